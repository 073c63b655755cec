"""The packed EDR cells' word arithmetic on the host, at limits where every value of its range occurs."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cpp") / "edr_words")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "gat_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "edr_words.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    return exe


# limit, rows, columns, match matrices (0: every one); rows up to the limit, more columns than that too
@pytest.mark.parametrize("limit,rows,cols,count", [(2, 2, 2, 0), (2, 2, 5, 0), (4, 3, 5, 0), (4, 4, 4, 0), (4, 4, 13, 20000),
                                                   (8, 7, 30, 5000), (8, 8, 8, 20000), (8, 8, 30, 5000), (16, 16, 16, 5000),
                                                   (16, 16, 50, 2000)])
def test_every_cell(words, limit, rows, cols, count):
    r = subprocess.run([words, str(limit), str(rows), str(cols), str(count)], capture_output=True, text=True, check=True)
    rule, plain = map(int, r.stdout.split())
    assert rule == 0
    # the form without the exact step is wrong only with a row at the limit, which is why the rule names that row
    assert (plain > 0) == (rows == limit)
