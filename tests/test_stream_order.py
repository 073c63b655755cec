"""Every context works on a stream of its own that is not ordered with the legacy default stream. A copy or a
memset on the latter may return before its data has arrived, so a kernel of the context that follows it
would read what is not there yet: device memory is written in the order of a stream that the call names."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gat_b200", "csrc")


def _calls(text, name):
    """The argument lists of the calls of `name`, comments left out."""
    text = re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)
    for m in re.finditer(r"\b%s\s*\(" % name, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_device_memory_is_written_in_stream_order():
    bad = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        bad += [f"{name}: cudaMemset({a})" for a in _calls(text, "cudaMemset")]
        # a copy to the host is complete when it returns
        bad += [f"{name}: cudaMemcpy({a})" for a in _calls(text, "cudaMemcpy") if not a.rstrip().endswith("cudaMemcpyDeviceToHost")]
    assert not bad, "\n".join(bad)
