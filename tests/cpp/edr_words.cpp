/* The word arithmetic of the packed EDR cells (edr_words.h) against the recurrence, cell by cell, at a small
 * limit: argv = limit (TOP = 2 limit), rows, columns, matrices (0: every one). Two match matrices share the words,
 * one in the low halves and one in the high halves. The tile of the last `limit / 2` rows takes the exact form when
 * it holds row `limit`, as in the kernel. Prints the cells that differ, by the kernel's rule and without the
 * exact form. */
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "edr_words.h"

using namespace gat::edr;

/* E of every cell of a rows x cols problem, by 32-bit values */
static std::vector<int> recurrence(const std::vector<char>& match, int rows, int cols) {
    std::vector<int> D((rows + 1) * (cols + 1));
    auto at = [&](int r, int c) -> int& { return D[r * (cols + 1) + c]; };
    for (int c = 0; c <= cols; c++) at(0, c) = c;
    for (int r = 1; r <= rows; r++) {
        at(r, 0) = r;
        for (int c = 1; c <= cols; c++) {
            const int m = at(r - 1, c - 1) + (match[(r - 1) * cols + c - 1] ? 0 : 1), u = at(r - 1, c) + 1, l = at(r, c - 1) + 1;
            at(r, c) = m < u && m < l ? m : l < m && l < u ? l : u;
        }
    }
    for (int r = 0; r <= rows; r++)
        for (int c = 0; c <= cols; c++) at(r, c) -= c;
    return D;
}

template <unsigned TOP>
static int wrong_cells(const std::vector<char>& a, const std::vector<char>& b, int rows, int cols, bool by_rule) {
    const int limit = TOP / 2, bias = limit;
    const std::vector<int> ea = recurrence(a, rows, cols), eb = recurrence(b, rows, cols);
    std::vector<unsigned> W((rows + 1) * (cols + 1));
    auto at = [&](int r, int c) -> unsigned& { return W[r * (cols + 1) + c]; };
    auto both = [&](int e) { return (unsigned)(e + bias) * 0x00010001u; };
    int wrong = 0;
    for (int c = 0; c <= cols; c++) at(0, c) = both(0);
    for (int r = 1; r <= rows; r++) {
        at(r, 0) = both(r);
        const bool exact = by_rule && rows == limit && r > limit / 2;
        for (int c = 1; c <= cols; c++) {
            const int i = (r - 1) * cols + c - 1;
            const unsigned hit = (a[i] ? 0xffffu : 0u) | (b[i] ? 0xffff0000u : 0u);
            const unsigned m = add_u16x2(at(r - 1, c - 1), hit), l = at(r, c - 1);
            const unsigned mml = exact ? min_or_top<TOP, true>(m, l, 1u) : min_or_top<TOP, false>(m, l, 1u);
            at(r, c) = inc_min_u16x2(at(r - 1, c), mml);
            const int k = r * (cols + 1) + c;
            wrong += (int)(at(r, c) & 0xffffu) - bias != ea[k];
            wrong += (int)(at(r, c) >> 16) - bias != eb[k];
        }
    }
    return wrong;
}

template <unsigned TOP>
static void run(int rows, int cols, long count) {
    const int cells = rows * cols;
    const bool all = count == 0;
    if (all) count = 1l << cells;
    std::mt19937 rng(17);
    long rule = 0, plain = 0;
    std::vector<char> a(cells), b(cells);
    for (long k = 0; k < count; k++) {
        const unsigned density = rng() % 9 + 1;
        for (int i = 0; i < cells; i++) {
            a[i] = all ? (k >> i) & 1 : rng() % 10 < density;
            b[i] = all ? ((count - 1 - k) >> i) & 1 : rng() % 10 < 10 - density;
        }
        rule += wrong_cells<TOP>(a, b, rows, cols, true);
        plain += wrong_cells<TOP>(a, b, rows, cols, false);
    }
    printf("%ld %ld\n", rule, plain);
}

int main(int argc, char** argv) {
    if (argc != 5) return 2;
    const int limit = atoi(argv[1]), rows = atoi(argv[2]), cols = atoi(argv[3]);
    const long count = atol(argv[4]);
    if (limit == 2)
        run<4>(rows, cols, count);
    else if (limit == 4)
        run<8>(rows, cols, count);
    else if (limit == 8)
        run<16>(rows, cols, count);
    else if (limit == 16)
        run<32>(rows, cols, count);
    else
        return 2;
    return 0;
}
