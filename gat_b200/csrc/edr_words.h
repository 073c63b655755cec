/* The choice of a DP cell on two 16-bit distances per 32-bit word (edr_kernel.cuh), for the device and, in
 * plain C++, for the host tests of its range.
 *
 * A half holds E + TOP / 2, E the column-shifted distance. Row r has |E| <= r, so with at most TOP / 2 rows every
 * half lies in [0, TOP], and only the last of them, row TOP / 2, reaches TOP itself. m == l is read from
 * (m ^ l) + (TOP - 1): with both below TOP the sum's TOP bit is clear exactly when m ^ l is 0. Where l is TOP the
 * XOR has that bit itself and the sum carries it out, so the word that holds row TOP / 2 (EXACT) adds
 * without the bit and joins it again. TOP is 0x8000 on the device: 16,384 rows. */
#pragma once

#if defined(__CUDACC__)
#define GAT_WORD_FN __device__ __forceinline__
#else
#define GAT_WORD_FN inline
#endif

namespace gat {
namespace edr {

#if defined(__CUDACC__)
GAT_WORD_FN unsigned add_u16x2(unsigned a, unsigned b) {
    unsigned d;
    asm("add.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
GAT_WORD_FN unsigned min_u16x2(unsigned a, unsigned b) {
    unsigned d;
    asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
/* min(a + 1, c) in both halves */
GAT_WORD_FN unsigned inc_min_u16x2(unsigned a, unsigned c) { return __viaddmin_u16x2(a, 0x00010001u, c); }
#else
GAT_WORD_FN unsigned add_u16x2(unsigned a, unsigned b) { return ((a + b) & 0xffffu) | (((a >> 16) + (b >> 16)) << 16); }
GAT_WORD_FN unsigned min_u16x2(unsigned a, unsigned b) {
    const unsigned lo = (a & 0xffffu) < (b & 0xffffu) ? a : b, hi = (a >> 16) < (b >> 16) ? a : b;
    return (lo & 0xffffu) | (hi & 0xffff0000u);
}
GAT_WORD_FN unsigned inc_min_u16x2(unsigned a, unsigned c) { return min_u16x2(add_u16x2(a, 0x00010001u), c); }
#endif

/* min(m, l), with the TOP bit set where m == l: no value is above it then, and the cell takes the value
 * above plus one. one: 1 (the device passes it as unknown, so that the sum is a multiply-add). */
template <unsigned TOP, bool EXACT>
GAT_WORD_FN unsigned min_or_top(unsigned m, unsigned l, unsigned one) {
    constexpr unsigned kTops = TOP * 0x00010001u, kRest = (TOP - 1u) * 0x00010001u;
    const unsigned x = m ^ l;
    if (EXACT) return min_u16x2(m, l) | (~(((x & kRest) + kRest) | x) & kTops);
    return min_u16x2(m, l) | (~(x * one + kRest) & kTops);
}

}  // namespace edr
}  // namespace gat
