/* The EDR wavefront kernel, shared by the pair API (edr.cu) and the top-k walk (topk.cu).
 *
 * Recurrence (Grid::SimilarityExecuter, Grid.cpp:1274-1306): with m = D[r-1][c-1] + subcost,
 * u = D[r-1][c] + 1, l = D[r][c-1] + 1, the reference takes m when m is below both others,
 * else l when l is below both others, else u. That is min(m, u, l) except when m == l, where
 * it is u (also when u is larger); the kernel evaluates exactly that. subcost is 0 when
 * |x1 - x2| < eps and |y1 - y2| < eps with float differences compared in double
 * (Grid.cpp:1281); the kernel compares the float |difference| with u_eps, the smallest float
 * not below eps, which is the same predicate. Orientation: rows are the query when the
 * candidate is at least as long, else the candidate (Grid.cpp:1234-1247).
 *
 * Three kernels: k_edr_rows (row tiles as work items, longest pairs first, consecutive tiles of a
 * pair pipelined across warps, two cells per 32-bit word; every caller but the next two),
 * k_edr_cols (column tiles, one cell per word; GAT_TUNE_EDR_FORM = 2) and k_edr (one warp per pair,
 * its tiles in sequence; the allocation-free entry point). Everything is integer arithmetic plus
 * float subtractions and compares for the match test.
 */
#pragma once
#include <algorithm>
#include <type_traits>

#include "edr_words.h"
#include "internal.h"
#include "launch.cuh"

namespace gat {
namespace edr {

constexpr int kWarps = 8; /* k_edr (one warp per pair) */
constexpr int kRowWarps = 16; /* k_edr_rows: one CTA per SM, 128 registers per thread */
template <int R>
constexpr int kColWarps = R == 8 ? 10 : 8; /* k_edr_cols */
constexpr int kBig = 1 << 29; /* above any distance; up + 1 never overflows against it */

/* Pair source over (a_off, a_len, b_off, b_len) arrays; results to out[p]. A pair with a side
 * outside 1..lim gets -1, raises GAT_ERR_ARG in the status word and runs as an empty problem
 * whose result goes to the sink word (flag + 1). */
struct SoaPairs {
    int npairs;
    const int* d_npairs;
    const int64_t* a_off;
    const int32_t* a_len;
    const int64_t* b_off;
    const int32_t* b_len;
    const float2* A;
    const float2* B;
    int32_t* out;
    int lim;
    int32_t* flag;
    static constexpr int kKind = 0;
    __device__ int count() const { return d_npairs ? *d_npairs : npairs; }
    /* whether the pair is known to share no match (the arrays carry no boxes) */
    __device__ bool apart(int, float) const { return false; }
    __device__ void get(int p, const float2*& a, int& la, const float2*& b, int& lb, int32_t*& o) const {
        la = a_len[p];
        lb = b_len[p];
        if (la < 1 || lb < 1 || la > lim || lb > lim) {
            out[p] = -1;
            atomicCAS(flag, 0, GAT_ERR_ARG);
            a = A;
            b = B;
            la = lb = 0;
            o = flag + 1;
            return;
        }
        a = A + a_off[p];
        b = B + b_off[p];
        o = out + p;
    }
};

template <int R, class Src>
__global__ void __launch_bounds__(kWarps * 32) k_edr(Src src, float u, int* __restrict__ carry, int carry_stride,
                                                     unsigned* __restrict__ work, unsigned long long* __restrict__ cells) {
    __shared__ float2 bring[kWarps][64];
    __shared__ int cring[kWarps][64];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = blockIdx.x * kWarps + wib;
    int* cbuf0 = carry + (size_t)gw * 2 * carry_stride;
    int* cbuf1 = cbuf0 + carry_stride;
    const int n = src.count();
    for (;;) {
        unsigned p = 0;
        if (lane == 0) p = atomicAdd(work, 1u);
        p = __shfl_sync(FULL, p, 0);
        if ((int)p >= n) break;
        const float2 *pa, *pb;
        int la, lb;
        int32_t* outp;
        src.get((int)p, pa, la, pb, lb, outp);
        const float2* rows;
        const float2* cols;
        int len1, len2;
        if (lb >= la) {
            rows = pa;
            cols = pb;
            len1 = la;
            len2 = lb;
        } else {
            rows = pb;
            cols = pa;
            len1 = lb;
            len2 = la;
        }
        int result;
        if (len1 == 0 || len2 == 0) {
            result = len1 + len2;
        } else {
            constexpr int kTile = 32 * R;
            const int ntiles = (len1 + kTile - 1) / kTile;
            const int last_row = len1 - 1;
            result = 0;
            for (int t = 0; t < ntiles; t++) {
                const int* cin = (t & 1) ? cbuf1 : cbuf0;
                int* cout = (t & 1) ? cbuf0 : cbuf1;
                const bool write_carry = t + 1 < ntiles;
                const int r0 = t * kTile + lane * R;
                float ax[R], ay[R];
                int left[R];
#pragma unroll
                for (int i = 0; i < R; i++) {
                    int r = r0 + i;
                    if (r < len1) {
                        float2 v = rows[r];
                        ax[i] = v.x;
                        ay[i] = v.y;
                    } else {
                        ax[i] = __int_as_float(0x7f800000); /* +inf never matches */
                        ay[i] = ax[i];
                    }
                    left[i] = r + 1; /* D[r+1][0] */
                }
                const bool owns_last = (last_row >= r0) && (last_row < r0 + R);
                const int last_i = last_row - r0;
                int diag_in = r0; /* D[r0][0] */
                int bottom = 0;
                const int steps = len2 + 31;
                for (int s = 0; s < steps; s++) {
                    if ((s & 31) == 0) {
                        __syncwarp();
                        int c = s + lane;
                        if (c < len2) {
                            bring[wib][c & 63] = cols[c];
                            cring[wib][c & 63] = t == 0 ? c + 1 : cin[c + 1];
                        }
                        __syncwarp();
                    }
                    const int from_above = __shfl_up_sync(FULL, bottom, 1);
                    const int j = s - lane;
                    if (j >= 0 && j < len2) {
                        const float2 b = bring[wib][j & 63];
                        const int upf = lane == 0 ? cring[wib][j & 63] : from_above;
                        /* Everything except the carry from the row above depends only on the
                         * previous column: with m = diag + subcost and l = left + 1, the
                         * reference's choice equals min(up + 1, mml) where mml = min(m, l),
                         * or +inf when m == l (then it takes up + 1 whatever the others are).
                         * The chain down the lane's rows is then one add-min per cell. */
                        int mml[R];
#pragma unroll
                        for (int i = 0; i < R; i++) {
                            const bool match = (fabsf(__fsub_rn(ax[i], b.x)) < u) & (fabsf(__fsub_rn(ay[i], b.y)) < u);
                            const int m = (i == 0 ? diag_in : left[i - 1]) + (match ? 0 : 1);
                            const int l = left[i] + 1;
                            mml[i] = (m == l) ? kBig : min(m, l);
                        }
                        int up = upf;
#pragma unroll
                        for (int i = 0; i < R; i++) {
                            up = __viaddmin_s32(up, 1, mml[i]);
                            left[i] = up;
                        }
                        bottom = up;
                        diag_in = upf;
                        if (write_carry && lane == 31) cout[j + 1] = bottom;
                        if (owns_last && j == len2 - 1) {
#pragma unroll
                            for (int i = 0; i < R; i++)
                                if (i == last_i) result = left[i];
                        }
                    }
                }
                __syncwarp();
            }
            /* the owner of the last row holds the answer */
            const int owner = (last_row % (32 * R)) / R;
            result = __shfl_sync(FULL, result, owner);
        }
        if (lane == 0) {
            *outp = result;
            if (cells) atomicAdd(cells, (unsigned long long)len1 * (unsigned long long)len2);
        }
    }
}

/* ================================================================ tiled, load-balanced form
 * Work items are row tiles. A pair whose rows span T >= 2 tiles contributes T items and its
 * tiles run on different warps, pipelined: tile t consumes the bottom row of tile t-1 through a
 * carry row in L2 while tile t-1 is still producing it. Pairs with one tile, and multi-tile
 * pairs beyond the cooperative pool, are one item that a single warp walks tile by tile with
 * its own carry rows.
 *
 * Carry words: each column's carry value is one 64-bit word, tag << 16 | (uint16) value, with
 * tag = launch epoch << 8 | producing tile (mod 256). The consumer polls the words it needs and
 * accepts a word whose tag is the one it expects, so the hand-over needs neither a progress
 * flag nor a memory fence: a 64-bit store is seen whole or not at all. Values are the
 * column-shifted distances E = D - c, which lie in [-16384, 16384] and fit 16 bits; epochs
 * come from a per-context device counter and only grow (2^40 launches before a repeat), and carry
 * buffers are zeroed when allocated, so a stale word never carries the expected tag. A tile rewrites the buffer its predecessor read
 * (double buffering per pair) only for columns that predecessor has already consumed.
 *
 * Schedule (longest first): a count pass puts every pair in one of kClasses duration classes
 * (half-octaves of the pair's critical path in column steps: len2 + 32 (T - 1) when its tiles
 * are pipelined, T (len2 + 31) on one warp) and a write pass lays the items out class by
 * class, longest class first, a pair's tiles consecutive. Warps take items in that order from
 * one counter, so the long pairs start first and the short ones fill in behind them.
 *
 * Waits are bounded: after kSpinLimit polls the warp raises GAT_ERR_TIMEOUT in the status word
 * and abandons the pair (its result becomes -1). The producer of the tile a warp waits for
 * took the preceding item from the same counter, so it is already running. */
constexpr int kSpinLimit = 1 << 22;
constexpr int kClasses = 48;
/* counter block: [0] item counter, [1] cooperative slots taken, [2] total items,
 * [4, 4 + kClasses) items per class, [4 + kClasses, 4 + 2 kClasses) class cursors, then the
 * launch's epoch (64-bit, 8-byte aligned) */
constexpr int kCtrEpoch = 4 + 2 * kClasses;
constexpr int kCtrWords = kCtrEpoch + 2;
typedef unsigned long long carry_t;

constexpr int kEdrCarveoutPct = 100; /* preferred shared-memory share of the SM for the tile kernels (launch_tiles) */

struct TileCtl {
    const int4* items; /* (pair, tile or -1 for a whole pair on one warp, cooperative slot, tiles) */
    const int* total;
    carry_t* pair_carry; /* cooperative slot s: rows pair_carry + s * 2 * stride */
    carry_t* warp_carry; /* per-warp double carry rows for single-warp pairs */
    int stride;
    const unsigned long long* epoch; /* written by the schedule's write pass */
    int32_t* flag;
    int spin_limit;  /* polls before a carry wait gives up (kSpinLimit) */
    int stall_pair;  /* tests of the bounded wait: this pair's first pipelined tile writes no carries (-1: none) */
    unsigned one;    /* 1, unknown to the compiler: x * one + c is a multiply-add on the FMA pipe (row_step) */
};

/* The carry word is the only datum exchanged, so neither access needs to order other memory
 * operations (no "memory" clobber: the step loop's shared-memory loads may move across them);
 * volatile keeps every poll a fresh load. */
__device__ __forceinline__ carry_t ld_carry(const carry_t* p) {
    carry_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_carry(carry_t* p, carry_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v));
}

/* floor(2 log2(d)) for d >= 1, clamped to the class range */
__device__ __forceinline__ int duration_class(long long d) {
    if (d < 1) d = 1;
    const int e = 63 - __clzll(d);
    const int half = (d * d >= (1LL << (2 * e + 1))) ? 1 : 0;
    return min(2 * e + half, kClasses - 1);
}

/* E of row r at column c when no point of the first r rows matches any of the first c columns.
 * Let k be the highest bit set in r and clear in c: E = (r mod 2^(k+1)) - (c mod 2^(k+1)), and 0
 * when there is no such bit. (The recurrence without matches depends on r and c alone. Row r has
 * period 2^(k+1) in c for 2^k <= r < 2^(k+1): over a period E falls r, r - 1, ..., r - 2^k + 1,
 * then repeats row r - 2^k from its start, where E = r - 2^k; by induction on r the rule m == l ->
 * u restarts the fall at each period, as m and l meet there.) */
__device__ __forceinline__ int unmatched_e(int r, int c) {
    const int x = r & ~c;
    if (x == 0) return 0;
    const int mask = (2 << (31 - __clz(x))) - 1;
    return (r & mask) - (c & mask);
}
/* Whether boxes a and b (x0, y0, x1, y1 of the points) are too far apart for any match: rounding is
 * monotone, so a difference of edges of at least u bounds every difference of points from below. False
 * when an edge is NaN. */
__device__ __forceinline__ bool boxes_apart(const float4& a, const float4& b, float u) {
    return __fsub_rn(b.x, a.z) >= u || __fsub_rn(a.x, b.z) >= u || __fsub_rn(b.y, a.w) >= u || __fsub_rn(a.y, b.w) >= u;
}

/* How a pair is cut: column tiles of 32 R columns, row tiles of 32 R rows (2H = R rows per lane),
 * the last row tile of the smallest height 64 h, h a power of two, that holds the rest. */
template <int R>
__device__ __forceinline__ int tile_count(int nlane) {
    return nlane <= 0 ? 1 : (nlane + 32 * R - 1) / (32 * R);
}

/* The count pass also answers the pairs whose boxes are apart (most candidates of a top-k walk are far
 * from the query): their distance is the lengths' alone (unmatched_e) and they take no item. */
template <int R, bool COL, class Src>
__global__ void k_sched_count(Src src, int cap, int coop_cap, int* __restrict__ ctr, int2* __restrict__ meta, float u,
                              unsigned long long* __restrict__ cells) {
    dep_wait();
    unsigned long long done = 0; /* cells of the pairs answered here */
    __shared__ int hist[kClasses];
    for (int i = threadIdx.x; i < kClasses; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int n = min(src.count(), cap);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float2 *a, *b;
        int la, lb;
        int32_t* o;
        src.get(p, a, la, b, lb, o);
        const int len1 = min(la, lb), len2 = max(la, lb);
        if (src.apart(p, u)) {
            *o = len2 + unmatched_e(len1, len2);
            done += (unsigned long long)len1 * (unsigned long long)len2;
            meta[p] = make_int2(-1, 0);
            continue;
        }
        const int nlane = COL ? len2 : len1, nstep = COL ? len1 : len2;
        const int T = tile_count<R>(nlane);
        int slot = -1, items = 1;
        if (T >= 2) {
            const int sl = atomicAdd(&ctr[1], 1);
            if (sl < coop_cap) {
                slot = sl;
                items = T;
            }
        }
        /* steps of the critical path: a row tile starts 96 steps behind its predecessor, a column
         * tile 32 */
        constexpr int kLag = COL ? 32 : 96, kRamp = COL ? 31 : 63;
        const long long dur = slot >= 0 ? (long long)nstep + (long long)kLag * (T - 1) : (long long)T * (nstep + kRamp);
        const int c = duration_class(dur);
        atomicAdd(&hist[c], items);
        meta[p] = make_int2(slot, (c << 16) | items);
    }
    if (cells) {
        for (int o = 16; o > 0; o >>= 1) done += __shfl_xor_sync(0xffffffffu, done, o);
        if ((threadIdx.x & 31) == 0 && done) atomicAdd(cells, done);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kClasses; i += blockDim.x)
        if (hist[i]) atomicAdd(&ctr[4 + i], hist[i]);
}

template <class Src>
__global__ void k_sched_write(Src src, int cap, int* __restrict__ ctr, const int2* __restrict__ meta,
                              int4* __restrict__ items, unsigned long long* __restrict__ epochs) {
    dep_wait();
    __shared__ int off[kClasses];
    __shared__ int lcnt[kClasses];
    __shared__ int lbase[kClasses];
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int c = kClasses - 1; c >= 0; c--) {
            off[c] = acc;
            acc += ctr[4 + c];
        }
        if (blockIdx.x == 0) {
            ctr[2] = acc;
            /* a fresh epoch per launch from the context's device counter, so launches replayed
             * from a CUDA graph never reuse a tag */
            *reinterpret_cast<unsigned long long*>(ctr + kCtrEpoch) = atomicAdd(epochs, 1ull) + 1ull;
        }
    }
    const int n = min(src.count(), cap);
    /* block-sized chunks (uniform trip count over the block) so the local counters reset */
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        for (int i = threadIdx.x; i < kClasses; i += blockDim.x) lcnt[i] = 0;
        __syncthreads();
        const int p = base + threadIdx.x;
        int c = 0, nit = 0, loc = 0, slot = -1;
        if (p < n) {
            const int2 m = meta[p];
            slot = m.x;
            c = m.y >> 16;
            nit = m.y & 0xffff;
            loc = atomicAdd(&lcnt[c], nit);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kClasses; i += blockDim.x)
            if (lcnt[i]) lbase[i] = atomicAdd(&ctr[4 + kClasses + i], lcnt[i]);
        __syncthreads();
        if (p < n) {
            const int pos = off[c] + lbase[c] + loc;
            if (nit == 0)
                ; /* answered by the count pass */
            else if (slot < 0)
                items[pos] = make_int4(p, -1, -1, 1);
            else
                for (int t = 0; t < nit; t++) items[pos + t] = make_int4(p, t, slot, nit);
        }
        __syncthreads();
    }
}

/* Match mask of one cell: -1 when |x1 - x2| < u and |y1 - y2| < u (float differences, no
 * contraction), else 0. */
__device__ __forceinline__ int match_mask(float ax, float ay, float2 b, float u) {
    const float dx = __fsub_rn(ax, b.x), dy = __fsub_rn(ay, b.y);
    int m;
    asm("{\n\t.reg .pred p;\n\t.reg .f32 t0, t1;\n\t"
        "abs.f32 t0, %1;\n\tabs.f32 t1, %2;\n\t"
        "setp.lt.f32 p, t0, %3;\n\t"
        "set.lt.and.s32.f32 %0, t1, %3, p;\n\t}"
        : "=r"(m)
        : "f"(dx), "f"(dy), "f"(u));
    return m;
}

/* ---------------------------------------------------------------- row tiles, two cells per word
 * The row form works on column-shifted distances E[r][c] = D[r][c] - c: in column c's shift the
 * reference's three operands at (r, c) become m = E[r-1][c-1] + (match ? -1 : 0), l = E[r][c-1]
 * and u = E[r-1][c] + 1; a common shift keeps every comparison, so the choice min(u, mml), with
 * mml = min(m, l) or +inf when m == l, is taken on shifted values unchanged.
 *
 * |E[r][c]| <= r (D <= c + r along the column boundary; D >= |r - c|), so with a bias of 16384 every
 * value of a supported pair lies in [0, 0x8000] and two of them share a 32-bit word (edr_words.h; the
 * last of 16,384 rows, where 0x8000 occurs, by row_tile_top). A lane owns
 * 2H consecutive rows: word i holds row i of the lane (low half) and row H + i (high half). The
 * high half runs one column behind the low half, and the next lane's low half one column behind
 * that, so the value above a half's first row is always one step old: the lane's own low bottom
 * row for the high half, the lane above's high bottom row (one shuffle) for the low half. At step
 * s lane L handles columns s - 2L (low) and s - 2L - 1 (high).
 *
 * What bounds it: the ALU pipe, at half the issue rate (16-bit min / add, min.f32, lop3 and prmt all
 * ran at 62 lanes per clock and SM on a B200, float adds at 117 and multiply-adds at 62 beside
 * them). Two cells take 8 ALU and 7 FMA-pipe instructions where a match is possible and 4 + 1 where
 * it is not, against 14 ALU and 4 FMA for two cells held one per word. Measured on 4,096 pairs of
 * log-uniform [16, 4096] lengths: 0.84 ms, 2.6 Tcell/s; one cell per word: 1.62 ms, 1.34 Tcell/s. */
constexpr int kBias = 16384;
constexpr unsigned kTop = 0x8000u; /* E + kBias of row kBias at column 0, and where its fall restarts */
static_assert(kBias == GAT_EDR_MAX_LEN && kTop == 2u * kBias && kBias % 256 == 0, "the last row of the longest side ends a tile");

/* Negative exactly when |dx| < u and |dy| < u: max propagates a NaN (no match, as the compares
 * have it), and a difference of unequal floats is never zero. */
__device__ __forceinline__ float match_sign(float dx, float dy, float u) {
    float t;
    asm("{\n\t.reg .f32 a, b;\n\tabs.f32 a, %1;\n\tabs.f32 b, %2;\n\tmax.NaN.f32 %0, a, b;\n\t}" : "=f"(t) : "f"(dx), "f"(dy));
    return __fsub_rn(t, u);
}
/* 0xffff in each half whose float is negative (prmt with replicated sign bits) */
__device__ __forceinline__ unsigned sign_halves(float lo, float hi) {
    unsigned d;
    asm("prmt.b32 %0, %1, %2, 0xffbb;" : "=r"(d) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
    return d;
}

__device__ __forceinline__ unsigned unmatched_pair(int rlo, int rhi, int c) {
    return (unsigned)(kBias + unmatched_e(rlo, c)) | (unsigned)(kBias + unmatched_e(rhi, c)) << 16;
}

/* A box of row points. near() is true when a column point may match one of them: rounding is
 * monotone, so a difference to the box's edge of at least u bounds the difference to every row
 * from below. NaN rows widen nothing (they match nothing), a NaN point is near nothing. */
struct RowBox {
    float x0, y0, x1, y1;
    __device__ __forceinline__ void clear() {
        x0 = y0 = __int_as_float(0x7f800000);
        x1 = y1 = __int_as_float(0xff800000);
    }
    __device__ __forceinline__ void add(float x, float y) {
        x0 = fminf(x0, x);
        y0 = fminf(y0, y);
        x1 = fmaxf(x1, x);
        y1 = fmaxf(y1, y);
    }
    __device__ __forceinline__ void add(const RowBox& o) {
        x0 = fminf(x0, o.x0);
        y0 = fminf(y0, o.y0);
        x1 = fmaxf(x1, o.x1);
        y1 = fmaxf(y1, o.y1);
    }
    __device__ __forceinline__ void warp_union() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
            y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
            y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
        }
    }
    __device__ __forceinline__ bool near(float2 p, float u) const {
        return (__fsub_rn(p.x, x1) < u) & (__fsub_rn(x0, p.x) < u) & (__fsub_rn(p.y, y1) < u) & (__fsub_rn(y0, p.y) < u);
    }
};

/* Where the distances of a row tile stop being unmatched_e: `mine` is the first column (rounded
 * down to 32) that may match one of the rows [0, r1), `above` the same for the rows [0, r0) above
 * the tile; both are kNever when there is none. Every value left of the first match of the rows
 * so far is known without any work, so a tile starts at `mine`, takes the values above its first
 * row from its predecessor from column `above` on and by formula before it, and a pair without a
 * possible match (most candidates of a top-k walk) costs one pass over its points. The tile above
 * evaluates the same rows and columns, so its `mine` is this tile's `above`. Called by a warp. */
constexpr int kNever = 1 << 30;
struct Front {
    int above, mine;
};
__device__ __forceinline__ Front row_front(const float2* __restrict__ rows, const float2* __restrict__ cols, int len2, int r0,
                                           int r1, float u) {
    const int lane = threadIdx.x & 31;
    RowBox up, all;
    up.clear();
#pragma unroll 4
    for (int i = lane; i < r0; i += 32) {
        const float2 v = rows[i];
        up.add(v.x, v.y);
    }
    all = up;
#pragma unroll 4
    for (int i = r0 + lane; i < r1; i += 32) {
        const float2 v = rows[i];
        all.add(v.x, v.y);
    }
    if (r0 > 0) up.warp_union();
    all.warp_union();
    Front f{kNever, kNever};
    for (int c0 = 0; c0 < len2; c0 += 128) {
        /* four loads in flight per lane */
        float2 p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = c0 + 32 * q + lane;
            p[q] = c < len2 ? cols[c] : make_float2(__int_as_float(0x7fffffff), 0.f);
        }
        bool done = false;
#pragma unroll
        for (int q = 3; q >= 0; q--)
            if (__any_sync(0xffffffffu, all.near(p[q], u))) done = true;
        if (!done) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (f.mine == kNever && __any_sync(0xffffffffu, all.near(p[q], u))) f.mine = c0 + 32 * q;
            if (r0 > 0 && f.above == kNever && __any_sync(0xffffffffu, up.near(p[q], u))) f.above = c0 + 32 * q;
        }
        if (r0 == 0 || f.above != kNever) break;
    }
    return f;
}

/* One step of a lane: up0 holds the values above its two halves' first rows, d0 the same one
 * column earlier. L[i] goes from column c - 1 to column c of its half, where `keep` (MASKED: the
 * halves whose column lies inside the pair) allows it. The choice is min_or_top's; EXACT for the tile
 * that holds row kBias. */
template <int H, bool MATCH, bool MASKED, bool EXACT>
__device__ __forceinline__ void row_step(const float (&ax)[2 * H], const float (&ay)[2 * H], unsigned (&L)[H], unsigned& d0,
                                         float2 blo, float2 bhi, unsigned up0, float u, unsigned one, unsigned keep) {
    unsigned mml[H];
#pragma unroll
    for (int i = 0; i < H; i++) {
        unsigned m = i == 0 ? d0 : L[i - 1];
        if (MATCH) {
            const float slo = match_sign(__fsub_rn(ax[i], blo.x), __fsub_rn(ay[i], blo.y), u);
            const float shi = match_sign(__fsub_rn(ax[H + i], bhi.x), __fsub_rn(ay[H + i], bhi.y), u);
            m = add_u16x2(m, sign_halves(slo, shi));
        }
        mml[i] = min_or_top<kTop, EXACT>(m, L[i], one);
    }
    unsigned up = up0;
#pragma unroll
    for (int i = 0; i < H; i++) {
        up = inc_min_u16x2(up, mml[i]);
        if (MASKED)
            L[i] = (up & keep) | (L[i] & ~keep);
        else
            L[i] = up;
    }
    d0 = MASKED ? (up0 & keep) | (d0 & ~keep) : up0;
}

/* Per-warp shared memory of a row tile: the window of 96 column points (at the start of the chunk of
 * steps [s0, s0 + 32): columns s0 - 64 .. s0 + 31), the chunk's carry values (in the high half) and
 * the bottom-row words lane 31 leaves during the chunk. */
struct RowShared {
    float4 pts[48]; /* two points each */
    uint4 in[8], out[8];
};

/* Stores four words to shared memory where `on` is set: predicated, and without a memory clobber, so
 * that the compiler neither branches around it nor orders the next loads of the window behind it
 * (they never touch these words; a warp barrier follows the last store of a chunk). */
__device__ __forceinline__ void put_words(unsigned addr, const unsigned (&v)[4], bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p st.shared.v4.u32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"((int)on),
                 "r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
}

/* The first `kend` steps (rounded up to 4) of one chunk. Four steps at a time: their points and
 * carry values come in 128-bit shared loads, their bottom-row words leave in one store. UN groups of
 * four are unrolled: two where the kernel holds the loops of one or two tile heights, one where it
 * holds three, since warps in loops that do not fit the instruction cache together wait for
 * instructions (4,096 pairs of log-uniform [16, 4096] lengths, 8 rows per lane: 0.85 ms with one
 * group, 1.03 ms with two; 4 rows: 0.94 and 0.91 ms). */
template <int H, int UN, bool MATCH, bool MASKED, bool EXACT>
__device__ __forceinline__ void row_chunk(const float (&ax)[2 * H], const float (&ay)[2 * H], unsigned (&L)[H], unsigned& d0,
                                          RowShared& sh, int s0, int kend, int c0, int len2, bool writer, float u,
                                          unsigned one) {
    const int lane = threadIdx.x & 31;
    const float4* pb = sh.pts + 32 - lane; /* the lane's low column of step k: point k of pb */
    float2 bhi = make_float2(0.f, 0.f);
    if (MATCH) bhi = reinterpret_cast<const float2*>(pb)[-1];
    const int groups = MASKED ? (kend + 3) >> 2 : 8;
    const unsigned out = (unsigned)__cvta_generic_to_shared(sh.out);
    constexpr int kUnroll = MASKED ? 1 : UN;
#pragma unroll(kUnroll)
    for (int g = 0; g < groups; g++) {
        float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
        if (MATCH) {
            p0 = pb[2 * g];
            p1 = pb[2 * g + 1];
        }
        const uint4 in = sh.in[g];
        const float2 b[4] = {make_float2(p0.x, p0.y), make_float2(p0.z, p0.w), make_float2(p1.x, p1.y), make_float2(p1.z, p1.w)};
        const unsigned cv[4] = {in.x, in.y, in.z, in.w};
        unsigned o[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned above = __shfl_up_sync(0xffffffffu, L[H - 1], 1);
            const unsigned up0 = __byte_perm(lane == 0 ? cv[k] : above, L[H - 1], 0x5432);
            unsigned keep = 0xffffffffu;
            if (MASKED) {
                const int j = s0 + 4 * g + k - 2 * lane;
                keep = (j >= c0 && j < len2 ? 0xffffu : 0u) | (j > c0 && j <= len2 ? 0xffff0000u : 0u);
            }
            row_step<H, MATCH, MASKED, EXACT>(ax, ay, L, d0, b[k], bhi, up0, u, one, keep);
            bhi = b[k];
            o[k] = L[H - 1];
        }
        put_words(out + 16 * g, o, writer);
    }
}

/* One row tile of one pair: the 64H rows of the shorter side from t0 on, steps over the columns from the
 * tile's front on. cin: the carry words of tile t-1's bottom row (used from column fr.above on),
 * accepted with tag tag_in; cout: this tile's bottom row for tile t+1 (nullptr for the last tile),
 * written with tag tag_out. Returns false when a wait gave up. The owner lane of the pair's last
 * row leaves the distance in `result`. The next chunk's points and carry words are loaded one
 * chunk early. A chunk none of whose columns is near the tile's rows (their box) takes the steps
 * without the match test: 29% of the chunks over pairs of log-uniform [16, 4096] lengths that follow
 * one another, nearly all over a top-k walk's candidates. */
template <int H, int UN, bool EXACT>
__device__ __forceinline__ bool row_tile(const float2* __restrict__ rows, const float2* __restrict__ cols, int len1, int len2,
                                      int t0, Front fr, const carry_t* cin, carry_t* cout, carry_t tag_in, carry_t tag_out,
                                      float u, RowShared& sh, int& result, int spin_limit, unsigned one) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool writer = cout != nullptr && lane == 31;
    const int r0 = t0 + lane * 2 * H; /* the lane's first row */
    const int c0 = fr.mine;
    float ax[2 * H], ay[2 * H];
    RowBox box;
    box.clear();
#pragma unroll
    for (int i = 0; i < 2 * H; i++) {
        ax[i] = ay[i] = __int_as_float(0x7f800000); /* +inf never matches */
        if (r0 + i < len1) {
            const float2 v = rows[r0 + i];
            ax[i] = v.x;
            ay[i] = v.y;
            box.add(v.x, v.y);
        }
    }
    box.warp_union();
    unsigned L[H];
#pragma unroll
    for (int i = 0; i < H; i++) L[i] = unmatched_pair(r0 + i + 1, r0 + H + i + 1, c0);
    unsigned d0 = unmatched_pair(r0, r0 + H, c0);
    const int steps = len2 + 63;
    const carry_t tag_hi = tag_out << 16;
    const int from = cin ? fr.above : kNever; /* first column whose value above comes from cin */
    float2 nb = make_float2(0.f, 0.f);
    /* The next chunk's carry word as loaded; its tag is looked at when that chunk starts, never beside
     * the load, where the compare would hold the warp for an L2 round trip in every chunk (two tiles of
     * 64 rows over 16,384 columns: 95 cycles a step with the compare there, 82 without; chunks without
     * matches 78 and 64). A load later in the chunk's loop, closer to its use, shortens the lag between
     * tiles but costs more: the loop waits for it (95 again), and the loop cut in two for it does not
     * stay in the instruction cache (4,096 pairs of mid length, 4 rows a lane: 0.166 -> 0.193 ms). */
    carry_t nw = 0; /* no tag is 0: epochs start at 1 */
    if (c0 + lane < len2) {
        nb = cols[c0 + lane];
        if (c0 + lane >= from) nw = ld_carry(cin + c0 + lane + 1);
    }
    float2* pts = reinterpret_cast<float2*>(sh.pts);
    unsigned near = 0; /* bit 0: this chunk holds a near column, bits 1 and 2: the two before */
    for (int s0 = c0; s0 < steps; s0 += 32) {
        const int c = s0 + lane;
        near = (near << 1) & 7u;
        if (s0 < len2) {
            unsigned cv = s0 < from ? (unsigned)(kBias + unmatched_e(t0, c + 1)) : 0u;
            if (s0 + 31 >= from) {
                const bool want = c >= from && c < len2;
                bool ok = !want || (nw >> 16) == tag_in;
                for (int polls = 0;; polls++) {
                    if (!ok) {
                        nw = ld_carry(cin + c + 1);
                        ok = (nw >> 16) == tag_in;
                    }
                    if (__all_sync(FULL, ok)) break;
                    if (polls >= spin_limit) return false;
                    if (polls >= 16) __nanosleep(64); /* each poll is an L2 round trip already */
                }
                if (want) cv = (unsigned)nw & 0xffffu;
            }
            near |= __any_sync(FULL, c < len2 && box.near(nb, u)) ? 1u : 0u;
            __syncwarp();
            pts[lane] = pts[32 + lane];
            pts[32 + lane] = pts[64 + lane];
            pts[64 + lane] = nb;
            reinterpret_cast<unsigned*>(sh.in)[lane] = cv << 16;
            __syncwarp();
            const int cn = c + 32;
            if (cn < len2) {
                nb = cols[cn];
                if (cn >= from) nw = ld_carry(cin + cn + 1);
            }
        } else {
            __syncwarp();
            pts[lane] = pts[32 + lane];
            pts[32 + lane] = pts[64 + lane];
            __syncwarp();
        }
        if (s0 >= c0 + 64 && s0 + 32 <= len2) {
            /* both columns of every lane lie in [c0, len2) throughout */
            if (EXACT || near)
                row_chunk<H, UN, true, false, EXACT>(ax, ay, L, d0, sh, s0, 32, c0, len2, writer, u, one);
            else
                row_chunk<H, UN, false, false, EXACT>(ax, ay, L, d0, sh, s0, 32, c0, len2, writer, u, one);
        } else {
            const int kend = min(32, steps - s0);
            row_chunk<H, UN, true, true, EXACT>(ax, ay, L, d0, sh, s0, kend, c0, len2, writer, u, one);
        }
        if (cout) {
            /* lane 31's high half was at column s0 + k - 63 in step k */
            __syncwarp();
            const int j = s0 + lane - 63;
            if (j >= c0 && j < len2) st_carry(cout + (j + 1), tag_hi | (carry_t)(reinterpret_cast<const unsigned*>(sh.out)[lane] >> 16));
        }
    }
    const int last = len1 - 1 - r0;
    if (last >= 0 && last < 2 * H) {
#pragma unroll
        for (int i = 0; i < 2 * H; i++)
            if (i == last) result = (int)(i < H ? L[i] & 0xffffu : L[i - H] >> 16) - kBias + len2; /* D = E + column */
    }
    __syncwarp();
    return true;
}

/* The tile that holds row kBias (the last one of a pair whose shorter side has that many points): a
 * function of its own, so that its loops stay out of the kernel's. One chunk form less: it always
 * tests for matches. */
struct TileEnd {
    bool ok;
    int result;
};
template <int H>
__device__ __noinline__ TileEnd row_tile_top(const float2* rows, const float2* cols, int len1, int len2, int t0, int above,
                                             int mine, const carry_t* cin, carry_t tag_in, float u, RowShared* sh,
                                             int spin_limit) {
    TileEnd e{false, 0};
    e.ok = row_tile<H, 1, true>(rows, cols, len1, len2, t0, Front{above, mine}, cin, nullptr, tag_in, 0, u, *sh, e.result,
                                spin_limit, 1u);
    return e;
}

/* Column-tile form of the same recurrence: a lane owns R consecutive DP columns and a step
 * advances one DP row r. Values are held shifted by their row: F[r][c] = D[r][c] - r, so in
 * row r's shift u = F[r-1][c] needs no add, m = F[r-1][c-1] + (match ? -1 : 0) and
 * l = F[r][c-1] + 1, whose chain runs along the lane's columns: with mm1 = m - 1 and
 * prev = F[r][c-1], m == l exactly when mm1 == prev, min(m, l) = min(mm1, prev) + 1, and the
 * cell is u when they are equal, else min(u, min(m, l)). State per column j: F[j] =
 * F[r-1][c_j] on entry, F[r][c_j] on exit; diag0 = F[r-1][c_0 - 1]; left = F[r][c_0 - 1] (the
 * value to the left of the lane's first column). Returns the value in the last column. */
template <int R>
__device__ __forceinline__ int cf_step(const float (&bx)[R], const float (&by)[R], int (&F)[R], int& diag0, float2 a,
                                       int left, float u) {
    int prev = left;
    int diag = diag0;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const int up = F[j];
        const int mm1 = diag + match_mask(bx[j], by[j], a, u) - 1;
        const int mn = min(mm1, prev);
        const int d = (mm1 == prev) ? up : __viaddmin_s32(mn, 1, up);
        diag = up;
        F[j] = d;
        prev = d;
    }
    diag0 = left;
    return prev;
}

/* One column tile of one pair: lanes own the columns lpts[t * 32R ..], steps walk the rows spts. cin:
 * the carry words of tile t-1's last column (nullptr for t == 0), accepted with tag tag_in; cout:
 * this tile's last column for tile t+1 (nullptr for the last tile), written with tag tag_out.
 * Returns false when a wait gave up. The owner lane of the pair's last column leaves the distance
 * in `result`.
 *
 * Step points move through a per-warp window of 64 points in shared memory: at the start of the
 * chunk of steps [s0, s0 + 32) the window holds points s0 - 32 .. s0 + 31, so lane L reads point
 * s0 + k - L of step k at window index 32 + k - L (a per-lane base plus a constant). The next
 * chunk's points and carry words are loaded one chunk early. Chunks where every lane's point is
 * inside the pair skip the bounds test. */
template <int R>
__device__ __forceinline__ bool col_tile(const float2* __restrict__ rows, const float2* __restrict__ cols, int len1,
                                         int len2, int t, const carry_t* cin, carry_t* cout, carry_t tag_in,
                                         carry_t tag_out, float u, float2* sb, int* sc, int& result,
                                         int spin_limit) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool lane0 = lane == 0;
    const bool writer = cout != nullptr && lane == 31;
    constexpr int kTile = 32 * R;
    const int r0 = t * kTile + lane * R;
    float ax[R], ay[R];
    int Lp[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int r = r0 + i;
        if (r < len1) {
            const float2 v = rows[r];
            ax[i] = v.x;
            ay[i] = v.y;
        } else {
            ax[i] = __int_as_float(0x7f800000); /* +inf never matches */
            ay[i] = ax[i];
        }
        Lp[i] = r + 1; /* E[r+1][0] = D[r+1][0] */
    }
    int diag0 = r0; /* E[r0][0] */
    int bottom = 0;
    const float2* pb = sb + 32 - lane;
    const int steps = len2 + 31;
    const carry_t tag_hi = tag_out << 16;
    /* prefetched inputs of the next chunk: column point and carry word of column s0 + lane */
    float2 nb = make_float2(0.f, 0.f);
    carry_t nw = 0;
    bool nw_ok = false;
    if (lane < len2) {
        nb = cols[lane];
        if (cin) {
            nw = ld_carry(cin + lane + 1);
            nw_ok = (nw >> 16) == tag_in;
        }
    }
    for (int s0 = 0; s0 < steps; s0 += 32) {
        const int c = s0 + lane;
        if (s0 < len2) {
            int cv = 0; /* E[0][c+1] = D[0][c+1] - (c+1) for the first tile */
            if (cin) {
                bool ok = c >= len2 || nw_ok;
                for (int polls = 0;; polls++) {
                    if (!ok) {
                        nw = ld_carry(cin + c + 1);
                        ok = (nw >> 16) == tag_in;
                    }
                    if (__all_sync(FULL, ok)) break;
                    if (polls >= spin_limit) return false;
                    if (polls >= 16) __nanosleep(64); /* each poll is an L2 round trip already */
                }
                cv = (int)(short)(nw & 0xffffu);
            }
            __syncwarp();
            sb[lane] = sb[32 + lane];
            sb[32 + lane] = nb;
            sc[lane] = cv;
            __syncwarp();
            /* next chunk */
            const int cn = c + 32;
            nw_ok = false;
            if (cn < len2) {
                nb = cols[cn];
                if (cin) {
                    nw = ld_carry(cin + cn + 1);
                    nw_ok = (nw >> 16) == tag_in;
                }
            }
        } else {
            __syncwarp();
            sb[lane] = sb[32 + lane];
            __syncwarp();
        }
        if (s0 >= 32 && s0 + 32 <= len2) {
            /* every lane's column s0 + k - lane lies in [1, len2) */
#pragma unroll 8
            for (int k = 0; k < 32; k++) {
                const int from_above = __shfl_up_sync(FULL, bottom, 1);
                const int up0 = lane0 ? sc[k] : from_above;
                bottom = cf_step<R>(ax, ay, Lp, diag0, pb[k], up0, u);
                if (writer) st_carry(cout + (s0 + k - 30), tag_hi | (carry_t)(unsigned short)bottom);
            }
        } else {
            const int kend = min(32, steps - s0);
            for (int k = 0; k < kend; k++) {
                const int from_above = __shfl_up_sync(FULL, bottom, 1);
                const int j = s0 + k - lane;
                if (j >= 0 && j < len2) {
                    const int up0 = lane0 ? sc[k] : from_above;
                    bottom = cf_step<R>(ax, ay, Lp, diag0, pb[k], up0, u);
                    if (writer) st_carry(cout + (j + 1), tag_hi | (carry_t)(unsigned short)bottom);
                }
            }
        }
    }
    const int last_i = len1 - 1 - r0;
    if (last_i >= 0 && last_i < R) {
#pragma unroll
        for (int i = 0; i < R; i++)
            if (i == last_i) result = Lp[i] + len2; /* D = E + column */
    }
    __syncwarp();
    return true;
}

/* The work items of one warp: orients each pair (rows are the query when the candidate is at least
 * as long, else the candidate, Grid.cpp:1234-1247) and hands the tile to `run`, which returns
 * whether its waits succeeded and leaves the distance in the owner lane's `result` (owner < 0: in
 * every lane) when it finished the pair. */
template <class Src, class Run>
__device__ __forceinline__ void walk_tiles(const Src& src, const TileCtl& ctl, unsigned* work, unsigned long long* cells,
                                           Run run) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned total = (unsigned)*ctl.total;
    for (;;) {
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(work, 1u);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= total) break;
        const int4 it = ctl.items[idx];
        const float2 *pa, *pb;
        int la, lb;
        int32_t* outp;
        src.get(it.x, pa, la, pb, lb, outp);
        const bool swap = lb < la;
        const float2 *rows = swap ? pb : pa, *cols = swap ? pa : pb;
        const int len1 = swap ? lb : la, len2 = swap ? la : lb;
        if (len1 == 0) {
            if (lane == 0) *outp = len2;
            continue;
        }
        int result = 0, owner = -1;
        bool finished = false;
        if (!run(it, rows, cols, len1, len2, result, owner, finished)) {
            if (lane == 0) {
                atomicCAS(ctl.flag, 0, GAT_ERR_TIMEOUT);
                *outp = -1;
            }
            continue;
        }
        if (finished) {
            if (owner >= 0) result = __shfl_sync(FULL, result, owner);
            if (lane == 0) {
                *outp = result;
                if (cells) atomicAdd(cells, (unsigned long long)len1 * (unsigned long long)len2);
            }
        }
    }
}

/* Row tiles of at most 32 R rows (R = 2, 4 or 8 rows per lane). */
constexpr int kSpread = 500; /* cycles between the first items of a CTA's warps (below) */

template <int R, class Src>
__global__ void __launch_bounds__(kRowWarps * 32, 1) k_edr_rows(Src src, float u, TileCtl ctl, unsigned* __restrict__ work,
                                                                unsigned long long* __restrict__ cells) {
    dep_wait();
    __shared__ RowShared shared[kRowWarps];
    const int wib = threadIdx.x >> 5;
    RowShared& sh = shared[wib];
    carry_t* wc0 = ctl.warp_carry + (size_t)(blockIdx.x * kRowWarps + wib) * 2 * ctl.stride;
    const carry_t ep = *ctl.epoch << 8;
    /* Warp w of every CTA asks for its first item about w * kSpread cycles after the start, so the
     * first items go to the first warps of all SMs, the next to the second warps, and a launch with
     * fewer items than warps (a few long pairs) spreads over the SMs and their four schedulers
     * instead of filling the SMs that start first. A delay, not a rule: whichever warp comes takes
     * the next item, so a tile's predecessor has always been taken before it. */
    for (const long long start = clock64(); clock64() - start < (long long)wib * kSpread;) __nanosleep(20);
    walk_tiles(src, ctl, work, cells, [&](const int4& it, const float2* rows, const float2* cols, int len1, int len2,
                                          int& result, int& owner, bool& finished) {
        constexpr int kHeight = 32 * R;
        constexpr int kGroups = R == 8 ? 1 : 2; /* row_chunk's unrolled groups */
        const int T = tile_count<R>(len1);
        const bool pipelined = it.y >= 0;
        carry_t* buf = pipelined ? ctl.pair_carry + (size_t)it.z * 2 * ctl.stride : wc0;
        finished = !pipelined || it.y == T - 1;
        for (int t = pipelined ? it.y : 0; t < (pipelined ? it.y + 1 : T); t++) {
            const int t0 = t * kHeight, left = len1 - t0;
            const Front fr = row_front(rows, cols, len2, t0, min(len1, t0 + kHeight), u);
            if (fr.mine == kNever) {
                /* no match so far: known values below this tile too */
                result = len2 + unmatched_e(len1, len2);
                owner = -1;
                continue;
            }
            const carry_t* cin = t > 0 ? buf + (size_t)((t - 1) & 1) * ctl.stride : nullptr;
            const bool stalled = pipelined && it.x == ctl.stall_pair && t == 0;
            carry_t* cout = t + 1 < T && !stalled ? buf + (size_t)(t & 1) * ctl.stride : nullptr;
            const carry_t tin = ep | ((t - 1) & 0xff), tout = ep | (t & 0xff);
            bool ok = false;
            auto tile = [&](auto half) {
                constexpr int H = decltype(half)::value;
                if constexpr (2 * H <= R) {
                    ok = row_tile<H, kGroups, false>(rows, cols, len1, len2, t0, fr, cin, cout, tin, tout, u, sh, result, ctl.spin_limit, ctl.one);
                    owner = (left - 1) / (2 * H); /* the last tile's */
                }
            };
            if (len1 == kBias && t == T - 1) {
                /* full: kBias is a multiple of every tile height */
                const TileEnd e = row_tile_top<R / 2>(rows, cols, len1, len2, t0, fr.above, fr.mine, cin, tin, u, &sh, ctl.spin_limit);
                ok = e.ok;
                result = e.result;
                owner = 31;
            } else if (left <= 64 || R == 2)
                tile(std::integral_constant<int, 1>{});
            else if (left <= 128 || R == 4)
                tile(std::integral_constant<int, 2>{});
            else
                tile(std::integral_constant<int, 4>{});
            if (!ok) return false;
        }
        return true;
    });
}

/* Column tiles of 32 R columns. What bounds few pairs is the chain of a step's cells: with 8 columns a lane and 24
 * warps per SM (80 registers) values of the chain spilled, 64 x 16,384 points took 0.82 ms. Two CTAs of ten warps
 * (92 registers) take 0.68 ms, 64 pairs of 1 x 16,384 points 0.49 (two of eight warps: 0.56), and 4,096 pairs of
 * log-uniform [16, 4096] lengths 1.56 ms (24 warps: 1.69). */
template <int R, class Src>
__global__ void __launch_bounds__(kColWarps<R> * 32, R == 2 ? 4 : R == 4 ? 3 : 2) k_edr_cols(Src src, float u, TileCtl ctl,
                                                                              unsigned* __restrict__ work,
                                                                              unsigned long long* __restrict__ cells) {
    dep_wait();
    __shared__ float2 bring[kColWarps<R>][64];
    __shared__ int cring[kColWarps<R>][32];
    const int wib = threadIdx.x >> 5;
    carry_t* wc0 = ctl.warp_carry + (size_t)(blockIdx.x * kColWarps<R> + wib) * 2 * ctl.stride;
    const carry_t ep = *ctl.epoch << 8;
    walk_tiles(src, ctl, work, cells, [&](const int4& it, const float2* rows, const float2* cols, int len1, int len2,
                                          int& result, int& owner, bool& finished) {
        const int T = tile_count<R>(len2);
        const bool pipelined = it.y >= 0;
        carry_t* buf = pipelined ? ctl.pair_carry + (size_t)it.z * 2 * ctl.stride : wc0;
        finished = !pipelined || it.y == T - 1;
        owner = ((len2 - 1) % (32 * R)) / R;
        for (int t = pipelined ? it.y : 0; t < (pipelined ? it.y + 1 : T); t++) {
            const bool stalled = pipelined && it.x == ctl.stall_pair && t == 0;
            if (!col_tile<R>(cols, rows, len2, len1, t, t > 0 ? buf + (size_t)((t - 1) & 1) * ctl.stride : nullptr,
                             t + 1 < T && !stalled ? buf + (size_t)(t & 1) * ctl.stride : nullptr, ep | ((t - 1) & 0xff),
                             ep | (t & 0xff), u, bring[wib], cring[wib], result, ctl.spin_limit))
                return false;
        }
        return true;
    });
}

template <int R, bool COL, class Src>
struct TileKernel {
    static constexpr int kWarps = kRowWarps;
    static constexpr auto get() { return k_edr_rows<R, Src>; }
};
template <int R, class Src>
struct TileKernel<R, true, Src> {
    static constexpr int kWarps = kColWarps<R>;
    static constexpr auto get() { return k_edr_cols<R, Src>; }
};

/* Host side: schedule (count, write) -> tiled kernel. cap is the number of pairs (exact for
 * host-known lists, an upper bound for device-counted ones); max_rows / max_cols bound the
 * shorter / longer side of every pair. ev0/ev1, when given, bracket the tile kernel. */
template <int R, bool COL, class Src>
int launch_tiles(gat_ctx* ctx, const Src& src, int64_t cap, int max_rows, int max_cols, float u,
                 unsigned long long* cells, cudaEvent_t ev0 = nullptr, cudaEvent_t ev1 = nullptr) {
    int st = GAT_OK;
    cudaStream_t s = ctx->stream;
    int per_sm = 0;
    /* An SM's split between L1 and shared memory changes only while no block is resident on it, so a
     * persistent grid that leaves room on its SMs and asks for no split keeps out the blocks of other streams
     * that need more shared memory, until it ends: range batches beside a long top-k round waited for it (16
     * rectangles, 1.1 ms alone: 10.5 ms median beside 18 ms EDR launches that left half the SMs free; 2.5 ms with
     * the largest split; measured with CTAs of 256 threads, 5 KB each, and range blocks of 48 KB). It holds for
     * the column kernel. A CTA of the row kernel takes all 65,536 registers of its SM: beside it only the SMs
     * that the grid leaves (sm_reserve) are free. The tile kernels read their points once and use little L1. */
    constexpr auto kernel = TileKernel<R, COL, Src>::get();
    constexpr int kWarps = TileKernel<R, COL, Src>::kWarps;
    prefer_split(reinterpret_cast<const void*>(kernel), ctx->device, kEdrCarveoutPct);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarps * 32, 0);
    /* a serving lane leaves sm_reserve SMs free of this persistent grid for other streams */
    const int grid = std::max(1, ctx->sm_count - ctx->sm_reserve) * (per_sm > 0 ? per_sm : 1);
    /* carry rows run along the step side; tiles are cut along the lane side */
    const int max_lane = COL ? max_cols : max_rows, max_step = COL ? max_rows : max_cols;
    const int stride = max_step + 2;
    const int maxT = max_lane <= 0 ? 1 : (max_lane + 32 * R - 1) / (32 * R);
    const size_t budget = (size_t)512 << 20; /* cooperative carry rows */
    int64_t coop = (int64_t)(budget / ((size_t)2 * stride * sizeof(carry_t)));
    if (coop > cap) coop = cap;
    if (maxT < 2) coop = 0;
    const int64_t item_cap = cap + coop * (maxT - 1);
    if (item_cap >= (int64_t)1 << 31) return fail(ctx, GAT_ERR_ARG, "edr: too many work items in one launch");
    int* ctr = (int*)scratch(ctx, S_EDR_COUNTERS, kCtrWords * sizeof(int), &st);
    int2* meta = (int2*)scratch(ctx, S_EDR_META, (size_t)cap * sizeof(int2), &st);
    int4* items = (int4*)scratch(ctx, S_EDR_ITEMS, (size_t)item_cap * sizeof(int4), &st);
    carry_t* pcarry =
        coop > 0 ? (carry_t*)scratch_zeroed(ctx, S_EDR_PCARRY, (size_t)coop * 2 * stride * sizeof(carry_t), &st) : nullptr;
    carry_t* wcarry = (carry_t*)scratch_zeroed(ctx, S_EDR_CARRY, (size_t)grid * kWarps * 2 * stride * sizeof(carry_t), &st);
    if (!ctr || !meta || !items || !wcarry || (coop > 0 && !pcarry)) return st;
    (void)launch_dep(ctx, k_zero_words, dim3(1), dim3(256), 0, s, ctr, (int)kCtrWords);
    const int pgrid = (int)std::max<int64_t>(1, std::min<int64_t>((cap + 255) / 256, (int64_t)ctx->sm_count * 8));
    (void)launch_dep(ctx, k_sched_count<R, COL, Src>, dim3(pgrid), dim3(256), 0, s, src, (int)cap, (int)coop, ctr, meta, u,
                     cells);
    count_launch(ctx);
    (void)launch_dep(ctx, k_sched_write<Src>, dim3(pgrid), dim3(256), 0, s, src, (int)cap, ctr, meta, items, edr_epochs(ctx));
    count_launch(ctx);
    /* the stall knob (tests of the bounded wait) also shortens the wait to ~2^12 polls */
    const int stall = ctx->test_stall_pair - 1;
    TileCtl ctl{items, ctr + 2, pcarry, wcarry, stride, reinterpret_cast<const unsigned long long*>(ctr + kCtrEpoch),
                ctx->d_flag, stall >= 0 ? (1 << 12) : kSpinLimit, stall, 1u};
    /* serving lanes: after the previous EDR grid of any sibling lane (not inside a capture, whose
     * graph cannot wait on an event recorded outside it) */
    std::unique_lock<std::mutex> chain;
    if (ctx->edr_chain) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(s, &cs);
        if (cs == cudaStreamCaptureStatusNone) {
            chain = std::unique_lock<std::mutex>(ctx->edr_chain->mu);
            GAT_CUDA_TRY(ctx, cudaStreamWaitEvent(s, ctx->edr_chain->ev, 0), "edr chain");
        }
    }
    timed_begin(ctx, GAT_KERNEL_EDR);
    if (ev0) cudaEventRecord(ev0, s);
    (void)launch_dep(ctx, kernel, dim3(grid), dim3(kWarps * 32), 0, s, src, u, ctl, reinterpret_cast<unsigned*>(ctr), cells);
    if (ev1) cudaEventRecord(ev1, s);
    timed_end(ctx, GAT_KERNEL_EDR, 0.0);
    if (chain.owns_lock()) GAT_CUDA_TRY(ctx, cudaEventRecord(ctx->edr_chain->ev, s), "edr chain");
    count_launch(ctx);
    GAT_CUDA_TRY(ctx, cudaGetLastError(), "edr launch");
    return GAT_OK;
}

/* Tile shapes: rows (or columns) per lane 2, 4, 8, in row or column form. shape = R | COL << 4 */
constexpr int kShapeCol = 16;

template <class Src>
int launch_shape(gat_ctx* ctx, int shape, const Src& src, int64_t cap, int max_rows, int max_cols, float u,
                 unsigned long long* cells, cudaEvent_t ev0 = nullptr, cudaEvent_t ev1 = nullptr) {
    switch (shape) {
        case 2: return launch_tiles<2, false, Src>(ctx, src, cap, max_rows, max_cols, u, cells, ev0, ev1);
        case 4: return launch_tiles<4, false, Src>(ctx, src, cap, max_rows, max_cols, u, cells, ev0, ev1);
        case 8: return launch_tiles<8, false, Src>(ctx, src, cap, max_rows, max_cols, u, cells, ev0, ev1);
        case 2 | kShapeCol: return launch_tiles<2, true, Src>(ctx, src, cap, max_rows, max_cols, u, cells, ev0, ev1);
        case 8 | kShapeCol: return launch_tiles<8, true, Src>(ctx, src, cap, max_rows, max_cols, u, cells, ev0, ev1);
        default: return launch_tiles<4, true, Src>(ctx, src, cap, max_rows, max_cols, u, cells, ev0, ev1);
    }
}

inline uint64_t ceil_log2(int64_t v) {
    uint64_t e = 0;
    while (e < 62 && ((int64_t)1 << e) < v) e++;
    return e;
}

/* Column tiles pay for a few pairs with a side of a handful of points: a row tile then walks the longer side on
 * one warp whatever it holds (16,384 columns 0.50 ms), while the longer side's 64 column tiles are short. One
 * pair of 1, 8, 16 and 64 x 16,384 points: 0.35, 0.43, 0.51 and 0.68 ms by columns of 8 a lane; 64 pairs of
 * 1 x 16,384: 0.49 ms and 0.51 ms by rows, and beyond kColPairs pairs their tiles no longer run at one time
 * (256 pairs of 16 x 16,384: 1.7 ms, rows 0.55). They are timed when no pair has a second tile of 64 rows. */
constexpr int kColPairs = 64;

/* EDR over a pair source with the context's tile shape. Rows per lane (GAT_TUNE_EDR_ROWS) and
 * form (GAT_TUNE_EDR_FORM) are fixed by the knobs or autotuned: the first launch of a shape
 * class times the open candidates on this launch's own pairs (every candidate writes the same
 * results; the cell counter is fed once) and records the fastest; later launches of the class
 * use it. */
template <class Src>
int edr_launch(gat_ctx* ctx, const Src& src, int64_t cap, int max_rows, int max_cols, float u,
               unsigned long long* cells) {
    if (cap <= 0) return GAT_OK;
    int cand[4], nc = 0;
    for (int r : {8, 4, 2}) {
        if (ctx->edr_rows && ctx->edr_rows != r) continue;
        cand[nc++] = r | (ctx->edr_form == 2 ? kShapeCol : 0);
    }
    const bool columns = ctx->edr_form == 0 && ctx->edr_rows == 0 && cap <= kColPairs;
    if (columns) cand[nc++] = 8 | kShapeCol;
    if (nc == 1) return launch_shape(ctx, cand[0], src, cap, max_rows, max_cols, u, cells);
    const uint64_t key = ((uint64_t)Src::kKind << 60) | ((uint64_t)(ctx->edr_rows | ctx->edr_form << 4) << 52) |
                         (ceil_log2(cap) << 40) | (ceil_log2(max_rows) << 20) | ceil_log2(max_cols);
    /* worker contexts share their parent's table (one tuning per shape class per device) */
    gat_ctx* tab = ctx->root ? ctx->root : ctx;
    {
        std::lock_guard<std::mutex> lk(tab->tune_mu);
        auto hit = tab->edr_tune.find(key);
        if (hit != tab->edr_tune.end()) {
            const int shape = hit->second;
            return launch_shape(ctx, shape, src, cap, max_rows, max_cols, u, cells);
        }
    }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        if (e0) cudaEventDestroy(e0);
        cudaGetLastError();
        return launch_shape(ctx, cand[0], src, cap, max_rows, max_cols, u, cells);
    }
    int best = cand[0], st = GAT_OK;
    float best_ms = 0.f;
    for (int i = 0; i < nc && st == GAT_OK; i++) {
        if (columns && i == nc - 1) {
            /* the items of the launch before, in tiles of 64 rows */
            int* items = reinterpret_cast<int*>(ctx->h_pinned + 20);
            if (cudaMemcpyAsync(items, (const int*)ctx->slot_ptr[S_EDR_COUNTERS] + 2, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream) !=
                    cudaSuccess ||
                cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
                st = cuda_fail(ctx, cudaGetLastError(), "edr autotune");
                break;
            }
            if (*items > cap) break;
        }
        st = launch_shape(ctx, cand[i], src, cap, max_rows, max_cols, u, i == 0 ? cells : nullptr, e0, e1);
        if (st != GAT_OK) break;
        float ms = 0.f;
        if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
            st = cuda_fail(ctx, cudaGetLastError(), "edr autotune");
            break;
        }
        if (i == 0 || ms < best_ms) {
            best_ms = ms;
            best = cand[i];
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st == GAT_OK) {
        std::lock_guard<std::mutex> lk(tab->tune_mu);
        tab->edr_tune[key] = best;
    }
    return st;
}

}  // namespace edr
}  // namespace gat
