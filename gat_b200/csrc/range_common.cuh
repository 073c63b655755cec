/* Device helpers shared by the range kernels (range.cu, range_groups.cu) and the builder of the
 * per-trajectory point groups (groups.cu): the reference's box predicates, the shared-memory id set
 * and the warp sorts. */
#pragma once

#include "internal.h"

namespace gat {

struct Box {
    float xmin, ymin, xmax, ymax;
};

__device__ __forceinline__ bool in_box(const Box& q, float x, float y) {
    /* MBB::pInBox (MBB.cpp:21-26) */
    return x <= q.xmax && x >= q.xmin && y <= q.ymax && y >= q.ymin;
}

/* BoxIntersect (MBB.cpp:28-73) reduced to its zero / non-zero outcome, the only use the
 * traversals make of it. */
__device__ __forceinline__ bool box_intersect(const Box& a1, const Box& b1) {
    Box a, b;
    if (a1.xmin < b1.xmin) {
        a = a1;
        b = b1;
    } else if (a1.xmin == b1.xmin) {
        if (a1.xmax > b1.xmax) {
            a = a1;
            b = b1;
        } else {
            b = a1;
            a = b1;
        }
    } else {
        b = a1;
        a = b1;
    }
    if (b.xmin >= a.xmax) return false;
    if (b.ymax <= a.ymin) return false;
    if (b.ymin >= a.ymax) return false;
    return true;
}

__device__ __forceinline__ Box load_box(const gat_mbb* q, int i) {
    gat_mbb m = q[i];
    return Box{m.xmin, m.ymin, m.xmax, m.ymax};
}

__device__ __forceinline__ void set_flag(int32_t* flag, int code) { atomicCAS(flag, 0, code); }

/* a node box strictly inside the query (see grid_walk in range.cu) */
__device__ __forceinline__ bool box_inside(const Box& q, const float4& m) {
    return q.xmin < m.x && m.z < q.xmax && q.ymin < m.y && m.w < q.ymax;
}

constexpr int kRankSortMax = 512; /* lists up to this length are sorted by run ranks */
template <int HB>
__device__ __forceinline__ unsigned hs_slot(int t) { return ((unsigned)t * 2654435761u) >> (32 - HB); }

/* inserts t; a new id is appended to list (count: ids inserted; ovf: the list or a probe ran out) */
template <int HB>
__device__ __forceinline__ void hs_insert(int* tab, int* list, int t, int* count, int* ovf) {
    unsigned h = hs_slot<HB>(t);
    for (int p = 0; p < 64; p++) {
        int v = tab[h];
        if (v == t) return;
        if (v == -1) {
            v = atomicCAS(&tab[h], -1, t);
            if (v == -1) {
                const int pos = atomicAdd(count, 1);
                if (pos < (1 << (HB - 1)))
                    list[pos] = t;
                else
                    *ovf = 1;
                return;
            }
            if (v == t) return;
        }
        h = (h + 1) & ((1u << HB) - 1);
    }
    *ovf = 1;
}

/* empties the slot holding t (t is in the set) */
template <int HB>
__device__ __forceinline__ void hs_erase(int* tab, int t) {
    unsigned h = hs_slot<HB>(t);
    for (int p = 0; p < (1 << HB); p++) {
        if (tab[h] == t) {
            tab[h] = -1;
            return;
        }
        h = (h + 1) & ((1u << HB) - 1);
    }
}

/* ascending sort of the 32 values of a warp (one per lane), bitonic network over shuffles */
__device__ __forceinline__ int warp_sort32(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int o = __shfl_xor_sync(0xffffffffu, v, j);
            const bool up = (lane & k) == 0;
            const bool lower = (lane & j) == 0;
            v = (lower == up) ? min(v, o) : max(v, o);
        }
    return v;
}

/* number of the 32 ascending values run[0..32) below x: a binary search over the first 31
 * (it leaves lo = how many of them are below x), then the last */
__device__ __forceinline__ int lower_bound32(const int* run, int x) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
        if (run[lo + step - 1] < x) lo += step;
    return lo + (run[31] < x ? 1 : 0);
}

}  // namespace gat
