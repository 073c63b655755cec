/* Point groups of an index: the structure the trajectory-id range scan reads (range_groups.cu).
 *
 * A group is a maximal run of index positions with one trajectory inside one leaf (Grid) or cell
 * (FSG). Both layouts keep a cell's points sorted by trajectory (Grid::addDatasetToGrid,
 * Grid.cpp:210-316; FSG.cpp:95-143), so a walk that re-enters a cell still has one group there:
 * on 1M walks of 200 points in cells ten steps wide a group holds about 17 points. Per group: the
 * trajectory, the first position and the exact box of the points. A query takes a group by its box
 * (inside: the walk is in the result; outside: it is not, by these points) and reads points only
 * where the box straddles the query's border.
 *
 * Grid: every node's record holds its box, the exact box of its points, its first child and a range
 * of ids: a leaf's groups, or for an inner node of at most kNodeIds distinct trajectories their
 * list, so that a node inside a query costs its distinct walks instead of its points. The lists
 * follow the groups' trajectories in one array. FSG: the first group of every cell.
 *
 * STIG: a leaf keeps its points in the order std::sort left them, so its groups are made on a copy of
 * the coordinates sorted by (leaf, trajectory); a leaf of 10,240 points then is about a hundred boxes.
 * The index's own arrays stay as the reference lays them out. MortonGrid: its Grid's groups and the
 * first group of every Morton cell.
 *
 * Derived like the point boxes (pbox.cu), after a build or a snapshot load, and not part of the
 * snapshot format. A Grid of 200M points: 270 MB beside 3.3 GB, and 2 ms of a 16 ms build (its point
 * boxes come from the groups, so the pass over the points that made them is gone). When the memory
 * for it is not there the index is left without groups and queries take the point scan. */
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>

#include "range_common.cuh"

namespace gat {
namespace {

constexpr int kTile = 4096; /* positions per block of the head passes */
constexpr int kWordsPerWarp = kTile / 32 / 8;

__global__ void k_leaf_starts(int n, const int32_t* __restrict__ child, const int32_t* __restrict__ beg,
                              const int32_t* __restrict__ end, uint32_t* bits) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        if ((!child || child[j] < 0) && beg[j] < end[j]) atomicOr(bits + (beg[j] >> 5), 1u << (beg[j] & 31));
}

/* bits holds the leaf starts on entry, every group's first position on exit; counts per tile */
__global__ void __launch_bounds__(256) k_heads(int64_t P, const int32_t* __restrict__ tid, uint32_t* bits, int64_t* cnt) {
    __shared__ int warp_cnt[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t w0 = (int64_t)blockIdx.x * (kTile / 32) + warp * kWordsPerWarp;
    int c = 0;
    /* all of the warp's loads in flight at once */
    int t[kWordsPerWarp];
#pragma unroll
    for (int w = 0; w < kWordsPerWarp; w++) {
        const int64_t i = (w0 + w) * 32 + lane;
        t[w] = i < P ? __ldg(tid + i) : -1;
    }
    const unsigned starts = lane < kWordsPerWarp && (w0 + lane) * 32 < P ? bits[w0 + lane] : 0u;
    int before = w0 > 0 && w0 * 32 <= P ? __ldg(tid + w0 * 32 - 1) : -1; /* the point before the word */
    unsigned mine = 0;
#pragma unroll
    for (int w = 0; w < kWordsPerWarp; w++) {
        int prev = __shfl_up_sync(0xffffffffu, t[w], 1);
        if (lane == 0) prev = before;
        before = __shfl_sync(0xffffffffu, t[w], 31);
        const unsigned word = __ballot_sync(0xffffffffu, (w0 + w) * 32 + lane < P && t[w] != prev) | __shfl_sync(0xffffffffu, starts, w);
        if (lane == w) mine = word;
        c += __popc(word);
    }
    if (lane < kWordsPerWarp && (w0 + lane) * 32 < P) bits[w0 + lane] = mine;
    if (lane == 0) warp_cnt[warp] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < 8; w++) t += warp_cnt[w];
        cnt[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(256) k_groups(int64_t P, const int32_t* __restrict__ tid, const uint32_t* __restrict__ bits,
                                                const int64_t* __restrict__ off, int32_t* gbeg, int32_t* ids) {
    __shared__ int warp_cnt[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t w0 = (int64_t)blockIdx.x * (kTile / 32) + warp * kWordsPerWarp;
    /* lane w holds word w of the warp's words */
    const unsigned mine = lane < kWordsPerWarp && (w0 + lane) * 32 < P ? bits[w0 + lane] : 0u;
    int incl = __popc(mine);
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_cnt[warp] = incl;
    __syncthreads();
    int base = (int)off[blockIdx.x];
    for (int w = 0; w < warp; w++) base += warp_cnt[w];
    const int excl = incl - __popc(mine);
    for (int w = 0; w < kWordsPerWarp; w++) {
        const unsigned word = __shfl_sync(0xffffffffu, mine, w);
        const int first = base + __shfl_sync(0xffffffffu, excl, w);
        if ((word >> lane) & 1u) {
            const int64_t i = (w0 + w) * 32 + lane;
            const int g = first + __popc(word & ((1u << lane) - 1u));
            gbeg[g] = (int32_t)i;
            ids[g] = __ldg(tid + i);
        }
    }
}

/* The exact box of every group's points (NaN when a coordinate is NaN: no comparison holds, so the
 * query tests the points). A warp takes 32 consecutive groups, whose points are one range; it
 * stages 512 of them at a time in shared memory with coalesced loads, each lane then folds the
 * part of its own group. */
constexpr int kStage = 512;
__global__ void __launch_bounds__(128) k_group_boxes(int G, const int32_t* __restrict__ gbeg, const float* __restrict__ X,
                                                     const float* __restrict__ Y, float4* box) {
    __shared__ float sx[4][kStage], sy[4][kStage];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inf = 0x7f800000;
    for (int g0 = (blockIdx.x * 4 + warp) * 32; g0 < G; g0 += gridDim.x * 128) {
        const int g = g0 + lane, b = gbeg[min(g, G)], e = gbeg[min(g + 1, G)];
        const int lo = __shfl_sync(0xffffffffu, b, 0), hi = __shfl_sync(0xffffffffu, e, 31);
        float4 v = make_float4(__int_as_float(inf), __int_as_float(inf), __int_as_float(inf | 0x80000000), __int_as_float(inf | 0x80000000));
        bool nan = false;
        for (int s = lo; s < hi; s += kStage) {
            const int n = min(kStage, hi - s);
            __syncwarp();
#pragma unroll
            for (int k0 = 0; k0 < kStage; k0 += 256) {
                float x[8], y[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int k = k0 + 32 * u + lane;
                    x[u] = k < n ? X[s + k] : 0.f;
                    y[u] = k < n ? Y[s + k] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    sx[warp][k0 + 32 * u + lane] = x[u];
                    sy[warp][k0 + 32 * u + lane] = y[u];
                }
            }
            __syncwarp();
            for (int k = max(b, s) - s; k < min(e, s + n) - s; k++) {
                const float x = sx[warp][k], y = sy[warp][k];
                nan |= (x != x) || (y != y);
                v.x = fminf(v.x, x);
                v.y = fminf(v.y, y);
                v.z = fmaxf(v.z, x);
                v.w = fmaxf(v.w, y);
            }
        }
        if (nan) v.x = v.y = v.z = v.w = __int_as_float(0x7fffffff);
        if (g < G) box[g] = v;
    }
}

/* the first group at or after position p (p is a group's first position, or the end) */
__device__ __forceinline__ int group_at(const int32_t* __restrict__ gbeg, int G, int p) {
    int lo = 0, hi = G;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (gbeg[mid] < p)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__global__ void k_cell_groups(int ncells, const int32_t* __restrict__ cbeg, int G, const int32_t* __restrict__ gbeg,
                              int32_t* cell_g) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncells; c += gridDim.x * blockDim.x)
        cell_g[c] = c < ncells ? group_at(gbeg, G, cbeg[c]) : G;
}

__device__ __forceinline__ float4 no_points() {
    return make_float4(__int_as_float(0x7f800000), __int_as_float(0x7f800000), __int_as_float(0xff800000),
                       __int_as_float(0xff800000));
}
__device__ __forceinline__ float4 join_boxes(const float4& a, const float4& b) {
    if (a.x != a.x || b.x != b.x) return make_float4(__int_as_float(0x7fffffff), 0.f, 0.f, 0.f);
    return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
}

/* Records of all nodes, a warp each; a leaf's ids and point box are final, an inner node's follow by level. (One
 * thread per node walked a crowded cell's groups in sequence: a Grid over 1M walks of which 30% of the points
 * stand at one place took 169 ms to build, 24.5 ms now.) */
__global__ void __launch_bounds__(256) k_node_records(GridDev t, int G, const int32_t* __restrict__ gbeg,
                                                      const float4* __restrict__ gbox, NodeRec* rec, float4* pbox) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < t.nnodes; j += (gridDim.x * blockDim.x) >> 5) {
        const int child = t.node_child[j], pb = t.node_pbeg[j], pe = t.node_pend[j];
        int ib = 0, ie = 0;
        float4 box = no_points();
        if (child < 0 && pb < pe) {
            ib = group_at(gbeg, G, pb);
            ie = group_at(gbeg, G, pe);
#pragma unroll 4
            for (int g = ib + lane; g < ie; g += 32) box = join_boxes(box, gbox[g]);
            for (int o = 16; o > 0; o >>= 1) {
                float4 b;
                b.x = __shfl_xor_sync(FULL, box.x, o);
                b.y = __shfl_xor_sync(FULL, box.y, o);
                b.z = __shfl_xor_sync(FULL, box.z, o);
                b.w = __shfl_xor_sync(FULL, box.w, o);
                box = join_boxes(box, b);
            }
        }
        if (lane == 0) {
            NodeRec r;
            r.mbb = t.node_mbb[j];
            r.pbox = box;
            r.child = child;
            r.ib = ib;
            r.ie = ie;
            r.aux = 0;
            rec[j] = r;
            pbox[j] = box;
        }
    }
}

/* level[l + 1] = the end of level l + 1 in the breadth-first order: the last child of level l */
__global__ void k_next_level(int l, const int32_t* __restrict__ child, int* level) {
    const int b = level[l], e = max(level[l + 1], b);
    int last = e;
    for (int j = b + blockIdx.x * blockDim.x + threadIdx.x; j < e; j += gridDim.x * blockDim.x)
        if (child[j] >= 0) last = max(last, child[j] + 4);
    for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&level[l + 2], last);
}

/* The node covering square (x, y) of the 2^L x 2^L squares, by descending L levels or to a leaf;
 * *bad is set when a node on the way is not wide against the coordinates' rounding (about 100 units
 * in the last place): the walk then starts at the root (walk_grid in range_groups.cu). */
__global__ void k_jump(int L, const NodeRec* __restrict__ rec, int32_t* jump, int* bad) {
    const int n = 1 << (2 * L);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int x = i & ((1 << L) - 1), y = i >> L;
        int nd = 0;
        for (int l = 0; l < L && rec[nd].child >= 0; l++) {
            nd = rec[nd].child + ((x >> (L - 1 - l)) & 1) + 2 * ((y >> (L - 1 - l)) & 1);
            const float4 m = rec[nd].mbb;
            if (!(m.z - m.x > 1e-5f * fmaxf(fabsf(m.x), fabsf(m.z))) || !(m.w - m.y > 1e-5f * fmaxf(fabsf(m.y), fabsf(m.w)))) *bad = 1;
        }
        jump[i] = nd;
    }
}

constexpr int kJumpLevel = 6;
constexpr int kSmallIds = 256; /* nodes whose children hold at most this many ids: one warp each */

/* the ids of a node's four children into the set; false when a child has no list */
template <int HB>
__device__ __forceinline__ void take_children(const NodeRec* __restrict__ rec, int child, const int32_t* ids, int first,
                                              int step, int* tab, int* list, int* cnt, int* ovf) {
    for (int c = 0; c < 4; c++) {
        const int b = rec[child + c].ib, e = rec[child + c].ie;
        for (int i = b + first; i < e; i += step) hs_insert<HB>(tab, list, ids[i], cnt, ovf);
    }
}

/* Inner nodes of one level, a warp each: point box, and the distinct ids of its children. Larger
 * nodes go on a list for k_big_lists. */
__global__ void __launch_bounds__(256) k_small_lists(int l, const int* __restrict__ level, NodeRec* rec, float4* pbox,
                                                     int32_t* ids, unsigned long long* cursor, unsigned long long cap,
                                                     int* big, int* nbig) {
    constexpr int HB = 9;
    __shared__ int tab[8][1 << HB], list[8][1 << (HB - 1)], cnt[8], ovf[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = lane; i < (1 << HB); i += 32) tab[warp][i] = -1;
    if (lane == 0) cnt[warp] = ovf[warp] = 0;
    __syncwarp();
    const int e = level[l + 1];
    for (int j = level[l] + blockIdx.x * 8 + warp; j < e; j += gridDim.x * 8) {
        const int child = rec[j].child;
        if (child < 0) continue;
        const int ib = rec[child + (lane & 3)].ib, n = rec[child + (lane & 3)].ie - ib;
        int total = n;
        total += __shfl_xor_sync(0xffffffffu, total, 1);
        total += __shfl_xor_sync(0xffffffffu, total, 2);
        const bool none = __any_sync(0xffffffffu, ib < 0);
        if (lane == 0) {
            const float4 b = join_boxes(join_boxes(rec[child].pbox, rec[child + 1].pbox),
                                        join_boxes(rec[child + 2].pbox, rec[child + 3].pbox));
            rec[j].pbox = b;
            pbox[j] = b;
        }
        if (none) {
            if (lane == 0) rec[j].ib = rec[j].ie = -1;
            continue;
        }
        if (total > kSmallIds) {
            if (lane == 0) big[atomicAdd(nbig, 1)] = j;
            continue;
        }
        take_children<HB>(rec, child, ids, lane, 32, tab[warp], list[warp], &cnt[warp], &ovf[warp]);
        __syncwarp();
        const int m = min(cnt[warp], 1 << (HB - 1));
        const bool lost = ovf[warp] != 0; /* a probe sequence ran out */
        unsigned long long at = 0;
        if (lane == 0 && !lost) at = atomicAdd(cursor, (unsigned long long)m);
        at = __shfl_sync(0xffffffffu, at, 0);
        const bool fits = !lost && at + m <= cap;
        if (fits)
            for (int i = lane; i < m; i += 32) ids[at + i] = list[warp][i];
        for (int i = lane; i < (1 << HB); i += 32) tab[warp][i] = -1;
        __syncwarp();
        if (lane == 0) {
            rec[j].ib = fits ? (int)at : -1;
            rec[j].ie = fits ? (int)(at + m) : -1;
            cnt[warp] = ovf[warp] = 0;
        }
        __syncwarp();
    }
}

/* The listed larger nodes, a block each; a node of more than kNodeIds distinct ids gets no list. */
__global__ void __launch_bounds__(256) k_big_lists(NodeRec* rec, int32_t* ids, unsigned long long* cursor,
                                                   unsigned long long cap, const int* __restrict__ big, const int* nbig) {
    constexpr int HB = 13;
    static_assert((1 << (HB - 1)) == kNodeIds, "the set holds a node's ids at half load");
    extern __shared__ int smem[];
    int* tab = smem;
    int* list = smem + (1 << HB);
    __shared__ int cnt, ovf;
    __shared__ unsigned long long at_sh;
    for (int k = blockIdx.x; k < *nbig; k += gridDim.x) {
        for (int i = threadIdx.x; i < (1 << HB); i += blockDim.x) tab[i] = -1;
        if (threadIdx.x == 0) cnt = ovf = 0;
        __syncthreads();
        const int j = big[k], child = rec[j].child;
        /* a child's own list already holds distinct ids, so four full ones cannot fit either */
        for (int c = 0; c < 4; c++) {
            const int b = rec[child + c].ib, e = rec[child + c].ie;
            for (int i = b + threadIdx.x; i < e; i += blockDim.x) {
                if (*(volatile int*)&ovf) break;
                hs_insert<HB>(tab, list, ids[i], &cnt, &ovf);
            }
        }
        __syncthreads();
        const int m = cnt;
        if (threadIdx.x == 0) at_sh = ovf ? cap : atomicAdd(cursor, (unsigned long long)m);
        __syncthreads();
        const unsigned long long at = at_sh;
        const bool fits = !ovf && at + m <= cap;
        if (fits)
            for (int i = threadIdx.x; i < m; i += blockDim.x) ids[at + i] = list[i];
        if (threadIdx.x == 0) {
            rec[j].ib = fits ? (int)at : -1;
            rec[j].ie = fits ? (int)(at + m) : -1;
        }
        __syncthreads();
    }
}

/* ---------------------------------------------------------------- STIG */
__global__ void k_leaf_sizes(StigDev t, int64_t* size) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < t.nnodes; j += gridDim.x * blockDim.x)
        size[j] = t.kind[j] ? t.hi[j] - t.lo[j] + 1 : 0;
}

/* entry e of leaf j: key (j, trajectory) and the point's position; neighbouring leaves share a point, so
 * there are more entries than points. The leaf's first entry is marked in `bits`. */
__global__ void k_leaf_entries(StigDev t, const int64_t* __restrict__ off, const int32_t* __restrict__ tid,
                               unsigned long long* key, int32_t* at, uint32_t* bits) {
    const int lane = threadIdx.x & 31;
    for (int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < t.nnodes; j += (gridDim.x * blockDim.x) >> 5) {
        const int64_t b = off[j], n = off[j + 1] - b;
        if (n <= 0) continue;
        if (lane == 0) atomicOr(bits + (b >> 5), 1u << (b & 31));
        for (int64_t k = lane; k < n; k += 32) {
            const int p = t.lo[j] + (int)k;
            key[b + k] = (unsigned long long)j << 32 | (unsigned)tid[p];
            at[b + k] = p;
        }
    }
}

__global__ void k_regroup(int64_t E, const unsigned long long* __restrict__ key, const int32_t* __restrict__ at,
                          const float* __restrict__ X, const float* __restrict__ Y, int32_t* tid, float* gx, float* gy) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        tid[e] = (int32_t)(key[e] & 0xffffffffull);
        gx[e] = X[at[e]];
        gy[e] = Y[at[e]];
    }
}

__global__ void k_stig_records(StigDev t, const int64_t* __restrict__ off, int G, const int32_t* __restrict__ gbeg, NodeRec* rec) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < t.nnodes; j += gridDim.x * blockDim.x) {
        NodeRec r;
        r.mbb = make_float4(t.median[j], 0.f, 0.f, 0.f);
        r.pbox = make_float4(0.f, 0.f, 0.f, 0.f);
        r.child = t.left[j];
        r.ib = r.ie = 0;
        r.aux = t.right[j] * 2 + t.dim[j];
        if (t.kind[j]) {
            r.mbb = t.mbb[j];
            r.pbox = t.pbox[j];
            r.child = -1;
            r.aux = 0;
            if (off[j] < off[j + 1]) {
                r.ib = group_at(gbeg, G, (int)off[j]);
                r.ie = group_at(gbeg, G, (int)off[j + 1]);
            }
        }
        rec[j] = r;
    }
}

int blocks_for(const gat_ctx* ctx, int64_t threads, int per = 256) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((threads + per - 1) / per, (int64_t)ctx->sm_count * 16));
}

/* device temporaries of one build, returned in stream order */
struct Temp {
    gat_ctx* ctx;
    cudaMemPool_t pool;
    std::vector<void*> p;
    explicit Temp(gat_ctx* c) : ctx(c), pool(build_pool(c)) {}
    Temp(const Temp&) = delete;
    ~Temp() {
        for (void* q : p) pool ? cudaFreeAsync(q, ctx->stream) : cudaFree(q);
    }
    template <class T>
    T* get(size_t n) {
        void* q = nullptr;
        const size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
        if ((pool ? cudaMallocFromPoolAsync(&q, bytes, pool, ctx->stream) : cudaMalloc(&q, bytes)) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        p.push_back(q);
        return static_cast<T*>(q);
    }
};

}  // namespace

void index_groups_free(gat_index* ix) {
    for (void* p : ix->group_allocs) cudaFree(p);
    ix->group_allocs.clear();
    ix->device_bytes -= ix->group_bytes;
    ix->group_bytes = 0;
    ix->groups = GroupsDev{};
}

int index_groups(gat_index* ix) {
    gat_ctx* ctx = ix->ctx;
    const bool grid = ix->kind == GAT_INDEX_GRID, stig = ix->kind == GAT_INDEX_STIG, morton = ix->kind == GAT_INDEX_MORTON;
    if (ctx->device < 0 || ix->npoints <= 0) return GAT_OK;
    if (morton && ix->base->groups.n == 0) return GAT_OK;
    cudaStream_t s = ctx->stream;
    auto dev = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (cudaMalloc(&p, std::max<size_t>(bytes, 16)) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        ix->group_allocs.push_back(p);
        ix->group_bytes += bytes;
        ix->device_bytes += bytes;
        return p;
    };
    /* no room: the index works without groups */
    auto without = [&]() {
        index_groups_free(ix);
        return GAT_OK;
    };
    if (morton) {
        GroupsDev g = ix->base->groups;
        const int ncells = ix->grid.cellnum;
        int32_t* cell_g = (int32_t*)dev((size_t)(ncells + 1) * 4);
        if (!cell_g) return without();
        k_cell_groups<<<blocks_for(ctx, ncells + 1), 256, 0, s>>>(ncells, ix->morton.cbeg, g.n, g.gbeg, cell_g);
        count_launch(ctx);
        GAT_CUDA_TRY(ctx, cudaGetLastError(), "point groups");
        GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
        g.cell_g = cell_g;
        ix->groups = g;
        return GAT_OK;
    }
    Temp tmp(ctx);
    GroupsDev g;
    int64_t P = ix->npoints; /* entries to group */
    const int32_t* tid = ix->d_tid;
    int64_t* leaf_off = nullptr;
    g.X = ix->d_x;
    g.Y = ix->d_y;
    if (stig) {
        if (int st = index_point_boxes(ix)) return st;
        const int n = ix->stig.nnodes;
        leaf_off = tmp.get<int64_t>((size_t)n + 1);
        if (!leaf_off) return without();
        k_leaf_sizes<<<blocks_for(ctx, n), 256, 0, s>>>(ix->stig, leaf_off);
        if (int st = scan_i64(ctx, leaf_off, leaf_off, n)) return st;
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_pinned, leaf_off + n, 8, cudaMemcpyDeviceToHost, s), "point groups");
        GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
        P = ctx->h_pinned[0];
    }
    if (P >= (int64_t)1 << 31) return without();
    const int64_t words = (P + 31) / 32, tiles = (P + kTile - 1) / kTile;
    uint32_t* bits = tmp.get<uint32_t>(words);
    int64_t* off = tmp.get<int64_t>(tiles + 1);
    if (!bits || !off) return without();
    GAT_CUDA_TRY(ctx, cudaMemsetAsync(bits, 0, words * 4, s), "point groups");
    if (stig) {
        const int n = ix->stig.nnodes;
        auto* key = tmp.get<unsigned long long>(P);
        auto* key_s = tmp.get<unsigned long long>(P);
        int32_t* at = tmp.get<int32_t>(P);
        int32_t* at_s = tmp.get<int32_t>(P);
        int32_t* etid = tmp.get<int32_t>(P);
        float* gx = (float*)dev((size_t)P * 4);
        float* gy = gx ? (float*)dev((size_t)P * 4) : nullptr;
        if (!key || !key_s || !at || !at_s || !etid || !gy) return without();
        k_leaf_entries<<<blocks_for(ctx, (int64_t)n * 32), 256, 0, s>>>(ix->stig, leaf_off, ix->d_tid, key, at, bits);
        int nbits = 32;
        while (nbits < 63 && ((int64_t)n >> (nbits - 32))) nbits++;
        size_t need = 0;
        GAT_CUDA_TRY(ctx, cub::DeviceRadixSort::SortPairs(nullptr, need, key, key_s, at, at_s, P, 0, nbits, s), "point groups");
        void* t = tmp.get<char>(need);
        if (!t) return without();
        GAT_CUDA_TRY(ctx, cub::DeviceRadixSort::SortPairs(t, need, key, key_s, at, at_s, P, 0, nbits, s), "point groups");
        k_regroup<<<blocks_for(ctx, P), 256, 0, s>>>(P, key_s, at_s, ix->d_x, ix->d_y, etid, gx, gy);
        count_launch(ctx, 3 + 2 * ((nbits + 7) / 8));
        tid = etid;
        g.X = gx;
        g.Y = gy;
    } else if (grid) {
        k_leaf_starts<<<blocks_for(ctx, ix->grid.nnodes), 256, 0, s>>>(ix->grid.nnodes, ix->grid.node_child, ix->grid.node_pbeg,
                                                                       ix->grid.node_pend, bits);
    } else {
        k_leaf_starts<<<blocks_for(ctx, ix->fsg.cellnum), 256, 0, s>>>(ix->fsg.cellnum, nullptr, ix->fsg.cbeg, ix->fsg.cend, bits);
    }
    k_heads<<<(unsigned)tiles, 256, 0, s>>>(P, tid, bits, off);
    if (int st = scan_i64(ctx, off, off, tiles)) return st;
    GAT_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_pinned, off + tiles, 8, cudaMemcpyDeviceToHost, s), "point groups");
    GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
    const int64_t total = ctx->h_pinned[0];
    const int G = (int)total;
    /* room for a Grid's node lists: each level holds at most as many ids as the one below, in practice
     * half as many until the nodes outgrow the walks; a node that does not fit goes without */
    const int64_t cap = std::min<int64_t>(grid ? total + total * 3 / 2 + 4096 : total, ((int64_t)1 << 31) - 2);
    /* all that is kept in one allocation: each costs the build 0.1 ms and more (an FSG over 20M points: 3.7 ms with one
     * per array, 2.9 now) */
    const int nodes_n = grid ? ix->grid.nnodes : stig ? ix->stig.nnodes : 0;
    if (grid) g.jump_level = std::min(kJumpLevel, ix->grid.total_level);
    const size_t per_node = (size_t)nodes_n * sizeof(NodeRec);
    const size_t cells = grid ? (size_t)1 << (2 * g.jump_level) : stig ? 0 : (size_t)ix->fsg.cellnum + 1;
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    char* mem = (char*)dev(up((size_t)total * 16) + up(per_node) + up((size_t)(total + 1) * 4) + up((size_t)cap * 4) + up(cells * 4));
    if (!mem) return without();
    auto part = [&](size_t bytes) {
        char* p = mem;
        mem += up(bytes);
        return p;
    };
    float4* gbox = (float4*)part((size_t)total * 16);
    NodeRec* rec = (NodeRec*)part(per_node);
    int32_t* gbeg = (int32_t*)part((size_t)(total + 1) * 4);
    int32_t* ids = (int32_t*)part((size_t)cap * 4);
    int32_t* cell_mem = (int32_t*)part(cells * 4); /* FSG: cell_g, Grid: jump */
    k_groups<<<(unsigned)tiles, 256, 0, s>>>(P, tid, bits, off, gbeg, ids);
    ctx->h_pinned[2] = P; /* the low word closes gbeg */
    GAT_CUDA_TRY(ctx, cudaMemcpyAsync(gbeg + total, ctx->h_pinned + 2, 4, cudaMemcpyHostToDevice, s), "point groups");
    k_group_boxes<<<blocks_for(ctx, total, 128), 128, 0, s>>>(G, gbeg, g.X, g.Y, gbox);
    count_launch(ctx, 4);
    g.n = G;
    g.gbeg = gbeg;
    g.ids = ids;
    g.gbox = gbox;
    if (ix->kind == GAT_INDEX_FSG) {
        k_cell_groups<<<blocks_for(ctx, ix->fsg.cellnum + 1), 256, 0, s>>>(ix->fsg.cellnum, ix->fsg.cbeg, G, gbeg, cell_mem);
        count_launch(ctx);
        g.cell_g = cell_mem;
    } else if (stig) {
        k_stig_records<<<blocks_for(ctx, ix->stig.nnodes), 256, 0, s>>>(ix->stig, leaf_off, G, gbeg, rec);
        count_launch(ctx);
        g.rec = rec;
    } else {
        const int n = ix->grid.nnodes, levels = ix->grid.total_level + 1;
        int* level = tmp.get<int>(levels + 3);
        int* big = tmp.get<int>((size_t)n + 1);
        unsigned long long* cursor = tmp.get<unsigned long long>(1);
        if (!level || !big || !cursor) return without();
        if (!ix->d_pbox) {
            GAT_CUDA_TRY(ctx, cudaMalloc(&ix->d_pbox, (size_t)n * sizeof(float4)), "point boxes");
            ix->device_bytes += (size_t)n * sizeof(float4);
        }
        k_node_records<<<blocks_for(ctx, (int64_t)n * 32), 256, 0, s>>>(ix->grid, G, gbeg, gbox, rec, ix->d_pbox);
        /* level l is [level[l], level[l + 1]); the root is level 0 */
        ctx->h_pinned[3] = 1;
        ctx->h_pinned[4] = total;
        GAT_CUDA_TRY(ctx, cudaMemsetAsync(level, 0, (size_t)(levels + 3) * 4, s), "point groups");
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(level + 1, ctx->h_pinned + 3, 4, cudaMemcpyHostToDevice, s), "point groups");
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(cursor, ctx->h_pinned + 4, 8, cudaMemcpyHostToDevice, s), "point groups");
        for (int l = 0; l + 1 < levels; l++)
            k_next_level<<<blocks_for(ctx, n, 1024), 256, 0, s>>>(l, ix->grid.node_child, level);
        constexpr size_t kBigSmem = (size_t)(2 * kNodeIds + kNodeIds) * 4;
        allow_smem(k_big_lists, kBigSmem);
        for (int l = levels - 1; l >= 0; l--) {
            const int64_t nodes = l < 15 ? std::min<int64_t>(n, (int64_t)1 << (2 * l)) : n;
            GAT_CUDA_TRY(ctx, cudaMemsetAsync(big + n, 0, 4, s), "point groups");
            k_small_lists<<<blocks_for(ctx, nodes, 8), 256, 0, s>>>(l, level, rec, ix->d_pbox, ids, cursor,
                                                                     (unsigned long long)cap, big, big + n);
            k_big_lists<<<(int)std::min<int64_t>(nodes, (int64_t)ctx->sm_count * 4), 256, kBigSmem, s>>>(
                rec, ids, cursor, (unsigned long long)cap, big, big + n);
        }
        int32_t* jump = cell_mem;
        GAT_CUDA_TRY(ctx, cudaMemsetAsync(big + n, 0, 4, s), "point groups");
        k_jump<<<16, 256, 0, s>>>(g.jump_level, rec, jump, big + n);
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_pinned + 5, big + n, 4, cudaMemcpyDeviceToHost, s), "point groups");
        GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
        if (*reinterpret_cast<int32_t*>(ctx->h_pinned + 5) == 0) g.jump = jump;
        count_launch(ctx, 2 + levels * 3);
        ix->grid.node_pbox = ix->d_pbox;
        g.rec = rec;
    }
    GAT_CUDA_TRY(ctx, cudaGetLastError(), "point groups");
    GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
    ix->groups = g;
    return GAT_OK;
}

}  // namespace gat
