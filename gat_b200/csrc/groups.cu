/* Point groups of a Grid or FSG: the structure the trajectory-id range scan reads (range_groups.cu).
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
 * Derived like the point boxes (pbox.cu), after a build or a snapshot load, and not part of the
 * snapshot format. On 200M points: about 360 MB (the points take 3.2 GB). When the memory for it
 * is not there the index is left without groups and queries take the point scan. */
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
#pragma unroll 4
    for (int w = 0; w < kWordsPerWarp; w++) {
        const int64_t i = (w0 + w) * 32 + lane;
        const int t = i < P ? __ldg(tid + i) : -1;
        int prev = __shfl_up_sync(0xffffffffu, t, 1);
        if (lane == 0) prev = i > 0 && i < P ? __ldg(tid + i - 1) : -1;
        unsigned word = __ballot_sync(0xffffffffu, i < P && t != prev);
        if ((w0 + w) * 32 >= P) break;
        word |= bits[w0 + w];
        __syncwarp();
        if (lane == 0) bits[w0 + w] = word;
        c += __popc(word);
    }
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
#pragma unroll 4
            for (int k = lane; k < n; k += 32) {
                sx[warp][k] = X[s + k];
                sy[warp][k] = Y[s + k];
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

__global__ void k_cell_groups(int ncells, const int32_t* __restrict__ cbeg, const int32_t* __restrict__ cend, int G,
                              const int32_t* __restrict__ gbeg, int32_t* cell_g) {
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

/* records of all nodes; a leaf's ids and point box are final, an inner node's follow by level */
__global__ void k_node_records(GridDev t, int G, const int32_t* __restrict__ gbeg, const float4* __restrict__ gbox,
                               NodeRec* rec, float4* pbox) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < t.nnodes; j += gridDim.x * blockDim.x) {
        NodeRec r;
        r.mbb = t.node_mbb[j];
        r.child = t.node_child[j];
        r.ib = r.ie = 0;
        r.pbox = no_points();
        r.pad = 0;
        if (r.child < 0 && t.node_pbeg[j] < t.node_pend[j]) {
            r.ib = group_at(gbeg, G, t.node_pbeg[j]);
            r.ie = group_at(gbeg, G, t.node_pend[j]);
            for (int g = r.ib; g < r.ie; g++) r.pbox = join_boxes(r.pbox, gbox[g]);
        }
        rec[j] = r;
        pbox[j] = r.pbox;
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
    const int64_t P = ix->npoints;
    const bool grid = ix->kind == GAT_INDEX_GRID;
    if (ctx->device < 0 || P <= 0 || P >= (int64_t)1 << 31 || (!grid && ix->kind != GAT_INDEX_FSG)) return GAT_OK;
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
    Temp tmp(ctx);
    const int64_t words = (P + 31) / 32, tiles = (P + kTile - 1) / kTile;
    uint32_t* bits = tmp.get<uint32_t>(words);
    int64_t* off = tmp.get<int64_t>(tiles + 1);
    if (!bits || !off) return without();
    GAT_CUDA_TRY(ctx, cudaMemsetAsync(bits, 0, words * 4, s), "point groups");
    if (grid)
        k_leaf_starts<<<blocks_for(ctx, ix->grid.nnodes), 256, 0, s>>>(ix->grid.nnodes, ix->grid.node_child, ix->grid.node_pbeg,
                                                                       ix->grid.node_pend, bits);
    else
        k_leaf_starts<<<blocks_for(ctx, ix->fsg.cellnum), 256, 0, s>>>(ix->fsg.cellnum, nullptr, ix->fsg.cbeg, ix->fsg.cend, bits);
    k_heads<<<(unsigned)tiles, 256, 0, s>>>(P, ix->d_tid, bits, off);
    if (int st = scan_i64(ctx, off, off, tiles)) return st;
    int64_t total = 0;
    GAT_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_pinned, off + tiles, 8, cudaMemcpyDeviceToHost, s), "point groups");
    GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
    total = ctx->h_pinned[0];
    const int G = (int)total;
    /* room for the node lists: each level holds at most as many ids as the one below, in practice
     * half as many until the nodes outgrow the walks; a node that does not fit goes without */
    const int64_t cap = std::min<int64_t>(grid ? total + total * 3 / 2 + 4096 : total, ((int64_t)1 << 31) - 2);
    int32_t* gbeg = (int32_t*)dev((size_t)(total + 1) * 4);
    int32_t* ids = gbeg ? (int32_t*)dev((size_t)cap * 4) : nullptr;
    float4* gbox = ids ? (float4*)dev((size_t)total * 16) : nullptr;
    if (!gbox) return without();
    k_groups<<<(unsigned)tiles, 256, 0, s>>>(P, ix->d_tid, bits, off, gbeg, ids);
    const int32_t end = (int32_t)P;
    GAT_CUDA_TRY(ctx, cudaMemcpyAsync(gbeg + total, &end, 4, cudaMemcpyHostToDevice, s), "point groups");
    k_group_boxes<<<blocks_for(ctx, total, 128), 128, 0, s>>>(G, gbeg, ix->d_x, ix->d_y, gbox);
    count_launch(ctx, 4);
    GroupsDev g;
    g.n = G;
    g.gbeg = gbeg;
    g.ids = ids;
    g.gbox = gbox;
    if (!grid) {
        int32_t* cell_g = (int32_t*)dev((size_t)(ix->fsg.cellnum + 1) * 4);
        if (!cell_g) return without();
        k_cell_groups<<<blocks_for(ctx, ix->fsg.cellnum + 1), 256, 0, s>>>(ix->fsg.cellnum, ix->fsg.cbeg, ix->fsg.cend, G, gbeg,
                                                                          cell_g);
        count_launch(ctx);
        g.cell_g = cell_g;
    } else {
        const int n = ix->grid.nnodes, levels = ix->grid.total_level + 1;
        NodeRec* rec = (NodeRec*)dev((size_t)n * sizeof(NodeRec));
        int* level = tmp.get<int>(levels + 3);
        int* big = tmp.get<int>((size_t)n + 1);
        unsigned long long* cursor = tmp.get<unsigned long long>(1);
        if (!rec || !level || !big || !cursor) return without();
        if (!ix->d_pbox) {
            GAT_CUDA_TRY(ctx, cudaMalloc(&ix->d_pbox, (size_t)n * sizeof(float4)), "point boxes");
            ix->device_bytes += (size_t)n * sizeof(float4);
        }
        k_node_records<<<blocks_for(ctx, n), 256, 0, s>>>(ix->grid, G, gbeg, gbox, rec, ix->d_pbox);
        /* level l is [level[l], level[l + 1]); the root is level 0 */
        ctx->h_pinned[2] = total;
        GAT_CUDA_TRY(ctx, cudaMemsetAsync(level, 0, (size_t)(levels + 3) * 4, s), "point groups");
        const int one = 1;
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(level + 1, &one, 4, cudaMemcpyHostToDevice, s), "point groups");
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(cursor, ctx->h_pinned + 2, 8, cudaMemcpyHostToDevice, s), "point groups");
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
        g.jump_level = std::min(kJumpLevel, ix->grid.total_level);
        int32_t* jump = (int32_t*)dev(((size_t)1 << (2 * g.jump_level)) * 4);
        if (!jump) return without();
        GAT_CUDA_TRY(ctx, cudaMemsetAsync(big + n, 0, 4, s), "point groups");
        k_jump<<<16, 256, 0, s>>>(g.jump_level, rec, jump, big + n);
        GAT_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_pinned + 3, big + n, 4, cudaMemcpyDeviceToHost, s), "point groups");
        GAT_CUDA_TRY(ctx, cudaStreamSynchronize(s), "point groups");
        if ((int32_t)ctx->h_pinned[3] == 0) g.jump = jump;
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
