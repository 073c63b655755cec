/* Batched trajectory-id range queries over point groups (groups.cu).
 *
 * A query's candidates are the reference's: the leaves the quadtree walk takes (BoxIntersect,
 * Grid.cpp:428-446, MortonGrid.cpp:356-393) or the median slabs and leaf boxes select (STIG.cpp:179-252),
 * or the cells of the candidate rectangle (FSG.cpp:183-262). Their points are not scanned one by one:
 *   - a node inside the query (by its box and the exact box of its points), or the FSG cells strictly
 *     inside the candidate rectangle, have every point in the query: their ids are taken as they
 *     are, a node's from its list of distinct trajectories;
 *   - of the other candidate leaves and cells each group is taken or left by its box; only a group
 *     that straddles the query's border, of a trajectory not yet found, has its points tested
 *     (MBB::pInBox, MBB.cpp:21-26) until one is inside.
 * On 100k rectangles of log-U[0.001, 0.05] degree sides over 1M walks (200M points) that reads about
 * 1/20 of the candidates' bytes, and the walk, the scan, the sort and the output of a query run in
 * one kernel without items in global memory.
 *
 * One kernel, three kinds of team by the ids a query is expected to hold (k_order_class): a warp, a
 * pair of warps, or the CTA of 256 threads, each with its share of the CTA's shared memory (an eighth,
 * a quarter, all). Small teams keep more queries in flight and wait less at barriers: 15k rectangles
 * of 0.02 to 0.05 degrees over 1M walks took 2.07 ms by CTAs alone, 1.86 ms with pairs for those of
 * 400 to 1,100 expected ids. A query that outgrows its team
 * runs again on the CTA; one with more ids than that holds goes to the bitmap scan, one whose walk outgrows it to
 * the point scan (range.cu; a rectangle over the whole of an FSG of 1,000 rows and 300 long walks: 1.16 ms by
 * the point scan, 3.57 ms by the bitmap).
 *
 * Plain execution (one query per launch): the CTA answers one query and writes it where the query before
 * it ended. Each launch lets the next start at once; a query waits for the one before only to read its
 * end, so the walks, scans and sorts of neighbouring launches overlap.
 *
 * Point lists (Grid, MortonGrid): the same walk gives ranges of points, the CTA collects the keys of
 * those inside, sorts and writes them.
 */
#include <algorithm>
#include <climits>
#include <cmath>

#include "cells.cuh"
#include "launch.cuh"
#include "range_common.cuh"

namespace gat {
namespace {

constexpr int kNT = 256, kW = kNT / 32;
/* id set slots (log2), ids, walk frontier and candidate ranges of a team in each mode */
constexpr int kBlockBits = 13, kBlockIds = 4096, kBlockFront = 512, kBlockItems = 2048;
constexpr int kMidBits = 11, kMidIds = 1408, kMidFront = 128, kMidItems = 320;
constexpr int kSmallBits = 10, kSmallIds = 512, kSmallFront = 64, kSmallItems = 256;
constexpr int kMidTeams = kW / 2; /* pairs of warps */
constexpr int kCtl = 24; /* control words of a team */
/* expected ids up to which a query is small or mid: short of the set, since the estimate is not exact */
constexpr float kSmallMax = 400.f, kMidMax = 1100.f;
constexpr int kSmallScan = 4096, kMidScan = 8192; /* groups a small or a mid team takes on */
constexpr float kBoundToOutgrow = 1.2f; /* plain execution: expected ids, as a multiple of the set's, that are not tried */
constexpr int kFarCell = 1 << 20; /* FSG cell coordinates beyond this take the general scan */
constexpr int kBorder = (int)0x80000000; /* item end flag: groups to be tested by box */

/* shared memory of one query's team */
template <int HB_, int IDS_, int FRONT_, int ITEMS_, int NTHREADS_>
struct Team {
    static constexpr int HB = HB_, IDS = IDS_, FRONT = FRONT_, ITEMS = ITEMS_, NTHREADS = NTHREADS_;
    static constexpr int kInts = (1 << HB) + IDS + 2 * FRONT + 2 * ITEMS;
    static_assert((1 << HB) / 8 + IDS <= (1 << HB), "sort_ids keeps buckets and ids in the set's slots");
    int* tab;    /* 2^HB slots, -1 = empty */
    int* list;   /* IDS ids in insertion order */
    int* front;  /* 2 x FRONT first children of the nodes to open */
    int2* items; /* ITEMS ranges of ids / groups */
    int* nitems;
    int* nfront; /* [2] */
    int* cnt;
    int* ovf;
    int* next;                /* items handed out */
    unsigned long long* base; /* the answer's place in the arena */
    int* sort;                /* sort_ids: [0] least id, [1] greatest, [2] largest bucket, [4 + w] bucket totals per warp */
    int* query;               /* the query being answered */
    int id;                   /* which of the CTA's teams */
    __device__ Team(int* mem, int* ctl, int id_)
        : tab(mem), list(mem + (1 << HB)), front(list + IDS), items(reinterpret_cast<int2*>(front + 2 * FRONT)), nitems(ctl),
          nfront(ctl + 1), cnt(ctl + 3), ovf(ctl + 4), next(ctl + 5), base(reinterpret_cast<unsigned long long*>(ctl + 6)),
          sort(ctl + 8), query(ctl + 20), id(id_) {}
    __device__ __forceinline__ void sync() const {
        if (NTHREADS == 32)
            __syncwarp();
        else if (NTHREADS == kNT)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(NTHREADS) : "memory");
    }
    /* hs_insert with this team's list length */
    __device__ __forceinline__ void insert(int t) {
        unsigned h = hs_slot<HB>(t);
        for (int p = 0; p < 64; p++) {
            int v = tab[h];
            if (v == t) return;
            if (v == -1) {
                v = atomicCAS(&tab[h], -1, t);
                if (v == -1) {
                    const int pos = atomicAdd(cnt, 1);
                    if (pos < IDS)
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
    __device__ __forceinline__ bool has(int t) const {
        unsigned h = hs_slot<HB>(t);
        for (int p = 0; p < 64; p++) {
            const int v = *(const volatile int*)(tab + h);
            if (v == t) return true;
            if (v == -1) return false;
            h = (h + 1) & ((1u << HB) - 1);
        }
        return false;
    }
};
using BlockTeam = Team<kBlockBits, kBlockIds, kBlockFront, kBlockItems, kNT>;
using LongTeam = Team<14, 14336, kBlockFront, kBlockItems, kNT>; /* point lists: one CTA per SM */
using MidTeam = Team<kMidBits, kMidIds, kMidFront, kMidItems, 64>;
using SmallTeam = Team<kSmallBits, kSmallIds, kSmallFront, kSmallItems, 32>;
constexpr int kInts = BlockTeam::kInts;
static_assert(kW * SmallTeam::kInts <= kInts && kMidTeams * MidTeam::kInts <= kInts, "the warps share the CTA's memory");
constexpr size_t kSmem = (size_t)kInts * sizeof(int);

__device__ __forceinline__ bool pbox_inside(const Box& q, const float4& b) {
    return b.x >= q.xmin && b.z <= q.xmax && b.y >= q.ymin && b.w <= q.ymax;
}

template <class T>
__device__ __forceinline__ void put_item(T& t, int b, int e, bool border) {
    if (b >= e) return;
    const int k = atomicAdd(t.nitems, 1);
    if (k < T::ITEMS)
        t.items[k] = make_int2(b, border ? e | kBorder : e);
    else
        *t.ovf = 1;
}

/* The quadtree walk, one level of the frontier at a time, by thread `me` of the team. The root is
 * taken without a test (Grid.cpp:428-433), every other node when BoxIntersect holds for it and all its
 * ancestors. A node's box lies within its ancestors' and has a width, and then BoxIntersect with the
 * node implies BoxIntersect with them (both ask for open overlap in y, and in x for the larger xmin
 * below the other's xmax, which a wider box keeps), so a query smaller than a few squares of the jump
 * table starts at the nodes of its squares (one more on every side, for the rounding of the division)
 * and skips the levels above. */
constexpr int kJumpMax = 64; /* squares a walk starts from at most */

template <bool PTS, class T>
__device__ void walk_grid(const GroupsDev& g, const GridDev& tree, const Box& q, T& t, int me) {
    constexpr int FRONT = T::FRONT;
    const NodeRec* __restrict__ rec = g.rec;
    /* PTS: ranges of points instead of ids and groups */
    auto take = [&](int nd, const NodeRec& r, bool border) {
        if (PTS)
            put_item(t, tree.node_pbeg[nd], tree.node_pend[nd], border);
        else
            put_item(t, r.ib, r.ie, border);
    };
    auto classify = [&](int nd, const NodeRec& r, int* out, int* nout) {
        const bool in = pbox_inside(q, r.pbox);
        if (r.child < 0)
            take(nd, r, !in);
        else if (in && (PTS || r.ib >= 0) && box_inside(q, r.mbb))
            take(nd, r, false);
        else {
            const int k = atomicAdd(nout, 1);
            if (k < FRONT)
                out[k] = r.child;
            else
                *t.ovf = 1;
        }
    };
    bool jumped = false;
    if (g.jump) {
        const int n = 1 << g.jump_level;
        const float inv = 1.f / (tree.cell * (float)(tree.axis >> g.jump_level));
        auto square = [&](float d, int off) { return min(n - 1, max(0, (int)fminf(fmaxf(d * inv, -4.f), 1e6f) + off)); };
        const int x0 = square(q.xmin - tree.rxmin, -1), x1 = square(q.xmax - tree.rxmin, 1);
        const int y0 = square(tree.rymax - q.ymax, -1), y1 = square(tree.rymax - q.ymin, 1);
        const int w = x1 - x0 + 1, h = y1 - y0 + 1;
        jumped = w > 0 && h > 0 && w * h <= kJumpMax;
        if (jumped)
            for (int k = me; k < w * h; k += T::NTHREADS) {
                const int x = x0 + k % w, y = y0 + k / w;
                const int nd = g.jump[y * n + x];
                /* a leaf above the table's level covers several squares: the first of the query's takes it */
                if ((x > x0 && g.jump[y * n + x - 1] == nd) || (y > y0 && g.jump[(y - 1) * n + x] == nd)) continue;
                const NodeRec r = rec[nd];
                if (nd == 0 || box_intersect(q, Box{r.mbb.x, r.mbb.y, r.mbb.z, r.mbb.w})) classify(nd, r, t.front, t.nfront);
            }
    }
    if (!jumped && me == 0) {
        const NodeRec r = rec[0];
        classify(0, r, t.front, t.nfront);
    }
    t.sync();
    for (int cur = 0;; cur ^= 1) {
        /* read by all before any thread opens nodes (and may flag an overflow) again */
        const int n = min(t.nfront[cur], FRONT);
        const bool lost = *(volatile int*)t.ovf != 0;
        t.sync();
        if (n == 0 || lost) break;
        for (int k = me; k < 4 * n; k += T::NTHREADS) {
            const int nd = t.front[cur * FRONT + (k >> 2)] + (k & 3);
            const NodeRec r = rec[nd];
            if (box_intersect(q, Box{r.mbb.x, r.mbb.y, r.mbb.z, r.mbb.w}))
                classify(nd, r, t.front + (cur ^ 1) * FRONT, t.nfront + (cur ^ 1));
        }
        t.sync();
        if (me == 0) t.nfront[cur] = 0;
    }
}

/* STIG::searchNode (STIG.cpp:201-252), one level at a time: an inner node sends the walk left and right
 * by its median (intersectBlock, STIG.cpp:340-347), a leaf is taken when BoxIntersect(its box, query). */
template <class T>
__device__ void walk_stig(const NodeRec* __restrict__ rec, const Box& q, T& t, int me) {
    if (me == 0) {
        t.front[0] = 0;
        t.nfront[0] = 1;
    }
    t.sync();
    for (int cur = 0;; cur ^= 1) {
        const int n = min(t.nfront[cur], T::FRONT);
        const bool lost = *(volatile int*)t.ovf != 0;
        t.sync();
        if (n == 0 || lost) break;
        int* out = t.front + (cur ^ 1) * T::FRONT;
        auto push = [&](int nd) {
            const int k = atomicAdd(t.nfront + (cur ^ 1), 1);
            if (k < T::FRONT)
                out[k] = nd;
            else
                *t.ovf = 1;
        };
        for (int k = me; k < n; k += T::NTHREADS) {
            const NodeRec r = rec[t.front[cur * T::FRONT + k]];
            if (r.child < 0) {
                if (box_intersect(Box{r.mbb.x, r.mbb.y, r.mbb.z, r.mbb.w}, q)) put_item(t, r.ib, r.ie, !pbox_inside(q, r.pbox));
                continue;
            }
            const float lo = r.aux & 1 ? q.ymin : q.xmin, hi = r.aux & 1 ? q.ymax : q.xmax, med = r.mbb.x;
            if (!(hi < 0.0f) && !(lo > med)) push(r.child);
            if (!(hi < med) && !(lo > 180.0f)) push(r.aux >> 1);
        }
        t.sync();
        if (me == 0) t.nfront[cur] = 0;
    }
}

/* The implicit quadtree of the MortonGrid (morton_walk in range.cu): frontier entries pack
 * (id << 4) | level. The groups of what it takes are tested by their boxes, whole subtrees included
 * (their points may lie a rounding outside the computed boxes). */
template <class T>
__device__ void walk_morton(const MortonDev& m, const int32_t* __restrict__ cell_g, const Box& q, T& t, int me) {
    auto emit = [&](int level, uint32_t id) {
        const uint32_t span = 1u << (2 * (m.total_level - level));
        put_item(t, cell_g[id * span], cell_g[id * span + span], true);
    };
    auto leaf = [&](int level, uint32_t id) {
        const uint64_t idx = (((uint64_t)1 << (2 * level)) - 1) / 3 + id;
        return (__ldg(m.leaf + (idx >> 5)) >> (idx & 31)) & 1u;
    };
    if (me == 0) {
        if (leaf(0, 0))
            emit(0, 0);
        else
            t.nfront[0] = 1, t.front[0] = 0;
    }
    t.sync();
    for (int cur = 0;; cur ^= 1) {
        const int n = min(t.nfront[cur], T::FRONT);
        const bool lost = *(volatile int*)t.ovf != 0;
        t.sync();
        if (n == 0 || lost) break;
        for (int k = me; k < 4 * n; k += T::NTHREADS) {
            const uint32_t e = (uint32_t)t.front[cur * T::FRONT + (k >> 2)];
            const int level = (int)(e & 15u) + 1;
            const uint32_t id = ((e >> 4) << 2) + (k & 3), span = 1u << (2 * (m.total_level - level));
            const float4 a = morton_cell_box(m.rxmin, m.rymax, m.cell, (int)(id * span));
            const float4 b = morton_cell_box(m.rxmin, m.rymax, m.cell, (int)(id * span + span - 1));
            const float4 box = make_float4(a.x, b.y, b.z, a.w);
            if (!box_intersect(q, Box{box.x, box.y, box.z, box.w})) continue;
            if (leaf(level, id) || box_inside(q, box)) {
                emit(level, id);
                continue;
            }
            const int o = atomicAdd(t.nfront + (cur ^ 1), 1);
            if (o < T::FRONT)
                t.front[(cur ^ 1) * T::FRONT + o] = (int)((id << 4) | (uint32_t)level);
            else
                *t.ovf = 1;
        }
        t.sync();
        if (me == 0) t.nfront[cur] = 0;
    }
}

/* The FSG's candidate cells row by row (fsg_walk in range.cu): row r covers the cells g1 + r nx ..
 * g2 + r nx, unclamped as in the reference. f(v) = (int)((v - origin) / cell) is monotone in float
 * arithmetic, so a point in a column strictly between g1 and g2 and a row strictly between g3 and g4
 * lies inside the query: those cells are taken whole, the rest by their groups' boxes. (A NaN
 * coordinate would break the ordering: no cell is then taken whole.) */
template <class T>
__device__ void walk_fsg(const FsgDev& f, const int32_t* __restrict__ cell_g, const Box& q, T& t, int me) {
    auto begin = [&](int c) { return cell_g[c]; }; /* the cell's first group */
    const int g1 = (int)__fdiv_rn(__fsub_rn(q.xmin, f.rxmin), f.cell), g2 = (int)__fdiv_rn(__fsub_rn(q.xmax, f.rxmin), f.cell);
    const int g3 = (int)__fdiv_rn(__fsub_rn(f.rymax, q.ymax), f.cell), g4 = (int)__fdiv_rn(__fsub_rn(f.rymax, q.ymin), f.cell);
    if (max(max(g1, g2), max(g3, g4)) > kFarCell || min(min(g1, g2), min(g3, g4)) < -kFarCell || g4 - g3 > 4 * T::ITEMS) {
        if (me == 0) *t.ovf = 1;
        t.sync();
        return;
    }
    const bool ordered = q.xmin <= q.xmax && q.ymin <= q.ymax;
    for (int r = g3 + me; r <= g4; r += T::NTHREADS) {
        const long long row = (long long)r * f.nx;
        const long long lo_ = max(0ll, row + g1), hi_ = min((long long)f.cellnum - 1, row + g2);
        if (lo_ > hi_) continue;
        const int lo = (int)lo_, hi = (int)hi_;
        int a = hi + 1, b = hi + 1; /* cells [a, b) taken whole */
        if (ordered && r > g3 && r < g4 && r >= 0 && r < f.ny) {
            const int c0 = max(g1 + 1, 0), c1 = min(g2 - 1, f.nx - 1);
            if (c0 <= c1) {
                a = (int)row + c0;
                b = (int)row + c1 + 1;
            }
        }
        const int ga = begin(a), gb = begin(b);
        put_item(t, begin(lo), ga, true);
        put_item(t, ga, gb, false);
        put_item(t, gb, begin(hi + 1), true);
    }
    t.sync();
}

/* groups a warp has found to straddle the query's border, tested kOpen / 2 or more at a time */
constexpr int kOpen = 64;
struct OpenGroups {
    int at[kOpen], id[kOpen]; /* group and trajectory */
};

/* Tests the points of `n` open groups whose trajectory is not in the set yet, eight groups at a time with
 * four lanes each and kFly points per lane in flight (24 points: most groups in one trip to L2), until
 * one lies in the query. (Four groups with two points per lane in flight took two trips each: 100k
 * rectangles over 1M walks 2.24 ms, 2.05 ms now.) */
constexpr int kFly = 6;

template <class T>
__device__ __forceinline__ void test_open(const OpenGroups& og, int n, const Box& q, const int32_t* __restrict__ gbeg,
                                          const float* __restrict__ X, const float* __restrict__ Y, T& t, unsigned& bytes) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const bool on = k0 + lane < n;
        int b = 0, e = 0, id = -1;
        if (on) {
            const int g = og.at[k0 + lane];
            id = og.id[k0 + lane];
            b = __ldg(gbeg + g);
            e = __ldg(gbeg + g + 1);
            bytes += 8;
        }
        const unsigned m = __ballot_sync(FULL, on && !t.has(id));
        const int total = __popc(m);
        /* the lanes of the open groups, in order: lane i holds the i-th */
        int nth = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            if (__popc(m & ((1u << (nth + s)) - 1u)) <= lane) nth += s;
        for (int k = 0; k < total; k += 8) {
            const int g = k + (lane >> 2);
            const int src = __shfl_sync(FULL, nth, g & 31);
            const int b0 = __shfl_sync(FULL, b, src), e1 = __shfl_sync(FULL, e, src), e0 = g < total ? e1 : b0;
            const int tid = __shfl_sync(FULL, id, src);
            bool found = false;
            for (int i = b0 + (lane & 3); i < e0 && !found; i += 4 * kFly) {
                float x[kFly], y[kFly];
#pragma unroll
                for (int u = 0; u < kFly; u++) {
                    const int p = min(i + 4 * u, e0 - 1);
                    x[u] = __ldg(X + p);
                    y[u] = __ldg(Y + p);
                }
#pragma unroll
                for (int u = 0; u < kFly; u++) found |= in_box(q, x[u], y[u]);
                bytes += 8 * kFly;
            }
            const unsigned hits = __ballot_sync(FULL, found);
            if ((lane & 3) == 0 && ((hits >> lane) & 0xfu)) t.insert(tid);
        }
    }
    __syncwarp();
}

/* One warp takes the `n` <= 32 ranges from items[0]: their ids are dealt to the lanes as one sequence
 * (a mask of where ranges begin tells a lane its range), so that short ranges fill the warp. The ids and
 * boxes of the next 32 are loaded before the current 32 are looked at: with a load after each test
 * a step waited for three trips to L2 (100k rectangles over 1M walks 4.6 ms). Groups that straddle
 * the border gather in `og`. */
template <class T>
__device__ __forceinline__ void take_items(const int2* items, int n, const Box& q, const int32_t* __restrict__ ids,
                                           const int32_t* __restrict__ gbeg, const float4* __restrict__ gbox,
                                           const float* __restrict__ X, const float* __restrict__ Y, T& t, OpenGroups& og,
                                           unsigned long long& work) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int2 it = lane < n ? items[lane] : make_int2(0, 0);
    const int len = (it.y & ~kBorder) - it.x;
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    const int shift = it.x - (incl - len); /* position = shift + sequence index */
    unsigned bytes = len * (it.y < 0 ? 20 : 4); /* ids, and boxes of border groups */
    int nopen = 0;
    struct Next {
        int id, pos;
        float4 box;
        bool border;
    };
    int begun = 0; /* ranges that begin before the current 32 */
    auto load = [&](int e0) {
        Next x;
        /* the owner: the last range that begins at or before the lane's element */
        const unsigned at = (unsigned)(incl - len - e0);
        const unsigned heads = __reduce_or_sync(FULL, lane < n && at < 32u ? 1u << at : 0u);
        const int l = begun + __popc(heads & ((2u << lane) - 1u)) - 1;
        begun += __popc(heads);
        x.pos = __shfl_sync(FULL, shift, l) + e0 + lane;
        x.border = __shfl_sync(FULL, it.y, l) < 0;
        x.id = -1;
        x.box = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e0 + lane < total) {
            x.id = __ldg(ids + x.pos);
            if (x.border) x.box = __ldg(gbox + x.pos);
        }
        return x;
    };
    Next nx = load(0);
    for (int e0 = 0; e0 < total; e0 += 32) {
        const Next x = nx;
        if (e0 + 32 < total) nx = load(e0 + 32);
        const bool in = pbox_inside(q, x.box);
        const bool out = x.box.x > q.xmax || x.box.z < q.xmin || x.box.y > q.ymax || x.box.w < q.ymin;
        if (__shfl_sync(FULL, *(volatile int*)t.ovf, 0)) break;
        if (x.id >= 0 && (!x.border || in)) t.insert(x.id);
        const bool open = x.id >= 0 && x.border && !in && !out;
        const unsigned m = __ballot_sync(FULL, open);
        if (open) {
            const int k = nopen + __popc(m & ((1u << lane) - 1u));
            og.at[k] = x.pos;
            og.id[k] = x.id;
        }
        nopen += __popc(m);
        __syncwarp();
        if (nopen > kOpen - 32) {
            test_open(og, nopen, q, gbeg, X, Y, t, bytes);
            nopen = 0;
        }
    }
    if (nopen) test_open(og, nopen, q, gbeg, X, Y, t, bytes);
    work += bytes;
}

/* The team's m ids, ascending, to out (nothing when `write` is false); leaves the set empty. Ids are
 * counted into buckets of equal width between the least and the greatest (about two to a bucket),
 * scattered to their buckets, and placed by the number of smaller ids in their own bucket. When ids
 * crowd in a few buckets the list is sorted in runs of 32 that are merged in pairs instead. (Sorting
 * runs and searching every id in every run took half of a query's instructions.) `out` may be the list
 * itself. FLIP is xored into what is written (point keys are held with their top bit flipped). */
/* Fullest bucket that is ranked: ids, and point keys, which lie in clusters (1,500 rectangles of 0.003 to 0.03
 * degrees on 100k walks: 1270 us with 32, 1132 us with 512). The second pass of point lists sorts by
 * digits instead as soon as a bucket holds more than kCrowd: a key is compared with every other of its bucket, a
 * walk's hundred or more points (148 lists of 10k points 248 us by ranks, 139 by digits; a thousand 1409 and 912). The
 * first pass keeps to ranks: the digits' code in it cost 1,000 lists of about 110 points 5 us of 38. */
constexpr int kCrowd = 32, kKeyCrowd = 512;

/* The m keys of the team's list by a stable radix sort in shared memory, 8 bits of (key - lo) a pass, between the
 * list and the set's slots: each warp counts the digits of its share, a scan over digits and warps gives it
 * its places, and it puts its keys there in order. */
template <class T, unsigned FLIP>
__device__ void radix_keys(T& t, int m, unsigned range, unsigned lo, uint32_t* out, bool write, int me) {
    constexpr int W = T::NTHREADS / 32;
    static_assert(T::NTHREADS == 256 && T::IDS + W * 256 <= (1 << T::HB), "the keys and the counters share the set's slots");
    const unsigned FULL = 0xffffffffu;
    const int lane = me & 31, warp = me >> 5;
    int* const hist = t.tab + (1 << T::HB) - W * 256;
    const int share = ((m + W - 1) / W + 31) & ~31, begin = min(m, warp * share), end = min(m, begin + share);
    int *src = t.list, *dst = t.tab;
    t.sync(); /* the counts in the slots have been read */
    for (int shift = 0; shift < 32 && (range >> shift) != 0; shift += 8) {
        for (int i = me; i < W * 256; i += T::NTHREADS) hist[i] = 0;
        t.sync();
        for (int i = begin + lane; i < end; i += 32) atomicAdd(&hist[warp * 256 + ((((unsigned)src[i] - lo) >> shift) & 255u)], 1);
        t.sync();
        int c[W], sum = 0;
#pragma unroll
        for (int w = 0; w < W; w++) {
            c[w] = hist[w * 256 + me];
            sum += c[w];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) t.sort[4 + warp] = incl;
        t.sync();
        int at = incl - sum;
        for (int w = 0; w < warp; w++) at += t.sort[4 + w];
#pragma unroll
        for (int w = 0; w < W; w++) {
            hist[w * 256 + me] = at;
            at += c[w];
        }
        t.sync();
        for (int i0 = begin; i0 < end; i0 += 32) {
            const int i = i0 + lane;
            const int x = i < end ? src[i] : 0;
            const int d = i < end ? (int)((((unsigned)x - lo) >> shift) & 255u) : -1;
            const unsigned peers = __match_any_sync(FULL, d);
            const int rank = __popc(peers & ((1u << lane) - 1u));
            int at0 = 0;
            if (d >= 0) at0 = hist[warp * 256 + d];
            __syncwarp();
            if (d >= 0) {
                if (rank == 0) hist[warp * 256 + d] = at0 + __popc(peers);
                dst[at0 + rank] = x;
            }
            __syncwarp();
        }
        t.sync();
        int* s = src;
        src = dst;
        dst = s;
    }
    if (write)
        for (int i = me; i < m; i += T::NTHREADS) out[i] = (uint32_t)src[i] ^ FLIP;
}

template <class T, unsigned FLIP = 0>
__device__ void sort_ids(T& t, int m, uint32_t* out, bool write, int me) {
    constexpr int HB = T::HB, NTHREADS = T::NTHREADS;
    int *const tab = t.tab, *const list = t.list;
    constexpr int B = 1 << (HB - 3); /* buckets, counted in tab[0..B); the scattered ids follow */
    constexpr int kPer = B / NTHREADS;
    const unsigned FULL = 0xffffffffu;
    const int lane = me & 31, warp = me >> 5;
    int* lo_hi = t.sort;
    /* the list is complete and the set no longer needed */
    int lo = INT_MAX, hi = INT_MIN;
    for (int i = me; i < m; i += NTHREADS) {
        lo = min(lo, list[i]);
        hi = max(hi, list[i]);
    }
    for (int b = me; b < B; b += NTHREADS) tab[b] = 0;
    if (NTHREADS > 32 && me == 0) {
        lo_hi[0] = INT_MAX;
        lo_hi[1] = INT_MIN;
        lo_hi[2] = 0;
    }
    t.sync();
    lo = __reduce_min_sync(FULL, lo);
    hi = __reduce_max_sync(FULL, hi);
    if (NTHREADS > 32) {
        if (lane == 0) {
            atomicMin(&lo_hi[0], lo);
            atomicMax(&lo_hi[1], hi);
        }
        t.sync();
        lo = lo_hi[0];
        hi = lo_hi[1];
    }
    /* bucket of t: (t - lo) B / width by a rounded-down 0.32 reciprocal, monotone in t, which is all
     * that the placement needs */
    const unsigned scale = (unsigned)min(0xffffffffull, ((unsigned long long)B << 32) / ((unsigned long long)((unsigned)hi - (unsigned)lo) + 1ull));
    auto bucket = [&](int x) -> int {
        const unsigned long long p = (unsigned long long)((unsigned)x - (unsigned)lo) * scale;
        return min(B - 1, (int)(p >> 32));
    };
    for (int i = me; i < m; i += NTHREADS) atomicAdd(&tab[bucket(list[i])], 1);
    t.sync();
    /* exclusive scan of the counts, kPer consecutive buckets per thread */
    int c[kPer], sum = 0, most = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        c[k] = tab[me * kPer + k];
        most = max(most, c[k]);
        sum += c[k];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
    }
    most = __reduce_max_sync(FULL, most);
    int start = incl - sum;
    if (NTHREADS > 32) {
        if (lane == 31) lo_hi[4 + warp] = incl;
        if (lane == 0) atomicMax(&lo_hi[2], most);
        t.sync();
        most = lo_hi[2];
        for (int w = 0; w < warp; w++) start += lo_hi[4 + w];
    }
    bool placed = false;
    if constexpr (FLIP != 0 && T::IDS > kBlockIds) {
        placed = most > kCrowd;
        if (placed) radix_keys<T, FLIP>(t, m, (unsigned)hi - (unsigned)lo, (unsigned)lo, out, write, me);
    }
    if (placed) {
    } else if (most <= (FLIP ? kKeyCrowd : kCrowd)) {
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            tab[me * kPer + k] = start;
            start += c[k];
        }
        t.sync();
        int* dst = tab + B;
        for (int i = me; i < m; i += NTHREADS) {
            const int x = list[i];
            dst[atomicAdd(&tab[bucket(x)], 1)] = x;
        }
        t.sync();
        /* tab[b] is now the end of bucket b */
        if (write)
            for (int i = me; i < m; i += NTHREADS) {
                const int x = dst[i], b = bucket(x), first = b ? tab[b - 1] : 0, end = tab[b];
                int rank = first;
                for (int k = first; k < end; k++) rank += dst[k] < x ? 1 : 0;
                out[rank] = (uint32_t)x ^ FLIP;
            }
    } else {
        /* runs of 32 sorted by the warps, then merged in pairs: an id's place in the merged run is its
         * place in its own run plus the ids below it in the partner run */
        t.sync();
        const int runs = (m + 31) >> 5;
        for (int r = warp; r < runs; r += NTHREADS / 32) {
            const int i = 32 * r + lane;
            const int v = warp_sort32(i < m ? list[i] : INT_MAX);
            __syncwarp();
            if (i < m) list[i] = v;
        }
        t.sync();
        int* src = list;
        int* dst = tab;
        for (int L = 32; L < m; L <<= 1) {
            for (int i = me; i < m; i += NTHREADS) {
                const int x = src[i];
                const int begin = i & ~(2 * L - 1);
                const int mid = min(begin + L, m), end = min(begin + 2 * L, m);
                const bool in_a = i < mid;
                const int first = in_a ? mid : begin;
                int at = first, len = in_a ? end - mid : mid - begin;
                while (len > 0) {
                    const int half = len >> 1;
                    if (src[at + half] < x) {
                        at += half + 1;
                        len -= half + 1;
                    } else {
                        len = half;
                    }
                }
                dst[begin + (i - (in_a ? begin : mid)) + (at - first)] = x;
            }
            t.sync();
            int* s = src;
            src = dst;
            dst = s;
        }
        if (write)
            for (int i = me; i < m; i += NTHREADS) out[i] = (uint32_t)src[i] ^ FLIP;
    }
    t.sync();
    int4* slots = reinterpret_cast<int4*>(tab);
    for (int i = me; i < (1 << HB) / 4; i += NTHREADS) slots[i] = make_int4(-1, -1, -1, -1);
}

struct GroupQuery {
    const gat_mbb* queries;
    GridDev grid;
    FsgDev fsg;
    MortonDev morton;
    GroupsDev g;
    uint32_t* arena;
    /* Fields of one mode share their place with the other's: 16 bytes more of parameters cost every plain launch 0.3
     * us (24 plain rectangles on an FSG 128 -> 136 us). */
    union {
        int64_t cap;
        float share[2]; /* plain execution: new ids per group of a border item, per id of an inside one */
    };
    /* [0] arena cursor, [1] work bytes, [2] big queries taken, [3] queries for the bitmap scan, [4] small
     * queries taken, [5] queries that outgrew their team, [6] queries for the point scan, [7] mid queries taken */
    unsigned long long* ctr;
    int64_t* segbase;
    int64_t* segcnt;
    /* plain execution: offsets, ids, their capacity, and the state of the call (answer) */
    int64_t* p_off;
    int32_t* p_out;
    union {
        int64_t p_cap;
        float points; /* batches: points per group of the index */
    };
    int* p_state;
    int2* retry;   /* queries that outgrew their team, chained per CTA: (query, next or -1) */
    int* ovf_list; /* queries for the bitmap scan from its front, for the point scan from its end */
    unsigned long long* work;
};

/* How a query ended: answered; more ids than the team's set holds; a walk beyond its frontier or ranges (nothing is
 * scanned then). */
enum Ending { kAnswered, kManyIds, kLongWalk };

/* Whether a walk's candidates are left unscanned, by the groups to be tested by their boxes and the ids and groups
 * inside (small and mid teams scan what they get: their class goes by the expected length too, k_order_class):
 *   - by the CTA to the point scan when there are very many and they hold few points each: a group costs about as much
 *     as four points of that scan when its box is looked at and two when it is inside (16 rectangles of 0.3 degrees on a
 *     MortonGrid with 1.2 points a group, 450k groups each: 5.2 times the point scan's time by groups, the same now). That
 *     scan begins when the batch is done, which a shorter query does not make up for (20k rectangles of up to 0.05 degrees
 *     there: 1.2 times the point scan's time, 1.8 when those of 12k groups are left too);
 *   - by plain execution, where one CTA stands against a grid that scans a long query's points (16k groups take it 50
 *     us, about what it costs to change over), and which fills the set in vain when the query is bound to hold more ids
 *     (a rectangle of 0.3 degrees on a MortonGrid of 100k walks: 528 us, 146 now, 120 by the point scan's three launches
 *     alone). Candidates that count groups twice are kept: an FSG's rows overlap when the rectangle is wider than the
 *     FSG, and the plain point scan has room for every point once.
 * A Grid's batches are not weighed: its nodes' lists stand for many points each. */
constexpr int kPlainScan = 16384, kBatchScan = 24576;
template <int KIND, bool PLAIN>
constexpr bool kWeighed = PLAIN || KIND != GAT_INDEX_GRID;

template <bool PLAIN, class T>
__device__ __forceinline__ bool too_long(const GroupQuery& a, int border, int inside) {
    const float b = (float)border, i = (float)inside;
    if (PLAIN)
        return (b + 0.25f * i > (float)kPlainScan || b * a.share[0] + i * a.share[1] > kBoundToOutgrow * (float)T::IDS) &&
               border + inside <= a.g.n;
    return b + i > (float)kBatchScan && 4.f * b + 2.f * i > (b + i) * a.points;
}

/* one query of a team: walk, scan, sort, write; the team's memory is empty again when it could not answer */
template <int KIND, bool PLAIN = false, class T>
__device__ Ending answer(const GroupQuery& a, int qi, T& t, OpenGroups& og, int me, unsigned long long& bytes) {
    const Box q = load_box(a.queries, qi);
    if (KIND == GAT_INDEX_GRID)
        walk_grid<false>(a.g, a.grid, q, t, me);
    else if (KIND == GAT_INDEX_STIG)
        walk_stig(a.g.rec, q, t, me);
    else if (KIND == GAT_INDEX_MORTON)
        walk_morton(a.morton, a.g.cell_g, q, t, me);
    else
        walk_fsg(a.fsg, a.g.cell_g, q, t, me);
    const int n = min(*t.nitems, T::ITEMS);
    if constexpr (kWeighed<KIND, PLAIN> && T::NTHREADS == kNT) {
        /* groups to be tested by their boxes, and ids and groups inside: every warp adds them up for itself, which
         * for a few dozen ranges is shorter than barriers */
        constexpr int kEnough = 1 << 24; /* a lane's share: the sums stay below 2^31 */
        int border = 0, inside = 0;
        for (int i = me & 31; i < n; i += 32) {
            const int2 it = t.items[i];
            const int len = min((it.y & ~kBorder) - it.x, kEnough);
            border = min(border + (it.y < 0 ? len : 0), kEnough);
            inside = min(inside + (it.y < 0 ? 0 : len), kEnough);
        }
        border = __reduce_add_sync(0xffffffffu, border);
        inside = __reduce_add_sync(0xffffffffu, inside);
        if ((me & 31) == 0 && too_long<PLAIN, T>(a, border, inside)) *t.ovf = 1; /* the same in every warp */
        __syncwarp();
    }
    if (!__shfl_sync(0xffffffffu, *(volatile int*)t.ovf, 0)) {
        /* ranges per turn: enough turns for every warp, up to 32 a turn */
        constexpr int kWarps = T::NTHREADS / 32;
        const int per = kWarps == 1 ? 32 : max(1, min(32, (n + kWarps - 1) / kWarps));
        for (;;) {
            int k = 0;
            if ((me & 31) == 0) k = atomicAdd(t.next, per);
            k = __shfl_sync(0xffffffffu, k, 0);
            if (k >= n) break;
            take_items(t.items + k, min(per, n - k), q, a.g.ids, a.g.gbeg, a.g.gbox, a.g.X, a.g.Y, t, og, bytes);
        }
    }
    t.sync();
    const int m = *t.cnt;
    const bool lost = *(volatile int*)t.ovf != 0;
    if (PLAIN) {
        if (!lost) sort_ids(t, m, reinterpret_cast<uint32_t*>(t.list), true, me);
        dep_wait(); /* the query before has written its end */
        /* state: [0] ids that do not fit, [1] 1 + the first query that outgrew the CTA, [2..3] the end */
        const int stop = qi > 0 ? a.p_state[1] : 0;
        const bool go = stop == 0 && !lost;
        const int64_t at = go && qi > 0 ? a.p_off[qi] : 0;
        t.sync();
        if (me == 0) {
            if (qi == 0) {
                a.p_off[0] = 0;
                a.p_state[0] = a.p_state[1] = 0;
            }
            if (go) {
                a.p_off[qi + 1] = at + m;
                *reinterpret_cast<int64_t*>(a.p_state + 2) = at + m;
                if (at + m > a.p_cap) a.p_state[0] = 1;
            } else if (stop == 0) {
                a.p_state[1] = qi + 1;
            }
        }
        if (go && at + m <= a.p_cap)
            for (int i = me; i < m; i += T::NTHREADS) a.p_out[at + i] = t.list[i];
        return go ? kAnswered : kManyIds;
    }
    if (me == 0 && !lost) {
        *t.base = atomicAdd(&a.ctr[0], (unsigned long long)m);
        a.segcnt[qi] = m;
        a.segbase[qi] = (int64_t)*t.base;
    }
    t.sync();
    if (lost) {
        for (int i = me; i < (1 << T::HB); i += T::NTHREADS) t.tab[i] = -1;
    } else {
        const int64_t at = (int64_t)*t.base;
        sort_ids(t, m, a.arena + at, at + m <= a.cap, me);
    }
    t.sync();
    if (me == 0) *t.nitems = t.nfront[0] = t.nfront[1] = *t.cnt = *t.ovf = *t.next = 0;
    return !lost ? kAnswered : m > 0 ? kManyIds : kLongWalk;
}

/* A team's share of the queries list[0..n), taken from *ctr; the ones that outgrow it go on the CTA's chain. */
template <int KIND, class T>
__device__ void answer_list(const GroupQuery& a, const int* __restrict__ list, int n, unsigned long long* ctr, T t,
                            OpenGroups& og, int* chain, unsigned long long& bytes) {
    const int me = threadIdx.x % T::NTHREADS;
    for (;;) {
        if (me == 0) *t.query = (int)atomicAdd(ctr, 1ull);
        t.sync(); /* also: the set and the counters are clear */
        const int j = *t.query;
        t.sync();
        if (j >= n) break;
        const int qi = list[j];
        if (answer<KIND>(a, qi, t, og, me, bytes) != kAnswered && me == 0) {
            const int k = (int)atomicAdd(&a.ctr[5], 1ull);
            a.retry[k] = make_int2(qi, atomicExch(chain, k));
        }
    }
}

/* Big queries by the CTA, then mid and small ones by its teams, then those that outgrew their team.
 * list: the queries by class, small, mid, big (k_order), *counts how many of them (ends of the small and
 * the mid part, then nq); list null: queries 0..nq-1, all big. */
template <int KIND>
__global__ void __launch_bounds__(kNT, 3) k_range_groups(GroupQuery a, const int* __restrict__ list, const int* counts, int nq) {
    dep_wait();
    extern __shared__ int4 smem4[];
    int* mem = reinterpret_cast<int*>(smem4);
    __shared__ __align__(8) int ctl[kW][kCtl];
    __shared__ int q_sh, chain;
    __shared__ OpenGroups open[kW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto empty = [&] {
        int4* m = smem4;
        for (int i = threadIdx.x; i < kInts / 4; i += kNT) m[i] = make_int4(-1, -1, -1, -1);
    };
    empty();
    if (lane < kCtl) ctl[warp][lane] = 0;
    if (threadIdx.x == 0) chain = -1;
    __syncthreads();
    unsigned long long bytes = 0;
    int first_big = 0;
    BlockTeam t(mem, ctl[0], 0);
    auto block_query = [&](int qi) {
        const Ending e = answer<KIND>(a, qi, t, open[warp], threadIdx.x, bytes);
        if (e != kAnswered && threadIdx.x == 0) {
            if (e == kManyIds)
                a.ovf_list[atomicAdd(&a.ctr[3], 1ull)] = qi;
            else
                a.ovf_list[nq - 1 - (int)atomicAdd(&a.ctr[6], 1ull)] = qi;
            a.segcnt[qi] = 0;
            a.segbase[qi] = 0;
        }
    };
    if (counts) first_big = counts[1];
    for (const int nbig = nq - first_big;;) {
        if (threadIdx.x == 0) q_sh = nbig > 0 ? (int)atomicAdd(&a.ctr[2], 1ull) : 0;
        __syncthreads(); /* also: the set and the counters are clear */
        const int j = q_sh;
        __syncthreads();
        if (j >= nbig) break;
        block_query(list ? list[first_big + j] : j);
    }
    if (counts) {
        const int nsmall = counts[0], nmid = counts[1] - nsmall;
        empty();
        __syncthreads();
        const int pair = warp >> 1;
        answer_list<KIND>(a, list + nsmall, nmid, &a.ctr[7], MidTeam(mem + pair * MidTeam::kInts, ctl[2 * pair], pair), open[warp],
                          &chain, bytes);
        __syncthreads();
        empty();
        __syncthreads();
        answer_list<KIND>(a, list, nsmall, &a.ctr[4], SmallTeam(mem + warp * SmallTeam::kInts, ctl[warp], warp), open[warp],
                          &chain, bytes);
        __syncthreads();
        if (chain >= 0) {
            empty();
            __syncthreads();
            for (int k = chain; k >= 0;) {
                const int2 r = a.retry[k];
                block_query(r.x);
                __syncthreads();
                k = r.y;
            }
        }
    }
    if (a.work) {
        for (int o = 16; o > 0; o >>= 1) bytes += __shfl_down_sync(0xffffffffu, bytes, o);
        if (lane == 0 && bytes) atomicAdd(a.work, bytes);
    }
}

/* Plain execution: query qi of the call. The next query's instance starts at once; until dep_wait (in answer) an
 * instance may read nothing that an earlier one writes (offsets, ids, state) and write nothing outside its
 * shared memory, and none may return before it (launch.cuh). */
template <int KIND>
__global__ void __launch_bounds__(kNT, 2) k_plain_groups(GroupQuery a, int qi) {
    asm volatile("griddepcontrol.launch_dependents;");
    extern __shared__ int4 smem4[];
    int* mem = reinterpret_cast<int*>(smem4);
    __shared__ __align__(8) int ctl[kCtl];
    __shared__ OpenGroups open[kW];
    for (int i = threadIdx.x; i < (1 << kBlockBits) / 4; i += kNT) smem4[i] = make_int4(-1, -1, -1, -1);
    if (threadIdx.x < kCtl) ctl[threadIdx.x] = 0;
    __syncthreads();
    BlockTeam t(mem, ctl, 0);
    unsigned long long bytes = 0;
    answer<KIND, true>(a, qi, t, open[threadIdx.x >> 5], threadIdx.x, bytes);
    if (a.work) {
        for (int o = 16; o > 0; o >>= 1) bytes += __shfl_down_sync(0xffffffffu, bytes, o);
        if ((threadIdx.x & 31) == 0 && bytes) atomicAdd(a.work, bytes);
    }
}

/* Point lists: the keys (trajectory << bits | point index) of the points inside, ascending. A query of
 * more than T::IDS points, or with more than twice as many candidates, is left by the first pass to the second
 * (AGAIN, the list `again` of ctr[5] queries), which has 3.5 times the list and one CTA per SM. What outgrows
 * that too goes on the overflow list for k_range_points, and so do at once the queries with far more candidates
 * than the second pass holds and those whose walk outgrows its frontier or its ranges, of which both passes
 * have the same.
 * Without the second pass a batch with some long lists paid the items and the host's wait for them (710
 * rectangles of 0.0055 to 0.05 degrees on 16k walks: 303 us and 254 us with it).
 * Keys are held with the top bit flipped, so that signed compares order them. */
template <int KIND, class T, bool AGAIN>
__global__ void __launch_bounds__(kNT, AGAIN ? 1 : 3) k_group_points(GroupQuery a, const uint32_t* __restrict__ key, int nq,
                                                                      int* __restrict__ again) {
    dep_wait();
    extern __shared__ int4 smem4[];
    int* mem = reinterpret_cast<int*>(smem4);
    __shared__ __align__(8) int ctl[kCtl];
    __shared__ int q_sh;
    const int lane = threadIdx.x & 31, me = threadIdx.x;
    const unsigned FULL = 0xffffffffu;
    if (me < kCtl) ctl[me] = 0;
    T t(mem, ctl, 0);
    const float *X = a.g.X, *Y = a.g.Y;
    const int todo = AGAIN ? (int)a.ctr[5] : nq;
    for (;;) {
        if (me == 0) q_sh = (int)atomicAdd(&a.ctr[AGAIN ? 4 : 2], 1ull);
        __syncthreads();
        const int turn = q_sh;
        __syncthreads();
        if (turn >= todo) break;
        const int qi = AGAIN ? again[turn] : turn;
        const Box q = load_box(a.queries, qi);
        if (KIND == GAT_INDEX_GRID)
            walk_grid<true>(a.g, a.grid, q, t, me);
        else
            walk_morton(a.morton, a.morton.cbeg, q, t, me);
        const int n = min(*t.nitems, T::ITEMS);
        /* the candidate points: far more than the list holds go on unread, past the second pass where they
         * are far more than it holds */
        int all = 0;
        for (int i = me; i < n; i += kNT) all += (t.items[i].y & ~kBorder) - t.items[i].x;
        all = __reduce_add_sync(FULL, all);
        if (lane == 0 && all) atomicAdd(t.query, all);
        __syncthreads();
        const int points = *t.query;
        const bool many = !AGAIN && points > 2 * kBlockIds;
        if (!many && !__shfl_sync(FULL, *(volatile int*)t.ovf, 0)) {
            for (;;) {
                int k = 0;
                if (lane == 0) k = atomicAdd(t.next, 1);
                k = __shfl_sync(FULL, k, 0);
                if (k >= n) break;
                const int2 r = t.items[k];
                const int end = r.y & ~kBorder;
                const bool test = r.y < 0;
                for (int i0 = r.x; i0 < end; i0 += 128) {
                    /* four points per lane in flight */
                    float x[4], y[4];
                    uint32_t kk[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int i = i0 + 32 * u + lane;
                        const bool on = i < end;
                        x[u] = on && test ? __ldg(X + i) : 0.f;
                        y[u] = on && test ? __ldg(Y + i) : 0.f;
                        kk[u] = on ? __ldg(key + i) : 0u;
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const bool hit = i0 + 32 * u + lane < end && (!test || in_box(q, x[u], y[u]));
                        const unsigned m = __ballot_sync(FULL, hit);
                        if (m == 0) continue;
                        int at = 0;
                        if (lane == 0) at = atomicAdd(t.cnt, __popc(m));
                        at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
                        if (hit && at < T::IDS) t.list[at] = (int)(kk[u] ^ 0x80000000u);
                    }
                }
                if (__shfl_sync(FULL, *(volatile int*)t.cnt, 0) > T::IDS) break;
            }
        }
        __syncthreads();
        const int m = *t.cnt;
        const bool lost = many || *(volatile int*)t.ovf != 0 || m > T::IDS;
        if (me == 0) {
            if (lost) {
                /* a walk that outgrew its memory would do so in the second pass too */
                const bool last = AGAIN || *(volatile int*)t.ovf != 0 || points > LongTeam::IDS + LongTeam::IDS / 4;
                (last ? a.ovf_list : again)[atomicAdd(&a.ctr[last ? 3 : 5], 1ull)] = qi;
                a.segcnt[qi] = 0;
                a.segbase[qi] = 0;
            } else {
                *t.base = atomicAdd(&a.ctr[0], (unsigned long long)m);
                a.segcnt[qi] = m;
                a.segbase[qi] = (int64_t)*t.base;
            }
        }
        __syncthreads();
        if (!lost) {
            const int64_t at = (int64_t)*t.base;
            sort_ids<T, 0x80000000u>(t, m, a.arena + at, at + m <= a.cap, me);
        }
        __syncthreads();
        if (me == 0) *t.nitems = t.nfront[0] = t.nfront[1] = *t.cnt = *t.ovf = *t.next = *t.query = 0;
        __syncthreads();
    }
}

/* ---------------------------------------------------------------- order and class of a batch */
/* The queries of a batch in one counting sort: by class (small, mid, big), then by where they start in
 * the index's point order, bucketed: queries that run at one time then read overlapping groups, which
 * stay in L2. The order changes no result. */
constexpr int kBuckets = 8192;
constexpr int kBins = 3 * kBuckets;

/* The class: by the distinct ids a query is expected to hold. A box of sides w, h meets about
 * D (w + e)(h + e) walks, D the density of walks there and e how far a walk reaches (from the mean
 * number of cells a walk has groups in, range_groups_launch). Grid: D from the list of the smallest
 * node around the query's centre that is no smaller than it, or the largest one with a list; the
 * bucket from the last node of that descent. FSG: D from the groups in the query's middle row of
 * cells, the bucket from its first cell. MortonGrid: D from the groups of the cells of a square about
 * as large as the query around its centre. STIG: the groups of the leaf at the query's lower corner,
 * times how often the query covers that leaf's sides. */
template <int KIND>
__global__ void k_order_class(const gat_mbb* queries, int nq, GroupsDev g, GridDev tree, FsgDev f, float reach, int* __restrict__ hist,
                              int* __restrict__ bin) {
    const int qi = blockIdx.x * blockDim.x + threadIdx.x;
    if (qi >= nq) return;
    const Box q = load_box(queries, qi);
    const float w = q.xmax - q.xmin, h = q.ymax - q.ymin;
    float density = 0.f; /* walks per unit area */
    float est = -1.f;
    float scan = 0.f;    /* groups of the candidates */
    int at = 0;          /* a group near the query's first one */
    if (KIND == GAT_INDEX_GRID) {
        const float cx = q.xmin + 0.5f * w, cy = q.ymin + 0.5f * h;
        NodeRec r = g.rec[0];
        bool set = false;
        for (int guard = 0; guard < 32; guard++) {
            const float nw = r.mbb.z - r.mbb.x, nh = r.mbb.w - r.mbb.y;
            if (!set && (r.child < 0 || (r.ib >= 0 && (0.5f * nw < w || 0.5f * nh < h)))) {
                density = (float)(r.ie - r.ib) / ((nw + reach) * (nh + reach));
                set = true;
            }
            if (r.child < 0) break;
            /* children UL, UR, DL, DR around the middle */
            const int c = (cx >= r.mbb.x + 0.5f * nw ? 1 : 0) + (cy < r.mbb.y + 0.5f * nh ? 2 : 0);
            r = g.rec[r.child + c];
        }
        at = max(r.ib, 0);
    } else if (KIND == GAT_INDEX_STIG) {
        NodeRec r = g.rec[0];
        for (int guard = 0; guard < 64 && r.child >= 0; guard++) {
            const float lo = r.aux & 1 ? q.ymin : q.xmin;
            r = g.rec[!(lo > r.mbb.x) ? r.child : r.aux >> 1];
        }
        at = max(r.ib, 0);
        const float kw = w / fmaxf(r.mbb.z - r.mbb.x, 1e-30f), kh = h / fmaxf(r.mbb.w - r.mbb.y, 1e-30f);
        est = (float)(r.ie - r.ib) * fmaxf(kw, 1.f) * fmaxf(kh, 1.f);
    } else if (KIND == GAT_INDEX_MORTON) {
        /* level whose squares are just larger than the query */
        const float side = fmaxf(fmaxf(w, h), tree.cell);
        int l = tree.total_level;
        while (l > 0 && tree.cell * (float)(1 << (tree.total_level - l)) < side) l--;
        const int cells = 1 << (tree.total_level - l), n = 1 << l;
        const float inv = 1.f / (tree.cell * (float)cells);
        const int x = min(n - 1, max(0, (int)fminf((q.xmin + 0.5f * w - tree.rxmin) * inv, 1e6f)));
        const int y = min(n - 1, max(0, (int)fminf((tree.rymax - q.ymin - 0.5f * h) * inv, 1e6f)));
        const uint32_t id = spread_bits((uint32_t)x) | (spread_bits((uint32_t)y) << 1), span = (uint32_t)cells * (uint32_t)cells;
        const float c = tree.cell + reach;
        at = g.cell_g[id * span];
        const float groups = (float)(g.cell_g[id * span + span] - at) / (float)span; /* per cell */
        density = groups / (c * c);
        scan = groups * (w / tree.cell) * (h / tree.cell);
    } else {
        const int g1 = max((int)__fdiv_rn(__fsub_rn(q.xmin, f.rxmin), f.cell), 0);
        const int g2 = min((int)__fdiv_rn(__fsub_rn(q.xmax, f.rxmin), f.cell), f.nx - 1);
        const int g3 = max((int)__fdiv_rn(__fsub_rn(f.rymax, q.ymax), f.cell), 0);
        const int g4 = min((int)__fdiv_rn(__fsub_rn(f.rymax, q.ymin), f.cell), f.ny - 1);
        if (g1 <= g2 && g3 <= g4) {
            const int row = ((g3 + g4) >> 1) * f.nx;
            const float c = f.cell + reach;
            at = g.cell_g[row + g1];
            const float groups = (float)(g.cell_g[row + g2 + 1] - at); /* of one row */
            density = groups / ((float)(g2 - g1 + 1) * c * c);
            scan = groups * (float)(g4 - g3 + 1);
        }
    }
    if (KIND == GAT_INDEX_STIG) scan = est;
    if (KIND != GAT_INDEX_STIG) est = density * (w + reach) * (h + reach);
    int cls = est <= kSmallMax ? 0 : est <= kMidMax ? 1 : 2; /* NaN: big */
    if (scan > (float)kSmallScan) cls = max(cls, scan <= (float)kMidScan ? 1 : 2);
    const int b = cls * kBuckets + (int)min((long long)kBuckets - 1, (long long)at * kBuckets / (g.n + 1));
    bin[qi] = b;
    atomicAdd(&hist[b], 1);
}

/* one CTA: exclusive scan of the bins in place; counts: queries below the mid and the big class */
__global__ void __launch_bounds__(1024) k_order_scan(int* hist, int* counts) {
    constexpr int kPer = kBins / 1024;
    __shared__ int warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int c[kPer], sum = 0;
    int4* mine = reinterpret_cast<int4*>(hist + threadIdx.x * kPer);
#pragma unroll
    for (int k = 0; k < kPer / 4; k++) {
        const int4 v = mine[k];
        c[4 * k] = v.x, c[4 * k + 1] = v.y, c[4 * k + 2] = v.z, c[4 * k + 3] = v.w;
        sum += v.x + v.y + v.z + v.w;
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int run = incl - sum;
    for (int w = 0; w < warp; w++) run += warp_sum[w];
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int b = threadIdx.x * kPer + k, n = c[k];
        if (b == kBuckets) counts[0] = run;
        if (b == 2 * kBuckets) counts[1] = run;
        c[k] = run;
        run += n;
    }
#pragma unroll
    for (int k = 0; k < kPer / 4; k++) mine[k] = make_int4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
}

__global__ void k_order(int nq, const int* __restrict__ bin, int* __restrict__ base, int* __restrict__ list) {
    const int qi = blockIdx.x * blockDim.x + threadIdx.x;
    if (qi < nq) list[atomicAdd(&base[bin[qi]], 1)] = qi;
}

}  // namespace

int range_groups_launch(gat_ctx* ctx, const gat_index* ix, const gat_mbb* d_q, int nq, uint32_t* arena, int64_t cap,
                        unsigned long long* ctr, int64_t* segbase, int64_t* segcnt, int* ovf_list, bool timed) {
    cudaStream_t s = ctx->stream;
    auto kernel = ix->kind == GAT_INDEX_GRID     ? k_range_groups<GAT_INDEX_GRID>
                  : ix->kind == GAT_INDEX_STIG   ? k_range_groups<GAT_INDEX_STIG>
                  : ix->kind == GAT_INDEX_MORTON ? k_range_groups<GAT_INDEX_MORTON>
                                                 : k_range_groups<GAT_INDEX_FSG>;
    auto classify = ix->kind == GAT_INDEX_GRID     ? k_order_class<GAT_INDEX_GRID>
                    : ix->kind == GAT_INDEX_STIG   ? k_order_class<GAT_INDEX_STIG>
                    : ix->kind == GAT_INDEX_MORTON ? k_order_class<GAT_INDEX_MORTON>
                                                   : k_order_class<GAT_INDEX_FSG>;
    allow_smem(kernel, kSmem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kNT, kSmem);
    const int full = std::max(1, per_sm) * ctx->sm_count;
    GAT_CUDA_TRY(ctx, cudaMemsetAsync(ctr, 0, 8 * sizeof(unsigned long long), s), "range");
    GroupQuery a{d_q, ix->grid, ix->fsg, ix->morton, ix->groups, arena, cap, ctr, segbase, segcnt, nullptr, nullptr, 0, nullptr, nullptr,
                 ovf_list, timed ? ctr + 1 : nullptr};
    a.points = (float)ix->npoints / (float)std::max(1, ix->groups.n);
    if (nq <= full) {
        /* no more queries than resident CTAs: one each, in block mode */
        kernel<<<nq, kNT, kSmem, s>>>(a, nullptr, nullptr, nq);
        count_launch(ctx);
        GAT_CUDA_TRY(ctx, cudaGetLastError(), "range scan launch");
        return GAT_OK;
    }
    /* [retry nq int2 | bins | counts 4 | bin nq | list nq] */
    int st = GAT_OK;
    char* p = (char*)scratch(ctx, S_RANGE_SPLIT, (size_t)nq * 16 + (size_t)(kBins + 4) * 4, &st);
    if (!p) return st;
    int* hist = reinterpret_cast<int*>(p);
    int* counts = hist + kBins;
    a.retry = reinterpret_cast<int2*>(counts + 4);
    int* bin = reinterpret_cast<int*>(a.retry + nq);
    int* list = bin + nq;
    const int tb = (nq + 255) / 256;
    GAT_CUDA_TRY(ctx, cudaMemsetAsync(hist, 0, kBins * 4, s), "range");
    const float cell = ix->kind == GAT_INDEX_STIG ? 0.f : ix->kind == GAT_INDEX_FSG ? ix->fsg.cell : ix->grid.cell;
    const float reach = cell * (std::sqrt(std::max(1.f, (float)ix->groups.n / (float)std::max(1, ix->db->n))) - 1.f);
    classify<<<tb, 256, 0, s>>>(d_q, nq, ix->groups, ix->grid, ix->fsg, reach, hist, bin);
    k_order_scan<<<1, 1024, 0, s>>>(hist, counts);
    k_order<<<tb, 256, 0, s>>>(nq, bin, hist, list);
    kernel<<<full, kNT, kSmem, s>>>(a, list, counts, nq);
    count_launch(ctx, 4);
    GAT_CUDA_TRY(ctx, cudaGetLastError(), "range scan launch");
    return GAT_OK;
}

int plain_groups_launch(gat_ctx* ctx, const gat_index* ix, const gat_mbb* d_q, int qi, int64_t* off, int32_t* out, int64_t capacity,
                        int* state, unsigned long long* work) {
    auto kernel = ix->kind == GAT_INDEX_GRID     ? k_plain_groups<GAT_INDEX_GRID>
                  : ix->kind == GAT_INDEX_STIG   ? k_plain_groups<GAT_INDEX_STIG>
                  : ix->kind == GAT_INDEX_MORTON ? k_plain_groups<GAT_INDEX_MORTON>
                                                 : k_plain_groups<GAT_INDEX_FSG>;
    if (qi == 0) allow_smem(kernel, kSmem);
    /* a walk has about G / n groups in all and no more of them in a rectangle; it is in one or two of a Grid's lists */
    const bool may_outgrow = ix->db->n > kBlockIds;
    const float share = may_outgrow ? std::min(1.f, (float)ix->db->n / (float)std::max(1, ix->groups.n)) : 0.f;
    GroupQuery a{d_q, ix->grid, ix->fsg, ix->morton, ix->groups, nullptr, 0, nullptr, nullptr, nullptr, off, out, capacity, state,
                 nullptr, nullptr, work};
    a.share[0] = share;
    a.share[1] = ix->kind == GAT_INDEX_GRID && may_outgrow ? 0.75f : share;
    /* the first launch of a call waits for all before it: the queries may come from a kernel */
    if (qi == 0)
        kernel<<<1, kNT, kSmem, ctx->stream>>>(a, qi);
    else
        (void)launch_dep(ctx, kernel, dim3(1), dim3(kNT), kSmem, ctx->stream, a, qi);
    count_launch(ctx);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? GAT_OK : cuda_fail(ctx, e, "range plain launch");
}

int group_points_launch(gat_ctx* ctx, const gat_index* ix, const gat_mbb* d_q, int nq, uint32_t* arena, int64_t cap,
                        unsigned long long* ctr, int64_t* segbase, int64_t* segcnt, int* ovf_list, int* again) {
    cudaStream_t s = ctx->stream;
    auto launch = [&](auto kind) -> int {
        constexpr int KIND = decltype(kind)::value;
        auto first = k_group_points<KIND, BlockTeam, false>;
        auto second = k_group_points<KIND, LongTeam, true>;
        constexpr size_t kLongSmem = (size_t)LongTeam::kInts * sizeof(int);
        allow_smem(first, kSmem);
        allow_smem(second, kLongSmem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, first, kNT, kSmem);
        GAT_CUDA_TRY(ctx, cudaMemsetAsync(ctr, 0, 8 * sizeof(unsigned long long), s), "range");
        GroupQuery a{d_q, ix->grid, ix->fsg, ix->morton, ix->groups, arena, cap, ctr, segbase, segcnt, nullptr, nullptr, 0,
                     nullptr, nullptr, ovf_list, nullptr};
        first<<<std::min(nq, std::max(1, per_sm) * ctx->sm_count), kNT, kSmem, s>>>(a, ix->d_key, nq, again);
        (void)launch_dep(ctx, second, dim3(std::min(nq, ctx->sm_count)), dim3(kNT), kLongSmem, s, a, (const uint32_t*)ix->d_key, nq,
                         again);
        count_launch(ctx);
        count_launch(ctx);
        GAT_CUDA_TRY(ctx, cudaGetLastError(), "range scan launch");
        return GAT_OK;
    };
    if (ix->kind == GAT_INDEX_GRID) return launch(std::integral_constant<int, GAT_INDEX_GRID>{});
    return launch(std::integral_constant<int, GAT_INDEX_MORTON>{});
}

}  // namespace gat
