// Treelet restructuring (Karras & Aila 2013) for sm_100a: one warp per treelet root,
// walking bottom-up from the leaves with an arrival counter per node, dynamic
// programming over the 128 leaf subsets staged in shared memory.
//
// Output is that of the reference's optimizeBVH (BVH/Optimization.cu:467-525 with
// optimizeTreelet :49-462) up to the rounding of surface areas (subset_area below): same
// treelet formation (expand the largest-area
// node, first lane on ties), same partition enumeration order per subset, the same
// warp min-reduction tree for the 6- and 7-leaf subsets, and the same reuse of node
// ids by lane during reconstruction.  It differs in mechanics only:
//   * a round starts from the nodes that are leaves when it starts (the reference tests
//     `isLeaf` inside the same launch that restructures the tree, Optimization.cu:479): a
//     separate pass climbs from them, a thread per leaf, to the lowest nodes with 7 leaves;
//   * the formation lanes keep their node records in registers, so every read of the
//     old treelet precedes every write, and the bottom-up box/cost refresh runs on
//     registers with explicit warp synchronisation (the reference iterates 7 times over
//     global memory without __syncwarp, :445-460; its converged values are the same);
//   * subsets of 2..5 leaves are processed grouped by size instead of by the
//     reference's hand-packed 5-round table (each subset's result depends only on the
//     smaller subsets, so the order between subsets does not change any value);
//   * a node whose subtree holds fewer than 7 leaves is not visited by the formation at
//     all (the reference's formation expands such a subtree and gives up without writing);
//   * the walkers are persistent warps that claim their starting nodes from a counter.
#include <cuda_runtime.h>

#include <algorithm>

#include "cav_internal.cuh"

namespace cav {

namespace {

constexpr unsigned kFull = 0xffffffffu;

struct SubsetTable {
    unsigned char s[112];
    int off[5];  // start of popcount 2,3,4,5 and the end
};

constexpr int popc7(int x) { return (x & 1) + ((x >> 1) & 1) + ((x >> 2) & 1) + ((x >> 3) & 1) + ((x >> 4) & 1) + ((x >> 5) & 1) + ((x >> 6) & 1); }

constexpr SubsetTable make_table() {
    SubsetTable t{};
    int k = 0;
    for (int pc = 2; pc <= 5; ++pc) {
        t.off[pc - 2] = k;
        for (int s = 1; s < 128; ++s)
            if (popc7(s) == pc) t.s[k++] = (unsigned char)s;
    }
    t.off[4] = k;
    return t;
}

__constant__ SubsetTable kSubsets = make_table();

struct __align__(16) WarpSmem {
    float area[128];
    float cost[128];
    float lbox[7][8];    // the treelet leaves' boxes (lo, hi, two unused: 16-byte loads, broadcast)
    int32_t lrec[7][4];  // and their left, right, prim, is_leaf
    float carea[8];      // and their areas as stored
    float pcost[64];     // partial minima of subsets whose partitions are split over lanes
    signed char ppart[64];
    signed char part[128];
};

struct Rec {
    float lo_x, lo_y, lo_z, hi_x, hi_y, hi_z;
    int32_t left, right, parent, prim;
    float area, cost;
    int32_t is_leaf;
};

__device__ inline Rec load_rec(const BNode* nodes, int32_t id) {
    const float4* p = reinterpret_cast<const float4*>(nodes + id);
    float4 a = __ldcg(p), b = __ldcg(p + 1), c = __ldcg(p + 2), d = __ldcg(p + 3);
    Rec r;
    r.lo_x = a.x; r.lo_y = a.y; r.lo_z = a.z; r.hi_x = a.w;
    r.hi_y = b.x; r.hi_z = b.y; r.left = __float_as_int(b.z); r.right = __float_as_int(b.w);
    r.parent = __float_as_int(c.x); r.prim = __float_as_int(c.y); r.area = c.z; r.cost = c.w;
    r.is_leaf = __float_as_int(d.x);
    return r;
}

__device__ inline void store_rec(BNode* nodes, int32_t id, const Rec& r) {
    float4* p = reinterpret_cast<float4*>(nodes + id);
    __stcg(p, make_float4(r.lo_x, r.lo_y, r.lo_z, r.hi_x));
    __stcg(p + 1, make_float4(r.hi_y, r.hi_z, __int_as_float(r.left), __int_as_float(r.right)));
    __stcg(p + 2, make_float4(__int_as_float(r.parent), __int_as_float(r.prim), r.area, r.cost));
    __stcg(p + 3, make_float4(__int_as_float(r.is_leaf), 0.f, 0.f, 0.f));
}

__device__ inline bool is_pow2(int n) { return (n & (n - 1)) == 0; }

// The reference's warp reduction of partition costs (Optimization.cu:224-266, :271-324): for
// d = 16, 8, 4, 2, 1 lane l takes lane min(l + d, 31)'s candidate when its own is the empty
// -1 or the other is smaller.  Lane 0 ends with the smallest cost; among equal costs with the
// lane whose 5-bit index read backwards is smallest (the bracket keeps the lower lane of
// every pair), and an empty candidate (only lane 0's can be) loses to any other.  Costs are
// non-negative floats, whose bit patterns order like their values, so two min-reductions find
// the same winner; a NaN or negative cost anywhere takes the reference's own loop.  Every lane
// returns lane 0's result.
__device__ inline void reduce_partition(float& tc, int& p) {
    const int lane = threadIdx.x & 31;
    const bool empty = tc == -1.f;
    if (__any_sync(kFull, !empty && !(tc >= 0.f))) {
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            const int o = min(lane + d, 31);
            const float oc = __shfl_sync(kFull, tc, o);
            const int op = __shfl_sync(kFull, p, o);
            if (tc == -1.f || oc < tc) {
                tc = oc;
                p = op;
            }
        }
        tc = __shfl_sync(kFull, tc, 0);
        p = __shfl_sync(kFull, p, 0);
        return;
    }
    const unsigned key = empty ? 0xffffffffu : __float_as_uint(tc + 0.f);  // +0 for a -0 cost
    const unsigned best = __reduce_min_sync(kFull, key);
    const unsigned rev = __brev((unsigned)lane) >> 27;
    const unsigned win = __brev(__reduce_min_sync(kFull, key == best ? rev : 0xffffffffu)) >> 27;
    tc = __shfl_sync(kFull, tc, (int)win);
    p = __shfl_sync(kFull, p, (int)win);
}

// The area of a union of treelet leaves, rounded as this pass always has: the other order of the
// contraction than surface_area (the build's, and the one that the reference's build kernels were
// seen to have).  Partitions whose costs are a rounding apart can fall the other way for it: trees
// of icospheres differ from the oracle's own rounding in a part of their nodes, and are the
// oracle's node for node with this one.
__device__ __forceinline__ float subset_area(f3 lo, f3 hi) {
    const f3 e = hi - lo;
    return 2.f * fmaf(e.x, e.z, fmaf(e.y, e.z, __fmul_rn(e.x, e.y)));
}

__device__ __forceinline__ void load_box(const WarpSmem& S, int k, f3& lo, f3& hi) {
    const float4 a = *reinterpret_cast<const float4*>(S.lbox[k]);
    const float2 b = *reinterpret_cast<const float2*>(S.lbox[k] + 4);
    lo = mk(a.x, a.y, a.z);
    hi = mk(a.w, b.x, b.y);
}

__device__ __forceinline__ void unite_box(const WarpSmem& S, int k, f3& lo, f3& hi) {
    f3 blo, bhi;
    load_box(S, k, blo, bhi);
    lo = vmin3(lo, blo);
    hi = vmax3(hi, bhi);
}

// The cost of subset `s` split into p and the rest.
__device__ __forceinline__ float split_cost(const WarpSmem& S, int s, int p) { return S.cost[p] + S.cost[s ^ p]; }

// Partitions first..last of subset s in the reference's order (Optimization.cu:180-216: the
// j-th is the j-th subset of s without its lowest bit, in increasing order), from partition p
// on; the first smallest wins.
__device__ __forceinline__ void best_of(const WarpSmem& S, int s, int p, int count, float& best, int& bestp) {
    const int cleared = (s - 1) & s;
    best = split_cost(S, s, p);
    bestp = p;
#pragma unroll 1
    for (int k = 1; k < count; ++k) {
        p = (p - cleared) & s;
        const float c = split_cost(S, s, p);
        if (c < best) {
            best = c;
            bestp = p;
        }
    }
}

// The j-th subset of `m` in increasing order (bit i of j to the i-th bit of m), m of at most
// four bits.
__device__ __forceinline__ int nth_subset(int m, int j) {
    int r = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int low = m & -m;
        if ((j >> i) & 1) r |= low;
        m ^= low;
    }
    return r;
}

__device__ __forceinline__ void put_subset(WarpSmem& S, int s, float best, int bestp) {
    S.cost[s] = internal_cost(S.area[s], best);
    S.part[s] = (signed char)bestp;
}

// The best partition of every subset of 2..7 leaves, with the reference's choice among equal
// costs (the first smallest in its order).  Subsets of 2 and 3 leaves take a lane each; the
// last three of the 35 of 4 leaves and all 21 of 5 leaves are split over lanes, whose partial
// minima are then taken in order; the 7 of 6 leaves take four lanes each: the reference's
// bracket keeps, among equal costs, the partition whose 5-bit number read backwards is
// smallest, so lane c of a subset takes the numbers 8 c .. 8 c + 7 in that reading.  21
// steps of a cost sum and a comparison, where a lane per subset and a warp reduction per
// 6-leaf subset took 36 and seven reductions.  With the boxes and records
// taken from the subsets (below) a round over the 1M-triangle soup executes 644 M warp
// instructions, 795 M before, and three rounds take 4.13 ms, 4.47 before; issue slots (57 %
// used) and the waits for node fetches bound the walk.
__device__ __forceinline__ void split_subsets(WarpSmem& S) {
    const int lane = threadIdx.x & 31;
    float best;
    int bestp;
    // 2 leaves: one partition each
    if (lane < 21) {
        const int s = kSubsets.s[lane], p = (s - 1) & s;
        put_subset(S, s, split_cost(S, s, p), p);
    }
    __syncwarp();
    // 3 leaves: three partitions each, 35 subsets
#pragma unroll 1
    for (int k = lane; k < 35; k += 32) {
        const int s = kSubsets.s[kSubsets.off[1] + k];
        best_of(S, s, -((s - 1) & s) & s, 3, best, bestp);
        put_subset(S, s, best, bestp);
    }
    __syncwarp();
    // 4 leaves: seven partitions each; the last three subsets one partition per lane
    {
        const int s = kSubsets.s[kSubsets.off[2] + lane];
        best_of(S, s, -((s - 1) & s) & s, 7, best, bestp);
        put_subset(S, s, best, bestp);
        if (lane < 21) {
            const int k = lane / 7;
            const int s3 = kSubsets.s[kSubsets.off[2] + 32 + k];
            const int p = nth_subset((s3 - 1) & s3, lane - 7 * k + 1);
            S.pcost[lane] = split_cost(S, s3, p);
            S.ppart[lane] = (signed char)p;
        }
        __syncwarp();
        if (lane < 3) {
            best = S.pcost[7 * lane];
            int at = 7 * lane;
#pragma unroll
            for (int j = 1; j < 7; ++j)
                if (S.pcost[7 * lane + j] < best) {
                    best = S.pcost[7 * lane + j];
                    at = 7 * lane + j;
                }
            put_subset(S, kSubsets.s[kSubsets.off[2] + 32 + lane], best, S.ppart[at]);
        }
    }
    __syncwarp();
    // 5 leaves: fifteen partitions each, in three parts of five
    {
#pragma unroll 1
        for (int k = lane; k < 63; k += 32) {
            const int q = k / 3;
            const int s = kSubsets.s[kSubsets.off[3] + q];
            best_of(S, s, nth_subset((s - 1) & s, 5 * (k - 3 * q) + 1), 5, best, bestp);
            S.pcost[k] = best;
            S.ppart[k] = (signed char)bestp;
        }
        __syncwarp();
        if (lane < 21) {
            best = S.pcost[3 * lane];
            int at = 3 * lane;
#pragma unroll
            for (int j = 1; j < 3; ++j)
                if (S.pcost[3 * lane + j] < best) {
                    best = S.pcost[3 * lane + j];
                    at = 3 * lane + j;
                }
            put_subset(S, kSubsets.s[kSubsets.off[3] + lane], best, S.ppart[at]);
        }
    }
    __syncwarp();
    // 6 leaves (Optimization.cu:224-266): partition number l of the subset without leaf eb
    // (lane l's in the reference) is l with a zero bit put in at eb, for eb = 6 with its upper
    // bits dropped (the reference's shift by -1)
    {
        const int eb = min(lane >> 2, 6), c = lane & 3;
        const int s = 0x7f ^ (1 << eb);
        best = INFINITY;
        bestp = 0;
        bool none = true;
#pragma unroll
        for (int r = 0; r < 8; ++r) {  // l = bit-reversed (8 c + r)
            const int l = ((r & 1) << 4) | ((r & 2) << 2) | (r & 4) | ((c & 1) << 1) | (c >> 1);
            const int hi = eb <= 5 ? ((l << 1) & (((1 << (5 - eb)) - 1) << (eb + 1))) : 0;
            const int p = (l & ((1 << eb) - 1)) | hi;
            const float t = split_cost(S, s, p);
            if (p != 0 && (none || t < best)) {
                best = t;
                bestp = p;
                none = false;
            }
        }
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) {  // the lower lane keeps equal costs
            const float ob = __shfl_xor_sync(kFull, best, d);
            const int op = __shfl_xor_sync(kFull, bestp, d);
            const bool on = __shfl_xor_sync(kFull, none ? 1 : 0, d) != 0;
            const bool upper = (c & d) != 0;
            if (!on && (none || ob < best || (ob == best && upper))) {
                best = ob;
                bestp = op;
                none = false;
            }
        }
        if (c == 0 && lane < 28) put_subset(S, s, best, bestp);
    }
    __syncwarp();
    // all 7 leaves (Optimization.cu:271-324)
    {
        int p = lane;
        float tc = -1.f;
        if (p != 0) tc = split_cost(S, 0x7f, p);
        const int op = lane | 32;
        const float otc = split_cost(S, 0x7f, op);
        if (tc == -1.f || otc < tc) {
            tc = otc;
            p = op;
        }
        reduce_partition(tc, p);
        if (lane == 0) put_subset(S, 0x7f, tc, p);
    }
    __syncwarp();
}

// The same with the reference's own loops, for costs that do not order (NaN or negative).
__device__ __noinline__ void plain_subsets(WarpSmem& S) {
    const int lane = threadIdx.x & 31;
    // ---- subsets of 2..5 leaves (Optimization.cu:180-216), grouped by size
#pragma unroll 1
    for (int g = 0; g < 4; ++g) {
        const int b = kSubsets.off[g], e = kSubsets.off[g + 1];
#pragma unroll 1
        for (int k0 = b; k0 < e; k0 += 32) {
            int k = k0 + lane;
            if (k < e) {
                int s = kSubsets.s[k];
                float best = -1.f;
                int bestp = 0;
                int cleared = (s - 1) & s;
                int p = (0 - cleared) & s;
                do {
                    float tc = S.cost[p] + S.cost[s ^ p];
                    if (best == -1.f || tc < best) {
                        bestp = p;
                        best = tc;
                    }
                    p = (p - cleared) & s;
                } while (p != 0);
                S.cost[s] = internal_cost(S.area[s], best);
                S.part[s] = (signed char)bestp;
            }
        }
        __syncwarp();
    }

    // ---- 6-leaf subsets (Optimization.cu:224-266): partition per lane, then the
    // reference's lane-order min reduction (lane l reads lane min(l+d, 31)).
#pragma unroll 1
    for (int eb = 0; eb < 7; ++eb) {
        int s = 0x7f ^ (1 << eb);
        int hi = eb <= 5 ? ((lane << 1) & (((1 << (5 - eb)) - 1) << (eb + 1))) : 0;
        int p = (lane & ((1 << eb) - 1)) | hi;
        float tc = -1.f;
        if (p != 0) tc = S.cost[p] + S.cost[s ^ p];
        reduce_partition(tc, p);
        if (lane == 0) {
            S.cost[s] = internal_cost(S.area[s], tc);
            S.part[s] = (signed char)p;
        }
        __syncwarp();
    }

    // ---- all 7 leaves (Optimization.cu:271-324)
    {
        const int s = 0x7f;
        int p = lane;
        float tc = -1.f;
        if (p != 0) tc = S.cost[p] + S.cost[s ^ p];
        int op = lane | 32;
        float otc = S.cost[op] + S.cost[s ^ op];
        if (tc == -1.f || otc < tc) {
            tc = otc;
            p = op;
        }
        reduce_partition(tc, p);
        if (lane == 0) {
            S.cost[s] = internal_cost(S.area[s], tc);
            S.part[s] = (signed char)p;
        }
        __syncwarp();
    }
}

// optimizeTreelet semantics for the subtree rooted at `root`, whose parent it reports (it never
// changes).  Returns false only on
// an internal inconsistency (recorded in *err by the caller).
__device__ bool optimize_treelet(BNode* nodes, int32_t root, int32_t count, WarpSmem& S, int32_t& root_parent) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;

    // ---- formation (Optimization.cu:59-107)
    int32_t nid = -1;
    Rec rec{};
    if (lane == 0) {
        nid = root;
        rec = load_rec(nodes, root);
    }
    root_parent = __shfl_sync(kFull, rec.parent, 0);
    bool expanded = false;
    int size = 1;
    while (size < 13) {
        // the first of lanes 0..size-1 with the largest area above -1 (lane 0 when none):
        // areas are non-negative, so their bit patterns order like their values
        const bool cand = lane < size && !(rec.is_leaf || expanded) && rec.area > -1.f;
        int max_lane = 0;
        if (__any_sync(kFull, cand && !(rec.area >= 0.f))) {  // a negative area: a plain scan
            float my_area = rec.area;
            if (rec.is_leaf || expanded) my_area = -1.f;
            float max_area = -1.f;
            for (int i = 0; i < size; ++i) {
                float a = __shfl_sync(kFull, my_area, i);
                if (a > max_area) {
                    max_area = a;
                    max_lane = i;
                }
            }
        } else {
            const unsigned key = cand ? __float_as_uint(rec.area + 0.f) + 1u : 0u;
            const unsigned top = __reduce_max_sync(kFull, key);
            if (top != 0u) max_lane = __ffs(__ballot_sync(kFull, key == top)) - 1;
        }
        int stop = __shfl_sync(kFull, (int)(expanded || rec.is_leaf), max_lane);
        if (stop) return true;  // fewer than 7 leaves reachable: leave the subtree as it is
        int32_t cl = __shfl_sync(kFull, rec.left, max_lane);
        int32_t cr = __shfl_sync(kFull, rec.right, max_lane);
        if (cl < 0 || cr < 0 || cl >= count || cr >= count) return false;
        if (lane == max_lane) expanded = true;
        if (lane == size) {
            nid = cl;
            rec = load_rec(nodes, cl);
        }
        if (lane == size + 1) {
            nid = cr;
            rec = load_rec(nodes, cr);
        }
        size += 2;
    }
    const bool in_treelet = lane < 13;
    const unsigned leaf_mask = __ballot_sync(kFull, in_treelet && !expanded);
    const int my_leaf = __popc(leaf_mask & lt);

    // ---- subset areas (Optimization.cu:126-163)
    // the leaves' records go through shared memory rather than registers (the walk's
    // occupancy is set by its registers)
    if (in_treelet && !expanded) {
        float4* b = reinterpret_cast<float4*>(S.lbox[my_leaf]);
        b[0] = make_float4(rec.lo_x, rec.lo_y, rec.lo_z, rec.hi_x);
        b[1] = make_float4(rec.hi_y, rec.hi_z, 0.f, 0.f);
        *reinterpret_cast<int4*>(S.lrec[my_leaf]) = make_int4(rec.left, rec.right, rec.prim, rec.is_leaf);
    }
    __syncwarp();
    // Subset s = (q << 5) | lane: the union of the lane's leaves 0-4 (its low five bits) is
    // taken once, then leaves 5 and 6 per quarter q.
    f3 lo, hi;
    load_box(S, lane != 0 ? __ffs(lane) - 1 : 5, lo, hi);
#pragma unroll
    for (int k = 1; k < 5; ++k)
        if ((lane >> k) & 1) unite_box(S, k, lo, hi);
    S.area[lane] = lane != 0 ? subset_area(lo, hi) : 0.f;
    {
        f3 l6, h6;
        load_box(S, 6, l6, h6);
        if (lane != 0) {
            l6 = vmin3(lo, l6);
            h6 = vmax3(hi, h6);
            unite_box(S, 5, lo, hi);
        }
        S.area[32 | lane] = subset_area(lo, hi);
        S.area[64 | lane] = subset_area(l6, h6);
        unite_box(S, 6, lo, hi);
        S.area[96 | lane] = subset_area(lo, hi);
    }
    if (in_treelet && !expanded) {
        S.cost[1 << my_leaf] = rec.cost;
        S.carea[my_leaf] = rec.area;
    }
    __syncwarp();

    // costs are finite or infinite but never NaN or negative, or the reference's own loops run
    bool plain = in_treelet && !expanded && !(rec.cost >= 0.f);
#pragma unroll
    for (int q = 0; q < 4; ++q) plain = plain || !(S.area[(q << 5) | lane] >= 0.f);
    if (__any_sync(kFull, plain)) plain_subsets(S);
    else split_subsets(S);

    // ---- reconstruction (Optimization.cu:330-394): lane i keeps node nid and takes a role
    int my_subset = lane == 0 ? 0x7f : -1;
    bool exp_r = false;
    int par_lane = 0, cl_lane = lane, cr_lane = lane;
    int rsize = 1;
    while (rsize < 13) {
        const bool prop = lane < rsize && !exp_r && !is_pow2(my_subset);
        const unsigned m = __ballot_sync(kFull, prop);
        if (m == 0) return false;
        const int sel_lane = __ffs(m) - 1;
        const int sel = __shfl_sync(kFull, my_subset, sel_lane);
        if (sel <= 0 || sel > 127 || is_pow2(sel)) return false;
        const int pp = S.part[sel];
        if (pp <= 0 || (pp & ~sel) != 0) return false;
        if (lane == sel_lane) {
            exp_r = true;
            cl_lane = rsize;
            cr_lane = rsize + 1;
        }
        if (lane == rsize) my_subset = pp;
        if (lane == rsize + 1) my_subset = sel ^ pp;
        if (lane == rsize || lane == rsize + 1) par_lane = sel_lane;
        rsize += 2;
    }

    // ---- new records (Optimization.cu:400-461).  A node's box is the union of its leaves'
    // (min and max do not depend on the order), its area the subset's; a treelet leaf keeps
    // the cost it was stored with, which is what computing it again gives: its own treelet was
    // finished, and its children's costs final, before this root was reached.
    Rec nr;
    {
        const int32_t up = __shfl_sync(kFull, nid, par_lane);
        nr.parent = lane == 0 ? rec.parent : up;
    }
    const int32_t child_l = __shfl_sync(kFull, nid, cl_lane);
    const int32_t child_r = __shfl_sync(kFull, nid, cr_lane);
    const int subset = in_treelet ? my_subset : 1;
    const int leaf_id = __ffs(subset) - 1;
    f3 nlo, nhi;
    load_box(S, leaf_id, nlo, nhi);
#pragma unroll
    for (int k = 1; k < 7; ++k)
        if ((subset >> k) & 1) unite_box(S, k, nlo, nhi);
    nr.lo_x = nlo.x; nr.lo_y = nlo.y; nr.lo_z = nlo.z;
    nr.hi_x = nhi.x; nr.hi_y = nhi.y; nr.hi_z = nhi.z;
    nr.area = S.area[subset];
    int32_t old_l = 0, old_r = 0;
    if (exp_r) {
        nr.left = child_l;
        nr.right = child_r;
        nr.prim = -1;
        nr.is_leaf = 0;
        nr.cost = 0.f;
    } else {
        const int4 o = *reinterpret_cast<const int4*>(S.lrec[leaf_id]);
        nr.left = old_l = o.x;
        nr.right = old_r = o.y;
        nr.prim = o.z;
        nr.is_leaf = o.w;
        nr.cost = S.cost[1 << leaf_id];
        // where the stored area was rounded another way (a node that the refit wrote), the cost
        // follows the area; the children's costs are final
        if (in_treelet && nr.area != S.carea[leaf_id]) {
            if (nr.is_leaf) nr.cost = leaf_cost(nr.area, 1);
            else if (old_l >= 0 && old_r >= 0 && old_l < count && old_r < count)
                nr.cost = internal_cost(nr.area, __ldcg(&nodes[old_l].cost), __ldcg(&nodes[old_r].cost));
        }
    }
    // costs from the last pair of children to the first: lanes 2 k + 1 and 2 k + 2 hang
    // under the lane that took them, always a lower one
#pragma unroll
    for (int k = 11; k >= 1; k -= 2) {
        const float ca = __shfl_sync(kFull, nr.cost, k);
        const float cb = __shfl_sync(kFull, nr.cost, k + 1);
        if (cl_lane == k && lane != k) nr.cost = internal_cost(nr.area, ca, cb);
    }
    if (in_treelet) {
        store_rec(nodes, nid, nr);
        if (!exp_r && !nr.is_leaf && old_l >= 0 && old_r >= 0 && old_l < count && old_r < count) {
            __stcg(&nodes[old_l].parent, nid);
            __stcg(&nodes[old_r].parent, nid);
        }
    }
    __syncwarp();
    return true;
}

// A leaf's climb to the first node with 7 or more leaves under it (a subtree of fewer cannot form
// a treelet: the reference's formation then expands every internal node of it and gives up
// without writing anything; with 7 or more an internal node always remains to expand).  Each
// node's arrival counter holds the leaves of its first child to arrive (saturated at 7); the
// second arrival goes on, and returns the node once it counts 7.  -1: another leaf goes on.
__device__ int32_t seed_climb(const BNode* __restrict__ nodes, int32_t curr, int32_t count, uint32_t* visited, int* err) {
    uint32_t leaves = 1;
    while (curr != 0) {
        const int32_t parent = nodes[curr].parent;
        if (parent < 0 || parent >= count) {
            atomicExch(err, 2);
            return -1;
        }
        const uint32_t old = atomicAdd(visited + parent, (leaves << 2) | 1u);
        if ((old & 3u) != 1u) return -1;
        leaves = min(7u, leaves + (old >> 2));
        curr = parent;
        if (leaves >= 7) return curr;
    }
    return -1;
}

// The round's seeds: a thread per leaf climbs the small subtrees.  With a warp per leaf the
// walkers spent a third of the round on climbs that ended below a treelet (three rounds on the
// 1M-triangle soup 4.13 ms, 2.92 with this pass).
__global__ void k_treelet_seeds(const BNode* __restrict__ nodes, int64_t count, int32_t* __restrict__ list,
                                uint32_t* __restrict__ counter, uint32_t* visited, int* err) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t seed = -1;
    if (i < count && nodes[i].is_leaf) seed = seed_climb(nodes, (int32_t)i, (int32_t)count, visited, err);
    __syncwarp();
    const unsigned m = __ballot_sync(kFull, seed >= 0);
    if (m == 0) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(kFull, base, __ffs(m) - 1);
    const uint32_t pos = base + __popc(m & ((1u << lane) - 1u));
    if (seed >= 0 && pos < (uint32_t)((count + 1) / 2)) list[pos] = seed;
}

// optimizeBVHImpl (Optimization.cu:467-507): a warp per seed optimises its treelet and walks up;
// the second arrival at a node optimises the treelet rooted there and continues.  The
// counter's update is an acquire-release atomic: the lanes' record writes precede it (warp
// barrier), and the second arrival's reads follow it.
__device__ void treelet_walk(BNode* nodes, int32_t curr, int32_t count, uint32_t* visited, WarpSmem& S, int* err) {
    const int lane = threadIdx.x & 31;
    if (curr < 0 || curr >= count) {
        if (lane == 0) atomicExch(err, 2);
        return;
    }
    for (;;) {
        int32_t parent = -1;
        if (!optimize_treelet(nodes, curr, count, S, parent)) {
            if (lane == 0) atomicExch(err, 2);
            return;
        }
        __syncwarp();
        if (curr == 0) return;
        if (parent < 0 || parent >= count) {
            if (lane == 0) atomicExch(err, 2);
            return;
        }
        uint32_t old = 0;
        if (lane == 0)
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
                         : "=r"(old)
                         : "l"(visited + parent), "r"((7u << 2) | 1u)
                         : "memory");
        old = __shfl_sync(kFull, old, 0);
        if ((old & 3u) != 1u) return;  // first arrival stops; the second optimises the parent
        __syncwarp();
        curr = parent;
    }
}

// Persistent walkers: a fixed grid of 2-warp blocks, 24 per SM (48 warps at 40 registers),
// each warp claiming seeds from a counter until the list is exhausted.  The walk
// waits on atomics and dependent loads, so resident walkers matter more than registers,
// and a persistent warp never waits for a block launch after a first arrival ends its walk.
// Measured on 3 rounds over a 1M-triangle soup: one launched warp per leaf in 1-warp blocks
// (32 per SM, 64 registers) 7.14 ms; persistent 1-warp blocks at 64 registers 5.67;
// 2-warp blocks at 48 registers (40 per SM) 5.46; at 40 registers 5.34, 5.00 with the leaf
// boxes in shared memory, 4.93 with the leaf records there too, 4.72 with the subset boxes
// built from per-lane partial unions; at 32 registers (64 per SM) 5.99 (spills).
constexpr int kWalkWarps = 2;
constexpr int kWalkBlocksPerSm = 24;
__global__ void __launch_bounds__(kWalkWarps * 32, kWalkBlocksPerSm)
    k_treelet(BNode* nodes, const int32_t* __restrict__ list, int64_t n, uint32_t* visited, int* err,
              const uint32_t* __restrict__ seeds, uint32_t* claim) {
    __shared__ WarpSmem smem[kWalkWarps];
    WarpSmem& S = smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const uint32_t total = min(*seeds, (uint32_t)n);
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(claim, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= total) return;
        treelet_walk(nodes, list[i], (int32_t)(2 * n - 1), visited, S, err);
        __syncwarp();
    }
}

// ---- many trees per launch (the batched build): tree k owns leaves [leaf_off[k],
// leaf_off[k+1]) of the concatenated numbering and nodes [2 leaf_off[k] - k, ...) of the
// concatenated node numbering (2 n_k - 1 each).  A launch covers trees [k0, k1); a thread or
// warp finds its tree by binary search over the offsets.
__device__ inline int64_t node_off(const int64_t* leaf_off, int k) { return 2 * leaf_off[k] - k; }

__global__ void k_treelet_seeds_batch(const TreeletSeg* __restrict__ segs, const int64_t* __restrict__ leaf_off, int k0,
                                      int k1, int2* __restrict__ list, uint32_t* __restrict__ counter, uint32_t* visited,
                                      int* err) {
    const int64_t i = node_off(leaf_off, k0) + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int k = k0;
    int32_t seed = -1;
    if (i < node_off(leaf_off, k1)) {
        int lo = k0, hi = k1 - 1;  // the tree whose node range holds i
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (node_off(leaf_off, mid) <= i) lo = mid;
            else hi = mid - 1;
        }
        k = lo;
        const int64_t at = node_off(leaf_off, k), local = i - at;
        const int32_t count = (int32_t)(2 * segs[k].n - 1);
        if (local < count && segs[k].nodes[local].is_leaf)
            seed = seed_climb(segs[k].nodes, (int32_t)local, count, visited + at, err);
    }
    __syncwarp();
    const unsigned m = __ballot_sync(kFull, seed >= 0);
    if (m == 0) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(kFull, base, __ffs(m) - 1);
    const int64_t pos = (int64_t)base + __popc(m & ((1u << lane) - 1u));
    // a seed has 7 leaves or more of its own, so two words per seed fit the group's leaves
    if (seed >= 0 && 2 * pos + 1 < leaf_off[k1] - leaf_off[k0]) list[pos] = make_int2(k, seed);
}

// The same persistent walkers over a group of trees: a seed names its tree.
__global__ void __launch_bounds__(kWalkWarps * 32, kWalkBlocksPerSm)
    k_treelet_batch(const TreeletSeg* __restrict__ segs, const int64_t* __restrict__ leaf_off,
                    const int2* __restrict__ list, uint32_t most, uint32_t* visited, int* err,
                    const uint32_t* __restrict__ seeds, uint32_t* claim) {
    __shared__ WarpSmem smem[kWalkWarps];
    WarpSmem& S = smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const uint32_t total = min(*seeds, most);  // what the list holds, also of a build that failed
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(claim, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= total) return;
        const int2 s = list[i];
        treelet_walk(segs[s.x].nodes, s.y, (int32_t)(2 * segs[s.x].n - 1), visited + node_off(leaf_off, s.x), S, err);
        __syncwarp();
    }
}

}  // namespace

cav_status treelet_rounds(cav_ctx* ctx, BNode* nodes, int64_t n, int rounds, int32_t* leaf_list, uint32_t* visited,
                          uint32_t* counter, cudaStream_t s) {
    if (rounds <= 0) return CAV_OK;
    const int64_t count = 2 * n - 1;
    // counter[0]: the seeds listed, counter[1]: the walkers' claims; both in the
    // build's own scratch (builds on different streams, such as a server's lanes, never share it)
    // at most n / 7 seeds: their subtrees are disjoint
    const int64_t grid = std::min<int64_t>(div_up(div_up(n, 7) + 1, kWalkWarps), (int64_t)ctx->num_sms * kWalkBlocksPerSm);
    for (int r = 0; r < rounds; ++r) {
        CAV_CUDA(ctx, cudaMemsetAsync(visited, 0, sizeof(uint32_t) * count, s));
        CAV_CUDA(ctx, cudaMemsetAsync(counter, 0, 2 * sizeof(uint32_t), s));
        k_treelet_seeds<<<div_up(count, 256), 256, 0, s>>>(nodes, count, leaf_list, counter, visited, ctx->d_error + 1);
        k_treelet<<<(unsigned)grid, kWalkWarps * 32, 0, s>>>(nodes, leaf_list, n, visited, ctx->d_error + 1, counter,
                                                             counter + 1);
    }
    CAV_CUDA(ctx, cudaGetLastError());
    return CAV_OK;
}

// Treelet rounds of K trees, a group of consecutive trees at a time: per group and round one
// seeds launch and one treelet launch over all its trees (rather than two per tree).  A
// group holds at most kGroupLeaves leaves; a tree that fills a group alone runs the
// single-tree pass (measured: the grouped kernels were 1.3x slower than it on trees of
// 0.5-2M triangles, and launch overhead does not matter there).  Each tree's result is the
// single-tree one: within a tree the walk is the same, and trees share no nodes.  segs /
// leaf_off: device tables (K trees, K + 1 leaf offsets), segs_host / leaf_off_host the same
// on the host; leaf_list holds leaf_off[K] entries, visited 2 leaf_off[K] - K, counters K + 2
// (the last two are used).
cav_status treelet_rounds_batch(cav_ctx* ctx, const TreeletSeg* segs, const TreeletSeg* segs_host,
                                const int64_t* leaf_off, const int64_t* leaf_off_host, int K, int rounds,
                                int32_t* leaf_list, uint32_t* counters, uint32_t* visited, cudaStream_t s) {
    if (rounds <= 0 || K <= 0) return CAV_OK;
    constexpr int64_t kGroupLeaves = (int64_t)1 << 19;
    auto node_off_h = [&](int k) { return 2 * leaf_off_host[k] - k; };
    for (int k0 = 0; k0 < K;) {
        int k1 = k0 + 1;
        while (k1 < K && leaf_off_host[k1 + 1] - leaf_off_host[k0] <= kGroupLeaves) ++k1;
        const int64_t leaves = leaf_off_host[k1] - leaf_off_host[k0];
        const int64_t nodes = node_off_h(k1) - node_off_h(k0);
        if (k1 == k0 + 1 && leaves >= kGroupLeaves / 2) {
            cav_status st = treelet_rounds(ctx, segs_host[k0].nodes, segs_host[k0].n, rounds,
                                           leaf_list + leaf_off_host[k0], visited + node_off_h(k0), counters + K, s);
            if (st != CAV_OK) return st;
            k0 = k1;
            continue;
        }
        const int64_t grid =
            std::min<int64_t>(div_up(div_up(leaves, 7) + 1, kWalkWarps), (int64_t)ctx->num_sms * kWalkBlocksPerSm);
        for (int r = 0; r < rounds; ++r) {
            CAV_CUDA(ctx, cudaMemsetAsync(visited + node_off_h(k0), 0, sizeof(uint32_t) * nodes, s));
            CAV_CUDA(ctx, cudaMemsetAsync(counters + K, 0, 2 * sizeof(uint32_t), s));  // seeds, the walkers' claims
            int2* list = reinterpret_cast<int2*>(leaf_list);
            k_treelet_seeds_batch<<<div_up(nodes, 256), 256, 0, s>>>(segs, leaf_off, k0, k1, list, counters + K, visited,
                                                                     ctx->d_error + 1);
            k_treelet_batch<<<(unsigned)grid, kWalkWarps * 32, 0, s>>>(segs, leaf_off, list, (uint32_t)(leaves / 2), visited,
                                                                      ctx->d_error + 1, counters + K, counters + K + 1);
        }
        k0 = k1;
    }
    CAV_CUDA(ctx, cudaGetLastError());
    return CAV_OK;
}

}  // namespace cav
