// Device helpers shared by the traversal kernels (trace.cu: the binary exact mode;
// wide.cu: the compressed 8-wide fast mode): the triangle test, the triangle record load
// and the persistent warps' work claim.
#pragma once

#include "cav_internal.cuh"

namespace cav {

constexpr uint32_t kMaxSteps = 1u << 22;  // default node+triangle visits per ray before the ray is stopped
// Bits of a traversal kind's error word (cav_sync_check maps them to a cav_status).
constexpr int kFlagStackOverflow = 1;  // a push found the traversal stack full
constexpr int kFlagStepLimit = 2;      // a ray reached the context's step limit
// The exact mode always traverses the binary tree of up to this many triangles: a wide node costs
// as much as the few binary nodes it replaces (36 triangles, closest hit, 1M rays: 0.132 ms against
// 0.189; the room's shadow rays at 256x256, 16 samples 0.38 against 0.43).  Above it the two are
// level at first and the view gains with size (4,096 and 1M rays, binary and view: 129 triangles of
// a soup 33 and 32 us, 0.143 and 0.111 ms, 1,000 64 and 45 us, 0.246 and 0.232 ms; spheres of 298
// 35 and 35 us, 0.150 and 0.136 ms).
constexpr int64_t kTinyTris = 128;
constexpr int kDefaultRefill = 4;         // idle lanes that trigger a warp's next claim
// Node groups of the fast mode's stack kept per lane in shared memory when the autotuner
// picks that placement (a lane holds at most one group per wide level).
constexpr int kWideSmemStack = 8;
constexpr unsigned kFull = 0xffffffffu;

// rayTriangleIntersection (Core/Triangle.h:7-57) on precomputed edges.
__device__ inline bool tri_test(const f3& o, const f3& d, const f3& v0, const f3& e1, const f3& e2, float& t, float& u,
                                float& v) {
    f3 tvec = o - v0;
    f3 pvec = cross3(d, e2);
    float det = dot3(e1, pvec);
    if (det == 0) return false;
    det = 1.f / det;
    u = dot3(tvec, pvec) * det;
    if (u < 0.0f || u > 1.0f) return false;
    f3 qvec = cross3(tvec, e1);
    v = dot3(d, qvec) * det;
    if (v < 0.0f || (u + v) > 1.0f) return false;
    t = dot3(e2, qvec) * det;
    if (t <= 0.f) return false;
    return true;
}

__device__ inline void load_tri(const TriRec* __restrict__ tris, int64_t slot, f3& v0, f3& e1, f3& e2, int& id,
                                int& mesh) {
    const float4* p = reinterpret_cast<const float4*>(tris + slot);
    float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    v0 = mk(a.x, a.y, a.z);
    id = __float_as_int(a.w);
    e1 = mk(b.x, b.y, b.z);
    mesh = __float_as_int(b.w);
    e2 = mk(c.x, c.y, c.z);
}

// Device counters of one build of a tree's 8-wide view (wide.cu).  nodes[l % 3]: wide nodes
// allocated for level l; level l allocates from nodes[(l + 1) % 3] and nodes[l % 3] is cleared again
// one level later, so one grid barrier per level is enough.
struct WideCtr {
    uint32_t nodes[3];
    uint32_t tris;      // triangles placed
    uint32_t want;      // and to be placed
    uint32_t bar;       // arrivals at the grid barrier, all levels
    uint32_t failed;    // a barrier wait ran out, or the level bound was reached
    uint32_t unscreened;  // a triangle or the scene box outside the screening pass's range
    float margin;       // of the quantised boxes
    float area;         // the triangles' own boxes, half areas summed (in no fixed order)
    float root_area;    // and the scene box's
};

// Closest hits go through the view where a line through the scene meets few triangles' boxes, or
// the rays are few.  The search of the view follows the whole line, the binary traversal stops at
// the hit but walks more nodes, and its launch waits for its longest ray: lines that meet 4 boxes
// (1.3M triangles of spheres, 4M rays) 0.99 ms against 3.4 in the binary tree, 14 boxes (20,000 of a
// soup, 1M rays) 1.29 against 1.40, 40 boxes (60,000) 262,144 rays 1.19 against 1.41 and 1M rays 3.1
// against 2.6, 131 boxes (200,000) 65,536 rays 1.4 against 2.5 and 1M rays 9.0 against 6.0, 655 boxes
// (1M) 65,536 rays 6.1 against 8.9, 262,144 rays 14.8 against 11.9 and 4M rays 158 against 66.
constexpr float kSparse = 12.f;
constexpr int64_t kFewRays = 3 << 16;

// Whether the view serves n rays of the exact mode.
__device__ inline bool view_serves(const WideCtr* c, bool any_hit, int64_t n) {
    if (c->failed || c->tris != c->want || c->unscreened) return false;
    return any_hit || n <= kFewRays || c->area <= kSparse * c->root_area;
}

__device__ inline float imax_f(float a, float b) { return __int_as_float(max(__float_as_int(a), __float_as_int(b))); }
__device__ inline float imin_f(float a, float b) { return __int_as_float(min(__float_as_int(a), __float_as_int(b))); }

// AABB::intersect: returns the entry distance (>= 0) or -1 on a miss.
__device__ inline float slab(float lx, float ly, float lz, float hx, float hy, float hz, const f3& o, const f3& inv) {
    f3 t0 = (mk(lx, ly, lz) - o) * inv;
    f3 t1 = (mk(hx, hy, hz) - o) * inv;
    // fmin_fmax(a,b,c) = int max(int min(a,b), c); fmax_fmin(a,b,c) = int min(int max(a,b), c)
    float maxmin = imax_f(imin_f(t0.x, t1.x), imax_f(imin_f(t0.y, t1.y), fminf(t0.z, t1.z)));
    float minmax = imin_f(imax_f(t0.x, t1.x), imin_f(imax_f(t0.y, t1.y), fmaxf(t0.z, t1.z)));
    if (maxmin <= minmax) {
        if (minmax > 0) return fmaxf(0.f, maxmin);
    }
    return -1.f;
}

// One 64-byte node as two 256-bit read-only loads (sm_100 vector width): each load is one
// 32-byte sector, half the L1 sector lookups of four 16-byte loads.
__device__ __forceinline__ void ld_nc_v8(const void* p, float (&r)[8]) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "l"(p));
}

struct NodeRegs {
    float lo[8];  // L.lo.xyz L.hi.x L.hi.y L.hi.z R.lo.x R.lo.y
    float hi[8];  // R.lo.z R.hi.xyz left right - -
};

__device__ __forceinline__ void load_node(const TNode* __restrict__ nodes, int32_t ref, NodeRegs& nr) {
    const float* p = reinterpret_cast<const float*>(nodes + ref);
    ld_nc_v8(p, nr.lo);
    ld_nc_v8(p + 8, nr.hi);
}

// Claims new rays for the idle lanes of the warp.  Returns the claimed index for this lane
// (or -1) and clears `more` once the counter passed n.
__device__ inline int64_t claim(unsigned idle, unsigned long long* counter, int64_t n, bool& more) {
    const int lane = threadIdx.x & 31;
    const int cnt = __popc(idle);
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(counter, (unsigned long long)cnt);
    base = __shfl_sync(kFull, base, 0);
    if (base + (unsigned long long)cnt >= (unsigned long long)n) more = false;
    if (!((idle >> lane) & 1u)) return -1;
    int64_t my = (int64_t)base + __popc(idle & ((1u << lane) - 1u));
    return my < n ? my : -1;
}

// Segments: one traversal launch over the rays of several jobs, each with its own tree and
// outputs; a lane that claims global ray g finds its segment by binary search over the
// segment starts (staged in shared memory).
constexpr int kMaxSeg = 1024;

__device__ inline int find_seg(const int64_t* sbeg, int nseg, int64_t g) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (sbeg[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Per-lane visit counters of the instrumented traversal variants, summed per warp.
struct TraceStats {
    uint32_t nodes = 0, tris = 0;
};

template <bool kStats>
__device__ inline void flush_stats(const TraceStats& st, unsigned long long* stats) {
    if (!kStats) return;
    unsigned long long a = st.nodes, b = st.tris;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        a += __shfl_down_sync(kFull, a, o);
        b += __shfl_down_sync(kFull, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(stats, a);
        atomicAdd(stats + 1, b);
    }
}

// Blocks of a persistent traversal launch: every SM filled to the kernel's occupancy (or
// the context's configured blocks per SM).  The occupancy query costs a microsecond or two of
// the launch, so each host thread remembers its last answers.
template <typename K>
int grid_for(cav_ctx* ctx, K kernel, int block, size_t dyn_smem = 0) {
    if (dyn_smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_smem);
    int per_sm = ctx->trace_blocks_per_sm;
    if (per_sm <= 0) {
        struct Known {
            const void* kernel;
            size_t dyn;
            int block, device, per_sm;
        };
        thread_local Known known[16] = {};
        thread_local int next = 0;
        for (const Known& k : known)
            if (k.kernel == (const void*)kernel && k.dyn == dyn_smem && k.block == block && k.device == ctx->device)
                per_sm = k.per_sm;
        if (per_sm <= 0) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, dyn_smem);
            if (per_sm < 1) per_sm = 1;
            known[next] = Known{(const void*)kernel, dyn_smem, block, ctx->device, per_sm};
            next = (next + 1) & 15;
        }
    }
    return ctx->num_sms * per_sm;
}

// Rays a warp holds at least, when there are rays enough: fewer would leave most of each
// instruction idle.  With rays for every warp of the grid in one go, warp w takes rays [w cap,
// (w + 1) cap) and no others, and the work counter is not used (nor cleared by the launch).
__device__ __forceinline__ int warp_share(int64_t n, int min_cap, bool& once) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int cap = (int)min((int64_t)32, max((int64_t)min_cap, (n + warps - 1) / warps));
    once = n <= warps * cap;
    return cap;
}

// The launch's side of it: the blocks that n rays need, and whether the counter will be used.
inline int share_grid(int64_t n, int min_cap, int block, int grid, bool& counted) {
    const int64_t warps = (n + min_cap - 1) / min_cap, per_block = block / 32;
    grid = (int)(warps / per_block + 1 < grid ? (warps + per_block - 1) / per_block : grid);
    counted = n > (int64_t)grid * per_block * 32;
    return grid;
}

}  // namespace cav
