// The compressed 8-wide view of the binary tree, and persistent-warp traversal over it: the
// fast traversal mode (CAV_TRACE_FAST), and the screening pass that answers the rays of the exact
// mode that go this way (view_use).
//
// Layout (CNode, 96 bytes) after Ylitie, Karras and Laine, "Efficient Incoherent Ray
// Traversal on GPUs Through Compressed Wide BVHs" (HPG 2017): up to eight children per
// node with 8-bit quantised boxes, internal children and triangles each stored
// contiguously, and child slots chosen by direction so that a ray's octant alone gives a
// near-first visiting order.  The view is collapsed from the binary traversal tree
// (TNode) on the device, level by level: a wide node starts from a binary node's two
// children and repeatedly opens the internal child of largest surface area until it has
// eight children or only triangles remain.  Triangles are copied into wide-leaf order so
// that one node's triangles are adjacent in memory.
//
// Traversal keeps a node group (the remaining hit internal children of one node, as a
// bit mask over their visiting order) and a triangle group per ray; only node groups go
// on the stack, 8 bytes each.  A ray visits the same triangles' closest hit as the exact
// mode: the quantised boxes contain the exact ones with a margin, so the closest-hit
// distance is the same and only the choice between triangles at an equal distance may
// differ; the any-hit answer is the same.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <memory>
#include <mutex>

#include "trace_common.cuh"

namespace cav {

namespace {

constexpr int kBuildThreads = 128;
constexpr int kWideStack = 128;       // node groups; one per wide level at most
constexpr int kMaxWideLevels = 4096;  // a wide level consumes at least one binary level
// Relative growth of a box's exit distance, so that the rounding of the two-term plane
// distance never drops a box the ray touches.
constexpr float kGrow = 1.00000095f;  // 1 + 2^-20

// ------------------------------------------------------------------- building the view
// Coordinates up to this are screened (see the screening note below); larger or non-finite
// geometry always takes the binary traversal in the exact mode.
constexpr float kScreenCoord = 1e9f;

__device__ __forceinline__ float half_area(const float (&b)[6]) {
    const float ex = b[3] - b[0], ey = b[4] - b[1], ez = b[5] - b[2];
    return ex * ey + ey * ez + ez * ex;
}

__device__ void wide_init(const float* root_box, uint32_t tris, int32_t* task, WideCtr* ctr) {
    float mag = 0.f, b[6];
    bool ok = true;
    for (int k = 0; k < 6; ++k) {
        b[k] = root_box[k];
        mag = fmaxf(mag, fabsf(root_box[k]));
        ok = ok && fabsf(root_box[k]) <= kScreenCoord;
    }
    WideCtr c{};
    c.want = tris;
    c.margin = mag * 4.76837158e-7f + 1e-30f;  // 2^-21: 4 ulps of the largest coordinate
    c.unscreened = ok ? 0u : 1u;
    c.root_area = half_area(b);
    *ctr = c;
    task[0] = 0;  // the binary root becomes wide node 0
}

__global__ void k_wide_init(const float* root_box, uint32_t tris, int32_t* task, WideCtr* ctr) {
    if (threadIdx.x == 0) wide_init(root_box, tris, task, ctr);
}

// What came of a build of K views, in one word of pinned memory that the host looks at: kArrived,
// whether some view failed or cannot be screened, and in the upper half the most boxes per line.
// Also the sign that the views are complete.
constexpr unsigned long long kArrived = 1, kSomeFailed = 2, kSomeUnscreened = 4;

__global__ void k_wide_verdict(const WideCtr* __restrict__ ctr, int K, unsigned long long* host) {
    unsigned bits = (unsigned)kArrived, most = 0;
    for (int k = threadIdx.x; k < K; k += 32) {
        const WideCtr c = ctr[k];
        if (c.failed || c.tris != c.want) bits |= (unsigned)kSomeFailed;
        if (c.unscreened) bits |= (unsigned)kSomeUnscreened;
        const float lines = c.area / c.root_area;  // a NaN counts as infinitely many
        most = max(most, __float_as_uint(lines >= 0.f ? lines : INFINITY));
    }
    bits = __reduce_or_sync(kFull, bits);
    most = __reduce_max_sync(kFull, most);
    if (threadIdx.x == 0) {
        *(volatile unsigned long long*)host = ((unsigned long long)most << 32) | bits;
        __threadfence_system();
    }
}

// All blocks of the (co-resident, cooperatively launched) grid arrive; false once the build
// has failed in any of them (a wait that ran out among the reasons).
__device__ bool wide_barrier(WideCtr* ctr, uint32_t blocks, uint32_t target, uint64_t wait_ns) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        if (blocks > 1) {
            __threadfence();
            atomicAdd(&ctr->bar, 1u);
            uint64_t t0 = 0;
            volatile uint32_t* bar = &ctr->bar;
            while (*bar < target) {
                if (*(volatile uint32_t*)&ctr->failed) {
                    ok = 0;
                    break;
                }
                uint64_t t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                else if (t - t0 > wait_ns) {
                    atomicExch(&ctr->failed, 1u);
                    ok = 0;
                    break;
                }
            }
            __threadfence();
        }
        if (*(volatile uint32_t*)&ctr->failed) ok = 0;
    }
    __syncthreads();
    return ok != 0;
}

// One launch builds the whole view: eight lanes per wide node (lane k holds child k while the
// node is opened, then the child in slot k), the levels separated by a grid barrier (a block
// barrier for trees small enough for one block).  Latency bounds it: a level is a chain of six
// dependent node fetches and a barrier.  1M-triangle soup: 0.35 ms; 3.9 ms with a thread per
// node, its children in local memory, and two launches per level.
// `octet` of `octets` works on one tree with the threads of `blocks` blocks.
__device__ __forceinline__ void wide_levels(const TNode* __restrict__ tn, const TriRec* __restrict__ tris_in, int32_t* task,
                                            CNode* __restrict__ out, TriRec* __restrict__ tris_out,
                                            float4* __restrict__ lbox, WideCtr* ctr, uint32_t max_nodes, uint32_t max_tris,
                                            uint64_t wait_ns, uint32_t octet, uint32_t octets, uint32_t blocks) {
    const int lane = threadIdx.x & 31, k8 = lane & 7, lead = lane & 24;
    const float margin = *(volatile float*)&ctr->margin;
    uint32_t begin = 0, end = 1;
    float area = 0.f;  // of the own boxes that this lane places
    for (int level = 0; begin < end; ++level) {
        if (level >= kMaxWideLevels) {
            if (threadIdx.x == 0) atomicExch(&ctr->failed, 1u);
            return;
        }
        if (octet == 0 && k8 == 0) ctr->nodes[(level + 2) % 3] = 0;
        uint32_t* const alloc = &ctr->nodes[(level + 1) % 3];
        // the warp's four octets run together: w0 is the first one's node
        for (uint32_t w0 = begin + (octet & ~3u); w0 < end; w0 += octets) {
            const uint32_t w = w0 + (lane >> 3);
            const bool live = w < end;
            float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
            int32_t ref = -1, par = 0;  // the child, and the binary node that holds it
            int cnt = live ? 2 : 0;
            if (live && k8 < 2) {
                par = __ldcg(task + w);
                const TNode t = tn[par];
                if (k8 == 0) {
                    b[0] = t.a.x; b[1] = t.a.y; b[2] = t.a.z; b[3] = t.a.w; b[4] = t.b.x; b[5] = t.b.y;
                    ref = t.d.x;
                } else {
                    b[0] = t.b.z; b[1] = t.b.w; b[2] = t.c.x; b[3] = t.c.y; b[4] = t.c.z; b[5] = t.c.w;
                    ref = t.d.y;
                }
            }
            // open the internal child of largest area (the first on ties) until there are eight
#pragma unroll 1
            for (int step = 0; step < 6; ++step) {
                float pa = k8 < cnt && ref >= 0 ? half_area(b) : -1.f;
                if (!(pa > -1.f)) pa = -1.f;  // NaN areas are not opened
                int pick = k8;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    const float oa = __shfl_xor_sync(kFull, pa, o);
                    const int oi = __shfl_xor_sync(kFull, pick, o);
                    if (oa > pa || (oa == pa && oi < pick)) {
                        pa = oa;
                        pick = oi;
                    }
                }
                const bool open = pa > -1.f;
                const int32_t pref = __shfl_sync(kFull, ref, lead + pick);
                if (open && (k8 == pick || k8 == cnt)) {
                    const TNode t = tn[pref];
                    par = pref;
                    if (k8 == pick) {
                        b[0] = t.a.x; b[1] = t.a.y; b[2] = t.a.z; b[3] = t.a.w; b[4] = t.b.x; b[5] = t.b.y;
                        ref = t.d.x;
                    } else {
                        b[0] = t.b.z; b[1] = t.b.w; b[2] = t.c.x; b[3] = t.c.y; b[4] = t.c.z; b[5] = t.c.w;
                        ref = t.d.y;
                    }
                }
                if (open) ++cnt;
                if (!__any_sync(kFull, open)) break;
            }
            float lo[3] = {b[0], b[1], b[2]}, hi[3] = {b[3], b[4], b[5]};
#pragma unroll
            for (int o = 1; o < 8; o <<= 1)
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[a] = fminf(lo[a], __shfl_xor_sync(kFull, lo[a], o));
                    hi[a] = fmaxf(hi[a], __shfl_xor_sync(kFull, hi[a], o));
                }
            // slots: child i goes to the free slot whose octant diagonal best matches the
            // direction from the node's centre to the child's centre (greedy, largest first;
            // ties to the lower child, then the lower slot)
            const float cx = (b[0] + b[3]) - (lo[0] + hi[0]);
            const float cy = (b[1] + b[4]) - (lo[1] + hi[1]);
            const float cz = (b[2] + b[5]) - (lo[2] + hi[2]);
            int slot = -1;
            unsigned taken = 0;
#pragma unroll 1
            for (int round = 0; round < 8; ++round) {
                bool has = k8 < cnt && slot < 0;
                float bc = -FLT_MAX;
                int bs = -1, bi = k8;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const float c = ((s & 4) ? cx : -cx) + ((s & 2) ? cy : -cy) + ((s & 1) ? cz : -cz);
                    if (!((taken >> s) & 1u) && (bs < 0 || c > bc)) {
                        bc = c;
                        bs = s;
                    }
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    const bool oh = __shfl_xor_sync(kFull, has ? 1 : 0, o) != 0;
                    const float oc = __shfl_xor_sync(kFull, bc, o);
                    const int os = __shfl_xor_sync(kFull, bs, o), oi = __shfl_xor_sync(kFull, bi, o);
                    if (oh && (!has || oc > bc || (!(bc > oc) && oi < bi))) {
                        has = true;
                        bc = oc;
                        bs = os;
                        bi = oi;
                    }
                }
                if (has) {
                    if (bi == k8) slot = bs;
                    taken |= 1u << bs;
                }
                if (!__any_sync(kFull, has)) break;
            }
            // lane k takes the child in slot k
            int from = -1;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (__shfl_sync(kFull, slot, lead + i) == k8) from = i;
            const int srcl = lead + (from < 0 ? k8 : from);
#pragma unroll
            for (int a = 0; a < 6; ++a) b[a] = __shfl_sync(kFull, b[a], srcl);
            ref = __shfl_sync(kFull, ref, srcl);
            par = __shfl_sync(kFull, par, srcl);
            const bool full = from >= 0;
            const unsigned imask = (__ballot_sync(kFull, full && ref >= 0) >> lead) & 0xFFu;
            const unsigned tmask = (__ballot_sync(kFull, full && ref < 0) >> lead) & 0xFFu;
            // node and triangle ranges: one atomic each per warp
            const uint32_t ni = __popc(imask), nt = __popc(tmask);
            uint32_t si = k8 == 0 ? ni : 0u, stt = k8 == 0 ? nt : 0u;
#pragma unroll
            for (int o = 8; o < 32; o <<= 1) {
                const uint32_t a = __shfl_up_sync(kFull, si, o), c = __shfl_up_sync(kFull, stt, o);
                if (lane >= o) {
                    si += a;
                    stt += c;
                }
            }
            uint32_t cbase = 0, tbase = 0;
            if (lane == 24) {
                cbase = si ? atomicAdd(alloc, si) : 0u;
                tbase = stt ? atomicAdd(&ctr->tris, stt) : 0u;
            }
            cbase = end + __shfl_sync(kFull, cbase, 24) + __shfl_sync(kFull, si, lead) - ni;
            tbase = __shfl_sync(kFull, tbase, 24) + __shfl_sync(kFull, stt, lead) - nt;
            if (!live) continue;
            if ((uint64_t)cbase + ni > max_nodes || (uint64_t)tbase + nt > max_tris) {  // not a tree
                if (k8 == 0) atomicExch(&ctr->failed, 1u);
                continue;
            }
            // The node's grid: a power-of-two step per axis with 253 steps covering the box grown
            // by the margin, one spare step below it (the origin) and one above.  Every child plane
            // is then rounded outward and moved out by one more step, which absorbs the half-step
            // rounding of the traversal's folded plane distance (node_hits).
            unsigned char* const bytes = reinterpret_cast<unsigned char*>(out + w);
            uint32_t ebits = 0;
            float p[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float range = (hi[a] + margin) - (lo[a] - margin);
                int ex = 0;
                frexpf(range * (1.f / 253.f) * 1.0000010f, &ex);  // 2^ex > range / 253
                int eb = ex + 127;
                eb = eb < 1 ? 1 : (eb > 254 ? 254 : eb);
                ebits |= (uint32_t)eb << (8 * a);
                const double step_inv = ldexp(1.0, 127 - eb);
                p[a] = (lo[a] - margin) - __uint_as_float((uint32_t)eb << 23);
                double qlo = floor(((double)b[a] - (double)margin - (double)p[a]) * step_inv) - 1.0;
                double qhi = ceil(((double)b[3 + a] + (double)margin - (double)p[a]) * step_inv) + 1.0;
                qlo = qlo < 0.0 ? 0.0 : (qlo > 255.0 ? 255.0 : qlo);
                qhi = qhi < 0.0 ? 0.0 : (qhi > 255.0 ? 255.0 : qhi);
                bytes[32 + 8 * a + k8] = full ? (unsigned char)qlo : 0;
                bytes[56 + 8 * a + k8] = full ? (unsigned char)qhi : 0;
            }
            if (k8 == 0) {
                uint4* o = reinterpret_cast<uint4*>(bytes);
                o[0] = make_uint4(__float_as_uint(p[0]), __float_as_uint(p[1]), __float_as_uint(p[2]), ebits | (imask << 24));
                o[1] = make_uint4(cbase, tbase, tmask, 0u);
            }
            if (full && ref >= 0) {
                task[cbase + __popc(imask & ((1u << k8) - 1u))] = ref;
            } else if (full) {
                const uint32_t at = tbase + __popc(tmask & ((1u << k8) - 1u));
                const TriRec r = tris_in[~ref];
                tris_out[at] = r;
                lbox[2 * (size_t)at] = make_float4(b[0], b[1], b[2], b[3]);
                lbox[2 * (size_t)at + 1] = make_float4(b[4], b[5], __int_as_float(par), __int_as_float(ref));
                area += half_area(b);
                const float m = fmaxf(fmaxf(fmaxf(fabsf(r.e1.x), fabsf(r.e1.y)), fabsf(r.e1.z)),
                                      fmaxf(fmaxf(fabsf(r.e2.x), fabsf(r.e2.y)), fabsf(r.e2.z)));
                const float sum = r.v0.x + r.v0.y + r.v0.z + r.e1.x + r.e1.y + r.e1.z + r.e2.x + r.e2.y + r.e2.z;
                if (!(m <= 4.f * kScreenCoord) || !(fabsf(sum) <= 64.f * kScreenCoord)) ctr->unscreened = 1u;
            }
        }
        if (!wide_barrier(ctr, blocks, (uint32_t)(level + 1) * blocks, wait_ns)) return;
        begin = end;
        end = begin + __ldcg(alloc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) area += __shfl_xor_sync(kFull, area, o);
    if (lane == 0 && area > 0.f) atomicAdd(&ctr->area, area);
}

__global__ void __launch_bounds__(kBuildThreads)
    k_wide_build(const TNode* __restrict__ tn, const TriRec* __restrict__ tris_in, int32_t* task, CNode* __restrict__ out,
                 TriRec* __restrict__ tris_out, float4* __restrict__ lbox, WideCtr* ctr, uint32_t max_nodes,
                 uint32_t max_tris, uint64_t wait_ns) {
    wide_levels(tn, tris_in, task, out, tris_out, lbox, ctr, max_nodes, max_tris, wait_ns,
                (blockIdx.x * blockDim.x + threadIdx.x) >> 3, (gridDim.x * blockDim.x) >> 3, gridDim.x);
}

// The views of many small trees (a batched build's), a cluster of four blocks each (co-resident, as
// the levels' barriers need): a tree's levels are a chain of fetches, so one tree keeps the chip
// idle, and a launch, a copy back and a wait for each cost more than its view.  48 trees of 1,000 to
// 30,000 triangles: 31 views at 65 us each, one by one; the queries of 2,048 closest hits each, the
// views among them, 3.25 ms with a block for each tree, 2.87, 2.67 and 2.62 with two, four and
// eight blocks.
struct WideTree {
    const TNode* tn;
    const TriRec* tris_in;
    const float* root_box;
    int32_t* task;
    CNode* out;
    TriRec* tris_out;
    float4* lbox;
    uint32_t tris, nodes;
};
constexpr int kGroupThreads = 512;
constexpr int kGroupBlocks = 4;
constexpr int64_t kGroupTris = 1 << 16;             // larger trees take the grid
// And so does a tree of more than this many triangles for each of the group: few clusters leave most
// of the chip idle (views and queries of 2,048 rays: two trees of 5,000 triangles 0.23 ms together and
// 0.26 one by one, of 20,000 0.48 and 0.42, of 60,000 1.06 and 0.80; of 60,000 four 1.61 and 1.57,
// eight 2.77 and 3.18, sixteen 5.1 and 6.4).
constexpr int64_t kGroupShare = 1 << 13;
constexpr size_t kGroupBytes = (size_t)256 << 20;  // of the views together, at most

__global__ void __cluster_dims__(kGroupBlocks) __launch_bounds__(kGroupThreads)
    k_wide_build_group(const WideTree* __restrict__ trees, WideCtr* ctrs, uint64_t wait_ns) {
    const uint32_t rank = blockIdx.x % kGroupBlocks;
    const WideTree t = trees[blockIdx.x / kGroupBlocks];
    WideCtr* ctr = ctrs + blockIdx.x / kGroupBlocks;
    if (rank == 0 && threadIdx.x == 0) {
        wide_init(t.root_box, t.tris, t.task, ctr);
        __threadfence();
    }
    cooperative_groups::this_cluster().sync();
    wide_levels(t.tn, t.tris_in, t.task, t.out, t.tris_out, t.lbox, ctr, t.nodes, t.tris, wait_ns,
                (rank * kGroupThreads + threadIdx.x) >> 3, kGroupBlocks * kGroupThreads >> 3, kGroupBlocks);
}

// ----------------------------------------------------------------------- traversal
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Byte k of w as the float 2^23 + byte (bit pattern 0x4B0000bb).
__device__ __forceinline__ float biased_byte(uint32_t w, uint32_t k) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | k));
}

// Two plane distances in one instruction: {b0, b1} * {a, a} + {c, c}.
__device__ __forceinline__ float2 fma2(float b0, float b1, float2 a, float2 c) {
    unsigned long long r, q, x, y;
    asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(b0), "f"(b1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(c.x), "f"(c.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(q), "l"(x), "l"(y));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
    return d;
}

struct WideRay {
    f3 o, inv;
    uint32_t octinv;  // the visiting-order flip, 7 - direction octant
};

// Hit mask of one node: bits 24-31 the internal children in visiting order (slot ^ octinv),
// bits 0-7 the triangles by slot.  `lim` bounds the entry distance (closest hit so far, ray
// tmax, shadow limit).  A plane's distance is fma(2^23 + q, s * inv, (p - o) * inv - 2^23 * s
// * inv): one fma per plane on the byte's biased float, two children per packed instruction;
// the folded constant rounds by at most half a grid step in distance, inside the spare step
// every quantised plane carries.  ALU operations bound this function: a child costs six byte
// extractions, four three-input min/max and one predicated or; the children's order is applied
// to the eight-bit mask, not child by child.
__device__ __forceinline__ uint32_t node_hits(const CNode* __restrict__ cn, uint32_t idx, const WideRay& R, float lim,
                                              uint32_t& child_base, uint32_t& tri_base, uint32_t& masks) {
    uint32_t h[8], q[8];
    const char* at = reinterpret_cast<const char*>(cn + idx);
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]), "=r"(h[4]), "=r"(h[5]), "=r"(h[6]), "=r"(h[7])
        : "l"(at));
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7])
        : "l"(at + 32));
    const uint4 r = __ldg(reinterpret_cast<const uint4*>(at + 64));
    child_base = h[4];
    tri_base = h[5];
    const uint32_t imask = h[3] >> 24, tmask = h[6];
    masks = imask | (tmask << 8);
    const float ax = __uint_as_float((h[3] & 0xFFu) << 23) * R.inv.x;
    const float ay = __uint_as_float(((h[3] >> 8) & 0xFFu) << 23) * R.inv.y;
    const float az = __uint_as_float(((h[3] >> 16) & 0xFFu) << 23) * R.inv.z;
    const float bx = (__uint_as_float(h[0]) - R.o.x) * R.inv.x - 8388608.f * ax;
    const float by = (__uint_as_float(h[1]) - R.o.y) * R.inv.y - 8388608.f * ay;
    const float bz = (__uint_as_float(h[2]) - R.o.z) * R.inv.z - 8388608.f * az;
    const float2 ax2 = make_float2(ax, ax), ay2 = make_float2(ay, ay), az2 = make_float2(az, az);
    const float2 bx2 = make_float2(bx, bx), by2 = make_float2(by, by), bz2 = make_float2(bz, bz);
    // near / far planes by direction sign (octinv bit 2: x not negative, and so on)
    const bool nx = !(R.octinv & 4u), ny = !(R.octinv & 2u), nz = !(R.octinv & 1u);
    uint32_t hm = 0;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        if (w && ((imask | tmask) & 0xF0u) == 0u) break;  // slots 4-7 empty
        const uint32_t rx = w ? r.y : r.x, rz = w ? r.w : r.z;
        const uint32_t nxw = nx ? q[6 + w] : q[w], fxw = nx ? q[w] : q[6 + w];
        const uint32_t nyw = ny ? rx : q[2 + w], fyw = ny ? q[2 + w] : rx;
        const uint32_t nzw = nz ? rz : q[4 + w], fzw = nz ? q[4 + w] : rz;
#pragma unroll
        for (int k = 0; k < 4; k += 2) {
            const float2 tnx = fma2(biased_byte(nxw, k), biased_byte(nxw, k + 1), ax2, bx2);
            const float2 tny = fma2(biased_byte(nyw, k), biased_byte(nyw, k + 1), ay2, by2);
            const float2 tnz = fma2(biased_byte(nzw, k), biased_byte(nzw, k + 1), az2, bz2);
            const float2 tfx = fma2(biased_byte(fxw, k), biased_byte(fxw, k + 1), ax2, bx2);
            const float2 tfy = fma2(biased_byte(fyw, k), biased_byte(fyw, k + 1), ay2, by2);
            const float2 tfz = fma2(biased_byte(fzw, k), biased_byte(fzw, k + 1), az2, bz2);
            const float t0 = max3f(tnx.x, tny.x, fmaxf(tnz.x, 0.f)), t1 = max3f(tnx.y, tny.y, fmaxf(tnz.y, 0.f));
            if (t0 <= fminf(min3f(tfx.x, tfy.x, tfz.x) * kGrow, lim)) hm |= 1u << (4 * w + k);
            if (t1 <= fminf(min3f(tfx.y, tfy.y, tfz.y) * kGrow, lim)) hm |= 2u << (4 * w + k);
        }
    }
    uint32_t x = hm & imask;  // slot s to bit s ^ octinv
    if (!nz) x = ((x << 1) & 0xAAu) | ((x >> 1) & 0x55u);
    if (!ny) x = ((x << 2) & 0xCCu) | ((x >> 2) & 0x33u);
    if (!nx) x = ((x << 4) & 0xF0u) | (x >> 4);
    return (x << 24) | (hm & tmask);
}

// The first kSmemN node groups of a lane's stack in shared memory, [entry][thread] (a warp's
// push or pop is two conflict-free wavefronts whatever the lanes' depths), the rest in local
// memory; kSmemN == 0 keeps all of it in local memory.
template <int kSmemN>
__device__ __forceinline__ void wstack_put(uint2* sst, uint2* lst, int i, uint2 v) {
    if (kSmemN > 0 && i < kSmemN) sst[i * (int)blockDim.x] = v;
    else lst[i - kSmemN] = v;
}

template <int kSmemN>
__device__ __forceinline__ uint2 wstack_get(const uint2* sst, const uint2* lst, int i) {
    return kSmemN > 0 && i < kSmemN ? sst[i * (int)blockDim.x] : lst[i - kSmemN];
}

// ---- screening (kExact).  The exact mode's answer is the one the binary traversal of
// trace.cu gives (the reference's visiting order and pruning).  The wide traversal finds it
// faster, and proves it ray by ray:
//   * The binary slab test of a box that contains another passes whenever the inner box's
//     passes, with an entry distance no larger: subtraction and multiplication round
//     monotonically, and the boxes of the tree are exact unions.  So the slab test of a
//     triangle's own box, entry `ml`, bounds those of all its ancestors; and a triangle whose
//     own box fails is never tested by the binary traversal (leaves are tested as boxes).
//   * Any hit: the binary traversal prunes nothing, so it finds a hit exactly when some hit
//     triangle's own box passes.  The wide traversal prunes nothing either, boxes beyond the limit
//     among them: of a triangle that the ray's line lies in, the tested distance is rounding noise and
//     can be far below its box's entry (of 1M shadow rays laid in such planes 200 to 800 differed when
//     boxes beyond the limit were left out).  The rays that find no hit pay for it: 4M shadow rays
//     over the 1M-triangle soup 8.9 ms (5.9 with the pruning), 26.3 in the binary tree.
//   * Closest hit: the wide traversal tests every triangle whose box it enters up to the ray's
//     tmax, whatever it has hit so far, and keeps the two smallest distances.  If only one triangle
//     has the smallest, its own box passes and its `ml` is below the second, the binary traversal
//     cannot have pruned the winner at any of its ancestors (a hit that prunes one has a distance of
//     `ml` or less), and no triangle replaces it: that triangle is the answer.
//   * Of two triangles with the smallest distance (a ray through a shared edge) the same holds
//     for the one that the binary traversal tests first, the one on the side that it enters
//     first at their lowest common ancestor.  (Handed to the binary steps instead, such ties, 1 ray
//     in 10,000 of a path tracer's bounces, took up to 941 of them at the end of a launch.)
// The winner's own box is tested once per ray, when the ray ends; if it fails, the wide search
// runs again and leaves such triangles out as it goes (kModeCareful).  Every other ray (more
// ties, a second hit as close as the box entry, a ray or scene out of range) takes the binary
// steps themselves, in the same kernel (kModeBinary).
// Leaving out boxes that a ray enters beyond its closest hit (with some slack) would be much
// less work where boxes overlap densely, but no proof: a triangle that holds the ray's line in its
// plane can have any tested distance, and the binary traversal may come to it before the hit (15
// to 60 of 1M closest-hit rays laid in triangles' planes differed).  So the closest hits of many
// rays on such trees are the binary traversal's own (kSparse below).
constexpr float kSlack = 1.0009765625f;  // 1 + 2^-10, far above the rounding of an entry distance
constexpr float kScreenDir = 1e6f, kScreenDirMin = 1e-6f;

__device__ inline bool screenable(const f3& o, const f3& d) {
    const float mo = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z));
    const float md = fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    // NaN components fail the sums (fmaxf drops them)
    return mo <= kScreenCoord && md <= kScreenDir && md >= kScreenDirMin && fabsf(o.x + o.y + o.z) <= 4.f * kScreenCoord &&
           fabsf(d.x + d.y + d.z) <= 4.f * kScreenDir;
}

// ---- work sharing.  A launch ends when its slowest ray does, and the slowest of a batch
// visits hundreds of times the average (a ray nearly in a plane of a dense scene).  Once the
// queue is empty, an idle lane takes the oldest node group of a busy lane of its warp and
// searches it for the same ray.  The first lane of a shared ray lends its slot in this
// per-warp record; lanes that run out merge what they found, and the last one to finish
// writes the ray's result.  The largest part left (the bottom of the stack) is the better one
// to give: taking the nearest group instead made 65,536 closest-hit rays 1.85 against 1.44 ms.
// Waiting for a hit or a number of steps before sharing a ray measured slower too (2.7 and 2.2
// against 1.6 ms).  1M-triangle soup, fast mode, with and without sharing: 16,384 shadow rays
// 0.12 against 1.4 ms, 65,536 closest-hit rays 1.5 against 6.1, 4M 35.7 against 43.8.  (Closest-hit
// times of the kernel's variants here and below are of searches that end at the hit found, as the
// fast mode's do.)
struct ShareRec {
    int32_t bound[32];  // closest, fast mode: the smallest distance any lane of the ray has seen (float bits)
    float best[32], second[32];  // the two smallest distances of the merged lanes (second negative: a lane failed)
    float u[32], v[32];
    int32_t slot[32];     // closest: the triangle at `best`; any: bits 1 hit, 4 failed
    int32_t slot2[32];    // another triangle at `best`
    int32_t pending[32];  // lanes still searching
    int32_t donor[32];    // one hand-over's donors, in lane order
};
constexpr int kShareEvery = 2;  // iterations between two hand-overs

__device__ __forceinline__ int tri_id(const TriRec* __restrict__ tris, int32_t slot) {
    return __float_as_int(__ldg(&tris[slot].v0.w));
}

// The binary traversal's reciprocal direction: R.inv but for the components that were replaced.
__device__ __forceinline__ f3 own_inv(const WideRay& R, const f3& d) {
    if (fmaxf(fmaxf(fabsf(R.inv.x), fabsf(R.inv.y)), fabsf(R.inv.z)) < 7.37e19f) return R.inv;
    return mk(1.f / d.x, 1.f / d.y, 1.f / d.z);
}

// The binary slab test of triangle `slot`'s own box (the entry distance, or -1).
__device__ __forceinline__ float own_box(const TraceSeg& S, uint32_t slot, const WideRay& R, const f3& d) {
    const float4* lb = S.lbox + 2 * (size_t)slot;
    const float4 a = __ldg(lb), b = __ldg(lb + 1);
    return slab(a.x, a.y, a.z, a.w, b.x, b.y, R.o, own_inv(R, d));
}

// Which of two triangles the binary traversal tests first, both reached: the one on the side
// that it enters first at their lowest common ancestor.  1: `a`, 0: `b`, -1: the climb does
// not meet (not a tree).
__device__ __forceinline__ int tested_first(const TNode* __restrict__ nodes, const float4* __restrict__ lbox, int32_t a,
                                         int32_t b, f3 o, f3 inv) {
    const float4 la = __ldg(lbox + 2 * (size_t)a + 1), lb = __ldg(lbox + 2 * (size_t)b + 1);
    int32_t pa = __float_as_int(la.z), pb = __float_as_int(lb.z);  // nodes, and the child each climb came from
    int32_t ca = __float_as_int(la.w), cb = __float_as_int(lb.w);
    int da = 0, db = 0;
    constexpr int kMaxClimb = 4096;
    for (int32_t x = pa; x != 0 && da < kMaxClimb; x = __ldg(&nodes[x].d.z)) ++da;
    for (int32_t x = pb; x != 0 && db < kMaxClimb; x = __ldg(&nodes[x].d.z)) ++db;
    if (da >= kMaxClimb || db >= kMaxClimb) return -1;
    for (; da > db; --da) {
        ca = pa;
        pa = __ldg(&nodes[pa].d.z);
    }
    for (; db > da; --db) {
        cb = pb;
        pb = __ldg(&nodes[pb].d.z);
    }
    for (; pa != pb && da > 0; --da) {
        ca = pa;
        pa = __ldg(&nodes[pa].d.z);
        cb = pb;
        pb = __ldg(&nodes[pb].d.z);
    }
    if (pa != pb) return -1;
    NodeRegs nr;
    load_node(nodes, pa, nr);
    const float ml = slab(nr.lo[0], nr.lo[1], nr.lo[2], nr.lo[3], nr.lo[4], nr.lo[5], o, inv);
    const float mr = slab(nr.lo[6], nr.lo[7], nr.hi[0], nr.hi[1], nr.hi[2], nr.hi[3], o, inv);
    const int32_t first = ml > mr ? __float_as_int(nr.hi[5]) : __float_as_int(nr.hi[4]);
    return ca == first ? 1 : (cb == first ? 0 : -1);
}

enum { kModeWide = 0, kModeCareful = 1, kModeBinary = 2 };

// Idle lane iterations, per unit of the context's queue chunk (default 4), that pay for settling
// a warp's ended rays and claiming new ones.
constexpr int kSettleCost = 8;

// kSeg: one launch over several jobs' rays (segs[k] = one tree and its outputs, ray indices
// numbered across the launch); otherwise `one` describes the tree.
// A warp holds at most `cap` rays of its own at a time: 32, less when there are fewer rays
// than lanes (they are spread over the warps, and the other lanes help).
// Registers: 72 for the exact closest hit (the two smallest distances and the search mode ride
// along), 64 for the others; in the former 180,000 rays of the 1M soup took 11.4 ms at 72, 11.8 at
// 64 and 11.9 at 80 (2M camera rays over spheres 1.68, 1.64 and 1.62), 4M soup rays of the fast
// mode's closest hit 33.7, 35.4 and 38.2 ms at 64, 72 and 80.
template <bool kAny, bool kStats, bool kSeg, bool kExact, int kSmemN = 0>
__global__ void __maxnreg__(kExact && !kAny ? 72 : 64)
    k_trace_wide(TraceSeg one, const TraceSeg* __restrict__ segs, int nseg, int64_t n, unsigned long long* counter,
                 int refill, int min_cap, uint32_t max_steps, int* flag, unsigned long long* stats) {
    __shared__ int64_t sbeg[kSeg ? kMaxSeg : 1];
    __shared__ ShareRec shares[8];
    if (kSeg) {
        for (int i = threadIdx.x; i < nseg; i += blockDim.x) sbeg[i] = segs[i].begin;
        __syncthreads();
    }
    if (!kSeg && one.n_dev) n = *one.n_dev;
    if (kExact && one.gate && !view_serves(one.gate, kAny, n)) n = 0;
    bool once;
    const int cap = warp_share(n, min_cap, once);
    ShareRec& sh = shares[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const CNode* __restrict__ cn = one.cnodes;
    const TriRec* __restrict__ tris = one.ctris;
    int seg = 0;
    TraceStats st;
    extern __shared__ uint2 wsstack[];
    uint2* const sst = wsstack + threadIdx.x;
    uint2 lst[kWideStack - kSmemN];
    bool more = true;
    int64_t ray = -1;
    WideRay R{};
    f3 d = mk(0, 0, 0);
    // closest: ray tmax; any: the limit (FLT_MAX without one: a hit needs t < lim only with one)
    float tmax = 0.f;
    float best = 0.f, second = 0.f, bu = 0.f, bv = 0.f;
    int32_t slot = -1, src = -1, dst = -1;  // closest: the hit triangle; any: the bits of ShareRec::slot
    int32_t slot2 = -1;                     // another triangle at `best`; -2: there are several
    bool use_limit = false;
    uint2 grp = make_uint2(0, 0), tgrp = make_uint2(0, 0);
    int top = -1, bot = 0;  // stack entries bot..top
    // The record that the lane's ray uses when it is shared (its first lane's, which no other
    // ray can need); ~owner while the ray has one lane only.
    int owner = ~lane;
    int mode = kModeWide;
    bool finished = false;  // this lane's search has ended, its ray is not yet written
    uint32_t steps = 0;
    int turn = 0, waste = 0;  // waste: idle lanes, summed over iterations
    for (;;) {
        unsigned idle = __ballot_sync(kFull, ray < 0 || finished);
        // Rays that ended are proven and written, and their lanes take new rays, once the lanes
        // have waited long enough together to pay for the instructions (at once when the queue
        // is empty): after a few iterations where rays are short, with few lanes where they are
        // long.  Against a fixed four lanes: 1M rays of the 36-triangle
        // room 0.207 -> 0.189 ms, 1M camera rays over 20,498 triangles 0.157 -> 0.136, 4M soup
        // rays 38.1 -> 37.0.
        waste += __popc(idle);
        if (!more || idle == kFull || waste >= kSettleCost * refill) {
            waste = 0;
            if (!more) {  // lanes of shared rays that ran out merge; the last of a ray goes on to write it
                const bool out = finished && owner >= 0;
                if (__any_sync(kFull, out)) {
                    if (kAny) {
                        if (out && slot != 0) atomicOr(&sh.slot[owner], slot);
                    } else {
                        // most lanes found nothing and have nothing to add; the others one by one
                        unsigned fin = __ballot_sync(kFull, out && (slot >= 0 || second < FLT_MAX));
                        while (fin) {
                            const int f = __ffs(fin) - 1;
                            fin &= fin - 1u;
                            if (lane == f) {
                                const float rb = sh.best[owner];
                                const int32_t rs = sh.slot[owner];
                                second = fminf(second, sh.second[owner]);
                                bool keep = slot >= 0 && (rs < 0 || best < rb);
                                if (!kExact && slot >= 0 && rs >= 0 && best == rb) keep = tri_id(tris, slot) < tri_id(tris, rs);
                                if (keep) {
                                    if (kExact && rs >= 0) second = fminf(second, rb);
                                    sh.best[owner] = best;
                                    sh.slot[owner] = slot;
                                    sh.u[owner] = bu;
                                    sh.v[owner] = bv;
                                    sh.slot2[owner] = slot2;
                                } else if (kExact && slot >= 0 && best == rb) {
                                    sh.slot2[owner] = slot2 == -1 && sh.slot2[owner] == -1 ? slot : -2;
                                } else if (kExact && slot >= 0) {
                                    second = fminf(second, best);
                                }
                                sh.second[owner] = second;
                            }
                            __syncwarp();
                        }
                    }
                    __syncwarp();
                    if (out) {
                        if (atomicSub(&sh.pending[owner], 1) > 1) {
                            ray = -1;
                            finished = false;
                        } else {
                            slot = sh.slot[owner];
                            if (!kAny) {
                                best = sh.best[owner];
                                second = sh.second[owner];
                                slot2 = sh.slot2[owner];
                                bu = sh.u[owner];
                                bv = sh.v[owner];
                            }
                        }
                        owner = ~owner;
                    }
                }
            }
            if (finished && kExact) {  // proven, or searched again
                int next = -1;
                if (mode <= kModeCareful) {
                    if (kAny) {
                        if ((slot & 4) && !(slot & 1)) next = kModeBinary;
                    } else if (second < 0.f) {
                        next = kModeBinary;
                    } else if (slot >= 0) {
                        const float ml = own_box(one, slot, R, d);
                        if (!(ml >= 0.f)) {
                            next = kModeCareful;
                        } else if (ml > tmax) {
                            next = kModeBinary;
                        } else if (slot2 == -1) {
                            if (!(ml < second)) next = kModeBinary;
                        } else {  // a tie: of two, the first one tested keeps it
                            const float m2 = slot2 >= 0 ? own_box(one, slot2, R, d) : -1.f;
                            int first = slot2 >= 0 ? 1 : -1;
                            if (m2 >= 0.f) first = tested_first(one.nodes, one.lbox, slot, slot2, R.o, own_inv(R, d));
                            if (first == 0 && m2 < second && !(m2 > tmax)) {
                                tgrp = make_uint2((uint32_t)slot2, 0x101u);  // test it once more, alone
                                grp = make_uint2(0u, 0u);
                                best = second = FLT_MAX;
                                slot = slot2 = -1;
                                top = -1;
                                bot = 0;
                                finished = false;
                            } else if (first != 1 || !(ml < second)) {
                                next = kModeBinary;
                            }
                        }
                    }
                }
                if (next >= 0) {
                    best = second = FLT_MAX;
                    bu = bv = 0.f;
                    slot = kAny ? 0 : -1;
                    slot2 = -1;
                    grp = make_uint2(0u, next == kModeCareful ? (1u << (24u + R.octinv)) | 1u : 0u);
                    top = -1;
                    bot = 0;
                    steps = 0;
                    mode = next;
                    finished = false;
                }
            }
            if (finished) {
                const TraceSeg& S = kSeg ? segs[seg] : one;
                if (kAny) {
                    S.occ[ray] = (slot & 1) ? 1 : ((slot & 4) ? 2 : 0);
                } else {
                    const bool wide = mode <= kModeCareful;
                    const bool bad = wide ? second < 0.f : slot == -2;
                    const bool hit = !bad && slot >= 0;
                    S.prim[ray] = hit ? (wide ? tri_id(tris, slot) : slot) : (bad ? -2 : -1);
                    if (S.t) S.t[ray] = hit ? best : __int_as_float(0x7f800000);
                    if (S.uv) reinterpret_cast<float2*>(S.uv)[ray] = hit ? make_float2(bu, bv) : make_float2(0.f, 0.f);
                }
                ray = -1;
                finished = false;
            }
            idle = __ballot_sync(kFull, ray < 0);
            if (more) {
                const int busy = 32 - __popc(idle);
                const int want = min(cap - busy, 32 - busy);
                if (want > 0) {
                    const int rank = __popc(idle & ((1u << lane) - 1u));
                    const bool mine = ((idle >> lane) & 1u) && rank < want;
                    int64_t r;
                    if (once) {
                        r = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * cap + rank;
                        if (!mine || r >= n) r = -1;
                        more = false;
                    } else {
                        r = claim(__ballot_sync(kFull, mine), counter, n, more);
                    }
                    if (r >= 0) {
                        const TraceSeg* S = &one;
                        if (kSeg) {
                            seg = find_seg(sbeg, nseg, r);
                            S = segs + seg;
                            cn = S->cnodes;
                            tris = S->ctris;
                            r -= S->begin;
                        }
                        const float4* rp = reinterpret_cast<const float4*>(S->rays + r);
                        const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
                        R.o = mk(r0.x, r0.y, r0.z);
                        d = mk(r1.x, r1.y, r1.z);
                        tmax = r1.w;
                        // Box tests use a direction whose zero components are replaced by +-2^-66: a
                        // finite reciprocal keeps the folded plane distances finite (an infinite one
                        // turns them into NaN, which the min / max drop, so the axis would stop
                        // bounding the ray and a ray parallel to it would visit a whole slab of the
                        // tree).  The triangle test uses the ray's own direction.
                        const f3 db = mk(fabsf(d.x) < 1.3552527e-20f ? copysignf(1.3552527e-20f, d.x) : d.x,
                                         fabsf(d.y) < 1.3552527e-20f ? copysignf(1.3552527e-20f, d.y) : d.y,
                                         fabsf(d.z) < 1.3552527e-20f ? copysignf(1.3552527e-20f, d.z) : d.z);
                        R.inv = mk(1.f / db.x, 1.f / db.y, 1.f / db.z);
                        R.octinv = 7u - ((db.x < 0.f ? 4u : 0u) | (db.y < 0.f ? 2u : 0u) | (db.z < 0.f ? 1u : 0u));
                        // the root as the one internal child of a virtual parent: slot 0, imask 1
                        grp = make_uint2(0u, (1u << (24u + R.octinv)) | 1u);
                        tgrp = make_uint2(0u, 0u);
                        best = second = FLT_MAX;
                        bu = bv = 0.f;
                        slot = kAny ? 0 : -1;
                        slot2 = -1;
                        top = -1;
                        bot = 0;
                        owner = ~lane;
                        mode = kModeWide;
                        steps = 0;
                        if (kAny) {
                            use_limit = S->limit != nullptr;
                            tmax = use_limit ? __ldg(S->limit + r) : FLT_MAX;
                            src = dst = -1;
                            if (S->excl) {
                                const int2 e = __ldg(reinterpret_cast<const int2*>(S->excl) + r);
                                src = e.x;
                                dst = e.y;
                            }
                        }
                        ray = r;
                        if (kExact && !screenable(R.o, d)) {
                            mode = kModeBinary;
                            grp.x = 0u;
                        }
                    }
                }
            } else {
                if (idle == kFull) break;
                // The step limit counts one lane's visits, so rays are shared only under the default
                if (idle != 0 && max_steps >= kMaxSteps && (++turn & (kShareEvery - 1)) == 0) {
                    const bool on_stack = top >= bot;
                    const bool can = ray >= 0 && mode <= kModeCareful && (on_stack || __popc(grp.y >> 24) >= 2);
                    const unsigned donors = __ballot_sync(kFull, can);
                    const int pairs = min(__popc(donors), __popc(idle));
                    if (pairs > 0) {
                        const unsigned lt = (1u << lane) - 1u;
                        const bool give = can && __popc(donors & lt) < pairs;
                        const bool take = ray < 0 && __popc(idle & lt) < pairs;
                        uint2 g = make_uint2(0, 0);
                        if (give) {
                            if (on_stack) {
                                g = wstack_get<kSmemN>(sst, lst, bot++);  // the oldest: the largest part left
                                if (bot > top) {
                                    bot = 0;
                                    top = -1;
                                }
                            } else {  // all but the next child of the current group
                                const uint32_t keep = 0x80000000u >> __clz(grp.y & 0xFF000000u);
                                g = make_uint2(grp.x, grp.y & ~keep);
                                grp.y &= keep | 0x00FFFFFFu;
                            }
                            if (owner < 0) {
                                owner = ~owner;
                                sh.bound[owner] = __float_as_int(best);
                                sh.best[owner] = FLT_MAX;
                                sh.second[owner] = FLT_MAX;
                                sh.slot2[owner] = -1;
                                sh.slot[owner] = kAny ? 0 : -1;
                                sh.pending[owner] = 1;
                            }
                            atomicAdd(&sh.pending[owner], 1);
                            sh.donor[__popc(donors & lt)] = lane;
                        }
                        __syncwarp();
                        // the k-th idle lane takes from the k-th donor
                        const int from = take ? sh.donor[__popc(idle & lt)] : lane;
                        const float ox = __shfl_sync(kFull, R.o.x, from), oy = __shfl_sync(kFull, R.o.y, from),
                                    oz = __shfl_sync(kFull, R.o.z, from);
                        const float ix = __shfl_sync(kFull, R.inv.x, from), iy = __shfl_sync(kFull, R.inv.y, from),
                                    iz = __shfl_sync(kFull, R.inv.z, from);
                        const float dx = __shfl_sync(kFull, d.x, from), dy = __shfl_sync(kFull, d.y, from),
                                    dz = __shfl_sync(kFull, d.z, from);
                        const uint32_t oct = __shfl_sync(kFull, R.octinv, from);
                        const float tm = __shfl_sync(kFull, tmax, from), bb = __shfl_sync(kFull, best, from);
                        const int64_t rr = __shfl_sync(kFull, ray, from);
                        const int ow = __shfl_sync(kFull, owner, from), sg = __shfl_sync(kFull, seg, from);
                        const int es = __shfl_sync(kFull, src, from), ed = __shfl_sync(kFull, dst, from);
                        const uint32_t gx = __shfl_sync(kFull, g.x, from), gy = __shfl_sync(kFull, g.y, from);
                        const int how = __shfl_sync(kFull, mode | (use_limit ? 16 : 0), from);
                        if (take) {
                            R.o = mk(ox, oy, oz);
                            R.inv = mk(ix, iy, iz);
                            R.octinv = oct;
                            d = mk(dx, dy, dz);
                            tmax = tm;
                            best = bb;
                            second = FLT_MAX;
                            bu = bv = 0.f;
                            slot = kAny ? 0 : -1;
                            slot2 = -1;
                            src = es;
                            dst = ed;
                            use_limit = (how & 16) != 0;
                            ray = rr;
                            owner = ow;
                            if (kSeg) {
                                seg = sg;
                                cn = segs[seg].cnodes;
                                tris = segs[seg].ctris;
                            }
                            grp = make_uint2(gx, gy);
                            tgrp = make_uint2(0u, 0u);
                            top = -1;
                            bot = 0;
                            mode = how & 15;
                            steps = 0;
                        }
                    }
                }
            }
        }
        // The lanes take each phase together: without the barriers the compiler duplicates the
        // phases for the paths that lead to them, and the lanes of a warp run them apart (16,384
        // soup rays 1.43 against 0.76 ms, 4M 40.2 against 38.4).
        __syncwarp();
        const bool walk = ray >= 0 && !finished && (!kExact || mode <= kModeCareful);
        bool failed = false;
        if (walk) {
            if (kAny && owner >= 0 && (*(volatile int32_t*)&sh.slot[owner] & 1)) finished = true;
            // node phase: a lane without pending triangles takes its next internal child
            if (!finished && (tgrp.y & 0xFFu) == 0u) {
                if ((grp.y & 0xFF000000u) == 0u) {
                    if (top < bot) finished = true;
                    else grp = wstack_get<kSmemN>(sst, lst, top--);
                }
                if (!finished) {
                    const uint32_t bit = 31u - __clz(grp.y & 0xFF000000u);
                    grp.y &= ~(1u << bit);
                    const uint32_t s = (bit - 24u) ^ R.octinv;
                    const uint32_t idx = grp.x + __popc(grp.y & 0xFFu & ((1u << s) - 1u));
                    if (grp.y & 0xFF000000u) {
                        if (top + 1 >= kWideStack) failed = true;
                        else wstack_put<kSmemN>(sst, lst, ++top, grp);
                    }
                    uint32_t cbase, tbase, masks;
                    float bound;
                    if (kExact) {
                        bound = kAny ? __int_as_float(0x7f800000) : tmax * kSlack;
                    } else if (kAny) {
                        bound = tmax;
                    } else {
                        bound = best;
                        if (owner >= 0) bound = fminf(bound, __int_as_float(*(volatile int32_t*)&sh.bound[owner]));
                        bound = fminf(bound, tmax);
                    }
                    if (kStats) ++st.nodes;
                    const uint32_t h = node_hits(cn, idx, R, bound, cbase, tbase, masks);
                    grp = make_uint2(cbase, (h & 0xFF000000u) | (masks & 0xFFu));
                    tgrp = make_uint2(tbase, (h & 0xFFu) | (masks & 0xFF00u));
                }
            }
        }
        __syncwarp();
        if (walk) {
            // triangle phase: one triangle per iteration
            if (!finished && (tgrp.y & 0xFFu) != 0u) {
                const uint32_t s = (uint32_t)(__ffs(tgrp.y) - 1);
                tgrp.y &= tgrp.y - 1u;
                if (kStats) ++st.tris;
                const uint32_t at = tgrp.x + __popc((tgrp.y >> 8) & ((1u << s) - 1u));
                f3 v0, e1, e2;
                int id, mesh;
                load_tri(tris, (int64_t)at, v0, e1, e2, id, mesh);
                float t, u, v;
                if (kAny) {
                    if (mesh != src && mesh != dst && tri_test(R.o, d, v0, e1, e2, t, u, v) && (!use_limit || t < tmax)) {
                        if (!kExact || own_box(kSeg ? segs[seg] : one, at, R, d) >= 0.f) {
                            slot |= 1;
                            finished = true;
                        }
                    }
                } else if (tri_test(R.o, d, v0, e1, e2, t, u, v)) {
                    // slot < 0: no hit of this lane's own (best is then the bound it started from)
                    const bool mine = slot >= 0;
                    const bool better = !(t > tmax) && ((!mine && (t <= best || best == FLT_MAX)) || t < best);
                    bool reached = better;
                    if (kExact && better && mode == kModeCareful) reached = own_box(one, at, R, d) >= 0.f;
                    if (reached) {
                        if (mine) second = best;
                        slot2 = -1;
                        best = t;
                        slot = (int32_t)at;
                        bu = u;
                        bv = v;
                        if (!kExact && owner >= 0) atomicMin(&sh.bound[owner], __float_as_int(t));
                    } else if (!better && !(t > tmax)) {
                        if (kExact && mine && t == best) slot2 = slot2 == -1 ? (int32_t)at : -2;
                        else if (kExact) second = fminf(second, t);
                        if (!kExact && t == best && id < tri_id(tris, slot)) {  // at equal distances the lower triangle
                            slot = (int32_t)at;
                            bu = u;
                            bv = v;
                        }
                    }
                    if (kExact && !(t < FLT_MAX)) failed = true;  // not a distance that can be compared
                }
            }
            if (!finished && (failed || ++steps >= max_steps)) {
                if (!kExact) atomicOr(flag, failed ? kFlagStackOverflow : kFlagStepLimit);
                if (kAny) slot |= 4;
                else second = -1.f;
                finished = true;
            }
        } else if (kExact && ray >= 0 && !finished) {
            // the binary traversal's steps, exactly as in trace.cu; grp.x is the node reference
            const TraceSeg& S = kSeg ? segs[seg] : one;
            const f3 inv = mk(1.f / d.x, 1.f / d.y, 1.f / d.z);
            const int32_t ref = (int32_t)grp.x;
            bool pop = false, failed = false;
            if (!kAny && steps == 0) {  // a missed root box ends the ray
                const float* rb = S.root_box;
                if (!(slab(rb[0], rb[1], rb[2], rb[3], rb[4], rb[5], R.o, inv) >= 0.f)) finished = true;
            }
            if (finished) {
            } else if (ref >= 0) {
                NodeRegs nr;
                load_node(S.nodes, ref, nr);
                const int2 dd = make_int2(__float_as_int(nr.hi[4]), __float_as_int(nr.hi[5]));
                const float ml = slab(nr.lo[0], nr.lo[1], nr.lo[2], nr.lo[3], nr.lo[4], nr.lo[5], R.o, inv);
                const float mr = slab(nr.lo[6], nr.lo[7], nr.hi[0], nr.hi[1], nr.hi[2], nr.hi[3], R.o, inv);
                const bool okl = ml >= 0 && (kAny || (ml < best && !(ml > tmax)));
                const bool okr = mr >= 0 && (kAny || (mr < best && !(mr > tmax)));
                if (okl && okr) {
                    if (top + 1 >= kWideStack) {
                        failed = true;
                    } else {
                        const bool lfar = ml > mr;
                        wstack_put<kSmemN>(sst, lst, ++top, make_uint2((uint32_t)(lfar ? dd.x : dd.y), 0u));
                        grp.x = (uint32_t)(lfar ? dd.y : dd.x);
                    }
                } else if (okl) {
                    grp.x = (uint32_t)dd.x;
                } else if (okr) {
                    grp.x = (uint32_t)dd.y;
                } else {
                    pop = true;
                }
            } else {
                f3 v0, e1, e2;
                int id, mesh;
                load_tri(S.tris, ~ref, v0, e1, e2, id, mesh);
                float t, u, v;
                if (kAny) {
                    if (mesh != src && mesh != dst && tri_test(R.o, d, v0, e1, e2, t, u, v) && (!use_limit || t < tmax)) {
                        slot = 1;
                        finished = true;
                    }
                } else if (tri_test(R.o, d, v0, e1, e2, t, u, v)) {
                    if ((slot < 0 || t < best) && !(t > tmax)) {
                        best = t;
                        slot = id;
                        bu = u;
                        bv = v;
                    }
                }
                pop = true;
            }
            if (!finished) {
                if (failed || ++steps >= max_steps) {
                    atomicOr(flag, failed ? kFlagStackOverflow : kFlagStepLimit);
                    if (kAny) slot = 4;
                    else slot = -2;
                    finished = true;
                } else if (pop) {
                    if (top < 0) finished = true;
                    else grp.x = wstack_get<kSmemN>(sst, lst, top--).x;
                }
            }
        }
    }
    flush_stats<kStats>(st, stats);
}

constexpr int kMinCap = 4;  // rays a warp holds at least (fewer leave most of each instruction idle)

template <bool kAny, bool kStats, bool kSeg, bool kExact, int kSmemN>
cav_status launch_one(cav_ctx* ctx, const TraceSeg& one, const TraceSeg* segs, int nseg, int64_t n, int block, int batch,
                      cudaStream_t s, unsigned long long* counter, unsigned long long* stats) {
    const size_t dyn = sizeof(uint2) * kSmemN * (size_t)block;
    auto* kernel = k_trace_wide<kAny, kStats, kSeg, kExact, kSmemN>;
    int grid = grid_for(ctx, kernel, block, dyn);
    bool counted = true;
    if (!one.n_dev) grid = share_grid(n, kMinCap, block, grid, counted);
    if (counted) CAV_CUDA(ctx, cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s));
    kernel<<<grid, block, dyn, s>>>(one, segs, nseg, n, counter, batch, kMinCap, ctx->max_trace_steps,
                                    ctx->d_error + (kAny ? 3 : 2), stats);
    CAV_CUDA(ctx, cudaGetLastError());
    return CAV_OK;
}

template <bool kAny, bool kSeg>
cav_status launch_wide(cav_ctx* ctx, const TraceSeg& one, const TraceSeg* segs, int nseg, int64_t n, cudaStream_t s,
                       unsigned long long* counter, unsigned long long* stats) {
    const int block = ctx->wide_block > 0 ? ctx->wide_block : 128;
    const int batch = ctx->wide_batch > 0 ? ctx->wide_batch : kDefaultRefill;
    if (!kSeg && stats)
        return launch_one<kAny, !kSeg, kSeg, false, 0>(ctx, one, segs, nseg, n, block, batch, s, counter, stats);
    if (!kSeg && (ctx->wide_smem_stack > 0 || (ctx->wide_smem_stack < 0 && !kAny)))
        return launch_one<kAny, false, kSeg, false, kSeg ? 0 : kWideSmemStack>(ctx, one, segs, nseg, n, block, batch, s,
                                                                              counter, nullptr);
    return launch_one<kAny, false, kSeg, false, 0>(ctx, one, segs, nseg, n, block, batch, s, counter, nullptr);
}

TraceSeg wide_seg(const cav_bvh* bvh) {
    TraceSeg g{};
    g.nodes = bvh->tnodes;
    g.tris = bvh->tris;
    g.root_box = bvh->d_root_box;
    g.cnodes = bvh->cnodes;
    g.ctris = bvh->ctris;
    g.lbox = bvh->lbox;
    return g;
}

}  // namespace

// Several jobs' rays, each against its own tree, in one fast-mode launch (the server's merged
// wavefronts).  Every segment's cnodes / ctris must be set (ensure_wide on its tree).
cav_status trace_wide_segments(cav_ctx* ctx, bool any_hit, const TraceSeg* segs, int nseg, int64_t n, cudaStream_t s,
                               unsigned long long* counter) {
    if (nseg <= 0 || n == 0) return CAV_OK;
    if (nseg > kMaxSeg) return set_error(ctx, CAV_ERR_INVALID_ARGUMENT, "too many trace segments in one launch");
    const TraceSeg none{};
    return any_hit ? launch_wide<true, true>(ctx, none, segs, nseg, n, s, counter, nullptr)
                   : launch_wide<false, true>(ctx, none, segs, nseg, n, s, counter, nullptr);
}

// ------------------------------------------------------------------ the view on the host
// Pinned words for the verdicts of view builds, handed out one to a build.
struct VerdictSlots {
    static constexpr int kCount = 1024;
    std::mutex mu;
    unsigned long long* words = nullptr;
    std::vector<int> free;
    std::vector<int> late;  // given back before the verdict was written

    bool arrived(int k) const { return (__atomic_load_n(words + k, __ATOMIC_ACQUIRE) & kArrived) != 0; }
    int take() {
        std::lock_guard<std::mutex> lk(mu);
        for (size_t i = 0; i < late.size();)
            if (arrived(late[i])) {
                free.push_back(late[i]);
                late[i] = late.back();
                late.pop_back();
            } else {
                ++i;
            }
        if (free.empty()) return -1;
        const int k = free.back();
        free.pop_back();
        words[k] = 0;
        return k;
    }
    void give(int k, bool written) {
        std::lock_guard<std::mutex> lk(mu);
        (written || arrived(k) ? free : late).push_back(k);
    }
    ~VerdictSlots() {
        if (!late.empty()) cudaDeviceSynchronize();
        cudaFreeHost(words);
    }
};

std::shared_ptr<VerdictSlots> make_verdict_slots() {
    auto v = std::make_shared<VerdictSlots>();
    if (cudaMallocHost((void**)&v->words, sizeof(*v->words) * VerdictSlots::kCount) != cudaSuccess) {
        cudaGetLastError();
        v->words = nullptr;
        return nullptr;
    }
    for (int k = 0; k < VerdictSlots::kCount; ++k) v->free.push_back(k);
    return v;
}

// One build of one or several trees' views: enqueued on a stream, complete once its verdict has
// arrived (or `done`, for those who wait).
struct ViewJob {
    void* arena = nullptr;
    std::atomic<int> refs{0};  // trees with a view in it
    int trees = 0;
    cudaEvent_t done = nullptr;
    unsigned long long stream = 0;             // the streams on which work enqueued since comes after it
    std::atomic<unsigned long long> also{0};
    std::shared_ptr<VerdictSlots> slots;
    int slot = -1;
    ViewJob* before = nullptr;  // a build of the tree alone that had failed
};

// kViewBegun: enqueued, no verdict yet.  kViewMixed: complete, the tree's own verdict is on the device.
// kViewUnscreened: a view that the exact mode does not use; kViewReady: one that it does.
enum ViewState { kViewFailed = -1, kViewNone = 0, kViewUnscreened = 1, kViewReady = 2, kViewBegun = 3, kViewMixed = 4 };

namespace {

// Wide nodes that a view of n triangles has at most.  A node has eight children, or triangles only
// (two or more): with F of the former and L of the latter, F + L - 1 of the children are nodes, so
// n >= L + 7 F + 1 and L <= 7 F + 1, and F + L is at most 4 (n - 2) / 7 + 1.  A child whose box area is
// no number is never opened, so infinite geometry can need a node for each internal node of the
// tree: its build fails within the bound and is done again without it (full).
uint32_t most_nodes(int64_t n, bool full) { return (uint32_t)(full ? n - 1 : std::min(n - 1, 4 * (n - 2) / 7 + 1)); }

std::mutex& view_mutex(const cav_bvh* bvh) { return bvh->shared ? bvh->shared->mu : bvh->view_mu; }

unsigned long long stream_id(cudaStream_t s) {
    unsigned long long id = 0;
    if (cudaStreamGetId(s, &id) != cudaSuccess) {
        cudaGetLastError();
        return ~0ull;  // no stream's
    }
    return id;
}

bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) return false;
    cudaGetLastError();
    return true;
}

// The state of a tree's view, with a verdict that has arrived taken over.
int view_state(const cav_bvh* bvh) {
    int st = bvh->wide_state.load(std::memory_order_acquire);
    if (st != kViewBegun) return st;
    const ViewJob* job = bvh->view_job;
    const unsigned long long w = __atomic_load_n(job->slots->words + job->slot, __ATOMIC_ACQUIRE);
    if (!(w & kArrived)) return st;
    int next = kViewMixed;
    if (!(w & (kSomeFailed | kSomeUnscreened))) next = kViewReady;
    else if (job->trees == 1) next = (w & kSomeFailed) ? kViewFailed : kViewUnscreened;
    float lines;
    const uint32_t bits = (uint32_t)(w >> 32);
    memcpy(&lines, &bits, 4);
    bvh->boxes_per_line.store(lines);
    bvh->wide_state.compare_exchange_strong(st, next);
    return bvh->wide_state.load(std::memory_order_acquire);
}

// Enqueues the build of the view of `bvh` on the stream, together with the missing views of the
// small trees of its batch; view_mutex(bvh) is held.  Every tree of a batch is complete where `bvh`
// is: the same launches built them all.  Sets no error: the exact mode does without.
cudaError_t begin_view(cav_ctx* ctx, const cav_bvh* bvh, cudaStream_t s) {
    auto round = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const bool full = bvh->wide_state.load() == kViewFailed;
    auto bytes = [&](const cav_bvh* b) {
        return round(sizeof(CNode) * (size_t)most_nodes(b->n, full)) + round(sizeof(TriRec) * (size_t)b->n) +
               round(2 * sizeof(float4) * (size_t)b->n) + round(sizeof(int32_t) * (size_t)most_nodes(b->n, full));
    };
    std::vector<const cav_bvh*> g{bvh};
    size_t need = bytes(bvh);
    if (bvh->shared && bvh->n <= kGroupTris && bvh->wide_state.load() == kViewNone) {
        for (const cav_bvh* b : bvh->shared->trees)
            if (b && b != bvh && b->wide_state.load() == kViewNone && b->n <= kGroupTris && b->n > kTinyTris) {
                g.push_back(b);
                need += bytes(b);
            }
        if (need > kGroupBytes || bvh->n > kGroupShare * (int64_t)g.size()) {
            g.resize(1);
            need = bytes(bvh);
        }
    }
    const int K = (int)g.size();
    need += round(sizeof(WideTree) * K) + round(sizeof(WideCtr) * K);
    auto job = std::make_unique<ViewJob>();
    job->slots = ctx->verdicts;
    job->slot = job->slots->take();
    if (job->slot < 0) return cudaErrorMemoryAllocation;  // as many builds under way as there are words
    cudaError_t e = dev_alloc(ctx, &job->arena, need, s, true);
    if (e == cudaSuccess && (e = cudaEventCreateWithFlags(&job->done, cudaEventDisableTiming)) != cudaSuccess)
        cudaFreeAsync(job->arena, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        job->slots->give(job->slot, true);
        return e;
    }
    unsigned char* p = (unsigned char*)job->arena;
    auto carve = [&](size_t b) {
        unsigned char* r = p;
        p += round(b);
        return (void*)r;
    };
    std::vector<WideTree> t(K);
    for (int k = 0; k < K; ++k) {
        const cav_bvh* b = g[k];
        t[k].tn = b->tnodes;
        t[k].tris_in = b->tris;
        t[k].root_box = b->d_root_box;
        t[k].nodes = most_nodes(b->n, full);
        t[k].out = (CNode*)carve(sizeof(CNode) * (size_t)t[k].nodes);
        t[k].tris_out = (TriRec*)carve(sizeof(TriRec) * (size_t)b->n);
        t[k].lbox = (float4*)carve(2 * sizeof(float4) * (size_t)b->n);
        t[k].task = (int32_t*)carve(sizeof(int32_t) * (size_t)t[k].nodes);
        t[k].tris = (uint32_t)b->n;
    }
    WideTree* dt = (WideTree*)carve(sizeof(WideTree) * K);
    WideCtr* dc = (WideCtr*)carve(sizeof(WideCtr) * K);
    if (K > 1) {
        // pageable memory: staged before the call returns
        e = cudaMemcpyAsync(dt, t.data(), sizeof(WideTree) * K, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) {
            k_wide_build_group<<<K * kGroupBlocks, kGroupThreads, 0, s>>>(dt, dc, ctx->sort_wait_ns);
            e = cudaGetLastError();
        }
    } else {
        const WideTree& w = t[0];
        k_wide_init<<<1, 32, 0, s>>>(w.root_box, w.tris, w.task, dc);
        // about one wide node per four triangles, eight lanes each; every block co-resident
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_wide_build, kBuildThreads, 0);
        const int64_t room = (int64_t)ctx->num_sms * std::min(std::max(per_sm, 1), 8);
        const int grid = (int)std::min<int64_t>(room, std::max<int64_t>(1, bvh->n * 2 / kBuildThreads));
        uint32_t max_nodes = w.nodes, max_tris = w.tris;
        uint64_t wait_ns = ctx->sort_wait_ns;
        void* args[] = {(void*)&w.tn, (void*)&w.tris_in, (void*)&w.task, (void*)&w.out, (void*)&w.tris_out, (void*)&w.lbox,
                        &dc,          &max_nodes,        &max_tris,      &wait_ns};
        e = cudaLaunchCooperativeKernel((const void*)k_wide_build, dim3(grid), dim3(kBuildThreads), args, 0, s);
    }
    bool reports = false;
    if (e == cudaSuccess) {
        k_wide_verdict<<<1, 32, 0, s>>>(dc, K, job->slots->words + job->slot);
        e = cudaGetLastError();
        reports = e == cudaSuccess;
    }
    if (e == cudaSuccess) e = cudaEventRecord(job->done, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        cudaFreeAsync(job->arena, s);
        cudaEventDestroy(job->done);
        job->slots->give(job->slot, !reports);
        return e;
    }
    job->stream = stream_id(s);
    job->trees = K;
    job->refs = K;
    if (K == 1) job->before = bvh->view_job;
    ViewJob* held = job.release();
    for (int k = 0; k < K; ++k) {
        g[k]->view_job = held;
        g[k]->cnodes = t[k].out;
        g[k]->ctris = t[k].tris_out;
        g[k]->lbox = t[k].lbox;
        g[k]->wctr = dc + k;
        g[k]->wide_state.store(kViewBegun, std::memory_order_release);
    }
    return cudaSuccess;
}

}  // namespace

// The view of a tree, complete: built and waited for where it is missing.
cav_status ensure_wide(cav_ctx* ctx, const cav_bvh* bvh, cudaStream_t s) {
    for (bool again = false;;) {
        int st = view_state(bvh);
        if (st == kViewReady || st == kViewUnscreened) return CAV_OK;
        if (st == kViewBegun || st == kViewMixed) {
            WideCtr c;
            cudaError_t e = cudaEventSynchronize(bvh->view_job->done);
            if (e == cudaSuccess) e = cudaMemcpyAsync(&c, bvh->wctr, sizeof(c), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return cuda_error(ctx, e, "fast traversal layout");
            const bool good = !c.failed && c.tris == c.want;
            bvh->boxes_per_line.store(c.area / c.root_area);
            bvh->wide_state.compare_exchange_strong(st, !good ? kViewFailed : (c.unscreened ? kViewUnscreened : kViewReady));
            continue;
        }
        if (st == kViewFailed && again) return set_error(ctx, CAV_ERR_CUDA, "fast traversal layout: not every triangle placed");
        again = true;
        std::lock_guard<std::mutex> lk(view_mutex(bvh));  // several host threads may reach one tree at once
        if (bvh->wide_state.load() > 0) continue;
        const cudaError_t e = begin_view(ctx, bvh, s);
        if (e != cudaSuccess) return cuda_error(ctx, e, "fast traversal layout");
    }
}

void detach_wide(cav_bvh* bvh, cudaStream_t s, bool async, std::vector<void*>& mem) {
    for (ViewJob* job = bvh->view_job; job;) {
        ViewJob* const before = job->before;
        if (job->refs.fetch_sub(1) == 1) {
            if (async) cudaStreamWaitEvent(s, job->done, 0);
            mem.push_back(job->arena);
            cudaEventDestroy(job->done);
            job->slots->give(job->slot, false);
            delete job;
        }
        job = before;
    }
    bvh->view_job = nullptr;
    bvh->wide_state.store(kViewNone);
}

// Rays that a tree must have been asked about before the exact mode builds its view.  From 4,096
// triangles on the view is worth it with the first 512 rays or soon after (closest hits, the call
// with the view's build, the binary traversal, and the next call: soups of 4,200 triangles 124,
// 135 and 56 us, of 10,000 147, 234 and 73 us, of 100,000 0.41, 1.12 and 0.25 ms, of 1M 2.6, 7.3 and
// 1.8 ms; spheres, whose lines meet few boxes, of 20,498 136, 64 and 46 us, of 327,698 302, 279 and
// 64 us).  Smaller trees gain less than they pay for many calls (1,000 triangles and 16,384 rays
// 106, 66 and 60 us; 2,000 125, 94 and 71).  A batched build's trees get their views together.
static int64_t screen_min_rays(const cav_bvh* bvh) { return bvh->n >= 4096 || bvh->shared ? 512 : 16384; }

bool view_is_sparse(const cav_bvh* bvh) {
    return view_state(bvh) == kViewReady && bvh->boxes_per_line.load() <= kSparse;
}

// How n rays (negative: a number that only the device knows) of the exact mode go.  Once the tree
// has been asked about enough of them its view's build is enqueued on the stream; nothing waits for
// it.  Until its verdict has arrived, calls on that stream come after it and let the device
// decide, and those on other streams take the binary traversal.  So do a lowered step limit, a
// stream in capture without a complete view, no memory for one (asked for again after twice
// as many rays as the last time), geometry out of the screening range, and many closest hits where
// boxes overlap densely.
ViewUse view_use(cav_ctx* ctx, const cav_bvh* bvh, bool any_hit, int64_t n, cudaStream_t s) {
    if (bvh->n <= kTinyTris) return kUseBinary;
    if (ctx->max_trace_steps < kMaxSteps) return kUseBinary;  // a lowered limit counts binary visits
    int st = view_state(bvh);
    if (st == kViewNone) {
        const int64_t more = std::max<int64_t>(n, 0);
        const int64_t seen = bvh->rays_seen.fetch_add(more) + more;
        if (seen < screen_min_rays(bvh) << std::min(bvh->view_misses.load(), 24)) return kUseBinary;
        if (capturing(s)) return kUseBinary;
        std::lock_guard<std::mutex> lk(view_mutex(bvh));
        if (bvh->wide_state.load() == kViewNone && begin_view(ctx, bvh, s) != cudaSuccess) {
            bvh->view_misses.fetch_add(1);
            bvh->rays_seen.store(0);
            return kUseBinary;
        }
        st = view_state(bvh);
    }
    if (st == kViewBegun) {
        const unsigned long long id = stream_id(s);
        const bool after = id == bvh->view_job->stream || id == bvh->view_job->also.load();
        return after && !capturing(s) ? kUseBoth : kUseBinary;
    }
    if (st == kViewMixed) return kUseBoth;
    if (st != kViewReady) return kUseBinary;
    if (any_hit || view_is_sparse(bvh)) return kUseView;
    return n < 0 ? kUseBoth : (n <= kFewRays ? kUseView : kUseBinary);
}

cav_status share_view(cav_ctx* ctx, const cav_bvh* bvh, bool any_hit, int64_t n, cudaStream_t a, cudaStream_t b) {
    if (view_use(ctx, bvh, any_hit, n, a) != kUseBoth || view_state(bvh) != kViewBegun) return CAV_OK;
    ViewJob* job = bvh->view_job;
    if (job->stream != stream_id(a)) return CAV_OK;
    CAV_CUDA(ctx, cudaStreamWaitEvent(b, job->done, 0));
    job->also.store(stream_id(b));
    return CAV_OK;
}

cav_status trace_screened(cav_ctx* ctx, const cav_bvh* bvh, const TraceSeg& q, bool any_hit, int64_t n, cudaStream_t s,
                          unsigned long long* counter) {
    TraceSeg one = q;
    const TraceSeg w = wide_seg(bvh);
    one.cnodes = w.cnodes;
    one.ctris = w.ctris;
    one.lbox = w.lbox;
    const int block = ctx->trace_block > 0 ? std::min(ctx->trace_block, 256) : 128;
    const int batch = ctx->trace_batch > 0 ? ctx->trace_batch : kDefaultRefill;
    const bool smem = ctx->screen_smem_stack < 0 ? !any_hit : ctx->screen_smem_stack > 0;
    if (any_hit)
        return smem ? launch_one<true, false, false, true, kWideSmemStack>(ctx, one, nullptr, 0, n, block, batch, s, counter, nullptr)
                    : launch_one<true, false, false, true, 0>(ctx, one, nullptr, 0, n, block, batch, s, counter, nullptr);
    return smem ? launch_one<false, false, false, true, kWideSmemStack>(ctx, one, nullptr, 0, n, block, batch, s, counter, nullptr)
                : launch_one<false, false, false, true, 0>(ctx, one, nullptr, 0, n, block, batch, s, counter, nullptr);
}

cav_status trace_wide_closest(cav_ctx* ctx, const cav_bvh* bvh, const cav_ray* rays, int64_t n, const uint32_t* n_dev,
                              int32_t* prim, float* t, float* uv, cudaStream_t s, unsigned long long* counter,
                              unsigned long long* stats) {
    cav_status st = ensure_wide(ctx, bvh, s);
    if (st != CAV_OK) return st;
    TraceSeg one = wide_seg(bvh);
    one.rays = rays;
    one.prim = prim;
    one.t = t;
    one.uv = uv;
    one.n_dev = n_dev;
    return launch_wide<false, false>(ctx, one, nullptr, 0, n, s, counter, stats);
}

cav_status trace_wide_any(cav_ctx* ctx, const cav_bvh* bvh, const cav_ray* rays, const float* limit,
                          const int32_t* excl, int64_t n, const uint32_t* n_dev, uint8_t* occ, cudaStream_t s,
                          unsigned long long* counter, unsigned long long* stats) {
    cav_status st = ensure_wide(ctx, bvh, s);
    if (st != CAV_OK) return st;
    TraceSeg one = wide_seg(bvh);
    one.rays = rays;
    one.limit = limit;
    one.excl = excl;
    one.occ = occ;
    one.n_dev = n_dev;
    return launch_wide<true, false>(ctx, one, nullptr, 0, n, s, counter, stats);
}

}  // namespace cav
