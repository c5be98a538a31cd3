// Kernels of the render hot path and their launchers (declared in kernels.h).
// Compiled with -fmad=false (see x86sem.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "packet_refill.cuh"
#include "packet_warp.cuh"
#include "path_refill.cuh"
#include "shade.cuh"

namespace cvx {

__device__ ApproxTables g_tables;

// Copies the 8 KB approximation tables into shared memory.
__device__ __forceinline__ void load_tables(ApproxTables& sm) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&g_tables);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&sm);
    for (int i = threadIdx.x; i < (int)(sizeof(ApproxTables) / 4); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Scene preparation

__global__ void k_prep_geom(const cvx_triangle* __restrict__ tris, uint32_t n, float4* __restrict__ geom,
                            TriShade* __restrict__ shade) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const cvx_triangle& t = tris[i];
        F3 v0 = f3(t.v0[0], t.v0[1], t.v0[2]), v1 = f3(t.v1[0], t.v1[1], t.v1[2]), v2 = f3(t.v2[0], t.v2[1], t.v2[2]);
        F3 e1 = sub(v0, v2), e2 = sub(v1, v0);
        F3 n = cross(e1, e2);
        geom[3 * i] = make_float4(v0.x, v0.y, v0.z, n.x);
        geom[3 * i + 1] = make_float4(e1.x, e1.y, e1.z, n.y);
        geom[3 * i + 2] = make_float4(e2.x, e2.y, e2.z, n.z);
        TriShade s;
        s.uv[0] = t.uv0[0];
        s.uv[1] = t.uv0[1];
        s.uv[2] = t.uv1[0];
        s.uv[3] = t.uv1[1];
        s.uv[4] = t.uv2[0];
        s.uv[5] = t.uv2[1];
        s.material = t.material;
        s.pad = 0u;
        shade[i] = s;
    }
}

// The wide records (traverse.cuh) of a scene's node pairs.
__global__ void k_prep_wide(const float4* __restrict__ nodes, uint32_t n_pairs, float4* __restrict__ wide) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n_pairs; p += gridDim.x * blockDim.x) {
        const float4* np = nodes + 4 * (size_t)p;
        const float4 q0 = np[0], q1 = np[1], q2 = np[2], q3 = np[3];
        const float own[2][6] = {{q0.x, q0.y, q0.z, q0.w, q1.x, q1.y}, {q1.z, q1.w, q2.x, q2.y, q2.z, q2.w}};
        const uint32_t own_ref[2] = {__float_as_uint(q3.x), __float_as_uint(q3.y)};
        float b[4][6];
        uint32_t ref[4];
        for (int c = 0; c < 2; c++) {
            if ((own_ref[c] & 31u) == 0u) {  // internal: its children's boxes
                const float4* cp = nodes + 4 * (size_t)(own_ref[c] >> 6);
                const float4 c0 = cp[0], c1 = cp[1], c2 = cp[2], c3 = cp[3];
                const float kids[2][6] = {{c0.x, c0.y, c0.z, c0.w, c1.x, c1.y}, {c1.z, c1.w, c2.x, c2.y, c2.z, c2.w}};
                for (int k = 0; k < 2; k++)
                    for (int a = 0; a < 6; a++) b[2 * c + k][a] = kids[k][a];
                ref[2 * c] = __float_as_uint(c3.x);
                ref[2 * c + 1] = __float_as_uint(c3.y);
            } else {
                for (int a = 0; a < 6; a++) {
                    b[2 * c][a] = own[c][a];
                    b[2 * c + 1][a] = a < 3 ? kEmptyLo : -kEmptyLo;
                }
                ref[2 * c] = own_ref[c];
                ref[2 * c + 1] = 0u;
            }
        }
        float4* w = wide + 8 * (size_t)p;
        for (int a = 0; a < 3; a++) {
            const int lo = a == 0 ? 0 : a == 1 ? 4 : 3, hi = lo + (1 << a);
            w[lo] = make_float4(b[0][a], b[1][a], b[2][a], b[3][a]);
            w[hi] = make_float4(b[0][a + 3], b[1][a + 3], b[2][a + 3], b[3][a + 3]);
        }
        w[2] = make_float4(__uint_as_float(ref[0]), __uint_as_float(ref[1]), __uint_as_float(ref[2]),
                           __uint_as_float(ref[3]));
        w[5] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// LightRec (5 x float4): v0 area | e1 rnorm | e2 - | n - | normal -
__global__ void k_prep_lights(const cvx_triangle* __restrict__ tris, const uint32_t* __restrict__ ds, uint32_t n,
                              float4* __restrict__ lights) {
    __shared__ ApproxTables tab;
    load_tables(tab);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const cvx_triangle& t = tris[ds[i]];
        F3 v0 = f3(t.v0[0], t.v0[1], t.v0[2]), v1 = f3(t.v1[0], t.v1[1], t.v1[2]), v2 = f3(t.v2[0], t.v2[1], t.v2[2]);
        F3 e1 = sub(v0, v2), e2 = sub(v1, v0);
        F3 nn = cross(e1, e2);
        float rnorm = x_rsqrt(dot(nn, nn), tab);
        float area = 0.5f * x_rcp(rnorm, tab);
        F3 normal = mulk(nn, rnorm);
        lights[5 * i] = make_float4(v0.x, v0.y, v0.z, area);
        lights[5 * i + 1] = make_float4(e1.x, e1.y, e1.z, rnorm);
        lights[5 * i + 2] = make_float4(e2.x, e2.y, e2.z, 0.0f);
        lights[5 * i + 3] = make_float4(nn.x, nn.y, nn.z, 0.0f);
        lights[5 * i + 4] = make_float4(normal.x, normal.y, normal.z, 0.0f);
    }
}

// ---------------------------------------------------------------------------
// Nearest hit over SoA rays (Bvh::intersect_nearest, bvh.rs:659): eight
// consecutive rays are one reference packet, or each is traced by itself
// (k_intersect_packets, k_intersect_warp; k_intersect_refill, k_intersect_lanes
// below). k_intersect_octets walks the pairs with a packet per octet, and counts
// the boxes and triangles of packets (COUNT).

// Next unit (group or packet) index for the calling octet (one atomic by its lane 0).
__device__ __forceinline__ uint32_t octet_claim(uint32_t* counter, unsigned omask, int k) {
    uint32_t g = 0;
    if (k == 0) g = atomicAdd(counter, 1u);
    return __shfl_sync(omask, g, (int)(threadIdx.x & 24u));
}

template <bool COUNT>
__global__ void __launch_bounds__(256) k_intersect_octets(DeviceScene s, const RayCols rays, uint32_t n,
                                                          float far_dist, float* __restrict__ t_out,
                                                          int32_t* __restrict__ tri_out,
                                                          uint32_t* __restrict__ counters, uint32_t* __restrict__ err) {
    __shared__ ApproxTables tab;
    load_tables(tab);
    const unsigned omask = 0xffu << (threadIdx.x & 24u);
    const int k = threadIdx.x & 7;
    const uint32_t npk = (n + 7u) >> 3;
    // Packets (8 consecutive rays, one per octet) claimed one at a time from err[1].
    for (uint32_t pk = octet_claim(err + 1, omask, k); pk < npk; pk = octet_claim(err + 1, omask, k)) {
        uint32_t i = pk * 8u + (uint32_t)k;
        bool active = i < n;
        uint32_t src = active ? i : (i & ~7u);
        F3 o = f3(__ldg(rays.c[0] + src), __ldg(rays.c[1] + src), __ldg(rays.c[2] + src));
        F3 d = f3(__ldg(rays.c[3] + src), __ldg(rays.c[4] + src), __ldg(rays.c[5] + src));
        Hit h{far_dist, 0.0f, 0.0f, -1};
        Counters c{0u, 0u};
        bool ok;
        // The select-form slab test for a packet whose 8 rays all allow it,
        // decided once per packet outside the traversal loop (4M random rays:
        // 3.05 -> 2.92 ms; the same results).
        if (!COUNT && s.slab_sel &&
            oct_all(omask, select_form_recip(f3(x_rcp(d.x, tab), x_rcp(d.y, tab), x_rcp(d.z, tab)))))
            ok = traverse<true, true>(s, o, d, active, omask, h, tab, nullptr);
        else
            ok = traverse<true>(s, o, d, active, omask, h, tab, COUNT ? &c : nullptr);
        if (!ok) atomicOr(err, kErrStackOverflow);
        if (active) {
            t_out[i] = h.t;
            tri_out[i] = h.tri;
            if (COUNT) {
                counters[i] = c.aabb;
                counters[n + i] = c.tri;
            }
        }
    }
}

constexpr int32_t kDeferredRay = -2;  // never a hit index: -1 is the miss

// Ray source of the isolated nearest-hit query: SoA rays in, (t, index) out.
struct SoaRays {
    const float4* nodes;
    const float4* wide;
    const float4* geom;
    RayCols rays;
    uint32_t n;
    float far_dist;
    float* t_out;
    int32_t* tri_out;
    uint32_t* counters;
    uint32_t slab_sel;  // DeviceScene::slab_sel
    __device__ __forceinline__ bool load(uint32_t r, F3& o, F3& d, float& far, const float4*& nd,
                                         const float4*& gm) const {
        nd = nodes;
        gm = geom;
        o = f3(__ldg(rays.c[0] + r), __ldg(rays.c[1] + r), __ldg(rays.c[2] + r));
        d = f3(__ldg(rays.c[3] + r), __ldg(rays.c[4] + r), __ldg(rays.c[5] + r));
        far = far_dist;
        return true;
    }
    __device__ __forceinline__ void first_scene(const float4*& nd, const float4*& wd, const float4*& gm) const {
        nd = nodes;
        wd = wide;
        gm = geom;
    }
    // A ray left to k_intersect_deferred (its index word holds kDeferredRay).
    __device__ __forceinline__ void defer(uint32_t r) const { tri_out[r] = kDeferredRay; }
    __device__ __forceinline__ void store(uint32_t r, const Hit& h, uint32_t na, uint32_t nt) const {
        t_out[r] = h.t;
        tri_out[r] = h.tri;
        if (counters) {
            counters[r] = na;
            counters[n + r] = nt;
        }
    }
};

// Staged ray supply of the isolated query: a warp claims 32 consecutive rays
// at a time and copies them into shared memory with cp.async, one batch ahead
// of use. A lane that finishes a ray takes the next one from shared memory, so
// neither the claim's atomic nor the ray's DRAM load stalls the warp.
struct StagedSoaClaim {
    const SoaRays& src;
    uint32_t* next_ray;
    float (*buf)[6][32];  // this warp's two batches: [batch][component][slot]
    uint32_t base_cur, base_nxt, used;
    int cur;

    __device__ __forceinline__ uint32_t claim32(int lane) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(next_ray, 32u);
        return __shfl_sync(0xffffffffu, b, 0);
    }
    __device__ __forceinline__ void issue(int which, uint32_t base, int lane) {
        uint32_t r = base + (uint32_t)lane;
        if (r < src.n)
            for (int c = 0; c < 6; c++) cp_async4(&buf[which][c][lane], src.rays.c[c] + r);
        cp_async_commit();
    }
    __device__ __forceinline__ void init(int lane) {
        base_cur = claim32(lane);
        issue(0, base_cur, lane);
        base_nxt = claim32(lane);
        issue(1, base_nxt, lane);
        cp_async_wait_one_pending();
        __syncwarp();
        cur = 0;
        used = 0;
    }
    __device__ __forceinline__ int claim(unsigned b, bool want, int lane, uint32_t& r, RayIn& in) {
        uint32_t k = (uint32_t)__popc(b);
        if (used + k > 32u) {  // some lanes take from the next batch: it must have landed
            cp_async_wait_all();
            __syncwarp();
        }
        int res = kClaimNone;
        if (want) {
            uint32_t t = used + (uint32_t)__popc(b & ((1u << lane) - 1u));
            int which = t < 32u ? cur : cur ^ 1;
            uint32_t slot = t & 31u;
            r = (t < 32u ? base_cur : base_nxt) + slot;
            if (r < src.n) {
                in.o = f3(buf[which][0][slot], buf[which][1][slot], buf[which][2][slot]);
                in.d = f3(buf[which][3][slot], buf[which][4][slot], buf[which][5][slot]);
                in.far = src.far_dist;
                in.nodes = src.nodes;
                in.wide = src.wide;
                in.geom = src.geom;
                res = kClaimRay;
            } else {
                res = kClaimDone;
            }
        }
        used += k;
        if (used >= 32u) {  // the current batch is used up: the next one becomes current
            __syncwarp();    // every read of the old batch is done
            used -= 32u;
            cur ^= 1;
            base_cur = base_nxt;
            cp_async_wait_all();
            __syncwarp();
            base_nxt = claim32(lane);
            issue(cur ^ 1, base_nxt, lane);
        }
        return res;
    }
};

// MINB: resident blocks per SM the register allocation must allow (8: the
// compiler's choice, 64 registers; 10 and 12 cap registers for occupancy).
// CLAIM: lanes without a ray wait until this many want one. Short traversals
// (shallow trees) gain from large batches of claims, long ones lose more to
// the waiting: 16 for trees up to 40 levels, 8 beyond (measured on the
// 82k-triangle icosphere and on the 70-level tube).
// Wide records a lane walks per round of the warp's claim votes, before the
// round's leaf test (RefillRay::walk; traversal steps, leaves included, in the
// x86 form). The kernel is bound by instruction issue and the ALU pipe: with a
// leaf tested wherever a lane met one, the triangle code ran at nearly every
// step for one or two lanes; once per round it runs for about eight. A wide
// record replaces two to three pair steps (7.0 records against 13.2 pairs per
// random ray of the icosphere). 4M rays of the 28-level icosphere, 1M of the
// 70-level tube, 1M of the 19-level room: leaves at once 792, 580, 198 us;
// postponed, five pairs per round 684, 536, 179; records with the planes
// selected in registers 718, 522, 160; selected by address 673, 505, 155; and
// two planes per instruction 643, 490, 149; with the spare stack entry and one
// limit check per record 608, 468, 146. Two, three, four records per round:
// 615, 605, 719; 472, 475, 546; 145, 146, 168 us. Ending a round early when few
// lanes can walk on costs more in votes than it saves (748-794 us with pairs).
// Pairs (Form::kPairs and kX86), with the leaf of a step tested by the next one:
// 1, 3, 4 steps 0.798, 0.784, 0.777 ms per 4M rays of the icosphere, tube 1.538,
// 1.503, 1.499 (six: within noise).
constexpr int kQuerySteps = 2, kQueryPairSteps = 4;
// Each lane's traversal stack lies in local memory. A scene may keep the first 4, 8
// or 12 entries in shared memory instead (cvx_scene_set_query_stack, which the query
// autotuner sets per scene). Eight shared entries were the better default while
// pops of local entries waited for L1 (0.905 -> 0.878 ms per 4M rays); with pushes by
// selects one store to one memory is: 0 and 8 shared, us: 4M icosphere rays 564,
// 592, 1M tube rays 387, 408, room 136, 143; packets 598, 618, 1165, 1210, 290, 297.
// The other launch shapes keep 8.
constexpr int kQueryStackShared = 8;

// FORM kWide or, for scenes that allow the select form but have no wide records,
// kPairs: the rays that the form does not allow are marked kDeferredRay and traced
// by k_intersect_deferred.
// SHARED: stack entries of each lane in shared memory (the rest in local).
template <int MINB, bool COUNT, int CLAIM, Form FORM, int SHARED = kQueryStackShared>
__global__ void __launch_bounds__(128, MINB) k_intersect_refill(SoaRays src, uint32_t* __restrict__ next_ray,
                                                                uint32_t* __restrict__ err) {
    // The reciprocal table is read three times per ray: from global memory
    // (L1-resident), which leaves the shared-memory carve-out to L1.
    __shared__ float stage[4][2][6][32];
    __shared__ uint2 sstack[4][SHARED > 0 ? SHARED : 1][32];
    StagedSoaClaim claim{src, next_ray, stage[threadIdx.x >> 5], 0u, 0u, 0u, 0};
    claim.init(threadIdx.x & 31);
    constexpr bool kWide = FORM == Form::kWide;
    bool ok = traverse_refill<COUNT, false, CLAIM, SHARED, FORM, kWide ? kQuerySteps : kQueryPairSteps, kWide && CLAIM == 8>(
        src, claim, g_tables, &sstack[threadIdx.x >> 5][0][threadIdx.x & 31]);
    if (!ok) atomicOr(err, kErrStackOverflow);
}

// The packet query: packets of a warp stepped together (packet_refill.cuh). Rays
// are staged as in k_intersect_refill; an octet takes 8 consecutive ones.
// Bound by instruction issue and the ALU pipe. One packet per octet, each octet
// on its own path (the counting form below), against this: 1M rays of the
// 19-level room 345 -> 311 us, of the 28-level icosphere 817 -> 628 us, of the
// 70-level tube 1544 -> 1210 us. Stepping pairs instead of wide records 353, 738,
// 1340 us. 7 blocks per SM (72 registers; 8 blocks spill: 329, 676, 1355 us).
// STEPS records per round: 1, 2, 3 -> 309, 311, 379 us (room), 650, 628, 716
// (icosphere), 1210, 1279, 1543 (tube): 1 for trees deeper than 40 levels, else 2.
// Waiting for two finished packets before taking new ones 322, 701, 1312 us. With a
// round's second leaf tested at once and the stack in local memory: 290, 598, 1164
// us; 5, 6, 8 blocks 288, 287, 307 us (room), 601, 594, 642 (icosphere).
constexpr int kPacketBlocksPerSm = 7;
// Scenes without wide records, us at 131,072, 1M and 4M rays, a packet per octet
// (k_intersect_octets) against pairs in step, six per round (four: the same; one
// and two 1-5 % more): room with loose roots 102/120, 334/343, 1220/1151; icosphere
// 228/307, 806/725, 2988/2405; tube 526/547, 1479/1230, 5265/3949; a room under a
// chain of 80 levels 190/332, 912/961, 3513/3549. Pairs in step from 2^20 rays.
constexpr uint32_t kPairPacketRays = 1u << 20;
constexpr int kPairPacketSteps = 6;
template <int STEPS, Form FORM>
__global__ void __launch_bounds__(128, kPacketBlocksPerSm) k_intersect_packets(SoaRays src,
                                                                               uint32_t* __restrict__ next_ray,
                                                                               uint32_t* __restrict__ err) {
    __shared__ float stage[4][2][6][32];
    StagedSoaClaim claim{src, next_ray, stage[threadIdx.x >> 5], 0u, 0u, 0u, 0};
    claim.init(threadIdx.x & 31);
    bool ok = traverse_packets<STEPS, FORM>(src, claim, g_tables);
    if (!ok) atomicOr(err, kErrStackOverflow);
}

// Queries of up to kDirectRays rays in the default launch shape, whose time is
// that of their longest rays: no ray supply to set up, no counter to reset, no
// pass over deferred rays. Device time with the launch, before (k_intersect_
// packets, k_intersect_refill and its pass) -> one packet per warp / one ray per
// lane, us at 1021, 65,536, 262,144, 524,288 rays: packets, 28-level icosphere 93
// -> 68, 189 -> 130, 331 -> 270, 421 -> 449; single rays 69 -> 54, 121 -> 95, 145
// -> 124, 181 -> 182; packets, 19-level room 59 -> 46, 94 -> 63, 165 -> 123, 212 ->
// 198; 70-level tube 241 -> 163, 421 -> 255, 640 -> 497, 839 -> 787; single rays,
// room 52 -> 42, 68 -> 51, 91 -> 70, 112 -> 102, tube 234 -> 186, 218 -> 165, 312
// -> 287, 419 -> 470. Packets on scenes without wide records, a packet per octet
// -> this, at 4,096, 32,768, 65,536, 131,072 rays: room with loose roots 96 -> 58,
// 89 -> 72, 87 -> 82, 102 -> 120; icosphere 146 -> 112, 190 -> 163, 210 -> 201, 228 ->
// 307; under a chain of 80 levels (room) 165 -> 92, 164 -> 131, 167 -> 196, 191 -> 328.
// `err` may be page-locked host memory (it is stored to).
__global__ void __launch_bounds__(64) k_intersect_warp(DeviceScene s, const RayCols rays, uint32_t n, float far_dist,
                                                       float* __restrict__ t_out, int32_t* __restrict__ tri_out,
                                                       uint32_t* err) {
    __shared__ WarpStack stacks[2];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t i = (blockIdx.x * 2u + wid) * 8u + (lane & 7u);
    if ((i & ~7u) >= n) return;
    const bool active = i < n;
    const uint32_t src = active ? i : (i & ~7u);
    const F3 o = f3(__ldg(rays.c[0] + src), __ldg(rays.c[1] + src), __ldg(rays.c[2] + src));
    const F3 d = f3(__ldg(rays.c[3] + src), __ldg(rays.c[4] + src), __ldg(rays.c[5] + src));
    Hit h{far_dist, 0.0f, 0.0f, -1};
    const bool ok = traverse_warp(s, o, d, active, h, g_tables, stacks[wid]);
    if (active && lane < 8u) {
        t_out[i] = h.t;
        tri_out[i] = h.tri;
    }
    if (!ok) *reinterpret_cast<volatile uint32_t*>(err) = kErrStackOverflow;
}

__global__ void __launch_bounds__(32) k_intersect_lanes(DeviceScene s, const RayCols rays, uint32_t n, float far_dist,
                                                        float* __restrict__ t_out, int32_t* __restrict__ tri_out,
                                                        uint32_t* err) {
    const uint32_t i = blockIdx.x * 32u + threadIdx.x;
    if (i >= n) return;
    const F3 o = f3(__ldg(rays.c[0] + i), __ldg(rays.c[1] + i), __ldg(rays.c[2] + i));
    const F3 d = f3(__ldg(rays.c[3] + i), __ldg(rays.c[4] + i), __ldg(rays.c[5] + i));
    RefillRay ray;
    uint2 local_stack[kStackSlots];
    LocalStack stack{local_stack};
    ray.top = make_uint2(0u, 0u);
    ray.start(o, d, far_dist, s.nodes, s.wide, s.geom, g_tables);
    bool overflow = false;
    if (s.wide && select_form_ray(o, ray.inv)) {
        do {
            ray.walk(stack, overflow);
            ray.walk(stack, overflow);
        } while (!ray.test_leaf());
    } else {
        while (!ray.step<false, false>(stack, overflow)) {
        }
    }
    t_out[i] = ray.h.t;
    tri_out[i] = ray.h.tri;
    if (overflow) *reinterpret_cast<volatile uint32_t*>(err) = kErrStackOverflow;
}

// After k_intersect_refill: the rays it left (index word kDeferredRay:
// a reciprocal infinite or below 0.75 in magnitude) with the x86-form slab
// test. Such rays are rare (axis-parallel or very long directions), so the
// scan over the index words is most of the work: each thread reads
// kDeferredScan words spread over the whole array, independent coalesced loads
// in one round (a grid-stride loop of dependent loads took 16 us per 4M rays).
constexpr uint32_t kDeferredScan = 4;
__global__ void __launch_bounds__(256) k_intersect_deferred(SoaRays src, uint32_t* __restrict__ err) {
    const uint32_t stride = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    int32_t w[kDeferredScan];
#pragma unroll
    for (uint32_t k = 0; k < kDeferredScan; k++) {
        const uint64_t r = (uint64_t)t + (uint64_t)k * stride;
        w[k] = r < src.n ? __ldg(src.tri_out + r) : 0;
    }
    bool ok = true;
#pragma unroll 1
    for (uint32_t k = 0; k < kDeferredScan; k++) {
        if (w[k] != kDeferredRay) continue;
        const uint32_t r = t + k * stride;
        F3 o, d;
        float far;
        const float4 *nodes, *geom;
        src.load(r, o, d, far, nodes, geom);
        RefillRay ray;
        uint2 local_stack[kStackSlots];
        LocalStack stack{local_stack};
        ray.top = make_uint2(0u, 0u);
        ray.start(o, d, far, nodes, nullptr, geom, g_tables);
        bool overflow = false;
        while (!ray.step<false, false>(stack, overflow)) {
        }
        ok &= !overflow;
        src.store(r, ray.h, 0u, 0u);
    }
    if (!ok) atomicOr(err, kErrStackOverflow);
}

// ---------------------------------------------------------------------------
// Frame rendering: one octet renders one 8-pixel group (RNG_GROUP), or walks
// the 128 groups of one 32x32 patch in the reference's order (RNG_PATCH).

struct FrameArgs {
    DeviceScene s;
    DeviceCamera cam;
    uint32_t w, h, frame;
    uint32_t* rgba;
    uint32_t* gbuf;
    float* color;
    float* accum;
    unsigned long long* rays;
    uint32_t* err;
    uint32_t debug;  // Renderer::toggle_debug_view (renderer.rs:150-152)
    // patch order: patch width (a multiple of 16) and the patch origins
    // (x, y pairs; null: every patch of the frame, column by column)
    uint32_t patch;
    const uint32_t* patches;
    uint32_t n_patches;
    // per-lane path refill (k_render_refill): one word per 8-pixel group,
    // zero at launch
    uint32_t* group_em;
    // the counting form of k_render_refill: totals of boxes and triangles
    // tested and of light-PDF shading steps (3 words, zero at launch)
    unsigned long long* work;
    // k_render_refill: samples rendered by the launch (frames frame ..
    // frame + samples - 1, their paths claimed sample after sample). The last
    // sample writes the frame buffers as a one-sample launch does (without the
    // accumulator); sample s < samples - 1 writes its linear colour to
    // sample_color + 3 * w * h * s, for k_accumulate_samples.
    uint32_t samples;
    float* sample_color;
};

// Screen x (or y) of lane k of group g of the 16x4 block at (xb, yb), before
// jitter (renderer.rs:171-198).
__device__ __forceinline__ void block_coord(uint32_t w, uint32_t h, uint32_t xb, uint32_t yb, int g, int k,
                                            float* x, float* y, float* scale_out) {
    float scale = 2.0f / (float)w;
    float s2 = 2.0f * scale, s4 = 4.0f * scale, s8 = 8.0f * scale, s12 = 12.0f * scale;
    float bx = scale * ((float)(k & 3) + ((float)xb - (float)w * 0.5f));
    float by = scale * ((float)(k >> 2) + ((float)yb - (float)h * 0.5f));
    int col = g >> 1;
    float gx = col == 0 ? bx : col == 1 ? bx + s4 : col == 2 ? bx + s8 : bx + s12;
    float gy = (g & 1) ? by + s2 : by;
    *x = gx;
    *y = gy;
    *scale_out = scale;
}

__device__ __forceinline__ void store_pixel(const FrameArgs& a, uint32_t px, uint32_t py, const PixelOut& p) {
    if (px >= a.w || py >= a.h) return;
    size_t idx = (size_t)py * a.w + px;
    if (a.rgba) a.rgba[idx] = pack_color(p.color);
    if (a.gbuf) a.gbuf[idx] = pack_gbuffer(p);
    if (a.color) {
        a.color[3 * idx] = p.color.x;
        a.color[3 * idx + 1] = p.color.y;
        a.color[3 * idx + 2] = p.color.z;
    }
    if (a.accum) {
        a.accum[3 * idx] += p.color.x;
        a.accum[3 * idx + 1] += p.color.y;
        a.accum[3 * idx + 2] += p.color.z;
    }
}

__device__ __forceinline__ void flush_rays(const FrameArgs& a, uint32_t rays) {
    unsigned long long v = rays;
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31u) == 0u && v) atomicAdd(a.rays, v);
}

// An octet renders whole groups: single rays, the debug view, and packets of the
// scenes that k_render_packets leaves to it.
template <bool PACKET>
__global__ void __launch_bounds__(128, 8) k_render_group(FrameArgs a) {
    __shared__ ApproxTables tab;
    load_tables(tab);
    const int k = threadIdx.x & 7;
    const unsigned omask = 0xffu << (threadIdx.x & 24u);
    const uint32_t bw = (a.w + 15u) / 16u, bh = (a.h + 3u) / 4u;
    const uint32_t ngroups = bw * bh * 8u;
    uint32_t rays = 0;
    bool ok = true;
    // Octet index runs through the 8 groups of a 16x4 block, then blocks in
    // row-major order, so a warp covers half a block.
    // Groups are claimed one at a time by each octet (a counter in a.err[1]):
    // paths end after 1 to 5 bounces, so a fixed share of groups per octet
    // leaves some octets working long after the others (room scene frame
    // 0.815 against 0.874 ms with a grid-stride share).
    for (uint32_t gi = octet_claim(a.err + 1, omask, k); gi < ngroups; gi = octet_claim(a.err + 1, omask, k)) {
        uint32_t blk = gi >> 3;
        int g = (int)(gi & 7u);
        uint32_t xb = (blk % bw) * 16u, yb = (blk / bw) * 4u;
        uint32_t gx = xb + 4u * (uint32_t)(g >> 1), gy = yb + 2u * (uint32_t)(g & 1);
        if (gx >= a.w || gy >= a.h) continue;  // whole group outside the frame (octet-uniform)
        float x, y, scale;
        block_coord(a.w, a.h, xb, yb, g, k, &x, &y, &scale);
        LaneRng rng;
        rng.seed(gx, gy, a.frame, k);
        x = fmaf(unit_from(rng.next()), scale, x);
        y = fmaf(unit_from(rng.next()), scale, y);
        PixelOut p;
        if (a.debug) ok &= render_pixels_debug<PACKET>(a.s, a.cam, x, y, omask, tab, p, rays);
        else ok &= render_pixels<PACKET>(a.s, a.cam, x, y, rng, omask, tab, p, rays);
        store_pixel(a, gx + (uint32_t)(k & 3), gy + (uint32_t)(k >> 2), p);
    }
    if (!ok) atomicOr(a.err, kErrStackOverflow);
    flush_rays(a, rays);
}

// Pixel of path p (lane p & 7 of group p >> 3; groups numbered as in
// k_render_group) and its group's origin.
__device__ __forceinline__ void path_pixel(uint32_t p, uint32_t bw, uint32_t& gx, uint32_t& gy, uint32_t& px,
                                           uint32_t& py) {
    uint32_t gi = p >> 3, blk = gi >> 3, g = gi & 7u, k = p & 7u;
    uint32_t xb = (blk % bw) * 16u, yb = (blk / bw) * 4u;
    gx = xb + 4u * (g >> 1);
    gy = yb + 2u * (g & 1u);
    px = gx + (k & 3u);
    py = gy + (k >> 2);
}

// The paths of a launch for path_refill. One sample (MULTI false): path p is
// lane p & 7 of group p >> 3, groups numbered as in k_render_group. MULTI:
// a.samples samples, claimed one after the other: claim number p is path
// p mod per of sample p / per, per being the paths of one sample (a multiple
// of 64, so both numbers share their lane and group-in-block bits). The two
// forms are separate instantiations: the sample logic in the one-sample
// kernel's loop slowed it by 6-7 % (tube 2.945 -> 3.12 ms, room 0.705 ->
// 0.759 ms). The reference keeps the sample, so that only the path's start
// divides (tube 2.356 -> 2.248 ms per sample with 16 per launch, room 0.620 ->
// 0.588 ms).
template <bool MULTI>
struct FramePaths {
    static constexpr bool kOneScene = true;
    struct PathRef {
        uint32_t path;  // within its sample
        uint32_t smp;
    };
    const FrameArgs& a;
    uint32_t bw, bh, rays;

    __device__ __forceinline__ uint32_t per() const { return bw * bh * 64u; }
    __device__ __forceinline__ uint32_t n_paths() const { return MULTI ? per() * a.samples : per(); }
    __device__ __forceinline__ uint32_t claim(uint32_t n) { return atomicAdd(a.err + 1, n); }
    __device__ __forceinline__ bool begin(uint32_t p, PathRef& r, F3& o, F3& d, LaneRng& rng,
                                          const ApproxTables& tab) {
        const uint32_t smp = MULTI ? p / per() : 0u;
        p -= smp * per();
        uint32_t gx, gy, px, py;
        path_pixel(p, bw, gx, gy, px, py);
        if (gx >= a.w || gy >= a.h) return false;
        r.path = p;
        r.smp = smp;
        const int k = (int)(p & 7u);
        float x, y, scale;
        block_coord(a.w, a.h, gx & ~15u, gy & ~3u, (int)((p >> 3) & 7u), k, &x, &y, &scale);
        rng.seed(gx, gy, a.frame + smp, k);
        x = fmaf(unit_from(rng.next()), scale, x);
        y = fmaf(unit_from(rng.next()), scale, y);
        camera_ray(a.cam, x, y, unit_from(rng.next()), tab, o, d);
        return true;
    }
    __device__ __forceinline__ void first_scene(const float4*& nd, const float4*& wd, const float4*& gm) const {
        nd = a.s.nodes;
        wd = a.s.wide;
        gm = a.s.geom;
    }
    __device__ __forceinline__ DeviceScene scene(const PathRef&) const { return a.s; }
    __device__ __forceinline__ bool last(const PathRef& r) const { return !MULTI || r.smp + 1u == a.samples; }
    __device__ __forceinline__ void gbuffer(const PathRef& r, uint32_t word) {
        if (!a.gbuf || !last(r)) return;
        uint32_t gx, gy, px, py;
        path_pixel(r.path, bw, gx, gy, px, py);
        if (px < a.w && py < a.h) a.gbuf[(size_t)py * a.w + px] = word;
    }
    __device__ __forceinline__ void mark_emitter(const PathRef& r) {
        if (!a.gbuf || !last(r)) return;
        atomicOr(a.group_em + (r.path >> 3), 1u << (r.path & 7u));
    }
    __device__ __forceinline__ void store(const PathRef& r, F3 c) {
        uint32_t gx, gy, px, py;
        path_pixel(r.path, bw, gx, gy, px, py);
        if (px >= a.w || py >= a.h) return;
        const size_t idx = (size_t)py * a.w + px;
        if (!last(r)) {
            float* out = a.sample_color + (size_t)3 * a.w * a.h * r.smp + 3 * idx;
            out[0] = c.x;
            out[1] = c.y;
            out[2] = c.z;
            return;
        }
        if (a.rgba) a.rgba[idx] = pack_color(c);
        if (a.color) {
            a.color[3 * idx] = c.x;
            a.color[3 * idx + 1] = c.y;
            a.color[3 * idx + 2] = c.z;
        }
        if (a.accum) {
            a.accum[3 * idx] += c.x;
            a.accum[3 * idx + 1] += c.y;
            a.accum[3 * idx + 2] += c.z;
        }
    }
    __device__ __forceinline__ void count_ray(const PathRef&) { rays++; }
    __device__ __forceinline__ void finish(const PathRef&) { flush_rays(a, rays); }
    __device__ __forceinline__ void work(uint64_t boxes, uint64_t tris, uint64_t shades) {
        unsigned long long v[3] = {boxes, tris, shades};
        for (int k = 0; k < 3; k++) {
            for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
            if ((threadIdx.x & 31u) == 0u && v[k]) atomicAdd(a.work + k, v[k]);
        }
    }
};

// Launch shape and loop form of the per-lane path refill, each measured on the
// room (5k triangles), the 82k-triangle icosphere and the 870k-triangle tube at
// 1280x736: 7 resident blocks per SM (72 registers, no spill; 8 blocks spill
// and lose 2-7 %), and a leaf reached from a pair tested in the same step.
// Trees up to 40 levels: claim threshold 16 and two wide records per round with
// the leaves they lead to tested once, at its end (RefillRay::walk): 82k
// icosphere at 1920x1080 2.02 ms, room 1280x736 0.476 ms (2.79 and 0.70 with
// pairs and leaves tested at once, 2.31 and 0.61 with five pairs per round and
// postponed leaves; three and four records per round 1.99, 2.01 and 0.50, 0.48).
// With pairs: claim 12, 20, 24 icosphere 2.31, 2.41, 2.58 ms, room 0.63, 0.60,
// 0.61; 6 and 8 blocks per SM 2.44, 2.36 and 0.61, 0.65. Deeper trees: below
// (kDeepFrame*).
constexpr int kRefillFrameBlocksPerSm = 7;
constexpr int kRefillFrameSteps = 2;

// COUNT: the same frame, also counting its work (FrameArgs::work); the
// counters cost registers, so frames are rendered without them.
// Deep trees (the DEEP instantiation): claim threshold 12, two wide records per
// round, and the warp's leaves tested together. 870k tube, 1280x736, 16 samples in
// one launch: 23.2 ms (35.7 with pairs and leaves tested at once, 28.7 with four
// pairs per round and postponed leaves, 25.7 with two wide records per round;
// one and three records per round 24.1-25.6, 25.9; claim 8, 14: 23.9, 23.2; 6 and
// 8 resident blocks per SM 24.7 and 23.4); 21.9 with one pop per step, and 21.7
// with the whole stack in local memory as in shallow trees: 16 shared entries per
// lane helped while each push and pop was a branch of its own (4 entries 22.3 ms;
// one sample per launch 1.93 against 1.99 ms).
constexpr int kDeepFrameClaim = 12;
constexpr int kDeepFrameSteps = 2;
// DEEP: a tree deeper than 40 levels (the constants above).
// MULTI: a.samples samples in one launch (FramePaths<true>).
// FORM kPairs: a scene without wide records, and the counting form. Three steps
// per round; deep trees wait for 8 lanes, keep the first 16 stack entries of each
// lane in shared memory and read the tables from global memory (tube, ms per sample:
// local stack 3.07-3.11, 16 entries 2.99; at claim 8 one, two, three, four steps
// 3.15, 2.98, 2.93, 3.07). Icosphere and tube with loose roots, 1280x736: 1.42 and
// 2.92 ms; in the kWide kernel's x86 steps 1.48 and 3.18.
constexpr int kPairFrameSteps = 3, kDeepPairFrameClaim = 8, kDeepPairFrameStack = 16;
template <bool DEEP, bool COUNT, Form FORM, bool MULTI = false>
__global__ void __launch_bounds__(128, kRefillFrameBlocksPerSm) k_render_refill(FrameArgs a) {
    FramePaths<MULTI> P{a, (a.w + 15u) / 16u, (a.h + 3u) / 4u, 0u};
    bool ok;
    if constexpr (FORM == Form::kPairs && DEEP) {
        __shared__ uint2 sstack[4][kDeepPairFrameStack][32];
        ok = path_refill<kDeepPairFrameClaim, kPairFrameSteps, COUNT, FORM, false, kDeepPairFrameStack>(
            P, g_tables, &sstack[threadIdx.x >> 5][0][threadIdx.x & 31]);
    } else {
        __shared__ ApproxTables tab;
        load_tables(tab);
        if constexpr (FORM == Form::kPairs) ok = path_refill<16, kPairFrameSteps, COUNT, FORM>(P, tab);
        else if constexpr (DEEP) ok = path_refill<kDeepFrameClaim, kDeepFrameSteps, COUNT, FORM, true>(P, tab);
        else ok = path_refill<16, kRefillFrameSteps, COUNT, FORM>(P, tab);
    }
    if (!ok) atomicOr(a.err, kErrStackOverflow);
}

template <Form FORM>
static void launch_refill(const FrameArgs& a, uint32_t blocks, cudaStream_t st) {
    const bool deep = a.s.depth > 40;
    if (a.samples > 1) {
        if (deep) k_render_refill<true, false, FORM, true><<<blocks, 128, 0, st>>>(a);
        else k_render_refill<false, false, FORM, true><<<blocks, 128, 0, st>>>(a);
    } else {
        if (deep) k_render_refill<true, false, FORM><<<blocks, 128, 0, st>>>(a);
        else k_render_refill<false, false, FORM><<<blocks, 128, 0, st>>>(a);
    }
}

// Frames in packet traversal, per-group RNG order: an octet holds one 8-pixel
// group at a time and the packets of a warp step together (packet_refill.cuh).
// One group per octet traced to its end (k_render_group) against this, 1280x736:
// room 1.22 -> 1.13 ms, icosphere 3.66 -> 2.75, tube 8.88 -> 6.34; 320x184: room
// 0.65 -> 0.39, icosphere 1.06 -> 0.57 ms. Two wide records per round and 5 blocks
// per SM (80 registers and more, no spill; 6 and 7 blocks: room 1.14, 1.21 ms,
// icosphere 2.77, 2.76 ms, the small one 0.61, 0.64 ms); trees deeper than 40
// levels one record and 6 blocks (6.34 ms; two records 6.81-6.85).
// Scenes without wide records (kPairs), one group per octet against this, us at
// 320x184, 640x368, 900x516, 1280x736, 1920x1080: room with loose roots 608/395,
// 697/528, 809/757, 1210/1362, 2495/2844; icosphere 981/657, 1402/1106, 2019/1823,
// 3610/3316, 7550/6867; tube 3259/2381, 3976/2888, 5609/4292, 8787/7210, 16709/14228;
// the icosphere under a chain of 60 levels 1244/811, 2011/1669, 3063/2875, 5629/5399,
// 11833/11379; the room under one of 80 levels 957/606, 1227/1210, 2052/2130,
// 3888/4058, 8209/8655. Six pairs per round (one to four: 1439, 1402, 1364, 1362 us for
// the room at 1280x736; eight: the same).
constexpr int kPairGroupSteps = 6;
inline bool packets_in_step(const DeviceScene& s, uint32_t pixels) {
    if (s.wide) return true;
    return s.depth < 25u ? pixels <= 600000u : s.depth <= kWideMaxDepth || pixels <= 300000u;
}
template <bool DEEP, Form FORM>
__global__ void __launch_bounds__(128, DEEP ? 6 : 5) k_render_packets(FrameArgs a) {
    __shared__ ApproxTables tab;
    load_tables(tab);
    FramePaths<false> P{a, (a.w + 15u) / 16u, (a.h + 3u) / 4u, 0u};
    bool ok = group_refill<FORM == Form::kPairs ? kPairGroupSteps : DEEP ? 1 : 2, FORM>(P, tab);
    if (!ok) atomicOr(a.err, kErrStackOverflow);
}

// After k_render_refill: a group whose 8 lanes all hit an emitter at bounce 0
// leaves the reference's path loop before its gbuffer values are taken
// (renderer.rs:413-468), so its gbuffer words are 0.
__global__ void __launch_bounds__(256) k_emitter_groups(const uint32_t* __restrict__ mask, uint32_t ngroups,
                                                       uint32_t w, uint32_t h, uint32_t* __restrict__ gbuf) {
    const uint32_t bw = (w + 15u) / 16u;
    for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngroups; gi += gridDim.x * blockDim.x) {
        if (mask[gi] != 0xffu) continue;
        uint32_t gx, gy, px, py;
        path_pixel(gi << 3, bw, gx, gy, px, py);
        for (uint32_t q = 0; q < 8u; q++) {
            uint32_t qx = gx + (q & 3u), qy = gy + (q >> 2);
            if (qx < w && qy < h) gbuf[(size_t)qy * w + qx] = 0u;
        }
    }
}

// After a k_render_refill launch of n > 1 samples: adds each pixel's sample
// colours to the accumulator in sample order (samples 0 .. n - 2 from
// `samples`, the last from the frame's colour buffer). These are the additions
// one launch per frame makes (renderer.rs:339-410 accumulates a frame at a
// time), in the same order, so the accumulator gets the same bits.
__global__ void __launch_bounds__(256) k_accumulate_samples(float* __restrict__ accum,
                                                           const float* __restrict__ samples,
                                                           const float* __restrict__ last, size_t nf, uint32_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nf; i += (size_t)gridDim.x * blockDim.x) {
        float v = accum[i];
        for (uint32_t s = 0; s + 1u < n; s++) v += __ldg(samples + (size_t)s * nf + i);
        accum[i] = v + last[i];
    }
}

// Patch order for single rays, and the debug view (PACKET: of packets; their
// frames take k_render_patch_warp): an octet per patch. One resident block per SM
// is all the launch bound asks: the frame's few hundred chains leave most warp
// slots empty, so registers are free, and with the bound of 128 threads alone the
// compiler capped the kernel at 64 registers and spilled on the chains' critical
// path.
template <bool PACKET>
__global__ void __launch_bounds__(128, 1) k_render_patch(FrameArgs a) {
    __shared__ ApproxTables tab;
    load_tables(tab);
    const int k = threadIdx.x & 7;
    const unsigned omask = 0xffu << (threadIdx.x & 24u);
    const uint32_t pw = (a.w + a.patch - 1u) / a.patch, ph = (a.h + a.patch - 1u) / a.patch;
    const uint32_t n = a.patches ? a.n_patches : pw * ph;
    const uint32_t wb = a.patch / 16u, hb = a.patch / 4u;  // 16x4 blocks across and up a patch
    // One octet per warp: a patch is one long serial chain, so its octet gets a
    // scheduler slot of its own instead of sharing a warp (and diverging) with
    // three other patches, and the few hundred chains of a frame spread over
    // every SM.
    if ((threadIdx.x & 31u) >= 8u) return;
    const uint32_t octets = (gridDim.x * blockDim.x) >> 5;
    uint32_t rays = 0;
    bool ok = true;
    for (uint32_t pi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; pi < n; pi += octets) {
        uint32_t x0 = a.patches ? a.patches[2 * pi] : (pi / ph) * a.patch;
        uint32_t y0 = a.patches ? a.patches[2 * pi + 1] : (pi % ph) * a.patch;
        LaneRng rng;
        rng.seed(x0, y0, a.frame, k);
        for (uint32_t i = 0; i < wb; i++) {
            for (uint32_t j = 0; j < hb; j++) {
                uint32_t xb = x0 + i * 16u, yb = y0 + j * 4u;
                float jx[8], jy[8];
                for (int q = 0; q < 8; q++) jx[q] = unit_from(rng.next());
                for (int q = 0; q < 8; q++) jy[q] = unit_from(rng.next());
#pragma unroll 1
                for (int g = 0; g < 8; g++) {
                    float x, y, scale;
                    block_coord(a.w, a.h, xb, yb, g, k, &x, &y, &scale);
                    x = fmaf(jx[g], scale, x);
                    y = fmaf(jy[g], scale, y);
                    PixelOut p;
                    if (PACKET || a.debug) ok &= render_pixels_debug<PACKET>(a.s, a.cam, x, y, omask, tab, p, rays);
                    else ok &= render_pixels<false>(a.s, a.cam, x, y, rng, omask, tab, p, rays);
                    store_pixel(a, xb + 4u * (uint32_t)(g >> 1) + (uint32_t)(k & 3),
                                yb + 2u * (uint32_t)(g & 1) + (uint32_t)(k >> 2), p);
                }
            }
        }
    }
    if (!ok) atomicOr(a.err, kErrStackOverflow);
    // only the warp's first octet is alive here: reduce over it alone
    unsigned long long v = rays;
    for (int off = 4; off > 0; off >>= 1) v += __shfl_down_sync(0xffu, v, off, 8);
    if (k == 0 && v) atomicAdd(a.rays, v);
}

// Patch order in packet traversal: W warps per patch, one packet per warp
// (packet_warp.cuh). A patch is one chain: a group's generator state depends on
// how many bounces every group before it took. But the generator jumps to any
// state (after n draws it is s * f^n mod 2^64), so the warps of a round render
// the next groups at once, each from the state it has if the groups before it in
// the round take certain bounce counts. What counts is by how often each was met
// so far in the patch (top: the three most frequent): a chain of groups that all take
// the first; two guesses for the first group and a group beyond; or three guesses
// for it, whichever is expected to confirm the most groups. The groups whose
// predecessors took what was guessed are right and are stored; the others are
// rendered again.
//
// The frame's time is that of its slowest patches (the room's slowest takes four
// times the mean): in some nearly every group takes all five bounces (125 of 128), so
// chains hold; in others the counts are mixed, and a round confirms two groups of
// four. Room 1280x736: one octet per patch 16.6 ms, one warp per patch 12.0, a chain
// of four warps as long as the last round's was right 5.57, this 5.46; icosphere
// 26.8, 18.2, 11.6, 10.9 ms; the room at 320x184 (60 patches) 4.61, 4.26. (Two warps
// 7.8 ms, eight 6.5, sixteen 10.5, with chains: idle warps keep other patches' blocks
// off the SM.) 6 blocks of 4 warps per SM hold the frame's 920 patches at once (4, 5,
// 7, 8 blocks with chains: 5.7, 5.6, 5.9, 6.4 and 14.2, 13.6, 13.2, 13.7 ms).
// kPatchChance: 0, 0.18, 0.21 -> 5.58, 5.55, 5.48; 11.08, 10.94, 11.04; 4.31, 4.31,
// 4.29 ms (0.25, 0.35 and 0.5 3, 7 and 15 % slower).
constexpr int kPatchWarps = 4;
constexpr float kPatchChance = 0.2f;
__global__ void __launch_bounds__(32 * kPatchWarps, 24 / kPatchWarps) k_render_patch_warp(FrameArgs a) {
    __shared__ ApproxTables tab;
    __shared__ WarpStack stacks[kPatchWarps];
    __shared__ uint64_t draws[8][8], group_draws[6][8];
    __shared__ int taken[2][kPatchWarps];  // by parity of the round: bounces of each warp's group
    load_tables(tab);
    const uint32_t lane = threadIdx.x & 31u, k = lane & 7u;
    const int wid = (int)(threadIdx.x >> 5);
    const uint32_t ph = (a.h + a.patch - 1u) / a.patch;
    const uint32_t hb = a.patch / 4u, total = a.patch / 16u * hb * 8u;  // 16x4 blocks up a patch, groups of a patch
    const uint32_t pi = blockIdx.x;
    const uint32_t x0 = a.patches ? a.patches[2 * pi] : (pi / ph) * a.patch;
    const uint32_t y0 = a.patches ? a.patches[2 * pi + 1] : (pi % ph) * a.patch;
    LaneRng rng;
    rng.seed(x0, y0, a.frame, (int)k);
    // Powers of this lane's generator factor: 1 draw to 7, and those of a group of t
    // bounces (1 + 6 t draws).
    const uint64_t f = rng.f, f2 = f * f, f4 = f2 * f2, f8 = f4 * f4, f16 = f8 * f8;
    if (threadIdx.x < 8u) {
        uint64_t q = 1;
        for (int i = 0; i < 8; i++, q *= f) draws[i][k] = q;
        q = f;
        for (int t = 0; t < 6; t++, q *= f4 * f2) group_draws[t][k] = q;
    }
    __syncthreads();
    // Confirmed: the state before group `done` (before its block's jitter draws
    // if it is the block's first), and before its block's jitter draws.
    uint64_t state = rng.s, block = rng.s;
    uint32_t done = 0, rays = 0;
    int parity = 0;
    // Lane t < 6: how often t bounces were met (to start with, a guess).
    uint32_t met = lane >= 1u && lane < 6u ? lane == 5u ? 2u : 1u : 0u;
    bool ok = true;
    while (done < total) {
        const float all = (float)__reduce_add_sync(0xffffffffu, met);
        int top[3];
        float p[3];
        uint32_t rest = lane < 6u ? met << 3 | lane : 0u;
        for (int i = 0; i < 3; i++) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, rest);
            top[i] = (int)(m & 7u);
            p[i] = __fdividef((float)(m >> 3), all);
            if (rest == m) rest = 0u;
        }
        // Groups beyond the first expected to be confirmed: chain, two guesses, three.
        const float chain = p[0] + p[0] * p[0] * (1.0f + p[0]), two = p[0] + p[1] + p[0] * p[0], three = p[0] + p[1] + p[2];
        const int guesses = two > chain ? (three > two ? 3 : 2) : (three > chain ? 3 : 1);
        // Warp w renders group done + ahead(w), if the group before it takes last(w)
        // and those before that top[0].
        auto ahead = [&](int w) { return guesses == 1 ? w : guesses == 2 && w == 3 ? 2 : min(w, 1); };
        auto last = [&](int w) { return w < 2 || guesses == 1 || w > guesses ? top[0] : w == 2 ? top[1] : top[2]; };
        // The chance that warp w's group is confirmed; a small one is not worth the
        // issue slots it takes from other patches.
        const float q = wid == 0 ? 1.0f : wid == 1 ? p[0] : guesses == 1 ? (wid == 2 ? p[0] * p[0] : p[0] * p[0] * p[0])
                                : wid == 2 ? p[1] : guesses == 2 ? p[0] * p[0] : p[2];
        const uint32_t mine = done + (uint32_t)ahead(wid);
        PixelOut out;
        uint32_t px = 0, py = 0, r = 0;
        bool fits = true;
        if (lane == 0u) taken[parity][wid] = -1;
        if (mine < total && q >= kPatchChance) {
            uint64_t s = state, b = block;
            for (uint32_t i = done;; i++) {
                if ((i & 7u) == 0u) {
                    b = s;
                    s *= f16;
                }
                if (i == mine) break;
                s *= group_draws[i + 1u == mine ? last(wid) : top[0]][k];
            }
            const int g = (int)(mine & 7u);
            b *= draws[g][k];
            auto draw = [&](uint64_t v) { return unit_from(rng.hi ? (uint32_t)(v >> 32) : (uint32_t)v); };
            const uint32_t xb = x0 + (mine >> 3) / hb * 16u, yb = y0 + (mine >> 3) % hb * 4u;
            float x, y, scale;
            block_coord(a.w, a.h, xb, yb, g, (int)k, &x, &y, &scale);
            x = fmaf(draw(b), scale, x);
            y = fmaf(draw(b * f8), scale, y);
            rng.s = s;
            int bounces;
            fits = render_pixels_warp(a.s, a.cam, x, y, rng, tab, stacks[wid], out, r, bounces);
            px = xb + 4u * (uint32_t)(g >> 1) + (k & 3u);
            py = yb + 2u * (uint32_t)(g & 1) + (k >> 2);
            if (lane == 0u) taken[parity][wid] = bounces;
        }
        __syncthreads();
        // From group to group, by the warp that guessed what the last one took.
        bool firsts = true;  // the groups before the last one took top[0]
        for (int w = 0, d = 1; w >= 0; d++) {
            if (w == wid) {
                ok &= fits;
                if (lane < 8u) {
                    store_pixel(a, px, py, out);
                    rays += r;
                }
            }
            const int t = taken[parity][w];
            if ((done & 7u) == 0u) {
                block = state;
                state *= f16;
            }
            state *= group_draws[t][k];
            if (__any_sync(0xffffffffu, met >= 64u)) met >>= 1;
            met += (int)lane == t;
            w = -1;
            if (++done < total && firsts)
                for (int v = 1; v < kPatchWarps; v++)
                    if (ahead(v) == d && last(v) == t && taken[parity][v] >= 0) w = v;
            firsts &= t == top[0];
        }
        parity ^= 1;
    }
    if (!ok) atomicOr(a.err, kErrStackOverflow);
    flush_rays(a, rays);
}

__global__ void k_resolve(const float* __restrict__ accum, uint32_t npx, float factor, uint32_t* __restrict__ rgba) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < npx; i += gridDim.x * blockDim.x) {
        F3 c = f3(accum[3 * i] * factor, accum[3 * i + 1] * factor, accum[3 * i + 2] * factor);
        rgba[i] = pack_color(c);
    }
}

// ---------------------------------------------------------------------------
// Launchers

// SM count of the calling thread's current device, looked up once per device.
// Threads may call this concurrently and devices may differ in SM count, so
// each device has its own atomic slot (a racing first lookup stores the same
// value twice).
constexpr int kMaxCachedDevices = 64;
static std::atomic<int> g_sm_count[kMaxCachedDevices];
int sm_count() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    if (dev >= 0 && dev < kMaxCachedDevices) {
        const int v = g_sm_count[dev].load(std::memory_order_relaxed);
        if (v > 0) return v;
    }
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        return 1;
    }
    if (dev >= 0 && dev < kMaxCachedDevices) g_sm_count[dev].store(n, std::memory_order_relaxed);
    return n;
}
static int num_sms() { return sm_count(); }

cudaError_t set_stack_limit(int entries) {
    return cudaMemcpyToSymbol(c_stack_limit, &entries, sizeof entries);
}

cudaError_t upload_tables(const uint16_t* rcp, const uint16_t* rsqrt) {
    ApproxTables t;
    for (int i = 0; i < 2048; i++) {
        t.rcp[i] = rcp[i];
        t.rsqrt[i] = rsqrt[i];
    }
    return cudaMemcpyToSymbol(g_tables, &t, sizeof t);
}

cudaError_t launch_prep_geom(const cvx_triangle* tris, uint32_t n, float4* geom, TriShade* shade, cudaStream_t st) {
    uint32_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    if (blocks == 0) blocks = 1;
    k_prep_geom<<<blocks, 256, 0, st>>>(tris, n, geom, shade);
    return cudaGetLastError();
}

cudaError_t launch_prep_wide(const float4* nodes, uint32_t n_pairs, float4* wide, cudaStream_t st) {
    uint32_t blocks = (n_pairs + 127) / 128;
    if (blocks > 4096) blocks = 4096;
    if (blocks == 0) blocks = 1;
    k_prep_wide<<<blocks, 128, 0, st>>>(nodes, n_pairs, wide);
    return cudaGetLastError();
}

cudaError_t launch_prep_lights(const cvx_triangle* tris, const uint32_t* ds, uint32_t n, float4* lights,
                               cudaStream_t st) {
    uint32_t blocks = (n + 127) / 128;
    if (blocks > 1024) blocks = 1024;
    if (blocks == 0) blocks = 1;
    k_prep_lights<<<blocks, 128, 0, st>>>(tris, ds, n, lights);
    return cudaGetLastError();
}

// The select-form query with CLAIM at 8 blocks per SM and `shared` stack
// entries in shared memory (0, 4, 8 or 12).
template <int CLAIM>
static void launch_select_stack(uint32_t shared, uint32_t blocks, const SoaRays& src, uint32_t* err,
                                cudaStream_t st) {
    switch (shared) {
        case 4: k_intersect_refill<8, false, CLAIM, Form::kWide, 4><<<blocks, 128, 0, st>>>(src, err + 1, err); break;
        case 12: k_intersect_refill<8, false, CLAIM, Form::kWide, 12><<<blocks, 128, 0, st>>>(src, err + 1, err); break;
        case 8: k_intersect_refill<8, false, CLAIM, Form::kWide, 8><<<blocks, 128, 0, st>>>(src, err + 1, err); break;
        default: k_intersect_refill<8, false, CLAIM, Form::kWide, 0><<<blocks, 128, 0, st>>>(src, err + 1, err); break;
    }
}

cudaError_t launch_intersect(const DeviceScene& s, const RayCols& rays, uint32_t n, float far_dist, bool packet,
                             float* t_out, int32_t* tri_out, uint32_t* counters, uint32_t* err, uint32_t block,
                             uint32_t blocks_per_sm, cudaStream_t st, uint32_t shared_stack) {
    // Calls that do not fill the GPU several times over: one packet per warp, or
    // one ray per lane, with nothing claimed.
    if (!counters && direct_query(s, n, packet, blocks_per_sm)) {
        if (packet) k_intersect_warp<<<(n + 15u) / 16u, 64, 0, st>>>(s, rays, n, far_dist, t_out, tri_out, err);
        else k_intersect_lanes<<<(n + 31u) / 32u, 32, 0, st>>>(s, rays, n, far_dist, t_out, tri_out, err);
        return cudaGetLastError();
    }
    if (!packet) {
        // persistent ray-refill kernel; err[1] is its ray counter
        cudaError_t e = cudaMemsetAsync(err + 1, 0, 4, st);
        if (e != cudaSuccess) return e;
        uint32_t bps = blocks_per_sm ? blocks_per_sm : 8;
        uint32_t blocks = (uint32_t)num_sms() * bps;
        uint32_t need = (n + 127u) / 128u;
        if (blocks > need) blocks = need;
        SoaRays src{s.nodes, s.wide, s.geom, rays, n, far_dist, t_out, tri_out, counters, s.slab_sel};
        bool deep = s.depth > 40;
        const bool sel = s.slab_sel && !counters;
        if (counters) k_intersect_refill<8, true, 16, Form::kX86><<<blocks, 128, 0, st>>>(src, err + 1, err);
        else if (!sel) {  // x86-form slab test throughout
            if (deep) k_intersect_refill<8, false, 8, Form::kX86><<<blocks, 128, 0, st>>>(src, err + 1, err);
            else k_intersect_refill<8, false, 16, Form::kX86><<<blocks, 128, 0, st>>>(src, err + 1, err);
        } else if (!s.wide) {
            if (deep) k_intersect_refill<8, false, 8, Form::kPairs><<<blocks, 128, 0, st>>>(src, err + 1, err);
            else k_intersect_refill<8, false, 16, Form::kPairs><<<blocks, 128, 0, st>>>(src, err + 1, err);
        } else if (deep) {
            if (bps >= 12) k_intersect_refill<12, false, 8, Form::kWide><<<blocks, 128, 0, st>>>(src, err + 1, err);
            else if (bps >= 10) k_intersect_refill<10, false, 8, Form::kWide><<<blocks, 128, 0, st>>>(src, err + 1, err);
            else launch_select_stack<8>(shared_stack, blocks, src, err, st);
        } else {
            if (bps >= 12) k_intersect_refill<12, false, 16, Form::kWide><<<blocks, 128, 0, st>>>(src, err + 1, err);
            else if (bps >= 10) k_intersect_refill<10, false, 16, Form::kWide><<<blocks, 128, 0, st>>>(src, err + 1, err);
            else launch_select_stack<16>(shared_stack, blocks, src, err, st);
        }
        if (sel) {
            const uint32_t per_block = 256u * kDeferredScan;
            k_intersect_deferred<<<(n + per_block - 1u) / per_block, 256, 0, st>>>(src, err);
        }
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(err + 1, 0, 4, st);  // packet counter
    if (e != cudaSuccess) return e;
    if (!counters && (s.wide || n >= kPairPacketRays)) {
        uint32_t blocks = (uint32_t)num_sms() * (blocks_per_sm ? blocks_per_sm : (uint32_t)kPacketBlocksPerSm),
                 need = (n + 127u) / 128u;
        if (blocks > need) blocks = need;
        SoaRays src{s.nodes, s.wide, s.geom, rays, n, far_dist, t_out, tri_out, nullptr, s.slab_sel};
        if (!s.wide) k_intersect_packets<kPairPacketSteps, Form::kPairs><<<blocks, 128, 0, st>>>(src, err + 1, err);
        else if (s.depth > 40) k_intersect_packets<1, Form::kWide><<<blocks, 128, 0, st>>>(src, err + 1, err);
        else k_intersect_packets<2, Form::kWide><<<blocks, 128, 0, st>>>(src, err + 1, err);
        return cudaGetLastError();
    }
    if (block == 0) block = 128;
    if (blocks_per_sm == 0) blocks_per_sm = 8;
    uint32_t need = ((n + 7u) & ~7u) / block + 1u;
    uint32_t blocks = (uint32_t)num_sms() * blocks_per_sm;
    if (blocks > need) blocks = need;
    if (counters) k_intersect_octets<true><<<blocks, block, 0, st>>>(s, rays, n, far_dist, t_out, tri_out, counters, err);
    else k_intersect_octets<false><<<blocks, block, 0, st>>>(s, rays, n, far_dist, t_out, tri_out, nullptr, err);
    return cudaGetLastError();
}

cudaError_t launch_render(const DeviceScene& s, const DeviceCamera& cam, uint32_t w, uint32_t h, uint32_t frame,
                          bool packet, bool patch_order, uint32_t* rgba, uint32_t* gbuf, float* color, float* accum,
                          unsigned long long* rays, uint32_t* err, uint32_t block, bool debug, cudaStream_t st,
                          uint32_t patch, const uint32_t* patches, uint32_t n_patches, uint32_t* group_em,
                          unsigned long long* work, uint32_t samples, float* sample_color) {
    if (patch == 0) patch = 32;
    if (samples == 0) samples = 1;
    if (samples > 1 && (!accum || !color || !sample_color)) return cudaErrorInvalidValue;
    FrameArgs a{s,      cam,     w,         h,       frame, rgba, gbuf, color, samples > 1 ? nullptr : accum,
                rays,   err,     debug ? 1u : 0u, patch, patches, n_patches, group_em, work, samples, sample_color};
    if (block == 0) block = 128;
    if (group_em && !packet && !patch_order && !debug) {
        uint32_t ngroups = ((w + 15u) / 16u) * ((h + 3u) / 4u) * 8u;
        cudaError_t e = cudaMemsetAsync(group_em, 0, (size_t)ngroups * 4u, st);
        if (e != cudaSuccess) return e;
        uint32_t need = (uint32_t)(((uint64_t)ngroups * 8u * samples + 127u) / 128u),
                 blocks = (uint32_t)num_sms() * kRefillFrameBlocksPerSm;
        if (blocks > need) blocks = need;
        if (work) {
            if (samples > 1) return cudaErrorInvalidValue;
            if (s.depth > 40) k_render_refill<true, true, Form::kPairs><<<blocks, 128, 0, st>>>(a);
            else k_render_refill<false, true, Form::kPairs><<<blocks, 128, 0, st>>>(a);
        } else if (s.wide) {
            launch_refill<Form::kWide>(a, blocks, st);
        } else {
            launch_refill<Form::kPairs>(a, blocks, st);
        }
        if (gbuf) {
            uint32_t fb = (ngroups + 255u) / 256u, cap = (uint32_t)num_sms() * 8u;
            k_emitter_groups<<<fb < cap ? fb : cap, 256, 0, st>>>(group_em, ngroups, w, h, gbuf);
        }
        if (samples > 1 && accum) {
            const size_t nf = (size_t)3 * w * h;
            const uint32_t cap = (uint32_t)num_sms() * 8u;
            const uint32_t fb = (uint32_t)std::min<size_t>((nf + 255u) / 256u, cap);
            k_accumulate_samples<<<fb, 256, 0, st>>>(accum, sample_color, color, nf, samples);
        }
        return cudaGetLastError();
    }
    if (samples != 1) return cudaErrorInvalidValue;
    if (patch_order) {
        uint32_t units = patches ? n_patches : ((w + patch - 1) / patch) * ((h + patch - 1) / patch);
        uint32_t blocks = (units * 32 + block - 1) / block;  // one warp per patch
        if (packet && !debug) k_render_patch_warp<<<units, 32 * kPatchWarps, 0, st>>>(a);
        else if (packet) k_render_patch<true><<<blocks, block, 0, st>>>(a);
        else k_render_patch<false><<<blocks, block, 0, st>>>(a);
    } else {
        uint32_t units = ((w + 15) / 16) * ((h + 3) / 4) * 8;
        uint32_t need = (units * 8 + block - 1) / block;
        uint32_t blocks = (uint32_t)num_sms() * 16u;
        if (blocks > need) blocks = need;
        if (packet && !debug && packets_in_step(s, w * h)) {
            const bool deep = s.wide && s.depth > 40;
            blocks = std::min((uint32_t)num_sms() * ((deep ? 6u : 5u) * 128u / block), need);
            if (!s.wide) k_render_packets<false, Form::kPairs><<<blocks, block, 0, st>>>(a);
            else if (deep) k_render_packets<true, Form::kWide><<<blocks, block, 0, st>>>(a);
            else k_render_packets<false, Form::kWide><<<blocks, block, 0, st>>>(a);
        } else if (packet) k_render_group<true><<<blocks, block, 0, st>>>(a);
        else k_render_group<false><<<blocks, block, 0, st>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_resolve(const float* accum, uint32_t npx, float factor, uint32_t* rgba, cudaStream_t st) {
    uint32_t blocks = (npx + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    if (blocks == 0) blocks = 1;
    k_resolve<<<blocks, 256, 0, st>>>(accum, npx, factor, rgba);
    return cudaGetLastError();
}

}  // namespace cvx
