// One reference packet per warp, for the patch order (renderer.rs:306-362),
// whose groups are one serial chain per patch: what counts is the time of one
// packet, not the rate of many. Lane 8 q + k holds ray k of the packet; all four
// lanes of a ray keep the same ray and hit, and on a wide record lane 8 q + k
// tests the box of slot q, in a leaf every fourth triangle from the q-th.
#pragma once
#include "shade.cuh"
#include "traverse.cuh"

namespace cvx {

// The warp's stack: a node reference and the eight rays' entry distances.
struct WarpStack {
    float t[kStackSlots][8];
    uint32_t ref[kStackSlots];
};

// The decisions are those of traverse<true> (bvh.rs:589-657), by the argument at
// RefillRay::walk taken for each ray; a packet that does not allow the select
// form, or for one step one with an origin on a bound plane, takes the pairs in
// the x86 form. Returns false on a stack overflow. `h` starts at the far
// distance.
__device__ __forceinline__ bool traverse_warp(const DeviceScene& s, F3 o, F3 d, bool active, Hit& h,
                                              const ApproxTables& tab, WarpStack& st) {
    constexpr unsigned kAll = 0xffffffffu;
    const float inf = __int_as_float(0x7f800000);
    const uint32_t lane = threadIdx.x & 31u, k = lane & 7u, q = lane >> 3;
    const F3 inv = f3(x_rcp(d.x, tab), x_rcp(d.y, tab), x_rcp(d.z, tab)), no = f3(-o.x, -o.y, -o.z);
    const bool sel = s.wide && __all_sync(kAll, select_form_ray(o, inv));
    // This slot's planes in the records (WidePlanes): near and far by the signs.
    const uint32_t nx_at = 4u * q + (inv.x > 0.0f ? 0u : 16u), fx_at = 8u * q + 16u - nx_at;
    const uint32_t ny_at = 4u * q + (inv.y > 0.0f ? 64u : 96u), fy_at = 8u * q + 160u - ny_at;
    const uint32_t nz_at = 4u * q + (inv.z > 0.0f ? 48u : 112u), fz_at = 8u * q + 160u - nz_at;
    int sp = 0;
    uint32_t cur = 0;
    for (;;) {
        uint32_t ref = 0;  // the next node, if `have`
        bool have = false, pairs = !sel;
        if (sel) {
            const char* w = reinterpret_cast<const char*>(s.wide) + (size_t)cur * 2;
            auto ld = [](const char* p) { return __ldg(reinterpret_cast<const float*>(p)); };
            const float nx = (ld(w + nx_at) + no.x) * inv.x, fx = (ld(w + fx_at) + no.x) * inv.x;
            const float ny = (ld(w + ny_at) + no.y) * inv.y, fy = (ld(w + fy_at) + no.y) * inv.y;
            const float nz = (ld(w + nz_at) + no.z) * inv.z, fz = (ld(w + fz_at) + no.z) * inv.z;
            const uint32_t r = __float_as_uint(ld(w + 32 + 4u * q));
            const float t = max3(nx, ny, nz), e = min3(fx, fy, fz);
            // Entry distance of the child this slot belongs to, from both its boxes.
            const float tc = max3(fminf(nx, __shfl_xor_sync(kAll, nx, 8)), fminf(ny, __shfl_xor_sync(kAll, ny, 8)),
                                  fminf(nz, __shfl_xor_sync(kAll, nz, 8)));
            const float t_other = __shfl_xor_sync(kAll, t, 8);
            const bool mask = e >= t;
            const float c = mask ? t : inf;
            const unsigned hits = __ballot_sync(kAll, mask & active & (e > 0.0f));
            const unsigned kept = __ballot_sync(kAll, active & (c < h.t));
            pairs = __any_sync(kAll, !(fabsf(t * e * tc) > 0.0f));
            const float tc_other = __shfl_xor_sync(kAll, tc, 16);
            // Slots 0 and 2: the order of their child's boxes; slot 1: of the children.
            const unsigned order = __ballot_sync(kAll, ge0((q & 1u) ? tc - tc_other : t - t_other));
            if (__builtin_expect(!pairs, 1)) {
                const uint32_t in0 = (order & 0xffu) == 0xffu, in1 = (order & 0xff0000u) == 0xff0000u,
                               ch = (order & 0xff00u) == 0xff00u;
                // Rank of this slot's box: 3 is visited first. Ranks 2 and 3 are
                // the boxes of the child visited first (WideT's order).
                const uint32_t rank = ((q >> 1) == ch ? 2u : 0u) + ((q & 1u) == ((q >> 1) ? in1 : in0) ? 1u : 0u);
                const bool vis = (hits >> (8u * q) & 0xffu) && (kept >> (8u * q) & 0xffu);
                // By rank: which boxes are visited (the lanes of a slot agree).
                const unsigned v = __reduce_or_sync(kAll, vis ? 1u << rank : 0u);
                const int top = 31 - __clz((int)v);  // -1: none
                if (vis && (int)rank != top) {
                    const int at = sp + __popc(v & ((1u << rank) - 1u));
                    st.t[at][k] = c;
                    if (k == 0u) st.ref[at] = r;
                }
                ref = __reduce_or_sync(kAll, vis && (int)rank == top ? r : 0u);
                have = v != 0u;
                if (have) sp += __popc(v) - 1;
            }
        }
        if (__builtin_expect(pairs, 0)) {
            const float4* np = reinterpret_cast<const float4*>(reinterpret_cast<const char*>(s.nodes) + cur);
            const float4 q0 = __ldg(np), q1 = __ldg(np + 1), q2 = __ldg(np + 2), q3 = __ldg(np + 3);
            const BoxT b0 = box_test(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o, inv);
            const BoxT b1 = box_test(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o, inv);
            const bool first0 = __all_sync(kAll, !sneg(b0.tmin - b1.tmin));
            const bool hit0 = __any_sync(kAll, b0.mask & active & !sneg(b0.tmax));
            const bool hit1 = __any_sync(kAll, b1.mask & active & !sneg(b1.tmax));
            const float c0 = b0.mask ? b0.tmin : inf, c1 = b1.mask ? b1.tmin : inf;
            const uint32_t r0 = __float_as_uint(q3.x), r1 = __float_as_uint(q3.y);
            auto push = [&](bool v, uint32_t r, float c) {
                if (!v) return;
                if (q == 0u) st.t[sp][k] = c;
                if (lane == 0u) st.ref[sp] = r;
                sp++;
            };
            push(first0 ? hit0 : hit1, first0 ? r0 : r1, first0 ? c0 : c1);
            push(first0 ? hit1 : hit0, first0 ? r1 : r0, first0 ? c1 : c0);
        }
        if (sp > c_stack_limit) return false;
        __syncwarp();
        // Pop until an internal node, testing the leaves on the way.
        for (;;) {
            if (!have) {
                if (sp == 0) return true;
                sp--;
                ref = st.ref[sp];
                if (!__any_sync(kAll, active & !geq(st.t[sp][k], h.t))) continue;
            }
            have = false;
            uint32_t len = ref & 31u, idx = ref >> 5;
            if (len == 0u) break;
            leaf_range(s.nodes, idx, len);
            if (len == 1u) {
                tri_test(s.geom, idx, o, d, active, h);
                continue;
            }
            for (uint32_t b = 0; b < len; b += 4u) {
                Hit g = h;
                g.tri = -1;
                if (b + q < len) tri_test(s.geom, idx + b + q, o, d, active, g);
                // The nearest of the four, the first tested on a tie
                // (triangle.rs:122-147 takes a hit only if it is nearer).
#pragma unroll
                for (int off = 8; off <= 16; off *= 2) {
                    const Hit x{__shfl_xor_sync(kAll, g.t, off), __shfl_xor_sync(kAll, g.u, off),
                                __shfl_xor_sync(kAll, g.v, off), __shfl_xor_sync(kAll, g.tri, off)};
                    if (x.tri >= 0 && (g.tri < 0 || x.t < g.t || (x.t == g.t && x.tri < g.tri))) g = x;
                }
                if (g.tri >= 0) h = g;
            }
        }
        cur = ref;
        __syncwarp();  // the entries popped above may be overwritten now
    }
}

// render_pixels<true> (shade.cuh) with the warp's traversal: the four lanes of a
// ray compute the same values. `bounces`: how often the path was continued (the
// group took 1 + 6 * bounces draws).
__device__ __forceinline__ bool render_pixels_warp(const DeviceScene& s, const DeviceCamera& cam, float x, float y,
                                                   LaneRng& rng, const ApproxTables& tab, WarpStack& st,
                                                   PixelOut& out, uint32_t& rays, int& bounces) {
    constexpr unsigned kAll = 0xffffffffu;
    F3 o, d;
    camera_ray(cam, x, y, unit_from(rng.next()), tab, o, d);
    bool active = true, ok = true;
    F3 color = f3(1.0f, 1.0f, 1.0f);
    uint32_t hit_em = 0u;
    out.tex = 0;
    out.tu = out.tv = out.fresnel = 0.0f;
    int i = 0;
#pragma unroll 1
    for (; i < 5; i++) {
        rays += active ? 1u : 0u;
        Hit h{1.0e5f, 0.0f, 0.0f, -1};
        ok &= traverse_warp(s, o, d, active, h, tab, st);
        const Isect I = make_isect(s, h, o, d, tab);
        hit_em = I.mat;
        if (__all_sync(kAll, (I.mat >> 31) != 0u)) break;
        F3 cm;
        float fr;
        continue_path(s, o, d, active, I, rng, i == 0, tab, cm, fr);
        color = f3(color.x * cm.x, color.y * cm.y, color.z * cm.z);
        if (i == 0) {
            out.tex = ((int32_t)I.mat >> 24) & 3;
            out.tu = I.tu;
            out.tv = I.tv;
            out.fresnel = fr;
        }
    }
    bounces = i;
    const F3 em = sky_intensity(d);
    const F3 c = f3(color.x * em.x, color.y * em.y, color.z * em.z);
    out.color = (hit_em >> 31) ? c : f3(0.0f, 0.0f, 0.0f);
    return ok;
}

}  // namespace cvx
