// Reference packets (8 rays, one octet of a warp) with refill: the packet form
// of the nearest-hit query and of the path loop (renderer.rs:413-468).
//
// A warp holds four packets and steps them together: every vote is one ballot
// of the whole warp from which each octet reads its 8 bits, a packet that is
// finished is replaced while the others go on, and leaves are postponed as in
// RefillRay::walk. (With one packet per octet traced to its end, octets of a
// warp that diverge run their node pairs one after the other, and all wait for
// the longest.) Decisions and their order are the reference's for each packet
// (bvh.rs:589-657); they do not depend on the other packets of the warp.
#pragma once
#include "shade.cuh"
#include "traverse.cuh"

namespace cvx {

constexpr unsigned kFullWarp = 0xffffffffu;

// One packet; each thread is one of its lanes. nodes, geom, sp, cur, leaf and
// the references on the stack are the same in all 8 lanes, distances and hits
// are the lane's own.
struct PacketRay {
    static constexpr uint32_t kNone = RefillRay::kNone;
    const float4* nodes;
    const float4* wide;
    const float4* geom;
    F3 o, d, inv;
    Hit h;
    uint2 top;
    int sp;
    uint32_t cur, leaf;
    float cur_t;  // this lane's entry distance of cur (+inf: outside the box)
    bool active;

    // Votes over the calling lane's octet, as ballots of the whole warp.
    static __device__ __forceinline__ bool any(bool p) {
        return (__ballot_sync(kFullWarp, p) & (0xffu << (threadIdx.x & 24u))) != 0u;
    }
    static __device__ __forceinline__ bool all(bool p) { return !any(!p); }

    __device__ __forceinline__ void clear() {
        o = d = inv = f3(0, 0, 0);
        h = Hit{0.0f, 0.0f, 0.0f, -1};
        top = make_uint2(0u, 0u);
        sp = 0;
        cur = kNone;
        leaf = 0u;
        cur_t = 0.0f;
        active = false;
    }
    __device__ __forceinline__ void start(F3 o_, F3 d_, bool active_, float far, const float4* nodes_,
                                          const float4* wide_, const float4* geom_, const ApproxTables& tab) {
        o = o_;
        d = d_;
        active = active_;
        nodes = nodes_;
        wide = wide_;
        geom = geom_;
        inv = f3(x_rcp(d.x, tab), x_rcp(d.y, tab), x_rcp(d.z, tab));
        h = Hit{far, 0.0f, 0.0f, -1};
        sp = 0;
        cur = 0;  // the root pair
        leaf = 0u;
        cur_t = __int_as_float(0xff800000);
    }

    // One step of each packet that is `on` (the whole warp calls this): at most
    // one pop, and the wide record of its next node (kWide, walking on past one
    // waiting leaf) or that node's pair (a waiting leaf stops the packet).
    template <Form FORM, class Stack>
    __device__ __forceinline__ void walk(bool on, Stack& stack, bool& overflow) {
        constexpr bool kPast = FORM == Form::kWide;
        const bool pop = on && cur == kNone && sp > 0 && (kPast || leaf == 0u);
        const uint2 e = top;
        if (pop) top = stack.load(--sp);
        const bool kept = any(active & !geq(__uint_as_float(e.y), h.t));
        if (pop && kept) {
            if ((e.x & 31u) != 0u && leaf == 0u) {
                leaf = e.x;
            } else {
                cur = e.x;
                cur_t = __uint_as_float(e.y);
            }
        }
        const bool next = on && (cur & 31u) == 0u && (kPast || leaf == 0u);
        if constexpr (FORM == Form::kWide) wide_step(next, stack, overflow);
        else pair_step<FORM == Form::kPairs>(next, stack, overflow);
    }

    // The node pair of each packet with `pair`, in the select form or the x86 form.
    template <bool SELECT, class Stack>
    __device__ __forceinline__ void pair_step(bool pair, Stack& stack, bool& overflow) {
        BoxT b0{0.0f, 0.0f, false}, b1{0.0f, 0.0f, false};
        uint32_t r0 = 0u, r1 = 0u;
        if (pair) {
            const float4* np = reinterpret_cast<const float4*>(reinterpret_cast<const char*>(nodes) + cur);
            const float4 q0 = __ldg(np), q1 = __ldg(np + 1), q2 = __ldg(np + 2), q3 = __ldg(np + 3);
            if constexpr (SELECT) {
                b0 = box_test_sel(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o, inv);
                b1 = box_test_sel(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o, inv);
            } else {
                b0 = box_test(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o, inv);
                b1 = box_test(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o, inv);
            }
            r0 = __float_as_uint(q3.x);
            r1 = __float_as_uint(q3.y);
        }
        const bool first0 = all(!sneg(b0.tmin - b1.tmin));
        const bool hit0 = any(b0.mask & active & !sneg(b0.tmax));
        const bool hit1 = any(b1.mask & active & !sneg(b1.tmax));
        // Lanes outside a box never block a cull (aabb.rs:171-177): +inf.
        const float inf = __int_as_float(0x7f800000);
        const float c0 = b0.mask ? b0.tmin : inf, c1 = b1.mask ? b1.tmin : inf;
        // The reference pushes `first` then `second` and pops `second` first.
        const float t_first = first0 ? c0 : c1, t_second = first0 ? c1 : c0;
        // Either is culled when popped (aabb.rs:171-177), the first too if the second
        // is not visited: then it is next at once.
        const bool kept0 = any(active & !geq(t_first, h.t)), kept1 = any(active & !geq(t_second, h.t));
        if (!pair) return;
        const bool v[2] = {(first0 ? hit0 : hit1) && kept0, (first0 ? hit1 : hit0) && kept1};
        const uint32_t r[2] = {first0 ? r0 : r1, first0 ? r1 : r0};
        const float t[2] = {t_first, t_second};
        push<2>(v, r, t, stack, overflow);
    }

    // The wide record of each packet with `rec`. A box is visited when a lane
    // hits it and a lane enters it before its own hit distance (not necessarily
    // the same lane, bvh.rs:604-651). The visits and their order are those of
    // the pair steps, by the argument at RefillRay::walk taken for each lane. A
    // packet with an origin on a bound plane takes the pair instead.
    template <class Stack>
    __device__ __forceinline__ void wide_step(bool rec, Stack& stack, bool& overflow) {
        const float inf = __int_as_float(0x7f800000);
        const WidePlanes p(wide, rec ? cur : 0u, f3(-o.x, -o.y, -o.z), inv);
        const bool zero = any(p.zero) && rec;
        bool vis[4];
        float c[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool mask = p.e[k] >= p.t[k];
            c[k] = mask ? p.t[k] : inf;
            const bool hit = any(mask & active & (p.e[k] > 0.0f));
            vis[k] = any(active & (c[k] < h.t)) & hit;
        }
        const bool in0 = all(ge0(p.t[0] - p.t[1])), in1 = all(ge0(p.t[2] - p.t[3])), ch = all(ge0(p.tc0 - p.tc1));
        if (__builtin_expect(__any_sync(kFullWarp, zero), 0)) pair_step<false>(zero, stack, overflow);
        if (!rec || zero) return;
        const bool va0 = in0 ? vis[0] : vis[1], va1 = in0 ? vis[1] : vis[0];
        const bool vb0 = in1 ? vis[2] : vis[3], vb1 = in1 ? vis[3] : vis[2];
        const float a0 = in0 ? c[0] : c[1], a1 = in0 ? c[1] : c[0], b0 = in1 ? c[2] : c[3], b1 = in1 ? c[3] : c[2];
        const uint32_t ra0 = in0 ? p.r.x : p.r.y, ra1 = in0 ? p.r.y : p.r.x;
        const uint32_t rb0 = in1 ? p.r.z : p.r.w, rb1 = in1 ? p.r.w : p.r.z;
        const bool v[4] = {ch ? va0 : vb0, ch ? va1 : vb1, ch ? vb0 : va0, ch ? vb1 : va1};
        const float t[4] = {ch ? a0 : b0, ch ? a1 : b1, ch ? b0 : a0, ch ? b1 : a1};
        const uint32_t r[4] = {ch ? ra0 : rb0, ch ? ra1 : rb1, ch ? rb0 : ra0, ch ? rb1 : ra1};
        push<4>(v, r, t, stack, overflow);
    }

    // The boxes to visit, from the last to the first: each becomes the next
    // node, and the one before it is pushed, by selects (as branches, frames: room
    // 1.127 -> 1.119 ms, icosphere 2.76 -> 2.72, 320x184 of it 0.57 -> 0.53). Then a
    // leaf goes to wait, if none does.
    template <int N, class Stack>
    __device__ __forceinline__ void push(const bool (&v)[N], const uint32_t (&r)[N], const float (&t)[N], Stack& stack,
                                         bool& overflow) {
        cur = kNone;
#pragma unroll
        for (int k = 0; k < N; k++) {
            const bool p = k > 0 && v[k] && cur != kNone;
            if (p) stack.store(sp, top);
            top.x = p ? cur : top.x;
            top.y = p ? __float_as_uint(cur_t) : top.y;
            sp += p;
            cur = v[k] ? r[k] : cur;
            cur_t = v[k] ? t[k] : cur_t;
        }
        if (sp > c_stack_limit) {
            overflow = true;
            sp = 0;
            cur = kNone;
            leaf = 0u;
            return;
        }
        if (cur != kNone && (cur & 31u) != 0u && leaf == 0u) {
            leaf = cur;
            cur = kNone;
        }
    }

    // Tests the waiting leaf of each packet that is `on` and has one, and drops
    // `cur` if its hits cull it (the whole warp calls this). Returns true when
    // the packet is finished.
    __device__ __forceinline__ bool test_leaf(bool on) {
        const bool test = on && leaf != 0u;
        if (test) {
            uint32_t len = leaf & 31u, idx = leaf >> 5;
            leaf_range(nodes, idx, len);
#pragma unroll 1
            for (uint32_t i = idx; i < idx + len; i++) tri_test(geom, i, o, d, active, h);
        }
        const bool kept = any(active & !geq(cur_t, h.t));
        if (test) {
            leaf = 0u;
            if (!kept) cur = kNone;
            if (cur != kNone && (cur & 31u) != 0u) {  // the second leaf is next
                leaf = cur;
                cur = kNone;
            }
        }
        return cur == kNone && sp == 0 && leaf == 0u;
    }
    // One round of the warp: STEPS wide records of each packet, with the leaves
    // they lead to tested once (kWide), or STEPS pairs with each leaf tested at
    // once (kPairs); in the x86 form unless every packet `on` allows FORM (sel).
    // Returns true when the packet is finished.
    template <int STEPS, Form FORM, class Stack>
    __device__ __forceinline__ bool round(bool on, bool sel, Stack& stack, bool& overflow) {
        bool fin = false;
        if (!__any_sync(kFullWarp, on)) return false;  // (and then there may be no wide records)
        if (__all_sync(kFullWarp, !on || sel)) {
            if constexpr (FORM == Form::kWide) {
#pragma unroll 1
                for (int st = 0; st < STEPS; st++) walk<Form::kWide>(on, stack, overflow);
                fin = test_leaf(on);
                // Two records may lead to two leaves, of which the second stopped its packet:
                // tested now instead of after the next round (1M packets: room 311 -> 299
                // us, icosphere 632 -> 620; frames -0.6 and -1 %). With one record per round a
                // second test costs 1.5 %.
                if (STEPS > 1 && __any_sync(kFullWarp, on && leaf != 0u)) fin = test_leaf(on);
            } else {
                pairs<STEPS, FORM>(on, fin, stack, overflow);
            }
        } else {
            pairs<STEPS, Form::kX86>(on, fin, stack, overflow);
        }
        return fin;
    }
    template <int STEPS, Form FORM, class Stack>
    __device__ __forceinline__ void pairs(bool on, bool& fin, Stack& stack, bool& overflow) {
#pragma unroll 1
        for (int st = 0; st < STEPS; st++) {
            walk<FORM>(on && !fin, stack, overflow);
            fin = test_leaf(on && !fin);
        }
    }
    // Whether the packet, whose lanes call this with the rest of the warp, allows FORM.
    template <Form FORM>
    __device__ __forceinline__ bool allows(bool scene_allows) const {
        return all(form_allows<FORM>(o, inv)) && scene_allows;
    }
};

// The nearest-hit query over the packets of `claim` (which hands an octet 8
// consecutive rays; src as in traverse_refill, with one scene). A finished packet
// is replaced at once. The lanes of a last, partial packet beyond its rays are
// inactive copies of its first lane's ray.
template <int STEPS, Form FORM, class Src, class Claim>
__device__ __forceinline__ bool traverse_packets(const Src& src, Claim& claim, const ApproxTables& tab) {
    const int lane = threadIdx.x & 31;
    PacketRay ray;
    ray.clear();
    src.first_scene(ray.nodes, ray.wide, ray.geom);
    uint2 local_stack[kStackSlots];
    LocalStack stack{local_stack};
    uint32_t r_id = 0;
    bool have = false, done = false, sel = false, overflow = false;
    for (;;) {
        const bool want = !have && !done;
        const unsigned b = __ballot_sync(kFullWarp, want);
        if (b) {
            uint32_t r = 0;
            RayIn in{f3(0, 0, 0), f3(0, 0, 0), 0.0f, nullptr, nullptr, nullptr};
            const int got = claim.claim(b, want, lane, r, in);
            const unsigned rays = __ballot_sync(kFullWarp, want && got == kClaimRay);
            const bool any = ((rays >> (lane & 24)) & 0xffu) != 0u;
            const int l0 = lane & 24;
            const F3 o0 = f3(__shfl_sync(kFullWarp, in.o.x, l0), __shfl_sync(kFullWarp, in.o.y, l0),
                             __shfl_sync(kFullWarp, in.o.z, l0));
            const F3 d0 = f3(__shfl_sync(kFullWarp, in.d.x, l0), __shfl_sync(kFullWarp, in.d.y, l0),
                             __shfl_sync(kFullWarp, in.d.z, l0));
            if (want) {
                done = !any;
                have = any;
                if (any) {
                    const bool mine = got == kClaimRay;
                    r_id = r;
                    ray.start(mine ? in.o : o0, mine ? in.d : d0, mine, src.far_dist, src.nodes, src.wide, src.geom, tab);
                }
            }
            const bool all_sel = ray.allows<FORM>(FORM == Form::kWide ? src.wide != nullptr : src.slab_sel != 0u);
            if (want) sel = all_sel;
        }
        if (__all_sync(kFullWarp, done)) break;
        if (ray.round<STEPS, FORM>(have, sel, stack, overflow) && have) {
            if (ray.active) src.store(r_id, ray.h, 0u, 0u);
            have = false;
        }
    }
    return !overflow;
}

// The path loop for packets: an octet holds one 8-pixel group at a time. A group
// that has finished its packet is shaded: the hit records, the octet's
// all-emissive vote, the next bounce's packet, or the pixels' stores and a new
// group. (Waiting until two groups of the warp are to be shaded costs more than
// it saves: icosphere 2.77 -> 2.97 ms, tube 6.81 -> 7.57 ms.) Paths: as in
// path_refill, path numbers being claimed 8 at a time (a group's lanes);
// mark_emitter is not used.
template <int STEPS, Form FORM, class Paths>
__device__ __forceinline__ bool group_refill(Paths& P, const ApproxTables& tab) {
    typedef typename Paths::PathRef PathRef;
    const int lane = threadIdx.x & 31;
    const unsigned omask = 0xffu << (lane & 24);
    const uint32_t npaths = P.n_paths();
    PacketRay ray;
    ray.clear();
    P.first_scene(ray.nodes, ray.wide, ray.geom);
    uint2 local_stack[kStackSlots];
    LocalStack stack{local_stack};
    LaneRng rng;
    rng.s = rng.f = 0ull;
    rng.hi = 0u;
    PathRef ref{};
    F3 color = f3(1.0f, 1.0f, 1.0f);
    uint32_t bounce = 0;
    bool tracing = false, has_group = false, done = false, sel = false, overflow = false;
    for (;;) {
        const bool want = !tracing && !done;
        bool started = false;
        if (want && has_group) {
            const DeviceScene s = P.scene(ref);
            const Isect I = make_isect(s, ray.h, ray.o, ray.d, tab);
            const bool em = (I.mat >> 31) != 0u;
            const bool all_em = oct_all(omask, em);
            if (all_em || bounce == 4u) {
                // (At bounce 4 the reference still continues the path, which
                // changes neither an emitter lane's colour nor the others' black.)
                if (bounce == 0u) P.gbuffer(ref, 0u);
                const F3 sky = sky_intensity(ray.d);
                P.store(ref, em ? f3(color.x * sky.x, color.y * sky.y, color.z * sky.z) : f3(0.0f, 0.0f, 0.0f));
                has_group = false;
            } else {
                F3 o = ray.o, d = ray.d, cm;
                bool active = ray.active;
                float fr;
                continue_path(s, o, d, active, I, rng, bounce == 0u, tab, cm, fr);
                color = f3(color.x * cm.x, color.y * cm.y, color.z * cm.z);
                if (bounce == 0u) {
                    PixelOut g0;
                    g0.tex = ((int32_t)I.mat >> 24) & 3;
                    g0.tu = I.tu;
                    g0.tv = I.tv;
                    g0.fresnel = fr;
                    P.gbuffer(ref, pack_gbuffer(g0));
                }
                bounce++;
                ray.start(o, d, active, 1.0e5f, s.nodes, s.wide, s.geom, tab);
                started = true;
                if (active) P.count_ray(ref);
            }
        }
        // Octets without a group take the next ones (one atomic per warp).
        const bool need = want && !has_group;
        const unsigned nb = __ballot_sync(kFullWarp, need);
        if (nb) {
            uint32_t base = 0;
            const int first = __ffs(nb) - 1;
            if (lane == first) base = P.claim((uint32_t)__popc(nb));
            base = __shfl_sync(kFullWarp, base, first);
            if (need) {
                const uint32_t p = base + (uint32_t)__popc(nb & ((1u << lane) - 1u));
                if (p >= npaths) {
                    done = true;
                } else {
                    F3 o, d;
                    if (P.begin(p, ref, o, d, rng, tab)) {  // else: a group outside its image; take another
                        const DeviceScene s = P.scene(ref);
                        ray.start(o, d, true, 1.0e5f, s.nodes, s.wide, s.geom, tab);
                        color = f3(1.0f, 1.0f, 1.0f);
                        bounce = 0u;
                        has_group = true;
                        started = true;
                        P.count_ray(ref);
                    }
                }
            }
        }
        if (__all_sync(kFullWarp, done)) break;
        if (__any_sync(kFullWarp, started)) {
            const bool all_sel = ray.allows<FORM>(true);
            if (started) {
                const DeviceScene s = P.scene(ref);
                sel = all_sel && (FORM == Form::kWide ? s.wide != nullptr : s.slab_sel != 0u);
                tracing = true;
            }
        }
        if (ray.round<STEPS, FORM>(tracing, sel, stack, overflow)) tracing = false;
    }
    P.finish(ref);
    return !overflow;
}

}  // namespace cvx
