// Nearest-hit BVH traversal (bvh.rs:589-657) with the reference's box test
// (aabb.rs:105-141) and triangle test (triangle.rs:59-148), bit-exact.
//
// Two variants share the arithmetic:
//  * PACKET: the 8 threads of an octet (lanes 8k..8k+7 of a warp) are one
//    reference ray packet. Every decision the reference takes over the packet
//    (child order by should_try_before, push by any_masked, cull by
//    is_further_away_than) is a warp vote over the octet, so all 8 threads walk
//    the same node sequence as the reference's packet, node fetches are
//    broadcast loads, and the result is the reference's lane for lane.
//  * SINGLE: each thread walks its own ray with the same decisions taken over
//    itself alone. Results equal the packet traversal except where two
//    triangles tie in t, or where the approximate-reciprocal box test is not
//    conservative for a grazing ray.
#pragma once
#include <type_traits>

#include "layout.cuh"
#include "x86sem.cuh"

namespace cvx {

// Stack entries a traversal may hold before it reports kErrStackOverflow:
// kStackDepth, unless lowered to test that error path
// (cvx_set_traversal_stack_limit). Every stack array keeps kStackDepth
// entries, so any limit up to that keeps all accesses in bounds. Each
// translation unit that traverses has its own copy; set_stack_limit (in
// kernels.cu and wavefront.cu) writes each.
static __constant__ int c_stack_limit = kStackDepth;

struct Hit {
    float t, u, v;
    int32_t tri;
};

struct BoxT {
    float tmin, tmax;
    bool mask;
};

__device__ __forceinline__ BoxT box_test(float lx, float ly, float lz, float hx, float hy, float hz, F3 o, F3 inv) {
    float tx1 = (lx - o.x) * inv.x, tx2 = (hx - o.x) * inv.x;
    float ty1 = (ly - o.y) * inv.y, ty2 = (hy - o.y) * inv.y;
    float tz1 = (lz - o.z) * inv.z, tz2 = (hz - o.z) * inv.z;
    float tmin = xmax(xmin(tx1, tx2), xmax(xmin(ty1, ty2), xmin(tz1, tz2)));
    float tmax = xmin(xmax(tx1, tx2), xmin(xmax(ty1, ty2), xmax(tz1, tz2)));
    return BoxT{tmin, tmax, geq(tmax, tmin)};
}

// The slab test in select form: the near and far plane of each axis are
// picked by the sign of the ray's reciprocal instead of by the x86 min/max of
// the two plane distances (one select for each compare-and-select). It gives
// the bits of box_test when every bound is finite, lo <= hi and no bound is -0
// (DeviceScene::slab_sel), and the reciprocals are finite with |1/d| >= 0.75
// (select_form_recip). With a positive reciprocal, rounding keeps
// (lo - o) / d <= (hi - o) / d; x86 min takes the first and max the second, and
// on equal values the second, which then has the same bits: a zero difference
// is +0 without -0 bounds, and a non-zero one does not round to a zero at
// |1/d| >= 0.75. A negative reciprocal swaps the two.
__device__ __forceinline__ BoxT box_test_sel(float lx, float ly, float lz, float hx, float hy, float hz, F3 o,
                                             F3 inv) {
    const bool px = inv.x > 0.0f, py = inv.y > 0.0f, pz = inv.z > 0.0f;
    float tx1 = (lx - o.x) * inv.x, tx2 = (hx - o.x) * inv.x;
    float ty1 = (ly - o.y) * inv.y, ty2 = (hy - o.y) * inv.y;
    float tz1 = (lz - o.z) * inv.z, tz2 = (hz - o.z) * inv.z;
    float nx = px ? tx1 : tx2, fx = px ? tx2 : tx1;
    float ny = py ? ty1 : ty2, fy = py ? ty2 : ty1;
    float nz = pz ? tz1 : tz2, fz = pz ? tz2 : tz1;
    float tmin = xmax(nx, xmax(ny, nz));
    float tmax = xmin(fx, xmin(fy, fz));
    return BoxT{tmin, tmax, geq(tmax, tmin)};
}

// The wide record of a node pair, 128 B (8 x 16 B): the boxes of the pair's
// grandchildren, slots 0 and 1 the children of the pair's first node, 2 and 3 of
// its second. A node that is a leaf takes its first slot itself and leaves the
// other one empty (lo kEmptyLo, hi -kEmptyLo: never hit). w[0], w[4], w[3]: lo of
// the four slots on the x, y and z axis; w[1], w[6], w[7]: hi; w[2]: their
// references (the same as in the pair records: an internal node is its child
// pair, whose wide record is at 128 bytes times the pair's index); w[5]: unused.
// Lo and hi of an axis differ in one bit of their place, another for each axis,
// so that a plane's 32-bit offset is the record's and one bit of the ray's sign.
// With lo and hi side by side and 64-bit addresses: patch frame 5.68 -> 5.56 ms,
// 1M packets 315 -> 310 us, 1M tube rays 427 -> 419 us, the rest 0 to 1 %.
constexpr float kEmptyLo = 1.0e30f;

// A difference of two distances that is not negative (no NaN matters here).
__device__ __forceinline__ bool ge0(float x) { return (int32_t)fb(x) >= 0; }

// sm_100's three-operand minimum and maximum.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// A ray against a wide record in select form: the near and far plane of each
// axis are picked by the sign of the ray's reciprocal (box_test_sel), by address,
// so that no select is spent on them, and the four boxes' distances to them take
// two planes per instruction (packed FP32, sm_100; the negated origin `no` is
// added, which is the same operation). t, e: entry and exit distance of each
// slot's box; tc: entry distances of the pair's own two boxes.
//
// The axes are joined by max3 and min3. They differ from the x86 min and max
// only where the result is a zero (of two tied zeros x86 takes the later
// operand, max3 +0 and min3 -0); and where no exit distance is zero, a ray that
// hits a grandchild's box hits the child's. `zero` is set where one of the results
// is zero (an origin on a bound plane; rare): the step is then to be decided from
// the pair records in the x86 form. The products of the results show it (0, or
// NaN from inf * 0; an underflow only costs time).
struct WidePlanes {
    float t[4], e[4], tc0, tc1;
    uint4 r;
    bool zero;
    __device__ __forceinline__ WidePlanes(const float4* __restrict__ wide, uint32_t ref, F3 no, F3 inv) {
        const char* base = reinterpret_cast<const char*>(wide);
        auto ld = [&](uint32_t at) { return __ldg(reinterpret_cast<const float4*>(base + at)); };
        const uint32_t w = ref * 2u, sx = fb(inv.x) >> 27 & 16u, sy = fb(inv.y) >> 26 & 32u, sz = fb(inv.z) >> 25 & 64u;
        const uint32_t nx_at = w | sx, ny_at = w | sy, nz_at = w | sz;
        const float4 nx4 = ld(nx_at), fx4 = ld(nx_at ^ 16u), ny4 = ld(ny_at + 64u), fy4 = ld((ny_at ^ 32u) + 64u),
                     nz4 = ld(nz_at + 48u), fz4 = ld((nz_at ^ 64u) + 48u);
        r = __ldg(reinterpret_cast<const uint4*>(base + w + 32u));
        auto dist = [](float4 v, float n, float i, float* out) {
            const float2 n2 = make_float2(n, n), i2 = make_float2(i, i);
            const float2 a = __fmul2_rn(__fadd2_rn(make_float2(v.x, v.y), n2), i2);
            const float2 b = __fmul2_rn(__fadd2_rn(make_float2(v.z, v.w), n2), i2);
            out[0] = a.x;
            out[1] = a.y;
            out[2] = b.x;
            out[3] = b.y;
        };
        float nx[4], ny[4], nz[4], fx[4], fy[4], fz[4];
        dist(nx4, no.x, inv.x, nx);
        dist(ny4, no.y, inv.y, ny);
        dist(nz4, no.z, inv.z, nz);
        dist(fx4, no.x, inv.x, fx);
        dist(fy4, no.y, inv.y, fy);
        dist(fz4, no.z, inv.z, fz);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            t[k] = max3(nx[k], ny[k], nz[k]);
            e[k] = min3(fx[k], fy[k], fz[k]);
        }
        tc0 = max3(fminf(nx[0], nx[1]), fminf(ny[0], ny[1]), fminf(nz[0], nz[1]));
        tc1 = max3(fminf(nx[2], nx[3]), fminf(ny[2], ny[3]), fminf(nz[2], nz[3]));
        const float p0 = (t[0] * e[0]) * (t[1] * e[1]) * tc0, p1 = (t[2] * e[2]) * (t[3] * e[3]) * tc1;
        zero = !(fabsf(p0) > 0.0f && fabsf(p1) > 0.0f);
    }
};
// The decisions of one ray on a wide record. t: entry distance of each slot's box
// if it is hit, +inf if not.
struct WideT {
    float t[4], tc0, tc1;
    uint4 r;
    __device__ __forceinline__ WideT(const float4* __restrict__ nodes, const float4* __restrict__ wide, uint32_t ref,
                                     F3 no, F3 inv) {
        const WidePlanes p(wide, ref, no, inv);
        r = p.r;
        if (__builtin_expect(p.zero, 0)) {
            exact(nodes, ref, f3(-no.x, -no.y, -no.z), inv);
        } else {
            const float inf = __int_as_float(0x7f800000);
            tc0 = p.tc0;
            tc1 = p.tc1;
#pragma unroll
            for (int k = 0; k < 4; k++) t[k] = (p.e[k] >= p.t[k]) & (p.e[k] > 0.0f) ? p.t[k] : inf;
        }
    }
    // This step from the pair records: the pair's boxes, then those of its
    // children that are hit.
    __device__ __forceinline__ void exact(const float4* __restrict__ nodes, uint32_t ref, F3 o, F3 inv) {
        const float inf = __int_as_float(0x7f800000);
#pragma unroll
        for (int k = 0; k < 4; k++) t[k] = inf;
        BoxT b[2], c[2];
        uint32_t br[2], cr[2];
        pair(nodes, ref, o, inv, b, br);
        tc0 = b[0].tmin;
        tc1 = b[1].tmin;
        if (hit(b[0])) {
            if ((br[0] & 31u) != 0u) {
                t[0] = tc0;
            } else {
                pair(nodes, br[0], o, inv, c, cr);
                if (hit(c[0])) t[0] = c[0].tmin;
                if (hit(c[1])) t[1] = c[1].tmin;
            }
        }
        if (hit(b[1])) {
            if ((br[1] & 31u) != 0u) {
                t[2] = tc1;
            } else {
                pair(nodes, br[1], o, inv, c, cr);
                if (hit(c[0])) t[2] = c[0].tmin;
                if (hit(c[1])) t[3] = c[1].tmin;
            }
        }
    }
    static __device__ __forceinline__ bool hit(const BoxT& b) { return b.mask & !sneg(b.tmax); }
    static __device__ __forceinline__ void pair(const float4* __restrict__ nodes, uint32_t ref, F3 o, F3 inv, BoxT* b,
                                                uint32_t* r) {
        const float4* np = reinterpret_cast<const float4*>(reinterpret_cast<const char*>(nodes) + ref);
        const float4 q0 = __ldg(np), q1 = __ldg(np + 1), q2 = __ldg(np + 2), q3 = __ldg(np + 3);
        b[0] = box_test(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o, inv);
        b[1] = box_test(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o, inv);
        r[0] = __float_as_uint(q3.x);
        r[1] = __float_as_uint(q3.y);
    }
};

// Rays that may take the select form on the pair records: reciprocals as at
// box_test_sel.
__device__ __forceinline__ bool select_form_recip(F3 inv) {
    return isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z) && fabsf(inv.x) >= 0.75f &&
           fabsf(inv.y) >= 0.75f && fabsf(inv.z) >= 0.75f;
}
// And on the wide records: reciprocals and origin bounded too (as the bounds are,
// TreeFacts::wide), so that no plane distance overflows.
__device__ __forceinline__ bool select_form_ray(F3 o, F3 inv) {
    auto in = [](float x) { return fabsf(x) >= 0.75f && fabsf(x) <= kSelectMax; };
    return in(inv.x) && in(inv.y) && in(inv.z) && fabsf(o.x) <= kSelectMax && fabsf(o.y) <= kSelectMax &&
           fabsf(o.z) <= kSelectMax;
}

// One triangle against one ray: `in` when the reference's tests that do not look
// at the nearest hit so far pass (triangle.rs:122-147).
struct TriT {
    float t, u, v;
    bool in;
};
__device__ __forceinline__ TriT tri_eval(const float4* __restrict__ geom, uint32_t i, F3 o, F3 d) {
    float4 A = __ldg(geom + 3 * i), B = __ldg(geom + 3 * i + 1), C = __ldg(geom + 3 * i + 2);
    F3 v0 = f3(A.x, A.y, A.z), e1 = f3(B.x, B.y, B.z), e2 = f3(C.x, C.y, C.z), n = f3(A.w, B.w, C.w);
    F3 fr = sub(v0, o);
    float denom = 1.0f / dot(d, n);
    float t = dot(fr, n) * denom;
    F3 c = cross(d, fr);
    float u = dot(c, e2) * denom;
    float v = dot(c, e1) * denom;
    float w = (1.0f - u) - v;
    return TriT{t, u, v, !(sneg(t) | sneg(u) | sneg(v) | sneg(w))};
}

// The same; updates the hit when the reference would pick the new
// intersection.
__device__ __forceinline__ void tri_test(const float4* __restrict__ geom, uint32_t i, F3 o, F3 d, bool active,
                                         Hit& h) {
    const TriT x = tri_eval(geom, i, o, d);
    bool reject = !x.in | !active | geq(x.t, h.t);
    if (!reject) {
        h.t = x.t;
        h.u = x.u;
        h.v = x.v;
        h.tri = (int32_t)i;
    }
}

// Node references: the two children's entries in a node pair's last float4
// (q3.x, q3.y), as the scene upload writes them and the traversal stacks hold
// them. (index << 5) | len: len 0 is an internal node (index = its first
// child), len 1..30 a leaf of len triangles at index; len 31 escapes larger
// leaves, index being the slot of their (index, len) in the float4 at
// nodes[-1 - slot]. Indices are below 2^27 (checked at scene creation).
// The escape is marked unlikely: as an ordinary branch in the packet
// traversal's pop loop it made that traversal up to 1.6x slower, even never
// taken (with the hint, and the stack holding references, the room frame runs
// 0.823 against 0.840 ms with (index, len) pairs on the stack).
__device__ __forceinline__ void leaf_range(const float4* __restrict__ nodes, uint32_t& idx, uint32_t& len) {
    if (__builtin_expect(len == 31u, 0)) {
        const float4 e = __ldg(nodes - 1 - (size_t)idx);
        idx = __float_as_uint(e.x);
        len = __float_as_uint(e.y);
    }
}

__device__ __forceinline__ bool oct_all(unsigned m, bool p) { return (__ballot_sync(m, p) & m) == m; }
__device__ __forceinline__ bool oct_any(unsigned m, bool p) { return (__ballot_sync(m, p) & m) != 0u; }

struct Counters {
    uint32_t aabb, tri;
};

// omask: the octet's lanes in the warp (PACKET) or the calling lane (SINGLE).
// In SINGLE mode an inactive lane must not call this. Returns false on stack
// overflow (the hit is then incomplete). SELECT: the select-form slab test
// (box_test_sel), for a scene with DeviceScene::slab_sel and rays whose
// reciprocals meet select_form_recip (in PACKET mode: all 8 lanes').
template <bool PACKET, bool SELECT = false>
__device__ __forceinline__ bool traverse(const DeviceScene& s, F3 o, F3 d, bool active, unsigned omask, Hit& h,
                                         const ApproxTables& tab, Counters* cnt) {
    F3 inv = f3(x_rcp(d.x, tab), x_rcp(d.y, tab), x_rcp(d.z, tab));
    uint32_t st_ref[kStackDepth];  // node references (leaf_range)
    float st_t[kStackDepth];
    int sp = 0;
    uint32_t na = 2, nt = 0;
    bool ok = true;

    uint32_t pair = 0;
    for (;;) {
        // Test the two children of a pair and push them in the reference order.
        const float4* np = s.nodes + 4 * pair;
        float4 q0 = __ldg(np), q1 = __ldg(np + 1), q2 = __ldg(np + 2), q3 = __ldg(np + 3);
        BoxT b0, b1;
        if constexpr (SELECT) {
            b0 = box_test_sel(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o, inv);
            b1 = box_test_sel(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o, inv);
        } else {
            b0 = box_test(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o, inv);
            b1 = box_test(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o, inv);
        }
        bool first0 = !sneg(b0.tmin - b1.tmin);
        bool hit0 = b0.mask & active & !sneg(b0.tmax);
        bool hit1 = b1.mask & active & !sneg(b1.tmax);
        if (PACKET) {
            first0 = oct_all(omask, first0);
            hit0 = oct_any(omask, hit0);
            hit1 = oct_any(omask, hit1);
        }
        // Lanes outside the box never block a cull (aabb.rs:171-177): +inf.
        float c0 = b0.mask ? b0.tmin : __int_as_float(0x7f800000);
        float c1 = b1.mask ? b1.tmin : __int_as_float(0x7f800000);
        const uint32_t r0 = __float_as_uint(q3.x), r1 = __float_as_uint(q3.y);
        int need = (int)hit0 + (int)hit1;
        if (sp + need > c_stack_limit) {
            ok = false;
            break;
        }
        if (first0) {
            if (hit0) { st_ref[sp] = r0; st_t[sp] = c0; sp++; }
            if (hit1) { st_ref[sp] = r1; st_t[sp] = c1; sp++; }
        } else {
            if (hit1) { st_ref[sp] = r1; st_t[sp] = c1; sp++; }
            if (hit0) { st_ref[sp] = r0; st_t[sp] = c0; sp++; }
        }
        // Pop until an internal node whose children must be tested.
        bool descend = false;
        while (sp > 0) {
            sp--;
            uint32_t idx = st_ref[sp] >> 5, len = st_ref[sp] & 31u;
            bool skip = !active | geq(st_t[sp], h.t);
            if (PACKET) skip = oct_all(omask, skip);
            if (skip) continue;
            if (len == 0u) {
                na += 2;
                pair = idx >> 1;
                descend = true;
                break;
            }
            leaf_range(s.nodes, idx, len);
            for (uint32_t i = idx; i < idx + len; i++) tri_test(s.geom, i, o, d, active, h);
            nt += len;
        }
        if (!descend) break;
    }
    if (cnt) {
        cnt->aabb = na;
        cnt->tri = nt;
    }
    return ok;
}

// Asynchronous global-to-shared copies (cp.async) for staging rays.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(__cvta_generic_to_global(gmem)));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_one_pending() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Ray supply of the refill traversal. claim() is called by the whole warp in
// an iteration in which the lanes of `b` want a ray; for a wanting lane it
// returns kClaimRay with the ray's data, kClaimDone when the rays are used up,
// or kClaimNone when the ray it took needs no tracing (the source then stored
// that ray's result itself).
enum : int { kClaimNone = 0, kClaimRay = 1, kClaimDone = 2 };

// How a refill traversal tests boxes: node pairs with the x86 slab test, node
// pairs with the select form (for scenes with DeviceScene::slab_sel), or wide
// records (for scenes that have them). The last two leave a ray that does not
// meet select_form_recip or select_form_ray to the first.
enum class Form { kX86, kPairs, kWide };
template <Form FORM>
__device__ __forceinline__ bool form_allows(F3 o, F3 inv) {
    return FORM == Form::kWide ? select_form_ray(o, inv) : FORM == Form::kPairs ? select_form_recip(inv) : true;
}

struct RayIn {
    F3 o, d;
    float far;
    const float4* nodes;
    const float4* wide;  // Form::kWide only
    const float4* geom;
};

// A refill traversal's stack: entry 0 is a spare (what `top` holds while the
// stack is empty is stored there and never used, which saves a test per push
// and pop), and a wide step may push three entries before it checks the limit.
constexpr int kStackSlots = kStackDepth + 4;

// Where a refill traversal keeps the stack entries below its top. LocalStack:
// a local array. SharedLocalStack<N>: the first N entries in shared memory,
// in this lane's column of a warp's [N][32] block (no bank conflicts, and pops
// of those never miss the cache), the deeper ones in the local array.
struct LocalStack {
    uint2 (&a)[kStackSlots];
    __device__ __forceinline__ uint2 load(int i) const { return a[i]; }
    __device__ __forceinline__ void store(int i, uint2 v) { a[i] = v; }
};
template <int N>
struct SharedLocalStack {
    uint2* sm;  // entry i at sm[32 * i]
    uint2 (&a)[kStackSlots];
    __device__ __forceinline__ uint2 load(int i) const { return i < N ? sm[32 * i] : a[i]; }
    __device__ __forceinline__ void store(int i, uint2 v) {
        if (i < N) sm[32 * i] = v;
        else a[i] = v;
    }
};

// One lane's single-ray traversal in the refill form. step() does one
// iteration: one node pair (and, LEAF_AFTER_PAIR, the leaf it leads to) or one
// leaf. Decisions and their order are exactly those of traverse<false>: after a
// pair test the child the reference would pop next is processed at once (its
// cull test sees the same hit distance the pop would), the other one is
// pushed, and culled entries are popped within the same iteration.
struct RefillRay {
    static constexpr uint32_t kNone = 0xffffffffu;
    const float4* nodes;
    const float4* wide;
    const float4* geom;
    F3 no, d, inv;  // no: the negated origin
    Hit h;
    // The stack holds (ref, entry distance bits) entries. Its top entry lives
    // in `top`, the entries below it in the caller's local array: a pop takes
    // `top` at once and reloads the next one from memory, so that load's
    // latency hides behind the work on the popped node.
    uint2 top;
    int sp;
    uint32_t cur;  // ref of the node to process; kNone: pop
    uint32_t leaf;  // walk(): ref of the leaf to test; 0: none
    float cur_t;    // entry distance of cur
    uint32_t na, nt;

    __device__ __forceinline__ F3 o() const { return f3(-no.x, -no.y, -no.z); }
    __device__ __forceinline__ void start(F3 o_, F3 d_, float far, const float4* nodes_, const float4* wide_,
                                          const float4* geom_, const ApproxTables& tab) {
        no = f3(-o_.x, -o_.y, -o_.z);
        d = d_;
        nodes = nodes_;
        wide = wide_;
        geom = geom_;
        inv = f3(x_rcp(d.x, tab), x_rcp(d.y, tab), x_rcp(d.z, tab));
        h = Hit{far, 0.0f, 0.0f, -1};
        sp = 0;
        na = 2;
        nt = 0;
        cur = 0;  // the root pair: internal ref with index 0
        leaf = 0u;
        cur_t = __int_as_float(0xff800000);  // the roots are never culled (bvh.rs:604-634)
    }

    // The leaf loops are not unrolled: len is bounded by its 5 bits, and the
    // compiler's unrolled copies of tri_test cost more in instruction fetch
    // than the loop (4M-ray query 0.825 -> 0.808 ms, tube frame 3.24 -> 3.11 ms).
    //
    // Returns true when the ray is finished (its stack is empty): h is then
    // its nearest hit. Sets `overflow` (and finishes the ray) when the stack
    // would overflow. SELECT: the slab test in select form (box_test_sel; the
    // scene and the ray must meet its conditions).
    template <bool COUNT, bool LEAF_AFTER_PAIR, bool SELECT = false, class Stack>
    __device__ __forceinline__ bool step(Stack& stack, bool& overflow) {
        if (cur == kNone) {
            // Pop until an entry survives the cull test (aabb.rs:171-177).
            while (sp > 0) {
                uint2 e = top;
                top = stack.load(--sp);
                if (!geq(__uint_as_float(e.y), h.t)) {
                    cur = e.x;
                    cur_t = __uint_as_float(e.y);
                    break;
                }
            }
            if (cur == kNone) return true;
        }
        uint32_t len = cur & 31u, idx = cur >> 5;
        if (!LEAF_AFTER_PAIR && len != 0u) {  // a popped leaf; the pair loop continues next iteration
            leaf_range(nodes, idx, len);
#pragma unroll 1
            for (uint32_t i = idx; i < idx + len; i++) tri_test(geom, i, o(), d, true, h);
            if (COUNT) nt += len;
            cur = kNone;
            return false;
        }
        if (len == 0u) {
            // An internal node: test its two children.
            if (COUNT && cur != 0u) na += 2;  // every pair but the root pair (bvh.rs:604-634)
            // The reference of an internal node is its first child's index (even:
            // checked at scene creation) times 32, which is the byte offset of
            // the child pair (64 bytes per pair).
            const float4* np = reinterpret_cast<const float4*>(reinterpret_cast<const char*>(nodes) + cur);
            float4 q0 = __ldg(np), q1 = __ldg(np + 1), q2 = __ldg(np + 2), q3 = __ldg(np + 3);
            BoxT b0, b1;
            if constexpr (SELECT) {
                b0 = box_test_sel(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o(), inv);
                b1 = box_test_sel(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o(), inv);
            } else {
                b0 = box_test(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, o(), inv);
                b1 = box_test(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, o(), inv);
            }
            bool first0 = !sneg(b0.tmin - b1.tmin);
            bool hit0 = b0.mask & !sneg(b0.tmax);
            bool hit1 = b1.mask & !sneg(b1.tmax);
            const uint32_t r0 = __float_as_uint(q3.x), r1 = __float_as_uint(q3.y);
            // The reference pushes `first` then `second` and pops `second` first.
            bool hit_first = first0 ? hit0 : hit1, hit_second = first0 ? hit1 : hit0;
            uint32_t ref_first = first0 ? r0 : r1, ref_second = first0 ? r1 : r0;
            float t_first = first0 ? b0.tmin : b1.tmin, t_second = first0 ? b1.tmin : b0.tmin;
            if (sp + (int)hit_first + (int)hit_second > c_stack_limit) {
                overflow = true;
                sp = 0;
                cur = kNone;
                return false;
            }
            if (hit_first) {
                stack.store(sp, top);
                top = make_uint2(ref_first, __float_as_uint(t_first));
                sp++;
            }
            cur = (hit_second && !geq(t_second, h.t)) ? ref_second : kNone;
            cur_t = t_second;
            if (!LEAF_AFTER_PAIR || cur == kNone) return false;
            len = cur & 31u;
            idx = cur >> 5;
        }
        // LEAF_AFTER_PAIR: a leaf, popped or reached from the pair just tested
        // (the reference would pop it next with no decision in between).
        if (len != 0u) {
            leaf_range(nodes, idx, len);
#pragma unroll 1
            for (uint32_t i = idx; i < idx + len; i++) tri_test(geom, i, o(), d, true, h);
            if (COUNT) nt += len;
            cur = kNone;
        }
        return false;
    }

    // The same traversal over the wide records (select form), with the leaf
    // tests postponed: walk() goes on from record to record while at most one
    // leaf waits in `leaf`, and test_leaf() tests that leaf's triangles. A warp
    // alternates a few walk() steps with one test_leaf(), so the triangle code
    // runs once per round for all lanes that reached a leaf in it, not at nearly
    // every step for one or two lanes.
    //
    // A wide record holds the boxes of a pair's four grandchildren (WidePlanes):
    // one step does what step() does for the pair and for both its children.
    // The triangles tested and their order are those of step():
    //  * Bounds nest (checked at scene creation), and the differences, products,
    //    minima and maxima of the slab test are monotonic in the bounds, for
    //    finite values. So a ray that hits a grandchild's box hits the child's,
    //    with an entry distance not beyond the grandchild's: the child's own
    //    test and its cull when popped decide nothing that the grandchild's do
    //    not decide, at the same hit distance.
    //  * A child's bound on an axis is that of one of its two boxes, so its near
    //    plane distance is the smaller of theirs and its entry distance, which
    //    orders the children, the largest over the axes: the same bits, as the
    //    two boxes' zeros on an axis have one sign.
    //  * A box entered at or beyond the hit distance would be culled when popped,
    //    as the hit distance never grows: it is not pushed. One that a waiting
    //    leaf's hit culls is dropped when popped, or by test_leaf() where it is
    //    `cur`, and so are the boxes below it, entered no nearer.
    // (With the stack limit lowered, the overflow status may come at another
    // node; up to three boxes of a record are pushed, so trees of up to
    // kWideMaxDepth levels fit the stack.)
    //
    // Does nothing when the stack is empty, the entry popped is culled (a second
    // pop would run with few lanes: one per step 4M icosphere rays 609 -> 592 us,
    // tube sample 1.41 -> 1.37 ms), or the next node is a leaf and one waits already.
    template <class Stack>
    __device__ __forceinline__ void walk(Stack& stack, bool& overflow) {
        if (cur == kNone && sp > 0) {
            uint2 e = top;
            top = stack.load(--sp);
            if (!geq(__uint_as_float(e.y), h.t)) {
                if ((e.x & 31u) != 0u && leaf == 0u) {
                    leaf = e.x;
                } else {
                    cur = e.x;
                    cur_t = __uint_as_float(e.y);
                }
            }
        }
        if ((cur & 31u) != 0u) return;  // nothing left, or a second leaf
        const WideT w(nodes, wide, cur, no, inv);
        cur = kNone;
        // The order of step(): of two boxes the reference pops first the one it
        // pushes second (the second, unless the first is entered nearer), and
        // the boxes of the child it pops first before the other child's.
        const bool in0 = ge0(w.t[0] - w.t[1]), in1 = ge0(w.t[2] - w.t[3]), ch = ge0(w.tc0 - w.tc1);
        const float a0 = in0 ? w.t[0] : w.t[1], a1 = in0 ? w.t[1] : w.t[0];  // child 0: last, first
        const float b0 = in1 ? w.t[2] : w.t[3], b1 = in1 ? w.t[3] : w.t[2];
        const uint32_t ra0 = in0 ? w.r.x : w.r.y, ra1 = in0 ? w.r.y : w.r.x;
        const uint32_t rb0 = in1 ? w.r.z : w.r.w, rb1 = in1 ? w.r.w : w.r.z;
        const float t[4] = {ch ? a0 : b0, ch ? a1 : b1, ch ? b0 : a0, ch ? b1 : a1};
        const uint32_t r[4] = {ch ? ra0 : rb0, ch ? ra1 : rb1, ch ? rb0 : ra0, ch ? rb1 : ra1};
        // From the last to the first: each box hit becomes the next node, and
        // the one before it is pushed (selects and a predicated store: as branches
        // the four boxes took three lanes each).
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool c = t[k] < h.t;
            if (k > 0) {
                const bool p = c && cur != kNone;
                if (p) stack.store(sp, top);
                top.x = p ? cur : top.x;
                top.y = p ? __float_as_uint(cur_t) : top.y;
                sp += p;
            }
            cur = c ? r[k] : cur;
            cur_t = c ? t[k] : cur_t;
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
    // Tests the waiting leaf, if any, and drops `cur` if its hit culls it.
    // Returns true when the ray is finished.
    __device__ __forceinline__ bool test_leaf() {
        if (leaf != 0u) {
            uint32_t len = leaf & 31u, idx = leaf >> 5;
            leaf_range(nodes, idx, len);
#pragma unroll 1
            for (uint32_t i = idx; i < idx + len; i++) tri_test(geom, i, o(), d, true, h);
            leaf = 0u;
            if (geq(cur_t, h.t)) cur = kNone;
            if (cur != kNone && (cur & 31u) != 0u) {  // the second leaf is next
                leaf = cur;
                cur = kNone;
            }
        }
        return cur == kNone && sp == 0 && leaf == 0u;
    }
    // test_leaf() for a whole warp, which must call it converged (`on`: lanes that
    // trace a ray). Where some leaf has more than two triangles, the waiting
    // leaves' triangles are laid out one after the other over the warp's lanes,
    // each lane tests one of them for its ray's lane, and that lane then looks
    // at its triangles that are hit in their order: the same decisions as
    // test_leaf()'s, in about a pass per 32 triangles instead of one per triangle of
    // the longest leaf. Laying out, shuffling the rays and looking at the hits
    // make such a pass cost a little more than two of the others'.
    //
    // For trees deeper than 40 levels. A round of the 870k tube's frame has 15
    // leaves of 2 triangles on average and the longest 4.6: 4.6 passes of 7 lanes
    // become 1.4. One triangle at a time -> this, 1M random rays 470 -> 427 us, a
    // 1280x736 sample of 16 in one launch 25.7 -> 23.2 ms (also when leaves of up to
    // two or three triangles are laid out 23.9-24.3 at the old claim threshold).
    // Shallower trees reach 10 triangles a round and lose by the warp's votes: 4M
    // rays on the 28-level icosphere 614 -> 629 us, the room's samples 6.33 -> 6.20 ms,
    // the icosphere's frame 2.01 -> 2.06 ms.
    //
    // owner: 32 bytes of shared memory of the warp's own. ONE_SCENE: every lane's
    // `geom` is the same.
    template <bool ONE_SCENE>
    __device__ __forceinline__ bool test_leaves(uint8_t* owner, bool on) {
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t len = 0, idx = 0;
        if (on && leaf != 0u) {
            len = leaf & 31u;
            idx = leaf >> 5;
            leaf_range(nodes, idx, len);
        }
        for (;;) {
            if (!__any_sync(0xffffffffu, len != 0u)) break;
            if (__ballot_sync(0xffffffffu, len > 2u) == 0u) {
#pragma unroll 1
                for (uint32_t i = idx; i < idx + len; i++) tri_test(geom, i, o(), d, true, h);
                break;
            }
            // Slots p .. p + n - 1 are this lane's (at most seven triangles a pass).
            uint32_t n = min(len, 7u);
            const unsigned b0 = __ballot_sync(0xffffffffu, n & 1u), b1 = __ballot_sync(0xffffffffu, n & 2u),
                           b2 = __ballot_sync(0xffffffffu, n & 4u), lt = (1u << lane) - 1u;
            const uint32_t p = __popc(b0 & lt) + 2u * __popc(b1 & lt) + 4u * __popc(b2 & lt);
            const uint32_t total = __popc(b0) + 2u * __popc(b1) + 4u * __popc(b2);
            n = p < 32u ? min(n, 32u - p) : 0u;
            const unsigned starts = __reduce_or_sync(0xffffffffu, n ? 1u << p : 0u);
            __syncwarp();
            if (n) owner[p] = (uint8_t)lane;
            __syncwarp();
            const int start = 31 - __clz((int)(starts & (lt | 1u << lane)));  // slot 0 always starts a leaf
            const int w = owner[start];
            const uint32_t i = __shfl_sync(0xffffffffu, idx, w) + (lane - (uint32_t)start);
            const F3 ro = f3(-__shfl_sync(0xffffffffu, no.x, w), -__shfl_sync(0xffffffffu, no.y, w),
                             -__shfl_sync(0xffffffffu, no.z, w));
            const F3 rd = f3(__shfl_sync(0xffffffffu, d.x, w), __shfl_sync(0xffffffffu, d.y, w),
                             __shfl_sync(0xffffffffu, d.z, w));
            const float4* g = geom;
            if (!ONE_SCENE)
                g = reinterpret_cast<const float4*>(
                    __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(geom), w));
            TriT x{0.0f, 0.0f, 0.0f, false};
            if (lane < total) x = tri_eval(g, i, ro, rd);
            unsigned mine = __ballot_sync(0xffffffffu, x.in) >> (p & 31u) & ((1u << n) - 1u);
            while (__any_sync(0xffffffffu, mine != 0u)) {
                const uint32_t k = (uint32_t)__ffs((int)mine) - 1u;  // of no lane's hits: unused
                const int j = (int)(p + k);
                const float t = __shfl_sync(0xffffffffu, x.t, j), u = __shfl_sync(0xffffffffu, x.u, j),
                            v = __shfl_sync(0xffffffffu, x.v, j);
                if (mine != 0u && !geq(t, h.t)) {
                    h.t = t;
                    h.u = u;
                    h.v = v;
                    h.tri = (int32_t)(idx + k);
                }
                mine &= mine - 1u;
            }
            idx += n;
            len -= n;
        }
        if (on && leaf != 0u) {
            leaf = 0u;
            if (geq(cur_t, h.t)) cur = kNone;
            if (cur != kNone && (cur & 31u) != 0u) {
                leaf = cur;
                cur = kNone;
            }
        }
        return on && cur == kNone && sp == 0 && leaf == 0u;
    }
    // From postponed leaves back to step(): after test_leaf() a waiting leaf is
    // the next node.
    __device__ __forceinline__ void settle() {
        if (leaf != 0u) {
            cur = leaf;
            leaf = 0u;
        }
    }
};

template <int N>
__device__ __forceinline__ typename std::conditional<N == 0, LocalStack, SharedLocalStack<N>>::type make_stack(
    uint2* sm, uint2 (&a)[kStackSlots]) {
    if constexpr (N == 0) return LocalStack{a};
    else return SharedLocalStack<N>{sm, a};
}

// Persistent single-ray traversal with ray refill over the rays of `claim`.
// Every iteration each lane processes one node pair or one leaf (RefillRay);
// a lane whose ray is finished takes the next unclaimed ray, so warps stay
// full while rays of different lengths finish.
// The whole warp must call this. `src` provides
//   void first_scene(nodes, wide, geom): what the scene pointers hold before
//   the first ray (a source of one scene gives that scene's, so that the
//   pointers need no registers)
//   void store(r, const Hit&, uint32_t boxes, uint32_t triangles)
// (box and triangle counts when COUNT, else 0). LEAF_AFTER_PAIR: a lane whose
// pair test leads to a leaf tests that leaf in the same iteration (fewer
// iterations for deep trees; the order of decisions is the same either way).
// CLAIM_MIN: lanes without a ray wait until that many want one; results do
// not depend on it (each ray's traversal is independent of when it starts).
// Returns false if a ray overflowed the stack (its hit is then incomplete).
// FORM kWide: rays walk the wide records, with postponed leaves (RefillRay::
// walk); kPairs: step() in the select form. A ray that the form does not allow is
// handed to src.defer(r) untraced (the caller traces it afterwards in the x86
// form). STEPS: wide records or traversal steps per round of the warp's votes (a
// lane whose ray ends within a round waits for the next round's claim).
// POOL_LEAVES (with kWide): a round's leaves are tested by the whole warp
// (RefillRay::test_leaves).
template <bool COUNT, bool LEAF_AFTER_PAIR, int CLAIM_MIN, int SHARED_STACK = 0, Form FORM = Form::kX86, int STEPS = 1,
          bool POOL_LEAVES = false, class Src, class Claim>
__device__ __forceinline__ bool traverse_refill(const Src& src, Claim& claim, const ApproxTables& tab,
                                                uint2* shared_stack = nullptr) {
    __shared__ uint8_t owners[4][32];  // test_leaves(), blocks of four warps
    uint8_t* const owner = owners[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    RefillRay ray;
    uint2 local_stack[kStackSlots];
    typename std::conditional<SHARED_STACK == 0, LocalStack, SharedLocalStack<SHARED_STACK>>::type stack =
        make_stack<SHARED_STACK>(shared_stack, local_stack);
    ray.top = make_uint2(0u, 0u);
    ray.sp = 0;
    ray.cur = 0;
    ray.leaf = 0u;
    ray.cur_t = 0.0f;
    ray.na = ray.nt = 0;
    src.first_scene(ray.nodes, ray.wide, ray.geom);
    ray.no = ray.d = ray.inv = f3(0, 0, 0);
    ray.h = Hit{0.0f, 0.0f, 0.0f, -1};
    uint32_t r_id = 0;
    bool have = false, done = false, overflow = false;
    for (;;) {
        bool want = !have && !done;
        unsigned b = __ballot_sync(0xffffffffu, want);
        // Claim only when CLAIM_MIN lanes want a ray (or none has work): the
        // claim path then runs with many lanes at once instead of with one or
        // two lanes in nearly every iteration.
        if (CLAIM_MIN > 1 && b && __popc(b) < CLAIM_MIN && __any_sync(0xffffffffu, have)) b = 0u;
        want = want && b;
        if (b) {
            uint32_t r = 0;
            RayIn in;
            int got = claim.claim(b, want, lane, r, in);
            if (want) {
                if (got == kClaimRay) {
                    r_id = r;
                    ray.start(in.o, in.d, in.far, in.nodes, in.wide, in.geom, tab);
                    have = true;
                    if constexpr (FORM != Form::kX86) {
                        if (!form_allows<FORM>(ray.no, ray.inv)) {
                            src.defer(r);
                            have = false;
                        }
                    }
                } else if (got == kClaimDone) {
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if constexpr (FORM == Form::kWide) {
            if (have) {
#pragma unroll
                for (int st = 0; st < STEPS; st++) ray.walk(stack, overflow);
            }
            bool finished;
            if constexpr (POOL_LEAVES) finished = ray.test_leaves<true>(owner, have);
            else finished = have && ray.test_leaf();
            if (finished) {
                src.store(r_id, ray.h, 0u, 0u);
                have = false;
            }
        } else {
            for (int st = 0; st < STEPS && have; st++) {
                if (ray.step<COUNT, LEAF_AFTER_PAIR, FORM == Form::kPairs>(stack, overflow)) {
                    src.store(r_id, ray.h, ray.na, ray.nt);
                    have = false;
                }
            }
        }
    }
    return !overflow;
}

}  // namespace cvx
