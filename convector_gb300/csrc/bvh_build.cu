// Device BVH build: the binned TSAH build of bvh.rs:44-545 on the GPU, with
// the host build's node order, triangle order and statistics.
//
// Exactness. Every decision of the host build is reproduced:
//  * split costs are computed with the same float operations in the same
//    order (the n-dependent TSAH factors come from a host-made table, so the
//    libm powf/log2f results are the host's own);
//  * bin boxes only feed costs, whose values do not depend on the sign of a
//    zero bound, so they are plain min/max reductions;
//  * node boxes are written out and must be bit-identical: from_refs folds
//    the triangle boxes in node order with f32::min / f32::max, which keep
//    the first of equal operands (+0 / -0), so a node bound is the bound of
//    the first triangle in node order that attains the extreme value. The
//    reduction key is (value with -0 as +0, position).
//  * triangle order inside a child is the host's: bins concatenated in bin
//    order, each bin in insertion order (node order for coordinate binning,
//    sorted order for the uniform split of bvh.rs:176-201).
// Inputs with NaN or infinite coordinates are refused (the host build takes
// them; its min/max folds then depend on NaN placement).
//
// Structure. Nodes of more than 32 triangles are split level by level by the
// whole device (coordinate binning with shared-memory histograms, a segmented
// sort for the uniform fallback, a stable counting-sort partition); every
// node of 2..32 triangles is then built completely by one warp (per = 1 in
// the uniform split, so bins are single triangles in sorted order). The interim
// tree is then crystallized into the reference's node array on the device too.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <memory>
#include <vector>

#include "internal.h"

namespace cvx {
namespace {

constexpr int kBins = 64;
constexpr uint32_t kSmall = 32;      // nodes up to this size are built by one warp
constexpr int kTile = 256;           // positions per tile (one per thread)
constexpr uint32_t kBlockSort = 4096;  // uniform sorts up to this size run in one block
constexpr uint32_t kMaxTris = 1u << 26;

struct Refs {
    float* lo[3];
    float* hi[3];
    float* bc[3];
};

struct Tile {
    uint32_t slot, axis, start, len;
};

// Per-slot state of the level being split.
struct Slot {
    uint32_t id, beg, cnt;
};

// A slot's split, and what else the host reads of a level. axis 3: no axis had two
// non-empty bins. flags: bit 0 a leaf, bit 1 + a the mode of axis a (k_fallback).
// The entry after the last slot's holds the error bits in `flags`.
struct Decision {
    uint32_t axis, at, nl, flags;
};
// A split node and its children, l and l + 1: the first nl of its cnt triangles
// from beg, and the others.
struct Link {
    uint32_t id, l, beg, nl, cnt;
};

// Orderable key of a float with -0 and +0 equal (no NaN reaches here).
__device__ __forceinline__ uint32_t okey(float x) {
    uint32_t u = __float_as_uint(x);
    if ((u << 1) == 0u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_okey(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
// f32::min / f32::max of the host build (first operand on equal values).
__device__ __forceinline__ float fmin_rs(float a, float b) { return a != a ? b : (b < a ? b : a); }
__device__ __forceinline__ float fmax_rs(float a, float b) { return a != a ? b : (b > a ? b : a); }

struct Box {
    float lo[3], hi[3];
};
// aabb.rs:97-103
__device__ __forceinline__ float area(const Box& b) {
    float sx = b.hi[0] - b.lo[0], sy = b.hi[1] - b.lo[1], sz = b.hi[2] - b.lo[2];
    float x = sy * sz, y = sz * sx, z = sx * sy;
    return 2.0f * (x + y + z);
}

struct Tsah {
    const float* x;  // 2p - n p^log2(n)
    const float* t;  // n p^(log2(n) - 1)
    float y;         // p - 2p^2
};
// TreeSurfaceAreaHeuristic::aabb_cost (bvh.rs:452-474), the host's operation order.
__device__ __forceinline__ float tsah_cost(const Tsah& ts, float parent_area, const Box& b, uint32_t n) {
    float ac_ap = area(b) / parent_area;
    float aabb_term = 1.0f + ac_ap * ts.x[n] / ts.y;
    float tri_term = ts.t[n] * ac_ap;
    return aabb_term * 40.0f + tri_term * 120.0f;
}

// ---------------------------------------------------------------------------
// Triangle boxes and barycentres (bvh.rs:495-499).

__global__ void k_prep(const cvx_triangle* __restrict__ tris, uint32_t n, float third, Refs r,
                       uint32_t* __restrict__ order, uint32_t* __restrict__ bad) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const cvx_triangle& t = tris[i];
    bool ok = true;
    for (int c = 0; c < 3; c++) {
        float a = t.v0[c], b = t.v1[c], d = t.v2[c];
        ok = ok && isfinite(a) && isfinite(b) && isfinite(d);
        r.lo[c][i] = fmin_rs(fmin_rs(a, b), d);
        r.hi[c][i] = fmax_rs(fmax_rs(a, b), d);
        r.bc[c][i] = ((a + b) + d) * third;
    }
    order[i] = i;
    if (!ok) atomicOr(bad, 1u);
}

// ---------------------------------------------------------------------------
// Exact node boxes of a list of ranges (from_refs, bvh.rs:125-132): outer
// bounds as (key, position) extremes, the barycentre box (inner) by value.

struct BoxAcc {
    unsigned long long omin[3], omax[3];
    uint32_t imin[3], imax[3];
};

__global__ void k_box_init(BoxAcc* acc, uint32_t m) {
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    for (int c = 0; c < 3; c++) {
        acc[j].omin[c] = ~0ull;
        acc[j].omax[c] = 0ull;
        acc[j].imin[c] = ~0u;
        acc[j].imax[c] = 0u;
    }
}

__device__ __forceinline__ unsigned long long shfl64(unsigned long long v, int o) {
    uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
    lo = __shfl_xor_sync(0xffffffffu, lo, o);
    hi = __shfl_xor_sync(0xffffffffu, hi, o);
    return ((unsigned long long)hi << 32) | lo;
}

// One block per tile; the tile's slot indexes `acc`.
__global__ void __launch_bounds__(kTile) k_box(const Tile* __restrict__ tiles, uint32_t n_tiles, Refs r,
                                               const uint32_t* __restrict__ order, uint32_t n, BoxAcc* acc,
                                               uint32_t n_acc, uint32_t* err) {
    if (blockIdx.x >= n_tiles) return;
    Tile tl = tiles[blockIdx.x];
    if (tl.slot >= n_acc || tl.start > n || tl.len > (uint32_t)kTile || tl.start + tl.len > n) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    BoxAcc a;
    for (int c = 0; c < 3; c++) {
        a.omin[c] = ~0ull;
        a.omax[c] = 0ull;
        a.imin[c] = ~0u;
        a.imax[c] = 0u;
    }
    if (threadIdx.x < tl.len) {
        uint32_t p = tl.start + threadIdx.x;
        uint32_t t = order[p];
        for (int c = 0; c < 3; c++) {
            a.omin[c] = ((unsigned long long)okey(r.lo[c][t]) << 32) | p;
            a.omax[c] = ((unsigned long long)okey(r.hi[c][t]) << 32) | (0xffffffffu - p);
            uint32_t kb = okey(r.bc[c][t]);
            a.imin[c] = kb;
            a.imax[c] = kb;
        }
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int c = 0; c < 3; c++) {
            a.omin[c] = min(a.omin[c], shfl64(a.omin[c], o));
            a.omax[c] = max(a.omax[c], shfl64(a.omax[c], o));
            a.imin[c] = min(a.imin[c], __shfl_xor_sync(0xffffffffu, a.imin[c], o));
            a.imax[c] = max(a.imax[c], __shfl_xor_sync(0xffffffffu, a.imax[c], o));
        }
    __shared__ BoxAcc sm;
    if (threadIdx.x == 0) sm = a;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && threadIdx.x) {
        for (int c = 0; c < 3; c++) {
            atomicMin(&sm.omin[c], a.omin[c]);
            atomicMax(&sm.omax[c], a.omax[c]);
            atomicMin(&sm.imin[c], a.imin[c]);
            atomicMax(&sm.imax[c], a.imax[c]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        BoxAcc* g = acc + tl.slot;
        for (int c = 0; c < 3; c++) {
            atomicMin(&g->omin[c], sm.omin[c]);
            atomicMax(&g->omax[c], sm.omax[c]);
            atomicMin(&g->imin[c], sm.imin[c]);
            atomicMax(&g->imax[c], sm.imax[c]);
        }
    }
}

// Writes the decoded boxes into the interim nodes from `first` on, a thread per axis:
// four dependent loads bound it (a thread for all three axes 9 us, this 5).
__global__ void k_box_store(uint32_t first, uint32_t m, const BoxAcc* __restrict__ acc, Refs r,
                            const uint32_t* __restrict__ order, uint32_t n, InterimNode* nodes, uint32_t n_nodes,
                            float* inner, uint32_t* err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, j = i / 3u, c = i % 3u;
    if (j >= m) return;
    const uint32_t id = first + j;
    const uint32_t pmin = (uint32_t)acc[j].omin[c], pmax = 0xffffffffu - (uint32_t)acc[j].omax[c];
    if (id >= n_nodes || pmin >= n || pmax >= n) {
        atomicOr(err, 2u);
        return;
    }
    const float* const lo = c == 0u ? r.lo[0] : c == 1u ? r.lo[1] : r.lo[2];
    const float* const hi = c == 0u ? r.hi[0] : c == 1u ? r.hi[1] : r.hi[2];
    nodes[id].lo[c] = lo[order[pmin]];
    nodes[id].hi[c] = hi[order[pmax]];
    inner[6 * (size_t)id + c] = from_okey(acc[j].imin[c]);
    inner[6 * (size_t)id + 3 + c] = from_okey(acc[j].imax[c]);
}

// ---------------------------------------------------------------------------
// Level split of nodes above kSmall triangles.

// Bin statistics per (slot, axis, bin): count and the bin box as value keys.
struct BinStats {
    uint32_t* count;  // [K][3][64]
    uint32_t* key;    // [K][3][64][6]: lo x y z (min), hi x y z (max)
};

__global__ void k_stats_init(BinStats st, uint32_t entries) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= entries) return;
    st.count[i] = 0u;
    for (int c = 0; c < 3; c++) {
        st.key[6 * (size_t)i + c] = ~0u;
        st.key[6 * (size_t)i + 3 + c] = 0u;
    }
}

// Adds triangle t to the shared-memory histogram of (axis, bin).
__device__ __forceinline__ void sm_add(uint32_t* cnt, uint32_t* key, int a, int b, const Refs& r, uint32_t t) {
    int e = a * kBins + b;
    atomicAdd(&cnt[e], 1u);
    for (int c = 0; c < 3; c++) {
        atomicMin(&key[6 * e + c], okey(r.lo[c][t]));
        atomicMax(&key[6 * e + 3 + c], okey(r.hi[c][t]));
    }
}

__device__ __forceinline__ void sm_flush(const uint32_t* cnt, const uint32_t* key, BinStats st, uint32_t slot,
                                         int axis_lo, int axis_hi) {
    for (int e = threadIdx.x; e < 3 * kBins; e += blockDim.x) {
        int a = e / kBins;
        if (a < axis_lo || a > axis_hi || cnt[e] == 0u) continue;
        size_t g = (size_t)slot * 3 * kBins + e;
        atomicAdd(&st.count[g], cnt[e]);
        for (int c = 0; c < 3; c++) {
            atomicMin(&st.key[6 * g + c], key[6 * e + c]);
            atomicMax(&st.key[6 * g + 3 + c], key[6 * e + 3 + c]);
        }
    }
}

__device__ __forceinline__ void sm_init(uint32_t* cnt, uint32_t* key) {
    for (int e = threadIdx.x; e < 3 * kBins; e += blockDim.x) {
        cnt[e] = 0u;
        for (int c = 0; c < 3; c++) {
            key[6 * e + c] = ~0u;
            key[6 * e + 3 + c] = 0u;
        }
    }
}

// Coordinate binning of bvh.rs:142-171 on all three axes.
__global__ void __launch_bounds__(kTile) k_bin_float(const Tile* __restrict__ tiles, uint32_t n_tiles,
                                                     const Slot* __restrict__ slots, uint32_t n_slots, Refs r,
                                                     const uint32_t* __restrict__ order, uint32_t n,
                                                     const float* __restrict__ inner, uint8_t* __restrict__ binf,
                                                     BinStats st, uint32_t* err) {
    __shared__ uint32_t cnt[3 * kBins];
    __shared__ uint32_t key[3 * kBins * 6];
    if (blockIdx.x >= n_tiles) return;
    Tile tl = tiles[blockIdx.x];
    if (tl.slot >= n_slots || tl.len > (uint32_t)kTile || tl.start + tl.len > n) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    sm_init(cnt, key);
    __syncthreads();
    Slot s = slots[tl.slot];
    if (threadIdx.x < tl.len) {
        uint32_t p = tl.start + threadIdx.x;
        uint32_t t = order[p];
        for (int a = 0; a < 3; a++) {
            float mn = inner[6 * (size_t)s.id + a];
            float size = inner[6 * (size_t)s.id + 3 + a] - mn;
            float f = floorf((float)kBins * (r.bc[a][t] - mn) / size);
            // `as usize` saturates NaN and negatives to 0; clamp to the last bin.
            int b = (f != f || f <= 0.0f) ? 0 : (f >= (float)(kBins - 1) ? kBins - 1 : (int)f);
            binf[(size_t)a * n + p] = (uint8_t)b;
            sm_add(cnt, key, a, b, r, t);
        }
    }
    __syncthreads();
    sm_flush(cnt, key, st, tl.slot, 0, 2);
}

// bvh.rs:160-166: a bin above n/8 triangles (n > 64) sends the axis to the
// uniform split. mode[slot][axis]: 0 coordinate bins, 1 uniform; the statistics of
// those that k_sort_slots sorts are reset. One warp per (slot, axis): a thread
// per slot and a pass for the reset took 12 + 3 us a level.
__global__ void __launch_bounds__(128) k_fallback(const Slot* __restrict__ slots, uint32_t n_slots, BinStats st,
                                                  uint32_t* __restrict__ mode) {
    const uint32_t pair = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (pair >= 3u * n_slots) return;  // warp-uniform
    const uint32_t n = slots[pair / 3u].cnt;
    uint32_t* const cn = st.count + (size_t)pair * kBins;
    const uint32_t mx = __reduce_max_sync(0xffffffffu, max(cn[lane], cn[lane + 32u]));
    const bool uniform = mx > n / 8u && n > (uint32_t)kBins;
    if (lane == 0u) mode[pair] = uniform ? 1u : 0u;
    if (!uniform || n > kBlockSort) return;
    for (uint32_t b = lane; b < (uint32_t)kBins; b += 32u) {
        cn[b] = 0u;
        for (int c = 0; c < 3; c++) {
            st.key[6 * ((size_t)pair * kBins + b) + c] = ~0u;
            st.key[6 * ((size_t)pair * kBins + b) + 3 + c] = 0u;
        }
    }
}

// Uniform split keys: (barycentre coordinate key, position); ascending order
// is std::stable_sort by the coordinate (-0 and +0 compare equal).
__device__ __forceinline__ unsigned long long ukey(const Refs& r, const uint32_t* order, int a, uint32_t p) {
    return ((unsigned long long)okey(r.bc[a][order[p]]) << 32) | p;
}

// One block sorts the positions of one (slot, axis) of at most kBlockSort
// triangles; srt[axis][beg + rank] = position.
__device__ __forceinline__ void sort_pair(const Tile& pr, unsigned long long* k, const Refs& r,
                                          const uint32_t* __restrict__ order, uint32_t n,
                                          uint32_t* __restrict__ srt) {
    uint32_t m = 1;
    while (m < pr.len) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x)
        k[i] = i < pr.len ? ukey(r, order, pr.axis, pr.start + i) : ~0ull;
    __syncthreads();
    for (uint32_t size = 2; size <= m; size <<= 1)
        for (uint32_t j = size >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                uint32_t l = i ^ j;
                if (l > i) {
                    bool up = (i & size) == 0u;
                    unsigned long long x = k[i], y = k[l];
                    if ((x > y) == up) {
                        k[i] = y;
                        k[l] = x;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < pr.len; i += blockDim.x)
        srt[(size_t)pr.axis * n + pr.start + i] = (uint32_t)k[i];
}

// The uniform split of every (slot, axis) that fell back and fits one block:
// the sort, one block per slot and axis; the others return at once, which
// costs less than the host's look at the modes and its list (a round trip and
// three uploads per level).
__global__ void __launch_bounds__(1024) k_sort_slots(const Slot* __restrict__ slots, uint32_t n_slots,
                                                     const uint32_t* __restrict__ mode, Refs r,
                                                     const uint32_t* __restrict__ order, uint32_t n,
                                                     uint32_t* __restrict__ srt, uint32_t* err) {
    __shared__ unsigned long long k[kBlockSort];
    const uint32_t slot = blockIdx.x / 3u, axis = blockIdx.x % 3u;
    if (slot >= n_slots || !mode[3 * slot + axis]) return;
    const Slot sl = slots[slot];
    if (sl.cnt > kBlockSort) return;  // sorted through global memory
    if (sl.beg + sl.cnt > n) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    sort_pair(Tile{slot, axis, sl.beg, sl.cnt}, k, r, order, n, srt);
}

__global__ void k_sort_fill(Tile pr, uint32_t m, Refs r, const uint32_t* __restrict__ order,
                            unsigned long long* __restrict__ buf) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    buf[i] = i < pr.len ? ukey(r, order, pr.axis, pr.start + i) : ~0ull;
}
__global__ void k_sort_step(unsigned long long* __restrict__ buf, uint32_t m, uint32_t size, uint32_t j) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    uint32_t l = i ^ j;
    if (l <= i) return;
    bool up = (i & size) == 0u;
    unsigned long long x = buf[i], y = buf[l];
    if ((x > y) == up) {
        buf[i] = y;
        buf[l] = x;
    }
}
// All steps j < 2048 of stage `size` (from j0 down), on 4096-element chunks.
__global__ void __launch_bounds__(1024) k_sort_chunk(unsigned long long* __restrict__ buf, uint32_t m,
                                                     uint32_t size_lo, uint32_t size_hi, uint32_t j0) {
    __shared__ unsigned long long k[4096];
    uint32_t base = blockIdx.x * 4096u;
    if (base >= m) return;
    for (uint32_t i = threadIdx.x; i < 4096u; i += blockDim.x) k[i] = buf[base + i];
    __syncthreads();
    for (uint32_t size = size_lo; size <= size_hi; size <<= 1)
        for (uint32_t j = (size == size_lo ? j0 : (size >> 1)); j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < 4096u; i += blockDim.x) {
                uint32_t l = i ^ j;
                if (l > i) {
                    bool up = ((base + i) & size) == 0u;
                    unsigned long long x = k[i], y = k[l];
                    if ((x > y) == up) {
                        k[i] = y;
                        k[l] = x;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < 4096u; i += blockDim.x) buf[base + i] = k[i];
}
__global__ void k_sort_extract(Tile pr, const unsigned long long* __restrict__ buf, uint32_t n,
                               uint32_t* __restrict__ srt) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pr.len) return;
    srt[(size_t)pr.axis * n + pr.start + i] = (uint32_t)buf[i];
}

// Statistics of the uniform bins (bin = rank / per) of the (slot, axis) tiles;
// tile.start is a rank offset inside the slot.
__global__ void k_axis_reset(const Tile* __restrict__ pairs, uint32_t n_pairs, BinStats st) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pairs * kBins) return;
    Tile pr = pairs[i / kBins];
    size_t g = ((size_t)pr.slot * 3 + pr.axis) * kBins + (i % kBins);
    st.count[g] = 0u;
    for (int c = 0; c < 3; c++) {
        st.key[6 * g + c] = ~0u;
        st.key[6 * g + 3 + c] = 0u;
    }
}
// slot_mode: `tiles` are the level's tiles (absolute starts), one axis per
// blockIdx.y, of which the (slot, axis) pairs of k_sort_slots are taken; null:
// tiles list (slot, axis, relative start) themselves.
__global__ void __launch_bounds__(kTile) k_uniform_stats(const Tile* __restrict__ tiles, uint32_t n_tiles,
                                                         const uint32_t* __restrict__ slot_mode,
                                                         const Slot* __restrict__ slots, uint32_t n_slots, Refs r,
                                                         const uint32_t* __restrict__ order, uint32_t n,
                                                         const uint32_t* __restrict__ srt, BinStats st,
                                                         uint32_t* err) {
    __shared__ uint32_t cnt[3 * kBins];
    __shared__ uint32_t key[3 * kBins * 6];
    if (blockIdx.x >= n_tiles) return;
    Tile tl = tiles[blockIdx.x];
    if (tl.slot >= n_slots || tl.axis > 2 || tl.len > (uint32_t)kTile) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    Slot s = slots[tl.slot];
    if (slot_mode) {
        tl.axis = blockIdx.y;
        if (!slot_mode[3 * tl.slot + tl.axis] || s.cnt > kBlockSort) return;
        tl.start -= s.beg;
    }
    if (tl.start + tl.len > s.cnt || s.beg + s.cnt > n) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    sm_init(cnt, key);
    __syncthreads();
    uint32_t per = (s.cnt + kBins - 1) / kBins;  // bvh.rs:186-188
    if (threadIdx.x < tl.len) {
        uint32_t rank = tl.start + threadIdx.x;
        uint32_t p = srt[(size_t)tl.axis * n + s.beg + rank];
        if (p < n) sm_add(cnt, key, tl.axis, (int)(rank / per), r, order[p]);
    }
    __syncthreads();
    sm_flush(cnt, key, st, tl.slot, tl.axis, tl.axis);
}

// bvh.rs:218-322: the cheapest split over the three axes, or a leaf. One
// warp per slot and axis (lane l owns bins l and l + 32): prefix and suffix boxes
// and counts by warp scans, the candidate costs in parallel, and their first
// minimum; then the axes in order. Bound by the chain of shuffles: one warp for
// the three axes and the candidates one by one took 30 us a level.
__device__ __forceinline__ void box_scan_empty(Box& b) {
    for (int c = 0; c < 3; c++) {
        b.lo[c] = __int_as_float(0x7f800000);   // +inf
        b.hi[c] = __int_as_float((int)0xff800000u);  // -inf
    }
}
__device__ __forceinline__ void box_join(Box& a, const Box& b) {
    for (int c = 0; c < 3; c++) {
        a.lo[c] = fminf(a.lo[c], b.lo[c]);
        a.hi[c] = fmaxf(a.hi[c], b.hi[c]);
    }
}
__device__ __forceinline__ Box box_shfl_up(const Box& b, int o) {
    Box r;
    for (int c = 0; c < 3; c++) {
        r.lo[c] = __shfl_up_sync(0xffffffffu, b.lo[c], o);
        r.hi[c] = __shfl_up_sync(0xffffffffu, b.hi[c], o);
    }
    return r;
}
__device__ __forceinline__ Box box_shfl_down(const Box& b, int o) {
    Box r;
    for (int c = 0; c < 3; c++) {
        r.lo[c] = __shfl_down_sync(0xffffffffu, b.lo[c], o);
        r.hi[c] = __shfl_down_sync(0xffffffffu, b.hi[c], o);
    }
    return r;
}
__device__ __forceinline__ Box box_shfl(const Box& b, int src) {
    Box r;
    for (int c = 0; c < 3; c++) {
        r.lo[c] = __shfl_sync(0xffffffffu, b.lo[c], src);
        r.hi[c] = __shfl_sync(0xffffffffu, b.hi[c], src);
    }
    return r;
}

__global__ void __launch_bounds__(96) k_choose(const Slot* __restrict__ slots, uint32_t n_slots,
                                               const InterimNode* __restrict__ nodes, BinStats st, Tsah ts,
                                               const uint32_t* __restrict__ mode, const uint32_t* __restrict__ err,
                                               Decision* __restrict__ dec) {
    struct Choice {
        float cost;
        uint32_t at, nl;  // at 0: the axis has no two bins to split between
    };
    __shared__ Choice choice[3];
    const int lane = threadIdx.x & 31, a = threadIdx.x >> 5;
    const uint32_t k = blockIdx.x;
    if (k >= n_slots) return;  // block-uniform
    const Slot s = slots[k];
    Box outer;
    for (int c = 0; c < 3; c++) {
        outer.lo[c] = nodes[s.id].lo[c];
        outer.hi[c] = nodes[s.id].hi[c];
    }
    const float parent_area = area(outer);
    if (lane == 0) choice[a].at = 0u;
    const uint32_t* cn = st.count + ((size_t)k * 3 + a) * kBins;
    const uint32_t* ky = st.key + ((size_t)k * 3 + a) * kBins * 6;
    uint32_t c0 = cn[lane], c1 = cn[lane + 32];
    unsigned m0 = __ballot_sync(0xffffffffu, c0 != 0u), m1 = __ballot_sync(0xffffffffu, c1 != 0u);
    int nonempty = __popc(m0) + __popc(m1);
    if (nonempty > 1) {  // warp-uniform
        int first = (m0 ? __ffs(m0) - 1 : 32 + __ffs(m1) - 1) + 1;
        int last = (m1 ? 32 + 31 - __clz(m1) : 31 - __clz(m0)) + 1;
        Box b0, b1;
        box_scan_empty(b0);
        box_scan_empty(b1);
        if (c0)
            for (int c = 0; c < 3; c++) {
                b0.lo[c] = from_okey(ky[6 * lane + c]);
                b0.hi[c] = from_okey(ky[6 * lane + 3 + c]);
            }
        if (c1)
            for (int c = 0; c < 3; c++) {
                b1.lo[c] = from_okey(ky[6 * (lane + 32) + c]);
                b1.hi[c] = from_okey(ky[6 * (lane + 32) + 3 + c]);
            }
        // Inclusive prefix (bins 0..b) and suffix (bins b..63) of boxes and counts.
        Box p0 = b0, p1 = b1, q0 = b0, q1 = b1;
        uint32_t pc0 = c0, pc1 = c1, qc0 = c0, qc1 = c1;
        for (int o = 1; o < 32; o <<= 1) {
            Box u0 = box_shfl_up(p0, o), u1 = box_shfl_up(p1, o);
            uint32_t uc0 = __shfl_up_sync(0xffffffffu, pc0, o), uc1 = __shfl_up_sync(0xffffffffu, pc1, o);
            Box v0 = box_shfl_down(q0, o), v1 = box_shfl_down(q1, o);
            uint32_t vc0 = __shfl_down_sync(0xffffffffu, qc0, o), vc1 = __shfl_down_sync(0xffffffffu, qc1, o);
            if (lane >= o) {
                box_join(p0, u0);
                box_join(p1, u1);
                pc0 += uc0;
                pc1 += uc1;
            }
            if (lane + o < 32) {
                box_join(q0, v0);
                box_join(q1, v1);
                qc0 += vc0;
                qc1 += vc1;
            }
        }
        Box lowtot = box_shfl(p0, 31), hightot = box_shfl(q1, 0);
        uint32_t lowcnt = __shfl_sync(0xffffffffu, pc0, 31), highcnt = __shfl_sync(0xffffffffu, qc1, 0);
        box_join(p1, lowtot);  // prefix of bins 32 + lane includes all of 0..31
        pc1 += lowcnt;
        box_join(q0, hightot);  // suffix of bins lane includes all of 32..63
        qc0 += highcnt;
        // Split i = b + 1 puts bins 0..b left and i..63 right: left = prefix(b),
        // right = suffix(b + 1). Lane l evaluates i = l + 1 and i = l + 33.
        Box r0 = box_shfl_down(q0, 1), r1 = box_shfl_down(q1, 1);
        uint32_t rc0 = __shfl_down_sync(0xffffffffu, qc0, 1), rc1 = __shfl_down_sync(0xffffffffu, qc1, 1);
        Box q1_first = box_shfl(q1, 0);  // suffix(32) for i = 32
        uint32_t qc1_first = __shfl_sync(0xffffffffu, qc1, 0);
        if (lane == 31) {
            r0 = q1_first;
            rc0 = qc1_first;
        }
        int i0 = lane + 1, i1 = lane + 33;
        float cost0 = 0.0f, cost1 = 0.0f;
        if (i0 >= first && i0 < last) cost0 = tsah_cost(ts, parent_area, p0, pc0) + tsah_cost(ts, parent_area, r0, rc0);
        if (i1 >= first && i1 < last) cost1 = tsah_cost(ts, parent_area, p1, pc1) + tsah_cost(ts, parent_area, r1, rc1);
        // bvh.rs:241-258: the first candidate, then strictly cheaper ones, in bin
        // order: the first of the cheapest, unless the first is not a number.
        const bool v0 = i0 >= first && i0 < last && cost0 == cost0, v1 = i1 >= first && i1 < last && cost1 == cost1;
        const uint32_t k0 = v0 ? okey(cost0) : ~0u, k1 = v1 ? okey(cost1) : ~0u;
        const uint32_t kmin = __reduce_min_sync(0xffffffffu, min(k0, k1));
        const unsigned e0 = __ballot_sync(0xffffffffu, v0 && k0 == kmin), e1 = __ballot_sync(0xffffffffu, v1 && k1 == kmin);
        const float c_first = first <= 32 ? __shfl_sync(0xffffffffu, cost0, first - 1)
                                          : __shfl_sync(0xffffffffu, cost1, first - 33);
        const int at = c_first != c_first ? first : e0 ? __ffs((int)e0) : 32 + __ffs((int)e1);
        const float best = at <= 32 ? __shfl_sync(0xffffffffu, cost0, at - 1) : __shfl_sync(0xffffffffu, cost1, at - 33);
        // left count: prefix count of bin at - 1
        const uint32_t nl = at <= 32 ? __shfl_sync(0xffffffffu, pc0, at - 1) : __shfl_sync(0xffffffffu, pc1, at - 33);
        if (lane == 0) choice[a] = Choice{best, (uint32_t)at, nl};
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    float best_cost = 0.0f;
    bool is_first = true;
    Decision d{3u, 0u, 0u, 1u};
    for (int x = 0; x < 3; x++) {
        const Choice c = choice[x];
        if (c.at != 0u && (c.cost < best_cost || is_first)) {
            best_cost = c.cost;
            is_first = false;
            d = Decision{(uint32_t)x, c.at, c.nl, 0u};
        }
    }
    if (is_first || (float)s.cnt * 120.0f < best_cost) d.flags = 1u;
    for (int x = 0; x < 3; x++) d.flags |= mode[3 * k + x] << (1 + x);
    dec[k] = d;
    if (k == 0) dec[n_slots] = Decision{0u, 0u, 0u, *err};
}

// Partition of the split slots. Coordinate-binned axis: a stable counting
// sort by bin (bins in order, node order inside a bin); uniform axis: the
// sorted order. tile_off[t][b]: first new index (relative to beg) of tile t's
// triangles in bin b.
__global__ void __launch_bounds__(kTile) k_tile_hist(const Tile* __restrict__ tiles, uint32_t n_tiles,
                                                     const uint8_t* __restrict__ binf, uint32_t n,
                                                     uint32_t* __restrict__ tile_hist) {
    __shared__ uint32_t h[kBins];
    if (blockIdx.x >= n_tiles) return;
    Tile tl = tiles[blockIdx.x];
    if (threadIdx.x < kBins) h[threadIdx.x] = 0u;
    __syncthreads();
    if (threadIdx.x < tl.len && tl.start + threadIdx.x < n && tl.axis < 3)
        atomicAdd(&h[binf[(size_t)tl.axis * n + tl.start + threadIdx.x]], 1u);
    __syncthreads();
    if (threadIdx.x < kBins) tile_hist[(size_t)blockIdx.x * kBins + threadIdx.x] = h[threadIdx.x];
}

// One block per split slot with coordinate bins; its tiles are t0..t1-1.
__global__ void __launch_bounds__(1024) k_tile_offsets(const uint32_t* __restrict__ slot_tiles, uint32_t n_split,
                                                       const uint32_t* __restrict__ tile_hist,
                                                       uint32_t* __restrict__ tile_off) {
    __shared__ uint32_t part[16][kBins];
    __shared__ uint32_t bin_start[kBins];
    if (blockIdx.x >= n_split) return;
    uint32_t t0 = slot_tiles[2 * blockIdx.x], t1 = slot_tiles[2 * blockIdx.x + 1];
    uint32_t nt = t1 - t0;
    int b = threadIdx.x % kBins, ch = threadIdx.x / kBins;
    uint32_t per = (nt + 15) / 16;
    uint32_t c0 = t0 + min(nt, ch * per), c1 = t0 + min(nt, (ch + 1) * per);
    uint32_t sum = 0;
    for (uint32_t t = c0; t < c1; t++) sum += tile_hist[(size_t)t * kBins + b];
    part[ch][b] = sum;
    __syncthreads();
    if (threadIdx.x < kBins) {
        uint32_t tot = 0;
        for (int c = 0; c < 16; c++) tot += part[c][threadIdx.x];
        bin_start[threadIdx.x] = tot;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int k = 0; k < kBins; k++) {
            uint32_t v = bin_start[k];
            bin_start[k] = run;
            run += v;
        }
    }
    __syncthreads();
    uint32_t off = bin_start[b];
    for (int c = 0; c < ch; c++) off += part[c][b];
    for (uint32_t t = c0; t < c1; t++) {
        tile_off[(size_t)t * kBins + b] = off;
        off += tile_hist[(size_t)t * kBins + b];
    }
}

// tiles: the split slots' tiles; axis = 3 + axis for a uniform axis.
__global__ void __launch_bounds__(kTile) k_scatter(const Tile* __restrict__ tiles, uint32_t n_tiles,
                                                   const Slot* __restrict__ slots, uint32_t n_slots,
                                                   const uint8_t* __restrict__ binf, const uint32_t* __restrict__ srt,
                                                   const uint32_t* __restrict__ tile_off,
                                                   const uint32_t* __restrict__ order, uint32_t n,
                                                   uint32_t* __restrict__ order_tmp, uint32_t* err) {
    __shared__ uint32_t wcount[kTile / 32][kBins];
    if (blockIdx.x >= n_tiles) return;
    Tile tl = tiles[blockIdx.x];
    if (tl.slot >= n_slots || tl.len > (uint32_t)kTile || tl.start + tl.len > n || tl.axis > 5) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    Slot s = slots[tl.slot];
    uint32_t p = tl.start + threadIdx.x;
    bool live = threadIdx.x < tl.len;
    if (tl.axis >= 3) {  // uniform: new index = rank
        if (live) {
            uint32_t rank = p - s.beg;
            uint32_t src = srt[(size_t)(tl.axis - 3) * n + p];
            if (src < n && rank < s.cnt) order_tmp[p] = order[src];
            else atomicOr(err, 2u);
        }
        return;
    }
    int w = threadIdx.x / 32, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < (kTile / 32) * kBins; i += blockDim.x) (&wcount[0][0])[i] = 0u;
    __syncthreads();
    int b = live ? binf[(size_t)tl.axis * n + p] : kBins;  // kBins: no bin
    unsigned same = __match_any_sync(0xffffffffu, b);
    uint32_t rank = __popc(same & ((1u << lane) - 1u));
    if (live && rank == 0u) wcount[w][b] = __popc(same);
    __syncthreads();
    if (live) {
        uint32_t before = 0;
        for (int k = 0; k < w; k++) before += wcount[k][b];
        uint32_t dst = s.beg + tile_off[(size_t)blockIdx.x * kBins + b] + before + rank;
        if (dst < s.beg + s.cnt) order_tmp[dst] = order[p];
        else atomicOr(err, 2u);
    }
}

__global__ void k_copy_back(const Tile* __restrict__ tiles, uint32_t n_tiles, const uint32_t* __restrict__ src,
                            uint32_t* __restrict__ dst, uint32_t n) {
    if (blockIdx.x >= n_tiles) return;
    Tile tl = tiles[blockIdx.x];
    uint32_t p = tl.start + threadIdx.x;
    if (threadIdx.x < tl.len && p < n) dst[p] = src[p];
}

// Links split parents to their children, smaller box first (bvh.rs:333-335), and
// sets the children's ranges.
__global__ void k_link(const Link* __restrict__ links, uint32_t m, InterimNode* nodes, uint32_t n_nodes,
                       uint32_t* err) {
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    const Link k = links[j];
    const uint32_t l = k.l, r = k.l + 1u;
    if (k.id >= n_nodes || r >= n_nodes) {
        atomicOr(err, 2u);
        return;
    }
    Box bl, br;
    for (int c = 0; c < 3; c++) {
        bl.lo[c] = nodes[l].lo[c];
        bl.hi[c] = nodes[l].hi[c];
        br.lo[c] = nodes[r].lo[c];
        br.hi[c] = nodes[r].hi[c];
    }
    nodes[l].beg = k.beg;
    nodes[l].cnt = k.nl;
    nodes[r].beg = k.beg + k.nl;
    nodes[r].cnt = k.cnt - k.nl;
    bool swap = area(bl) > area(br);
    nodes[k.id].c0 = swap ? r : l;
    nodes[k.id].c1 = swap ? l : r;
}

// ---------------------------------------------------------------------------
// Warp build of a node of 2..32 triangles and its whole subtree. Every split
// is the uniform split with one triangle per bin, so the split candidates
// are the prefixes of the triangles sorted by barycentre coordinate. The
// node's range of `order` is rewritten in depth-first leaf order.

constexpr int kSmallWarps = 4;

__device__ __forceinline__ float shf(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }

__global__ void __launch_bounds__(32 * kSmallWarps) k_small(const uint32_t* __restrict__ ids, uint32_t m,
                                                            InterimNode* nodes, uint32_t n_nodes,
                                                            uint32_t* next_id, uint32_t* order, uint32_t n, Refs r,
                                                            Tsah ts, uint32_t* err) {
    __shared__ uint8_t lists[kSmallWarps][kSmall + 1][kSmall];
    __shared__ uint32_t st_id[kSmallWarps][kSmall + 1];
    __shared__ uint32_t st_cnt[kSmallWarps][kSmall + 1];
    __shared__ uint8_t perm[kSmallWarps][3][kSmall];
    const int w = threadIdx.x / 32, lane = threadIdx.x & 31;
    uint32_t job = blockIdx.x * kSmallWarps + w;
    if (job >= m) return;
    uint32_t root = ids[job];
    if (root >= n_nodes) {
        if (lane == 0) atomicOr(err, 2u);
        return;
    }
    uint32_t beg = nodes[root].beg, cnt = nodes[root].cnt;
    if (cnt < 2u || cnt > kSmall || beg + cnt > n) {
        if (lane == 0) atomicOr(err, 2u);
        return;
    }
    // Element e (0..cnt-1) = the triangle at beg + e; its data sits in lane e.
    uint32_t tri = lane < (int)cnt ? order[beg + lane] : 0u;
    float lo[3], hi[3], bc[3];
    for (int c = 0; c < 3; c++) {
        lo[c] = lane < (int)cnt ? r.lo[c][tri] : 0.0f;
        hi[c] = lane < (int)cnt ? r.hi[c][tri] : 0.0f;
        bc[c] = lane < (int)cnt ? r.bc[c][tri] : 0.0f;
    }
    __syncwarp();
    int sp = 0;
    if (lane < (int)cnt) lists[w][0][lane] = (uint8_t)lane;
    if (lane == 0) {
        st_id[w][0] = root;
        st_cnt[w][0] = cnt;
    }
    sp = 1;
    uint32_t out_pos = 0;
    __syncwarp();
    while (sp > 0) {
        sp--;
        uint32_t u = st_id[w][sp], mm = st_cnt[w][sp];
        int me = lane < (int)mm ? lists[w][sp][lane] : 0;  // element at node position `lane`
        __syncwarp();
        bool leaf = mm <= 1u;
        int best_axis = 0, best_at = 0;
        if (!leaf) {
            Box outer;
            for (int c = 0; c < 3; c++) {
                outer.lo[c] = nodes[u].lo[c];
                outer.hi[c] = nodes[u].hi[c];
            }
            float parent_area = area(outer);
            float best_cost = 0.0f;
            bool is_first = true;
            for (int a = 0; a < 3; a++) {
                uint32_t mykey = okey(shf(bc[a], me));
                int rank = 0;
                for (int j = 0; j < (int)mm; j++) {
                    uint32_t kj = __shfl_sync(0xffffffffu, mykey, j);
                    rank += (kj < mykey || (kj == mykey && j < lane)) ? 1 : 0;
                }
                if (lane < (int)mm) perm[w][a][rank] = (uint8_t)lane;
                __syncwarp();
                // Lane q holds the element of rank q.
                int eq = lane < (int)mm ? lists[w][sp][perm[w][a][lane]] : 0;
                Box pb, sb;
                for (int c = 0; c < 3; c++) {
                    float l = shf(lo[c], eq), h = shf(hi[c], eq);
                    pb.lo[c] = l;
                    pb.hi[c] = h;
                    sb.lo[c] = l;
                    sb.hi[c] = h;
                }
                for (int o = 1; o < 32; o <<= 1)
                    for (int c = 0; c < 3; c++) {
                        float pl = __shfl_up_sync(0xffffffffu, pb.lo[c], o);
                        float ph = __shfl_up_sync(0xffffffffu, pb.hi[c], o);
                        float sl = __shfl_down_sync(0xffffffffu, sb.lo[c], o);
                        float sh = __shfl_down_sync(0xffffffffu, sb.hi[c], o);
                        if (lane >= o) {
                            pb.lo[c] = fminf(pb.lo[c], pl);
                            pb.hi[c] = fmaxf(pb.hi[c], ph);
                        }
                        if (lane + o < (int)mm) {
                            sb.lo[c] = fminf(sb.lo[c], sl);
                            sb.hi[c] = fmaxf(sb.hi[c], sh);
                        }
                    }
                // Split i (1 <= i < mm): left = ranks 0..i-1, right = ranks i..mm-1.
                Box la;
                for (int c = 0; c < 3; c++) {
                    la.lo[c] = __shfl_up_sync(0xffffffffu, pb.lo[c], 1);
                    la.hi[c] = __shfl_up_sync(0xffffffffu, pb.hi[c], 1);
                }
                float cost = 0.0f;
                if (lane >= 1 && lane < (int)mm)
                    cost = tsah_cost(ts, parent_area, la, (uint32_t)lane) +
                           tsah_cost(ts, parent_area, sb, mm - (uint32_t)lane);
                float best = shf(cost, 1);
                int at = 1;
                for (int i = 2; i < (int)mm; i++) {
                    float ci = shf(cost, i);
                    if (ci < best) {
                        best = ci;
                        at = i;
                    }
                }
                if (best < best_cost || is_first) {
                    best_cost = best;
                    best_axis = a;
                    best_at = at;
                    is_first = false;
                }
            }
            leaf = (float)mm * 120.0f < best_cost;
        }
        if (leaf) {
            uint32_t tv = __shfl_sync(0xffffffffu, tri, me);
            if (lane < (int)mm) order[beg + out_pos + lane] = tv;
            if (lane == 0) {
                nodes[u].beg = beg + out_pos;
                nodes[u].cnt = mm;
                nodes[u].c0 = 0u;
                nodes[u].c1 = 0u;
            }
            out_pos += mm;
            __syncwarp();
            continue;
        }
        // Children in sorted order of the chosen axis; exact boxes with the
        // first of equal bounds in child order.
        uint32_t at = (uint32_t)best_at;
        int eq = lane < (int)mm ? lists[w][sp][perm[w][best_axis][lane]] : 0;
        bool in_left = lane < (int)at, in_right = lane >= (int)at && lane < (int)mm;
        Box cb[2];
        for (int side = 0; side < 2; side++) {
            bool mine = side == 0 ? in_left : in_right;
            for (int c = 0; c < 3; c++) {
                float vl = shf(lo[c], eq), vh = shf(hi[c], eq);
                unsigned long long kmin = mine ? (((unsigned long long)okey(vl) << 32) | (uint32_t)lane) : ~0ull;
                unsigned long long kmax =
                    mine ? (((unsigned long long)okey(vh) << 32) | (0xffffffffu - (uint32_t)lane)) : 0ull;
                for (int o = 16; o > 0; o >>= 1) {
                    kmin = min(kmin, shfl64(kmin, o));
                    kmax = max(kmax, shfl64(kmax, o));
                }
                int qmin = (int)((uint32_t)kmin & 31u), qmax = (int)((0xffffffffu - (uint32_t)kmax) & 31u);
                int emin = __shfl_sync(0xffffffffu, eq, qmin), emax = __shfl_sync(0xffffffffu, eq, qmax);
                float bl = shf(lo[c], emin), bh = shf(hi[c], emax);
                cb[side].lo[c] = bl;
                cb[side].hi[c] = bh;
            }
        }
        bool swap = area(cb[0]) > area(cb[1]);
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(next_id, 2u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base + 2u > n_nodes || sp + 2 > (int)kSmall + 1) {
            if (lane == 0) atomicOr(err, 4u);
            return;
        }
        uint32_t id_l = base, id_r = base + 1u;
        if (lane == 0) {
            for (int c = 0; c < 3; c++) {
                nodes[id_l].lo[c] = cb[0].lo[c];
                nodes[id_l].hi[c] = cb[0].hi[c];
                nodes[id_r].lo[c] = cb[1].lo[c];
                nodes[id_r].hi[c] = cb[1].hi[c];
            }
            nodes[id_l].cnt = at;
            nodes[id_r].cnt = mm - at;
            nodes[u].c0 = swap ? id_r : id_l;
            nodes[u].c1 = swap ? id_l : id_r;
        }
        // Element lists of the children (ranks in order); the second child
        // goes below the first on the stack so that the first is built first.
        uint32_t first = swap ? id_r : id_l, second = swap ? id_l : id_r;
        uint32_t first_cnt = swap ? mm - at : at, second_cnt = swap ? at : mm - at;
        uint32_t first_off = swap ? at : 0u, second_off = swap ? 0u : at;
        int v1 = __shfl_sync(0xffffffffu, eq, (int)((first_off + (uint32_t)lane) & 31u));
        int v2 = __shfl_sync(0xffffffffu, eq, (int)((second_off + (uint32_t)lane) & 31u));
        __syncwarp();  // every read of the popped list is done
        if (lane < (int)second_cnt) lists[w][sp][lane] = (uint8_t)v2;
        if (lane < (int)first_cnt) lists[w][sp + 1][lane] = (uint8_t)v1;
        if (lane == 0) {
            st_id[w][sp] = second;
            st_cnt[w][sp] = second_cnt;
            st_id[w][sp + 1] = first;
            st_cnt[w][sp + 1] = first_cnt;
        }
        sp += 2;
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// crystallize (bvh.rs:389-428) and the statistics of bvh.rs:536-545 over the
// interim tree: node 0 is the root, children have larger ids than their
// parents, a leaf's triangles are order[beg .. beg + cnt). The recursion becomes
// a climb from the leaves (subtree sizes, the summed area ratio with the
// operation order of bvh.rs:380-385) and, per node, the walk to the root that
// gives its place in the depth-first order: a node's first child goes to 2 + 2 *
// (internal nodes before it in that order), a leaf's triangles follow those of
// the leaves before it. Latency-bound at these sizes (a few hundred thousand
// nodes, tens of levels); on the host's threads the same took 4.8 ms of a build of
// 81,930 triangles and 27 ms of one of 869,900.

struct Crystal {
    uint32_t* parent;  // 2 * parent's id + (1: second child); kNoParent: none
    uint32_t* arrived;
    uint32_t* inner;  // internal nodes of the subtree
    uint32_t* tris;   // triangles of the subtree
    float* ratio;     // summed area ratio of the subtree
};
constexpr uint32_t kNoParent = 0xffffffffu;

__device__ __forceinline__ Box node_box(const InterimNode& n) {
    Box b;
    for (int c = 0; c < 3; c++) {
        b.lo[c] = n.lo[c];
        b.hi[c] = n.hi[c];
    }
    return b;
}

__global__ void __launch_bounds__(256) k_crystal_parents(const InterimNode* __restrict__ t,
                                                         const uint32_t* __restrict__ count, Crystal x, uint32_t* err) {
    const uint32_t n = *count;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t c0 = t[v].c0, c1 = t[v].c1;
        if (!c0) continue;
        if (c0 <= v || c1 <= v || c0 >= n || c1 >= n) {
            atomicOr(err, 8u);
            continue;
        }
        x.parent[c0] = 2u * v;
        x.parent[c1] = 2u * v + 1u;
    }
}

// One thread per leaf; of the two that reach a node, the second goes on.
__global__ void __launch_bounds__(256) k_crystal_up(const InterimNode* __restrict__ t,
                                                    const uint32_t* __restrict__ count, Crystal x,
                                                    const uint32_t* __restrict__ err) {
    if (*err) return;
    const uint32_t n = *count;
    for (uint32_t leaf = blockIdx.x * blockDim.x + threadIdx.x; leaf < n; leaf += gridDim.x * blockDim.x) {
        if (t[leaf].c0) continue;
        uint32_t v = leaf;
        x.inner[v] = 0u;
        x.tris[v] = t[v].cnt;
        x.ratio[v] = 0.0f;
        while (v != 0u && x.parent[v] != kNoParent) {
            v = x.parent[v] >> 1;
            __threadfence();
            if (atomicAdd(x.arrived + v, 1u) == 0u) break;
            __threadfence();
            const uint32_t c0 = t[v].c0, c1 = t[v].c1;
            x.inner[v] = 1u + __ldcg(x.inner + c0) + __ldcg(x.inner + c1);
            x.tris[v] = __ldcg(x.tris + c0) + __ldcg(x.tris + c1);
            float child_contrib = 0.0f;
            child_contrib += __ldcg(x.ratio + c0);
            child_contrib += __ldcg(x.ratio + c1);
            const float self_area = area(node_box(t[v]));
            float child_sum = 0.0f;
            child_sum += area(node_box(t[c0])) / self_area;
            child_sum += area(node_box(t[c1])) / self_area;
            x.ratio[v] = child_sum + child_contrib;
        }
    }
}

// Places every node but the root, and the triangles of the leaves.
__global__ void __launch_bounds__(256) k_crystal_emit(const InterimNode* __restrict__ t,
                                                      const uint32_t* __restrict__ count, Crystal x,
                                                      const uint32_t* __restrict__ order, uint32_t n_tris,
                                                      const float4* __restrict__ src, cvx_bvh_node* __restrict__ nodes,
                                                      float4* __restrict__ tris, uint32_t* __restrict__ source,
                                                      uint32_t* __restrict__ depth, const uint32_t* __restrict__ err) {
    const uint32_t n = *count;
    // (A tree that lost triangles or nodes is reported by the host from the root's sums.)
    if (*err || x.tris[0] != n_tris || 2u * x.inner[0] != n - 1u) return;
    uint32_t deepest = 0;
    for (uint32_t v = 1u + blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint32_t before = 0, first = 0, levels = 0, own = 0;  // own: what the last step to v added to `before`
        for (uint32_t u = v; u != 0u;) {
            const uint32_t link = x.parent[u], p = link >> 1;
            uint32_t add = p != 0u ? 1u : 0u;
            if (link & 1u) {
                const uint32_t c0 = t[p].c0;
                add += x.inner[c0];
                first += x.tris[c0];
            }
            if (u == v) own = add;
            before += add;
            levels++;
            u = p;
        }
        const InterimNode& nd = t[v];
        const uint32_t link = x.parent[v];
        const uint32_t at = (link >> 1) == 0u ? (link & 1u) : 2u + 2u * (before - own) + (link & 1u);
        cvx_bvh_node o;
        for (int c = 0; c < 3; c++) {
            o.origin[c] = nd.lo[c];
            o.far_[c] = nd.hi[c];
        }
        o.index = nd.c0 ? 2u + 2u * before : first;
        o.len = nd.c0 ? 0u : nd.cnt;
        nodes[at] = o;
        deepest = max(deepest, levels);
        if (nd.c0) continue;
        for (uint32_t j = 0; j < nd.cnt; j++) {
            const uint32_t s = order[nd.beg + j];
            source[first + j] = s;
            for (int q = 0; q < 4; q++) tris[4 * (size_t)(first + j) + q] = src[4 * (size_t)s + q];
        }
    }
    if (deepest) atomicMax(depth, deepest);
}

// ---------------------------------------------------------------------------

struct DevBuf {
    void* p = nullptr;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
};

#define BK(call, what)                                                                             \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) return set_error(CVX_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
static int32_t dalloc(DevBuf& b, size_t count, const char* what) {
    cudaError_t e = cudaMalloc(&b.p, std::max<size_t>(count, 1) * sizeof(T));
    if (e != cudaSuccess) return set_error(CVX_ERR_DEVICE, std::string("device BVH build: ") + what + ": " +
                                                                  cudaGetErrorString(e));
    return CVX_OK;
}

static void tiles_of(std::vector<Tile>& out, uint32_t slot, uint32_t axis, uint32_t beg, uint32_t cnt) {
    for (uint32_t s = 0; s < cnt; s += kTile) out.push_back(Tile{slot, axis, beg + s, std::min<uint32_t>(kTile, cnt - s)});
}

static unsigned blocks(size_t n, unsigned b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

// The lists of a phase, which go up in one copy (a level made eight, and three
// down, and lists that grew by the level: 81,920 triangles 5.77 -> 5.11 ms).
struct Lists {
    std::vector<unsigned char> bytes;
    template <class T>
    size_t add(const std::vector<T>& v) {
        const size_t at = (bytes.size() + 15) / 16 * 16, size = v.size() * sizeof(T);
        bytes.resize(at + size);
        if (size) std::memcpy(bytes.data() + at, v.data(), size);
        return at;
    }
};

int32_t bvh_build_device(const cvx_triangle* tris, uint32_t n, cvx_bvh** out) {
    if (n == 0) return set_error(CVX_ERR_INVALID, "cannot build a BVH of zero triangles");
    if (n > kMaxTris) return set_error(CVX_ERR_CAPACITY, "device BVH build: more than 2^26 triangles");
    std::vector<float> tx, tt;
    float ty;
    tsah_tables(n, tx, tt, &ty);
    std::unique_ptr<cvx_bvh> bvh(new cvx_bvh());
    cudaStream_t st = nullptr;
    BK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "cudaStreamCreate");
    // Host arrays of uploads in flight, kept until the stream has been waited for
    // (the guard, which goes before them and before what is declared above, waits on
    // every way out).
    std::vector<std::shared_ptr<void>> keep;
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() {
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    } guard{st};
    auto upload = [&](void* dst, auto&& host) -> int32_t {
        using V = std::decay_t<decltype(host)>;
        auto v = std::make_shared<V>(std::forward<decltype(host)>(host));
        keep.push_back(v);
        BK(cudaMemcpyAsync(dst, v->data(), v->size() * sizeof((*v)[0]), cudaMemcpyHostToDevice, st), "upload");
        return CVX_OK;
    };

    const uint32_t max_nodes = 2 * n;
    const uint32_t max_slots = n / (kSmall + 1) + 1;

    // The arrays whose sizes are known lie in one allocation: each one of its own
    // takes 20 us to make and 20 to release (81,920 triangles 5.10 -> 4.69 ms).
    size_t total = 0;
    auto place = [&](size_t bytes) {
        const size_t at = total;
        total += (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
        return at;
    };
    const size_t at_tris = place((size_t)n * sizeof(cvx_triangle)), at_refs = place((size_t)9 * n * 4),
                 at_order = place((size_t)n * 4), at_tmp = place((size_t)n * 4), at_srt = place((size_t)3 * n * 4),
                 at_binf = place((size_t)3 * n), at_nodes = place((size_t)max_nodes * sizeof(InterimNode)),
                 at_inner = place((size_t)6 * max_nodes * 4), at_tx = place(((size_t)n + 1) * 4),
                 at_tt = place(((size_t)n + 1) * 4), at_misc = place(4 * 4),
                 at_cnt = place((size_t)max_slots * 3 * kBins * 4), at_key = place((size_t)max_slots * 3 * kBins * 6 * 4),
                 at_mode = place((size_t)max_slots * 3 * 4), at_dec = place(((size_t)max_slots + 1) * sizeof(Decision)),
                 at_out_nodes = place((size_t)max_nodes * sizeof(cvx_bvh_node)),
                 at_out_tris = place((size_t)n * sizeof(cvx_triangle));
    DevBuf d_arrays, d_level, d_split, d_tiles2, d_hist, d_off, d_ids, d_acc, d_sortbuf, d_pairs;
    int32_t s = 0;
    if ((s = dalloc<char>(d_arrays, total, "arrays"))) return s;
    char* const base = (char*)d_arrays.p;
    cvx_triangle* tri_d = (cvx_triangle*)(base + at_tris);
    float* refs = (float*)(base + at_refs);
    Refs R;
    for (int c = 0; c < 3; c++) {
        R.lo[c] = refs + (size_t)c * n;
        R.hi[c] = refs + (size_t)(3 + c) * n;
        R.bc[c] = refs + (size_t)(6 + c) * n;
    }
    uint32_t* order = (uint32_t*)(base + at_order);
    uint32_t* order_tmp = (uint32_t*)(base + at_tmp);
    uint32_t* srt = (uint32_t*)(base + at_srt);
    uint8_t* binf = (uint8_t*)(base + at_binf);
    InterimNode* nodes = (InterimNode*)(base + at_nodes);
    float* inner = (float*)(base + at_inner);
    uint32_t* misc = (uint32_t*)(base + at_misc);  // [0] bad input, [1] error bits, [2] next node id, [3] depth
    BinStats bs{(uint32_t*)(base + at_cnt), (uint32_t*)(base + at_key)};
    float *d_tx = (float*)(base + at_tx), *d_tt = (float*)(base + at_tt);
    Tsah ts{d_tx, d_tt, ty};
    uint32_t* const dm = (uint32_t*)(base + at_mode);
    Decision* const d_dec = (Decision*)(base + at_dec);
    cvx_bvh_node* const out_nodes = (cvx_bvh_node*)(base + at_out_nodes);
    cvx_triangle* const out_tris = (cvx_triangle*)(base + at_out_tris);

    BK(cudaMemcpyAsync(tri_d, tris, (size_t)n * sizeof(cvx_triangle), cudaMemcpyHostToDevice, st), "upload");
    BK(cudaMemcpyAsync(d_tx, tx.data(), tx.size() * 4, cudaMemcpyHostToDevice, st), "upload");
    BK(cudaMemcpyAsync(d_tt, tt.data(), tt.size() * 4, cudaMemcpyHostToDevice, st), "upload");
    BK(cudaMemsetAsync(misc, 0, 16, st), "memset");
    BK(cudaMemsetAsync(nodes, 0, (size_t)max_nodes * sizeof(InterimNode), st), "memset");
    const float third = 1.0f / 3.0f;
    k_prep<<<blocks(n, 256), 256, 0, st>>>(tri_d, n, third, R, order, misc);

    // Host-side copies of every interim node's range.
    std::vector<uint32_t> h_beg(max_nodes, 0), h_cnt(max_nodes, 0);
    uint32_t next_id = 1;
    h_beg[0] = 0;
    h_cnt[0] = n;

    // Scratch that grows with the largest list of a level (to twice what is asked for:
    // an allocation waits for the device).
    size_t cap_level = 0, cap_split = 0, cap_tiles2 = 0, cap_ids = 0, cap_pairs = 0, cap_sort = 0;
    auto ensure = [&](DevBuf& b, size_t& cap, size_t bytes, const char* what) -> int32_t {
        if (bytes <= cap) return CVX_OK;
        if (b.p) cudaFree(b.p);
        b.p = nullptr;
        cap = 0;
        const size_t want = std::max(2 * bytes, (size_t)1 << 20);
        cudaError_t e = cudaMalloc(&b.p, want);
        if (e != cudaSuccess)
            return set_error(CVX_ERR_DEVICE, std::string("device BVH build: ") + what + ": " + cudaGetErrorString(e));
        cap = want;
        return CVX_OK;
    };
    size_t cap_hist = 0, cap_off = 0, cap_acc = 0;
    auto upload_lists = [&](DevBuf& b, size_t& cap, Lists& l) -> int32_t {
        int32_t e = ensure(b, cap, l.bytes.size(), "lists");
        return e ? e : upload(b.p, std::move(l.bytes));
    };

    // Exact boxes of the `count` interim nodes from `first` on, whose tiles are `tl`
    // (slot: index from `first`).
    auto node_boxes = [&](uint32_t first, uint32_t count, const Tile* tl, uint32_t n_tl) -> int32_t {
        int32_t e = ensure(d_acc, cap_acc, count * sizeof(BoxAcc), "boxes");
        if (e) return e;
        k_box_init<<<blocks(count, 128), 128, 0, st>>>((BoxAcc*)d_acc.p, count);
        k_box<<<n_tl, kTile, 0, st>>>(tl, n_tl, R, order, n, (BoxAcc*)d_acc.p, count, misc + 1);
        k_box_store<<<blocks(3 * (size_t)count, 128), 128, 0, st>>>(first, count, (const BoxAcc*)d_acc.p, R, order, n,
                                                                    nodes, max_nodes, inner, misc + 1);
        return CVX_OK;
    };

    // Root: range [0, n) in input order.
    const InterimNode r0{{0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}, 0u, n, 0u, 0u};
    {
        BK(cudaMemcpyAsync(nodes, &r0, sizeof r0, cudaMemcpyHostToDevice, st), "upload");
        std::vector<Tile> tl;
        tiles_of(tl, 0, 0, 0, n);
        const uint32_t n_tl = (uint32_t)tl.size();
        Lists l;
        l.add(tl);
        if ((s = upload_lists(d_split, cap_split, l)) || (s = node_boxes(0, 1, (const Tile*)d_split.p, n_tl))) return s;
    }
    uint32_t bad = 0;
    BK(cudaMemcpyAsync(&bad, misc, 4, cudaMemcpyDeviceToHost, st), "flags");
    BK(cudaStreamSynchronize(st), "root");
    keep.clear();
    if (bad)
        return set_error(CVX_ERR_INVALID,
                         "device BVH build: NaN or infinite vertex coordinates (the host build takes them)");

    std::vector<uint32_t> active, small;
    if (n > kSmall) active.push_back(0);
    else if (n >= 2) small.push_back(0);

    while (!active.empty()) {
        const uint32_t K = (uint32_t)active.size();
        std::vector<Slot> slots(K);
        std::vector<Tile> tl;
        for (uint32_t k = 0; k < K; k++) {
            uint32_t id = active[k];
            slots[k] = Slot{id, h_beg[id], h_cnt[id]};
            tiles_of(tl, k, 0, h_beg[id], h_cnt[id]);
        }
        const uint32_t n_tl = (uint32_t)tl.size();
        Lists lists;
        const size_t at_slots = lists.add(slots), at_tiles = lists.add(tl);
        if ((s = upload_lists(d_level, cap_level, lists))) return s;
        const Slot* ds = (const Slot*)((const char*)d_level.p + at_slots);
        const Tile* dt = (const Tile*)((const char*)d_level.p + at_tiles);
        k_stats_init<<<blocks((size_t)K * 3 * kBins, 256), 256, 0, st>>>(bs, K * 3 * kBins);
        k_bin_float<<<n_tl, kTile, 0, st>>>(dt, n_tl, ds, K, R, order, n, inner, binf, bs, misc + 1);
        k_fallback<<<blocks((size_t)K * 3 * 32, 128), 128, 0, st>>>(ds, K, bs, dm);
        // Uniform split (bvh.rs:176-201) where coordinate binning fell back.
        k_sort_slots<<<3 * K, 1024, 0, st>>>(ds, K, dm, R, order, n, srt, misc + 1);
        k_uniform_stats<<<dim3(n_tl, 3), kTile, 0, st>>>(dt, n_tl, dm, ds, K, R, order, n, srt, bs, misc + 1);
        k_choose<<<K, 96, 0, st>>>(ds, K, nodes, bs, ts, dm, misc + 1, d_dec);
        std::vector<Decision> dec((size_t)K + 1);
        auto decisions = [&]() -> int32_t {
            BK(cudaMemcpyAsync(dec.data(), d_dec, dec.size() * sizeof(Decision), cudaMemcpyDeviceToHost, st),
               "download");
            BK(cudaStreamSynchronize(st), "split choice");
            keep.clear();
            if (dec[K].flags) return set_error(CVX_ERR_DEVICE, "device BVH build: internal range check failed");
            return CVX_OK;
        };
        if ((s = decisions())) return s;
        auto uniform = [&](uint32_t k, uint32_t a) { return (dec[k].flags >> (1 + a) & 1u) != 0u; };

        // Uniform splits too large for one block: sorted through global memory,
        // and the level's choice made again.
        std::vector<Tile> uni_tiles, big_pairs;
        for (uint32_t k = 0; k < K; k++)
            for (uint32_t a = 0; a < 3; a++)
                if (uniform(k, a) && slots[k].cnt > kBlockSort) {
                    const Tile pr{k, a, slots[k].beg, slots[k].cnt};
                    big_pairs.push_back(pr);
                    for (uint32_t r0 = 0; r0 < pr.len; r0 += kTile)
                        uni_tiles.push_back(Tile{k, a, r0, std::min<uint32_t>(kTile, pr.len - r0)});
                }
        if (!big_pairs.empty()) {
            const uint32_t n_uni = (uint32_t)uni_tiles.size();
            if ((s = ensure(d_pairs, cap_pairs, big_pairs.size() * sizeof(Tile), "pairs")) ||
                (s = ensure(d_tiles2, cap_tiles2, n_uni * sizeof(Tile), "tiles")) ||
                (s = upload(d_pairs.p, big_pairs)) || (s = upload(d_tiles2.p, std::move(uni_tiles))))
                return s;
            for (const Tile& pr : big_pairs) {
                uint32_t m2 = 4096;
                while (m2 < pr.len) m2 <<= 1;
                if ((s = ensure(d_sortbuf, cap_sort, (size_t)m2 * 8, "sort buffer"))) return s;
                unsigned long long* buf = (unsigned long long*)d_sortbuf.p;
                k_sort_fill<<<blocks(m2, 256), 256, 0, st>>>(pr, m2, R, order, buf);
                // stages 2..4096 inside chunks, then the larger ones
                k_sort_chunk<<<m2 / 4096, 1024, 0, st>>>(buf, m2, 2, 4096, 1);
                for (uint32_t size = 8192; size <= m2; size <<= 1) {
                    uint32_t j = size >> 1;
                    for (; j >= 4096; j >>= 1) k_sort_step<<<blocks(m2, 256), 256, 0, st>>>(buf, m2, size, j);
                    k_sort_chunk<<<m2 / 4096, 1024, 0, st>>>(buf, m2, size, size, j);
                }
                k_sort_extract<<<blocks(pr.len, 256), 256, 0, st>>>(pr, buf, n, srt);
            }
            k_axis_reset<<<blocks(big_pairs.size() * kBins, 256), 256, 0, st>>>((const Tile*)d_pairs.p,
                                                                               (uint32_t)big_pairs.size(), bs);
            k_uniform_stats<<<n_uni, kTile, 0, st>>>((const Tile*)d_tiles2.p, n_uni, nullptr, ds, K, R, order, n, srt,
                                                     bs, misc + 1);
            k_choose<<<K, 96, 0, st>>>(ds, K, nodes, bs, ts, dm, misc + 1, d_dec);
            if ((s = decisions())) return s;
        }

        // Partition the split slots.
        std::vector<Tile> part;            // axis: 0..2 coordinate bins, 3..5 uniform
        std::vector<uint32_t> slot_tiles;  // per coordinate-binned split slot: [t0, t1) in `fl`
        std::vector<Tile> fl;              // coordinate-binned tiles (for the histograms)
        std::vector<Tile> boxes;           // of the children
        std::vector<Link> links;
        std::vector<uint32_t> next_active;
        const uint32_t first_child = next_id;
        for (uint32_t k = 0; k < K; k++) {
            const Decision& d = dec[k];
            if (d.flags & 1u) continue;
            if (d.axis > 2 || d.nl == 0 || d.nl >= slots[k].cnt)
                return set_error(CVX_ERR_DEVICE, "device BVH build: bad split");
            if (uniform(k, d.axis)) {
                tiles_of(part, k, 3 + d.axis, slots[k].beg, slots[k].cnt);
            } else {
                uint32_t t0 = (uint32_t)fl.size();
                tiles_of(fl, k, d.axis, slots[k].beg, slots[k].cnt);
                slot_tiles.push_back(t0);
                slot_tiles.push_back((uint32_t)fl.size());
            }
            const uint32_t l = next_id, r = next_id + 1;
            next_id += 2;
            if (next_id > max_nodes) return set_error(CVX_ERR_DEVICE, "device BVH build: node overflow");
            h_beg[l] = slots[k].beg;
            h_cnt[l] = d.nl;
            h_beg[r] = slots[k].beg + d.nl;
            h_cnt[r] = slots[k].cnt - d.nl;
            links.push_back(Link{slots[k].id, l, slots[k].beg, d.nl, slots[k].cnt});
            for (uint32_t c : {l, r}) {
                tiles_of(boxes, c - first_child, 0, h_beg[c], h_cnt[c]);
                if (h_cnt[c] > kSmall) next_active.push_back(c);
                else if (h_cnt[c] >= 2) small.push_back(c);
            }
        }
        if (!links.empty()) {
            // coordinate-binned tiles first (their block index is the tile_off row), then uniform
            const size_t n_fl = fl.size();
            fl.insert(fl.end(), part.begin(), part.end());
            const uint32_t n_all = (uint32_t)fl.size(), n_links = (uint32_t)links.size(),
                           n_boxes = (uint32_t)boxes.size();
            Lists sl;
            const size_t at_all = sl.add(fl), at_st = sl.add(slot_tiles), at_boxes = sl.add(boxes),
                         at_links = sl.add(links);
            if ((s = upload_lists(d_split, cap_split, sl)) ||
                (s = ensure(d_hist, cap_hist, std::max<size_t>(n_fl, 1) * kBins * 4, "histograms")) ||
                (s = ensure(d_off, cap_off, std::max<size_t>(n_fl, 1) * kBins * 4, "offsets")))
                return s;
            const char* lb = (const char*)d_split.p;
            const Tile* d_all = (const Tile*)(lb + at_all);
            if (n_fl) {
                k_tile_hist<<<(unsigned)n_fl, kTile, 0, st>>>(d_all, (uint32_t)n_fl, binf, n, (uint32_t*)d_hist.p);
                k_tile_offsets<<<(unsigned)(slot_tiles.size() / 2), 1024, 0, st>>>(
                    (const uint32_t*)(lb + at_st), (uint32_t)(slot_tiles.size() / 2), (const uint32_t*)d_hist.p,
                    (uint32_t*)d_off.p);
            }
            k_scatter<<<n_all, kTile, 0, st>>>(d_all, n_all, ds, K, binf, srt, (const uint32_t*)d_off.p, order, n,
                                               order_tmp, misc + 1);
            k_copy_back<<<n_all, kTile, 0, st>>>(d_all, n_all, order_tmp, order, n);
            // Children: exact boxes, then the parents' links and the ranges.
            if ((s = node_boxes(first_child, 2 * n_links, (const Tile*)(lb + at_boxes), n_boxes))) return s;
            k_link<<<blocks(n_links, 128), 128, 0, st>>>((const Link*)(lb + at_links), n_links, nodes, max_nodes,
                                                         misc + 1);
        }
        active.swap(next_active);
    }

    if (!small.empty()) {
        if ((s = ensure(d_ids, cap_ids, small.size() * 4, "ids"))) return s;
        if ((s = upload(d_ids.p, small))) return s;
        BK(cudaMemcpyAsync(misc + 2, &next_id, 4, cudaMemcpyHostToDevice, st), "upload");
        k_small<<<blocks(small.size(), kSmallWarps), 32 * kSmallWarps, 0, st>>>(
            (const uint32_t*)d_ids.p, (uint32_t)small.size(), nodes, max_nodes, misc + 2, order, n, R, ts, misc + 1);
    }
    else BK(cudaMemcpyAsync(misc + 2, &next_id, 4, cudaMemcpyHostToDevice, st), "upload");

    // The reference's node array and triangle order. The boxes of the levels
    // are no longer needed: their memory holds the crystallization's state.
    uint32_t* state = (uint32_t*)inner;  // 6 * max_nodes words
    const Crystal cr{state, state + max_nodes, state + 2 * (size_t)max_nodes, state + 3 * (size_t)max_nodes,
                     (float*)(state + 4 * (size_t)max_nodes)};
    BK(cudaMemsetAsync(cr.parent, 0xff, (size_t)max_nodes * 4, st), "memset");
    BK(cudaMemsetAsync(cr.arrived, 0, (size_t)max_nodes * 4, st), "memset");
    const unsigned cb = std::min(blocks(max_nodes, 256), 4096u);
    k_crystal_parents<<<cb, 256, 0, st>>>(nodes, misc + 2, cr, misc + 1);
    k_crystal_up<<<cb, 256, 0, st>>>(nodes, misc + 2, cr, misc + 1);
    k_crystal_emit<<<cb, 256, 0, st>>>(nodes, misc + 2, cr, order, n, (const float4*)tri_d,
                                       out_nodes, (float4*)out_tris, order_tmp, misc + 3,
                                       misc + 1);
    BK(cudaGetLastError(), "crystallize");
    // The result's memory, while the kernels run. There are one (room, tube) to two
    // (icosphere) nodes per triangle: room for the most there can be, which is not
    // resident until it is used, and the pages of five for four triangles.
    bvh->nodes.reserve(max_nodes);
    bvh->nodes.resize(std::min<size_t>(max_nodes, (size_t)n + n / 4));
    bvh->triangles.resize(n);
    bvh->source_index.resize(n);
    touch_pages(bvh->nodes.data(), bvh->nodes.size() * sizeof(cvx_bvh_node));
    touch_pages(bvh->triangles.data(), (size_t)n * sizeof(cvx_triangle));
    touch_pages(bvh->source_index.data(), (size_t)n * 4);
    uint32_t flags[4], root_c0 = 0, root_inner = 0, root_tris = 0;
    float root_ratio = 0.0f;
    BK(cudaMemcpyAsync(flags, misc, sizeof flags, cudaMemcpyDeviceToHost, st), "download");
    BK(cudaMemcpyAsync(&root_c0, &nodes[0].c0, 4, cudaMemcpyDeviceToHost, st), "download");
    BK(cudaMemcpyAsync(&root_inner, cr.inner, 4, cudaMemcpyDeviceToHost, st), "download");
    BK(cudaMemcpyAsync(&root_tris, cr.tris, 4, cudaMemcpyDeviceToHost, st), "download");
    BK(cudaMemcpyAsync(&root_ratio, cr.ratio, 4, cudaMemcpyDeviceToHost, st), "download");
    BK(cudaStreamSynchronize(st), "crystallize");
    if (flags[1] & 8u) return set_error(CVX_ERR_DEVICE, "device BVH build: malformed interim tree");
    if (flags[1]) return set_error(CVX_ERR_DEVICE, "device BVH build: internal range check failed");
    next_id = flags[2];
    if (next_id > max_nodes) return set_error(CVX_ERR_DEVICE, "device BVH build: node overflow");
    if (!root_c0)
        return set_error(CVX_ERR_INVALID,
                         "the BVH root did not split: the reference needs at least two root nodes (bvh.rs:509-512)");
    if (root_tris != n) return set_error(CVX_ERR_DEVICE, "device BVH build lost triangles");
    if (2u * root_inner != next_id - 1u)
        return set_error(CVX_ERR_DEVICE, "device BVH build: unreachable interim nodes");
    const size_t m = 2 * (size_t)root_inner, touched = bvh->nodes.size();
    bvh->nodes.resize(m);
    if (m > touched) touch_pages(bvh->nodes.data() + touched, (m - touched) * sizeof(cvx_bvh_node));
    BK(cudaMemcpyAsync(bvh->nodes.data(), out_nodes, m * sizeof(cvx_bvh_node), cudaMemcpyDeviceToHost, st),
       "download");
    BK(cudaMemcpyAsync(bvh->triangles.data(), out_tris, (size_t)n * sizeof(cvx_triangle), cudaMemcpyDeviceToHost,
                       st),
       "download");
    BK(cudaMemcpyAsync(bvh->source_index.data(), order_tmp, (size_t)n * 4, cudaMemcpyDeviceToHost, st), "download");
    BK(cudaStreamSynchronize(st), "download");
    bvh->depth = flags[3];
    bvh->avg_area_ratio = root_ratio / (float)(m + 1);  // the crystallized nodes and the root
    bvh->avg_tris_per_leaf = (float)n / (float)((size_t)root_inner + 1);
    *out = bvh.release();
    return CVX_OK;
}

}  // namespace cvx

extern "C" int32_t cvx_bvh_build_device(const cvx_triangle* triangles, uint32_t n, cvx_bvh** out) {
    if (!out || (!triangles && n)) return cvx::set_error(CVX_ERR_INVALID, "null argument");
    return cvx::bvh_build_device(triangles, n, out);
}
