// Shared host-side helpers of libconvector_gpu (not part of the C-ABI).
#pragma once
#include <cstdint>
#include <memory>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "../../include/convector_gpu.h"

namespace cvx {

int32_t set_error(int32_t status, const std::string& msg);

// Allocation-failure injection (cvx_inject_allocation_failure): called by the
// library's device-allocation helpers before each cudaMalloc; true when this
// allocation is to fail as if the device were out of memory.
bool injected_allocation_failure();

// Makes the pages of an output buffer present and writable before the device or a
// copy fills it. Pages the process has not used yet (a fresh large allocation) cost
// the driver's copies and the device's stores several times what they cost the CPU,
// and the CPU can do it while the kernels run. touch_pages stores a zero in each: for
// a buffer that is filled whole unless the device itself fails. populate_pages
// leaves the contents as they are, for calls that may yet return without filling
// it. Two images of 3.8 MB, fresh, on 64 KB pages, us: copied untouched 490; touched
// 249 and copied 83, populated 233 and 84. (A byte read and stored back, or exchanged
// for itself, 2,750: the read maps the shared zero page, and taking it away again
// invalidates the device's translations.) Where the pages are in use a touch costs 1
// us, but the system call 5 (a 320x184 frame 199 -> 205 us).
void touch_pages(void* p, size_t bytes);
void populate_pages(void* p, size_t bytes);

// Whether a kernel may access a caller's array of 32-bit values in place: copies
// take any address, a device's loads and stores only multiples of the size.
inline bool word_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3u) == 0u; }

// A node of the interim tree of the device BVH build (bvh.rs:52-62): its
// exact bounding box, its triangles order[beg .. beg + cnt) and its children
// (c0 == 0: a leaf; node 0 is the root and never a child).
struct InterimNode {
    float lo[3], hi[3];
    uint32_t beg, cnt;
    uint32_t c0, c1;
};

// TSAH factors for triangle counts 0..n (index 0 unused) and the constant
// denominator, as the host build computes them.
void tsah_tables(uint32_t n, std::vector<float>& x, std::vector<float>& t, float* y);
// A vector whose resize() leaves plain data uninitialised (it is filled whole
// right after).
template <class T>
struct NoInit : std::allocator<T> {
    template <class U>
    struct rebind {
        using other = NoInit<U>;
    };
    NoInit() = default;
    template <class U>
    NoInit(const NoInit<U>&) {}
    template <class U>
    void construct(U* p) {
        ::new ((void*)p) U;
    }
    template <class U, class... A>
    void construct(U* p, A&&... a) {
        ::new ((void*)p) U(std::forward<A>(a)...);
    }
};

struct MeshTri {
    uint32_t v[3];
    int64_t t[3];  // -1: the face has no texture coordinates
    uint32_t material;
};

}  // namespace cvx

struct cvx_mesh {
    std::vector<float> vertices;    // 3 per vertex
    std::vector<float> tex_coords;  // 2 per coordinate
    std::vector<cvx::MeshTri> triangles;
};

struct cvx_bvh {
    std::vector<cvx_bvh_node, cvx::NoInit<cvx_bvh_node>> nodes;
    std::vector<cvx_triangle, cvx::NoInit<cvx_triangle>> triangles;  // BVH (leaf) order
    std::vector<uint32_t, cvx::NoInit<uint32_t>> source_index;  // input index of each BVH-order triangle
    float avg_area_ratio = 0.0f;
    float avg_tris_per_leaf = 0.0f;
    uint32_t depth = 0;
};
