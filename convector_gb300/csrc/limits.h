// Limits that host and device code share.
#pragma once
#include <cstdint>

namespace cvx {

constexpr int kStackDepth = 128;  // >= BVH depth + 2 (checked at scene creation)
// Up to three boxes of a wide record wait on the stack: at most 1.5 per level.
constexpr uint32_t kWideMaxDepth = (kStackDepth - 8) / 3 * 2;
constexpr uint32_t kWideMaxPairs = 1u << 25;  // 32-bit offsets into the records
// Largest bound, origin and reciprocal of a ray on the wide records (traverse.cuh).
constexpr float kSelectMax = 1.0e18f;

}  // namespace cvx
