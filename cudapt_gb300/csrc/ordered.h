// Layout of the ordered walk's tree (made by ordered_tree.cpp, walked by ordered.cuh).
#pragma once
#include <cstdint>
#include <memory>

namespace gbpt {

// node, 24 words:  base.xyz, 32768 * cell.xyz, first child node | inner mask << 24,
//                  first leaf record | binary inner nodes it stands for << 24,
//                  per axis 8 low and 8 high child planes (bytes: base + q * cell),
//                  4 unused; children fill the slots from 0 in the reference's leaf order
// leaf, 16 words:  p0, p1 - p0, p2 - p0, box min, box max, triangle id (or kOrdManyTris | first
//                  id, with the triangle count in word 0)
constexpr uint32_t kOrdWidth = 8, kOrdNodeWords = 24, kOrdLeafWords = 16;
constexpr uint32_t kOrdMaxIndex = 1u << 24, kOrdManyTris = 0x80000000u;
constexpr uint32_t kOrdStack = 20;  // stack entries of a walk: at most one per level below the root

struct OrderedTree {
  std::unique_ptr<float[]> nodes;      // nodeN x kOrdNodeWords
  std::unique_ptr<uint32_t[]> leaves;  // binary leaf of each leaf record
  uint32_t nodeN = 0, leafN = 0;
  float range = 0.f;  // largest |origin coordinate| the walk is exact for
};

}  // namespace gbpt
