// Host side of the ordered walk (ordered.cuh): the binary tree of
// bvh_build.cpp collapsed to nodes of up to eight children that keep the order
// in which the reference's walk reaches leaves, with child boxes in 8 bits a
// plane, and one 64-byte record per leaf (its exact box and its triangle).
#include <cmath>
#include <cstring>

#include "gbpt_internal.h"

namespace gbpt {

namespace {

constexpr uint32_t kW = kOrdWidth;

float bits(uint32_t u) {
  float f;
  std::memcpy(&f, &u, 4);
  return f;
}

// cost[i] (1..8): least expected node visits (summed box areas) to cover a
// binary subtree with at most i children of one wide node; split[i]: how many
// of them the left subtree takes, 0 when i - 1 are as good; split[1] is the
// split of the eight children of a wide node made of the subtree itself.
struct Plan {
  float cost[kW + 1];
  uint8_t split[kW + 1];
};

struct Collapse {
  const HostBVH& bvh;
  std::vector<Plan> plan;
  explicit Collapse(const HostBVH& b) : bvh(b), plan(b.nodeN) {}

  bool inner(uint32_t i) const { return bvh.offOrTSTN[2 * (size_t)i + 1] == 0; }
  uint32_t left(uint32_t i) const { return i + 1; }
  uint32_t right(uint32_t i) const { return i + bvh.offOrTSTN[2 * (size_t)i]; }
  const float* box(uint32_t i) const { return &bvh.bounds[6 * (size_t)i]; }
  float area(uint32_t i) const {
    const float* b = box(i);
    const float x = b[3] - b[0], y = b[4] - b[1], z = b[5] - b[2];
    return x * y + y * z + z * x;
  }

  void make_plan() {
    for (uint32_t n = bvh.nodeN; n-- > 0;) {  // children have larger indices
      Plan& p = plan[n];
      const float a = area(n);
      if (!inner(n)) {
        for (uint32_t i = 1; i <= kW; i++) p.cost[i] = 0.5f * a, p.split[i] = 0;
        continue;
      }
      const float *l = plan[left(n)].cost, *r = plan[right(n)].cost;
      float best[kW + 1];
      uint8_t at[kW + 1];
      for (uint32_t i = 2; i <= kW; i++) {
        best[i] = l[1] + r[i - 1];
        at[i] = 1;
        for (uint32_t k = 2; k < i; k++)
          if (l[k] + r[i - k] < best[i]) best[i] = l[k] + r[i - k], at[i] = (uint8_t)k;
      }
      p.cost[1] = a + best[kW];
      p.split[1] = at[kW];
      for (uint32_t i = 2; i <= kW; i++) {
        const bool split = best[i] < p.cost[i - 1];
        p.cost[i] = split ? best[i] : p.cost[i - 1];
        p.split[i] = split ? at[i] : 0;
      }
    }
  }

  // children of a wide node in the reference's order (right subtree first)
  void children(uint32_t n, uint32_t slots, bool root, uint32_t* out, uint32_t& count, uint32_t& innerN) const {
    if (inner(n)) {
      uint32_t i = slots;
      if (!root)
        while (i > 1 && plan[n].split[i] == 0) i--;
      if (root || i > 1) {
        const uint32_t s = root ? plan[n].split[1] : plan[n].split[i];
        innerN++;
        children(right(n), i - s, false, out, count, innerN);
        children(left(n), s, false, out, count, innerN);
        return;
      }
    }
    out[count++] = n;
  }
};

}  // namespace

bool ordered_tree(const HostBVH& bvh, const float* tris, OrderedTree* out) {
  *out = OrderedTree{};
  const uint32_t n = bvh.nodeN, nt = (uint32_t)bvh.order.size();
  if (n == 0 || bvh.emptyChildren || n >= kOrdMaxIndex || nt >= kOrdMaxIndex) return false;
  Collapse c(bvh);
  // the walk's exactness rests on boxes inside their parents' boxes and on no
  // subtree being dropped by the reference's 29-entry stack test: an inner node
  // reached by r right turns is popped with r - 1 entries below it
  float M = 0.f;
  for (int k = 0; k < 6; k++) M = std::fmax(M, std::fabs(bvh.bounds[k]));
  if (!(M >= 1e-3f && M <= 1e9f)) return false;
  std::vector<uint8_t> turns(n, 0), depth(n, 0);
  for (uint32_t i = 0; i < n; i++) {
    if (!c.inner(i)) {
      const uint64_t first = bvh.offOrTSTN[2 * (size_t)i], cnt = bvh.offOrTSTN[2 * (size_t)i + 1];
      if (first + cnt > nt) return false;
      continue;
    }
    const uint32_t kids[2] = {c.left(i), c.right(i)};
    if (turns[i] > 29 || depth[i] > 60) return false;
    for (uint32_t k = 0; k < 2; k++) {
      if (kids[k] <= i || kids[k] >= n) return false;
      turns[kids[k]] = (uint8_t)(turns[i] + k);
      depth[kids[k]] = (uint8_t)(depth[i] + 1);
      const float *p = c.box(i), *q = c.box(kids[k]);
      for (int a = 0; a < 3; a++)
        if (!(q[a] >= p[a] && q[3 + a] <= p[3 + a] && q[a] <= q[3 + a])) return false;
    }
  }
  c.make_plan();

  // Every plane is moved outwards by `margin` before it is quantised.  With u =
  // 2^-24 and |origin| <= 8 M, in units of the axis (distance times direction):
  // the walk's plane is off by at most 27 u M + 2^-9 cells, the reference's by
  // 18 u M, and scaling by the closest hit adds 4 u of a distance of at most 9 M
  // to each of the two that are compared: 128 u M and 2^-7 cells cover all.
  const double margin = std::ldexp((double)M, -17);
  out->range = 8.f * M;
  struct Item {
    uint32_t bin, wide, depth;
  };
  std::vector<Item> todo{{0u, 0u, 1u}};
  out->nodes.resize(kOrdNodeWords);
  out->leaves.reserve((size_t)nt * kOrdLeafWords);
  while (!todo.empty()) {
    const Item it = todo.back();
    todo.pop_back();
    if (it.depth > kOrdStack + 1) return false;
    uint32_t kid[kW], count = 0, innerN = 0;
    c.children(it.bin, kW, true, kid, count, innerN);
    float node[kOrdNodeWords] = {0.f};
    uint8_t q[6][8];
    const float* nb = c.box(it.bin);
    for (int a = 0; a < 3; a++) {
      const double lo = (double)nb[a] - margin, hi = (double)nb[3 + a] + margin, cell = (hi - lo) / 253.0;
      const float base = std::nextafterf((float)(lo - cell / 32), -INFINITY);
      const float scale = std::nextafterf((float)((hi + cell / 32 - (double)base) / 254.5), INFINITY);
      node[a] = base;
      node[3 + a] = scale * 32768.f;
      for (uint32_t k = 0; k < 8; k++) {
        q[a][k] = 255, q[3 + a][k] = 0;  // an empty slot: its near planes lie behind its far ones
        if (k >= count) continue;
        const float* b = c.box(kid[k]);
        const double l = std::floor(((double)b[a] - margin - (double)base) / (double)scale - 0x1p-7);
        const double h = std::ceil(((double)b[3 + a] + margin - (double)base) / (double)scale + 0x1p-7);
        if (!(l >= 0.0 && h <= 255.0)) return false;
        q[a][k] = (uint8_t)l;
        q[3 + a][k] = (uint8_t)h;
      }
    }
    uint32_t imask = 0, kids = 0;
    const uint32_t childBase = (uint32_t)(out->nodes.size() / kOrdNodeWords);
    const uint32_t leafBase = (uint32_t)(out->leaves.size() / kOrdLeafWords);
    for (uint32_t k = 0; k < count; k++) {
      if (c.inner(kid[k])) {
        imask |= 1u << k;
        todo.push_back({kid[k], childBase + kids++, it.depth + 1});
        continue;
      }
      const uint32_t first = bvh.offOrTSTN[2 * (size_t)kid[k]], cnt = bvh.offOrTSTN[2 * (size_t)kid[k] + 1];
      float leaf[kOrdLeafWords];
      const float* tr = tris + 16 * (size_t)first;
      for (int a = 0; a < 3; a++) leaf[a] = tr[a], leaf[3 + a] = tr[4 + a], leaf[6 + a] = tr[8 + a];
      for (int a = 0; a < 6; a++) leaf[9 + a] = c.box(kid[k])[a];
      leaf[15] = bits(first);
      if (cnt != 1) {  // several triangles: the record names them, the walk reads them from the triangle array
        leaf[0] = bits(cnt);
        leaf[15] = bits(first | kOrdManyTris);
      }
      out->leaves.insert(out->leaves.end(), leaf, leaf + kOrdLeafWords);
    }
    if (childBase + kids >= kOrdMaxIndex || leafBase + count >= kOrdMaxIndex) return false;
    out->nodes.resize(out->nodes.size() + (size_t)kids * kOrdNodeWords, 0.f);
    node[6] = bits(childBase | imask << 24);
    node[7] = bits(leafBase | innerN << 24);
    for (int p = 0; p < 3; p++) {  // per axis: low planes of children 0-3, 4-7, high planes of 0-3, 4-7
      std::memcpy(&node[8 + 4 * p], q[p], 8);
      std::memcpy(&node[10 + 4 * p], q[3 + p], 8);
    }
    std::memcpy(&out->nodes[(size_t)it.wide * kOrdNodeWords], node, sizeof(node));
  }
  return true;
}

}  // namespace gbpt
