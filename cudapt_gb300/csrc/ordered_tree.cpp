// Host side of the ordered walk (ordered.cuh): the binary tree of
// bvh_build.cpp collapsed to nodes of up to eight children that keep the order
// in which the reference's walk reaches leaves, with child boxes in 8 bits a
// plane (compressed wide BVHs and their least-cost collapse: Ylitie, Karras and
// Laine, HPG 2017), and the binary leaf of every leaf record (the device fills
// the records in from the arrays it has: launch_ord_leaves).
//
// Binary subtrees are index ranges, so checks and plan run over some 64 of them
// on several threads, and so does the making of the nodes below the top ones.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <exception>
#include <memory>
#include <new>
#include <thread>

#include "gbpt_internal.h"

namespace gbpt {

namespace {

constexpr uint32_t kW = kOrdWidth;

// The most that the outward margin may make of the leaf boxes' summed area, which
// the leaves a ray visits grow with.  Scenes moved away from the origin, node-by-node
// walk / this one (200,000 rays; 640x360 passes): at 1.6 finer interior 1.37 / 1.35,
// at 1.9 hall 1.23 / 1.37, at 2.2 interior 1.17 / 1.19, finer 1.15 / 1.22, at 2.9
// finer 1.04 / 1.01, at 3.3 hall 0.94 / 0.91, at 4.0 interior 0.75 / 0.79, at 110 hall
// 0.15 / 0.09.  In a small tree there is less to gain: Cornell at 1.09 1.26 / 1.17,
// at 1.27 1.12 / 0.98, at 2.0 0.99 / 0.91.  Unmoved scenes are at 1.00 to 1.01.
double most_growth(uint32_t nodes) { return nodes <= 2048u ? 1.25 : 2.0; }

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
  std::unique_ptr<Plan[]> plan;  // written by make_plan: not cleared first
  explicit Collapse(const HostBVH& b) : bvh(b), plan(new Plan[b.nodeN]) {}

  bool inner(uint32_t i) const { return bvh.offOrTSTN[2 * (size_t)i + 1] == 0; }
  uint32_t left(uint32_t i) const { return i + 1; }
  uint32_t right(uint32_t i) const { return i + bvh.offOrTSTN[2 * (size_t)i]; }
  const float* box(uint32_t i) const { return &bvh.bounds[6 * (size_t)i]; }
  float area(uint32_t i) const {
    const float* b = box(i);
    const float x = b[3] - b[0], y = b[4] - b[1], z = b[5] - b[2];
    return x * y + y * z + z * x;
  }
  // area() of the box with every plane `out` further outwards
  double grown(uint32_t i, double out) const {
    const float* b = box(i);
    const double x = (double)b[3] - b[0] + 2 * out, y = (double)b[4] - b[1] + 2 * out, z = (double)b[5] - b[2] + 2 * out;
    return x * y + y * z + z * x;
  }

  // nodes from .. to - 1, whose children are in the range or planned already
  void make_plan(uint32_t from, uint32_t to) {
    for (uint32_t n = to; n-- > from;) {  // children have larger indices
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

struct Item {
  uint32_t bin, wide, depth;
};

// Wide nodes and leaves of a part of the tree, numbered within the part.
struct Part {
  std::vector<float> nodes;
  std::vector<uint32_t> leaves;  // binary leaf of each leaf record
  std::vector<Item> todo;
};

// Makes node `it` of the part: its children are appended to the part's todo.
bool emit(const Collapse& c, double margin, const Item& it, Part& out) {
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
  const size_t childBase = out.nodes.size() / kOrdNodeWords, leafBase = out.leaves.size();
  if (childBase + kW >= kOrdMaxIndex || leafBase + kW >= kOrdMaxIndex) return false;
  for (uint32_t k = 0; k < count; k++) {
    if (c.inner(kid[k])) {
      imask |= 1u << k;
      out.todo.push_back({kid[k], (uint32_t)childBase + kids++, it.depth + 1});
    } else {
      out.leaves.push_back(kid[k]);
    }
  }
  out.nodes.resize(out.nodes.size() + (size_t)kids * kOrdNodeWords, 0.f);
  node[6] = bits((uint32_t)childBase | imask << 24);
  node[7] = bits((uint32_t)leafBase | innerN << 24);
  for (int p = 0; p < 3; p++) {  // per axis: low planes of children 0-3, 4-7, high planes of 0-3, 4-7
    std::memcpy(&node[8 + 4 * p], q[p], 8);
    std::memcpy(&node[10 + 4 * p], q[3 + p], 8);
  }
  std::memcpy(&out.nodes[(size_t)it.wide * kOrdNodeWords], node, sizeof(node));
  return true;
}

// f(0) .. f(n - 1), each once, on up to `threads` threads; false when one said so or ran out of memory
template <typename F>
bool each(size_t n, uint32_t threads, const F& f) {
  std::atomic<size_t> next{0};
  std::atomic<bool> ok{true};
  auto work = [&]() {
    try {
      for (size_t i; ok && (i = next.fetch_add(1)) < n;)
        if (!f(i)) ok = false;
    } catch (const std::bad_alloc&) {
      ok = false;
    }
  };
  std::vector<std::thread> more;
  more.reserve(threads);
  for (uint32_t k = 1; k < threads && k < n; k++) {
    try {
      more.emplace_back(work);
    } catch (const std::exception&) {  // no thread, or no memory for one: fewer do the work
      break;
    }
  }
  work();
  for (std::thread& t : more) t.join();
  return ok;
}

}  // namespace

bool ordered_tree(const HostBVH& bvh, OrderedTree* out) {
  *out = OrderedTree{};
  const uint32_t n = bvh.nodeN, nt = (uint32_t)bvh.order.size();
  if (n == 0 || bvh.emptyChildren || n >= kOrdMaxIndex || nt >= kOrdMaxIndex) return false;
  Collapse c(bvh);
  float M = 0.f;
  for (int k = 0; k < 6; k++) M = std::fmax(M, std::fabs(bvh.bounds[k]));
  if (!(M >= 1e-3f && M <= 1e9f)) return false;
  // eight threads from 16384 nodes on: below, starting them costs more than the work
  const uint32_t threads = n < 16384u ? 1u : std::min(8u, std::max(1u, std::thread::hardware_concurrency()));
  const size_t parts = threads > 1 ? 64 : 1;

  // the walk's exactness rests on boxes inside their parents' boxes and on no
  // subtree being dropped by the reference's 29-entry stack test: an inner node
  // reached by r right turns is popped with r - 1 entries below it
  std::unique_ptr<uint8_t[]> turns(new uint8_t[n]), depth(new uint8_t[n]);
  turns[0] = depth[0] = 0;
  // node i of the subtree that ends before `end`
  auto check = [&](uint32_t i, uint32_t end) {
    if (!c.inner(i)) {
      const uint64_t first = bvh.offOrTSTN[2 * (size_t)i], cnt = bvh.offOrTSTN[2 * (size_t)i + 1];
      return first + cnt <= nt;
    }
    const uint32_t kids[2] = {c.left(i), c.right(i)};
    if (turns[i] > 29 || depth[i] > 60) return false;
    for (uint32_t k = 0; k < 2; k++) {
      if (kids[k] <= i || kids[k] >= end) return false;
      turns[kids[k]] = (uint8_t)(turns[i] + k);
      depth[kids[k]] = (uint8_t)(depth[i] + 1);
      const float *p = c.box(i), *q = c.box(kids[k]);
      for (int a = 0; a < 3; a++)
        if (!(q[a] >= p[a] && q[3 + a] <= p[3 + a] && q[a] <= q[3 + a])) return false;
    }
    return true;
  };
  struct Range {
    uint32_t from, to;
  };
  std::vector<Range> range{{0u, n}};
  std::vector<uint32_t> top;
  while (range.size() < parts) {  // split the largest subtree
    size_t big = 0;
    for (size_t k = 1; k < range.size(); k++)
      if (range[k].to - range[k].from > range[big].to - range[big].from) big = k;
    const Range r = range[big];
    if (r.to - r.from < 64u) break;
    if (!c.inner(r.from) || !check(r.from, r.to)) return false;
    const uint32_t mid = c.right(r.from);
    if (mid <= r.from + 1u) return false;
    top.push_back(r.from);
    range[big] = {r.from + 1u, mid};
    range.push_back({mid, r.to});
  }
  // Every plane is moved outwards by `margin` before it is quantised.  With u =
  // 2^-24 and |origin| <= 8 M, in units of the axis (distance times direction):
  // the walk's plane is off by at most 27 u M + 2^-9 cells, the reference's by
  // 18 u M, and scaling by the closest hit adds 4 u of a distance of at most 9 M
  // to each of the two that are compared: 128 u M and 2^-7 cells cover all.
  const double margin = std::ldexp((double)M, -17);
  struct Areas {
    double exact = 0, grown = 0;  // of the range's leaf boxes
  };
  std::vector<Areas> leafArea(range.size());
  if (!each(range.size(), threads, [&](size_t k) {
        Areas sum;
        for (uint32_t i = range[k].from; i < range[k].to; i++) {
          if (!check(i, range[k].to)) return false;
          if (!c.inner(i)) sum.exact += c.grown(i, 0.0), sum.grown += c.grown(i, margin);
        }
        leafArea[k] = sum;
        c.make_plan(range[k].from, range[k].to);
        return true;
      }))
    return false;
  Areas total;
  for (const Areas& a : leafArea) total.exact += a.exact, total.grown += a.grown;
  if (!(total.grown <= most_growth(n) * total.exact)) return false;
  for (size_t k = top.size(); k-- > 0;) c.make_plan(top[k], top[k] + 1u);  // a node was split after its parent

  out->range = 8.f * M;
  Part head;
  head.nodes.resize(kOrdNodeWords);
  head.todo.push_back({0u, 0u, 1u});
  size_t at = 0;
  for (; at < head.todo.size() && (parts == 1 || head.todo.size() - at < parts); at++) {
    const Item it = head.todo[at];
    if (!emit(c, margin, it, head)) return false;
  }
  const size_t rest = head.todo.size() - at, headN = head.nodes.size() / kOrdNodeWords;
  std::vector<Part> part(rest);
  if (!each(rest, threads, [&](size_t k) {
        Part& p = part[k];
        const Item root = head.todo[at + k];
        p.nodes.resize(kOrdNodeWords);
        p.todo.push_back({root.bin, 0u, root.depth});
        while (!p.todo.empty()) {
          const Item it = p.todo.back();
          p.todo.pop_back();
          if (!emit(c, margin, it, p)) return false;
        }
        return true;
      }))
    return false;
  // the parts one after another behind the top nodes; a part's node 0 is the
  // top node it hangs from
  std::vector<size_t> nodeAt(rest), leafAt(rest);
  size_t nodes = headN, leaves = head.leaves.size();
  for (size_t k = 0; k < rest; k++) {
    nodeAt[k] = nodes;
    leafAt[k] = leaves;
    nodes += part[k].nodes.size() / kOrdNodeWords - 1;
    leaves += part[k].leaves.size();
  }
  if (nodes >= kOrdMaxIndex || leaves >= kOrdMaxIndex) return false;
  out->nodeN = (uint32_t)nodes;
  out->leafN = (uint32_t)leaves;
  out->nodes.reset(new float[nodes * kOrdNodeWords]);
  out->leaves.reset(new uint32_t[leaves + 1]);
  std::memcpy(out->nodes.get(), head.nodes.data(), head.nodes.size() * 4);
  if (!head.leaves.empty()) std::memcpy(out->leaves.get(), head.leaves.data(), head.leaves.size() * 4);
  return each(rest, threads, [&](size_t k) {
    Part& p = part[k];
    const size_t count = p.nodes.size() / kOrdNodeWords;
    for (size_t i = 0; i < count; i++) {
      float* w = &p.nodes[i * kOrdNodeWords];
      uint32_t word[2];
      std::memcpy(word, w + 6, 8);
      word[0] += (uint32_t)(nodeAt[k] - 1);  // below 2^24 with the mask above: checked by the sums
      word[1] += (uint32_t)leafAt[k];
      std::memcpy(w + 6, word, 8);
    }
    std::memcpy(&out->nodes[(size_t)head.todo[at + k].wide * kOrdNodeWords], p.nodes.data(), kOrdNodeWords * 4);
    std::memcpy(&out->nodes[nodeAt[k] * kOrdNodeWords], p.nodes.data() + kOrdNodeWords,
                (count - 1) * kOrdNodeWords * 4);
    if (!p.leaves.empty()) std::memcpy(&out->leaves[leafAt[k]], p.leaves.data(), p.leaves.size() * 4);
    return true;
  });
}

}  // namespace gbpt
