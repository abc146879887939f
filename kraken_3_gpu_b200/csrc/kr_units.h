// kr_units.h -- host side of the solve schedule: a solve list (constraints in
// order, each with its one or two bodies) as units and passes of units (see
// kr::Island in kr_solver.cuh), and which pins take the short form.
#pragma once
#include <algorithm>
#include <vector>

#ifdef __CUDACC__
#define KR_HD __host__ __device__
#else
#define KR_HD
#endif

namespace kr {

// Levers and masses for which the quotients of kr_solver.cuh pin_near stay in
// range whatever the angles (every pin of a creature): with wI |l|^2 <= 16 wS
// the matrix entries lie in wS .. 33 wS and det in wS^2 .. 2^11 wS^2, wS in
// 2^-10 .. 2^10 (so |det| >= kEpsDet); k01 is 0 or above 2^-100, since |sin|
// and |cos| are above 2^-21 where sincos_near stands and a lever's components
// are not small unless the other is large.
KR_HD inline bool lever_tame(float x, float y, float wI, float wS) {
  const float ax = x < 0.f ? -x : x, ay = y < 0.f ? -y : y;
  if (!(wI >= 0.f && wI <= 0x1p10f && ax <= 0x1p20f && ay <= 0x1p20f)) return false;
  if (wI == 0.f || (ax == 0.f && ay == 0.f)) return true;
  if (wI < 0x1p-16f || !(ax >= 0x1p-4f || ay >= 0x1p-4f)) return false;
  if ((ax > 0x1p-30f && ax < 0x1p-4f) || (ay > 0x1p-30f && ay < 0x1p-4f)) return false;
  return wI * (ax * ax + ay * ay) <= 16.f * wS;
}
KR_HD inline bool pin_tame(float lax, float lay, float lbx, float lby, float wA, float wIA, float wB, float wIB) {
  const float wS = wA + wB;
  return wA >= 0.f && wB >= 0.f && wS >= 0x1p-10f && wS <= 0x1p10f && lever_tame(lax, lay, wIA, wS) &&
         lever_tame(lbx, lby, wIB, wS);
}

// The batched engine's unit records: flags of the ab word above body A, body B
// << 8 and the index of its pair in the motors' records << 16; motors come
// first, then (their words also hold the proprioception's 6 arms + 6) one
// pair per grip and one for idle lanes.
constexpr unsigned kRecJoint = 1u << 24, kRecIdle = 1u << 25;
KR_HD inline int grip_pair0(int arms, int segs) {
  const int m = 2 * arms * segs, o = 6 * arms + 6;
  return (m > o ? m : o) / 2;
}

struct SolveEntry {
  int angle;  // 1: angle constraint, 0: pin or grip
  int a, b;   // bodies, b < 0: the world
};

// One unit: list positions of its pin and of its angle constraint (-1: none).
struct SolveUnit {
  int pin, ang, a, b;
};

// The list's units in list order.  An angle constraint joins the unit before
// it when that unit is the last one on both of its bodies and is a pin of the
// same two bodies: the pair then runs back to back in any valid order.
inline void build_units(const std::vector<SolveEntry> &list, int n_bodies, std::vector<SolveUnit> *units,
                        std::vector<int> &last) {
  units->clear();
  last.assign(n_bodies, -1);
  for (int q = 0; q < (int)list.size(); q++) {
    const SolveEntry &c = list[q];
    const int u = last[c.a];
    if (c.angle && u >= 0 && (c.b < 0 || last[c.b] == u)) {
      SolveUnit &p = (*units)[u];
      if (p.pin >= 0 && p.ang < 0 && p.a == c.a && p.b == c.b) {
        p.ang = q;
        continue;
      }
    }
    const int id = (int)units->size();
    units->push_back(c.angle ? SolveUnit{-1, q, c.a, c.b} : SolveUnit{q, -1, c.a, c.b});
    last[c.a] = id;
    if (c.b >= 0) last[c.b] = id;
  }
}

// Passes of at most G body-disjoint units: units sharing a body keep their
// list order, and each pass takes the ready units with the longest chain of
// successors first (list scheduling: with 8 lanes the 25 bodies of 4-8 arms x
// 5-9 segments need no more passes than max(arms, units / 8 rounded up)).
// order: the units pass by pass; off: n_passes + 1 offsets into it.
inline void schedule_units(const std::vector<SolveUnit> &units, int n_bodies, int G, std::vector<int> *order,
                           std::vector<int> *off) {
  const int n = (int)units.size();
  std::vector<int> last(n_bodies, -1), need(n, 0), height(n, 1), by_height(n), succ(2 * (size_t)n, -1);
  for (int u = n - 1; u >= 0; u--) {  // the next unit on each body
    int k = 0;
    for (int b : {units[u].a, units[u].b}) {
      if (b < 0 || (k == 1 && units[u].a == b)) continue;
      const int s = last[b];
      if (s >= 0 && !(k == 1 && succ[2 * (size_t)u] == s)) {
        succ[2 * (size_t)u + k] = s;
        need[s]++;
        height[u] = std::max(height[u], height[s] + 1);
      }
      last[b] = u;
      k = 1;
    }
  }
  for (int u = 0; u < n; u++) by_height[u] = u;
  std::stable_sort(by_height.begin(), by_height.end(), [&](int x, int y) { return height[x] > height[y]; });
  order->clear();
  off->assign(1, 0);
  std::vector<int> left = by_height, rest;
  while (!left.empty()) {
    const size_t beg = order->size();
    rest.clear();
    for (int u : left) {
      if (need[u] == 0 && order->size() - beg < (size_t)G) order->push_back(u);
      else rest.push_back(u);
    }
    for (size_t k = beg; k < order->size(); k++)
      for (int j = 0; j < 2; j++) {
        const int s = succ[2 * (size_t)(*order)[k] + j];
        if (s >= 0) need[s]--;
      }
    off->push_back((int)order->size());
    left.swap(rest);
  }
}

}  // namespace kr
