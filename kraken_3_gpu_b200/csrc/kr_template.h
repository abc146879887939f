// kr_template.h -- native body templates of the batched engine.
//
// A template is the constraint graph of one body shape (A arms x S segments)
// with its solve schedule, built exactly as the reference builds a creature:
// spawnKraken's creation order (src/body/kraken.js:64-148), createSim's
// greedy colouring in creation order (src/sim/core.js:45-58 with
// assignColor, src/physics/xpbd.js:98-105), the stable grouping by colour
// (core.js:276-288), and from that list order the passes of body-disjoint
// units that the lanes sweep.  Spawn poses follow the same chain rule (kraken.js:64-101).
#pragma once
#include <cstdint>
#include <string>
#include <vector>

namespace kr {

constexpr int kMaxArms = 8;
constexpr int kMaxSegs = 9;
constexpr int kMaxTplBodies = 1 + kMaxArms * kMaxSegs;            // 73
constexpr int kMaxTplCons = kMaxArms * (2 * kMaxSegs + 1);        // 152
constexpr int kMaxTplPts = 8 + 2 * kMaxArms * kMaxSegs;           // 152
constexpr int kRecFloats = 12;                                     // one unit record: 3 float4

// Solve schedules per lane-group size: 32, 16 and 8 lanes per creature.
constexpr int kSchedules = 3;
constexpr int schedule_index(int lanes) { return lanes == 32 ? 0 : lanes == 16 ? 1 : 2; }

// One solve schedule of the constraint list: unit records pass by pass, one
// per lane (idle lanes included), 3 float4 each:
//   {A | B << 8 | pair << 16 | flags, lax, lay, lbx} {1 / mass A, 1 / inertia
//   A, 1 / mass B, 1 / inertia B} {rest, min, max, 1 / (sum of 1 / inertia)}
// (kr_units.h kRecJoint, grip_pair0; lby is 0).  B of a grip is nb + arm, the record
// that holds its anchor; an idle lane's bodies are nb + arms, a spare record.
struct Schedule {
  int npass = 0;
  std::vector<float> recs;              // npass x lanes x kRecFloats
};

struct Template {
  int arms = 0, segs = 0;
  int nb = 0, nc = 0, np = 0;
  // bodies
  std::vector<float> im, ii;            // f32 as uploaded (gpuworld.js:258-259)
  std::vector<int> boff, bcnt;          // collision points per body
  std::vector<float> breach;            // bound on their distance from the body's centre (+1 px)
  // per lane-group size (schedule_index): the solve list in passes of that
  // many lanes
  Schedule sched[kSchedules];
  // collision points grouped per body in creation order
  std::vector<float> plx, ply, pr;
  std::vector<int> pbody;
  // arms
  std::vector<int> arm_tip;             // tip body
  std::vector<int> arm_seg0;            // first segment body
  std::vector<int> arm_segs;            // arms x segs body ids
  float r_max = 0.f;                    // largest collision radius
  double reach = 0.0;                   // ARM_REACH for this segment count
};

// Builds the template of an arms x segs body; returns false with a message
// if the shape is out of range.
bool build_template(int arms, int segs, Template *t, std::string *err);

// spawnKraken's pose (kraken.js:64-101): body positions and angles of a
// creature spawned at (x, y, angle), in f64, body order of the template.
void spawn_pose(const Template &t, double x, double y, double angle, double curl, double *px,
                double *py, double *ang);

}  // namespace kr
