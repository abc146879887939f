// kr_template.cpp -- see kr_template.h.
#include "kr_template.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "kr_units.h"

namespace kr {

namespace {

// BODY, src/body/kraken.js:22-47
constexpr double kPi = 3.141592653589793;
constexpr double kSegLen = 13.5;
constexpr double kShoulderR = 24;
constexpr double kMantleR = 18;
constexpr double kMantleMass = 20;
constexpr double kMantleIF = 2.5;
constexpr double kSegMassProx = 3.2, kSegMassDist = 1.8;
constexpr double kSegThickProx = 11.9, kSegThickDist = 5.9;
constexpr double kStiffMin = 2000;

struct RawCon {
  int type, a, b;
  double lax, lay, lbx, lby, rest, minA, maxA;
  int motor;     // a * segs + j or -1
  int arm;       // owner arm for grips, else -1
  int color;
};

double rect_inertia(double m, double w, double h) { return m * (w * w + h * h) / 12; }

float word(unsigned u) {
  float f;
  std::memcpy(&f, &u, sizeof(f));
  return f;
}

}  // namespace

bool build_template(int arms, int segs, Template *t, std::string *err) {
  if (arms < 1 || arms > kMaxArms || segs < 1 || segs > kMaxSegs) {
    *err = "body shape " + std::to_string(arms) + "x" + std::to_string(segs) +
           " outside 1.." + std::to_string(kMaxArms) + " arms x 1.." + std::to_string(kMaxSegs) +
           " segments";
    return false;
  }
  *t = Template();
  t->arms = arms;
  t->segs = segs;
  t->reach = kShoulderR + segs * kSegLen;
  const double joint = kPi * 0.42, shoulder = kPi * 0.62;
  std::vector<double> im, ii;
  std::vector<int> pbody;
  std::vector<double> plx, ply, pr;
  std::vector<RawCon> cons;
  auto add_body = [&](double mass, double inertia) {
    im.push_back(mass > 0 ? 1 / mass : 0);
    ii.push_back(inertia > 0 ? 1 / inertia : 0);
    return (int)im.size() - 1;
  };
  auto add_pt = [&](int b, double lx, double ly, double r) {
    pbody.push_back(b); plx.push_back(lx); ply.push_back(ly); pr.push_back(r);
  };
  auto add_con = [&](int type, int a, int b, double lax, double lay, double lbx, double lby) {
    RawCon c{type, a, b, lax, lay, lbx, lby, 0, -INFINITY, INFINITY, -1, -1, -1};
    cons.push_back(c);
    return (int)cons.size() - 1;
  };
  // spawnKraken creation order (kraken.js:64-148)
  const double mantleI = (kMantleMass * kMantleR * kMantleR / 2) * kMantleIF;
  const int mantle = add_body(kMantleMass, mantleI);
  for (int i = 0; i < 8; i++) {
    const double a = ((double)i / 8) * kPi * 2;
    add_pt(mantle, std::cos(a) * kMantleR * 0.7, std::sin(a) * kMantleR * 0.7, kMantleR * 0.45);
  }
  t->arm_tip.resize(arms);
  t->arm_seg0.resize(arms);
  t->arm_segs.resize((size_t)arms * segs);
  for (int a = 0; a < arms; a++) {
    const double relAng = ((double)a / arms) * kPi * 2;
    std::vector<int> sg(segs);
    for (int i = 0; i < segs; i++) {
      const double tt = segs > 1 ? (double)i / (segs - 1) : 0;
      const double mass = kSegMassProx + (kSegMassDist - kSegMassProx) * tt;
      const double thick = kSegThickProx + (kSegThickDist - kSegThickProx) * tt;
      const int b = add_body(mass, rect_inertia(mass, kSegLen, thick));
      const double r = thick * 0.5;
      add_pt(b, -kSegLen * 0.5 + r * 0.4, 0, r);
      add_pt(b, kSegLen * 0.5 - r * 0.4, 0, r);
      sg[i] = b;
      t->arm_segs[(size_t)a * segs + i] = b;
    }
    add_con(0, mantle, sg[0], std::cos(relAng) * kShoulderR, std::sin(relAng) * kShoulderR,
            -kSegLen * 0.5, 0);
    int ms = add_con(1, mantle, sg[0], 0, 0, 0, 0);
    cons[ms].rest = relAng;
    cons[ms].minA = -shoulder;
    cons[ms].maxA = shoulder;
    cons[ms].motor = a * segs;
    for (int i = 0; i + 1 < segs; i++) {
      add_con(0, sg[i], sg[i + 1], kSegLen * 0.5, 0, -kSegLen * 0.5, 0);
      int m = add_con(1, sg[i], sg[i + 1], 0, 0, 0, 0);
      cons[m].rest = 0.28;  // spawnCurl: the spawn pose is the fixpoint
      cons[m].minA = -joint;
      cons[m].maxA = joint;
      cons[m].motor = a * segs + i + 1;
    }
    int g = add_con(2, sg[segs - 1], -1, kSegLen * 0.5, 0, 0, 0);
    cons[g].arm = a;
    t->arm_tip[a] = sg[segs - 1];
    t->arm_seg0[a] = sg[0];
  }
  const int nb = (int)im.size(), nc = (int)cons.size(), np = (int)pbody.size();
  // colouring in creation order (core.js:51-58 / assignColor) and stable grouping
  std::vector<uint32_t> mask(nb, 0u);
  for (auto &c : cons) {
    uint32_t used = mask[c.a] | (c.b >= 0 ? mask[c.b] : 0u);
    int col = 0;
    while (col < 31 && (used & (1u << col))) col++;
    mask[c.a] |= 1u << col;
    if (c.b >= 0) mask[c.b] |= 1u << col;
    c.color = col;
  }
  std::vector<int> list(nc);
  for (int i = 0; i < nc; i++) list[i] = i;
  std::stable_sort(list.begin(), list.end(),
                   [&](int x, int y) { return cons[x].color < cons[y].color; });
  t->nb = nb; t->nc = nc; t->np = np;
  t->im.resize(nb); t->ii.resize(nb);
  for (int i = 0; i < nb; i++) { t->im[i] = (float)im[i]; t->ii[i] = (float)ii[i]; }
  // units of the solve list and, per lane-group size, their passes
  std::vector<SolveEntry> entries(nc);
  for (int q = 0; q < nc; q++) {
    const RawCon &c = cons[list[q]];
    entries[q] = SolveEntry{c.type == 1 ? 1 : 0, c.a, c.b};
  }
  std::vector<SolveUnit> units;
  std::vector<int> last;
  build_units(entries, nb, &units, last);
  for (const SolveUnit &u : units) {
    // the engine's records hold a joint (pin and angle constraint) or a grip
    const bool joint = u.pin >= 0 && u.ang >= 0 && u.b >= 0;
    const bool grip = u.pin >= 0 && u.ang < 0 && u.b < 0 && cons[list[u.pin]].type == 2;
    bool tame = joint || grip;
    if (tame) {
      const RawCon &c = cons[list[u.pin]];
      tame = joint ? pin_tame((float)c.lax, (float)c.lay, (float)c.lbx, (float)c.lby, t->im[u.a], t->ii[u.a],
                              t->im[u.b], t->ii[u.b])
                   : pin_tame((float)c.lax, (float)c.lay, 0.f, 0.f, t->im[u.a], t->ii[u.a], 0.f, 0.f);
      tame = tame && c.lby == 0;
    }
    if (tame && joint) {
      // what the engine's angle constraint relies on (kr_solver.cuh angle_near)
      const RawCon &g = cons[list[u.ang]];
      const float w = t->ii[u.a] + t->ii[u.b];
      unsigned m;
      std::memcpy(&m, &w, sizeof(m));
      tame = g.rest >= 0 && g.rest <= 6.27 && w > 0x1p-60f && w < 0x1p60f && (m & 0x7fffffu) != 0x7fffffu;
    }
    if (!tame) {
      *err = "body shape " + std::to_string(arms) + "x" + std::to_string(segs) + ": a constraint outside the joints";
      return false;
    }
  }
  for (int v = 0; v < kSchedules; v++) {
    const int G = v == 0 ? 32 : v == 1 ? 16 : 8;
    std::vector<int> order, off;
    schedule_units(units, nb, G, &order, &off);
    Schedule &S = t->sched[v];
    S.npass = (int)off.size() - 1;
    S.recs.assign((size_t)S.npass * G * kRecFloats, 0.f);
    for (int p = 0; p < S.npass; p++) {
      for (int l = 0; l < G; l++) {
        float *r = &S.recs[((size_t)p * G + l) * kRecFloats];
        if (off[p] + l >= off[p + 1]) {
          const unsigned spare = (unsigned)(nb + arms);
          r[0] = word(spare | (spare << 8) | ((unsigned)(grip_pair0(arms, segs) + arms) << 16) | kRecIdle);
          r[4] = 1.f;
          continue;
        }
        const SolveUnit &u = units[order[off[p] + l]];
        const RawCon &c = cons[list[u.pin]];
        const unsigned B = u.b >= 0 ? (unsigned)u.b : (unsigned)(nb + c.arm);
        const unsigned m = u.ang >= 0 ? (unsigned)cons[list[u.ang]].motor | (kRecJoint >> 16)
                                      : (unsigned)(grip_pair0(arms, segs) + c.arm);
        r[0] = word((unsigned)u.a | (B << 8) | (m << 16));
        r[1] = (float)c.lax; r[2] = (float)c.lay;
        r[4] = t->im[u.a]; r[5] = t->ii[u.a];
        if (u.b >= 0) {
          r[3] = (float)c.lbx;
          r[6] = t->im[u.b]; r[7] = t->ii[u.b];
        }
        if (u.ang >= 0) {
          const RawCon &g = cons[list[u.ang]];
          r[8] = (float)g.rest; r[9] = (float)g.minA; r[10] = (float)g.maxA;
          // rounded once: no f32 reciprocal lies within a f64 rounding of a midpoint
          r[11] = (float)(1.0 / (double)(t->ii[u.a] + t->ii[u.b]));
        }
      }
    }
  }
  // points grouped per body, creation order within a body (groupCollPoints)
  t->boff.assign(nb, 0);
  t->bcnt.assign(nb, 0);
  t->breach.assign(nb, 0.f);
  for (int p = 0; p < np; p++) t->bcnt[pbody[p]]++;
  int acc = 0;
  for (int b = 0; b < nb; b++) { t->boff[b] = acc; acc += t->bcnt[b]; }
  t->plx.assign(np, 0.f); t->ply.assign(np, 0.f); t->pr.assign(np, 0.f); t->pbody.assign(np, 0);
  std::vector<int> pc = t->boff;
  for (int p = 0; p < np; p++) {
    const int q = pc[pbody[p]]++;
    t->plx[q] = (float)plx[p]; t->ply[q] = (float)ply[p]; t->pr[q] = (float)pr[p];
    t->pbody[q] = pbody[p];
    t->r_max = std::max(t->r_max, (float)pr[p]);
    const double off = std::sqrt((double)t->plx[q] * t->plx[q] + (double)t->ply[q] * t->ply[q]);
    t->breach[pbody[p]] = std::max(t->breach[pbody[p]], (float)off + 1.f);
  }
  return true;
}

void spawn_pose(const Template &t, double x, double y, double angle, double curl, double *px,
                double *py, double *ang) {
  px[0] = x; py[0] = y; ang[0] = angle;
  for (int a = 0; a < t.arms; a++) {
    const double relAng = ((double)a / t.arms) * kPi * 2;
    const double th0 = angle + relAng;
    double jx = x + std::cos(th0) * kShoulderR;
    double jy = y + std::sin(th0) * kShoulderR;
    double th = th0;
    for (int i = 0; i < t.segs; i++) {
      const double ux = std::cos(th), uy = std::sin(th);
      const double cx = jx + ux * kSegLen * 0.5;
      const double cy = jy + uy * kSegLen * 0.5;
      const int b = t.arm_segs[(size_t)a * t.segs + i];
      px[b] = cx; py[b] = cy; ang[b] = th;
      jx = cx + ux * kSegLen * 0.5;
      jy = cy + uy * kSegLen * 0.5;
      th += curl;
    }
  }
}

}  // namespace kr
