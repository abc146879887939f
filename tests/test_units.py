"""The solve schedule (csrc/kr_units.h, csrc/kr_template.cpp): units and
passes of a solve list, checked against the list itself.  Any two constraints
that share a body must keep their list order -- inside a unit the pin comes
first -- and the units of a pass must not share a body; every constraint
appears exactly once.  Those two properties make a pass sweep bit-identical
to the sequential sweep of the list.  Random lists (repeated pairs, world
anchors, angle constraints without a pin, reversed pairs) at 1, 8, 16 and 32
lanes, and the unit records of every body shape."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "kraken_3_gpu_b200", "csrc")

PROGRAM = r'''
#include <cstdio>
#include <cstring>
#include <random>
#include "kr_template.h"
#include "kr_units.h"

static int fail(const char *m, int x) { std::printf("FAIL %s %d\n", m, x); return 1; }

static int check(const std::vector<kr::SolveEntry> &list, int nb, int G) {
  std::vector<kr::SolveUnit> units;
  std::vector<int> last, order, off;
  kr::build_units(list, nb, &units, last);
  kr::schedule_units(units, nb, G, &order, &off);
  if (order.size() != units.size()) return fail("units scheduled", (int)order.size());
  if (off.back() != (int)order.size()) return fail("offsets", off.back());
  // the constraints in the order a pass sweep solves them
  std::vector<int> run, pass;
  for (size_t p = 0; p + 1 < off.size(); p++) {
    if (off[p + 1] <= off[p] || off[p + 1] - off[p] > G) return fail("pass size", (int)p);
    std::vector<int> used(nb, 0);
    for (int k = off[p]; k < off[p + 1]; k++) {
      const kr::SolveUnit &u = units[order[k]];
      if (used[u.a]++ || (u.b >= 0 && u.b != u.a && used[u.b]++)) return fail("body twice in a pass", (int)p);
      if (u.pin >= 0) { run.push_back(u.pin); pass.push_back((int)p); }
      if (u.ang >= 0) { run.push_back(u.ang); pass.push_back((int)p); }
    }
  }
  if (run.size() != list.size()) return fail("constraints", (int)run.size());
  std::vector<int> at(list.size(), -1);
  for (size_t k = 0; k < run.size(); k++) {
    if (at[run[k]] >= 0) return fail("constraint twice", run[k]);
    at[run[k]] = (int)k;
  }
  for (size_t i = 0; i < list.size(); i++)
    for (size_t j = i + 1; j < list.size(); j++) {
      const kr::SolveEntry &x = list[i], &y = list[j];
      const bool share = x.a == y.a || (y.b >= 0 && x.a == y.b) || (x.b >= 0 && (x.b == y.a || x.b == y.b));
      if (share && at[i] > at[j]) return fail("order", (int)i);
    }
  return 0;
}

int main() {
  std::mt19937 r(7);
  for (int t = 0; t < 400; t++) {
    const int nb = 1 + r() % 20, n = r() % 60;
    std::vector<kr::SolveEntry> list;
    for (int q = 0; q < n; q++) {
      if (!list.empty() && r() % 3 == 0) {  // the pair before, either way round
        kr::SolveEntry c = list.back();
        c.angle = r() % 2;
        if (c.b >= 0 && r() % 4 == 0) std::swap(c.a, c.b);
        list.push_back(c);
        continue;
      }
      const int a = r() % nb;
      int b = r() % 4 == 0 || nb == 1 ? -1 : (int)(r() % nb);
      if (b == a && r() % 2) b = -1;  // otherwise both bodies are one
      list.push_back({(int)(r() % 2), a, b});
    }
    for (int G : {1, 8, 16, 32})
      if (check(list, nb, G)) return 1;
  }
  int worst = 0;
  for (int A = 1; A <= kr::kMaxArms; A++)
    for (int S = 1; S <= kr::kMaxSegs; S++) {
      kr::Template T;
      std::string err;
      if (!kr::build_template(A, S, &T, &err)) { std::printf("FAIL %s\n", err.c_str()); return 1; }
      for (int v = 0; v < kr::kSchedules; v++) {
        const int G = v == 0 ? 32 : v == 1 ? 16 : 8;
        const kr::Schedule &s = T.sched[v];
        if (s.recs.size() != (size_t)s.npass * G * kr::kRecFloats) return fail("record count", A * 10 + S);
        std::vector<int> joint(A * S, 0), grip(A, 0);
        for (int p = 0; p < s.npass; p++) {
          std::vector<int> used(T.nb + A, 0);
          for (int l = 0; l < G; l++) {
            unsigned ab;
            std::memcpy(&ab, &s.recs[((size_t)p * G + l) * kr::kRecFloats], 4);
            const int a = ab & 0xff, b = (ab >> 8) & 0xff, m = (ab >> 16) & 0xff, g0 = kr::grip_pair0(A, S);
            if (ab & kr::kRecIdle) {
              if (a != T.nb + A || b != a || m != g0 + A || (ab & kr::kRecJoint)) return fail("idle", A * 10 + S);
              continue;
            }
            if (a >= T.nb || b >= T.nb + A || used[a]++ || used[b]++) return fail("record bodies", A * 10 + S);
            if (ab & kr::kRecJoint) { if (m >= A * S || joint[m]++ || b != T.arm_segs[m]) return fail("joint", m); }
            else if (b < T.nb || grip[b - T.nb]++ || a != T.arm_tip[b - T.nb] || m != g0 + b - T.nb) return fail("grip", m);
          }
        }
        for (int j : joint) if (j != 1) return fail("joints", A * 10 + S);
        for (int g : grip) if (g != 1) return fail("grips", A * 10 + S);
        const int need = std::max(A, (A * S + A + G - 1) / G);
        if (A > 1 && S > 1) worst = std::max(worst, s.npass - need);
      }
    }
  std::printf("ok %d\n", worst);
  return 0;
}
'''


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("units")
    src = d / "units.cpp"
    src.write_text(PROGRAM)
    exe = d / "units"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, "-o", str(exe), str(src),
                    os.path.join(CSRC, "kr_template.cpp")], check=True)
    return str(exe)


def test_units_keep_the_list_order(program):
    out = subprocess.run([program], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout


def test_every_shape_needs_the_fewest_passes(program):
    """Bodies of two arms and segments or more: no schedule is longer than the
    larger of the arms (each joins the mantle) and the units over the lanes."""
    assert subprocess.run([program], capture_output=True, text=True, timeout=120).stdout == "ok 0\n"
