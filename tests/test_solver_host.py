"""Device functions of csrc/kr_solver.cuh run on the CPU (tests/cuda_on_host.h),
where a test can look at more than a step's results: which form a value takes,
and how many rects a collision pass reads."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "kraken_3_gpu_b200", "csrc")

COMMON = r'''
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "cuda_on_host.h"
using namespace kr;
static float2 g_tab[kSinEntries];
static float bits(unsigned u) { return __uint_as_float(u); }
static bool same(float4 a, float4 b) { return std::memcmp(&a, &b, sizeof a) == 0; }
'''


def _run(tmp_path, body, *args):
    src = tmp_path / "t.cpp"
    src.write_text(COMMON + body)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-mfma", "-w", "-pthread", "-I", HERE, "-I", CSRC, "-o",
                    str(exe), str(src)], check=True)
    out = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout


DISABLED = r'''
// one unit of two bodies whose pin and angle constraint are broken (or not
// there): both bodies must stay as they are, whatever the records hold
int main() {
  stage_sin(g_tab);
  const float inf = kInf, nan = bits(0x7fc00000u);
  const float angles[] = {0.3f, 60.f, 70.f, 1e4f, 1e17f, 1e30f, -3e38f, inf, -inf};
  const float levers[] = {7.f, 1e25f, inf, nan};
  const float masses[] = {0.25f, 0.f, 1e31f, inf, -inf};
  int n = 0;
  for (float az : angles) for (float bz : angles) for (float lev : levers) for (float im : masses)
  for (int ref = 0; ref < 3; ref++) for (int pin = 0; pin < 2; pin++) for (int world = 0; world < 2; world++) {
    float4 Q[2] = {make_float4(10.f, 20.f, az, 0.f), make_float4(14.f, 22.f, bz, 0.f)}, in[2] = {Q[0], Q[1]};
    float4 body[2] = {make_float4(im, ref == 1 ? im : 0.01f, 0.f, 0.f), make_float4(0.5f, ref == 2 ? im : 0.02f, 0.f, 0.f)};
    const float lax = pin ? lev : 0.f, lay = pin ? 2.f : 0.f, lbx = pin ? 3.f : 0.f, lby = pin ? lev : 0.f;
    const float wB = world ? 0.f : body[1].x, wIB = world ? 0.f : body[1].y;
    const unsigned ab = 0u | (world ? 0xffu : 1u) << 8 | kHasAngle | kAngleBroken | (pin ? kHasPin | kPinBroken : 0u) |
                        unit_forms(pin, false, lax, lay, world ? 0.f : lbx, world ? 0.f : lby, body[0].x, body[0].y, wB, wIB);
    float4 rec[kWorldRec] = {{bits(ab), lax, lay, lbx}, {lby, body[0].x, body[0].y, wB}, {wIB, lev, -1.f, 1.f},
                             {lev, lev, lev, recip(fadd(body[0].y, wIB))}, {0.f, 0.f, 0.f, 100.f}};
    Island S{};
    int off[2] = {0, 1};
    S.Q = Q; S.tab = g_tab; S.units = rec; S.nu = 1; S.npass = 1; S.off = off; S.nb = 2;
    solve_world<1>(S, true, Lanes<1>(0));
    solve_world<1>(S, false, Lanes<1>(0));
    if (!same(Q[0], in[0]) || !same(Q[1], in[1])) {
      std::printf("FAIL angles %g %g lever %g mass %g: %g %g\n", az, bz, lev, im, Q[0].z, Q[1].z);
      return 1;
    }
    n++;
  }
  std::printf("ok %d\n", n);
  return 0;
}
'''


def test_disabled_constraints_leave_their_bodies_alone(tmp_path):
    assert _run(tmp_path, DISABLED).startswith("ok")


CLAMP = r'''
// clamp_speed against the reference's plain form for limits of every size
int main() {
  std::mt19937 r(3);
  std::vector<float> lim = {0.f, -1.f, kInf, -kInf, bits(0x7fc00000u), 1.f, 360.f, 3e38f, 1e20f, 1.9e19f, 1.8e19f, 1e-18f, 1e-22f, 1e-23f, 1e-40f};
  for (int i = 0; i < 200; i++) lim.push_back(bits(r() & 0x7f7fffffu));
  long n = 0;
  for (float m : lim) {
    SolverConsts K{};
    K.maxSpeed = m;
    for (int i = 0; i < 20000; i++) {
      float x, y;
      const float a = std::fabs(m) < 1e38f ? std::fabs(m) : 1e38f;
      if (i < 10000) { x = bits(r() & 0xff7fffffu); y = i % 3 ? bits(r() & 0xff7fffffu) : 0.f; }
      else { const float t = 6.2831853f * (r() >> 8) / 16777216.f, s = 0.9f + 0.2f * (r() >> 8) / 16777216.f;
             x = a * s * std::cos(t); y = a * s * std::sin(t); }
      if (i % 1000 == 0) x = i % 2000 ? kInf : bits(0x7fc00000u);
      float vx = x, vy = y, wx = x, wy = y;
      clamp_speed(K, vx, vy);
      const float sp = length2(wx, wy);
      if (sp > m) { const float k = fdiv(m, sp); wx = fmul(wx, k); wy = fmul(wy, k); }
      if (std::memcmp(&vx, &wx, 4) || std::memcmp(&vy, &wy, 4)) {
        std::printf("FAIL limit %g of (%g, %g): (%g, %g) for (%g, %g)\n", m, x, y, vx, vy, wx, wy);
        return 1;
      }
      n++;
    }
  }
  std::printf("ok %ld\n", n);
  return 0;
}
'''


def test_speed_clamp_equals_the_plain_form(tmp_path):
    assert _run(tmp_path, CLAMP).startswith("ok")


SINCOS = r'''
#include <thread>
// sincos_near against sincos_f64: no accepted value may differ, and how many
// it leaves to sincos_f64 per octave of the argument.  argv[1]: every step-th
// argument of an octave (1: all of them)
struct Count { long n = 0, refused = 0, wrong = 0; };
static Count octave(int e, unsigned step) {  // exponent field e of the argument, both signs
  Count c;
  const unsigned first = e < 0 ? 0 : (unsigned)e << 23, last = first + (1u << 23);
  for (unsigned u = first; u < last; u += step)
    for (int sign = 0; sign < 2; sign++) {
      const float a = bits(u | (unsigned)sign << 31);
      if (std::fabs(a) > kSinCosNearMax) continue;
      float s, co;
      c.n++;
      if (sincos_near(g_tab, a, &s, &co) != 0.f) { c.refused++; continue; }
      const float2 f = sincos_f64(a);
      if (std::memcmp(&s, &f.x, 4) || std::memcmp(&co, &f.y, 4)) {
        if (!c.wrong++) std::printf("FAIL sin/cos of %a: %a %a for %a %a\n", a, s, co, f.x, f.y);
      }
    }
  return c;
}
int main(int argc, char **argv) {
  stage_sin(g_tab);
  const unsigned step = (unsigned)std::max(1, std::atoi(argv[1]));
  std::vector<Count> per(134);  // exponent fields 0 (zero and subnormal) .. 133 (64)
  std::vector<std::thread> th;
  const int nt = (int)std::thread::hardware_concurrency();
  for (int t = 0; t < nt; t++)
    th.emplace_back([&, t] { for (int e = t; e < 134; e += nt) per[e] = octave(e, step); });
  for (auto &t : th) t.join();
  long n = 0, refused = 0, wrong = 0;
  for (int e = 0; e < 134; e++) {
    n += per[e].n; refused += per[e].refused; wrong += per[e].wrong;
    if (argc > 2 && per[e].n) std::printf("2^%d: %ld of %ld\n", e - 127, per[e].refused, per[e].n);
    // at most one in 500 of an octave
    if (per[e].refused > per[e].n / 500 + 1) { std::printf("FAIL 2^%d: %ld of %ld refused\n", e - 127, per[e].refused, per[e].n); wrong++; }
  }
  float s, c;
  for (float a : {0.f, -0.f})
    if (sincos_near(g_tab, a, &s, &c) != 0.f || s != 0.f || c != 1.f) { std::printf("FAIL %g\n", a); wrong++; }
  std::printf(wrong ? "FAIL\n" : "ok %ld arguments, %ld refused\n", n, refused);
  return wrong != 0;
}
'''


def test_sines_near_zero_take_the_short_form(tmp_path):
    """0, the angle of most hand-made bodies, and small angles are decided by
    the f32 sine as others are; every 1,009th argument of each octave up to
    64 (KRAKEN_SINCOS_STEP=1: every argument, 20 s of 8 cores)."""
    assert _run(tmp_path, SINCOS, os.environ.get("KRAKEN_SINCOS_STEP", "1009")).startswith("ok")


NEAR = r'''
// Collision passes of a group of bodies that drift, are thrown about and are
// pulled back into walls, against the fold over every rect; and the rects that
// the passes read.  argv: offset of the whole scene, rects, far anchors (an
// immovable body and one without points, this far away; 0: at the scene),
// pull (px a body is put back into the nearest wall in every pass), spread,
// more rects, all far away
struct Scene {
  std::vector<float4> rects, P, Q, body, pts;
  std::vector<unsigned short> cull = std::vector<unsigned short>(64);
  std::vector<unsigned char> list;
  Island S{};
};
int main(int, char **argv) {
  stage_sin(g_tab);
  const float off = std::atof(argv[1]), anchors = std::atof(argv[3]), pull = std::atof(argv[4]), spread = std::atof(argv[5]);
  const int nr = std::atoi(argv[2]);
  std::mt19937 r(11);
  auto u = [&](float a, float b) { return a + (b - a) * (r() >> 8) / 16777216.f; };
  Scene s;
  auto rect = [&](float x, float y, float w, float h) { s.rects.push_back(make_float4(off + x, off + y, off + x + w, off + y + h)); };
  rect(0, 0, 1400, 14); rect(0, 786, 1400, 14); rect(0, 0, 14, 800); rect(1386, 0, 14, 800);
  for (int i = 4; i < nr; i++) rect(u(20, 1360), u(20, 760), u(3, 8), u(3, 8));
  for (int i = 0; i < std::atoi(argv[6]); i++) rect(5000 + 10 * i, 5000, 5, 5);
  const int nb = 24;
  s.P.resize(nb); s.Q.resize(nb); s.body.resize(nb); s.list.resize(nb);
  for (int j = 0; j < nb; j++) {
    const bool fixed = j == 3, bare = j == 4;
    const int n = bare ? 0 : j == 0 ? 8 : 1 + j % 2;
    const float far = fixed || bare ? anchors : 0.f;
    s.Q[j] = make_float4(off + far + 640 + spread * u(-1, 1), off + far + 400 + spread * u(-1, 1), u(-3, 3), 0.f);
    const int at = (int)s.pts.size();
    float reach = 0.f;
    for (int k = 0; k < n; k++) {
      s.pts.push_back(make_float4(u(-9, 9), u(-9, 9), u(2, 9), 0.f));
      reach = std::max(reach, length2(s.pts.back().x, s.pts.back().y) + 1.f);
    }
    s.body[j] = make_float4(fixed ? 0.f : 0.2f, 0.01f, reach, __int_as_float(at | n << 16));
  }
  Island &S = s.S;
  S.P = s.P.data(); S.Q = s.Q.data(); S.body = s.body.data(); S.pts = s.pts.data(); S.tab = g_tab;
  S.cull = s.cull.data(); S.list = s.list.data(); S.nb = nb;
  const int nR = (int)s.rects.size();
  const float near_d = 9.f + 2.f + kCullPad;
  const Lanes<1> L(0);
  Near N;
  long hits = 0, wrong = 0, loads = 0;
  const int kSteps = 400, kPasses = 8;
  for (int step = 0; step < kSteps; step++) {
    for (int pass = 0; pass < kPasses; pass++) {
      for (int j = 0; j < nb; j++) {
        float4 &q = s.Q[j];
        if (s.body[j].x == 0.f) continue;
        q.x += u(-0.8f, 0.8f); q.y += u(-0.8f, 0.8f); q.z += u(-0.1f, 0.1f);
        if (pull != 0.f && j % 5 == 0) { q.x = off + 700.f + 3.f * j; q.y = off + 14.f - pull; }
      }
      std::vector<float4> want = s.Q;
      for (int j = 0; j < nb; j++) {
        if (s.body[j].x == 0.f) continue;
        float sa, ca;
        sincos_r(g_tab, want[j].z, &sa, &ca);
        const int pr = __float_as_int(s.body[j].w);
        for (int k = 0; k < pr >> 16; k++) {
          const float4 pt = s.pts[(pr & 0xffff) + k];
          SdfFold f;
          const float x = fadd(want[j].x, fsub(fmul(pt.x, ca), fmul(pt.y, sa)));
          const float y = fadd(want[j].y, fadd(fmul(pt.x, sa), fmul(pt.y, ca)));
          for (const float4 &c : s.rects) f.add(c, x, y);
          float dx, dy;
          if (f.push(pt.z, &dx, &dy)) { want[j].x = fadd(want[j].x, dx); want[j].y = fadd(want[j].y, dy); hits++; }
        }
      }
      const long before = g_rect_loads;
      collide_island<1, true, false>(S, N, s.rects.data(), nR, near_d, L);
      loads += g_rect_loads - before;
      for (int j = 0; j < nb; j++)
        if (std::memcmp(&s.Q[j], &want[j], 12)) {
          if (!wrong++) std::printf("FAIL step %d pass %d body %d: %a %a for %a %a\n", step, pass, j, s.Q[j].x, s.Q[j].y, want[j].x, want[j].y);
        }
    }
    if (step % 50 == 49)  // thrown across the scene
      for (int j = 0; j < nb; j++)
        if (s.body[j].x != 0.f) { s.Q[j].x = off + 640 + spread * u(-1, 1); s.Q[j].y = off + 400 + spread * u(-1, 1); }
  }
  std::printf(wrong ? "FAIL %ld wrong\n" : "ok %.1f rects a pass, %ld hits\n", wrong ? (double)wrong : (double)loads / (kSteps * kPasses), hits);
  return wrong != 0;
}
'''


def _loads(tmp_path, offset=0, rects=300, anchors=0, pull=0, spread=110, more=0):
    out = _run(tmp_path, NEAR, *map(str, (offset, rects, anchors, pull, spread, more)))
    assert out.startswith("ok"), out
    words = out.split()
    assert int(words[-2]) > 0
    return float(words[1])


@pytest.mark.parametrize("offset", [31500, 100000, -200000, 990000])
def test_near_sets_hold_anywhere(tmp_path, offset):
    """A scene far from the origin gives the full fold's bits, and its passes
    read as many rects as at the origin (within a tenth: its coordinates
    round, so its bodies drift differently)."""
    assert _loads(tmp_path, offset) < 1.1 * _loads(tmp_path)


def test_bodies_that_meet_no_rect_cost_no_rebuild(tmp_path):
    """An immovable body and one without points, out of any reference's range."""
    assert _loads(tmp_path, anchors=50000) <= 1.02 * _loads(tmp_path)


def test_bodies_held_in_a_wall_fold_over_the_near_list(tmp_path):
    """Bodies pushed out of a wall by more than their near set's margin in every
    pass: their remaining points fold over the group's list, not over the map.
    3,000 more rects on it cost a look each at a rebuild, which a drift of 0.8
    px a pass makes rarer than one pass in 20."""
    assert _loads(tmp_path, pull=9, more=3000) - _loads(tmp_path, pull=9) < 3000 / 20


@pytest.mark.parametrize("rects,spread", [(600, 110), (700, 110), (900, 110), (1500, 110), (1500, 320), (4000, 320)])
def test_crowded_groups_fold_over_a_map_of_near_rects(tmp_path, rects, spread):
    """A list that fits within 16 or 8 px only, and more near rects than it
    holds, at one, two and eight rects a bit: the full fold's bits.  Up to one
    a bit a fold reads the rects near the group, 336 px of 1,340 x 740, and not
    the map: with the rebuilds less than three tenths of it."""
    points = 8 + 11 + 2 * 11  # of the 22 bodies that move and have points
    loads = _loads(tmp_path, rects=rects, spread=spread)
    assert rects > 992 or loads < 0.3 * rects * points
