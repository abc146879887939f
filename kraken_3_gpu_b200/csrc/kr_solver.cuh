// kr_solver.cuh -- device side of the XPBD creature step (sm_100a).
//
// One connected component of the world (one creature, an "island") is
// advanced by a group of lanes of one warp.  Its bodies and constraints are
// staged in shared memory for the whole launch; lanes split each pass of
// solve units and the per-body collision work.  Nothing in here touches
// global memory except the read-only rect list of the map.
//
// Arithmetic follows tools/f32solver.mjs operation by operation: every
// intermediate is rounded to f32 with a non-contracting intrinsic
// (__fadd_rn/__fsub_rn/__fmul_rn/__fdiv_rn/__fsqrt_rn never fuse into an FMA),
// sin/cos are the f64 functions rounded once to f32 (Math.fround(Math.cos(x))),
// and the WGSL `%` uses the exact truncated quotient (f32solver.mjs:36-51).
#pragma once
#include <cstdint>
#include <type_traits>

#include "kr_sincos_tab.h"
#include "kr_units.h"

namespace kr {

// solver.wgsl:81, 93-94 and f32solver.mjs:26-33, as f32
constexpr float kSlackPos = 0.002f;
constexpr float kSlackAng = 0.0002f;
constexpr float kTau = 6.28318530718f;
constexpr float kPi = 3.14159265359f;
constexpr float kEpsDet = 1e-12f;
constexpr float kEpsSdf = 1e-12f;
constexpr float kSdfInf = 1e30f;
constexpr float kSdfValid = 1e29f;
constexpr float kInf = __builtin_huge_valf();

struct SolverConsts {
  float h, invH, invH2, linDamp, angDamp, maxSpeed, maxAngSpeed;
  int substeps, iterations;
};

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fsqrt(float a) { return __fsqrt_rn(a); }

// Math.fround(Math.sin(x)) and Math.fround(Math.cos(x)) for an f32 argument:
// both evaluated in f64 and rounded once to f32.  For |x| <= 2^20 the f64
// value comes from a three-part Cody-Waite reduction by pi/32, a table of
// sin / cos at k pi/32 and short Taylor series on |r| <= pi/64, the table
// value plus a small correction; larger or non-finite arguments use CUDA's
// f64 sincos.  Either way the f64 result is within a few f64 ulp of the
// exact value (measured on 4e7 arguments up to 2^20 against long-double
// sin / cos: relative error below 3.6e-16), so its rounding to f32 is the
// correctly rounded f32 except within a few 2^-29 of a rounding midpoint --
// the same class as glibc's and V8's f64 sin/cos.
//
// sin and cos of k pi / 32, k = 0..63, each the correctly rounded f64
__device__ const double2 kSinCosTab[64] = {
    {0.0, 1.0},
    {0.0980171403295606, 0.9951847266721969},
    {0.19509032201612828, 0.9807852804032304},
    {0.2902846772544624, 0.9569403357322088},
    {0.3826834323650898, 0.9238795325112867},
    {0.47139673682599764, 0.881921264348355},
    {0.5555702330196022, 0.8314696123025452},
    {0.6343932841636455, 0.773010453362737},
    {0.7071067811865476, 0.7071067811865476},
    {0.773010453362737, 0.6343932841636455},
    {0.8314696123025452, 0.5555702330196022},
    {0.881921264348355, 0.47139673682599764},
    {0.9238795325112867, 0.3826834323650898},
    {0.9569403357322088, 0.2902846772544624},
    {0.9807852804032304, 0.19509032201612828},
    {0.9951847266721969, 0.0980171403295606},
    {1.0, 0.0},
    {0.9951847266721969, -0.0980171403295606},
    {0.9807852804032304, -0.19509032201612828},
    {0.9569403357322088, -0.2902846772544624},
    {0.9238795325112867, -0.3826834323650898},
    {0.881921264348355, -0.47139673682599764},
    {0.8314696123025452, -0.5555702330196022},
    {0.773010453362737, -0.6343932841636455},
    {0.7071067811865476, -0.7071067811865476},
    {0.6343932841636455, -0.773010453362737},
    {0.5555702330196022, -0.8314696123025452},
    {0.47139673682599764, -0.881921264348355},
    {0.3826834323650898, -0.9238795325112867},
    {0.2902846772544624, -0.9569403357322088},
    {0.19509032201612828, -0.9807852804032304},
    {0.0980171403295606, -0.9951847266721969},
    {0.0, -1.0},
    {-0.0980171403295606, -0.9951847266721969},
    {-0.19509032201612828, -0.9807852804032304},
    {-0.2902846772544624, -0.9569403357322088},
    {-0.3826834323650898, -0.9238795325112867},
    {-0.47139673682599764, -0.881921264348355},
    {-0.5555702330196022, -0.8314696123025452},
    {-0.6343932841636455, -0.773010453362737},
    {-0.7071067811865476, -0.7071067811865476},
    {-0.773010453362737, -0.6343932841636455},
    {-0.8314696123025452, -0.5555702330196022},
    {-0.881921264348355, -0.47139673682599764},
    {-0.9238795325112867, -0.3826834323650898},
    {-0.9569403357322088, -0.2902846772544624},
    {-0.9807852804032304, -0.19509032201612828},
    {-0.9951847266721969, -0.0980171403295606},
    {-1.0, 0.0},
    {-0.9951847266721969, 0.0980171403295606},
    {-0.9807852804032304, 0.19509032201612828},
    {-0.9569403357322088, 0.2902846772544624},
    {-0.9238795325112867, 0.3826834323650898},
    {-0.881921264348355, 0.47139673682599764},
    {-0.8314696123025452, 0.5555702330196022},
    {-0.773010453362737, 0.6343932841636455},
    {-0.7071067811865476, 0.7071067811865476},
    {-0.6343932841636455, 0.773010453362737},
    {-0.5555702330196022, 0.8314696123025452},
    {-0.47139673682599764, 0.881921264348355},
    {-0.3826834323650898, 0.9238795325112867},
    {-0.2902846772544624, 0.9569403357322088},
    {-0.19509032201612828, 0.9807852804032304},
    {-0.0980171403295606, 0.9951847266721969}
};

// sin / cos beyond 2^20 and of non-finite arguments: CUDA's f64 sincos
// rounded to f32, out of line -- a cold path kept out of the instruction
// stream of the solve loops.
static __device__ __noinline__ float2 sincos_far(double x) {
  double sd, cd;
  sincos(x, &sd, &cd);
  return make_float2(static_cast<float>(sd), static_cast<float>(cd));
}

static __device__ __noinline__ float2 sincos_f64(float a) {
  const double x = static_cast<double>(a);
  if (!(fabs(x) <= 1048576.0)) return sincos_far(x);
  // x = k pi/32 + r, |r| <= pi/64: pi/32 in three parts (29, 29 and 53
  // bits), so k p1 and k p2 are exact for |k| < 2^24
  const double k = rint(x * 10.185916357881302);  // 32/pi
  double r = fma(-k, 0x1.921fb54000000p-4, x);
  r = fma(-k, 0x1.10b4611000000p-34, r);
  r = fma(-k, 0x1.4c4c6628b80dcp-63, r);
  const double r2 = r * r;
  // Taylor series on |r| <= pi/64: sin through r^7 (truncation below 5e-18
  // relative), cos - 1 through r^8 (below 3e-20)
  double ps = -1.0 / 5040;
  ps = fma(ps, r2, 1.0 / 120);
  ps = fma(ps, r2, -1.0 / 6);
  const double sr = fma(r * r2, ps, r);
  double pc = 1.0 / 40320;
  pc = fma(pc, r2, -1.0 / 720);
  pc = fma(pc, r2, 1.0 / 24);
  pc = fma(pc, r2, -0.5);
  const double cm1 = r2 * pc;                     // cos r - 1
  // sin(t + r) = S + (S (cos r - 1) + C sin r), cos(t + r) = C + (C (cos r - 1) - S sin r):
  // the table value plus a small correction
  const double2 t = __ldg(&kSinCosTab[static_cast<int>(static_cast<long long>(k) & 63)]);
  return make_float2(static_cast<float>(t.x + fma(t.x, cm1, t.y * sr)),
                     static_cast<float>(t.y + fma(t.y, cm1, -(t.x * sr))));
}

// The same values in f32 arithmetic (Ziv's rounding test): sin and cos as an
// unevaluated sum h + l of two f32 whose error bound err is known; where
// h + (l - err) and h + (l + err) round to one f32, that is the rounding of
// the exact value and of the f64 value above, whose own error err includes.
// Returns the distance of the two roundings, 0 where the values stand; where
// it is not (one value in 2,400 to 4,700 of an octave from 2^-7 up, one in
// 1,300 between 2^-8 and 2^-7, fewer and fewer below, none below 2^-13) and
// for |a| > kSinCosNearMax sincos_f64 decides.  The f64 chain cost 241 cycles,
// mostly conversions (18 cycles each) and the serial reduction and series.
//
// a = k pi/256 + r1 + rl: p1 = pi/256 to 24 bits, so r1 = a - k p1 is exact
// (a multiple of 2^-31 below 2^-7.3, or a itself for k = 0), and rl = -k p2
// with |rl| < 2^-18.6.  With the table's S + Sl, C + Cl, r = r1 + rl, m =
// cos r - 1 and n = rl - r^3 / 6:
//   sin = S + C r1 + (Sl + Cl r1 + C n + S m),
//   cos = C - S r1 + (Cl - Sl r1 - S n + C m),
// S + C r1 and its two rounding errors exact (the product by fma, the sum
// because |S| is 0 or above |C r1|).  Error: r^2 (|m| <= r^2 / 2) times
// below 12 units of 2^-24 for the roundings of r, r^2, m and the two sums
// it enters, Sl m among them, times |S| (cos: |C|); |k| 2^-53 for the
// roundings of rl, n, its sum and p2 (2^-55.4 |k| each); r^2 2^-28.9 for r^5 /
// 120 (|r| <= pi / 512).  Every term vanishes with a, so an angle of 0, as
// fixed bodies have it, and small ones are decided like any other (a bound of
// 2^-43 in the place of the last term left all below 2^-18 to sincos_f64: 256
// chains on fixed bodies at angle 0, 100 steps, 9.8 ms, now 4.0).  What is
// left, below 2^-47 (the other roundings, the f64 value), has no term: that
// the bound holds is checked, not proven, over all 2,231,369,730 arguments
// from -64 to 64 -- no accepted value differs from sincos_f64's
// (tests/test_solver_host.py repeats it).
//
// tab: kSinNear in shared memory.  As 16-byte __ldg gathers its look-ups were
// the longest part of a pin (32 lanes, 32 lines: two of them 360 of 550
// cycles); two 8-byte shared loads take a few bank conflicts each.
__device__ __forceinline__ float sincos_near(const float2 *tab, float a, float *s, float *c) {
  const float t = fmaf(a, 0x1.45f306p6f, 12582912.f);  // 256/pi; the sum's low bits hold k
  const float2 *e = tab + (__float_as_int(t) & 511);
  const float2 ts = e[0], tc = e[128];
  const float4 T = make_float4(ts.x, ts.y, tc.x, tc.y);
  const float k = fsub(t, 12582912.f);
  const float r1 = fmaf(-k, 0x1.921fb6p-7f, a), rl = fmul(-k, -0x1.777a5cp-32f);
  const float r = fadd(r1, rl), rr = fmul(r, r);
  const float n = fmaf(fmul(r, rr), -1.f / 6, rl);
  const float m = fmul(rr, fmaf(rr, 1.f / 24, -0.5f));
  const float w = fmul(rr, 0x1.8p-22f), e0 = fmaf(fabsf(k), 0x1p-53f, fmul(rr, 0x1.1p-29f));
  const float es = fmaf(fabsf(T.x), w, e0), ec = fmaf(fabsf(T.z), w, e0);
  const float qs = fmul(T.z, r1), hs = fadd(T.x, qs);
  const float ls = fadd(fmaf(T.x, m, fmaf(T.z, n, fmaf(T.w, r1, T.y))),
                        fadd(fmaf(T.z, r1, -qs), fsub(qs, fsub(hs, T.x))));
  const float qc = fmul(-T.x, r1), hc = fadd(T.z, qc);
  const float lc = fadd(fmaf(T.z, m, fmaf(-T.x, n, fmaf(-T.y, r1, T.w))),
                        fadd(fmaf(-T.x, r1, -qc), fsub(qc, fsub(hc, T.z))));
  *s = fadd(hs, fadd(ls, es));
  *c = fadd(hc, fadd(lc, ec));
  return fadd(fabsf(fsub(*s, fadd(hs, fsub(ls, es)))), fabsf(fsub(*c, fadd(hc, fsub(lc, ec)))));
}
constexpr float kSinCosNearMax = 64.f;

// The table into shared memory, by every thread of the block, its first
// quarter repeated at the end for the cosine; __syncthreads before its first
// use.
constexpr int kSinEntries = 640;
__device__ __forceinline__ void stage_sin(float2 *tab) {
  for (int i = threadIdx.x; i < kSinEntries; i += blockDim.x) tab[i] = kSinNear[i & 511];
}

__device__ __forceinline__ void sincos_r(const float2 *tab, float a, float *s, float *c) {
  if (!(sincos_near(tab, a, s, c) == 0.f && fabsf(a) <= kSinCosNearMax)) {
    const float2 f = sincos_f64(a);
    *s = f.x;
    *c = f.y;
  }
}

// Quotients by a shared reciprocal: y = 1 / b from the hardware estimate and
// one Newton step, then q = a y corrected once by its residual, q + y (a - b
// q), the residual exact in one fma (the scheme of P. Markstein, IBM J. Res.
// Dev. 34(1), 1990, where y rounded to nearest makes the result RN(a / b)).
// For this y it was checked instead of proven: all 2^46 pairs of mantissas of
// a and b give RN(a / b), and the estimate scales exactly with the exponent of
// b over 2^-60 .. 2^60.  The same holds with y = RN(1 / b), unless every
// mantissa bit of b is set.  Three instructions in sequence per quotient and
// no branch, against about 45 cycles and a branch per __fdiv_rn.
// Valid for |b| in 2^-60 .. 2^60 and |a| in 2^-100 .. 2^60 or a = 0: no
// exponent comes near its limits, a residual is a multiple of 2^-149.
__device__ __forceinline__ float recip(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return fmaf(fmaf(-b, y, 1.f), y, y);
}
__device__ __forceinline__ bool recip_ok(float b) { return fabsf(b) > 0x1p-60f && fabsf(b) < 0x1p60f; }
__device__ __forceinline__ float quot(float a, float b, float y) {
  const float q = fmul(a, y);
  return fmaf(fmaf(-b, q, a), y, q);
}

// trunc(x / TAU) exactly, as the f64 quotient of f32solver.mjs:38 gives it.
// The f32 estimate q = trunc(x * (1/TAU)) is off by at most one near an
// integer; the remainder x - q*TAU is then exact in one fma (both terms are
// multiples of 2^-21 for |x| >= 4 and it stays below 8 in magnitude) and
// decides the correction.  |x| < 4 has quotient 0.
__device__ __forceinline__ float trunc_quot_tau(float x) {
  if (fabsf(x) < 4.f) return 0.f;
  float q = truncf(__fmul_rn(x, 0.15915494f));
  const float r = fmaf(-q, kTau, x);
  if (x >= 0.f) {
    if (r < 0.f) q -= 1.f;
    else if (r >= kTau) q += 1.f;
  } else {
    if (r > 0.f) q += 1.f;
    else if (r <= -kTau) q -= 1.f;
  }
  return q;
}

// angleDeltaF, f32solver.mjs:36-43 (solver.wgsl:103-108) and wrapAngleF,
// f32solver.mjs:45-51 (solver.wgsl:96-101), of the difference x.  Out of
// line: angles of neighbouring bodies differ by more than kWrapNear only
// while one of them has been wrapped at 50 rad and the other has not.
static __device__ __noinline__ float wrap_far(float x) {
  const float q = trunc_quot_tau(x);
  const float d = fsub(x, fmul(kTau, q));
  if (d > kPi) return fsub(d, kTau);
  if (d < -kPi) return fadd(d, kTau);
  return d;
}

// The same for |x| <= kWrapNear < kTau + kPi (or NaN): the quotient is 0 or
// +-1, and either way a difference beyond pi moves by one kTau, rounded once.
// Five instructions instead of the quotient's twenty in sequence (the angle
// constraint evaluates five of these in a row: its chain is 441 cycles instead
// of 764 with the quotient).
constexpr float kWrapNear = 9.42f;
__device__ __forceinline__ float wrap_near(float x) {
  const float d = fsub(x, copysignf(kTau, x));
  return fabsf(x) <= kPi ? x : d;
}
__device__ __forceinline__ float wrap_angle(float x) { return fabsf(x) > kWrapNear ? wrap_far(x) : wrap_near(x); }
__device__ __forceinline__ float angle_delta(float a, float b) { return wrap_angle(fsub(a, b)); }

// lengthF, f32solver.mjs:54-56 (WGSL length(vec2f))
__device__ __forceinline__ float length2(float x, float y) {
  return fsqrt(fadd(fmul(x, x), fmul(y, y)));
}

// sdfF, f32solver.mjs:139-166 (solver.wgsl:114-147): the fold over rects
// stored as x, y, x + w, y + h (all f32, the sums rounded once as
// solver.wgsl:120-121 computes r.x + r.w), added in ascending order.  The
// division of the outward normal is deferred to the final winner: bnx/bny are
// overwritten by every later winner, so only the last winner's dx/best,
// dy/best survive.
struct SdfFold {
  float best, thr;  // thr: f32 best * best, +inf for 1e30 * 1e30
  float wdx, wdy, inx, iny;
  bool inside;
  __device__ __forceinline__ SdfFold()
      : best(kSdfInf), thr(kInf), wdx(0.f), wdy(0.f), inx(0.f), iny(0.f), inside(false) {}
  __device__ __forceinline__ void add(const float4 r, float x, float y) {
    const float cx = x < r.x ? r.x : (x > r.z ? r.z : x);
    const float cy = y < r.y ? r.y : (y > r.w ? r.w : y);
    const float dx = fsub(x, cx), dy = fsub(y, cy);
    const float d2 = fadd(fmul(dx, dx), fmul(dy, dy));
    if (d2 > kEpsSdf) {
      if (d2 < thr) {
        best = fsqrt(d2);
        thr = fmul(best, best);
        wdx = dx; wdy = dy;
        inside = false;
      }
    } else {
      const float dl = fsub(x, r.x), dr = fsub(r.z, x), dt = fsub(y, r.y), db = fsub(r.w, y);
      float m = dl, nx = -1.f, ny = 0.f;
      if (dr < m) { m = dr; nx = 1.f; ny = 0.f; }
      if (dt < m) { m = dt; nx = 0.f; ny = -1.f; }
      if (db < m) { m = db; nx = 0.f; ny = 1.f; }
      const float d = -m;
      if (d < best) {
        best = d;
        thr = fmul(best, best);
        inx = nx; iny = ny;
        inside = true;
      }
    }
  }
  // the correction of a point of radius r, false if it needs none
  __device__ __forceinline__ bool push(float r, float *dx, float *dy) const {
    if (best > kSdfValid) return false;
    const float pen = fsub(r, best);
    if (!(pen > kSlackPos)) return false;
    *dx = fmul(inside ? inx : fdiv(wdx, best), pen);
    *dy = fmul(inside ? iny : fdiv(wdy, best), pen);
    return true;
  }
};

// Exact rect culling.
//
// Let D = max(largest collision radius, largest half-thickness min(w,h)/2 of
// a rect) + 2.  Drop any rects farther than D from an evaluated point.  The
// sequential SDF fold then returns the same winner, or in both cases a
// winner farther than D - 1 (> radius + 1: no correction):
//  * a state's threshold f(best^2) never falls below the squared distance
//    of any rect processed so far, except that an inside winner sets it to
//    at most half-thickness^2 < (D - 1)^2; a dropped rect (d^2 > D^2) can
//    therefore only beat states with threshold >= (D - 1)^2 ("far" states);
//  * by monotone rounding, a rect that fails to beat a far state is itself
//    far, and an inside rect beats every far state; so the folds with and
//    without the dropped rects hold equal states or two far states.
//
// Each body keeps the set of rects that can lie within D of one of its points
// while its centre stays within kNearMove of a reference position (kFarMove
// if no rect is that near): a bit mask over the creature's near list (the
// rects near any of its bodies, ascending).
// Bodies move a few px per env step, so the sets are rebuilt every few steps
// instead of once per collision pass (3 % of the passes on the default maps),
// and a body whose set is empty needs nothing but the test that it still is
// near its reference.
//
// The list takes the rects within the widest of three moves for which it fits,
// kFarMove, half of it or kNearMove: a body that its joints hold in a wall is
// pushed by more than kNearMove in every pass, and its remaining points fold
// over the list as far as the list holds, else over the map.  A group with
// more rects within kNearMove is dense: the list's words are a bit map of the
// rects within kFarMove, 1 to 128 rects a bit.  A dense fold has more to
// look at and diverges (256 chains among 405 small rects, 100 steps: 34 to 37
// ms dense, 13.8 with a list within kNearMove), a fold over the map more yet
// (1,024 creatures x 200 steps among 1,024 rects, where a few groups have no
// list: 1,040 ms with every rect, 137 now).
constexpr int kMaxCulled = 62;      // near list entries; bit b of a mask covers entries b << shift ...
constexpr int kCullWords = 32;      // the near list, two entries a word, and the references' origin behind it
static_assert(2 * kCullWords >= kMaxCulled + 2, "");
constexpr unsigned kNearBit = 1u << 31;  // of a mask: the body holds within kNearMove only
constexpr float kNearMove = 8.f, kFarMove = 32.f;
constexpr float kCullPad = 1.f;     // rounding of the box tests

// A group of G lanes of one warp advancing one creature (G = 32, 16, 8):
// lanes of a group loop with stride G and synchronize, reduce and vote only
// among themselves, so a warp can carry 32 / G creatures of one template.
template <int G>
struct Lanes {
  int lane;        // 0 .. G-1
  int base;        // first warp lane of the group
  unsigned mask;   // the group's lanes in the warp
  __device__ __forceinline__ explicit Lanes(int warp_lane)
      : lane(warp_lane & (G - 1)), base(warp_lane & ~(G - 1)),
        mask(G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (warp_lane & ~(G - 1)))) {}
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  __device__ __forceinline__ unsigned ballot(bool p) const {
    const unsigned b = __ballot_sync(mask, p);
    return G == 32 ? b : (b >> base) & ((1u << G) - 1u);
  }
  __device__ __forceinline__ float min(float v) const {
    for (int o = G / 2; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(mask, v, o, G));
    return v;
  }
  __device__ __forceinline__ float max(float v) const {
    for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(mask, v, o, G));
    return v;
  }
};

// Shared-memory view of one island (one creature).
//
// The solve list is swept in units: a pin or grip constraint, an angle
// constraint, or a pin and the angle constraint of the same two bodies when
// no other constraint on either body lies between them in the list (every
// joint of a creature).  A unit's two bodies are loaded once, solved in
// registers -- pin, then angle, as the list orders them -- and stored once.
// Units are grouped in passes of body-disjoint units, one unit per lane; a
// pass order that keeps every pair of units sharing a body in list order
// gives the sequential sweep's bits (the harness check color-order-free,
// harness.js:1172-1193, pins this for the reference's colour classes).
// The sweep is bound by its chain of dependent passes, each a round trip
// through shared memory: per-constraint levels make a 6 x 7 body 12 of them,
// as units it is 6.
//
// Bodies are float4 records (one 16-byte load or store instead of three
// 4-byte ones).
struct Island {
  float4 *P;           // committed x, y, angle; w: the collision reference position (near_pack)
  float4 *Q;           // predicted x, y, angle; w: the mask of near rects
  float4 *V;           // velocity vx, vy, av (batched engine: the same records as Q, see below)
  const float2 *tab;   // kSinNear in shared memory
  const float4 *body;  // inverse mass, inverse inertia, reach, point offset | count << 16
  const float4 *pts;   // collision points: x, y, radius, body; grouped per body in groupCollPoints order
  unsigned short *cull;       // near list (kMaxCulled rect indices), origin
  unsigned char *list;        // bodies with near rects: one or two points from the front, more from the back
  int nb;
  // drop-in world: one dynamic record of 5 float4 per unit, pass offsets
  float4 *units;
  int nu, npass;
  const int *off;      // npass + 1 unit offsets
  float4 *force;       // fx, fy, torque
  // batched engine: the template's static records (3 float4 per lane and
  // pass), per motor {target, lambda}, from grip0 on per arm the grip's lambda
  // and one pair for idle lanes, break force per arm
  const float4 *recs;
  float2 *mot;
  float *brk;
  int grip0;
  float comp_m;        // motor compliance of the creature
  int arms;
};

// ab word of a unit: body A, body B << 8, and flags.  Drop-in world: B is 0xff
// for the world.
constexpr unsigned kHasPin = 1u << 16, kPinBroken = 1u << 17, kHasAngle = 1u << 18, kAngleBroken = 1u << 19,
                   kPinIsGrip = 1u << 20, kPinTame = 1u << 21,
                   // two bodies whose inverse masses are finite (an update of 0 times them is 0)
                   kBounded = 1u << 22;

// The flags by which a drop-in unit takes the short forms below: its pin is
// tame or it has none (a disabled pin's levers enter sums with 0, so they must
// be finite too), its masses are bounded
__device__ inline unsigned unit_forms(bool has_pin, bool self, float lax, float lay, float lbx, float lby, float wA,
                                      float wIA, float wB, float wIB) {
  return (!has_pin || pin_tame(lax, lay, lbx, lby, wA, wIA, wB, wIB) ? kPinTame : 0u) |
         (!self && fabsf(wA) + fabsf(wIA) + fabsf(wB) + fabsf(wIB) < 1e30f ? kBounded : 0u);
}

// The speed clamp of integrateF and finalizeF.  A squared speed of at most
// 0.999 maxSpeed^2 has a length of at most maxSpeed however it rounds, so the
// square root is taken only near the limit (and where a square overflows).
__device__ __forceinline__ void clamp_speed(const SolverConsts &K, float &vx, float &vy) {
  const float s2 = fadd(fmul(vx, vx), fmul(vy, vy));
  if (!(s2 < (K.maxSpeed > 0.f ? 0.999f * K.maxSpeed * K.maxSpeed : -1.f))) {
    const float sp = fsqrt(s2);
    if (sp > K.maxSpeed) {
      const float k = fdiv(K.maxSpeed, sp);
      vx = fmul(vx, k); vy = fmul(vy, k);
    }
  }
}

// integrateF, f32solver.mjs:177-200 (solver.wgsl:166-205).  World: the
// drop-in's bodies (forces, immovable bodies, velocities in their own
// records); otherwise the batched engine's, which have neither and whose
// predicted state takes the place of the velocity: a substep reads the
// velocity only here and writes it only in finalize_body.
template <bool World>
__device__ __forceinline__ void integrate_body(const SolverConsts &K, Island &S, int i) {
  const float4 bd = S.body[i];
  const float im = bd.x, ii = bd.y;
  const float4 p = S.P[i];
  const float mask = S.Q[i].w;  // of near rects: the collision pass's
  if (World && im == 0.f && ii == 0.f) {
    S.Q[i] = make_float4(p.x, p.y, p.z, mask);
    S.V[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  float4 v = S.V[i];
  const float4 f = World ? S.force[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  float vx = fmul(fadd(v.x, fmul(fmul(K.h, im), f.x)), K.linDamp);
  float vy = fmul(fadd(v.y, fmul(fmul(K.h, im), f.y)), K.linDamp);
  float av = fmul(fadd(v.z, fmul(fmul(K.h, ii), f.z)), K.angDamp);
  clamp_speed(K, vx, vy);
  if (av > K.maxAngSpeed) av = K.maxAngSpeed;
  else if (av < -K.maxAngSpeed) av = -K.maxAngSpeed;
  if (!(vx == vx) || !(vy == vy)) { vx = 0.f; vy = 0.f; }
  if (!(av == av)) av = 0.f;
  if (World) S.V[i] = make_float4(vx, vy, av, 0.f);
  S.Q[i] = make_float4(fadd(p.x, fmul(K.h, vx)), fadd(p.y, fmul(K.h, vy)), fadd(p.z, fmul(K.h, av)), mask);
  if (World) S.force[i] = make_float4(0.f, 0.f, 0.f, f.w);
}

// solvePinF, f32solver.mjs:203-256 (solver.wgsl:225-290) on two body records
// in registers; grips are pins against the world.  Without a body B: b holds
// the anchor as its position with angle 1 (any angle with positive sine and
// cosine), lb and the masses of B are 0 (the same values as the reference's
// branch).  lx, ly: the multiplier, updated.
struct PinArgs {
  float lax, lay, lbx, lby, wA, wIA, wB, wIB, alphaTilde;
  bool hasB;
};

// The reference form: every branch as the reference takes it, for the
// arguments pin_near cannot take, and for units whose two bodies are one
// (self: a and b the same record, the result in b).
struct PinOut {
  float4 a, b;
  float lx, ly;
};
__device__ inline PinOut pin_any(PinArgs U, float4 a, float4 b, float lx, float ly, bool self) {
  const PinOut in{a, b, lx, ly};
  const float2 ta = sincos_f64(a.z), tb = sincos_f64(b.z);
  const float sa = ta.x, ca = ta.y, sb = tb.x, cb = tb.y;
  const float rax = fsub(fmul(U.lax, ca), fmul(U.lay, sa)), ray = fadd(fmul(U.lax, sa), fmul(U.lay, ca));
  const float rbx = fsub(fmul(U.lbx, cb), fmul(U.lby, sb)), rby = fadd(fmul(U.lbx, sb), fmul(U.lby, cb));
  const float Cx = fsub(fadd(a.x, rax), fadd(b.x, rbx)), Cy = fsub(fadd(a.y, ray), fadd(b.y, rby));
  if (!(Cx == Cx) || !(Cy == Cy)) return in;
  if (fadd(fmul(Cx, Cx), fmul(Cy, Cy)) < fmul(kSlackPos, kSlackPos)) return in;
  const float pax = -ray, pay = rax, pbx = -rby, pby = rbx;
  const float wSum = fadd(U.wA, U.wB);
  const float k00 = fadd(fadd(wSum, fmul(fmul(U.wIA, pax), pax)), fmul(fmul(U.wIB, pbx), pbx));
  const float k01 = fadd(fmul(fmul(U.wIA, pax), pay), fmul(fmul(U.wIB, pbx), pby));
  const float k11 = fadd(fadd(wSum, fmul(fmul(U.wIA, pay), pay)), fmul(fmul(U.wIB, pby), pby));
  const float det = fsub(fmul(k00, k11), fmul(k01, k01));
  if (fabsf(det) < kEpsDet) return in;
  const float bx = fadd(Cx, fmul(U.alphaTilde, lx)), by = fadd(Cy, fmul(U.alphaTilde, ly));
  const float i00 = fdiv(k11, det), i11 = fdiv(k00, det), i01 = -fdiv(k01, det);
  const float dlx = -fadd(fmul(i00, bx), fmul(i01, by)), dly = -fadd(fmul(i01, bx), fmul(i11, by));
  if (!(dlx == dlx) || !(dly == dly)) return in;
  lx = fadd(lx, dlx);
  ly = fadd(ly, dly);
  a.x = fadd(a.x, fmul(U.wA, dlx));
  a.y = fadd(a.y, fmul(U.wA, dly));
  a.z = fadd(a.z, fmul(U.wIA, fadd(fmul(pax, dlx), fmul(pay, dly))));
  if (self) b = a;
  if (U.hasB) {
    b.x = fsub(b.x, fmul(U.wB, dlx));
    b.y = fsub(b.y, fmul(U.wB, dly));
    b.z = fsub(b.z, fmul(U.wIB, fadd(fmul(pbx, dlx), fmul(pby, dly))));
  }
  return PinOut{a, b, lx, ly};
}

// The same operations for a tame pin (kr_units.h pin_tame), without a branch:
// the reference's early returns become one condition on the update (on: the
// pin is there and not broken), which otherwise adds 0.  Returns false, with
// a, b, lx, ly of no use, where another path is needed: an angle the rounding
// test does not decide, an error beyond 1e15 or NaN.  A predicate costs about 13 cycles and a branch on it 25 more
// in a chain that nothing else hides, so the tests are folded into sums.
// World: lby and the compliance may be other than 0 (the engine's pins have
// neither, so their terms are left out: the same values).
template <bool World>
__device__ __forceinline__ bool pin_near(const float2 *tab, const PinArgs &U, bool on, float4 &a, float4 &b, float &lx,
                                         float &ly) {
  float sa, ca, sb, cb;
  const float spread = fadd(sincos_near(tab, a.z, &sa, &ca), sincos_near(tab, b.z, &sb, &cb));
  const float amax = fmaxf(fabsf(a.z), fabsf(b.z));
  const float rax = fsub(fmul(U.lax, ca), fmul(U.lay, sa)), ray = fadd(fmul(U.lax, sa), fmul(U.lay, ca));
  const float rbx = World ? fsub(fmul(U.lbx, cb), fmul(U.lby, sb)) : fmul(U.lbx, cb);
  const float rby = World ? fadd(fmul(U.lbx, sb), fmul(U.lby, cb)) : fmul(U.lbx, sb);
  const float Cx = fsub(fadd(a.x, rax), fadd(b.x, rbx)), Cy = fsub(fadd(a.y, ray), fadd(b.y, rby));
  const float pax = -ray, pay = rax, pbx = -rby, pby = rbx;
  const float wSum = fadd(U.wA, U.wB), csq = fadd(fmul(Cx, Cx), fmul(Cy, Cy));
  const float k00 = fadd(fadd(wSum, fmul(fmul(U.wIA, pax), pax)), fmul(fmul(U.wIB, pbx), pbx));
  const float k01 = fadd(fmul(fmul(U.wIA, pax), pay), fmul(fmul(U.wIB, pbx), pby));
  const float k11 = fadd(fadd(wSum, fmul(fmul(U.wIA, pay), pay)), fmul(fmul(U.wIB, pby), pby));
  const float det = fsub(fmul(k00, k11), fmul(k01, k01));
  const float bx = World ? fadd(Cx, fmul(U.alphaTilde, lx)) : Cx, by = World ? fadd(Cy, fmul(U.alphaTilde, ly)) : Cy;
  const float y = recip(det);
  const float i00 = quot(k11, det, y), i11 = quot(k00, det, y), i01 = -quot(k01, det, y);
  const bool upd = on && csq >= fmul(kSlackPos, kSlackPos);
  const float dlx = upd ? -fadd(fmul(i00, bx), fmul(i01, by)) : 0.f;
  const float dly = upd ? -fadd(fmul(i01, bx), fmul(i11, by)) : 0.f;
  lx = fadd(lx, dlx);
  ly = fadd(ly, dly);
  a.x = fadd(a.x, fmul(U.wA, dlx));
  a.y = fadd(a.y, fmul(U.wA, dly));
  a.z = fadd(a.z, fmul(U.wIA, fadd(fmul(pax, dlx), fmul(pay, dly))));
  b.x = fsub(b.x, fmul(U.wB, dlx));
  b.y = fsub(b.y, fmul(U.wB, dly));
  b.z = fsub(b.z, fmul(U.wIB, fadd(fmul(pbx, dlx), fmul(pby, dly))));
  const bool small = World ? fadd(fabsf(bx), fabsf(by)) < 1e15f : csq < 1e30f;
  // World: a disabled pin's levers must come out finite, since 0 times them is
  // added (the engine's grips have the template's levers, and angles that are
  // wrapped at 50 rad: 1 % of 12 creatures' step for a test that holds)
  const bool near = amax <= kSinCosNearMax;
  return World ? near && (!on || (small && spread == 0.f)) : !on || (near && small && spread == 0.f);
}

// solveAngleF, f32solver.mjs:258-301 (solver.wgsl:292-350): muscle
// (compliant) part, then the one-sided joint limit.  az, bz: the angles; l:
// the multiplier, updated.
struct AngleArgs {
  float rest, mn, mx, tgt, alphaTilde, wA, wB;
  bool hasB;
};

// The reference form (as pin_any)
__device__ inline float3 angle_any(AngleArgs U, float az, float bz, float l, bool self) {
  const float wSum = fadd(U.wA, U.wB);
  if (wSum <= 0.f) return make_float3(az, bz, l);
  const float dev = angle_delta(U.hasB ? angle_delta(bz, az) : az, U.rest);
  const float C = angle_delta(dev, U.tgt);
  if (!(C == C)) return make_float3(az, bz, l);
  if (fabsf(C) >= kSlackAng) {
    const float dl = -fdiv(fadd(C, fmul(U.alphaTilde, l)), fadd(wSum, U.alphaTilde));
    if (!(dl == dl)) return make_float3(az, bz, l);
    l = fadd(l, dl);
    if (U.hasB) {
      bz = fadd(bz, fmul(U.wB, dl));
      az = fsub(self ? bz : az, fmul(U.wA, dl));
      if (self) bz = az;
    } else {
      az = fadd(az, fmul(U.wA, dl));
    }
  }
  const float dev2 = angle_delta(U.hasB ? angle_delta(bz, az) : az, U.rest);
  float over = 0.f;
  if (dev2 > U.mx) over = fsub(dev2, U.mx);
  else if (dev2 < U.mn) over = fsub(dev2, U.mn);
  if (fabsf(over) >= kSlackAng) {
    const float dl2 = -fdiv(over, wSum);
    if (U.hasB) {
      bz = fadd(bz, fmul(U.wB, dl2));
      az = fsub(self ? bz : az, fmul(U.wA, dl2));
      if (self) bz = az;
    } else {
      az = fadd(az, fmul(U.wA, dl2));
    }
  }
  return make_float3(az, bz, l);
}

// The same operations in near form (as pin_near).  Where a term is used, |C|
// and |over| are at least kSlackAng, so the quotients' numerators are 0 or
// above 2^-40.  yw: 1 / (wA + wB) for quot; reach: kWrapNear, or negative
// where the compliance is out of quot's range.  World: any rest, target, masses and a
// missing body B; the engine's joints have 0 <= rest <= 6.27 and |target| <
// 1.95, so only the differences of the two angles can exceed kWrapNear.
template <bool World>
__device__ __forceinline__ bool angle_near(const AngleArgs &U, float yw, float reach, bool on, float &az, float &bz,
                                           float &l) {
  const bool hasB = !World || U.hasB;
  const float wSum = fadd(U.wA, U.wB), den = fadd(wSum, U.alphaTilde);
  const float y = recip(den);
  const float x1 = hasB ? fsub(bz, az) : 0.f;
  const float x2 = fsub(hasB ? wrap_near(x1) : az, U.rest);
  const float x3 = fsub(wrap_near(x2), U.tgt);
  const float C = wrap_near(x3);
  const float num = fadd(C, fmul(U.alphaTilde, l));
  const float dl = on && fabsf(C) >= kSlackAng ? -quot(num, den, y) : 0.f;
  l = fadd(l, dl);
  az = hasB ? fsub(az, fmul(U.wA, dl)) : fadd(az, fmul(U.wA, dl));
  bz = hasB ? fadd(bz, fmul(U.wB, dl)) : bz;
  const float x4 = hasB ? fsub(bz, az) : 0.f;
  const float x5 = fsub(hasB ? wrap_near(x4) : az, U.rest);
  const float dev2 = wrap_near(x5);
  const float o1 = fsub(dev2, U.mx), o2 = fsub(dev2, U.mn);
  // (limits the wrong way round: above the maximum the minimum does not act)
  const bool hi = o1 >= kSlackAng, lim = hi || (o2 <= -kSlackAng && !(World && dev2 > U.mx));
  const float dl2 = on && lim ? -quot(hi ? o1 : o2, wSum, yw) : 0.f;
  az = hasB ? fsub(az, fmul(U.wA, dl2)) : fadd(az, fmul(U.wA, dl2));
  bz = hasB ? fadd(bz, fmul(U.wB, dl2)) : bz;
  float far = fmaxf(fabsf(x1), fabsf(x4));
  if (World) far = fmaxf(fmaxf(far, fabsf(x2)), fmaxf(fabsf(x3), fabsf(x5)));
  const bool tame = !World || (recip_ok(den) && recip_ok(wSum) && wSum > 0.f);
  return !on || (tame && fabsf(num) < 0x1p60f && far <= reach);  // NaN fails by num
}

// A unit in the reference form.  Out of line, values in and values out:
// records passed by address would live in local memory on the near path too.
struct UnitOut {
  float4 a, b;
  float lx, ly, l;
};
static __device__ __noinline__ UnitOut unit_any(PinArgs U, AngleArgs V, bool pin, bool angle, bool self, float4 a,
                                                float4 b, float lx, float ly, float l) {
  if (pin) {
    const PinOut o = pin_any(U, a, b, lx, ly, self);
    a = self ? o.b : o.a; b = o.b; lx = o.lx; ly = o.ly;
  }
  if (angle) {
    const float3 o = angle_any(V, a.z, b.z, l, self);
    a.z = o.x; b.z = o.y; l = o.z;
  }
  return UnitOut{a, b, lx, ly, l};
}

// One sweep of the solve list, batched engine.  first: the first sweep of a
// substep, where every multiplier starts from 0.  A pin's multiplier only
// enters its own equation times its compliance, which is 0 for the
// template's pins and grips, so only the grips' (the break test) and the
// motors' are kept.  Joints, grips (held or not) and idle lanes run one
// instruction stream; a pass ends in its only branch, for units that need
// the reference form (their bodies are still in shared memory as they were).
// The pass's 230 + 340 cycles of dependent arithmetic are what a creature's
// step consists of.
template <int G>
__device__ __forceinline__ void solve_engine(const SolverConsts &K, Island &S, bool first, const Lanes<G> &L) {
  const float alpha_m = fmul(S.comp_m, K.invH2), reach = alpha_m < 0x1p59f ? kWrapNear : -1.f;
  const float4 *rec = S.recs + 3 * L.lane;
  for (int p = 0; p < S.npass; p++) {
    const float4 r0 = rec[0], r1 = rec[1], r2 = rec[2];
    const unsigned ab = __float_as_uint(r0.x);
    const int A = ab & 0xff, B = (ab >> 8) & 0xff, m = (ab >> 16) & 0xff;
    const bool joint = (ab & kRecJoint) != 0;
    float4 a = S.Q[A], b = S.Q[B];
    const float2 mo = S.mot[m];
    const PinArgs U{r0.y, r0.z, r0.w, 0.f, r1.x, r1.y, r1.z, r1.w, 0.f, joint};
    const AngleArgs V{r2.x, r2.y, r2.z, mo.x, alpha_m, r1.y, r1.w, true};
    const float yw = r2.w;
    rec += 3 * G;
    const bool held = joint || b.w == 0.f;  // b.w: an anchor's broken flag (the spare record: broken)
    // multipliers: a joint's is mo.y, a grip's are both (each ignores the other's)
    const float m0 = first ? 0.f : mo.x, m1 = first ? 0.f : mo.y;
    float lx = m0, ly = m1, l = m1;
    const bool op = pin_near<false>(S.tab, U, held, a, b, lx, ly);
    const bool oa = angle_near<false>(V, yw, reach, joint, a.z, b.z, l);
    if (__builtin_expect(!(op && oa), 0)) {
      const UnitOut o = unit_any(U, V, held, joint, false, S.Q[A], S.Q[B], joint ? 0.f : m0, joint ? 0.f : m1, m1);
      a = o.a; b = o.b; lx = o.lx; ly = o.ly; l = o.l;
    }
    S.Q[A] = a;
    if (joint) S.Q[B] = b;
    S.mot[m] = make_float2(joint ? mo.x : lx, joint ? l : ly);
    L.sync();
  }
}

// One sweep of the solve list, drop-in world: unit records
// {ab, lax, lay, lbx} {lby, 1 / mass A, 1 / inertia A, 1 / mass B}
// {1 / inertia B, rest, min, max} {target, pin compliance / h^2, angle
// compliance / h^2, recip of the inertias' sum} {lambda x, y, lambda, break
// force}; lb is 0 without a body B.  The next pass's offset loads while the
// current one computes.
constexpr int kWorldRec = 5;
template <int G>
__device__ __forceinline__ void solve_world(Island &S, bool first, const Lanes<G> &L) {
  int beg = 0, end = S.npass > 0 ? S.off[1] : 0;
  for (int p = 0; p < S.npass; p++) {
    const int u = beg + L.lane;  // passes hold at most 32 units
    const bool mine = u < end;
    const int next = p + 1 < S.npass ? S.off[p + 2] : end;
    const float4 *rec = S.units + kWorldRec * (mine ? u : beg);
    const float4 r0 = rec[0], r1 = rec[1], r2 = rec[2], r3 = rec[3];
    const unsigned ab = __float_as_uint(r0.x);
    const int A = ab & 0xff, B = (ab >> 8) & 0xff;
    const bool hasB = B != 0xff;
    const float4 anchor = make_float4(r0.w, r1.x, 1.f, 0.f);
    const PinArgs U{r0.y, r0.z, hasB ? r0.w : 0.f, hasB ? r1.x : 0.f, r1.y, r1.z, r1.w, r2.x, r3.y, hasB};
    const AngleArgs V{r2.y, r2.z, r2.w, r3.x, r3.z, r1.z, r2.x, hasB};
    const float yw = r3.w;
    if (mine) {
      float4 a = S.Q[A], b = hasB ? S.Q[B] : anchor;
      float4 d = S.units[kWorldRec * u + 4];
      if (first) d.x = d.y = d.z = 0.f;
      const bool pin = (ab & (kHasPin | kPinBroken)) == kHasPin, angle = (ab & (kHasAngle | kAngleBroken)) == kHasAngle;
      float lx = d.x, ly = d.y, l = d.z;
      const bool op = pin_near<true>(S.tab, U, pin, a, b, lx, ly) && (ab & kPinTame) != 0;
      const bool oa = angle_near<true>(V, yw, kWrapNear, angle, a.z, b.z, l);
      if (__builtin_expect(!(op && oa && (ab & kBounded)), 0)) {
        const UnitOut o = unit_any(U, V, pin, angle, A == B, S.Q[A], hasB ? S.Q[B] : anchor, d.x, d.y, d.z);
        a = o.a; b = o.b; lx = o.lx; ly = o.ly; l = o.l;
      }
      S.units[kWorldRec * u + 4] = make_float4(lx, ly, l, d.w);
      S.Q[A] = a;
      if (hasB && A != B) S.Q[B] = b;
    }
    beg = end;
    end = next;
    L.sync();
  }
}

// Collision pass: solveCollisionsF 'seq', f32solver.mjs:317-344
// (solver.wgsl:373-402) -- per body, its points in order, each correction
// cumulative.
//
// State of the near sets, the same in every lane of the group, in one word
// (a struct returned by the out-of-line rebuild would live in local memory):
// listed bodies with at most kFewPoints points, listed bodies with more, near
// list entries (dense: log2 of the rects per bit of the list), entries per
// mask bit (log2), valid (every body that can meet a rect has a reference),
// full (no usable list: every body against every rect), dense (more near rects
// than a list holds: its words are a bit map of the map's rects, and bit b of a
// mask covers word b), shifted (the references have an origin), tight (the list
// holds while the bodies stay within near_reach(tight) of their references).
struct Near {
  unsigned w = 0;
  __device__ __forceinline__ int few() const { return w & 0xff; }
  __device__ __forceinline__ int many() const { return (w >> 8) & 0xff; }
  __device__ __forceinline__ int n() const { return (w >> 16) & 0x7f; }
  __device__ __forceinline__ int shift() const { return (w >> 23) & 1; }
  __device__ __forceinline__ bool valid() const { return (w >> 24) & 1; }
  __device__ __forceinline__ bool full() const { return (w >> 25) & 1; }
  __device__ __forceinline__ bool dense() const { return (w >> 26) & 1; }
  __device__ __forceinline__ bool shifted() const { return (w >> 27) & 1; }
  __device__ __forceinline__ int tight() const { return (w >> 28) & 3; }
  // the mask of the whole near list
  __device__ __forceinline__ unsigned whole() const { return (1u << ((n() + shift()) >> shift())) - 1u; }
};
constexpr int kMapWords = kCullWords - 1;  // of the bit map; the origin stays behind it
// kFarMove, half of it, kNearMove
__device__ __forceinline__ float near_reach(int tight) {
  return __uint_as_float(__float_as_uint(kFarMove) - ((unsigned)tight << 23));
}
constexpr int kFewPoints = 2;
constexpr float kRefRange = 32000.f;   // of a reference's coordinates about the origin
constexpr float kOriginStep = 16384.f;
// mask of a body that meets no rect (immovable or without points; no other
// mask has rect bits without kNearBit): it needs no reference
constexpr unsigned kExempt = 1u;

// A reference position in one word: x and y rounded to integers + 2^15, less
// the origin, which is ox, oy times kOriginStep: 0 while every body is within
// kRefRange, else kept behind the near list.
__device__ __forceinline__ unsigned near_pack(float x, float y, int ox, int oy) {
  return (unsigned)(__float2int_rn(x) + 32768 - ox * (int)kOriginStep) |
         ((unsigned)(__float2int_rn(y) + 32768 - oy * (int)kOriginStep) << 16);
}
// bias: near_bias of the origin (every sum is an integer below 2^24, so exact)
__device__ __forceinline__ float2 near_unpack(unsigned w, const float2 bias) {
  return make_float2(__uint_as_float(0x4b000000u | (w & 0xffffu)) - bias.x,
                     __uint_as_float(0x4b000000u | (w >> 16)) - bias.y);
}
__device__ __forceinline__ float2 near_bias(int ox, int oy) {
  return make_float2(8421376.f - kOriginStep * (float)ox, 8421376.f - kOriginStep * (float)oy);
}
__device__ __forceinline__ float2 near_bias(const unsigned short *cull, const Near &N) {
  float2 bias = make_float2(8421376.f, 8421376.f);
  if (N.shifted()) bias = near_bias((short)cull[kMaxCulled], (short)cull[kMaxCulled + 1]);
  return bias;
}
__device__ __forceinline__ bool near_holds(const float2 ref, float x, float y, float r) {
  return fabsf(x - ref.x) <= r && fabsf(y - ref.y) <= r;
}
// false only if the rect lies outside the box x0..x1 x y0..y1 (extents of
// either sign; NaN counts as inside)
__device__ __forceinline__ bool in_box(const float4 r, float x0, float x1, float y0, float y1) {
  return !((r.z < x0 && r.x < x0) || (r.x > x1 && r.z > x1) || (r.w < y0 && r.y < y0) || (r.y > y1 && r.w > y1));
}

// New references, near list, masks and body lists from the bodies' predicted
// positions.  near_d = D + kCullPad.  Out of line: it runs once per several
// dozen passes.  World: bodies that meet no rect may be among them (the batched
// engine's templates have none).
template <int G, bool World>
__device__ __noinline__ unsigned near_rebuild(float4 *P, float4 *Q, const float4 *body, unsigned short *cull,
                                          unsigned char *list, int nb, const float4 *__restrict__ rects, int nR,
                                          float near_d, Lanes<G> L) {
  int few_n = 0, many_n = 0, n = 0;
  float lx = kInf, ly = kInf, hx = -kInf, hy = -kInf;
  bool bad = nR > 65535, out = false;
  auto exempt = [&](int j) { return World && (body[j].x == 0.f || (__float_as_int(body[j].w) >> 16) == 0); };
  for (int j = L.lane; j < nb; j += G) {
    if (exempt(j)) continue;
    const float4 q = Q[j];
    const float e = body[j].z + near_d + kFarMove + kCullPad;
    if (!(fabsf(q.x) < 1e6f && fabsf(q.y) < 1e6f && e < 1e6f)) { bad = true; continue; }
    out |= !(fabsf(q.x) < kRefRange && fabsf(q.y) < kRefRange);
    lx = fminf(lx, q.x - e); hx = fmaxf(hx, q.x + e);
    ly = fminf(ly, q.y - e); hy = fmaxf(hy, q.y + e);
  }
  lx = L.min(lx); ly = L.min(ly);
  hx = L.max(hx); hy = L.max(hy);
  bool full = L.ballot(bad) != 0;
  const bool shifted = L.ballot(out) != 0 && !full;
  int ox = 0, oy = 0;
  if (shifted) {
    ox = __float2int_rn((lx + hx) * (0.5f / kOriginStep));
    oy = __float2int_rn((ly + hy) * (0.5f / kOriginStep));
    for (int j = L.lane; j < nb; j += G)
      bad |= !exempt(j) && !near_holds(make_float2(kOriginStep * ox, kOriginStep * oy), Q[j].x, Q[j].y, kRefRange);
    full = L.ballot(bad) != 0;  // farther apart than references reach
    if (L.lane == 0) {
      cull[kMaxCulled] = (unsigned short)ox;
      cull[kMaxCulled + 1] = (unsigned short)oy;
    }
  }
  const float2 bias = near_bias(ox, oy);
  // the near list, within the widest move for which it fits, or the bit map
  int tight = 0;
  bool dense = false;
  for (int base = 0; base < nR && !full && !dense; base += G) {
    const int i = base + L.lane;
    const float d = kFarMove - near_reach(tight);
    const bool keep = i < nR && in_box(__ldg(rects + i), lx + d, hx - d, ly + d, hy - d);
    const unsigned m = L.ballot(keep);
    const int at = n + __popc(m & ((1u << L.lane) - 1u));
    if (keep && at < kMaxCulled) cull[at] = (unsigned short)i;
    n += __popc(m);
    if (n > kMaxCulled) {
      dense = near_reach(tight) == kNearMove;
      tight = dense ? 0 : tight + 1;
      n = 0;
      base = -G;
      L.sync();
    }
  }
  unsigned *map = reinterpret_cast<unsigned *>(cull);
  if (dense) {
    for (n = 0; (nR - 1) >> n >= 32 * kMapWords; n++) {}
    L.sync();
    for (int w = L.lane; w < kMapWords; w += G) {
      unsigned bits = 0u;
      for (int i = w << (5 + n); i < min((w + 1) << (5 + n), nR); i++)
        if (in_box(__ldg(rects + i), lx, hx, ly, hy)) bits |= 1u << ((i >> n) & 31);
      map[w] = bits;
    }
  }
  const int shift = n > 31 && !dense ? 1 : 0;
  L.sync();
  for (int base = 0; base < nb; base += G) {
    const int j = base + L.lane;
    bool few = false, many = false;
    if (j < nb) {
      const float4 bd = body[j];
      const int cnt = __float_as_int(bd.w) >> 16;
      unsigned mask = 0u;
      if (exempt(j)) {
        Q[j].w = __uint_as_float(kExempt);
      } else {
        const float4 q = Q[j];
        if (full) {
          mask = 1u;
        } else {
          const unsigned w = near_pack(q.x, q.y, ox, oy);
          const float2 ref = near_unpack(w, bias);
          const float e = bd.z + near_d, en = e + kNearMove, ef = e + kFarMove;
          bool wide = tight != 0;
          auto look = [&](int i, unsigned bit) {
            const float4 r = __ldg(rects + i);
            wide |= in_box(r, ref.x - ef, ref.x + ef, ref.y - ef, ref.y + ef);
            if (in_box(r, ref.x - en, ref.x + en, ref.y - en, ref.y + en)) mask |= bit;
          };
          if (dense) {
            for (int w = 0; w < kMapWords; w++)
              for (unsigned m = map[w]; m; m &= m - 1u)
                for (int i = (32 * w + __ffs(m) - 1) << n, e = min(i + (1 << n), nR); i < e; i++) look(i, 1u << w);
          } else {
#pragma unroll 4
            for (int i = 0; i < n; i++) look(cull[i], 1u << (i >> shift));
          }
          if (wide) mask |= kNearBit;
          P[j].w = __uint_as_float(w);
        }
        Q[j].w = __uint_as_float(mask);
      }
      few = (mask & ~kNearBit) != 0u && cnt <= kFewPoints;
      many = (mask & ~kNearBit) != 0u && cnt > kFewPoints;
    }
    const unsigned mf = L.ballot(few), mm = L.ballot(many), below = (1u << L.lane) - 1u;
    if (few) list[few_n + __popc(mf & below)] = (unsigned char)j;
    if (many) list[nb - 1 - (many_n + __popc(mm & below))] = (unsigned char)j;
    few_n += __popc(mf);
    many_n += __popc(mm);
  }
  L.sync();
  return full ? (unsigned)few_n | ((unsigned)many_n << 8) | (1u << 25)
              : (unsigned)few_n | ((unsigned)many_n << 8) | ((unsigned)n << 16) | ((unsigned)shift << 23) | (1u << 24) |
                    (dense ? 1u << 26 : 0u) | (shifted ? 1u << 27 : 0u) | ((unsigned)tight << 28);
}

// The fold at (x, y) over a body's near rects, or every rect.  Wide: for groups
// whose state is dense or full; of a dense list's words and of all rects it
// takes those that can matter at this point (near_d = D + kCullPad, which
// covers the box test's rounding below 1e6 px).
template <bool Wide>
__device__ __forceinline__ SdfFold near_fold(const Island &S, const Near &N, const float4 *__restrict__ rects, int nR,
                                             float near_d, bool all, unsigned mask, float x, float y) {
  SdfFold f;
  if constexpr (Wide) {
    const float d = fabsf(x) < 1e6f && fabsf(y) < 1e6f ? near_d : kInf;
    auto take = [&](int i) {
      const float4 r = __ldg(rects + i);
      if (in_box(r, x - d, x + d, y - d, y + d)) f.add(r, x, y);
    };
    if (all) {
#pragma unroll 4
      for (int i = 0; i < nR; i++) take(i);
    } else {
      const int g = N.n();
      for (unsigned words = mask & ~kNearBit; words; words &= words - 1u) {
        const int w = __ffs(words) - 1;
        for (unsigned m = reinterpret_cast<const unsigned *>(S.cull)[w]; m; m &= m - 1u) {
          const int i0 = (32 * w + __ffs(m) - 1) << g, e = min(i0 + (1 << g), nR);
          for (int i = i0; i < e; i++) take(i);
        }
      }
    }
  } else if (all) {
    for (int i = 0; i < nR; i++) f.add(__ldg(rects + i), x, y);
  } else {
    for (unsigned m = mask & ~kNearBit; m; m &= m - 1u) {
      const int b = (__ffs(m) - 1) << N.shift(), e = min(b + 1 + N.shift(), N.n());
      for (int i = b; i < e; i++) f.add(__ldg(rects + S.cull[i]), x, y);
    }
  }
  return f;
}

// The points [from, count) of body j in order, from its pose q
template <bool Wide>
__device__ __forceinline__ void collide_points(Island &S, const Near &N, const float4 *__restrict__ rects, int nR,
                                               float near_d, int j, float4 q, float sa, float ca, int from) {
  const int pr = __float_as_int(S.body[j].w), off = pr & 0xffff, cnt = pr >> 16;
  unsigned mask = __float_as_uint(q.w);
  const bool full = Wide && N.full();
  bool all = full, moved = false;
  for (int k = from; k < cnt; k++) {
    const float4 pt = S.pts[off + k];
    const float wx = fadd(q.x, fsub(fmul(pt.x, ca), fmul(pt.y, sa)));
    const float wy = fadd(q.y, fadd(fmul(pt.x, sa), fmul(pt.y, ca)));
    float dx, dy;
    if (near_fold<Wide>(S, N, rects, nR, near_d, all, mask, wx, wy).push(pt.z, &dx, &dy)) {
      q.x = fadd(q.x, dx);
      q.y = fadd(q.y, dy);
      moved = true;
      // pushed away from its reference its near set may miss a rect, farther
      // away the near list too (a body that its joints hold in a wall is pushed
      // by more than kNearMove in every pass)
      if (!full) {
        const float2 ref = near_unpack(__float_as_uint(S.P[j].w), near_bias(S.cull, N));
        mask = near_holds(ref, q.x, q.y, kNearMove) ? __float_as_uint(q.w) : Wide ? ~kNearBit : N.whole();
        all = !near_holds(ref, q.x, q.y, near_reach(N.tight()));
      }
    }
  }
  if (moved) S.Q[j] = q;
}

// The listed bodies of a collision pass.  Those with one or two points take a
// lane each; the points of a body with more (the mantle's eight) are evaluated
// side by side, and one lane repeats them in order from the first that
// corrects -- until then none has moved the body.
template <int G, bool Wide>
__device__ __forceinline__ void collide_listed(Island &S, const Near &N, const float4 *__restrict__ rects, int nR,
                                               float near_d, const Lanes<G> &L) {
  for (int t = L.lane; t < N.few(); t += G) {
    const int j = S.list[t];
    const float4 q = S.Q[j];
    float sa, ca;
    sincos_r(S.tab, q.z, &sa, &ca);
    collide_points<Wide>(S, N, rects, nR, near_d, j, q, sa, ca, 0);
  }
  for (int t = 0; t < N.many(); t++) {
    const int j = S.list[S.nb - 1 - t];
    const float4 q = S.Q[j];
    const int pr = __float_as_int(S.body[j].w), off = pr & 0xffff, cnt = pr >> 16;
    float sa, ca;
    sincos_r(S.tab, q.z, &sa, &ca);
    int first = -1;
    for (int base = 0; base < cnt && first < 0; base += G) {
      bool hit = false;
      if (base + L.lane < cnt) {
        const float4 pt = S.pts[off + base + L.lane];
        const float wx = fadd(q.x, fsub(fmul(pt.x, ca), fmul(pt.y, sa)));
        const float wy = fadd(q.y, fadd(fmul(pt.x, sa), fmul(pt.y, ca)));
        float dx, dy;
        hit = near_fold<Wide>(S, N, rects, nR, near_d, Wide && N.full(), __float_as_uint(q.w), wx, wy).push(pt.z, &dx, &dy);
      }
      const unsigned m = L.ballot(hit);
      if (m) first = base + __ffs(m) - 1;
    }
    if (first >= 0 && L.lane == 0) collide_points<Wide>(S, N, rects, nR, near_d, j, q, sa, ca, first);
  }
}
// (the members it needs one by one: a struct of the size of Island would pass
// through local memory)
template <int G, bool Wide>
__device__ __noinline__ void collide_listed_call(const float4 *P, float4 *Q, const float4 *body, const float4 *pts,
                                                 const float2 *tab, unsigned short *cull, unsigned char *list, int nb,
                                                 unsigned near, const float4 *__restrict__ rects, int nR, float near_d,
                                                 int warp_lane) {
  Island S{};
  S.P = const_cast<float4 *>(P); S.Q = Q; S.body = body; S.pts = pts; S.tab = tab;
  S.cull = cull; S.list = list; S.nb = nb;
  Near N;
  N.w = near;
  collide_listed<G, Wide>(S, N, rects, nR, near_d, Lanes<G>(warp_lane));
}

// One collision pass of the island.  OutOfLine: the listed bodies (most passes
// have none) as a call -- for the kernel with the net, whose step is larger
// than the instruction caches: 8,000 creatures under the net take 9 % longer
// with it in line, the others 3 % less.  The groups without a list that masks
// can cover take a call of their own in every kernel.
template <int G, bool World, bool OutOfLine>
__device__ __forceinline__ void collide_island(Island &S, Near &N, const float4 *__restrict__ rects, int nR,
                                               float near_d, const Lanes<G> &L) {
  bool stale = !N.valid();
  if (!stale) {
    bool moved = false;
    const float2 bias = near_bias(S.cull, N);
#pragma unroll 1
    for (int j = L.lane; j < S.nb; j += G) {
      const float4 q = S.Q[j];
      const unsigned mask = __float_as_uint(q.w);
      if (World && mask == kExempt) continue;
      moved |= !near_holds(near_unpack(__float_as_uint(S.P[j].w), bias), q.x, q.y,
                           (mask & kNearBit) ? kNearMove : kFarMove);
    }
    stale = L.ballot(moved) != 0;
  }
  if (stale) N.w = near_rebuild<G, World>(S.P, S.Q, S.body, S.cull, S.list, S.nb, rects, nR, near_d, L);
  auto call = [&](auto wide) {
    collide_listed_call<G, decltype(wide)::value>(S.P, S.Q, S.body, S.pts, S.tab, S.cull, S.list, S.nb, N.w, rects, nR,
                                                  near_d, L.base + L.lane);
  };
  if (__builtin_expect(N.full() || N.dense(), 0)) call(std::true_type{});
  else if (!OutOfLine) collide_listed<G, false>(S, N, rects, nR, near_d, L);
  else if (N.w & 0xffffu) call(std::false_type{});
  L.sync();
}

// finalizeF, f32solver.mjs:376-399 (solver.wgsl:405-430)
template <bool World>
__device__ __forceinline__ void finalize_body(const SolverConsts &K, Island &S, int i) {
  if (World) {
    const float4 bd = S.body[i];
    if (bd.x == 0.f && bd.y == 0.f) {
      S.V[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      return;
    }
  }
  float4 q = S.Q[i];
  const float4 p = S.P[i];
  float vx = fmul(fsub(q.x, p.x), K.invH);
  float vy = fmul(fsub(q.y, p.y), K.invH);
  float av = fmul(angle_delta(q.z, p.z), K.invH);
  clamp_speed(K, vx, vy);
  if (av > K.maxAngSpeed) av = K.maxAngSpeed;
  else if (av < -K.maxAngSpeed) av = -K.maxAngSpeed;
  if (q.z > 50.f || q.z < -50.f) {
    q.z = wrap_far(q.z);
    if (World) S.Q[i].z = q.z;
  }
  S.P[i] = make_float4(q.x, q.y, q.z, p.w);
  S.V[i] = make_float4(vx, vy, av, World ? 0.f : q.w);
}

// gripBreakF, f32solver.mjs:402-416 (solver.wgsl:433-442): true if the
// constraint with this multiplier and break force breaks
__device__ __forceinline__ bool grip_breaks(const SolverConsts &K, float lx, float ly, float brk) {
  return fmul(length2(lx, ly), K.invH) > brk;
}

// One env step of one island by a group of G lanes (xpbd.js:487-490 with the
// substep of f32solver.mjs:419-428): substeps x (reset lambda, integrate,
// iterations x (solve passes, collisions), finalize), then grip break.
// U: unroll factor of the substep loop (1: a loop; 2: its body twice per
// trip, remainder handled) -- the same operations in the same order, so the
// results do not depend on it; the batched engine's autotuner picks it.  The
// loops inside are not unrolled: an env step's code has to stay in the
// instruction caches (the pass loop unrolled twice: 16,384 creatures take
// 42 % longer; the body loops unrolled: 8,000 under the policy 15 %).
template <bool World, int G, int U = 1, bool OutOfLine = false>
__device__ __forceinline__ void island_step(const SolverConsts &K, Island &S,
                                            const float4 *__restrict__ rects, int nR, float near_d,
                                            const Lanes<G> &L, Near &N) {
#pragma unroll U
  for (int s = 0; s < K.substeps; s++) {
#pragma unroll 1
    for (int i = L.lane; i < S.nb; i += G) integrate_body<World>(K, S, i);
    L.sync();
    for (int it = 0; it < K.iterations; it++) {
      if constexpr (World) solve_world<G>(S, it == 0, L);
      else solve_engine<G>(K, S, it == 0, L);
      collide_island<G, World, OutOfLine>(S, N, rects, nR, near_d, L);
    }
#pragma unroll 1
    for (int i = L.lane; i < S.nb; i += G) finalize_body<World>(K, S, i);
    L.sync();
  }
  if constexpr (World) {
    for (int u = L.lane; u < S.nu; u += G) {
      float4 *rec = S.units + kWorldRec * u;
      const unsigned ab = __float_as_uint(rec[0].x);
      if ((ab & (kHasPin | kPinIsGrip | kPinBroken)) != (kHasPin | kPinIsGrip)) continue;
      const float4 d = rec[4];
      if (grip_breaks(K, d.x, d.y, d.w)) {
        rec[0].x = __uint_as_float(ab | kPinBroken);
        rec[4] = make_float4(0.f, 0.f, d.z, d.w);
      }
    }
  } else if (L.lane < S.arms) {
    const float2 g = S.mot[S.grip0 + L.lane];
    float4 &an = S.Q[S.nb + L.lane];
    if (an.w == 0.f && grip_breaks(K, g.x, g.y, S.brk[L.lane])) {
      an.w = 1.f;
      S.mot[S.grip0 + L.lane] = make_float2(0.f, 0.f);
    }
  }
  L.sync();
}

}  // namespace kr
