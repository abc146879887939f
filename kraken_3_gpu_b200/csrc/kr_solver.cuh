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

__device__ __forceinline__ void sincos_r(float a, float *s, float *c) {
  const double x = static_cast<double>(a);
  if (!(fabs(x) <= 1048576.0)) {
    const float2 f = sincos_far(x);
    *s = f.x;
    *c = f.y;
    return;
  }
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
  *s = static_cast<float>(t.x + fma(t.x, cm1, t.y * sr));
  *c = static_cast<float>(t.y + fma(t.y, cm1, -(t.x * sr)));
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

// angleDeltaF, f32solver.mjs:36-43 (solver.wgsl:103-108)
__device__ __forceinline__ float angle_delta(float a, float b) {
  float x = fsub(a, b);
  float q = trunc_quot_tau(x);
  float d = fsub(x, fmul(kTau, q));
  if (d > kPi) return fsub(d, kTau);
  if (d < -kPi) return fadd(d, kTau);
  return d;
}

// wrapAngleF, f32solver.mjs:45-51 (solver.wgsl:96-101)
__device__ __forceinline__ float wrap_angle(float a) {
  float q = trunc_quot_tau(a);
  float d = fsub(a, fmul(kTau, q));
  if (d > kPi) return fsub(d, kTau);
  if (d < -kPi) return fadd(d, kTau);
  return d;
}

// lengthF, f32solver.mjs:54-56 (WGSL length(vec2f))
__device__ __forceinline__ float length2(float x, float y) {
  return fsqrt(fadd(fmul(x, x), fmul(y, y)));
}

// Rect as stored on the device: x, y, x + w, y + h (all f32, the sums
// rounded once as solver.wgsl:120-121 computes r.x + r.w).
// sdfF, f32solver.mjs:139-166 (solver.wgsl:114-147), over the rects
// idx[0..n) in ascending order (or 0..n when idx is null).  The division of
// the outward normal is deferred to the final winner: bnx/bny are overwritten
// by every later winner, so only the last winner's dx/best, dy/best survive.
__device__ __forceinline__ bool sdf(const float4 *__restrict__ rects, const short *idx, int n,
                                    float x, float y, float *od, float *onx, float *ony) {
  float best = kSdfInf, thr = __int_as_float(0x7f800000);  // f32 1e30*1e30 = +inf
  float wdx = 0.f, wdy = 0.f, inx = 0.f, iny = 0.f;
  bool inside = false;
  for (int q = 0; q < n; q++) {
    const float4 r = __ldg(rects + (idx ? idx[q] : q));
    float cx = x < r.x ? r.x : (x > r.z ? r.z : x);
    float cy = y < r.y ? r.y : (y > r.w ? r.w : y);
    float dx = fsub(x, cx), dy = fsub(y, cy);
    float d2 = fadd(fmul(dx, dx), fmul(dy, dy));
    if (d2 > kEpsSdf) {
      if (d2 < thr) {
        best = fsqrt(d2);
        thr = fmul(best, best);
        wdx = dx; wdy = dy;
        inside = false;
      }
    } else {
      float dl = fsub(x, r.x), dr = fsub(r.z, x), dt = fsub(y, r.y), db = fsub(r.w, y);
      float m = dl, nx = -1.f, ny = 0.f;
      if (dr < m) { m = dr; nx = 1.f; ny = 0.f; }
      if (dt < m) { m = dt; nx = 0.f; ny = -1.f; }
      if (db < m) { m = db; nx = 0.f; ny = 1.f; }
      float d = -m;
      if (d < best) {
        best = d;
        thr = fmul(best, best);
        inx = nx; iny = ny;
        inside = true;
      }
    }
  }
  if (best > kSdfValid) return false;
  *od = best;
  if (inside) { *onx = inx; *ony = iny; }
  else { *onx = fdiv(wdx, best); *ony = fdiv(wdy, best); }
  return true;
}

// Exact rect culling for one collision pass of one creature.
//
// Let D = max(largest collision radius, largest half-thickness min(w,h)/2 of
// a rect) + 2.  Drop every rect farther than D from every point the pass
// evaluates.  The sequential SDF fold then returns the same winner, or in
// both cases a winner farther than D - 1 (> radius + 1: no correction):
//  * a state's threshold f(best^2) never falls below the squared distance
//    of any rect processed so far, except that an inside winner sets it to
//    at most half-thickness^2 < (D - 1)^2; a dropped rect (d^2 > D^2) can
//    therefore only beat states with threshold >= (D - 1)^2 ("far" states);
//  * by monotone rounding, a rect that fails to beat a far state is itself
//    far, and an inside rect beats every far state; so the folds with and
//    without the dropped rects hold equal states or two far states.
// The pass keeps a point's evaluation on the culled list only while the
// point lies in the box the list was built for (kCullSlack inside the cull
// margin); otherwise it uses the full list.
constexpr int kMaxCulled = 64;
constexpr float kCullSlack = 6.f;

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
// through shared memory: per-constraint levels made a 6 x 7 body 12 of them,
// as units it is 6 (12 creatures: 90 -> 64 us an env step; 16,384 mixed
// creatures to their horizons: 391 -> 308 ms).
//
// Bodies are float4 records (one 16-byte load or store instead of three
// 4-byte ones).
struct Island {
  float4 *P;           // committed x, y, angle
  float4 *Q;           // predicted x, y, angle
  float4 *V;           // velocity vx, vy, av (batched engine: the same records as Q, see below)
  const float4 *body;  // inverse mass, inverse inertia, reach, point offset | count << 16
  const float4 *pts;   // collision points: x, y, radius, body; grouped per body in groupCollPoints order
  float *bs, *bc;      // sin / cos of the predicted angle during a collision pass
  float *pdx, *pdy;    // speculative correction of each point
  int *pflag;          // 1 if the speculative evaluation corrects
  short *cull;         // culled rect list (kMaxCulled)
  int nb, np;
  // drop-in world: one dynamic record of 4 float4 per unit, pass offsets
  float4 *units;
  int nu, npass;
  const int *off;      // npass + 1 unit offsets
  float4 *force;       // fx, fy, torque
  // batched engine: the template's static records (3 float4 per lane and
  // pass), per motor {target, lambda}, per arm {lambda x, y, break force}
  const float4 *recs;
  float2 *mot;
  float4 *grip;
  float comp_m;        // motor compliance of the creature
  int arms;
};

// ab word of a unit: body A, body B (or, in the batched engine, the record
// of an arm's anchor; 0xff in the drop-in: the world), and flags.
constexpr unsigned kUnitIdle = 0xffffffffu;
// drop-in world flags
constexpr unsigned kHasPin = 1u << 16, kPinBroken = 1u << 17, kHasAngle = 1u << 18, kAngleBroken = 1u << 19,
                   kPinIsGrip = 1u << 20;
// batched engine: bits 16..23 the motor of a joint, or 0xff for a grip
constexpr unsigned kNoMotor = 0xffu;

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
  if (World && im == 0.f && ii == 0.f) {
    S.Q[i] = p;
    S.V[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  float4 v = S.V[i];
  const float4 f = World ? S.force[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  float vx = fmul(fadd(v.x, fmul(fmul(K.h, im), f.x)), K.linDamp);
  float vy = fmul(fadd(v.y, fmul(fmul(K.h, im), f.y)), K.linDamp);
  float av = fmul(fadd(v.z, fmul(fmul(K.h, ii), f.z)), K.angDamp);
  float sp = length2(vx, vy);
  if (sp > K.maxSpeed) {
    float k = fdiv(K.maxSpeed, sp);
    vx = fmul(vx, k); vy = fmul(vy, k);
  }
  if (av > K.maxAngSpeed) av = K.maxAngSpeed;
  else if (av < -K.maxAngSpeed) av = -K.maxAngSpeed;
  if (!(vx == vx) || !(vy == vy)) { vx = 0.f; vy = 0.f; }
  if (!(av == av)) av = 0.f;
  if (World) S.V[i] = make_float4(vx, vy, av, v.w);
  S.Q[i] = make_float4(fadd(p.x, fmul(K.h, vx)), fadd(p.y, fmul(K.h, vy)), fadd(p.z, fmul(K.h, av)), v.w);
  if (World) S.force[i] = make_float4(0.f, 0.f, 0.f, f.w);
}

// solvePinF, f32solver.mjs:203-256 (solver.wgsl:225-290) on two body records
// in registers; grips are pins against the world.  Without a body B: b holds
// the anchor as its position with angle 0, lb and the masses of B are 0 (the
// same values as the reference's branch).  lx, ly: the multiplier, updated.
__device__ __forceinline__ void pin_math(float lax, float lay, float lbx, float lby, float wA, float wIA, float wB,
                                         float wIB, float alphaTilde, bool hasB, float4 &a, float4 &b, float &lx,
                                         float &ly) {
  float sa, ca, sb, cb;
  sincos_r(a.z, &sa, &ca);
  sincos_r(b.z, &sb, &cb);
  const float rax = fsub(fmul(lax, ca), fmul(lay, sa)), ray = fadd(fmul(lax, sa), fmul(lay, ca));
  const float rbx = fsub(fmul(lbx, cb), fmul(lby, sb)), rby = fadd(fmul(lbx, sb), fmul(lby, cb));
  const float Cx = fsub(fadd(a.x, rax), fadd(b.x, rbx)), Cy = fsub(fadd(a.y, ray), fadd(b.y, rby));
  if (!(Cx == Cx) || !(Cy == Cy)) return;
  if (fadd(fmul(Cx, Cx), fmul(Cy, Cy)) < fmul(kSlackPos, kSlackPos)) return;
  const float pax = -ray, pay = rax, pbx = -rby, pby = rbx;
  const float wSum = fadd(wA, wB);
  const float k00 = fadd(fadd(wSum, fmul(fmul(wIA, pax), pax)), fmul(fmul(wIB, pbx), pbx));
  const float k01 = fadd(fmul(fmul(wIA, pax), pay), fmul(fmul(wIB, pbx), pby));
  const float k11 = fadd(fadd(wSum, fmul(fmul(wIA, pay), pay)), fmul(fmul(wIB, pby), pby));
  const float det = fsub(fmul(k00, k11), fmul(k01, k01));
  if (fabsf(det) < kEpsDet) return;
  const float bx = fadd(Cx, fmul(alphaTilde, lx)), by = fadd(Cy, fmul(alphaTilde, ly));
  const float i00 = fdiv(k11, det), i11 = fdiv(k00, det), i01 = -fdiv(k01, det);
  const float dlx = -fadd(fmul(i00, bx), fmul(i01, by)), dly = -fadd(fmul(i01, bx), fmul(i11, by));
  if (!(dlx == dlx) || !(dly == dly)) return;
  lx = fadd(lx, dlx);
  ly = fadd(ly, dly);
  a.x = fadd(a.x, fmul(wA, dlx));
  a.y = fadd(a.y, fmul(wA, dly));
  a.z = fadd(a.z, fmul(wIA, fadd(fmul(pax, dlx), fmul(pay, dly))));
  if (hasB) {
    b.x = fsub(b.x, fmul(wB, dlx));
    b.y = fsub(b.y, fmul(wB, dly));
    b.z = fsub(b.z, fmul(wIB, fadd(fmul(pbx, dlx), fmul(pby, dly))));
  }
}

// solveAngleF, f32solver.mjs:258-301 (solver.wgsl:292-350): muscle
// (compliant) part, then the one-sided joint limit.  az, bz: the angles; l:
// the multiplier, updated.
__device__ __forceinline__ void angle_math(float rest, float mn, float mx, float tgt, float alphaTilde, float wA,
                                           float wB, bool hasB, float &az, float &bz, float &l) {
  const float rel = hasB ? angle_delta(bz, az) : az;
  const float wSum = fadd(wA, wB);
  if (wSum <= 0.f) return;
  const float dev = angle_delta(rel, rest);
  const float C = angle_delta(dev, tgt);
  if (!(C == C)) return;
  if (fabsf(C) >= kSlackAng) {
    const float dl = -fdiv(fadd(C, fmul(alphaTilde, l)), fadd(wSum, alphaTilde));
    if (!(dl == dl)) return;
    l = fadd(l, dl);
    if (hasB) {
      bz = fadd(bz, fmul(wB, dl));
      az = fsub(az, fmul(wA, dl));
    } else {
      az = fadd(az, fmul(wA, dl));
    }
  }
  const float dev2 = angle_delta(hasB ? angle_delta(bz, az) : az, rest);
  float over = 0.f;
  if (dev2 > mx) over = fsub(dev2, mx);
  else if (dev2 < mn) over = fsub(dev2, mn);
  if (fabsf(over) >= kSlackAng) {
    const float dl2 = -fdiv(over, wSum);
    if (hasB) {
      bz = fadd(bz, fmul(wB, dl2));
      az = fsub(az, fmul(wA, dl2));
    } else {
      az = fadd(az, fmul(wA, dl2));
    }
  }
}

// One sweep of the solve list, batched engine.  first: the first sweep of a
// substep, where every multiplier starts from 0.  A pin's multiplier only
// enters its own equation times its compliance, which is 0 for the
// template's pins and grips, so only the grips' (the break test) and the
// motors' are kept.
template <int G>
__device__ __forceinline__ void solve_engine(const SolverConsts &K, Island &S, bool first, const Lanes<G> &L) {
  const float alpha_m = fmul(S.comp_m, K.invH2);
  const float4 *rec = S.recs + 3 * L.lane;
  for (int p = 0; p < S.npass; p++, rec += 3 * G) {
    const float4 r0 = rec[0];
    const unsigned ab = __float_as_uint(r0.x);
    if (ab != kUnitIdle) {
      const int A = ab & 0xff, B = (ab >> 8) & 0xff, m = (ab >> 16) & 0xff;
      float4 a = S.Q[A], b = S.Q[B];
      const float4 r1 = rec[1], r2 = rec[2];
      if (m != (int)kNoMotor) {
        float lx = 0.f, ly = 0.f;
        pin_math(r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, 0.f, true, a, b, lx, ly);
        const float2 mo = S.mot[m];
        float l = first ? 0.f : mo.y;
        angle_math(r2.y, r2.z, r2.w, mo.x, alpha_m, r1.z, r2.x, true, a.z, b.z, l);
        S.mot[m].y = l;
        S.Q[A] = a;
        S.Q[B] = b;
      } else {
        float4 g = S.grip[B - S.nb];
        if (first) g.x = g.y = 0.f;
        if (b.w == 0.f) {  // holding
          pin_math(r0.y, r0.z, 0.f, 0.f, r1.y, r1.z, 0.f, 0.f, 0.f, false, a, b, g.x, g.y);
          S.Q[A] = a;
        }
        S.grip[B - S.nb] = g;
      }
    }
    L.sync();
  }
}

// A drop-in unit whose two bodies are one: every update sees the one before
// it (a and b are the same record).  Out of line: no creature has one.
static __device__ __noinline__ void solve_self(const SolverConsts &K, unsigned ab, float4 wa, float4 &a, float4 *rec) {
  const float4 r0 = rec[0], r2 = rec[2];
  float4 r1 = rec[1], r3 = rec[3];
  if ((ab & (kHasPin | kPinBroken)) == kHasPin)
    pin_math(r0.y, r0.z, r0.w, r1.x, wa.x, wa.y, wa.x, wa.y, fmul(r1.y, K.invH2), true, a, a, r1.z, r1.w);
  if ((ab & (kHasAngle | kAngleBroken)) == kHasAngle)
    angle_math(r2.x, r2.y, r2.z, r2.w, fmul(r3.x, K.invH2), wa.y, wa.y, true, a.z, a.z, r3.y);
  rec[1] = r1;
  rec[3] = r3;
}

// One sweep of the solve list, drop-in world: unit records
// {ab, lax, lay, lbx} {lby, pin compliance, lambda x, y}
// {rest, min, max, target} {angle compliance, lambda, break force, -}.
template <int G>
__device__ __forceinline__ void solve_world(const SolverConsts &K, Island &S, bool first, const Lanes<G> &L) {
  for (int p = 0; p < S.npass; p++) {
    for (int u = S.off[p] + L.lane; u < S.off[p + 1]; u += G) {  // at most one: passes hold up to 32 units
      float4 *rec = S.units + 4 * u;
      const float4 r0 = rec[0];
      const unsigned ab = __float_as_uint(r0.x);
      const int A = ab & 0xff, B = (ab >> 8) & 0xff;
      const bool hasB = B != 0xff;
      float4 a = S.Q[A], b = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 wa = S.body[A];
      if (A == B) {
        if (first) { rec[1].z = rec[1].w = 0.f; rec[3].y = 0.f; }
        solve_self(K, ab, wa, a, rec);
        S.Q[A] = a;
        continue;
      }
      float4 wb = b;
      if (hasB) { b = S.Q[B]; wb = S.body[B]; }
      if (ab & kHasPin) {
        float4 r1 = rec[1];
        if (first) r1.z = r1.w = 0.f;
        if (!(ab & kPinBroken)) {
          float4 anchor = make_float4(r0.w, r1.x, 0.f, 0.f);
          pin_math(r0.y, r0.z, hasB ? r0.w : 0.f, hasB ? r1.x : 0.f, wa.x, wa.y, wb.x, wb.y, fmul(r1.y, K.invH2),
                   hasB, a, hasB ? b : anchor, r1.z, r1.w);
        }
        rec[1] = r1;
      }
      if (ab & kHasAngle) {
        float4 r3 = rec[3];
        if (first) r3.y = 0.f;
        if (!(ab & kAngleBroken)) {
          const float4 r2 = rec[2];
          angle_math(r2.x, r2.y, r2.z, r2.w, fmul(r3.x, K.invH2), wa.y, wb.y, hasB, a.z, b.z, r3.y);
        }
        rec[3] = r3;
      }
      S.Q[A] = a;
      if (hasB) S.Q[B] = b;
    }
    L.sync();
  }
}

// One collision pass of the island: solveCollisionsF 'seq',
// f32solver.mjs:317-344 (solver.wgsl:373-402) -- per body, its points in
// order, each correction cumulative.  Evaluated as
//   1. sin/cos of angP per body (angP does not change in the pass),
//   2. every point at its body's pose at the start of the pass, plus the
//      bounding box of those positions, and the culled rect list,
//   3. per body, the points in order: a point's evaluation from step 2 is
//      the sequential one as long as no earlier point of that body moved
//      it; after the first correction the remaining points of that body are
//      re-evaluated at the moved pose, exactly as the sequential loop does.
// The collision pass with the culled list taken from the box of the bodies'
// centres widened by reach (>= every collision point's distance from its
// body's centre, plus 1 px for rounding): the rects within cull_d of that
// box, in ascending order.  The box holds every point the pass evaluates, so
// the list keeps every rect within cull_d of them and the fold over it is
// exact by the argument above kMaxCulled.  A body with no listed rect within
// reach + cull_d of its centre has no point that any rect can correct: its
// sin/cos, point positions and SDF evaluations are skipped (bc[j] = 2, an
// impossible cosine, marks it) -- its points are unflagged, as the full
// evaluation would leave them.  With an empty list the pass changes nothing
// and ends at once.  Returns false, having changed nothing, when the box is
// not finite or reaches 1e6 px (where 1 px no longer covers f32 rounding) or
// the list would exceed kMaxCulled; the caller then runs the pass below.
template <int G>
__device__ __forceinline__ bool collide_bodies(Island &S, const float4 *__restrict__ rects, int nR, float cull_d,
                                               const Lanes<G> &L, float reach) {
  float lx = __int_as_float(0x7f800000), ly = lx, hx = -lx, hy = -lx;
  for (int j = L.lane; j < S.nb; j += G) {
    lx = fminf(lx, S.Q[j].x); hx = fmaxf(hx, S.Q[j].x);
    ly = fminf(ly, S.Q[j].y); hy = fmaxf(hy, S.Q[j].y);
  }
  lx = L.min(lx); ly = L.min(ly);
  hx = L.max(hx); hy = L.max(hy);
  const float e = reach + cull_d;
  const float x0 = lx - e, x1 = hx + e, y0 = ly - e, y1 = hy + e;
  if (!(x0 <= x1 && y0 <= y1 && fmaxf(fmaxf(fabsf(x0), fabsf(x1)), fmaxf(fabsf(y0), fabsf(y1))) < 1e6f))
    return false;
  int ncull = 0;
  for (int base = 0; base < nR; base += G) {
    const int i = base + L.lane;
    bool keep = false;
    if (i < nR) {
      const float4 r = __ldg(rects + i);
      keep = !(r.z < x0 || r.x > x1 || r.w < y0 || r.y > y1);
    }
    const unsigned m = L.ballot(keep);
    const int at = ncull + __popc(m & ((1u << L.lane) - 1u));
    if (keep && at < kMaxCulled) S.cull[at] = static_cast<short>(i);
    ncull += __popc(m);
    if (ncull > kMaxCulled) {
      L.sync();
      return false;
    }
  }
  if (ncull == 0) return true;
  L.sync();
  for (int j = L.lane; j < S.nb; j += G) {
    const float cx = S.Q[j].x, cy = S.Q[j].y;
    bool near = false;
    for (int q = 0; q < ncull && !near; q++) {
      const float4 r = __ldg(rects + S.cull[q]);
      near = !(r.z < cx - e || r.x > cx + e || r.w < cy - e || r.y > cy + e);
    }
    if (near) {
      float sn, cs;
      sincos_r(S.Q[j].z, &sn, &cs);
      S.bs[j] = sn;
      S.bc[j] = cs;
    } else {
      S.bc[j] = 2.f;
    }
  }
  L.sync();
  for (int p = L.lane; p < S.np; p += G) {
    const float4 pt = S.pts[p];
    const int j = __float_as_int(pt.w);
    const float ca = S.bc[j];
    int flag = 0;
    float cx = 0.f, cy = 0.f;
    if (ca != 2.f && S.body[j].x != 0.f) {
      const float sa = S.bs[j], ox = pt.x, oy = pt.y;
      const float wx = fadd(S.Q[j].x, fsub(fmul(ox, ca), fmul(oy, sa)));
      const float wy = fadd(S.Q[j].y, fadd(fmul(ox, sa), fmul(oy, ca)));
      float d, nx, ny;
      if (sdf(rects, S.cull, ncull, wx, wy, &d, &nx, &ny)) {
        const float pen = fsub(pt.z, d);
        if (pen > kSlackPos) {
          flag = 1;
          cx = fmul(nx, pen);
          cy = fmul(ny, pen);
        }
      }
    }
    S.pflag[p] = flag;
    S.pdx[p] = cx;
    S.pdy[p] = cy;
  }
  L.sync();
  const float sx0 = lx - reach - kCullSlack, sx1 = hx + reach + kCullSlack;
  const float sy0 = ly - reach - kCullSlack, sy1 = hy + reach + kCullSlack;
  for (int j = L.lane; j < S.nb; j += G) {
    if (S.body[j].x == 0.f || S.bc[j] == 2.f) continue;
    const int pr = __float_as_int(S.body[j].w), o = pr & 0xffff, cnt = pr >> 16;
    float px = S.Q[j].x, py = S.Q[j].y;
    const float ca = S.bc[j], sa = S.bs[j];
    bool moved = false;
    for (int q = 0; q < cnt; q++) {
      const int p = o + q;
      if (!moved) {
        if (S.pflag[p]) {
          px = fadd(px, S.pdx[p]);
          py = fadd(py, S.pdy[p]);
          moved = true;
        }
        continue;
      }
      const float4 pt = S.pts[p];
      const float ox = pt.x, oy = pt.y;
      const float wx = fadd(px, fsub(fmul(ox, ca), fmul(oy, sa)));
      const float wy = fadd(py, fadd(fmul(ox, sa), fmul(oy, ca)));
      const bool in_box = wx >= sx0 && wx <= sx1 && wy >= sy0 && wy <= sy1;
      float d, nx, ny;
      if (!sdf(rects, in_box ? S.cull : nullptr, in_box ? ncull : nR, wx, wy, &d, &nx, &ny)) continue;
      const float pen = fsub(pt.z, d);
      if (pen <= kSlackPos) continue;
      px = fadd(px, fmul(nx, pen));
      py = fadd(py, fmul(ny, pen));
    }
    S.Q[j].x = px;
    S.Q[j].y = py;
  }
  L.sync();
  return true;
}

// cull_d = D + kCullSlack with D as in the comment above kMaxCulled.  reach
// >= 0 (the batched engine's templates): collide_bodies; reach < 0 (the
// drop-in world, arbitrary collision points): the culled list from the box
// of the evaluated points.
template <int G>
__device__ __forceinline__ void collide_island(Island &S, const float4 *__restrict__ rects, int nR,
                                               float cull_d, const Lanes<G> &L, float reach) {
  if (reach >= 0.f && collide_bodies<G>(S, rects, nR, cull_d, L, reach)) return;
  for (int j = L.lane; j < S.nb; j += G) {
    float s, c;
    sincos_r(S.Q[j].z, &s, &c);
    S.bs[j] = s;
    S.bc[j] = c;
  }
  L.sync();
  float mnx = __int_as_float(0x7f800000), mny = mnx, mxx = -mnx, mxy = -mnx;
  for (int p = L.lane; p < S.np; p += G) {
    const float4 pt = S.pts[p];
    const int j = __float_as_int(pt.w);
    const float ca = S.bc[j], sa = S.bs[j], lx = pt.x, ly = pt.y;
    const float wx = fadd(S.Q[j].x, fsub(fmul(lx, ca), fmul(ly, sa)));
    const float wy = fadd(S.Q[j].y, fadd(fmul(lx, sa), fmul(ly, ca)));
    S.pdx[p] = wx;  // position for now, correction below
    S.pdy[p] = wy;
    mnx = fminf(mnx, wx); mxx = fmaxf(mxx, wx);
    mny = fminf(mny, wy); mxy = fmaxf(mxy, wy);
  }
  mnx = L.min(mnx); mny = L.min(mny);
  mxx = L.max(mxx); mxy = L.max(mxy);
  // culled list, ascending rect order
  const float bx0 = mnx - cull_d, bx1 = mxx + cull_d, by0 = mny - cull_d, by1 = mxy + cull_d;
  int ncull = 0;
  bool full = !(bx0 <= bx1 && by0 <= by1);  // no finite point: use the full list
  for (int base = 0; base < nR && !full; base += G) {
    const int i = base + L.lane;
    bool keep = false;
    if (i < nR) {
      const float4 r = __ldg(rects + i);
      keep = !(r.z < bx0 || r.x > bx1 || r.w < by0 || r.y > by1);
    }
    const unsigned m = L.ballot(keep);
    const int at = ncull + __popc(m & ((1u << L.lane) - 1u));
    if (keep && at < kMaxCulled) S.cull[at] = static_cast<short>(i);
    ncull += __popc(m);
    if (ncull > kMaxCulled) full = true;
  }
  L.sync();
  const short *list = full ? nullptr : S.cull;
  const int nlist = full ? nR : ncull;
  const float sx0 = mnx - kCullSlack, sx1 = mxx + kCullSlack;
  const float sy0 = mny - kCullSlack, sy1 = mxy + kCullSlack;
  for (int p = L.lane; p < S.np; p += G) {
    const float4 pt = S.pts[p];
    const int j = __float_as_int(pt.w);
    int flag = 0;
    float cx = 0.f, cy = 0.f;
    if (S.body[j].x != 0.f) {
      float d, nx, ny;
      if (sdf(rects, list, nlist, S.pdx[p], S.pdy[p], &d, &nx, &ny)) {
        const float pen = fsub(pt.z, d);
        if (pen > kSlackPos) {
          flag = 1;
          cx = fmul(nx, pen);
          cy = fmul(ny, pen);
        }
      }
    }
    S.pflag[p] = flag;
    S.pdx[p] = cx;
    S.pdy[p] = cy;
  }
  L.sync();
  for (int j = L.lane; j < S.nb; j += G) {
    if (S.body[j].x == 0.f) continue;
    const int pr = __float_as_int(S.body[j].w), o = pr & 0xffff, cnt = pr >> 16;
    float px = S.Q[j].x, py = S.Q[j].y;
    const float ca = S.bc[j], sa = S.bs[j];
    bool moved = false;
    for (int q = 0; q < cnt; q++) {
      const int p = o + q;
      if (!moved) {
        if (S.pflag[p]) {
          px = fadd(px, S.pdx[p]);
          py = fadd(py, S.pdy[p]);
          moved = true;
        }
        continue;
      }
      const float4 pt = S.pts[p];
      const float lx = pt.x, ly = pt.y;
      const float wx = fadd(px, fsub(fmul(lx, ca), fmul(ly, sa)));
      const float wy = fadd(py, fadd(fmul(lx, sa), fmul(ly, ca)));
      const bool in_box = wx >= sx0 && wx <= sx1 && wy >= sy0 && wy <= sy1;
      float d, nx, ny;
      if (!sdf(rects, in_box ? list : nullptr, in_box ? nlist : nR, wx, wy, &d, &nx, &ny)) continue;
      const float pen = fsub(pt.z, d);
      if (pen <= kSlackPos) continue;
      px = fadd(px, fmul(nx, pen));
      py = fadd(py, fmul(ny, pen));
    }
    S.Q[j].x = px;
    S.Q[j].y = py;
  }
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
  float sp = length2(vx, vy);
  if (sp > K.maxSpeed) {
    float k = fdiv(K.maxSpeed, sp);
    vx = fmul(vx, k); vy = fmul(vy, k);
  }
  if (av > K.maxAngSpeed) av = K.maxAngSpeed;
  else if (av < -K.maxAngSpeed) av = -K.maxAngSpeed;
  if (q.z > 50.f || q.z < -50.f) {
    q.z = wrap_angle(q.z);
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
// results do not depend on it; the batched engine's autotuner picks it.
template <bool World, int G, int U = 1>
__device__ __forceinline__ void island_step(const SolverConsts &K, Island &S,
                                            const float4 *__restrict__ rects, int nR, float cull_d,
                                            const Lanes<G> &L, float reach) {
#pragma unroll U
  for (int s = 0; s < K.substeps; s++) {
    for (int i = L.lane; i < S.nb; i += G) integrate_body<World>(K, S, i);
    L.sync();
    for (int it = 0; it < K.iterations; it++) {
      if constexpr (World) solve_world<G>(K, S, it == 0, L);
      else solve_engine<G>(K, S, it == 0, L);
      collide_island<G>(S, rects, nR, cull_d, L, reach);
    }
    for (int i = L.lane; i < S.nb; i += G) finalize_body<World>(K, S, i);
    L.sync();
  }
  if constexpr (World) {
    for (int u = L.lane; u < S.nu; u += G) {
      float4 *rec = S.units + 4 * u;
      const unsigned ab = __float_as_uint(rec[0].x);
      if ((ab & (kHasPin | kPinIsGrip | kPinBroken)) != (kHasPin | kPinIsGrip)) continue;
      const float4 r1 = rec[1];
      if (grip_breaks(K, r1.z, r1.w, rec[3].z)) {
        rec[0].x = __uint_as_float(ab | kPinBroken);
        rec[1] = make_float4(r1.x, r1.y, 0.f, 0.f);
      }
    }
  } else if (L.lane < S.arms) {
    const float4 g = S.grip[L.lane];
    float4 &an = S.Q[S.nb + L.lane];
    if (an.w == 0.f && grip_breaks(K, g.x, g.y, g.z)) {
      an.w = 1.f;
      S.grip[L.lane] = make_float4(0.f, 0.f, g.z, g.w);
    }
  }
  L.sync();
}

}  // namespace kr
