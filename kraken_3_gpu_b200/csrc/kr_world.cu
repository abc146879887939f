// kr_world.cu -- the gpuworld.js drop-in: handle, schedule and the plain
// step kernel (one launch per kr_step call of up to 128 env steps, one warp per
// creature).
//
// Device buffers hold the reference's own AoS blocks (48 B bodies, 80 B
// constraints, 16 B forces / collision points), so upload and download are
// single copies and mirrorInto/packControls keep their exact field offsets.
// The kernel stages each creature into shared memory for the launch, bodies and
// solve units as 16-byte records.
//
// Schedule.  The reference runs one dispatch per colour class
// (gpuworld.js:353-366); a colour class is body-disjoint, so the classes in
// order are one valid sequential order of the solve list.  Here every
// connected component of the constraint graph (a creature) gets its own
// schedule of solve units in passes (kr_units.h, kr::Island): any order that
// keeps every pair of constraints sharing a body in list order gives
// bit-identical results (the harness check color-order-free,
// harness.js:1172-1193, pins this property for the reference), so the warp's
// pass sweep reproduces the list order exactly.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/kraken_b200.h"
#include "kr_solver.cuh"
#include "kr_units.h"

namespace {

thread_local std::string g_last_error;

constexpr int kWarpsPerBlock = 4;
// Env steps of one launch at most (a few ms): a launch stages the whole world
// from and to global memory, which took a fifth of a one-step launch.
constexpr int kStepsPerLaunch = 128;

// Per-island record, one int array of kIslandInts per island.
enum { I_BODY_OFF = 0, I_NB, I_UNIT_OFF, I_NU, I_PT_OFF, I_PASS_OFF, I_NPASS, kIslandInts };

struct DeviceTables {
  const int *isl;          // nI x kIslandInts
  const int *bodies;       // global body id per island body
  const int4 *units;       // per unit, pass by pass: local a | b << 8 (0xff: the world), global constraint
                           // index of its pin and of its angle constraint (-1: none)
  const int *pts;          // global collision point index, local-body grouped
  const int2 *bpt;         // per island body: (offset within island points, count)
  const int *pass;         // pass offsets per island (npass + 1 each)
};

struct StepArgs {
  kr::SolverConsts K;
  float *bodies;           // nB x 12
  uint32_t *cons;          // nC x 20
  float *forces;           // nB x 4
  const uint4 *coll;       // nP x 4 words
  const float4 *rects;     // nR x (x, y, x+w, y+h)
  int nR;
  float near_d;            // rect culling distance of a collision pass (kr_solver.cuh)
  int nI;
  int n_steps;             // env steps of the launch
  int maxB, maxU, maxP;    // smem carve sizes (per warp)
  DeviceTables T;
};

__host__ __device__ constexpr int warp_smem_words(int mb, int mu, int mp) {
  return 20 * mb + 4 * kr::kWorldRec * mu + 4 * mp + kr::kCullWords + mb;
}

// a block's dynamic shared memory when every warp holds the largest island
constexpr int kMaxWorldSmem =
    (int)sizeof(float) * kWarpsPerBlock *
    warp_smem_words(KR_MAX_ISLAND_BODIES, KR_MAX_ISLAND_CONSTRAINTS, KR_MAX_ISLAND_COLLPTS);

// Writable views of the statics while they are staged; the solver reads them
// through the const pointers of kr::Island.
struct StageView {
  float4 *body, *pts;
};

__device__ inline void carve(kr::Island &S, StageView &V, float *base, int mb, int mu, int mp) {
  float4 *q = reinterpret_cast<float4 *>(base);
  S.P = q; q += mb; S.Q = q; q += mb; S.V = q; q += mb; S.force = q; q += mb;
  V.body = q; q += mb;
  S.units = q; q += kr::kWorldRec * mu;
  V.pts = q; q += mp;
  S.cull = reinterpret_cast<unsigned short *>(q); q += kr::kCullWords / 4;
  S.list = reinterpret_cast<unsigned char *>(q);
  S.body = V.body; S.pts = V.pts;
}

// One launch of the plain step for the island of this warp (shared by the
// plain kernel and its allocation-free variant).
__device__ __forceinline__ void plain_step_body(const StepArgs &A) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float2 s_sin[kr::kSinEntries];
  kr::stage_sin(s_sin);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int island = blockIdx.x * kWarpsPerBlock + warp;
  if (island >= A.nI) return;
  kr::Island S;
  StageView V;
  carve(S, V, smem + warp * warp_smem_words(A.maxB, A.maxU, A.maxP), A.maxB, A.maxU, A.maxP);
  const int *rec = A.T.isl + island * kIslandInts;
  const int bo = rec[I_BODY_OFF], uo = rec[I_UNIT_OFF], po = rec[I_PT_OFF];
  S.nb = rec[I_NB]; S.nu = rec[I_NU];
  S.npass = rec[I_NPASS];
  S.off = A.T.pass + rec[I_PASS_OFF];
  S.tab = s_sin;

  // stage bodies (48 B AoS), forces and the bodies' collision points
  for (int i = lane; i < S.nb; i += 32) {
    const int g = A.T.bodies[bo + i];
    const float4 *b4 = reinterpret_cast<const float4 *>(A.bodies + 12 * (size_t)g);
    const float4 q0 = b4[0], q1 = b4[1], q2 = b4[2];
    S.P[i] = make_float4(q0.x, q0.y, q1.z, 0.f);
    S.Q[i] = make_float4(q0.z, q0.w, q1.w, 0.f);
    S.V[i] = make_float4(q1.x, q1.y, q2.x, 0.f);
    S.force[i] = reinterpret_cast<const float4 *>(A.forces)[g];
    const int2 bp = A.T.bpt[bo + i];
    float reach = 0.f;  // every point lies within it of the centre (+1 px for rounding)
    for (int q = 0; q < bp.y; q++) {
      const uint4 cp = A.coll[A.T.pts[po + bp.x + q]];
      const float lx = __uint_as_float(cp.y), ly = __uint_as_float(cp.z);
      V.pts[bp.x + q] = make_float4(lx, ly, __uint_as_float(cp.w), __int_as_float(i));
      const float d = kr::length2(lx, ly) + 1.f;
      if (!(d <= reach)) reach = d;  // NaN, unless a later point replaces it (it corrects nothing): no list
    }
    V.body[i] = make_float4(q2.y, q2.z, reach, __int_as_float(bp.x | (bp.y << 16)));
  }
  __syncwarp();  // the units read the bodies' masses
  // stage the units' constraints (80 B AoS -> unit records)
  for (int u = lane; u < S.nu; u += 32) {
    const int4 t = A.T.units[uo + u];
    unsigned ab = (unsigned)t.x;
    const int bA = ab & 0xffu, bB = (ab >> 8) & 0xffu;
    const bool has_b = bB != 0xff;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 wa = S.body[bA], wb = has_b ? S.body[bB] : zero;
    float4 r0 = zero, r1 = make_float4(0.f, wa.x, wa.y, wb.x), r2 = make_float4(wb.y, 0.f, 0.f, 0.f), r3 = zero;
    float brk = 0.f;
    if (t.y >= 0) {
      const uint4 *c4 = reinterpret_cast<const uint4 *>(A.cons + 20 * (size_t)t.y);
      const uint4 w0 = c4[0], w1 = c4[1], w2 = c4[2], w4 = c4[4];
      ab |= kr::kHasPin | (w4.y != 0u ? kr::kPinBroken : 0u) | ((w0.z & 0xffu) == 2u ? kr::kPinIsGrip : 0u);
      r0.y = __uint_as_float(w1.x); r0.z = __uint_as_float(w1.y);
      r0.w = __uint_as_float(w1.z); r1.x = __uint_as_float(w1.w);
      r3.y = kr::fmul(__uint_as_float(w2.x), A.K.invH2);
      brk = __uint_as_float(w4.x);
    }
    if (t.z >= 0) {
      const uint4 *c4 = reinterpret_cast<const uint4 *>(A.cons + 20 * (size_t)t.z);
      const uint4 w2 = c4[2], w3 = c4[3], w4 = c4[4];
      ab |= kr::kHasAngle | (w4.y != 0u ? kr::kAngleBroken : 0u);
      r2 = make_float4(wb.y, __uint_as_float(w2.y), __uint_as_float(w2.w), __uint_as_float(w3.x));
      r3.x = __uint_as_float(w2.z);
      r3.z = kr::fmul(__uint_as_float(w2.x), A.K.invH2);
      r3.w = kr::recip(kr::fadd(wa.y, wb.y));
    }
    ab |= kr::unit_forms(t.y >= 0, bA == bB, r0.y, r0.z, has_b ? r0.w : 0.f, has_b ? r1.x : 0.f, wa.x, wa.y, wb.x, wb.y);
    r0.x = __uint_as_float(ab);
    float4 *rec = S.units + kr::kWorldRec * u;
    rec[0] = r0; rec[1] = r1; rec[2] = r2; rec[3] = r3; rec[4] = make_float4(0.f, 0.f, 0.f, brk);
  }
  __syncwarp();

  // env steps back to back: what a launch per step would write back and stage
  // again is what shared memory holds
  kr::Near near;
  for (int s = 0; s < A.n_steps; s++)
    kr::island_step<true, 32, 1, true>(A.K, S, A.rects, A.nR, A.near_d, kr::Lanes<32>(lane), near);

  // write back bodies, consumed forces and constraint multipliers / flags
  for (int i = lane; i < S.nb; i += 32) {
    const int g = A.T.bodies[bo + i];
    float4 *b4 = reinterpret_cast<float4 *>(A.bodies + 12 * (size_t)g);
    const float pad = A.bodies[12 * (size_t)g + 11];
    const float4 p = S.P[i], q = S.Q[i], v = S.V[i], bd = S.body[i];
    b4[0] = make_float4(p.x, p.y, q.x, q.y);
    b4[1] = make_float4(v.x, v.y, p.z, q.z);
    b4[2] = make_float4(v.z, bd.x, bd.y, pad);
    if (!(bd.x == 0.f && bd.y == 0.f)) {
      float *f = A.forces + 4 * (size_t)g;
      f[0] = 0.f; f[1] = 0.f; f[2] = 0.f;  // consumed, adhesion kept (solver.wgsl:204)
    }
  }
  // every multiplier starts each substep at 0, so a pin's angle multiplier
  // and an angle constraint's pin multiplier end at 0
  for (int u = lane; u < S.nu; u += 32) {
    const int4 t = A.T.units[uo + u];
    const unsigned ab = __float_as_uint(S.units[kr::kWorldRec * u].x);
    const float4 d = S.units[kr::kWorldRec * u + 4];
    if (t.y >= 0) {
      uint32_t *c = A.cons + 20 * (size_t)t.y;
      c[13] = __float_as_uint(d.x);
      c[14] = __float_as_uint(d.y);
      c[15] = 0u;
      c[17] = (ab & kr::kPinBroken) ? 1u : 0u;
    }
    if (t.z >= 0) {
      uint32_t *c = A.cons + 20 * (size_t)t.z;
      c[13] = 0u;
      c[14] = 0u;
      c[15] = __float_as_uint(d.z);
      c[17] = (ab & kr::kAngleBroken) ? 1u : 0u;
    }
  }
}

__global__ void __launch_bounds__(32 * kWarpsPerBlock, 4) plain_step_kernel(StepArgs A) {
  plain_step_body(A);
}

// The copy runs on the handle's stream: after the steps that still read the
// old table, before those that read the new one (the handle's stream does not
// wait for the legacy one, on which a plain copy would run).
template <typename T>
cudaError_t dev_upload(T **dptr, size_t *cap, const std::vector<T> &v, cudaStream_t st) {
  size_t n = std::max<size_t>(v.size(), 1);
  if (*dptr == nullptr || *cap < n) {
    if (*dptr) cudaFree(*dptr);
    *dptr = nullptr;
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(dptr), n * sizeof(T));
    if (e != cudaSuccess) return e;
    *cap = n;
  }
  if (v.empty()) return cudaSuccess;
  return cudaMemcpyAsync(*dptr, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st);
}

}  // namespace

struct kr_world {
  kr_solver_params p{};
  kr::SolverConsts K{};
  uint32_t nB = 0, nC = 0, nP = 0, nR = 0;
  float *d_bodies = nullptr;
  uint32_t *d_cons = nullptr;
  uint32_t *d_stage = nullptr;          // staging copy of a control upload
  size_t smem_bytes = 0;
  float *d_forces = nullptr;
  float4 *d_rects = nullptr;
  uint4 *d_coll = nullptr;
  std::vector<uint32_t> h_coll_range;   // 2 x nB
  // island tables
  int *d_isl = nullptr, *d_ibodies = nullptr, *d_ipts = nullptr, *d_pass = nullptr;
  int4 *d_units = nullptr;
  int2 *d_bpt = nullptr;
  size_t c_isl = 0, c_ibodies = 0, c_units = 0, c_ipts = 0, c_pass = 0, c_bpt = 0;
  float near_d = 0.f;
  int nI = 0, maxB = 1, maxU = 1, maxP = 1, maxLv = 0;
  bool uploaded = false;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;

  int fail(int code, const std::string &msg) {
    err = msg;
    return code;
  }
  int cuda_fail(cudaError_t e, const char *what) {
    err = std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e);
    return KR_ERR_CUDA;
  }
};

extern "C" int kr_device_count(void) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess) {
    g_last_error = std::string("cudaGetDeviceCount: ") + cudaGetErrorString(e);
    cudaGetLastError();
    return 0;
  }
  return n;
}

extern "C" const char *kr_last_error(const kr_world *w) {
  if (w) return w->err.c_str();
  return g_last_error.c_str();
}

extern "C" int kr_create(const kr_solver_params *params, uint32_t n_bodies, uint32_t n_constraints,
                         const float *rects, uint32_t n_rects, const uint32_t *coll_pts,
                         uint32_t n_coll_pts, const uint32_t *coll_range, kr_world **out) {
  if (!out || !params) {
    g_last_error = "kr_create: null argument";
    return KR_ERR_INVALID;
  }
  *out = nullptr;
  const kr_solver_params &p = *params;
  // sanity guards of writeStatic (gpuworld.js:224-229), same bounds
  if (!(p.iterations >= 1 && p.iterations <= 64)) {
    g_last_error = "iterations implausible: " + std::to_string(p.iterations);
    return KR_ERR_INVALID;
  }
  if (!(n_rects >= 1 && n_rects <= 100000)) {
    g_last_error = "nRects implausible: " + std::to_string(n_rects);
    return KR_ERR_INVALID;
  }
  if (!(n_bodies >= 1 && n_bodies <= 4000000)) {
    g_last_error = "nBodies implausible: " + std::to_string(n_bodies);
    return KR_ERR_INVALID;
  }
  const float hf = static_cast<float>(p.h);
  if (!(hf > 0.f && hf < 1.f)) {
    g_last_error = "h implausible: " + std::to_string(p.h);
    return KR_ERR_INVALID;
  }
  if (p.substeps < 1 || p.substeps > 64) {
    g_last_error = "substeps implausible: " + std::to_string(p.substeps);
    return KR_ERR_INVALID;
  }
  if ((n_coll_pts > 0 && (!coll_pts || !coll_range)) || !rects) {
    g_last_error = "kr_create: missing rects or collision points";
    return KR_ERR_INVALID;
  }
  // collRange must cover the points exactly (gpuworld.js:193-199)
  uint64_t acc = 0;
  if (coll_range) {
    for (uint32_t b = 0; b < n_bodies; b++) {
      if (coll_range[b] != acc) {
        g_last_error = "collRange offsets are not contiguous at body " + std::to_string(b);
        return KR_ERR_INVALID;
      }
      acc += coll_range[n_bodies + b];
    }
    for (uint32_t i = 0; i < n_coll_pts; i++) {
      if (coll_pts[4 * i] >= n_bodies) {
        g_last_error = "collPt " + std::to_string(i) + " refers to body " +
                       std::to_string(coll_pts[4 * i]) + " of " + std::to_string(n_bodies);
        return KR_ERR_INDEX;
      }
    }
  }
  if (acc != n_coll_pts) {
    g_last_error = "collRange covers " + std::to_string(acc) + " of " +
                   std::to_string(n_coll_pts) + " points";
    return KR_ERR_INVALID;
  }
  int dev_count = 0;
  if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count == 0) {
    cudaGetLastError();
    g_last_error = "no CUDA device available";
    return KR_ERR_NODEVICE;
  }

  kr_world *w = new kr_world();
  w->p = p;
  w->nB = n_bodies; w->nC = n_constraints; w->nP = n_coll_pts; w->nR = n_rects;
  // f32 constants: writeStatic F[0], F[10], F[11] and f32solver.mjs:79-85
  kr::SolverConsts &K = w->K;
  K.h = hf;
  K.invH = static_cast<float>(1.0 / p.h);
  K.invH2 = static_cast<float>(1.0 / (p.h * p.h));
  const float nl = -static_cast<float>(p.lin_drag), na = -static_cast<float>(p.ang_drag);
  K.linDamp = static_cast<float>(std::exp(static_cast<double>(nl * hf)));
  K.angDamp = static_cast<float>(std::exp(static_cast<double>(na * hf)));
  K.maxSpeed = static_cast<float>(p.max_speed);
  K.maxAngSpeed = static_cast<float>(p.max_ang_speed);
  K.substeps = p.substeps;
  K.iterations = p.iterations;

  cudaError_t e;
  auto cleanup_fail = [&](cudaError_t ce, const char *what) {
    g_last_error = std::string("CUDA error in ") + what + ": " + cudaGetErrorString(ce);
    kr_destroy(w);
    return KR_ERR_CUDA;
  };
  if ((e = cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking)) != cudaSuccess)
    return cleanup_fail(e, "cudaStreamCreate");
  w->own_stream = true;
  if ((e = cudaMalloc(&w->d_bodies, sizeof(float) * 12 * n_bodies)) != cudaSuccess)
    return cleanup_fail(e, "cudaMalloc(bodies)");
  if ((e = cudaMalloc(&w->d_cons, sizeof(uint32_t) * 20 * std::max<uint32_t>(n_constraints, 1))) !=
      cudaSuccess)
    return cleanup_fail(e, "cudaMalloc(cons)");
  if ((e = cudaMalloc(&w->d_stage, sizeof(uint32_t) * 20 * std::max<uint32_t>(n_constraints, 1))) !=
      cudaSuccess)
    return cleanup_fail(e, "cudaMalloc(control staging)");
  if ((e = cudaMalloc(&w->d_forces, sizeof(float) * 4 * n_bodies)) != cudaSuccess)
    return cleanup_fail(e, "cudaMalloc(forces)");
  if ((e = cudaMemsetAsync(w->d_forces, 0, sizeof(float) * 4 * n_bodies, w->stream)) != cudaSuccess)
    return cleanup_fail(e, "cudaMemset(forces)");
  std::vector<float4> r4(n_rects);
  double half_thick = 0.0, r_max = 0.0;
  for (uint32_t i = 0; i < n_rects; i++) {
    const float x = rects[4 * i], y = rects[4 * i + 1], rw = rects[4 * i + 2], rh = rects[4 * i + 3];
    r4[i] = make_float4(x, y, x + rw, y + rh);  // f32 sums, as solver.wgsl:120-121
    const double ht = 0.5 * std::min(std::fabs((double)rw), std::fabs((double)rh));
    if (std::isfinite(ht)) half_thick = std::max(half_thick, ht);
    else half_thick = HUGE_VAL;
  }
  for (uint32_t i = 0; i < n_coll_pts; i++) {
    float r;
    std::memcpy(&r, &coll_pts[4 * i + 3], sizeof(float));
    if (std::isfinite(r)) r_max = std::max(r_max, std::fabs((double)r));
    else r_max = HUGE_VAL;
  }
  // D = max(radius, half thickness) + 2; the f32 rounding of the box tests is
  // covered by the pad
  const double cull = std::max(r_max, half_thick) + 2.0 + kr::kCullPad;
  w->near_d = std::isfinite(cull) && cull < 1e30 ? (float)cull : 1e30f;
  if ((e = cudaMalloc(&w->d_rects, sizeof(float4) * n_rects)) != cudaSuccess)
    return cleanup_fail(e, "cudaMalloc(rects)");
  if ((e = cudaMemcpyAsync(w->d_rects, r4.data(), sizeof(float4) * n_rects, cudaMemcpyHostToDevice,
                           w->stream)) != cudaSuccess)
    return cleanup_fail(e, "cudaMemcpy(rects)");
  if ((e = cudaMalloc(&w->d_coll, sizeof(uint4) * std::max<uint32_t>(n_coll_pts, 1))) != cudaSuccess)
    return cleanup_fail(e, "cudaMalloc(collPts)");
  if (n_coll_pts &&
      (e = cudaMemcpyAsync(w->d_coll, coll_pts, sizeof(uint4) * n_coll_pts, cudaMemcpyHostToDevice,
                           w->stream)) != cudaSuccess)
    return cleanup_fail(e, "cudaMemcpy(collPts)");
  if ((e = cudaStreamSynchronize(w->stream)) != cudaSuccess) return cleanup_fail(e, "create(sync)");
  w->h_coll_range.assign(2 * (size_t)n_bodies, 0u);
  if (coll_range) std::memcpy(w->h_coll_range.data(), coll_range, sizeof(uint32_t) * 2 * n_bodies);
  *out = w;
  return KR_OK;
}

namespace {

// Connected components, per-component unit passes and lane tables (see the file
// comment).  Returns KR_OK or an error code with w->err set.
int build_schedule(kr_world *w, const float *bodies, const uint32_t *cons) {
  const uint32_t nB = w->nB, nC = w->nC;
  std::vector<int> parent(nB);
  std::iota(parent.begin(), parent.end(), 0);
  auto find = [&](int x) {
    while (parent[x] != x) { parent[x] = parent[parent[x]]; x = parent[x]; }
    return x;
  };
  for (uint32_t k = 0; k < nC; k++) {
    const uint32_t a = cons[20 * k], b = cons[20 * k + 1];
    if (a >= nB || (b != 0xffffffffu && b >= nB)) {
      return w->fail(KR_ERR_INDEX, "Constraint " + std::to_string(k) + ": body index " +
                                       std::to_string(a) + "/" +
                                       (b == 0xffffffffu ? std::string("-1") : std::to_string(b)) +
                                       " outside of " + std::to_string(nB) +
                                       " (an out-of-bounds read in the kernel)");
    }
    if (b != 0xffffffffu) {
      int ra = find((int)a), rb = find((int)b);
      if (ra != rb) parent[std::max(ra, rb)] = std::min(ra, rb);
    }
  }
  // islands in order of their smallest body
  std::vector<int> island_of(nB), local(nB);
  std::vector<std::vector<int>> ib;  // bodies per island
  std::vector<int> root_island(nB, -1);
  for (uint32_t g = 0; g < nB; g++) {
    int r = find((int)g);
    if (root_island[r] < 0) { root_island[r] = (int)ib.size(); ib.emplace_back(); }
    int I = root_island[r];
    island_of[g] = I;
    local[g] = (int)ib[I].size();
    ib[I].push_back((int)g);
  }
  const int nI = (int)ib.size();
  std::vector<std::vector<int>> ic(nI);  // constraints per island, list order
  for (uint32_t k = 0; k < nC; k++) ic[island_of[cons[20 * k]]].push_back((int)k);

  std::vector<int> isl(nI * (size_t)kIslandInts), h_bodies, h_pts, h_pass;
  std::vector<int4> h_units;
  std::vector<int2> h_bpt;
  h_bodies.reserve(nB); h_units.reserve(nC);
  int maxB = 1, maxU = 1, maxP = 1, maxLv = 0;
  std::vector<int> last_level, order, off;
  std::vector<kr::SolveEntry> list, list_of;
  int list_nb = 0;
  std::vector<kr::SolveUnit> units;
  for (int I = 0; I < nI; I++) {
    const auto &bl = ib[I];
    const auto &cl = ic[I];
    const int nb = (int)bl.size(), nc = (int)cl.size();
    if (nb > KR_MAX_ISLAND_BODIES || nc > KR_MAX_ISLAND_CONSTRAINTS)
      return w->fail(KR_ERR_CAPACITY, "connected component " + std::to_string(I) + " has " +
                                          std::to_string(nb) + " bodies and " +
                                          std::to_string(nc) + " constraints; the kernel holds " +
                                          std::to_string(KR_MAX_ISLAND_BODIES) + " / " +
                                          std::to_string(KR_MAX_ISLAND_CONSTRAINTS));
    int *rec = &isl[I * (size_t)kIslandInts];
    rec[I_BODY_OFF] = (int)h_bodies.size();
    rec[I_NB] = nb;
    for (int g : bl) h_bodies.push_back(g);
    // the list, and its constraint levels (each on the first level after
    // every earlier constraint sharing a body)
    last_level.assign(nb, -1);
    list.resize(nc);
    int nlv = 0;
    for (int q = 0; q < nc; q++) {
      const uint32_t *c = cons + 20 * (size_t)cl[q];
      const int a = local[c[0]];
      const int b = c[1] == 0xffffffffu ? -1 : local[c[1]];
      int L = last_level[a] + 1;
      if (b >= 0) L = std::max(L, last_level[b] + 1);
      last_level[a] = L;
      if (b >= 0) last_level[b] = L;
      nlv = std::max(nlv, L + 1);
      list[q] = kr::SolveEntry{(c[2] & 0xffu) == 1u ? 1 : 0, a, b};
    }
    if (nlv > KR_MAX_LEVELS)
      return w->fail(KR_ERR_CAPACITY, "connected component " + std::to_string(I) + " needs " +
                                          std::to_string(nlv) + " constraint levels; the kernel holds " +
                                          std::to_string(KR_MAX_LEVELS));
    // islands of one structure (a population of one body shape) follow one
    // another: the last one's units serve again
    const bool again = I > 0 && nb == list_nb && list.size() == list_of.size() &&
                       std::equal(list.begin(), list.end(), list_of.begin(), [](const auto &x, const auto &y) {
                         return x.angle == y.angle && x.a == y.a && x.b == y.b;
                       });
    if (!again) {
      kr::build_units(list, nb, &units, last_level);
      kr::schedule_units(units, nb, 32, &order, &off);
      list_of = list;
      list_nb = nb;
    }
    rec[I_PASS_OFF] = (int)h_pass.size();
    rec[I_NPASS] = (int)off.size() - 1;
    h_pass.insert(h_pass.end(), off.begin(), off.end());
    rec[I_UNIT_OFF] = (int)h_units.size();
    rec[I_NU] = (int)units.size();
    for (int u : order) {
      const kr::SolveUnit &x = units[u];
      h_units.push_back(make_int4(x.a | ((x.b >= 0 ? x.b : 0xff) << 8), x.pin >= 0 ? cl[x.pin] : -1,
                                  x.ang >= 0 ? cl[x.ang] : -1, 0));
    }
    // collision points in local body order
    rec[I_PT_OFF] = (int)h_pts.size();
    int np = 0;
    for (int j = 0; j < nb; j++) {
      const int g = bl[j];
      const uint32_t off = w->h_coll_range[g], cnt = w->h_coll_range[nB + g];
      h_bpt.push_back(make_int2(np, (int)cnt));
      for (uint32_t q = 0; q < cnt; q++) h_pts.push_back((int)(off + q));
      np += (int)cnt;
    }
    if (np > KR_MAX_ISLAND_COLLPTS)
      return w->fail(KR_ERR_CAPACITY, "connected component " + std::to_string(I) + " has " +
                                          std::to_string(np) + " collision points; the kernel holds " +
                                          std::to_string(KR_MAX_ISLAND_COLLPTS));
    maxB = std::max(maxB, nb);
    maxU = std::max(maxU, (int)units.size());
    maxP = std::max(maxP, np);
    maxLv = std::max(maxLv, nlv);
  }
  // steps in flight read the tables that are replaced or freed now
  cudaError_t e = cudaStreamSynchronize(w->stream);
  if (e != cudaSuccess) return w->cuda_fail(e, "upload(steps in flight)");
  if ((e = dev_upload(&w->d_isl, &w->c_isl, isl, w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(islands)");
  if ((e = dev_upload(&w->d_ibodies, &w->c_ibodies, h_bodies, w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(island bodies)");
  if ((e = dev_upload(&w->d_units, &w->c_units, h_units, w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(island units)");
  if ((e = dev_upload(&w->d_ipts, &w->c_ipts, h_pts, w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(island points)");
  if ((e = dev_upload(&w->d_bpt, &w->c_bpt, h_bpt, w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(body point ranges)");
  if ((e = dev_upload(&w->d_pass, &w->c_pass, h_pass, w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(passes)");
  w->nI = nI;
  // round up so every per-warp region keeps 16-byte alignment of its arrays
  w->maxB = (maxB + 3) & ~3;
  w->maxU = maxU;
  w->maxP = (maxP + 3) & ~3;
  w->maxLv = maxLv;
  w->smem_bytes =
      sizeof(float) * kWarpsPerBlock * (size_t)warp_smem_words(w->maxB, w->maxU, w->maxP);
  // the limit belongs to the kernel, not to the handle: always the largest
  // island's, so that no upload lowers it below another handle's launches
  if ((e = cudaFuncSetAttribute(plain_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxWorldSmem)) !=
      cudaSuccess)
    return w->cuda_fail(e, "cudaFuncSetAttribute(plain_step_kernel)");
  return KR_OK;
}

}  // namespace

extern "C" int kr_upload(kr_world *w, const float *bodies, const uint32_t *cons, const float *forces,
                         const uint32_t *color_info) {
  if (!w) return KR_ERR_INVALID;
  if (!bodies || (w->nC && !cons)) return w->fail(KR_ERR_INVALID, "kr_upload: null buffer");
  if (color_info) {
    uint32_t acc = 0;
    for (int c = 0; c < 16; c++) {
      if (color_info[c] != acc)
        return w->fail(KR_ERR_INVALID, "colorInfo: colour " + std::to_string(c) +
                                           " does not start where the previous one ends");
      acc += color_info[16 + c];
    }
    if (acc != w->nC)
      return w->fail(KR_ERR_INVALID, "colorInfo covers " + std::to_string(acc) + " of " +
                                         std::to_string(w->nC) + " constraints");
  }
  int rc = build_schedule(w, bodies, cons);
  if (rc != KR_OK) return rc;
  cudaError_t e;
  if ((e = cudaMemcpyAsync(w->d_bodies, bodies, sizeof(float) * 12 * w->nB, cudaMemcpyHostToDevice,
                           w->stream)) != cudaSuccess)
    return w->cuda_fail(e, "upload(bodies)");
  if (w->nC && (e = cudaMemcpyAsync(w->d_cons, cons, sizeof(uint32_t) * 20 * w->nC,
                                    cudaMemcpyHostToDevice, w->stream)) != cudaSuccess)
    return w->cuda_fail(e, "upload(cons)");
  if (forces) {
    if ((e = cudaMemcpyAsync(w->d_forces, forces, sizeof(float) * 4 * w->nB, cudaMemcpyHostToDevice,
                             w->stream)) != cudaSuccess)
      return w->cuda_fail(e, "upload(forces)");
  } else if ((e = cudaMemsetAsync(w->d_forces, 0, sizeof(float) * 4 * w->nB, w->stream)) !=
             cudaSuccess) {
    return w->cuda_fail(e, "upload(forces)");
  }
  if ((e = cudaStreamSynchronize(w->stream)) != cudaSuccess) return w->cuda_fail(e, "upload(sync)");
  w->uploaded = true;
  return KR_OK;
}

namespace {
// Copies the control fields of the 80 B records (packControls, gpuworld.js:331-341).
__global__ void controls_kernel(uint32_t *dst, const uint32_t *src, int nC) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nC) return;
  const uint32_t *s = src + 20 * (size_t)k;
  uint32_t *d = dst + 20 * (size_t)k;
  d[6] = s[6]; d[7] = s[7]; d[8] = s[8]; d[10] = s[10]; d[16] = s[16]; d[17] = s[17];
}
}  // namespace

extern "C" int kr_upload_controls(kr_world *w, const uint32_t *cons) {
  if (!w) return KR_ERR_INVALID;
  if (!w->uploaded) return w->fail(KR_ERR_STATE, "uploadControls before upload");
  if (!w->nC) return KR_OK;
  if (!cons) return w->fail(KR_ERR_INVALID, "kr_upload_controls: null buffer");
  // stage the whole block once, then scatter the six control words per record
  cudaError_t e = cudaMemcpyAsync(w->d_stage, cons, sizeof(uint32_t) * 20 * w->nC,
                                  cudaMemcpyHostToDevice, w->stream);
  if (e != cudaSuccess) return w->cuda_fail(e, "uploadControls(copy)");
  controls_kernel<<<(w->nC + 255) / 256, 256, 0, w->stream>>>(w->d_cons, w->d_stage, (int)w->nC);
  e = cudaGetLastError();
  if (e != cudaSuccess) return w->cuda_fail(e, "uploadControls(scatter)");
  return KR_OK;
}

extern "C" int kr_step(kr_world *w, int32_t n_steps) {
  if (!w) return KR_ERR_INVALID;
  if (!w->uploaded) return w->fail(KR_ERR_STATE, "step before upload");
  if (n_steps < 0) return w->fail(KR_ERR_INVALID, "n_steps < 0");
  if (n_steps == 0 || w->nI == 0) return KR_OK;
  StepArgs A;
  A.K = w->K;
  A.bodies = w->d_bodies;
  A.cons = w->d_cons;
  A.forces = w->d_forces;
  A.coll = w->d_coll;
  A.rects = w->d_rects;
  A.nR = (int)w->nR;
  A.nI = w->nI;
  A.maxB = w->maxB; A.maxU = w->maxU; A.maxP = w->maxP;
  A.T = DeviceTables{w->d_isl, w->d_ibodies, w->d_units, w->d_ipts, w->d_bpt, w->d_pass};
  A.near_d = w->near_d;
  const size_t smem = w->smem_bytes;
  cudaError_t e;
  const int grid = (w->nI + kWarpsPerBlock - 1) / kWarpsPerBlock;
  for (int s = 0; s < n_steps; s += kStepsPerLaunch) {
    A.n_steps = std::min(kStepsPerLaunch, n_steps - s);
    plain_step_kernel<<<grid, 32 * kWarpsPerBlock, smem, w->stream>>>(A);
    e = cudaGetLastError();
    if (e != cudaSuccess) return w->cuda_fail(e, "plain_step_kernel launch");
  }
  return KR_OK;
}

extern "C" int kr_download(kr_world *w, float *bodies, uint32_t *cons) {
  if (!w) return KR_ERR_INVALID;
  if (!w->uploaded) return w->fail(KR_ERR_STATE, "download before upload");
  cudaError_t e;
  const size_t nb = sizeof(float) * 12 * (size_t)w->nB, nc = cons ? sizeof(uint32_t) * 20 * (size_t)w->nC : 0;
  if (bodies && (e = cudaMemcpyAsync(bodies, w->d_bodies, nb, cudaMemcpyDeviceToHost, w->stream)) != cudaSuccess)
    return w->cuda_fail(e, "download(bodies)");
  if (nc && (e = cudaMemcpyAsync(cons, w->d_cons, nc, cudaMemcpyDeviceToHost, w->stream)) != cudaSuccess)
    return w->cuda_fail(e, "download(cons)");
  if ((e = cudaStreamSynchronize(w->stream)) != cudaSuccess) return w->cuda_fail(e, "download(sync)");
  return KR_OK;
}

extern "C" int kr_sync(kr_world *w) {
  if (!w) return KR_ERR_INVALID;
  cudaError_t e = cudaStreamSynchronize(w->stream);
  if (e != cudaSuccess) return w->cuda_fail(e, "cudaStreamSynchronize");
  return KR_OK;
}

extern "C" int kr_set_stream(kr_world *w, void *stream) {
  if (!w) return KR_ERR_INVALID;
  cudaError_t e = cudaStreamSynchronize(w->stream);
  if (e != cudaSuccess) return w->cuda_fail(e, "cudaStreamSynchronize");
  if (stream) {
    if (w->own_stream) cudaStreamDestroy(w->stream);
    w->own_stream = false;
    w->stream = static_cast<cudaStream_t>(stream);
  } else if (!w->own_stream) {
    e = cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return w->cuda_fail(e, "cudaStreamCreate");
    w->own_stream = true;
  }
  return KR_OK;
}

extern "C" int kr_world_islands(const kr_world *w, int32_t *n_islands, int32_t *max_levels) {
  if (!w) return KR_ERR_INVALID;
  if (n_islands) *n_islands = w->nI;
  if (max_levels) *max_levels = w->maxLv;
  return KR_OK;
}

extern "C" void kr_destroy(kr_world *w) {
  if (!w) return;
  if (w->stream) cudaStreamSynchronize(w->stream);
  void *ptrs[] = {w->d_bodies, w->d_cons, w->d_stage, w->d_forces, w->d_rects, w->d_coll, w->d_isl,
                  w->d_ibodies, w->d_units, w->d_ipts, w->d_pass, w->d_bpt};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (w->own_stream && w->stream) cudaStreamDestroy(w->stream);
  delete w;
}

// ---------------------------------------------------------------------------
// Allocation-free step (kr_step_noalloc).
//
// For callers that cannot allocate GPU memory -- code running inside a
// host-side memory pool, an embedding that owns every device allocation, a
// real-time loop where cudaMalloc's implicit synchronization is not
// allowed.  Everything the step needs beyond the caller's own buffers (the
// per-creature schedule, the converted rect list, the culling distance)
// lives in one file-scope device array of fixed size, so the call allocates
// nothing on the device or the host.
//
// Scratch layout (words): island records, island bodies, units, island
// points, body point ranges, pass offsets, rects.  The builder's temporaries
// are in its block's shared memory.  The array is shared by every call on a
// device and keeps the last call's contents; the builder initializes every
// word it reads before reading it.
// ---------------------------------------------------------------------------
namespace {

constexpr int kNaB = KR_NOALLOC_MAX_BODIES;
constexpr int kNaC = KR_NOALLOC_MAX_CONSTRAINTS;
constexpr int kNaP = KR_NOALLOC_MAX_COLLPTS;
constexpr int kNaR = KR_NOALLOC_MAX_RECTS;
// region offsets in words
constexpr int kOffHdr = 0;                                  // n_islands, near_d, status, pad
constexpr int kOffIsl = 4;
constexpr int kOffBodies = kOffIsl + kNaB * kIslandInts;
constexpr int kOffUnits = (kOffBodies + kNaB + 3) & ~3;    // int4, 16-byte aligned
constexpr int kOffPts = kOffUnits + 4 * kNaC;
constexpr int kOffBpt = ((kOffPts + kNaP) + 1) & ~1;       // int2, 8-byte aligned
constexpr int kOffPass = kOffBpt + 2 * kNaB;
constexpr int kOffRects = ((kOffPass + kNaC + kNaB) + 3) & ~3;  // float4, 16-byte aligned
constexpr int kScratchWords = kOffRects + 4 * kNaR;

static __device__ __align__(256) int g_noalloc_scratch[kScratchWords];

// Schedule builder, one block: the islands, bodies and point ranges of
// build_schedule() and the same units, in passes by level.  A single thread
// over global memory took 5.3 ms for 40 creatures, all of it load latency;
// here (a 40-creature call of 4 steps: 5.9 -> 0.24 ms) the temporaries are in
// shared memory and only what is sequential by nature runs in order -- the
// ranks within an island by one warp, 32 entries at a time, and an island's
// units by one thread per island.
constexpr int kBuildThreads = 1024;

// Exclusive scan of v[0..n) in place, n <= 2 * kBuildThreads; returns the
// total.  sums: 32 ints.  Every thread of the block calls it.
__device__ __forceinline__ int block_scan(int *v, int n, int *sums) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int x0 = 2 * t < n ? v[2 * t] : 0, x1 = 2 * t + 1 < n ? v[2 * t + 1] : 0;
  int x = x0 + x1;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int s = sums[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    sums[lane] = s;
  }
  __syncthreads();
  const int before = x - x0 - x1 + (warp ? sums[warp - 1] : 0), total = sums[31];
  if (2 * t < n) v[2 * t] = before;
  if (2 * t + 1 < n) v[2 * t + 1] = before + x0;
  __syncthreads();
  return total;
}

// The builder's shared memory
struct BuildSmem {
  int par[kNaB];             // union-find parent
  int isl[kNaB];             // island of a body
  int loc[kNaB];             // its index in the island
  int bo[kNaB + 1];          // islands' body offsets
  int co[kNaB + 1];          // islands' constraint offsets
  int po[kNaB + 1];          // islands' point offsets
  int cnt[kNaB + 1];
  int last[kNaB], last_unit[kNaB];  // level and unit last on a body (by its place in island order)
  int con[kNaC];             // island order: local a | b << 8 | angle << 16
  int cur[kNaC + kNaB];      // level counts, nc + 1 words per island
  unsigned short list[kNaC]; // island order: constraint index
  short pin[kNaC], ang[kNaC];  // units in list order: place of their constraints
  short level[kNaC];
  int sums[32];
  int bad;
  double half_thick, r_max;
};

// Ranks by key in index order, by one warp: rank(i) = how many of 0..i-1 have
// key(i); count[key] ends up as the number of entries.
template <class Key, class Out>
__device__ __forceinline__ void ordered_ranks(int n, int *count, Key key, Out out) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const int k = i < n ? key(i) : -1;
    const unsigned m = __match_any_sync(0xffffffffu, k);
    const int before = k >= 0 ? count[k] : 0;
    __syncwarp();
    const int r = __popc(m & ((1u << lane) - 1u));
    if (k >= 0) {
      out(i, before + r);
      if (r == 0) count[k] = before + __popc(m);
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kBuildThreads) noalloc_schedule_kernel(
    int *W, const float *bodies, const uint32_t *cons, const float *rects, const uint32_t *coll_pts,
    const uint32_t *coll_range, int nB, int nC, int nP, int nR) {
  extern __shared__ __align__(16) unsigned char build_smem[];
  BuildSmem &M = *reinterpret_cast<BuildSmem *>(build_smem);
  const int t = threadIdx.x;
  int *isl = W + kOffIsl, *ib = W + kOffBodies, *ipts = W + kOffPts, *pass = W + kOffPass;
  int4 *units = reinterpret_cast<int4 *>(W + kOffUnits);
  int2 *bpt = reinterpret_cast<int2 *>(W + kOffBpt);
  float4 *r4 = reinterpret_cast<float4 *>(W + kOffRects);
  auto fail = [&](int code) {
    if (t == 0) {
      W[kOffHdr + 0] = 0;
      W[kOffHdr + 2] = code;
    }
  };
  // collRange must tile the points in body order (gpuworld.js:193-199).  A
  // count above nP is refused by itself, so the 32-bit prefix sums of the
  // others stay below 2^24 and every range lies inside [0, nP).
  bool bad = false;
  for (int g = t; g < nB; g += kBuildThreads) {
    const uint32_t c = coll_range[nB + g];
    bad |= c > (uint32_t)nP;
    M.cnt[g] = c > (uint32_t)nP ? 0 : (int)c;
  }
  if (__syncthreads_or(bad)) { fail(KR_ERR_INVALID); return; }
  const int total = block_scan(M.cnt, nB, M.sums);
  for (int g = t; g < nB; g += kBuildThreads) bad |= coll_range[g] != (uint32_t)M.cnt[g];
  if (__syncthreads_or(bad || total != nP)) { fail(KR_ERR_INVALID); return; }
  // connected components: hook the larger root below the smaller until no
  // constraint joins two; a component's root is its smallest body
  for (int k = t; k < nC; k += kBuildThreads) {
    const uint32_t a = cons[20 * (size_t)k], b = cons[20 * (size_t)k + 1];
    bad |= a >= (uint32_t)nB || (b != 0xffffffffu && b >= (uint32_t)nB);
  }
  if (__syncthreads_or(bad)) { fail(KR_ERR_INDEX); return; }
  for (int g = t; g < nB; g += kBuildThreads) M.par[g] = g;
  __syncthreads();
  auto root = [&](int x) {
    for (;;) {
      const int p = *(volatile int *)&M.par[x];
      if (p == x) return x;
      x = p;
    }
  };
  for (int round = 0; round < nB; round++) {  // ends after a few rounds: every round joins what it finds apart
    bool joined = false;
    for (int k = t; k < nC; k += kBuildThreads) {
      const uint32_t b = cons[20 * (size_t)k + 1];
      if (b == 0xffffffffu) continue;
      const int ra = root((int)cons[20 * (size_t)k]), rb = root((int)b);
      if (ra != rb) {
        atomicMin(&M.par[max(ra, rb)], min(ra, rb));
        joined = true;
      }
    }
    if (!__syncthreads_or(joined)) break;
    for (int g = t; g < nB; g += kBuildThreads) M.par[g] = root(g);
    __syncthreads();
  }
  // islands in order of their smallest body
  for (int g = t; g < nB; g += kBuildThreads) M.last[g] = M.par[g] == g ? 1 : 0;
  __syncthreads();
  const int nI = block_scan(M.last, nB, M.sums);
  for (int g = t; g < nB; g += kBuildThreads) {
    M.isl[g] = M.last[M.par[g]];
    M.cnt[g] = 0;
  }
  __syncthreads();
  // bodies per island, ascending; constraints per island, list order
  if (t < 32) ordered_ranks(nB, M.cnt, [&](int g) { return M.isl[g]; }, [&](int g, int r) { M.loc[g] = r; });
  __syncthreads();
  for (int I = t; I < nI; I += kBuildThreads) {
    bad |= M.cnt[I] > KR_MAX_ISLAND_BODIES;
    M.bo[I] = M.cnt[I];
    M.co[I] = 0;
    M.cnt[I] = 0;
  }
  if (__syncthreads_or(bad)) { fail(KR_ERR_CAPACITY); return; }
  const int nb_all = block_scan(M.bo, nI, M.sums);
  for (int k = t; k < nC; k += kBuildThreads) {
    const int I = M.isl[cons[20 * (size_t)k]];
    M.con[k] = I;  // for now: the constraint's island
    atomicAdd(&M.co[I], 1);
  }
  if (t == 0) M.bo[nI] = nb_all;
  __syncthreads();
  for (int I = t; I < nI; I += kBuildThreads) bad |= M.co[I] > KR_MAX_ISLAND_CONSTRAINTS;
  if (__syncthreads_or(bad)) { fail(KR_ERR_CAPACITY); return; }
  const int nc_all = block_scan(M.co, nI, M.sums);
  if (t == 0) M.co[nI] = nc_all;
  __syncthreads();
  if (t < 32)
    ordered_ranks(nC, M.cnt, [&](int k) { return M.con[k]; },
                  [&](int k, int r) { M.list[M.co[M.con[k]] + r] = (unsigned short)k; });
  for (int g = t; g < nB; g += kBuildThreads) {
    const int at = M.bo[M.isl[g]] + M.loc[g];
    ib[at] = g;
    M.last[at] = -1;
    M.last_unit[at] = -1;
  }
  __syncthreads();
  for (int q = t; q < nC; q += kBuildThreads) {
    const uint32_t *c = cons + 20 * (size_t)M.list[q];
    const int b = c[1] == 0xffffffffu ? 0xff : M.loc[c[1]];
    M.con[q] = M.loc[c[0]] | (b << 8) | ((c[2] & 0xffu) == 1u ? 1 << 16 : 0);
  }
  __syncthreads();
  // per island: units and their levels (each on the first level after every
  // earlier unit sharing a body), a stable counting sort by level (a level of
  // more than 32 units takes several passes), point ranges of its bodies
  for (int I = t; I < nI; I += kBuildThreads) {
    const int co = M.co[I], nc = M.co[I + 1] - co, bo = M.bo[I], nb = M.bo[I + 1] - bo;
    int *last = M.last + bo, *last_unit = M.last_unit + bo;
    int nlv = 0, nu = 0, nul = 0;
    for (int q = co; q < co + nc; q++) {
      const int c = M.con[q], a = c & 0xff, b = (c >> 8) & 0xff, angle = c >> 16;
      int L = last[a] + 1;
      if (b != 0xff) L = max(L, last[b] + 1);
      last[a] = L;
      if (b != 0xff) last[b] = L;
      nlv = max(nlv, L + 1);
      const int u = last_unit[a], ub = b != 0xff ? last_unit[b] : u;
      if (angle && u >= 0 && ub == u && M.pin[co + u] >= 0 && M.ang[co + u] < 0 &&
          (M.con[M.pin[co + u]] & 0xffff) == (c & 0xffff)) {
        M.ang[co + u] = (short)q;
        continue;
      }
      int ul = u >= 0 ? M.level[co + u] + 1 : 0;
      if (ub >= 0) ul = max(ul, M.level[co + ub] + 1);
      M.pin[co + nu] = angle ? -1 : (short)q;
      M.ang[co + nu] = angle ? (short)q : -1;
      M.level[co + nu] = (short)ul;
      nul = max(nul, ul + 1);
      last_unit[a] = nu;
      if (b != 0xff) last_unit[b] = nu;
      nu++;
    }
    bad |= nlv > KR_MAX_LEVELS;
    // cur has nc + 1 words per island
    int *cur = M.cur + co + I, *po = pass + co + I;
    for (int L = 0; L <= nul; L++) cur[L] = 0;
    for (int u = 0; u < nu; u++) cur[M.level[co + u] + 1]++;
    int np = 0;
    po[0] = 0;
    for (int L = 0; L < nul; L++) {
      cur[L + 1] += cur[L];
      for (int s = cur[L]; s < cur[L + 1]; s += 32) po[++np] = min(s + 32, cur[L + 1]);
    }
    for (int u = 0; u < nu; u++) {
      const int p = M.pin[co + u], q = M.ang[co + u];
      units[co + cur[M.level[co + u]]++] =
          make_int4(M.con[p >= 0 ? p : q] & 0xffff, p >= 0 ? (int)M.list[p] : -1, q >= 0 ? (int)M.list[q] : -1, 0);
    }
    int pts = 0;
    for (int j = 0; j < nb; j++) {
      const int cn = (int)coll_range[nB + ib[bo + j]];
      bpt[bo + j] = make_int2(pts, cn);
      pts += cn;
    }
    bad |= pts > KR_MAX_ISLAND_COLLPTS;
    M.po[I] = pts;
    int *rec = isl + I * kIslandInts;
    rec[I_BODY_OFF] = bo;
    rec[I_NB] = nb;
    rec[I_UNIT_OFF] = co;
    rec[I_NU] = nu;
    rec[I_PASS_OFF] = co + I;
    rec[I_NPASS] = np;
  }
  if (__syncthreads_or(bad)) { fail(KR_ERR_CAPACITY); return; }
  block_scan(M.po, nI, M.sums);
  for (int I = t; I < nI; I += kBuildThreads) isl[I * kIslandInts + I_PT_OFF] = M.po[I];
  for (int g = t; g < nB; g += kBuildThreads) {
    const int I = M.isl[g], at = M.bo[I] + M.loc[g];
    const int2 r = bpt[at];
    for (int q = 0; q < r.y; q++) ipts[M.po[I] + r.x + q] = (int)coll_range[g] + q;
  }
  // rects and the culling distance, as kr_create derives them: the largest
  // half thickness and radius (an infinite or undefined one counts as no
  // bound), as the bit patterns of non-negative doubles
  if (t == 0) M.half_thick = M.r_max = 0.0;
  __syncthreads();
  auto raise = [](double *m, double v) {
    atomicMax(reinterpret_cast<unsigned long long *>(m), (unsigned long long)__double_as_longlong(v));
  };
  for (int i = t; i < nR; i += kBuildThreads) {
    const float x = rects[4 * i], y = rects[4 * i + 1], rw = rects[4 * i + 2], rh = rects[4 * i + 3];
    r4[i] = make_float4(x, y, x + rw, y + rh);
    const double ht = 0.5 * fmin(fabs((double)rw), fabs((double)rh));
    raise(&M.half_thick, isfinite(ht) ? ht : HUGE_VAL);
  }
  for (int i = t; i < nP; i += kBuildThreads) {
    const float r = __uint_as_float(coll_pts[4 * i + 3]);
    raise(&M.r_max, isfinite(r) ? fabs((double)r) : HUGE_VAL);
  }
  __syncthreads();
  if (t == 0) {
    const double cull = fmax(M.r_max, M.half_thick) + 2.0 + kr::kCullPad;
    reinterpret_cast<float *>(W)[kOffHdr + 1] = (isfinite(cull) && cull < 1e30) ? (float)cull : 1e30f;
    W[kOffHdr + 0] = nI;
    W[kOffHdr + 2] = KR_OK;
  }
}

__global__ void __launch_bounds__(32 * kWarpsPerBlock, 4) noalloc_step_kernel(StepArgs A, const int *W) {
  StepArgs B = A;
  B.nI = W[kOffHdr + 0];
  B.near_d = reinterpret_cast<const float *>(W)[kOffHdr + 1];
  if (W[kOffHdr + 2] != KR_OK) return;
  plain_step_body(B);
}

int g_noalloc_status_host = 0;
void *g_noalloc_ptr[64] = {nullptr};

}  // namespace

extern "C" int kr_step_noalloc(const kr_solver_params *params, uint32_t n_bodies, uint32_t n_constraints,
                               float *bodies, uint32_t *cons, float *forces, const float *rects,
                               uint32_t n_rects, const uint32_t *coll_pts, uint32_t n_coll_pts,
                               const uint32_t *coll_range, int32_t n_steps, void *stream) {
  if (!params || !bodies || !forces || !rects || !coll_range || (n_constraints && !cons) ||
      (n_coll_pts && !coll_pts) || n_steps < 0)
    return KR_ERR_INVALID;
  // The kernels move bodies, forces, constraints and collision points as
  // 16-byte vectors and read rects and collRange as 4-byte words; a caller's
  // pool may hand out any address, so misaligned buffers are refused here,
  // before the device is touched.
  auto misaligned = [](const void *q, uintptr_t a) { return (reinterpret_cast<uintptr_t>(q) & (a - 1)) != 0; };
  if (misaligned(bodies, 16) || misaligned(forces, 16) || (cons && misaligned(cons, 16)) ||
      (coll_pts && misaligned(coll_pts, 16)) || misaligned(rects, 4) || misaligned(coll_range, 4))
    return KR_ERR_INVALID;
  const kr_solver_params &p = *params;
  const float hf = static_cast<float>(p.h);
  if (!(p.iterations >= 1 && p.iterations <= 64) || !(p.substeps >= 1 && p.substeps <= 64) ||
      !(hf > 0.f && hf < 1.f) || n_bodies < 1 || n_rects < 1)
    return KR_ERR_INVALID;
  if (n_bodies > (uint32_t)kNaB || n_constraints > (uint32_t)kNaC || n_coll_pts > (uint32_t)kNaP ||
      n_rects > (uint32_t)kNaR)
    return KR_ERR_CAPACITY;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return KR_ERR_CUDA;
  // set-up once per device, with that device current: the device address of
  // the scratch array (its host-side name is only a stand-in)
  if (!g_noalloc_ptr[dev]) {
    void *ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) return KR_ERR_CUDA;
    g_noalloc_ptr[dev] = ptr;
  }
  int *W = static_cast<int *>(g_noalloc_ptr[dev]);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n_steps == 0) return KR_OK;
  if (cudaFuncSetAttribute(noalloc_schedule_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(BuildSmem)) != cudaSuccess)
    return KR_ERR_CUDA;
  noalloc_schedule_kernel<<<1, kBuildThreads, sizeof(BuildSmem), st>>>(W, bodies, cons, rects, coll_pts, coll_range,
                                           (int)n_bodies, (int)n_constraints, (int)n_coll_pts,
                                           (int)n_rects);
  if (cudaGetLastError() != cudaSuccess) return KR_ERR_CUDA;
  // the builder's verdict decides the return code (a 4-byte copy into static
  // host memory, which also orders this call after the builder)
  if (cudaMemcpyAsync(&g_noalloc_status_host, W + kOffHdr + 2, sizeof(int), cudaMemcpyDeviceToHost,
                      st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return KR_ERR_CUDA;
  if (g_noalloc_status_host != KR_OK) return g_noalloc_status_host;
  StepArgs A;
  A.K.h = hf;
  A.K.invH = static_cast<float>(1.0 / p.h);
  A.K.invH2 = static_cast<float>(1.0 / (p.h * p.h));
  const float nl = -static_cast<float>(p.lin_drag), na = -static_cast<float>(p.ang_drag);
  A.K.linDamp = static_cast<float>(std::exp(static_cast<double>(nl * hf)));
  A.K.angDamp = static_cast<float>(std::exp(static_cast<double>(na * hf)));
  A.K.maxSpeed = static_cast<float>(p.max_speed);
  A.K.maxAngSpeed = static_cast<float>(p.max_ang_speed);
  A.K.substeps = p.substeps;
  A.K.iterations = p.iterations;
  A.bodies = bodies;
  A.cons = cons;
  A.forces = forces;
  A.coll = reinterpret_cast<const uint4 *>(coll_pts);
  A.rects = reinterpret_cast<const float4 *>(W + kOffRects);
  A.nR = (int)n_rects;
  A.near_d = 0.f;
  A.nI = 0;
  // shared memory for the largest island the world can hold
  A.maxB = ((int)std::min<uint32_t>(n_bodies, KR_MAX_ISLAND_BODIES) + 3) & ~3;
  A.maxU = (int)std::min<uint32_t>(std::max<uint32_t>(n_constraints, 1), KR_MAX_ISLAND_CONSTRAINTS);
  A.maxP = ((int)std::min<uint32_t>(std::max<uint32_t>(n_coll_pts, 1), KR_MAX_ISLAND_COLLPTS) + 3) & ~3;
  A.T = DeviceTables{W + kOffIsl, W + kOffBodies, reinterpret_cast<const int4 *>(W + kOffUnits), W + kOffPts,
                     reinterpret_cast<const int2 *>(W + kOffBpt), W + kOffPass};
  const size_t smem = sizeof(float) * kWarpsPerBlock * (size_t)warp_smem_words(A.maxB, A.maxU, A.maxP);
  if (cudaFuncSetAttribute(noalloc_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return KR_ERR_CUDA;
  const int grid = ((int)n_bodies + kWarpsPerBlock - 1) / kWarpsPerBlock;  // islands <= bodies
  for (int s = 0; s < n_steps; s += kStepsPerLaunch) {
    A.n_steps = std::min(kStepsPerLaunch, n_steps - s);
    noalloc_step_kernel<<<grid, 32 * kWarpsPerBlock, smem, st>>>(A, W);
    if (cudaGetLastError() != cudaSuccess) return KR_ERR_CUDA;
  }
  return KR_OK;
}
