// cuda_on_host.h -- enough of CUDA C++ for g++ to compile csrc/kr_solver.cuh,
// so that tests can run the device functions on the CPU, one lane at a time
// (kr::Lanes<1>).  The arithmetic is the device's (separately rounded f32,
// fmaf, f64) except for the hardware's reciprocal estimate, which is 1 / b
// rounded here.  g_rect_loads counts the loads of read-only 16-byte records:
// the rects a collision pass looked at.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#define __restrict__

struct float2 { float x, y; };
struct float3 { float x, y, z; };
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float3 make_float3(float x, float y, float z) { return {x, y, z}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }

inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline int __float_as_int(float f) { int i; std::memcpy(&i, &f, 4); return i; }
inline unsigned __float_as_uint(float f) { unsigned i; std::memcpy(&i, &f, 4); return i; }
inline float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
inline float __uint_as_float(unsigned i) { float f; std::memcpy(&f, &i, 4); return f; }
inline int __float2int_rn(float f) { return (int)std::lrintf(f); }
inline int __popc(unsigned m) { return __builtin_popcount(m); }
inline int __ffs(unsigned m) { return __builtin_ffs((int)m); }
using std::min;

static long g_rect_loads = 0;
inline float4 __ldg(const float4 *p) { g_rect_loads++; return *p; }
inline double2 __ldg(const double2 *p) { return *p; }

inline void __syncwarp(unsigned) {}
inline unsigned __ballot_sync(unsigned, bool p) { return p ? 1u : 0u; }
inline float __shfl_xor_sync(unsigned, float v, int, int) { return v; }
struct { unsigned x = 0; } static threadIdx;
struct { unsigned x = 1; } static blockDim;

// rcp.approx.ftz.f32 of kr::recip, the one asm statement of the header
#define asm(...) y = 1.f / b
#include "kr_solver.cuh"
#undef asm
