// Shared macros and small helpers for the TACE sm_100a kernels.
//
// The arithmetic helpers are plain C++ templates marked TACE_HD so the same
// code runs inside the CUDA kernels and, compiled by g++, inside the CPU unit
// tests of the generated contraction code.
#pragma once
#include <cmath>
#include <cstdint>

#if defined(__CUDACC__)
#define TACE_HD __host__ __device__
#define TACE_D __device__
#define TACE_INLINE __forceinline__
#define TACE_CONST static __device__ const
#else
#define TACE_HD
#define TACE_D
#define TACE_INLINE inline
#define TACE_CONST static const
#ifndef __restrict__
#define __restrict__
#endif
#endif

namespace tace {

// Four consecutive table entries; under nvcc one (fp32) or two (fp64) 16-byte loads, p 16-byte aligned.
#if defined(__CUDACC__)
TACE_HD TACE_INLINE void ld4(const float* p, float& a, float& b, float& c, float& d) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = v.x; b = v.y; c = v.z; d = v.w;
}
TACE_HD TACE_INLINE void ld4(const double* p, double& a, double& b, double& c, double& d) {
  const double2 u = *reinterpret_cast<const double2*>(p), v = *reinterpret_cast<const double2*>(p + 2);
  a = u.x; b = u.y; c = v.x; d = v.y;
}
#else
template <typename T>
inline void ld4(const T* p, T& a, T& b, T& c, T& d) { a = p[0]; b = p[1]; c = p[2]; d = p[3]; }
#endif

// Four consecutive entries written, the counterpart of ld4.
TACE_HD TACE_INLINE void st4(float* p, float a, float b, float c, float d) {
#if defined(__CUDACC__)
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
#else
  p[0] = a; p[1] = b; p[2] = c; p[3] = d;
#endif
}

// A pair of fp32 values (two channels of one thread) and the packed arithmetic on it: one instruction per pair, each half
// rounded as the scalar operation would be.  The packed FMA occupies the FMA pipe for as long as two scalar ones but takes
// one issue slot, and its scalar operand is broadcast without a move, which is what the contraction kernels need: they are
// bound by FP32 work, and address arithmetic, loads and shared-memory reads fit into the freed slots.
struct F2 { float x, y; };
#if defined(__CUDA_ARCH__)
TACE_D TACE_INLINE unsigned long long f2_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
TACE_D TACE_INLINE F2 f2_unpack(unsigned long long r) {
  F2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
  return v;
}
#endif
TACE_HD TACE_INLINE F2 fma2(F2 a, F2 b, F2 c) {
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)), "l"(f2_pack(c.x, c.y)));
  return f2_unpack(r);
#else
  return F2{a.x * b.x + c.x, a.y * b.y + c.y};
#endif
}
TACE_HD TACE_INLINE F2 mul2(F2 a, F2 b) {
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)));
  return f2_unpack(r);
#else
  return F2{a.x * b.x, a.y * b.y};
#endif
}
TACE_HD TACE_INLINE F2 fma2s(float s, F2 b, F2 c) { return fma2(F2{s, s}, b, c); }
TACE_HD TACE_INLINE F2 mul2s(float s, F2 b) { return mul2(F2{s, s}, b); }
// sum of products over the 2 NV channels of a thread
template <int NV>
TACE_HD TACE_INLINE float dot2(const F2 (&a)[NV], const F2 (&b)[NV]) {
  float r = a[0].x * b[0].x;
  r += a[0].y * b[0].y;
#pragma unroll
  for (int v = 1; v < NV; ++v) {
    r += a[v].x * b[v].x;
    r += a[v].y * b[v].y;
  }
  return r;
}

// Path weights of a generated backward pass held in arrays: get<p>() reads w[p], put<p>(v) stores dE/dw_p.
template <typename T>
struct TpArrayWeights {
  const T* w;
  T* dw;
  template <int P> TACE_HD TACE_INLINE T get() const { return w[P]; }
  template <int P> TACE_HD TACE_INLINE void put(T v) { dw[P] = v; }
};

template <typename T>
TACE_HD TACE_INLINE T sigmoid_(T x) { return T(1) / (T(1) + exp(-x)); }
template <>
TACE_HD TACE_INLINE float sigmoid_<float>(float x) { return 1.0f / (1.0f + expf(-x)); }

template <typename T>
TACE_HD TACE_INLINE T silu_(T x) { return x * sigmoid_(x); }

// d/dx [x * sigmoid(x)] = s * (1 + x * (1 - s))
template <typename T>
TACE_HD TACE_INLINE T silu_grad_(T x) {
  const T s = sigmoid_(x);
  return s * (T(1) + x * (T(1) - s));
}

}  // namespace tace
