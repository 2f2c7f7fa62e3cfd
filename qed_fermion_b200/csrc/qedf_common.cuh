// Common device helpers for the qed_fermion B200 kernels.
//
// Complex numbers are stored interleaved (re, im), the layout of torch
// complex64 / complex128, so vectors are passed as plain float / double
// pointers of twice the length.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/qedf.h"

namespace qedf {

// 8-byte (complex64) / 16-byte (complex128) alignment, so that one complex
// moves with one vector access
template <typename R>
struct alignas(2 * sizeof(R)) Cx {
  R re, im;
};

template <typename R>
__host__ __device__ __forceinline__ Cx<R> mk(R a, R b) {
  Cx<R> z;
  z.re = a;
  z.im = b;
  return z;
}
template <typename R>
__device__ __forceinline__ Cx<R> operator+(Cx<R> a, Cx<R> b) { return mk<R>(a.re + b.re, a.im + b.im); }
template <typename R>
__device__ __forceinline__ Cx<R> operator-(Cx<R> a, Cx<R> b) { return mk<R>(a.re - b.re, a.im - b.im); }
template <typename R>
__device__ __forceinline__ Cx<R> operator*(R s, Cx<R> a) { return mk<R>(s * a.re, s * a.im); }
template <typename R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) {
  return mk<R>(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
// conj(a) * b
template <typename R>
__device__ __forceinline__ Cx<R> cjmul(Cx<R> a, Cx<R> b) {
  return mk<R>(a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re);
}
// a + m * b
template <typename R>
__device__ __forceinline__ Cx<R> cfma(Cx<R> m, Cx<R> b, Cx<R> a) {
  Cx<R> z;
  z.re = fma(m.re, b.re, fma(-m.im, b.im, a.re));
  z.im = fma(m.re, b.im, fma(m.im, b.re, a.im));
  return z;
}
// a + conj(m) * b
template <typename R>
__device__ __forceinline__ Cx<R> cjfma(Cx<R> m, Cx<R> b, Cx<R> a) {
  Cx<R> z;
  z.re = fma(m.re, b.re, fma(m.im, b.im, a.re));
  z.im = fma(m.re, b.im, fma(-m.im, b.re, a.im));
  return z;
}
template <typename R>
__device__ __forceinline__ Cx<R> cneg(Cx<R> a) { return mk<R>(-a.re, -a.im); }

// e^{i x} scaled by t.  Single precision: the argument is first reduced to
// [-pi, pi] (two-constant Cody-Waite reduction with 2*pi split into its
// float value and the remainder), then the hardware approximations
// __sinf/__cosf are used, whose maximum absolute error on [-pi, pi] is
// documented as 2^-21.41 (sin) and 2^-21.19 (cos).  The phase always enters
// multiplied by tanh(dtau/2) <= tanh(dtau), so its contribution to an
// operator application is below 1e-7 relative for dtau <= 0.1.
__device__ __forceinline__ Cx<float> tphase(float x, float t) {
  const float k = rintf(x * 0.15915494309189535f);
  float r = fmaf(-k, 6.28318548202514648f, x);
  r = fmaf(-k, -1.7484556000744487e-07f, r);
  float s, c;
  __sincosf(r, &s, &c);
  return mk<float>(t * c, t * s);
}
// Double precision: CUDA's sincos().
__device__ __forceinline__ Cx<double> tphase(double x, double t) {
  double s, c;
  sincos(x, &s, &c);
  return mk<double>(t * c, t * s);
}

// Vector loads/stores of two consecutive complex numbers (16 B for complex64,
// 32 B for complex128).  Addresses are 16-byte aligned by construction: the
// first site of each pair has an even x and L is even.
__device__ __forceinline__ void ld2(const float* p, Cx<float>& a, Cx<float>& b) {
  float4 q = __ldg(reinterpret_cast<const float4*>(p));
  a = mk<float>(q.x, q.y);
  b = mk<float>(q.z, q.w);
}
__device__ __forceinline__ void ld2(const double* p, Cx<double>& a, Cx<double>& b) {
  double2 q0 = __ldg(reinterpret_cast<const double2*>(p));
  double2 q1 = __ldg(reinterpret_cast<const double2*>(p) + 1);
  a = mk<double>(q0.x, q0.y);
  b = mk<double>(q1.x, q1.y);
}
// plain (coherent) loads for buffers written earlier in the same kernel
__device__ __forceinline__ void ld2c(const float* p, Cx<float>& a, Cx<float>& b) {
  float4 q = *reinterpret_cast<const float4*>(p);
  a = mk<float>(q.x, q.y);
  b = mk<float>(q.z, q.w);
}
__device__ __forceinline__ void ld2c(const double* p, Cx<double>& a, Cx<double>& b) {
  double2 q0 = *reinterpret_cast<const double2*>(p);
  double2 q1 = *(reinterpret_cast<const double2*>(p) + 1);
  a = mk<double>(q0.x, q0.y);
  b = mk<double>(q1.x, q1.y);
}
__device__ __forceinline__ void st2(float* p, Cx<float> a, Cx<float> b) {
  *reinterpret_cast<float4*>(p) = make_float4(a.re, a.im, b.re, b.im);
}
__device__ __forceinline__ void st2(double* p, Cx<double> a, Cx<double> b) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a.re, a.im);
  reinterpret_cast<double2*>(p)[1] = make_double2(b.re, b.im);
}
// Storage of single-precision iteration vectors: float (complex64) or bf16
// pairs (4 bytes per complex number, the PCG's BF16 storage option for its
// search direction and preconditioned residual).
// ld2s / st2s move two consecutive complex numbers (16 B as float, 8 B as
// bf16); arithmetic stays in float.  round_st returns the value the storage
// keeps (round to nearest even for bf16), so that values kept in registers
// equal the stored ones.
using bf16 = __nv_bfloat16;
__device__ __forceinline__ void ld2s(const float* p, Cx<float>& a, Cx<float>& b) { ld2c(p, a, b); }
__device__ __forceinline__ void ld2s(const bf16* p, Cx<float>& a, Cx<float>& b) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.y));
  a = mk<float>(lo.x, lo.y);
  b = mk<float>(hi.x, hi.y);
}
__device__ __forceinline__ void ld2s(const double* p, Cx<double>& a, Cx<double>& b) { ld2c(p, a, b); }
__device__ __forceinline__ void st2s(float* p, Cx<float> a, Cx<float> b) { st2(p, a, b); }
__device__ __forceinline__ void st2s(double* p, Cx<double> a, Cx<double> b) { st2(p, a, b); }
__device__ __forceinline__ void st2s(bf16* p, Cx<float> a, Cx<float> b) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a.re, a.im);
  const __nv_bfloat162 hi = __floats2bfloat162_rn(b.re, b.im);
  uint2 q;
  q.x = *reinterpret_cast<const unsigned*>(&lo);
  q.y = *reinterpret_cast<const unsigned*>(&hi);
  *reinterpret_cast<uint2*>(p) = q;
}
template <typename S, typename R>
__device__ __forceinline__ Cx<R> round_st(Cx<R> v) {
  if constexpr (std::is_same<S, bf16>::value) {
    const float2 f = __bfloat1622float2(__floats2bfloat162_rn(v.re, v.im));
    return mk<R>(f.x, f.y);
  } else {
    return v;
  }
}

// Scaled fp16 storage (the PCG's F16 option): a vector is kept as fp16 pairs
// of v / sc, with sc a power of two chosen per vector from its norm, so the
// stored values sit in fp16's range whatever the residual's size and keep its
// 11-bit significand.  Scaling by a power of two is exact, so sc * (stored)
// is exactly the value the registers hold after round_st.  The overloads for
// the other storage types ignore the scale.
__device__ __forceinline__ void ld2s(const __half* p, Cx<float>& a, Cx<float>& b, float sc) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
  const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
  a = mk<float>(lo.x * sc, lo.y * sc);
  b = mk<float>(hi.x * sc, hi.y * sc);
}
__device__ __forceinline__ void st2s(__half* p, Cx<float> a, Cx<float> b, float inv) {
  const __half2 lo = __floats2half2_rn(a.re * inv, a.im * inv);
  const __half2 hi = __floats2half2_rn(b.re * inv, b.im * inv);
  uint2 q;
  q.x = *reinterpret_cast<const unsigned*>(&lo);
  q.y = *reinterpret_cast<const unsigned*>(&hi);
  *reinterpret_cast<uint2*>(p) = q;
}
template <typename S, typename R>
__device__ __forceinline__ void ld2s(const S* p, Cx<R>& a, Cx<R>& b, R) { ld2s(p, a, b); }
template <typename S, typename R>
__device__ __forceinline__ void st2s(S* p, Cx<R> a, Cx<R> b, R) { st2s(p, a, b); }
template <typename S, typename R>
__device__ __forceinline__ Cx<R> round_st(Cx<R> v, R sc, R inv) {
  if constexpr (std::is_same<S, __half>::value) {
    const float2 f = __half22float2(__floats2half2_rn(v.re * inv, v.im * inv));
    return mk<R>(f.x * sc, f.y * sc);
  } else {
    return round_st<S>(v);
  }
}
// the power-of-two scale of a vector with squared norm nn: about its norm
// / 1024, so entries of vectors of 10^3-10^7 sites stay well inside fp16's
// normal range; 1 for a zero or non-finite norm
__device__ __forceinline__ float st_scale(double nn) {
  if (!(nn > 0.0) || !isfinite(nn)) return 1.0f;
  int e;
  frexp(nn, &e);                         // nn in [2^(e-1), 2^e)
  int es = ((e - 1) >> 1) - 10;          // floor(log2 |v|) - 10
  es = es < -120 ? -120 : (es > 120 ? 120 : es);
  return ldexpf(1.0f, es);
}

// four reals (angles or forces of two sites, both components)
__device__ __forceinline__ void ld4(const float* p, float (&a)[4]) {
  float4 q = __ldg(reinterpret_cast<const float4*>(p));
  a[0] = q.x; a[1] = q.y; a[2] = q.z; a[3] = q.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&a)[4]) {
  double2 q0 = __ldg(reinterpret_cast<const double2*>(p));
  double2 q1 = __ldg(reinterpret_cast<const double2*>(p) + 1);
  a[0] = q0.x; a[1] = q0.y; a[2] = q1.x; a[3] = q1.y;
}
__device__ __forceinline__ void st4(float* p, const float (&a)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1], a[2], a[3]);
}
__device__ __forceinline__ void st4(double* p, const double (&a)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a[0], a[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(a[2], a[3]);
}

// Asynchronous 16-byte copies global -> shared, cached in L2 only (data that
// other SMs wrote before a grid barrier is seen).  Both addresses are 16-byte
// aligned.  cp_async_wait<N>: at most the N most recent groups still pending.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
// the same with an L2 policy: evict first, for data not read again before much
// else has passed through L2
__device__ __forceinline__ unsigned long long evict_first_policy() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, unsigned long long policy) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "l"(policy) : "memory");
}
__device__ __forceinline__ void st2_first(float* p, Cx<float> a, Cx<float> b) {
  __stcs(reinterpret_cast<float4*>(p), make_float4(a.re, a.im, b.re, b.im));
}
__device__ __forceinline__ void st2_first(double* p, Cx<double> a, Cx<double> b) {
  __stcs(reinterpret_cast<double2*>(p), make_double2(a.re, a.im));
  __stcs(reinterpret_cast<double2*>(p) + 1, make_double2(b.re, b.im));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Coefficients of the checkerboard factors F_g = c_g (I + t_g K_g):
// g1 uses cosh/tanh(dtau), g2..g4 cosh/tanh(dtau/2); Cb = c1 c2^2 c3^2 c4^2
// is the scalar that B = F4 F3 F2 F1 F2 F3 F4 carries in front of the
// product of the unscaled factors.
struct FactorCoeffs {
  double c1, ch, t1, th, Cb;
};

inline FactorCoeffs factor_coeffs(double dtau) {
  FactorCoeffs f;
  f.c1 = cosh(dtau);
  f.ch = cosh(dtau / 2);
  f.t1 = tanh(dtau);
  f.th = tanh(dtau / 2);
  f.Cb = f.c1 * f.ch * f.ch * f.ch * f.ch * f.ch * f.ch;
  return f;
}

}  // namespace qedf
