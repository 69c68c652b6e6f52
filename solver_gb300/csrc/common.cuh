// Shared device/host helpers for the GB300 FFT-PEEC kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>

template <typename R>
struct alignas(2 * sizeof(R)) cx {
  R x, y;
};
using c64 = cx<double>;
using c32 = cx<float>;

template <typename R>
__host__ __device__ __forceinline__ cx<R> mk(R a, R b) {
  cx<R> r;
  r.x = a;
  r.y = b;
  return r;
}
template <typename R>
__host__ __device__ __forceinline__ cx<R> operator+(cx<R> a, cx<R> b) {
  return mk<R>(a.x + b.x, a.y + b.y);
}
template <typename R>
__host__ __device__ __forceinline__ cx<R> operator-(cx<R> a, cx<R> b) {
  return mk<R>(a.x - b.x, a.y - b.y);
}
template <typename R>
__host__ __device__ __forceinline__ cx<R> operator*(cx<R> a, cx<R> b) {
  return mk<R>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename R>
__host__ __device__ __forceinline__ cx<R> cmulc(cx<R> a, cx<R> b) {  // a * conj(b)
  return mk<R>(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
template <typename R>
__host__ __device__ __forceinline__ cx<R> cscale(cx<R> a, R s) {
  return mk<R>(a.x * s, a.y * s);
}
template <typename R>
__host__ __device__ __forceinline__ cx<R> cconj(cx<R> a) {
  return mk<R>(a.x, -a.y);
}
template <typename To, typename From>
__host__ __device__ __forceinline__ cx<To> ccast(cx<From> a) {
  return mk<To>((To)a.x, (To)a.y);
}

__host__ __device__ __forceinline__ int ilog2(int v) {
  int r = 0;
  while ((1 << r) < v) ++r;
  return r;
}
__host__ __device__ __forceinline__ int brev(int v, int bits) {
  int r = 0;
  for (int i = 0; i < bits; ++i) {
    r = (r << 1) | (v & 1);
    v >>= 1;
  }
  return r;
}

#define PEEC_CUDA_TRY(expr)                                       \
  do {                                                            \
    cudaError_t _e = (expr);                                      \
    if (_e != cudaSuccess) return peec::fail_cuda(_e, #expr, __FILE__, __LINE__); \
  } while (0)

// Float-float ("double-float") scalar: value = hi + lo with |lo| <= ulp(hi)/2, about 48
// significant bits from FP32 arithmetic. Error-free transformations (Knuth two-sum,
// Dekker fast two-sum, FMA two-product) use the _rn intrinsics so the compiler can
// neither contract nor reassociate them. Used for the refinement residual operator,
// where GB300's FP32 pipes are far faster than its FP64 ones.
struct ff {
  float hi, lo;
  ff() = default;
  __host__ __device__ constexpr ff(float h, float l) : hi(h), lo(l) {}
  __host__ __device__ ff(double d) : hi((float)d), lo((float)(d - (double)(float)d)) {}
  __host__ __device__ ff(int i) : ff((double)i) {}
  __host__ __device__ explicit operator double() const { return (double)hi + (double)lo; }
};

#ifdef __CUDA_ARCH__
#define PEEC_FADD(a, b) __fadd_rn(a, b)
#define PEEC_FSUB(a, b) __fsub_rn(a, b)
#define PEEC_FMUL(a, b) __fmul_rn(a, b)
#define PEEC_FMA(a, b, c) __fmaf_rn(a, b, c)
#else
#define PEEC_FADD(a, b) ((a) + (b))
#define PEEC_FSUB(a, b) ((a) - (b))
#define PEEC_FMUL(a, b) ((a) * (b))
#define PEEC_FMA(a, b, c) fmaf(a, b, c)
#endif

__host__ __device__ __forceinline__ ff ff_two_sum(float a, float b) {
  const float s = PEEC_FADD(a, b);
  const float bb = PEEC_FSUB(s, a);
  const float e = PEEC_FADD(PEEC_FSUB(a, PEEC_FSUB(s, bb)), PEEC_FSUB(b, bb));
  return ff(s, e);
}
__host__ __device__ __forceinline__ ff ff_fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = PEEC_FADD(a, b);
  return ff(s, PEEC_FSUB(b, PEEC_FSUB(s, a)));
}
// Sum with the low parts added in FP32 after an exact two-sum of the high parts: the
// error is within a few units of 2^-48 (|a| + |b|), which is the norm-wise accuracy
// the transforms need (their error bounds are norm-wise, not element-wise).
__host__ __device__ __forceinline__ ff operator+(ff a, ff b) {
  const ff s = ff_two_sum(a.hi, b.hi);
  return ff_fast_two_sum(s.hi, PEEC_FADD(s.lo, PEEC_FADD(a.lo, b.lo)));
}
__host__ __device__ __forceinline__ ff operator-(ff a) { return ff(-a.hi, -a.lo); }
__host__ __device__ __forceinline__ ff operator-(ff a, ff b) { return a + (-b); }
__host__ __device__ __forceinline__ ff operator*(ff a, ff b) {
  const float p = PEEC_FMUL(a.hi, b.hi);
  float e = PEEC_FMA(a.hi, b.hi, -p);
  e = PEEC_FMA(a.hi, b.lo, e);
  e = PEEC_FMA(a.lo, b.hi, e);
  return ff_fast_two_sum(p, e);
}
// Double to float-float and back by integer operations: a conversion instruction holds the FP64
// pipe as long as a double multiply (64 cycles a warp and sub-partition), and the constructor
// and cast above take four and three such instructions. Same roundings (to nearest but for ties
// of the high part, which only move half a unit between the parts); values outside the range
// handled here, and sums that leave the high part's binade, take the plain forms.
__device__ __forceinline__ ff ff_split(double d) {
  const int h = __double2hiint(d), l = __double2loint(d);
  const int e = (h >> 20) & 0x7ff;
  if (e < 950 || e >= 1150) return d == 0.0 ? ff(0.f, 0.f) : ff(d);
  const int r = (int)((unsigned)l << 3) >> 3;  // the low 29 bits, signed
  const unsigned m = (((unsigned)(h & 0x7fffffff) - (896u << 20)) << 3 | (unsigned)l >> 29) +
                     (r < 0 ? 1u : 0u);
  const unsigned sg = (unsigned)h & 0x80000000u;
  const float lo = __fmul_rn((float)r, __uint_as_float((unsigned)(e - 948) << 23));
  return ff(__uint_as_float(m | sg), __uint_as_float(__float_as_uint(lo) ^ sg));
}
__device__ __forceinline__ double ff_join(ff a) {
  const unsigned h = __float_as_uint(a.hi);
  const int e = (int)(h >> 23) & 0xff;
  if (e >= 60 && e < 255) {
    // the low part in units of the double's last place
    const float u = __fmul_rn(a.lo, __uint_as_float((unsigned)(306 - e) << 23));
    int r = __float2int_rn(u);
    if ((int)h < 0) r = -r;
    if (fabsf(u) <= 268435456.f && ((h & 0x7fffffu) != 0 || r >= 0)) {
      const long long b = (((long long)(h & 0x7fffffffu) + (896ll << 23)) << 29) + r;
      return __longlong_as_double(b | (long long)((unsigned long long)(h & 0x80000000u) << 32));
    }
  }
  return (double)a;
}
using cff = cx<ff>;

// Sums of float-float values with the precision of an FP64 sum of them, in FP32 instructions: the
// high and the low parts are added exactly, what is below them gathers in a third part. An
// addition is 21 FP32 instructions (an FP64 one holds its pipe as long as 64 of them).
struct ffsum {
  float hi, lo, c;
};
__host__ __device__ __forceinline__ ffsum ffsum_of(ff a) { return ffsum{a.hi, a.lo, 0.f}; }
__host__ __device__ __forceinline__ ffsum operator+(const ffsum& a, const ffsum& b) {
  const ff s = ff_two_sum(a.hi, b.hi), t = ff_two_sum(a.lo, b.lo), u = ff_two_sum(s.lo, t.hi);
  return ffsum{s.hi, u.hi, PEEC_FADD(PEEC_FADD(a.c, b.c), PEEC_FADD(t.lo, u.lo))};
}
__host__ __device__ __forceinline__ double ffsum_double(const ffsum& a) {
  const ff s = ff_two_sum(a.hi, a.lo), t = ff_two_sum(s.lo, a.c);
#ifdef __CUDA_ARCH__
  // as ff_join, with the third part in units of the double's last place
  const unsigned h = __float_as_uint(s.hi);
  const int e = (int)(h >> 23) & 0xff;
  if (e >= 60 && e < 255) {
    const float unit = __uint_as_float((unsigned)(306 - e) << 23);
    const float u = __fmul_rn(t.hi, unit);
    int r = __float2int_rn(u) + __float2int_rn(__fmul_rn(t.lo, unit));
    if ((int)h < 0) r = -r;
    if (fabsf(u) <= 268435456.f && ((h & 0x7fffffu) != 0 || r >= 0)) {
      const long long b = (((long long)(h & 0x7fffffffu) + (896ll << 23)) << 29) + r;
      return __longlong_as_double(b | (long long)((unsigned long long)(h & 0x80000000u) << 32));
    }
  }
#endif
  return (double)s.hi + ((double)t.hi + (double)t.lo);
}

// acc += u x and acc += conj(u) x, products and sums one after the other: in float-float, 72
// operations. Adding the high parts of both products and of the sum exactly and all error terms
// before one normalisation takes 54, but a chain of 8 to 512 such sums rounds 1.5 times worse.
template <typename A>
__host__ __device__ __forceinline__ void cmac(cx<A>& acc, const cx<A>& u, const cx<A>& x) {
  acc.x = acc.x + (u.x * x.x - u.y * x.y);
  acc.y = acc.y + (u.x * x.y + u.y * x.x);
}
template <typename A>
__host__ __device__ __forceinline__ void cmac_conj(cx<A>& acc, const cx<A>& u, const cx<A>& x) {
  acc.x = acc.x + (u.x * x.x + u.y * x.y);
  acc.y = acc.y + (u.x * x.y - u.y * x.x);
}
