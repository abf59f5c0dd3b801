// Device code shared by the kernels that run a whole CG loop (team.cu, grid.cu): their scalars and
// the rows of a CSR operator.
#pragma once

#include "team.cuh"

namespace ruv {

constexpr int kTeamDirect = 64;            // rows solved by the dense inverse (amg.cu kDirect)

// 1 / d for a finite d whose reciprocal is normal: an FP32 seed of the significand and two Newton
// steps, within about an ulp.  d outside that goes to the division.
__device__ __forceinline__ double rcp64(double d) {
  const uint64_t u = (uint64_t)__double_as_longlong(d);
  const int e = (int)(u >> 52) & 0x7ff;
  if (e < 2 || e > 2044) return 1.0 / d;
  const double m = __longlong_as_double((long long)((u & 0x000fffffffffffffull) | 0x3ff0000000000000ull));
  double r = (double)(1.0f / (float)m);
  r = fma(r, fma(-m, r, 1.0), r);
  r = fma(r, fma(-m, r, 1.0), r);
  const uint64_t scale = ((uint64_t)(2046 - e) << 52) | (u & 0x8000000000000000ull);
  return r * __longlong_as_double((long long)scale);
}
// a / b from r = rcp64(b): the product and one correction by its exact remainder (the rounding of
// the division up to the last bit; a chain of three FP64 operations, where the division takes ten).
// Quotients that leave the normal range go to the division.
__device__ __forceinline__ double div_by(double a, double b, double r) {
  const double q = a * r;
  if (a == 0.0) return q;
  const int e = (int)((uint64_t)__double_as_longlong(q) >> 52) & 0x7ff;
  if (e < 64 || e > 1982) return a / b;
  return fma(fma(-q, b, a), r, q);
}
__device__ __forceinline__ double div64(double a, double b) { return div_by(a, b, rcp64(b)); }

// A sum in double-float: an unevaluated FP32 pair (48 bits).  The mixed loop's scalars are formed in
// these -- its partial sums are FP32, its vectors take alpha and beta rounded to FP32 -- because a
// dependent FP64 operation takes 64 clocks here and an FP32 one four (a reduction with its
// division: 2,000 clocks in FP64 against 700).
struct Pair {
  float h, l;
  __device__ __forceinline__ double f64() const { return (double)h + (double)l; }
};
__device__ __forceinline__ Pair pair_of(float a) { return Pair{a, 0.0f}; }
__device__ __forceinline__ Pair pair_of(double a) {
  Pair r;
  split_f64(a, r.h, r.l);
  return r;
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
  float s, e;
  two_sum(a.h, b.h, s, e);
  e += a.l + b.l;
  const float h = s + e;
  return Pair{h, e - (h - s)};
}
__device__ __forceinline__ Pair pair_div(Pair a, Pair b) {
  const float q1 = a.h / b.h;
  if (!(fabsf(q1) < 3e38f) || q1 == 0.0f) return Pair{q1, 0.0f};
  // the remainder a - q1 b to twice FP32, and its quotient
  const float p = q1 * b.h, pe = fmaf(q1, b.h, -p);
  const float q2 = ((a.h - p) - pe + (a.l - q1 * b.l)) / b.h;
  const float h = q1 + q2;
  return Pair{h, q2 - (h - q1)};
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {
  const float p = a.h * b.h;
  const float e = fmaf(a.h, b.h, -p) + (a.h * b.l + a.l * b.h);
  const float h = p + e;
  return Pair{h, e - (h - p)};
}
// What a reduction's totals and the scalars formed from them are held in.
template <class S>
struct ScalarOf {
  using type = double;
};
template <>
struct ScalarOf<float> {
  using type = Pair;
};
__device__ __forceinline__ double sc_add(double a, double b) { return a + b; }
__device__ __forceinline__ Pair sc_add(Pair a, Pair b) { return pair_add(a, b); }
__device__ __forceinline__ double sc_div(double a, double b) { return div64(a, b); }
__device__ __forceinline__ Pair sc_div(Pair a, Pair b) { return pair_div(a, b); }
__device__ __forceinline__ double sc_neg_mul(double a, double b) { return -a * b; }
__device__ __forceinline__ Pair sc_neg_mul(Pair a, Pair b) { return pair_mul(Pair{-a.h, -a.l}, b); }
__device__ __forceinline__ double sc_hi(double a) { return a; }
__device__ __forceinline__ float sc_hi(Pair a) { return a.h; }
__device__ __forceinline__ bool vanishes(double a) { return fabs(a) <= 1e-300; }
__device__ __forceinline__ bool vanishes(Pair a) { return a.h == 0.0f; }
__device__ __forceinline__ double sc_zero(double) { return 0.0; }
__device__ __forceinline__ Pair sc_zero(Pair) { return Pair{0.0f, 0.0f}; }
__device__ __forceinline__ double sc_from(double, double v) { return v; }
__device__ __forceinline__ Pair sc_from(Pair, double v) { return pair_of(v); }
__device__ __forceinline__ double sc_f64(double a) { return a; }
__device__ __forceinline__ double sc_f64(Pair a) { return a.f64(); }
__device__ __forceinline__ double sc_shfl(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ Pair sc_shfl(Pair a, int o) {
  return Pair{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)};
}
__device__ __forceinline__ unsigned long long sc_bits(double a) { return (unsigned long long)__double_as_longlong(a); }
__device__ __forceinline__ unsigned long long sc_bits(Pair a) {
  return ((unsigned long long)__float_as_uint(a.h) << 32) | __float_as_uint(a.l);
}
__device__ __forceinline__ double sc_of_bits(double, unsigned long long b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ Pair sc_of_bits(Pair, unsigned long long b) {
  return Pair{__uint_as_float((unsigned)(b >> 32)), __uint_as_float((unsigned)b)};
}
// sqrt(rr) <= norm (norm2 = square_of(norm)); an FP32 sum of squares against the FP32 square
__device__ __forceinline__ double square_of(double, double norm) {
  return norm > 1e-140 && norm < 1e140 ? norm * norm : -1.0;
}
__device__ __forceinline__ float square_of(float, double norm) {
  return norm > 1e-18 && norm < 1e18 ? (float)(norm * norm) : -1.0f;
}
template <class R>
__device__ __forceinline__ bool at_most(R rr, double norm, R norm2) {
  return norm2 > R(0) ? rr <= norm2 : sqrt((double)rr) <= norm;
}

// A CSR operator's column stream (see ColsWide, ColsNarrow, ColsRowRel).
struct Cols {
  const int32_t* c32;
  const uint16_t* c16;
  int kind;
  int32_t cb;
  __device__ __forceinline__ int32_t base(int32_t i) const { return kind == 2 ? i - kRowRelBias : cb; }
  __device__ __forceinline__ int32_t at(int32_t e, int32_t rb) const {
    return kind ? rb + (int32_t)__ldg(c16 + e) : __ldg(c32 + e);
  }
};

// sum_e val(e) get(col(e)) over the entries [lo, hi) of one row, eight in flight (a mesh Laplacian's row
// in one sweep), entry order.
template <class S, int NR, class Val, class Col, class Get>
__device__ __forceinline__ V<S, NR> entries_dot(int32_t lo, int32_t hi, Val val, Col col, Get get) {
  V<S, NR> s;
#pragma unroll
  for (int c = 0; c < NR; ++c) s.c[c] = S(0);
  for (int32_t e0 = lo; e0 < hi; e0 += 8) {
    S a[8];
    int32_t j[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in = e0 + k < hi;
      a[k] = in ? val(e0 + k) : S(0);
      j[k] = in ? col(e0 + k) : -1;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j[k] >= 0) {
        const V<S, NR> g = get(j[k]);
#pragma unroll
        for (int c = 0; c < NR; ++c) s.c[c] += a[k] * g.c[c];
      }
  }
  return s;
}

}  // namespace ruv
