// The batched CG's per-chart state and its vector types, shared by the launch-per-step solver
// (pcg.cu) and the team kernels (team.cu).
#pragma once

#include "system.cuh"

namespace ruv {

enum : int32_t { kActive = 0, kDone = 1 };

struct ChartState {
  double rz;       // r.z of the current iterate
  double alpha;
  double beta;
  double tol_abs;  // tol * ||b|| (tol when ||b|| <= 1e-300), solver.rs:465-466
  double r_ref;    // ||r|| at the last true-residual (mixed)
  double rr;       // last ||r||^2 (FP64 true residual for mixed)
  double bnorm;
  int32_t iters;
  int32_t status;
  int32_t state;
  int32_t refresh;  // mixed: a true-residual refresh is due
  int32_t refinements;
  float alpha32;  // alpha / beta rounded once per chart for the FP32 tile kernels
  float beta32;
  float rscale;   // 1 / ||b|| as FP32 (1 when b = 0): FP32 sums of squares of r * rscale stay in range
};

template <class S, int NR>
struct V {
  S c[NR];
};
template <class S, int NR>
__device__ __forceinline__ V<S, NR> ldv(const S* p, int64_t i) {
  V<S, NR> r;
  if constexpr (NR == 2 && sizeof(S) == 8) {
    double2 t = reinterpret_cast<const double2*>(p)[i];
    r.c[0] = t.x;
    r.c[1] = t.y;
  } else if constexpr (NR == 2 && sizeof(S) == 4) {
    float2 t = reinterpret_cast<const float2*>(p)[i];
    r.c[0] = t.x;
    r.c[1] = t.y;
  } else {
    r.c[0] = p[i];
  }
  return r;
}
template <class S, int NR>
__device__ __forceinline__ void stv(S* p, int64_t i, const V<S, NR>& v) {
  if constexpr (NR == 2 && sizeof(S) == 8) {
    reinterpret_cast<double2*>(p)[i] = make_double2(v.c[0], v.c[1]);
  } else if constexpr (NR == 2 && sizeof(S) == 4) {
    reinterpret_cast<float2*>(p)[i] = make_float2(v.c[0], v.c[1]);
  } else {
    p[i] = v.c[0];
  }
}

// Double-float arithmetic: TwoSum (Knuth) and the FMA TwoProduct carry the rounding error
// of an FP32 add / multiply exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
// (Sh, Sl) += (ah + al) * (dh + dl), dropping the al * dl term (2^-48 relative).
__device__ __forceinline__ void df_fma(float ah, float al, float dh, float dl, float& Sh, float& Sl) {
  const float p = ah * dh;
  const float t = fmaf(ah, dl, fmaf(al, dh, fmaf(ah, dh, -p)));
  float sh, se;
  two_sum(Sh, p, sh, se);
  Sh = sh;
  Sl += se + t;
}
// A row's double-float value: NR hi parts then NR lo parts (one 16- / 8-byte access).
template <int NR>
struct DF {
  float h[NR], l[NR];
};
template <int NR>
__device__ __forceinline__ DF<NR> lddf(const float* p, int64_t i) {
  DF<NR> r;
  if constexpr (NR == 2) {
    const float4 t = reinterpret_cast<const float4*>(p)[i];
    r.h[0] = t.x;
    r.h[1] = t.y;
    r.l[0] = t.z;
    r.l[1] = t.w;
  } else {
    const float2 t = reinterpret_cast<const float2*>(p)[i];
    r.h[0] = t.x;
    r.l[0] = t.y;
  }
  return r;
}
template <int NR>
__device__ __forceinline__ void stdf(float* p, int64_t i, const DF<NR>& v) {
  if constexpr (NR == 2) reinterpret_cast<float4*>(p)[i] = make_float4(v.h[0], v.h[1], v.l[0], v.l[1]);
  else reinterpret_cast<float2*>(p)[i] = make_float2(v.h[0], v.l[0]);
}
__device__ __forceinline__ void split_f64(double v, float& h, float& l) {
  h = (float)v;
  l = (float)(v - (double)h);
}


}  // namespace ruv
