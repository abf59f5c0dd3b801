// Device code of the kernels that run a whole CG loop (team.cu): their scalars and the rows of a CSR
// operator.
#pragma once

#include "fp64rn.cuh"
#include "team.cuh"

namespace ruv {

constexpr int kTeamDirect = 64;            // rows solved by the dense inverse (amg.cu kDirect)

// sqrt(rr) <= norm, by its square (norm2 = square_of(norm)) where that is in range
__device__ __forceinline__ double square_of(double norm) { return norm > 1e-140 && norm < 1e140 ? norm * norm : -1.0; }
__device__ __forceinline__ bool at_most(double rr, double norm, double norm2) {
  return norm2 > 0.0 ? rr <= norm2 : sqrt(rr) <= norm;
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
