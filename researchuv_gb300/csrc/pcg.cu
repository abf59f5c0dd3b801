// Batched preconditioned conjugate gradients over the packed block-diagonal operator
// (every chart of a mesh in one launch sequence, each chart with its own scalars,
// convergence test and status) — the sm_103a replacement for the reference's host-driven
// single-system loop (gpu/src/solver.rs:284-565) and its kernels (gpu/src/kernels.cu:7-75).
//
// Work decomposition: rows are cut into tiles that never span two charts; one CTA owns a
// tile.  A tile-level kernel writes one partial per reduction; a chart-level kernel (one
// CTA per chart) combines its chart's partials in tile order, so every reduction is
// deterministic and no host round trip happens inside an iteration.  Charts that are done
// exit at the top of every kernel.  One iteration is captured once as a CUDA graph and
// replayed; the host reads the count of active charts every `kCheckEvery` iterations.
//
// SpMV: CSR-vector with `LPR` lanes per row (sub-warp per row, chosen from the row-length
// profile), coalesced 32-bit value/column loads across the lanes, (u, v) pairs moved as one
// 64-bit (FP32) / 128-bit (FP64) vector, shuffle reduction inside the sub-warp, and the
// p.q product fused into the same pass.
//
// Precision: RUV_PREC_FP64 runs the reference's recurrence in FP64.  RUV_PREC_MIXED runs
// the SpMV, preconditioner and CG recurrence in FP32 and keeps an extended-precision
// solution accumulator and true residual r = b - A x, recomputed per chart whenever the
// FP32 residual has dropped by `kDelta` (1000x) since the last true residual ("reliable
// updates"); convergence is decided on the true residual only.  The extended precision is
// double-float (a value is an unevaluated FP32 pair hi + lo, ~48 significant bits, FP32
// instructions only: GB300's FP64 pipe is a small fraction of its FP32 rate).  The true
// residual is formed as r_i = b_i - rs_i x_i - sum_j a_ij (x_j - x_i), rs_i the FP64 row
// sum: for a Laplacian with eliminated pins rs_i is zero away from the pins, so the
// products are of the small differences x_j - x_i rather than of x itself and the
// cancellation in b - A x costs no more than the FP64 product does.
#include "pcg.cuh"
#include "team.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>

namespace ruv {
namespace {

constexpr int kTileThreads = 256;
constexpr int kChartThreads = 128;
constexpr int kCheckEvery = 16;
// refresh after a 1000x drop of the FP32 residual: the FP32 recurrence then drifts from the
// true residual by about 1e-7 x 1e3 relative, far inside CG's tolerance of an inexact residual,
// and the solve needs fewer double-float refreshes (4096 disks, AMG-SA: the same iterations,
// PCG 92.2 -> 91.1 ms against 100x)
constexpr double kDelta = 0.001;
inline double refresh_delta() {
  const char* e = std::getenv("RUV_REFRESH_DELTA");
  return e ? std::atof(e) : kDelta;
}

struct Tiles {
  const int64_t* tab;      // [begin, end) pairs
  const int32_t* chart;    // chart of each tile
  const int64_t* chart_tile;
  int64_t n;
  // bulk-copy SpMV (k_spmv_tma): the largest tile's rows and nonzeros (0: not set up), the
  // flag a timed-out staging wait sets, and the wait's iteration limit
  int64_t max_rows = 0, max_nnz = 0;
  int* err = nullptr;
  int64_t spin_limit = 0;
};

// ---------------------------------------------------------------- chart steps
// What follows a tile kernel's partial sums, once per chart: alpha, beta, convergence.  The last of a
// chart's tiles to arrive does it (every tile's sum is in global memory by then), combining the
// partials in tile order as k_chart_step does -- the same bits whichever tile is last,
// without a kernel of its own between the tile kernels (4 to 9 us each, five an iteration).
enum : int { kStepAlpha, kStepBeta, kStepBetaMixed, kStepAfterRefresh, kStepCheck64, kStepRz0, kStepBetaPc };
struct ChartStep {
  int kind = kStepAlpha;
  int precond_none = 0;  // rz is r.r
  int separate = 0;      // the preconditioner is applied by its own launches: beta comes after it
  int flexible = 0;
  int64_t max_iter = 0;
  double delta = 0.0;
  ChartState* st = nullptr;
  int* n_active = nullptr;
  int32_t* done = nullptr;  // the separate preconditioner's mask
  int32_t* arrived = nullptr;  // tiles of each chart that have their sums in place (zero between kernels)
};

__device__ __forceinline__ void chart_over(ChartState& s, const ChartStep& F, int64_t c, int status) {
  s.status = status;
  s.state = kDone;
  if (F.done) F.done[c] = 1;
  atomicSub(F.n_active, 1);
}

// One lane: the step from the chart's sums v.
__device__ __forceinline__ void chart_step(const ChartStep& F, int64_t c, double v0, double v1) {
  ChartState& s = F.st[c];
  auto plain_beta = [&](double rznew) {
    s.beta = rznew / s.rz;
    s.beta32 = (float)s.beta;
    s.rz = rznew;
  };
  switch (F.kind) {
    case kStepAlpha:
      if (fabs(v0) <= 1e-300 || !isfinite(v0)) return chart_over(s, F, c, RUV_ERR_BREAKDOWN);  // solver.rs:505-508
      s.alpha = s.rz / v0;
      s.alpha32 = (float)s.alpha;
      break;
    case kStepBeta:  // FP64: convergence on the recurrence residual (solver.rs:518-522), then beta
      s.iters += 1;
      s.rr = v0;
      if (sqrt(v0) <= s.tol_abs) return chart_over(s, F, c, RUV_OK);
      if (s.iters >= F.max_iter) return chart_over(s, F, c, RUV_ERR_NOT_CONVERGED);
      plain_beta(F.precond_none ? v0 : v1);
      break;
    case kStepCheck64:  // the same with a separate preconditioner
      s.iters += 1;
      s.rr = v0;
      if (sqrt(v0) <= s.tol_abs) return chart_over(s, F, c, RUV_OK);
      if (!isfinite(v0)) return chart_over(s, F, c, RUV_ERR_BREAKDOWN);
      if (s.iters >= F.max_iter) return chart_over(s, F, c, RUV_ERR_NOT_CONVERGED);
      break;
    case kStepBetaMixed: {  // mixed: the FP32 residual only schedules true-residual refreshes
      s.iters += 1;
      const double rn = sqrt(v0);
      if (rn <= F.delta * s.r_ref || rn <= s.tol_abs || !isfinite(rn) || s.iters >= F.max_iter) {
        s.refresh = 1;  // beta is formed after the refresh, from the true residual
      } else {
        s.refresh = 0;
        if (!F.separate) plain_beta(F.precond_none ? v0 : v1);
      }
      break;
    }
    case kStepAfterRefresh: {
      s.refinements += 1;
      s.rr = v0;
      const double rn = sqrt(v0);
      if (rn <= s.tol_abs) return chart_over(s, F, c, RUV_OK);
      if (!isfinite(rn)) return chart_over(s, F, c, RUV_ERR_BREAKDOWN);
      if (s.iters >= F.max_iter) return chart_over(s, F, c, RUV_ERR_NOT_CONVERGED);
      s.r_ref = rn;
      if (F.separate) {
        s.refresh = 2;  // refreshed: beta is the plain Fletcher-Reeves ratio
        break;
      }
      plain_beta(F.precond_none ? v0 : v1);
      s.refresh = 0;
      break;
    }
    case kStepRz0:
      s.rz = v0;
      break;
    case kStepBetaPc: {
      // after a separate apply: flexible (Polak-Ribiere, as the reference's FCG for AMG,
      // solver.rs:474-481, :526-539) using r_new - r_old = -alpha q, or Fletcher-Reeves right
      // after a true-residual refresh (r jumped)
      double beta = (F.flexible && s.refresh != 2) ? (-s.alpha * v1) / s.rz : v0 / s.rz;
      if (!isfinite(beta)) beta = 0.0;
      s.beta = beta;
      s.beta32 = (float)beta;
      s.rz = v0;
      s.refresh = 0;
      break;
    }
    default: break;
  }
}

// A tile's end: its sums v (thread 0's) into part, and the chart's step by the last tile; or (NoStep, a kernel
// of its own follows) the sums alone.
struct NoStep {};
template <int LPR, int U>
constexpr bool steps_built() {
  return (LPR <= 2 && U == 2) || (LPR == 8 && U == 4) || LPR >= 16;
}
template <int NV>
__device__ __forceinline__ void tile_end(const Tiles&, const NoStep&, int64_t t, int32_t, const double (&v)[NV],
                                         double* part) {
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) part[NV * t + k] = v[k];
}
template <int NV>
__device__ __forceinline__ void tile_end(const Tiles& T, const ChartStep& F, int64_t t, int32_t ch, const double (&v)[NV],
                                         double* part) {
  tile_end<NV>(T, NoStep(), t, ch, v, part);
  const int64_t t0 = T.chart_tile[ch], n = T.chart_tile[ch + 1] - t0;
  if (n == 1) {
    if (threadIdx.x == 0) chart_step(F, ch, v[0], NV > 1 ? v[NV - 1] : 0.0);
    return;
  }
  __shared__ int last;
  __shared__ double sh[NV * 32];
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&F.arrived[ch], 1) == (int)n - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double w[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) w[k] = 0.0;
  if (threadIdx.x < kChartThreads)
    for (int64_t q = t0 + threadIdx.x; q < t0 + n; q += kChartThreads)
#pragma unroll
      for (int k = 0; k < NV; ++k) w[k] += __ldcg(part + NV * q + k);
  block_sum_first<NV>(w, sh);
  if (threadIdx.x == 0) {
    F.arrived[ch] = 0;
    chart_step(F, ch, w[0], NV > 1 ? w[NV - 1] : 0.0);
  }
}

// ---------------------------------------------------------------- tile kernels
// Accumulator type of the per-element loops: float in the FP32 solver (GB300's FP64 pipe is
// a small fraction of its FP32 rate, so FP64 appears only per tile and per chart), double in
// the FP64 solver.

// Inverse diagonal (Jacobi) once per solve: dinv in the solver's precision; zero diagonals
// are counted so the chart can report a breakdown (precond.rs:595-611).
template <class S>
__global__ void __launch_bounds__(kTileThreads) k_dinv(int64_t n, const double* __restrict__ diag, S* __restrict__ dinv) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dinv[i] = diag[i] == 0.0 ? S(0) : S(1) / (S)diag[i];
}

// Initial state: x = 0, r = b, z = M^-1 r, p = z.  Partials (FP64, once per solve): b.b, r.z,
// #zero diagonals.
// Mixed precision also: the double-float solution xdf = 0 and right-hand side bdf = b.
template <class S, int NR>
__global__ void __launch_bounds__(kTileThreads) k_init(Tiles T, const double* __restrict__ b, const double* __restrict__ diag,
                                                       const S* __restrict__ dinv, int use_jacobi, double* __restrict__ x64,
                                                       S* __restrict__ xs, S* __restrict__ r, S* __restrict__ z,
                                                       S* __restrict__ p, double* __restrict__ part,
                                                       float* __restrict__ xdf, float* __restrict__ bdf) {
  __shared__ double sh[3 * 32];
  int64_t t = blockIdx.x;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int64_t i = T.tab[2 * t] + threadIdx.x; i < T.tab[2 * t + 1]; i += blockDim.x) {
    V<double, NR> bv = ldv<double, NR>(b, i);
    V<S, NR> rv, zv, zero;
    if (diag[i] == 0.0) acc[2] += 1.0;
    const S di = use_jacobi ? dinv[i] : S(1);
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      rv.c[k] = (S)bv.c[k];
      zv.c[k] = rv.c[k] * di;
      zero.c[k] = (S)0;
      acc[0] += bv.c[k] * bv.c[k];
      acc[1] += (double)rv.c[k] * (double)zv.c[k];
    }
    V<double, NR> z64;
#pragma unroll
    for (int k = 0; k < NR; ++k) z64.c[k] = 0.0;
    stv<double, NR>(x64, i, z64);
    if (xs) stv<S, NR>(xs, i, zero);
    if (xdf) {
      DF<NR> xz, bd;
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        xz.h[k] = xz.l[k] = 0.0f;
        split_f64(bv.c[k], bd.h[k], bd.l[k]);
      }
      stdf<NR>(xdf, i, xz);
      stdf<NR>(bdf, i, bd);
    }
    stv<S, NR>(r, i, rv);
    stv<S, NR>(z, i, zv);
    stv<S, NR>(p, i, zv);
  }
  block_sum<3>(acc, sh);
  if (threadIdx.x == 0) {
    part[3 * t] = acc[0];
    part[3 * t + 1] = acc[1];
    part[3 * t + 2] = acc[2];
  }
}

// The row loop of one SpMV tile (see k_spmv_pq); `col` maps an entry to its column.
template <class S, int NR, int LPR, int U, class Col>
__device__ __forceinline__ void spmv_pq_tile(int64_t beg, int64_t end, const int32_t* __restrict__ row_ptr, Col col,
                                             const S* __restrict__ vals, const S* __restrict__ p, S* __restrict__ q,
                                             S (&acc)[1]) {
  constexpr int K = (8 + LPR - 1) / LPR;
  const int sub = threadIdx.x % LPR;
  const int rpp = kTileThreads / LPR;
  for (int64_t base = beg; base < end; base += (int64_t)rpp * U) {
    int lo[U], hi[U];
    int32_t rb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + threadIdx.x / LPR + (int64_t)u * rpp;
      rb[u] = col.row_base(i);
      const bool valid = i < end;
      lo[u] = valid ? row_ptr[i] : 0;
      hi[u] = valid ? row_ptr[i + 1] : 0;
    }
    S av[U][K];
    int cv[U][K];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int e = lo[u] + sub + k * LPR;
        const bool in = e < hi[u];
        av[u][k] = in ? vals[e] : S(0);
        cv[u][k] = in ? col(e, rb[u]) : -1;
      }
    V<S, NR> s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int c = 0; c < NR; ++c) s[u].c[c] = S(0);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (cv[u][k] >= 0) {
          const V<S, NR> pv = ldv<S, NR>(p, cv[u][k]);
#pragma unroll
          for (int c = 0; c < NR; ++c) s[u].c[c] += av[u][k] * pv.c[c];
        }
      for (int e = lo[u] + sub + K * LPR; e < hi[u]; e += LPR) {  // rows longer than K * LPR
        const S a = vals[e];
        const V<S, NR> pv = ldv<S, NR>(p, col(e, rb[u]));
#pragma unroll
        for (int c = 0; c < NR; ++c) s[u].c[c] += a * pv.c[c];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < NR; ++c) s[u].c[c] += __shfl_xor_sync(0xffffffffu, s[u].c[c], o, LPR);
    if (sub == 0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = base + threadIdx.x / LPR + (int64_t)u * rpp;
        if (i < end) {
          stv<S, NR>(q, i, s[u]);
          const V<S, NR> pi = ldv<S, NR>(p, i);
#pragma unroll
          for (int c = 0; c < NR; ++c) acc[0] += pi.c[c] * s[u].c[c];
        }
      }
    }
  }
}

// q = A p on the tile's rows fused with the partial p.q.  CSR-vector: LPR lanes per row,
// each lane covering K = ceil(8 / LPR) entries in one unrolled sweep (rows of a mesh
// Laplacian hold <= 8 entries almost always; longer rows finish in a remainder loop), U rows
// per sub-warp in flight so a warp keeps U * K independent value/column loads and U * K
// gathers outstanding.  Block-uniform trip counts keep every lane in the shuffles.  NW: the
// column stream's kind (ColsWide, ColsNarrow, ColsRowRel).
template <class S, int NR, int LPR, int U, int NW, class Step>
__global__ void __launch_bounds__(kTileThreads) k_spmv_pq_k(Tiles T, const ChartState* __restrict__ st,
                                                            const int32_t* __restrict__ row_ptr,
                                                            const int32_t* __restrict__ cols,
                                                            const uint16_t* __restrict__ c16,
                                                            const int32_t* __restrict__ cbase, const S* __restrict__ vals,
                                                            const S* __restrict__ p, S* __restrict__ q,
                                                            double* __restrict__ part, Step F) {
  __shared__ S sh[32];
  const int64_t t = blockIdx.x;
  const int32_t ch = T.chart[t];
  if (st[ch].state != kActive) return;
  S acc[1] = {S(0)};
  const int64_t beg = T.tab[2 * t], end = T.tab[2 * t + 1];
  if constexpr (NW == 1) spmv_pq_tile<S, NR, LPR, U>(beg, end, row_ptr, ColsNarrow{c16, cbase[ch]}, vals, p, q, acc);
  else if constexpr (NW == 2) spmv_pq_tile<S, NR, LPR, U>(beg, end, row_ptr, ColsRowRel{c16}, vals, p, q, acc);
  else spmv_pq_tile<S, NR, LPR, U>(beg, end, row_ptr, ColsWide{cols}, vals, p, q, acc);
  block_sum_first<1, S>(acc, sh);
  const double v[1] = {(double)acc[0]};
  tile_end<1>(T, F, t, ch, v, part);
}

// ---------------------------------------------------------------- bulk-copy SpMV
// the largest tile's nonzeros and rows (for the bulk-copy SpMV's staging size)
__global__ void k_tile_max(Tiles T, const int32_t* __restrict__ row_ptr, unsigned long long* __restrict__ mx) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T.n) return;
  const int64_t b = T.tab[2 * t], e = T.tab[2 * t + 1];
  atomicMax(mx, (unsigned long long)(row_ptr[e] - row_ptr[b]));
  atomicMax(mx + 1, (unsigned long long)(e - b));
}


// The same q = A p with the fused p.q as k_spmv_pq_k, but each CTA first stages its tile's
// row pointers, FP32 values and column stream into shared memory with 1-D bulk asynchronous
// copies (cp.async.bulk, completing on an mbarrier) and then runs the row loop from shared
// memory: the per-row chain of dependent global loads (row pointers, then values and
// columns, then the gathers of p) loses its first two links, and the copy engine keeps a
// whole tile of bytes in flight per CTA.  Windows are widened to 16-byte boundaries (the
// bulk copy's alignment rule); the workspace allocations carry the slack that the widened
// end may read.  The staging wait is bounded: past its iteration limit the CTA sets T.err,
// waits once more (bounded) for its own copies and returns.
// bytes of one tile's stage (row pointers, values, columns) for the largest tile
template <class S, int NW>
inline size_t spmv_stage_bytes(const Tiles& T) {
  auto up16 = [](int64_t b) { return (size_t)((b + 15) & ~(int64_t)15); };
  return up16(4 * (T.max_rows + 1) + 16) + up16((int64_t)sizeof(S) * T.max_nnz + 16) +
         up16((NW ? 2 : 4) * T.max_nnz + 16);
}
template <class S, int NW>
inline size_t spmv_tma_smem(const Tiles& T) {
  return 16 + spmv_stage_bytes<S, NW>(T);
}
constexpr size_t kSpmvTmaMaxSmem = 100 * 1024;  // two CTAs per SM at least

// One tile's windows and where they sit in a stage buffer.
struct SpmvWin {
  Win r, v, c;
};
template <class S, int NW>
__device__ __forceinline__ SpmvWin spmv_windows(const int32_t* row_ptr, const S* vals, const int32_t* cols,
                                                const uint16_t* c16, int64_t beg, int64_t end) {
  const int64_t e0 = row_ptr[beg], e1 = row_ptr[end];
  return SpmvWin{stage_window(row_ptr, beg, end + 1, 4), stage_window(vals, e0, e1, (int)sizeof(S)),
                 NW ? stage_window(c16, e0, e1, 2) : stage_window(cols, e0, e1, 4)};
}
// thread 0: arm `bar` for the tile's bytes and start its three copies into `buf`
__device__ __forceinline__ void spmv_issue(const SpmvWin& w, unsigned char* buf, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(w.r.bytes + w.v.bytes + w.c.bytes)
               : "memory");
  bulk_g2s(buf, w.r.src, w.r.bytes, bar);
  bulk_g2s(buf + w.r.bytes, w.v.src, w.v.bytes, bar);
  bulk_g2s(buf + w.r.bytes + w.v.bytes, w.c.src, w.c.bytes, bar);
}

// The row loop of spmv_pq_tile over a staged tile: row pointers, values and columns read from
// the stage buffer (the same arithmetic in the same order, so the same bits).
template <class S, int NR, int LPR, int U, int NW>
__device__ __forceinline__ void spmv_staged_tile(int64_t beg, int64_t end, const SpmvWin& w,
                                                 const unsigned char* buf, int32_t cb, const S* __restrict__ p,
                                                 S* __restrict__ q, S& acc) {
  const int32_t* rs = reinterpret_cast<const int32_t*>(buf);
  const S* vs = reinterpret_cast<const S*>(buf + w.r.bytes);
  const unsigned char* sc = buf + w.r.bytes + w.v.bytes;
  struct {
    const unsigned char* sc;
    int64_t first;
    int32_t cb;
    __device__ __forceinline__ int32_t row_base(int64_t i) const { return narrow_row_base<NW>(cb, i); }
    __device__ __forceinline__ int32_t operator()(int64_t e, int32_t rb) const {
      if constexpr (NW != 0) return rb + (int32_t)(reinterpret_cast<const uint16_t*>(sc)[e - first]);
      else return reinterpret_cast<const int32_t*>(sc)[e - first];
    }
  } col{sc, w.c.first, cb};
  constexpr int K = (8 + LPR - 1) / LPR;
  const int sub = threadIdx.x % LPR;
  const int rpp = kTileThreads / LPR;
  for (int64_t base = beg; base < end; base += (int64_t)rpp * U) {
    int lo[U], hi[U];
    int32_t rb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + threadIdx.x / LPR + (int64_t)u * rpp;
      rb[u] = col.row_base(i);
      const bool valid = i < end;
      lo[u] = valid ? rs[i - w.r.first] : 0;
      hi[u] = valid ? rs[i + 1 - w.r.first] : 0;
    }
    S av[U][K];
    int cv[U][K];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int e = lo[u] + sub + k * LPR;
        const bool in = e < hi[u];
        av[u][k] = in ? vs[e - w.v.first] : S(0);
        cv[u][k] = in ? col(e, rb[u]) : -1;
      }
    V<S, NR> sm[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int c = 0; c < NR; ++c) sm[u].c[c] = S(0);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (cv[u][k] >= 0) {
          const V<S, NR> pv = ldv<S, NR>(p, cv[u][k]);
#pragma unroll
          for (int c = 0; c < NR; ++c) sm[u].c[c] += av[u][k] * pv.c[c];
        }
      for (int e = lo[u] + sub + K * LPR; e < hi[u]; e += LPR) {  // rows longer than K * LPR
        const S a = vs[e - w.v.first];
        const V<S, NR> pv = ldv<S, NR>(p, col(e, rb[u]));
#pragma unroll
        for (int c = 0; c < NR; ++c) sm[u].c[c] += a * pv.c[c];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < NR; ++c) sm[u].c[c] += __shfl_xor_sync(0xffffffffu, sm[u].c[c], o, LPR);
    if (sub == 0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = base + threadIdx.x / LPR + (int64_t)u * rpp;
        if (i < end) {
          stv<S, NR>(q, i, sm[u]);
          const V<S, NR> pi = ldv<S, NR>(p, i);
#pragma unroll
          for (int c = 0; c < NR; ++c) acc += pi.c[c] * sm[u].c[c];
        }
      }
    }
  }
}

template <class S, int NR, int LPR, int U, int NW>
__global__ void __launch_bounds__(kTileThreads) k_spmv_tma(Tiles T, const ChartState* __restrict__ st,
                                                           const int32_t* __restrict__ row_ptr,
                                                           const int32_t* __restrict__ cols,
                                                           const uint16_t* __restrict__ c16,
                                                           const int32_t* __restrict__ cbase, const S* __restrict__ vals,
                                                           const S* __restrict__ p, S* __restrict__ q,
                                                           double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char stage[];
  __shared__ S sh[32];
  const int64_t t = blockIdx.x;
  const int32_t ch = T.chart[t];
  if (st[ch].state != kActive) return;
  const int64_t beg = T.tab[2 * t], end = T.tab[2 * t + 1];
  const SpmvWin w = spmv_windows<S, NW>(row_ptr, vals, cols, c16, beg, end);
  uint64_t* bar = reinterpret_cast<uint64_t*>(stage);
  unsigned char* buf = stage + 16;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    spmv_issue(w, buf, bar);
  }
  __syncthreads();  // the barrier is initialised before anyone waits on it
  // one decision for the whole CTA: a wait that ran out in any thread sends every thread out
  if (__syncthreads_or(!mbar_wait(bar, 0, T.spin_limit))) {
    if (threadIdx.x == 0) atomicOr(T.err, 1);
    mbar_wait(bar, 0, T.spin_limit);  // (bounded) let this CTA's own copies land before it exits
    return;
  }
  S acc = S(0);
  spmv_staged_tile<S, NR, LPR, U, NW>(beg, end, w, buf, NW == 1 ? cbase[ch] : 0, p, q, acc);
  S accv[1] = {acc};
  block_sum_first<1, S>(accv, sh);
  const double v[1] = {(double)accv[0]};
  tile_end<1>(T, NoStep(), t, ch, v, part);
}

// One launch of the SpMV for a column stream of kind nw (0 wide, 1 chart-relative, 2 row-
// relative): the bulk-copy kernel when the context set it up (upload_tiles) and its stage fits,
// else the CSR-vector kernel.
template <class S, int NR, int LPR, int U, int NW, class Step>
void launch_spmv_nw(cudaStream_t s, unsigned grid, const Tiles& T, const ChartState* st, const int32_t* row_ptr,
                    const int32_t* cols, const uint16_t* c16, const int32_t* cbase, const S* vals, const S* p, S* q,
                    double* part, const Step& F) {
  if constexpr (std::is_same<S, float>::value && NR == 2 && std::is_same<Step, NoStep>::value) {
    const size_t sm = spmv_tma_smem<S, NW>(T);
    if (T.max_rows > 0 && sm <= kSpmvTmaMaxSmem) {
      k_spmv_tma<S, NR, LPR, U, NW><<<grid, kTileThreads, sm, s>>>(T, st, row_ptr, cols, c16, cbase, vals, p, q, part);
      return;
    }
  }
  k_spmv_pq_k<S, NR, LPR, U, NW><<<grid, kTileThreads, 0, s>>>(T, st, row_ptr, cols, c16, cbase, vals, p, q, part, F);
}
template <class S, int NR, int LPR, int U, class Step>
void launch_spmv(cudaStream_t s, unsigned grid, const Tiles& T, const ChartState* st, const DevSystem& sys,
                 const S* vals, const S* p, S* q, double* part, const Step& F) {
  if (sys.cols16 && sys.rowrel16)
    launch_spmv_nw<S, NR, LPR, U, 2>(s, grid, T, st, sys.row_ptr, sys.cols, sys.cols16, sys.cbase, vals, p, q, part, F);
  else if (sys.cols16)
    launch_spmv_nw<S, NR, LPR, U, 1>(s, grid, T, st, sys.row_ptr, sys.cols, sys.cols16, sys.cbase, vals, p, q, part, F);
  else
    launch_spmv_nw<S, NR, LPR, U, 0>(s, grid, T, st, sys.row_ptr, sys.cols, sys.cols16, sys.cbase, vals, p, q, part, F);
}

// Allows the bulk-copy kernels the dynamic shared memory they need (outside any capture).
template <class S, int NR, int LPR, int U>
void spmv_tma_attributes(const Tiles& T) {
  if constexpr (std::is_same<S, float>::value && NR == 2) {
    if (T.max_rows <= 0) return;
    RUV_CUDA(cudaFuncSetAttribute(k_spmv_tma<S, NR, LPR, U, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kSpmvTmaMaxSmem));
    RUV_CUDA(cudaFuncSetAttribute(k_spmv_tma<S, NR, LPR, U, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kSpmvTmaMaxSmem));
    RUV_CUDA(cudaFuncSetAttribute(k_spmv_tma<S, NR, LPR, U, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kSpmvTmaMaxSmem));
  }
}

// x += alpha p; r -= alpha q; z = M^-1 r.  Partials: r.r, r.z.  precond: 0 = none (z = r),
// 1 = Jacobi, 2 = applied separately afterwards (z is not written).
template <class S, int NR, class Step>
__global__ void __launch_bounds__(kTileThreads) k_update(Tiles T, const ChartState* __restrict__ st,
                                                         const S* __restrict__ dinv, int use_jacobi,
                                                         S* __restrict__ x, S* __restrict__ r, S* __restrict__ z,
                                                         const S* __restrict__ p, const S* __restrict__ q,
                                                         double* __restrict__ part, Step F) {
  __shared__ S sh[2 * 32];
  int64_t t = blockIdx.x;
  const int32_t ch = T.chart[t];
  const ChartState& cs = st[ch];
  if (cs.state != kActive) return;
  const S alpha = std::is_same<S, float>::value ? (S)cs.alpha32 : (S)cs.alpha;
  S acc[2] = {S(0), S(0)};
  for (int64_t i = T.tab[2 * t] + threadIdx.x; i < T.tab[2 * t + 1]; i += blockDim.x) {
    V<S, NR> xv = ldv<S, NR>(x, i), rv = ldv<S, NR>(r, i), pv = ldv<S, NR>(p, i), qv = ldv<S, NR>(q, i), zv;
    const S di = use_jacobi == 1 ? dinv[i] : S(1);
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      xv.c[k] += alpha * pv.c[k];
      rv.c[k] -= alpha * qv.c[k];
      zv.c[k] = rv.c[k] * di;
      acc[0] += rv.c[k] * rv.c[k];
      acc[1] += rv.c[k] * zv.c[k];
    }
    stv<S, NR>(x, i, xv);
    stv<S, NR>(r, i, rv);
    if (use_jacobi != 2) stv<S, NR>(z, i, zv);
  }
  block_sum_first<2, S>(acc, sh);
  const double v[2] = {(double)acc[0], (double)acc[1]};
  tile_end<2>(T, F, t, ch, v, part);
}

// p = z + beta p
template <class S, int NR>
__global__ void __launch_bounds__(kTileThreads) k_direction(Tiles T, const ChartState* __restrict__ st,
                                                            const S* __restrict__ z, S* __restrict__ p) {
  int64_t t = blockIdx.x;
  const ChartState& cs = st[T.chart[t]];
  if (cs.state != kActive) return;
  const S beta = std::is_same<S, float>::value ? (S)cs.beta32 : (S)cs.beta;
  for (int64_t i = T.tab[2 * t] + threadIdx.x; i < T.tab[2 * t + 1]; i += blockDim.x) {
    V<S, NR> zv = ldv<S, NR>(z, i), pv = ldv<S, NR>(p, i);
#pragma unroll
    for (int k = 0; k < NR; ++k) pv.c[k] = zv.c[k] + beta * pv.c[k];
    stv<S, NR>(p, i, pv);
  }
}

// Mixed precision, once per solve: the low FP32 halves of the FP64 values (vals32 holds the
// high halves) and the FP64 row sums as double-float pairs.
__global__ void k_split_rows(int64_t n, const int32_t* __restrict__ row_ptr, const double* __restrict__ vals,
                             const float* __restrict__ vals32, float* __restrict__ vals_lo, float2* __restrict__ rsum) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double acc = 0.0;
  for (int e = row_ptr[i]; e < row_ptr[i + 1]; ++e) {
    const double v = vals[e];
    vals_lo[e] = (float)(v - (double)vals32[e]);
    acc += v;
  }
  float h, l;
  split_f64(acc, h, l);
  rsum[i] = make_float2(h, l);
}

// Mixed precision, refresh step 1 (charts that asked for a refresh, or every chart when
// `all`): fold the FP32 increment into the double-float solution, xs = 0.  A separate launch
// from the true residual, which reads the solution of neighbouring rows in other tiles.
// With `all` (end of the solve) the FP64 solution x64 = hi + lo is written too.
template <int NR>
__global__ void __launch_bounds__(kTileThreads) k_fold(Tiles T, const ChartState* __restrict__ st, int all,
                                                       float* __restrict__ xdf, float* __restrict__ xs,
                                                       double* __restrict__ x64) {
  int64_t t = blockIdx.x;
  const ChartState& cs = st[T.chart[t]];
  if (!all && (cs.state != kActive || !cs.refresh)) return;
  for (int64_t i = T.tab[2 * t] + threadIdx.x; i < T.tab[2 * t + 1]; i += blockDim.x) {
    DF<NR> xv = lddf<NR>(xdf, i);
    V<float, NR> dv = ldv<float, NR>(xs, i), zero;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      float sh, se;
      two_sum(xv.h[k], dv.c[k], sh, se);
      se += xv.l[k];
      xv.h[k] = sh + se;  // renormalise: |lo| <= ulp(hi) / 2
      xv.l[k] = se - (xv.h[k] - sh);
      zero.c[k] = 0.f;
    }
    stdf<NR>(xdf, i, xv);
    stv<float, NR>(xs, i, zero);
    if (all) {
      V<double, NR> x;
#pragma unroll
      for (int k = 0; k < NR; ++k) x.c[k] = (double)xv.h[k] + (double)xv.l[k];
      stv<double, NR>(x64, i, x);
    }
  }
}

// Mixed precision, refresh step 2: r = b - A x in double-float (see the file comment),
// r32 = r, z = M^-1 r (precond 0: z = r, 1: Jacobi, 2: applied separately, z not written).
// Partials: r.r and r.z, summed in FP32 over r * rscale and rescaled per tile.  The CSR-vector
// shape (LPR lanes, K = ceil(8 / LPR) slots, U rows in flight) is the tuned SpMV's.
template <int NR, int LPR, int U, int NW, class Step>
__global__ void __launch_bounds__(kTileThreads) k_true_residual(Tiles T, const ChartState* __restrict__ st,
                                                                const int32_t* __restrict__ row_ptr,
                                                                const int32_t* __restrict__ cols,
                                                                const uint16_t* __restrict__ c16,
                                                                const int32_t* __restrict__ cbase, const float* __restrict__ vh,
                                                                const float* __restrict__ vl, const float2* __restrict__ rsum,
                                                                const float* __restrict__ bdf, const float* __restrict__ dinv,
                                                                int precond, const float* __restrict__ xdf,
                                                                float* __restrict__ r, float* __restrict__ z,
                                                                double* __restrict__ part, Step F) {
  constexpr int K = (8 + LPR - 1) / LPR;
  __shared__ float sh[2 * 32];
  const int64_t t = blockIdx.x;
  const ChartState& cs = st[T.chart[t]];
  if (cs.state != kActive || !cs.refresh) return;
  const float rsc = cs.rscale;
  const int sub = threadIdx.x % LPR;
  const int rpp = kTileThreads / LPR;
  float acc[2] = {0.0f, 0.0f};
  const int64_t beg = T.tab[2 * t], end = T.tab[2 * t + 1];
  auto run = [&](auto col) {
  for (int64_t base = beg; base < end; base += (int64_t)rpp * U) {
    int lo[U], hi[U];
    int32_t rb[U];
    DF<NR> xi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + threadIdx.x / LPR + (int64_t)u * rpp;
      rb[u] = col.row_base(i);
      const bool valid = i < end;
      lo[u] = valid ? row_ptr[i] : 0;
      hi[u] = valid ? row_ptr[i + 1] : 0;
      xi[u] = lddf<NR>(xdf, valid ? i : beg);
    }
    float ah[U][K], al[U][K];
    int cv[U][K];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int e = lo[u] + sub + k * LPR;
        const bool in = e < hi[u];
        ah[u][k] = in ? vh[e] : 0.0f;
        al[u][k] = in ? vl[e] : 0.0f;
        cv[u][k] = in ? col(e, rb[u]) : -1;
      }
    float Sh[U][NR], Sl[U][NR];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int c = 0; c < NR; ++c) Sh[u][c] = Sl[u][c] = 0.0f;
      auto entry = [&](float a_h, float a_l, int j) {
        const DF<NR> xj = lddf<NR>(xdf, j);
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          float dh, dl;
          two_sum(xj.h[c], -xi[u].h[c], dh, dl);
          dl += xj.l[c] - xi[u].l[c];
          df_fma(a_h, a_l, dh, dl, Sh[u][c], Sl[u][c]);
        }
      };
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (cv[u][k] >= 0) entry(ah[u][k], al[u][k], cv[u][k]);
      for (int e = lo[u] + sub + K * LPR; e < hi[u]; e += LPR) entry(vh[e], vl[e], col(e, rb[u]));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          const float oh = __shfl_xor_sync(0xffffffffu, Sh[u][c], o, LPR);
          const float ol = __shfl_xor_sync(0xffffffffu, Sl[u][c], o, LPR);
          float s2, e2;
          two_sum(Sh[u][c], oh, s2, e2);
          Sh[u][c] = s2;
          Sl[u][c] += ol + e2;
        }
      const int64_t i = base + threadIdx.x / LPR + (int64_t)u * rpp;
      if (sub == 0 && i < end) {
        const float2 rs = rsum[i];
        const DF<NR> bv = lddf<NR>(bdf, i);
        const float di = precond == 1 ? dinv[i] : 1.0f;
        V<float, NR> rv, zv;
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          // A x = rs * x_i + S
          float th = 0.0f, tl = 0.0f;
          df_fma(rs.x, rs.y, xi[u].h[c], xi[u].l[c], th, tl);
          float ah2, ae2;
          two_sum(th, Sh[u][c], ah2, ae2);
          const float axl = tl + Sl[u][c] + ae2;
          // r = b - A x
          float uh, ue;
          two_sum(bv.h[c], -ah2, uh, ue);
          ue += bv.l[c] - axl;
          rv.c[c] = uh + ue;
          zv.c[c] = rv.c[c] * di;
          const float rs_ = rv.c[c] * rsc;
          acc[0] += rs_ * rs_;
          acc[1] += rs_ * (zv.c[c] * rsc);
        }
        stv<float, NR>(r, i, rv);
        if (precond != 2) stv<float, NR>(z, i, zv);
      }
    }
  }
  };
  if constexpr (NW == 1) run(ColsNarrow{c16, cbase[T.chart[t]]});
  else if constexpr (NW == 2) run(ColsRowRel{c16});
  else run(ColsWide{cols});
  block_sum_first<2, float>(acc, sh);
  double v[2] = {0.0, 0.0};
  if (threadIdx.x == 0) {
    const double inv = 1.0 / ((double)rsc * (double)rsc);
    v[0] = (double)acc[0] * inv;
    v[1] = (double)acc[1] * inv;
  }
  tile_end<2>(T, F, t, T.chart[t], v, part);
}

// One launch of the true residual for the system's column stream kind.
template <int NR, int LPR, int U, class MX, class Step>
void launch_true_residual(cudaStream_t s, unsigned grid, const Tiles& T, const ChartState* st, const DevSystem& sys,
                          const MX& mx, const float* dinv32, int precond, float* r, float* z, double* part,
                          const Step& F) {
#define RUV_TR(NWV)                                                                                                   \
  k_true_residual<NR, LPR, U, NWV><<<grid, kTileThreads, 0, s>>>(T, st, sys.row_ptr, sys.cols, sys.cols16, sys.cbase, \
                                                                sys.vals32, mx.vals_lo, mx.rsum, mx.bdf, dinv32,      \
                                                                precond, mx.xdf, r, z, part, F)
  if (sys.cols16 && sys.rowrel16) RUV_TR(2);
  else if (sys.cols16) RUV_TR(1);
  else RUV_TR(0);
#undef RUV_TR
}

template <class S, int NR, class Step>
__global__ void __launch_bounds__(kTileThreads) k_dots_rz(Tiles T, const ChartState* __restrict__ st, const S* __restrict__ r,
                                                          const S* __restrict__ z, const S* __restrict__ q,
                                                          double* __restrict__ part, Step F) {
  __shared__ S sh[2 * 32];
  int64_t t = blockIdx.x;
  const int32_t ch = T.chart[t];
  if (st[ch].state != kActive) return;
  S acc[2] = {S(0), S(0)};
  for (int64_t i = T.tab[2 * t] + threadIdx.x; i < T.tab[2 * t + 1]; i += blockDim.x) {
    const V<S, NR> rv = ldv<S, NR>(r, i), zv = ldv<S, NR>(z, i), qv = ldv<S, NR>(q, i);
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      acc[0] += rv.c[k] * zv.c[k];
      acc[1] += zv.c[k] * qv.c[k];
    }
  }
  block_sum_first<2, S>(acc, sh);
  const double v[2] = {(double)acc[0], (double)acc[1]};
  tile_end<2>(T, F, t, ch, v, part);
}

// ---------------------------------------------------------------- chart kernels
template <int NV>
__device__ __forceinline__ void chart_reduce(const Tiles& T, int64_t c, const double* part, int stride, double (&v)[NV],
                                             double* sh) {
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int64_t t = T.chart_tile[c] + threadIdx.x; t < T.chart_tile[c + 1]; t += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += part[stride * t + k];
  block_sum<NV>(v, sh);
}

__global__ void __launch_bounds__(kChartThreads) k_chart_init(Tiles T, ChartState* __restrict__ st, const double* __restrict__ part,
                                                              double tol, int precond_none, int* __restrict__ n_active) {
  __shared__ double sh[3 * 32];
  int64_t c = blockIdx.x;
  double v[3];
  chart_reduce<3>(T, c, part, 3, v, sh);
  if (threadIdx.x != 0) return;
  ChartState s{};
  s.bnorm = sqrt(v[0]);
  s.tol_abs = s.bnorm <= 1e-300 ? tol : tol * s.bnorm;
  s.rscale = s.bnorm > 0.0 ? (float)fmin(fmax(1.0 / s.bnorm, 1e-30), 1e30) : 1.0f;
  s.rr = v[0];
  s.r_ref = s.bnorm;
  s.rz = precond_none ? v[0] : v[1];
  s.iters = 0;
  s.refinements = 0;
  s.refresh = 0;
  if (v[2] > 0.0 && !precond_none) {
    s.status = RUV_ERR_BREAKDOWN;  // Jacobi with a zero diagonal (precond.rs:595-611)
    s.state = kDone;
  } else if (sqrt(v[0]) <= s.tol_abs) {
    s.status = RUV_OK;
    s.state = kDone;
  } else if (T.chart_tile[c] == T.chart_tile[c + 1]) {
    s.status = RUV_ERR_BREAKDOWN;  // no rows under a tolerance that zero does not meet: p.q is 0, and no tile takes that step
    s.state = kDone;
  } else {
    s.status = RUV_ERR_NOT_CONVERGED;
    s.state = kActive;
    atomicAdd(n_active, 1);
  }
  st[c] = s;
}

// A chart step as a kernel of its own, one CTA per chart.
template <int NV>
__global__ void __launch_bounds__(kChartThreads) k_chart_step(Tiles T, ChartStep F, const double* __restrict__ part) {
  __shared__ double sh[NV * 32];
  const int64_t c = blockIdx.x;
  if (F.st[c].state != kActive || (F.kind == kStepAfterRefresh && !F.st[c].refresh)) return;
  double v[NV];
  chart_reduce<NV>(T, c, part, NV, v, sh);
  if (threadIdx.x == 0) chart_step(F, c, v[0], NV > 1 ? v[NV - 1] : 0.0);
}

// ---------------------------------------------------------------- separate preconditioner
// (AMG) support: done mask, r.z / z.q partials, chart-level beta.
__global__ void k_mark_done(const ChartState* __restrict__ st, int64_t n, int32_t* __restrict__ done) {
  int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) done[c] = st[c].state != kActive ? 1 : 0;
}

template <class S, int NR>
__global__ void __launch_bounds__(kTileThreads) k_copy_dir(Tiles T, const ChartState* __restrict__ st, const S* __restrict__ z,
                                                           S* __restrict__ p) {
  int64_t t = blockIdx.x;
  if (st[T.chart[t]].state != kActive) return;
  for (int64_t i = T.tab[2 * t] + threadIdx.x; i < T.tab[2 * t + 1]; i += blockDim.x) stv<S, NR>(p, i, ldv<S, NR>(z, i));
}

// FP64 <-> FP32 copies of the preconditioner's input / output (FP64 outer loop).
template <class A, class Bt>
__global__ void k_convert(int64_t n, const A* __restrict__ in, Bt* __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (Bt)in[i];
}

// ---------------------------------------------------------------- host driver
struct TileTable {
  std::vector<int64_t> tab, chart_tile;
  std::vector<int32_t> chart;
};

// Mixed precision's double-float state: solution and right-hand side (2 * NR floats per
// row), the low halves of the FP64 values and the FP64 row sums (k_split_rows, launched here).
struct MixedExtras {
  float* xdf = nullptr;
  float* bdf = nullptr;
  float* vals_lo = nullptr;
  float2* rsum = nullptr;
};

MixedExtras mixed_extras(Ctx& ctx, DevSystem& sys, int nr) {
  MixedExtras m;
  if (nr == 0) return m;
  const int64_t N = sys.n_rows;
  m.xdf = ctx.ws.get<float>("pcg.xdf", 2 * nr * N);
  m.bdf = ctx.ws.get<float>("pcg.bdf", 2 * nr * N);
  if (sys.vals_lo && sys.rsum) {  // formed by the assembly's fill pass
    m.vals_lo = sys.vals_lo;
    m.rsum = sys.rsum;
    return m;
  }
  m.vals_lo = ctx.ws.get<float>("pcg.vals_lo", sys.nnz);
  m.rsum = ctx.ws.get<float2>("pcg.rsum", N);
  if (N > 0) {
    k_split_rows<<<div_up(N, kTileThreads), kTileThreads, 0, ctx.stream>>>(N, sys.row_ptr, sys.vals, sys.vals32, m.vals_lo,
                                                                           m.rsum);
    count_launches(1);
    RUV_LAUNCH_CHECK();
  }
  return m;
}

// The chart steps' arrival counters, zero (a step leaves them so; a failed solve may not have).
int32_t* arrived_counters(Ctx& ctx, int64_t n_charts) {
  int32_t* d = ctx.ws.get<int32_t>("pcg.arrived", n_charts);
  RUV_CUDA(cudaMemsetAsync(d, 0, sizeof(int32_t) * std::max<int64_t>(n_charts, 1), ctx.stream));
  return d;
}

// Whether the tile kernels take the chart steps: up to eight tiles an SM.  With more, the fence and the
// atomic that end every tile cost the kernels' throughput as much as a kernel between them, or more (ms, in
// the tiles / kernels between: one chart of 88,800 rows in FP64, 152 tiles, 10.5 / 10.9 for 400 iterations;
// a 1024^2 field, 1,021 tiles, 28.6 / 28.8; 1,000 disks, 2,500 tiles, 14.8 / 15.0; a 1448^2 field, 2,048
// tiles, 48.4 / 48.2; 4096 disks, 14,900 tiles, 99.8 / 99.6).  Only shapes that pick_shape takes, and not
// the bulk-copy SpMV, are built with the steps; RUV_TILE_STEPS=1 / 0 takes them in the tiles whatever the
// count / never (bit-identical results).
template <int LPR, int U>
bool steps_in_tiles(const Ctx& ctx, const Tiles& T) {
  const char* e = std::getenv("RUV_TILE_STEPS");
  return steps_built<LPR, U>() && T.max_rows == 0 && (e ? e[0] == '1' : T.n <= 8 * (int64_t)ctx.sm_count);
}

template <class S, int NR, int LPR, int U>
void run_pcg(Ctx& ctx, DevSystem& sys, double* x64, const SolveOpts& o, Tiles T, ChartState* st, int* n_active,
             std::vector<ChartState>& out) {
  cudaStream_t s = ctx.stream;
  Workspace& ws = ctx.ws;
  const bool mixed = std::is_same<S, float>::value;
  const int64_t NR_ = sys.n_rows, NC = sys.n_charts, NTL = T.n;
  const int jac = o.precond == RUV_PRECOND_JACOBI ? 1 : 0;
  const int none = o.precond == RUV_PRECOND_NONE ? 1 : 0;
  S* xs = mixed ? ws.get<S>("pcg.xs", NR * NR_) : nullptr;
  S* r = ws.get<S>("pcg.r", NR * NR_);
  S* z = ws.get<S>("pcg.z", NR * NR_);
  S* p = ws.get<S>("pcg.p", NR * NR_);
  S* q = ws.get<S>("pcg.q", NR * NR_);
  S* dinv = ws.get<S>("pcg.dinv", NR_);
  float* dinv32 = mixed ? reinterpret_cast<float*>(dinv) : nullptr;
  double* part = ws.get<double>("pcg.part", 3 * NTL);
  const S* vals = mixed ? reinterpret_cast<const S*>(sys.vals32) : reinterpret_cast<const S*>(sys.vals);
  MixedExtras mx = mixed_extras(ctx, sys, mixed ? NR : 0);
  RUV_CUDA(cudaMemsetAsync(n_active, 0, sizeof(int), s));
  if (NR_ > 0) {
    k_dinv<S><<<div_up(NR_, kTileThreads), kTileThreads, 0, s>>>(NR_, sys.diag, dinv);
    count_launches(1);
    RUV_LAUNCH_CHECK();
  }
  if (NTL > 0) {
    k_init<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, sys.b, sys.diag, dinv, jac, x64, xs, r, z, p, part, mx.xdf,
                                                         mx.bdf);
    count_launches(1);
    RUV_LAUNCH_CHECK();
  }
  k_chart_init<<<(unsigned)NC, kChartThreads, 0, s>>>(T, st, part, o.tol, none, n_active);
  count_launches(1);
  RUV_LAUNCH_CHECK();
  // the charts a team solves in one kernel (team.cu); the loop below takes the others
  int64_t left = NTL > 0 ? 1 : 0;
  if constexpr (std::is_same<S, double>::value || NR == 2) {
    if (left && o.teams && o.max_iter > -kCheckEvery) {  // (the loop below replays nothing under that)
      const TeamLoop<S> loop{vals, dinv, mixed ? xs : reinterpret_cast<S*>(x64), r, z, p, q, x64, nullptr, nullptr, mx.vals_lo, mx.rsum, mx.bdf, mx.xdf, st, n_active,
                             o.max_iter, refresh_delta(), jac};
      left = team_solve<S, NR>(ctx, sys, loop, nullptr);
    }
  }
  int* h_active = static_cast<int*>(ctx.pinned.get(3 * sizeof(int)));
  *h_active = 0;
  if (left > 0) {
    spmv_tma_attributes<S, NR, LPR, U>(T);
    RUV_CUDA(cudaMemcpyAsync(h_active, n_active, sizeof(int), cudaMemcpyDeviceToHost, s));
    RUV_CUDA(cudaStreamSynchronize(s));
  }
  if (*h_active > 0) {
    ChartStep base;
    base.precond_none = none;
    base.max_iter = o.max_iter;
    base.delta = refresh_delta();
    base.st = st;
    base.n_active = n_active;
    base.arrived = arrived_counters(ctx, NC);
    const bool in_tiles = steps_in_tiles<LPR, U>(ctx, T);
    // a tile kernel and the chart step behind its sums: in the kernel, or in one of its own
    auto with_step = [&](auto nv, int kind, auto launch) {
      ChartStep f = base;
      f.kind = kind;
      if constexpr (steps_built<LPR, U>())
        if (in_tiles) return launch(f);
      launch(NoStep());
      k_chart_step<decltype(nv)::value><<<(unsigned)NC, kChartThreads, 0, s>>>(T, f, part);
    };
    constexpr std::integral_constant<int, 1> one{};
    constexpr std::integral_constant<int, 2> two{};
    // capture kCheckEvery iterations as one graph, replay it
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    RUV_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    for (int rep = 0; rep < kCheckEvery; ++rep) {
      with_step(one, kStepAlpha, [&](const auto& f) {
        launch_spmv<S, NR, LPR, U>(s, (unsigned)NTL, T, st, sys, vals, p, q, part, f);
      });
      with_step(two, mixed ? kStepBetaMixed : kStepBeta, [&](const auto& f) {
        k_update<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, dinv, jac, mixed ? xs : reinterpret_cast<S*>(x64), r,
                                                               z, p, q, part, f);
      });
      if (mixed) {
        k_fold<NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, 0, mx.xdf, reinterpret_cast<float*>(xs), x64);
        with_step(two, kStepAfterRefresh, [&](const auto& f) {
          launch_true_residual<NR, LPR, U>(s, (unsigned)NTL, T, st, sys, mx, dinv32, jac, reinterpret_cast<float*>(r),
                                           reinterpret_cast<float*>(z), part, f);
        });
      }
      k_direction<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, z, p);
    }
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (ce != cudaSuccess) throw Error{RUV_ERR_LAUNCH, std::string("graph capture: ") + cudaGetErrorString(ce)};
    ce = cudaGraphInstantiate(&exec, graph, 0);
    if (ce != cudaSuccess) {
      cudaGraphDestroy(graph);
      throw Error{RUV_ERR_LAUNCH, std::string("graph instantiate: ") + cudaGetErrorString(ce)};
    }
    int64_t launched = 0;
    try {
      while (launched < o.max_iter + kCheckEvery) {
        RUV_CUDA(cudaGraphLaunch(exec, s));
        count_launches((int64_t)kCheckEvery * ((mixed ? 5 : 3) + (in_tiles ? 0 : mixed ? 3 : 2)));
        launched += kCheckEvery;
        RUV_CUDA(cudaMemcpyAsync(h_active, n_active, sizeof(int), cudaMemcpyDeviceToHost, s));
        if (T.err) RUV_CUDA(cudaMemcpyAsync(h_active + 2, T.err, sizeof(int), cudaMemcpyDeviceToHost, s));
        RUV_CUDA(cudaStreamSynchronize(s));
        if (T.err && h_active[2] != 0) {
          RUV_CUDA(cudaMemsetAsync(T.err, 0, sizeof(int), s));
          throw Error{RUV_ERR_TIMEOUT, "SpMV: a bounded wait for the staged tile ran out"};
        }
        if (*h_active <= 0) break;
      }
    } catch (...) {
      cudaGraphExecDestroy(exec);
      cudaGraphDestroy(graph);
      throw;
    }
    cudaGraphExecDestroy(exec);
    cudaGraphDestroy(graph);
  }
  if (mixed && NTL > 0) {
    // fold any FP32 increment still pending (charts that stopped between refreshes); x64 = xdf
    k_fold<NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, 1, mx.xdf, reinterpret_cast<float*>(xs), x64);
    count_launches(1);
    RUV_LAUNCH_CHECK();
  }
  out.resize(NC);
  RUV_CUDA(cudaMemcpyAsync(out.data(), st, sizeof(ChartState) * NC, cudaMemcpyDeviceToHost, s));
  RUV_CUDA(cudaStreamSynchronize(s));
}

// Batched PCG with a separately applied preconditioner (AMG V-cycle, IC(0) sweeps): the
// mixed loop (FP32 recurrences, double-float true-residual refreshes) or the FP64 loop.
// A preconditioner that has no FP64 form gets FP32 copies of r and z under the FP64 loop.
template <class S, int NR, int LPR, int U>
void run_pcg_sep(Ctx& ctx, DevSystem& sys, double* x64, const SolveOpts& o, Tiles T, ChartState* st, int* n_active,
                 std::vector<ChartState>& out, SepPrecond& P) {
  constexpr bool mixed = std::is_same<S, float>::value;
  cudaStream_t s = ctx.stream;
  Workspace& ws = ctx.ws;
  const int64_t NR_ = sys.n_rows, NC = sys.n_charts, NTL = T.n;
  S* xs = mixed ? ws.get<S>("pcg.xs", NR * NR_) : nullptr;
  S* r = ws.get<S>("pcg.r", NR * NR_);
  S* z = ws.get<S>("pcg.z", NR * NR_);
  S* p = ws.get<S>("pcg.p", NR * NR_);
  S* q = ws.get<S>("pcg.q", NR * NR_);
  S* dinv = ws.get<S>("pcg.dinv", NR_);
  float* dinv32 = mixed ? reinterpret_cast<float*>(dinv) : nullptr;
  const bool copies = !mixed && !P.native_fp64();
  float* r32 = copies ? ws.get<float>("pcg.r32", NR * NR_) : reinterpret_cast<float*>(r);
  float* z32 = copies ? ws.get<float>("pcg.z32", NR * NR_) : reinterpret_cast<float*>(z);
  const S* vals = mixed ? reinterpret_cast<const S*>(sys.vals32) : reinterpret_cast<const S*>(sys.vals);
  S* xiter = mixed ? xs : reinterpret_cast<S*>(x64);
  double* part = ws.get<double>("pcg.part", 3 * NTL);
  double* part2 = ws.get<double>("pcg.part2", 2 * NTL);
  MixedExtras mx = mixed_extras(ctx, sys, mixed ? NR : 0);
  int32_t* done = ws.get<int32_t>("pcg.done", NC);
  if (copies) P.bind(ctx, r32, z32, false);
  else P.bind(ctx, r, z, !mixed);
  const int flex = P.flexible() ? 1 : 0;
  const unsigned gv = div_up(NR * NR_, 256);
  auto to32 = [&]() {
    if (copies) k_convert<S, float><<<gv, 256, 0, s>>>(NR * NR_, r, r32);
  };
  auto to64 = [&]() {
    if (copies) k_convert<float, S><<<gv, 256, 0, s>>>(NR * NR_, z32, z);
  };
  const int conv = copies ? 2 : 0;
  RUV_CUDA(cudaMemsetAsync(n_active, 0, sizeof(int), s));
  if (NR_ > 0) {
    k_dinv<S><<<div_up(NR_, kTileThreads), kTileThreads, 0, s>>>(NR_, sys.diag, dinv);
    count_launches(1);
  }
  if (NTL > 0) {
    k_init<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, sys.b, sys.diag, dinv, 1, x64, xs, r, z, p, part, mx.xdf,
                                                         mx.bdf);
    count_launches(1);
  }
  k_chart_init<<<(unsigned)NC, kChartThreads, 0, s>>>(T, st, part, o.tol, 0, n_active);  // (rz replaced below)
  count_launches(1);
  RUV_LAUNCH_CHECK();
  constexpr int kRep = 8;  // iterations of a graph
  // the charts a team solves in one kernel (team.cu); the loop below takes the others
  int64_t left = NTL > 0 ? 1 : 0;
  if constexpr (std::is_same<S, double>::value || NR == 2) {
    if (left && o.teams && o.max_iter > -kRep) {  // (the loop below replays nothing under that)
      const TeamLoop<S> loop{vals, dinv, xiter, r, z, p, q, x64, r32, z32, mx.vals_lo, mx.rsum, mx.bdf, mx.xdf, st, n_active,
                             o.max_iter, refresh_delta(), 0};
      TeamPrecond tp;
      P.team(tp);
      left = team_solve<S, NR>(ctx, sys, loop, &tp);
    }
  }
  int* h_active = static_cast<int*>(ctx.pinned.get(3 * sizeof(int)));
  *h_active = 0;
  if (left > 0) {
    spmv_tma_attributes<S, NR, LPR, U>(T);
    RUV_CUDA(cudaMemcpyAsync(h_active, n_active, sizeof(int), cudaMemcpyDeviceToHost, s));
    RUV_CUDA(cudaStreamSynchronize(s));
  }
  if (*h_active > 0) {
    // z0 = M^-1 r0, rz = r.z, p = z
    k_mark_done<<<div_up(NC, 256), 256, 0, s>>>(st, NC, done);
    to32();
    count_launches(1 + conv + P.apply(ctx, done));
    to64();
    ChartStep base;
    base.precond_none = base.separate = 1;
    base.flexible = flex;
    base.max_iter = o.max_iter;
    base.delta = refresh_delta();
    base.st = st;
    base.n_active = n_active;
    base.done = done;
    base.arrived = arrived_counters(ctx, NC);
    const bool in_tiles = steps_in_tiles<LPR, U>(ctx, T);
    // a tile kernel and the chart step behind its sums: in the kernel, or in one of its own; the launches
    auto with_step = [&](auto nv, int kind, const double* sums, auto launch) -> int {
      ChartStep f = base;
      f.kind = kind;
      if constexpr (steps_built<LPR, U>())
        if (in_tiles) {
          launch(f);
          return 1;
        }
      launch(NoStep());
      k_chart_step<decltype(nv)::value><<<(unsigned)NC, kChartThreads, 0, s>>>(T, f, sums);
      return 2;
    };
    auto dots = [&](const auto& f) {
      k_dots_rz<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, r, z, q, part2, f);
    };
    constexpr std::integral_constant<int, 1> one{};
    constexpr std::integral_constant<int, 2> two{};
    count_launches(1 + with_step(two, kStepRz0, part2, dots));
    k_copy_dir<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, z, p);
    RUV_LAUNCH_CHECK();
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int per_iter = 0;
    RUV_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    for (int rep = 0; rep < kRep; ++rep) {
      int l = 0;
      l += with_step(one, kStepAlpha, part, [&](const auto& f) {
        launch_spmv<S, NR, LPR, U>(s, (unsigned)NTL, T, st, sys, vals, p, q, part, f);
      });
      l += with_step(two, mixed ? kStepBetaMixed : kStepCheck64, part, [&](const auto& f) {
        k_update<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, dinv, 2, xiter, r, z, p, q, part, f);
      });
      if (mixed) {
        k_fold<NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, 0, mx.xdf, reinterpret_cast<float*>(xs), x64);
        l += 1 + with_step(two, kStepAfterRefresh, part, [&](const auto& f) {
          launch_true_residual<NR, LPR, U>(s, (unsigned)NTL, T, st, sys, mx, dinv32, 2, reinterpret_cast<float*>(r),
                                           reinterpret_cast<float*>(z), part, f);
        });
      }
      to32();
      l += conv + P.apply(ctx, done);
      to64();
      l += 1 + with_step(two, kStepBetaPc, part2, dots);
      k_direction<S, NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, z, p);
      per_iter = l;
    }
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (ce != cudaSuccess) throw Error{RUV_ERR_LAUNCH, std::string("graph capture: ") + cudaGetErrorString(ce)};
    ce = cudaGraphInstantiate(&exec, graph, 0);
    if (ce != cudaSuccess) {
      cudaGraphDestroy(graph);
      throw Error{RUV_ERR_LAUNCH, std::string("graph instantiate: ") + cudaGetErrorString(ce)};
    }
    int64_t launched = 0;
    const int* perr = P.error_flag();
    try {
      while (launched < o.max_iter + kRep) {
        RUV_CUDA(cudaGraphLaunch(exec, s));
        count_launches((int64_t)kRep * per_iter);
        launched += kRep;
        RUV_CUDA(cudaMemcpyAsync(h_active, n_active, sizeof(int), cudaMemcpyDeviceToHost, s));
        if (perr) RUV_CUDA(cudaMemcpyAsync(h_active + 1, perr, sizeof(int), cudaMemcpyDeviceToHost, s));
        if (T.err) RUV_CUDA(cudaMemcpyAsync(h_active + 2, T.err, sizeof(int), cudaMemcpyDeviceToHost, s));
        RUV_CUDA(cudaStreamSynchronize(s));
        if (T.err && h_active[2] != 0) {
          RUV_CUDA(cudaMemsetAsync(T.err, 0, sizeof(int), s));
          throw Error{RUV_ERR_TIMEOUT, "SpMV: a bounded wait for the staged tile ran out"};
        }
        if (perr && h_active[1] != 0) {
          RUV_CUDA(cudaMemsetAsync(const_cast<int*>(perr), 0, sizeof(int), s));
          throw Error{RUV_ERR_TIMEOUT, "preconditioner: a bounded device-side wait ran out"};
        }
        if (*h_active <= 0) break;
      }
    } catch (...) {
      cudaGraphExecDestroy(exec);
      cudaGraphDestroy(graph);
      throw;
    }
    cudaGraphExecDestroy(exec);
    cudaGraphDestroy(graph);
  }
  if (mixed && NTL > 0) {
    k_fold<NR><<<(unsigned)NTL, kTileThreads, 0, s>>>(T, st, 1, mx.xdf, reinterpret_cast<float*>(xs), x64);
    count_launches(1);
    RUV_LAUNCH_CHECK();
  }
  out.resize(NC);
  RUV_CUDA(cudaMemcpyAsync(out.data(), st, sizeof(ChartState) * NC, cudaMemcpyDeviceToHost, s));
  RUV_CUDA(cudaStreamSynchronize(s));
}

// The SpMV shape: lanes per row (LPR) and rows in flight per sub-warp (U).  Instantiated
// for the shapes the tuner explores; see pick_shape.
struct Shape {
  int lpr, unroll;
};

#define RUV_SHAPES(X) X(1, 2) X(2, 2) X(2, 4) X(4, 1) X(4, 2) X(4, 4) X(8, 1) X(8, 2) X(8, 4) X(16, 1) X(32, 1)

template <class S, int NR>
void dispatch_pcg(Shape sh, Ctx& ctx, DevSystem& sys, double* x64, const SolveOpts& o, Tiles T, ChartState* st,
                  int* n_active, std::vector<ChartState>& out) {
#define RUV_CASE(L, UU) \
  if (sh.lpr == L && sh.unroll == UU) return run_pcg<S, NR, L, UU>(ctx, sys, x64, o, T, st, n_active, out);
  RUV_SHAPES(RUV_CASE)
#undef RUV_CASE
  throw Error{RUV_ERR_BAD_INPUT, "unsupported SpMV shape"};
}

TileTable make_tiles(const std::vector<int64_t>& chart_row, int64_t tile_rows);

// Rows per tile of a solve: the context's where one was chosen.  Else, for a system too small to give
// every SM four tiles of the default size: the mixed loop halves them, down to 128; the FP64 loop, which
// the SMs' FP64 pipes bound, splits a large chart evenly -- a tile an SM, or as few more as keep them
// at about the default -- since the SM with most rows is the one waited for (89,401 rows in 88 tiles
// of 1024 left 64 SMs idle: 55 -> 49 ms; 160,000 in 157 gave five SMs twice the rows: 17.3 -> 14.9 ms)
// and smaller tiles only add block sums (128 rows: 65 ms).
int64_t solve_tile_rows(const Ctx& ctx, const DevSystem& sys, bool mixed) {
  int64_t tile = ctx.tile_rows;
  if (ctx.tile_set || sys.n_rows >= 4 * tile * ctx.sm_count) return tile;
  if (mixed) {
    while (tile > 128 && sys.n_rows < 4 * tile * ctx.sm_count) tile /= 2;
    return tile;
  }
  const int64_t per_sm = std::max<int64_t>(1, (sys.n_rows + 1100 * ctx.sm_count - 1) / (1100 * ctx.sm_count));
  const int64_t even = (sys.n_rows + per_sm * ctx.sm_count - 1) / (per_sm * ctx.sm_count);
  return std::max<int64_t>(512, (even + 15) & ~(int64_t)15);
}

Tiles upload_tiles(Ctx& ctx, const DevSystem& sys, const std::string& tag, int64_t tile_rows) {
  cudaStream_t s = ctx.stream;
  TileTable TT = make_tiles(sys.h_chart_row, tile_rows);
  const int64_t NTL = (int64_t)TT.chart.size(), NC = sys.n_charts;
  int64_t* d_tab = ctx.ws.get<int64_t>(tag + ".tab", 2 * NTL);
  int32_t* d_chart = ctx.ws.get<int32_t>(tag + ".tchart", NTL);
  int64_t* d_ctile = ctx.ws.get<int64_t>(tag + ".ctile", NC + 1);
  if (NTL > 0) {
    RUV_CUDA(cudaMemcpyAsync(d_tab, TT.tab.data(), sizeof(int64_t) * 2 * NTL, cudaMemcpyHostToDevice, s));
    RUV_CUDA(cudaMemcpyAsync(d_chart, TT.chart.data(), sizeof(int32_t) * NTL, cudaMemcpyHostToDevice, s));
  }
  RUV_CUDA(cudaMemcpyAsync(d_ctile, TT.chart_tile.data(), sizeof(int64_t) * (NC + 1), cudaMemcpyHostToDevice, s));
  Tiles T{d_tab, d_chart, d_ctile, NTL};
  // the bulk-copy SpMV (when the context chose it, or RUV_SPMV_TMA=1 / =0 says so): its
  // staging size from the largest tile
  const char* te = std::getenv("RUV_SPMV_TMA");
  const bool tma = te ? te[0] == '1' : ctx.spmv_tma == 1;
  if (NTL > 0 && sys.row_ptr && tma) {
    unsigned long long* mx = ctx.ws.get<unsigned long long>(tag + ".tmax", 2);
    int* err = ctx.ws.get<int>(tag + ".terr", 1);
    RUV_CUDA(cudaMemsetAsync(mx, 0, 2 * sizeof(unsigned long long), s));
    RUV_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    k_tile_max<<<div_up(NTL, 256), 256, 0, s>>>(T, sys.row_ptr, mx);
    count_launches(1);
    unsigned long long h[2] = {0, 0};
    RUV_CUDA(cudaMemcpyAsync(h, mx, sizeof(h), cudaMemcpyDeviceToHost, s));
    RUV_CUDA(cudaStreamSynchronize(s));
    T.max_nnz = (int64_t)h[0];
    T.max_rows = (int64_t)h[1];
    T.err = err;
    const char* le = std::getenv("RUV_SPIN_LIMIT");
    T.spin_limit = le ? std::max<int64_t>(1, std::atoll(le)) : (int64_t(1) << 22);
  }
  RUV_CUDA(cudaStreamSynchronize(s));  // the host tables go out of scope
  return T;
}

// SpMV shape: explicit (RUV_LPR / RUV_UNROLL via the context) or from the row-length
// profile: enough lanes to cover a typical row once, then as many rows in flight as keep
// 8 independent loads per lane.
// The launch shape without the autotuner: for mesh Laplacians (at most 8 entries per row) two
// lanes per row and two rows in flight, which the autotuner picked on every such operator
// measured (4096 disks, 1024^2 and 2048^2 height fields); wider sub-warps for denser rows.
Shape pick_shape(const Ctx& ctx, const DevSystem& sys, bool one_lane = false) {
  double avg = sys.n_rows > 0 ? (double)sys.nnz / (double)sys.n_rows : 1.0;
  int lpr = ctx.lanes_per_row > 0 ? ctx.lanes_per_row : (avg <= 8 ? 2 : avg <= 12 ? 8 : avg <= 24 ? 16 : 32);
  int u = ctx.unroll > 0 ? ctx.unroll : (lpr <= 4 ? 2 : lpr == 8 ? 4 : 1);
  // FP64: one lane per row, whose sum needs no additions across lanes (a quarter of a two-lane row's FP64
  // instructions).  Solves, two lanes / one (ms): Jacobi, one chart of 89,401 rows 41.5 / 38.2, of 357,604
  // 152 / 138; AMG-SA, of 1.0 million 24.7 / 24.2, 2.1 million 38.5 / 37.5, 4.2 million 71.9 / 69.8, 4096 disks of
  // 14.4 million 90.8 / 87.2
  if (one_lane && ctx.lanes_per_row == 0 && lpr == 2) lpr = 1;
  return Shape{lpr, u};
}

template <class S, int NR, int LPR, int U>
double time_spmv(Ctx& ctx, DevSystem& sys, Tiles T, int reps, int nbuf, bool iter) {
  cudaStream_t s = ctx.stream;
  spmv_tma_attributes<S, NR, LPR, U>(T);
  const int64_t N = sys.n_rows, NC = sys.n_charts;
  ChartState* st = ctx.ws.get<ChartState>("bench.state", NC);
  RUV_CUDA(cudaMemsetAsync(st, 0, sizeof(ChartState) * NC, s));  // every chart active
  double* part = ctx.ws.get<double>("bench.part", T.n);
  // iter: also the tile kernels of a CG iteration that run over the same tiles (update, dots,
  // direction), whose cost depends on the tile height as well
  S* xv = iter ? ctx.ws.get<S>("bench.x", NR * N) : nullptr;
  S* rv = iter ? ctx.ws.get<S>("bench.r", NR * N) : nullptr;
  double* part2 = iter ? ctx.ws.get<double>("bench.part2", 2 * T.n) : nullptr;
  if (iter) {
    RUV_CUDA(cudaMemsetAsync(xv, 0, sizeof(S) * NR * N, s));
    RUV_CUDA(cudaMemsetAsync(rv, 0, sizeof(S) * NR * N, s));
  }
  std::vector<S*> ps(nbuf), qs(nbuf);
  for (int k = 0; k < nbuf; ++k) {
    ps[k] = ctx.ws.get<S>("bench.p" + std::to_string(k), NR * N);
    qs[k] = ctx.ws.get<S>("bench.q" + std::to_string(k), NR * N);
    RUV_CUDA(cudaMemsetAsync(ps[k], 0, sizeof(S) * NR * N, s));
  }
  const S* vals = std::is_same<S, float>::value ? reinterpret_cast<const S*>(sys.vals32) : reinterpret_cast<const S*>(sys.vals);
  auto launch = [&](int k) {
    launch_spmv<S, NR, LPR, U>(s, (unsigned)T.n, T, st, sys, vals, ps[k % nbuf],
                               qs[k % nbuf], part, NoStep());
    count_launches(1);
    if (iter && T.n > 0) {
      k_update<S, NR><<<(unsigned)T.n, kTileThreads, 0, s>>>(T, st, nullptr, 2, xv, rv, nullptr, ps[k % nbuf],
                                                             qs[k % nbuf], part2, NoStep());
      k_dots_rz<S, NR><<<(unsigned)T.n, kTileThreads, 0, s>>>(T, st, rv, rv, qs[k % nbuf], part2, NoStep());
      k_direction<S, NR><<<(unsigned)T.n, kTileThreads, 0, s>>>(T, st, rv, ps[k % nbuf]);
      count_launches(3);
    }
  };
  for (int k = 0; k < 3; ++k) launch(k);
  RUV_LAUNCH_CHECK();
  cudaEvent_t e0, e1;
  RUV_CUDA(cudaEventCreate(&e0));
  RUV_CUDA(cudaEventCreate(&e1));
  RUV_CUDA(cudaEventRecord(e0, s));
  for (int k = 0; k < reps; ++k) launch(k);
  RUV_CUDA(cudaEventRecord(e1, s));
  RUV_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  RUV_LAUNCH_CHECK();
  return (double)ms / reps;
}

template <class S, int NR>
void dispatch_pcg_sep(Shape sh, Ctx& ctx, DevSystem& sys, double* x64, const SolveOpts& o, Tiles T, ChartState* st,
                      int* n_active, std::vector<ChartState>& out, SepPrecond& P) {
#define RUV_CASE(L, UU) \
  if (sh.lpr == L && sh.unroll == UU) return run_pcg_sep<S, NR, L, UU>(ctx, sys, x64, o, T, st, n_active, out, P);
  RUV_SHAPES(RUV_CASE)
#undef RUV_CASE
  throw Error{RUV_ERR_BAD_INPUT, "unsupported SpMV shape"};
}

template <class S, int NR>
double dispatch_time(Shape sh, Ctx& ctx, DevSystem& sys, Tiles T, int reps, int nbuf, bool iter = false) {
#define RUV_CASE(L, UU) \
  if (sh.lpr == L && sh.unroll == UU) return time_spmv<S, NR, L, UU>(ctx, sys, T, reps, nbuf, iter);
  RUV_SHAPES(RUV_CASE)
#undef RUV_CASE
  throw Error{RUV_ERR_BAD_INPUT, "unsupported SpMV shape"};
}

TileTable make_tiles(const std::vector<int64_t>& chart_row, int64_t tile_rows) {
  TileTable T;
  int64_t nc = (int64_t)chart_row.size() - 1;
  T.chart_tile.assign(nc + 1, 0);
  for (int64_t c = 0; c < nc; ++c) {
    T.chart_tile[c] = (int64_t)T.chart.size();
    for (int64_t a = chart_row[c]; a < chart_row[c + 1]; a += tile_rows) {
      T.tab.push_back(a);
      T.tab.push_back(std::min(a + tile_rows, chart_row[c + 1]));
      T.chart.push_back((int32_t)c);
    }
  }
  T.chart_tile[nc] = (int64_t)T.chart.size();
  return T;
}

// 16-bit column stream, one thread per row: every entry as an offset from its chart's first
// row (all charts of at most 65536 rows), or with `rowrel` as an offset from its row's index
// minus 32768, *bad set where an entry lies more than 32767 rows from its row.
constexpr int64_t kNarrowRows = 65536;
__global__ void k_narrow_cols(int64_t n, const int64_t* __restrict__ chart_row, int64_t n_charts,
                              const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ cols, int rowrel,
                              uint16_t* __restrict__ c16, int* __restrict__ bad) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (rowrel) {
    for (int e = row_ptr[i]; e < row_ptr[i + 1]; ++e) {
      const int64_t d = (int64_t)cols[e] - i + kRowRelBias;
      if (d < 0 || d > 65535) {
        atomicOr(bad, 1);
        return;
      }
      c16[e] = (uint16_t)d;
    }
    return;
  }
  int64_t lo = 0, hi = n_charts;  // the chart of row i: largest c with chart_row[c] <= i
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (chart_row[mid] <= i) lo = mid; else hi = mid;
  }
  const int64_t r0 = chart_row[lo];
  for (int e = row_ptr[i]; e < row_ptr[i + 1]; ++e) c16[e] = (uint16_t)(cols[e] - r0);
}
__global__ void k_chart_base(int64_t n_charts, const int64_t* __restrict__ chart_row, int32_t* __restrict__ cbase) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n_charts) cbase[c] = (int32_t)chart_row[c];
}

}  // namespace

// The 16-bit column stream of a chart-blocked CSR operator: chart-relative (cbase = each
// chart's first row) when every chart has at most 65536 rows, else row-relative (*rowrel,
// cbase null) when every entry lies within 32767 rows of its row.  Returns false and leaves
// the pointers null otherwise (the one case that reads a flag back: only operators with a
// chart above 65536 rows pay that synchronisation).  RUV_NARROW_COLS=chart: chart-relative
// streams only.
bool narrow_operator(Ctx& ctx, int64_t n, int64_t nnz, int64_t n_charts, const std::vector<int64_t>& h_chart_row,
                     const int64_t* chart_row, const int32_t* row_ptr, const int32_t* cols, const std::string& tag,
                     uint16_t** c16, int32_t** cbase, bool* rowrel) {
  *c16 = nullptr;
  *cbase = nullptr;
  *rowrel = false;
  bool large = false;
  for (int64_t c = 0; c < n_charts; ++c)
    if (h_chart_row[c + 1] - h_chart_row[c] > kNarrowRows) large = true;
  const char* env = std::getenv("RUV_NARROW_COLS");
  if (large && env && std::string(env) == "chart") return false;
  cudaStream_t s = ctx.stream;
  uint16_t* d16 = ctx.ws.get<uint16_t>(tag + ".c16", std::max<int64_t>(nnz, 1));
  int32_t* dbase = large ? nullptr : ctx.ws.get<int32_t>(tag + ".cbase", std::max<int64_t>(n_charts, 1));
  int* bad = ctx.ws.get<int>(tag + ".c16bad", 1);
  RUV_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s));
  if (n > 0) {
    k_narrow_cols<<<div_up(n, 256), 256, 0, s>>>(n, chart_row, n_charts, row_ptr, cols, large ? 1 : 0, d16, bad);
    count_launches(1);
  }
  if (!large && n_charts > 0) {
    k_chart_base<<<div_up(n_charts, 256), 256, 0, s>>>(n_charts, chart_row, dbase);
    count_launches(1);
  }
  RUV_LAUNCH_CHECK();
  if (large) {
    int h = 0;
    RUV_CUDA(cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    RUV_CUDA(cudaStreamSynchronize(s));
    if (h != 0) return false;
  }
  *c16 = d16;
  *cbase = dbase;
  *rowrel = large;
  return true;
}

// On unless RUV_NARROW_COLS=0: on the 4096-disk operator the 16-bit stream cuts the SpMV's
// bytes by 18% and its time by 13% (0.215 -> 0.187 ms); RUV_NARROW_COLS=chart keeps it to
// charts of at most 65536 rows (larger charts then make the whole operator 32-bit).
void narrow_columns(Ctx& ctx, DevSystem& sys) {
  const char* e = std::getenv("RUV_NARROW_COLS");
  if (e && e[0] == '0') {  // 32-bit columns only
    sys.cols16 = nullptr;
    sys.cbase = nullptr;
    sys.rowrel16 = false;
    return;
  }
  narrow_operator(ctx, sys.n_rows, sys.nnz, sys.n_charts, sys.h_chart_row, sys.chart_row, sys.row_ptr, sys.cols,
                  "sys", &sys.cols16, &sys.cbase, &sys.rowrel16);
}

double bench_spmv(Ctx& ctx, DevSystem& sys, bool mixed, int reps, int n_buffers, double* bytes,
                  double* stream_bytes) {
  narrow_columns(ctx, sys);
  Tiles T = upload_tiles(ctx, sys, "bench", ctx.tile_rows);
  const Shape sh = pick_shape(ctx, sys);
  const double N = (double)sys.n_rows, NNZ = (double)sys.nnz, nr = (double)sys.nrhs;
  const double vb = mixed ? 4.0 : 8.0;
  // column bytes per entry: 2 with the 16-bit stream (every chart has it then), 4 otherwise
  const double cb = sys.cols16 ? 2.0 : 4.0;
  // algorithmic bytes: values, 32-bit columns, row pointers, p read once, q written; the
  // stream bytes count the columns the kernel actually reads (16-bit where narrowed)
  if (bytes) *bytes = NNZ * (vb + 4.0) + (N + 1.0) * 4.0 + 2.0 * N * nr * vb;
  if (stream_bytes) *stream_bytes = NNZ * (vb + cb) + (N + 1.0) * 4.0 + 2.0 * N * nr * vb;
  if (T.n == 0) return 0.0;
  if (sys.nrhs == 2)
    return mixed ? dispatch_time<float, 2>(sh, ctx, sys, T, reps, n_buffers)
                 : dispatch_time<double, 2>(sh, ctx, sys, T, reps, n_buffers);
  return dispatch_time<double, 1>(sh, ctx, sys, T, reps, n_buffers);
}

// Autotuner: time the batched SpMV for every instantiated (lanes per row, rows in flight)
// shape, tile height and SpMV form (CSR-vector or bulk-copy staged) on the assembled operator,
// each with the update, dots and direction kernels of a CG iteration over the same tiles (the
// tile height sets their grid too); keep the fastest in the context.
TuneResult autotune_spmv(Ctx& ctx, DevSystem& sys, bool mixed, int reps) {
  narrow_columns(ctx, sys);
  TuneResult best{0, 0, 0, 0, 1e30};
  const int tiles[] = {128, 256, 512, 1024};
  const Shape shapes[] = {
#define RUV_SH(L, UU) Shape{L, UU},
      RUV_SHAPES(RUV_SH)
#undef RUV_SH
  };
  const int saved_tile = ctx.tile_rows, saved_tma = ctx.spmv_tma;
  // the bulk-copy kernel exists for the mixed solver's two-column SpMV only
  const int n_tma = mixed && sys.nrhs == 2 ? 2 : 1;
  for (int tr : tiles) {
    ctx.tile_rows = tr;
    for (int tma = 0; tma < n_tma; ++tma) {
      ctx.spmv_tma = tma;
      Tiles T = upload_tiles(ctx, sys, "tune", ctx.tile_rows);
      if (T.n == 0) break;
      for (const Shape& sh : shapes) {
        double ms = sys.nrhs == 2 ? (mixed ? dispatch_time<float, 2>(sh, ctx, sys, T, reps, 2, true)
                                           : dispatch_time<double, 2>(sh, ctx, sys, T, reps, 2, true))
                                  : dispatch_time<double, 1>(sh, ctx, sys, T, reps, 2, true);
        if (ms < best.ms) best = TuneResult{sh.lpr, sh.unroll, tr, tma, ms};
      }
    }
  }
  if (best.lpr > 0) {
    ctx.lanes_per_row = best.lpr;
    ctx.unroll = best.unroll;
    ctx.tile_rows = best.tile_rows;
    ctx.tile_set = true;
    ctx.spmv_tma = best.tma;
  } else {
    ctx.tile_rows = saved_tile;
    ctx.spmv_tma = saved_tma;
  }
  return best;
}

std::vector<ChartResult> pcg_solve(Ctx& ctx, DevSystem& sys, double* x, const SolveOpts& o) {
  const bool sep = o.precond == RUV_PRECOND_AMG || o.precond == RUV_PRECOND_AMG_SA || o.precond == RUV_PRECOND_IC0 ||
                   o.precond == RUV_PRECOND_IC0_COLOR;
  if (o.precond != RUV_PRECOND_NONE && o.precond != RUV_PRECOND_JACOBI && !sep)
    throw Error{RUV_ERR_BAD_INPUT, "unknown preconditioner"};
  const int64_t NC = sys.n_charts;
  narrow_columns(ctx, sys);
  Tiles T = upload_tiles(ctx, sys, "pcg", o.teams ? solve_tile_rows(ctx, sys, o.precision == RUV_PREC_MIXED) : ctx.tile_rows);
  ChartState* st = ctx.ws.get<ChartState>("pcg.state", NC);
  int* n_active = ctx.ws.get<int>("pcg.nactive", 1);
  const bool mixed = o.precision == RUV_PREC_MIXED;
  const Shape sh = pick_shape(ctx, sys, !mixed && o.teams);
  std::vector<ChartState> out;
  ctx.timings[3] = 0.0;
  if (sep) {
    // preconditioner set-up, timed on the stream
    cudaEvent_t e[2];
    RUV_CUDA(cudaEventCreate(&e[0]));
    RUV_CUDA(cudaEventCreate(&e[1]));
    struct EvGuard {
      cudaEvent_t* e;
      ~EvGuard() {
        cudaEventDestroy(e[0]);
        cudaEventDestroy(e[1]);
      }
    } guard{e};
    RUV_CUDA(cudaEventRecord(e[0], ctx.stream));
    std::unique_ptr<SepPrecond> P = (o.precond == RUV_PRECOND_AMG || o.precond == RUV_PRECOND_AMG_SA)
                                        ? make_amg(ctx, sys, o.precond == RUV_PRECOND_AMG_SA, !o.teams)
                                        : make_ic0(ctx, sys, o.precond == RUV_PRECOND_IC0_COLOR);
    RUV_CUDA(cudaEventRecord(e[1], ctx.stream));
    RUV_CUDA(cudaEventSynchronize(e[1]));
    float ms = 0.f;
    RUV_CUDA(cudaEventElapsedTime(&ms, e[0], e[1]));
    ctx.timings[3] = ms;
    if (sys.nrhs == 2) {
      if (mixed) dispatch_pcg_sep<float, 2>(sh, ctx, sys, x, o, T, st, n_active, out, *P);
      else dispatch_pcg_sep<double, 2>(sh, ctx, sys, x, o, T, st, n_active, out, *P);
    } else {
      if (mixed) dispatch_pcg_sep<float, 1>(sh, ctx, sys, x, o, T, st, n_active, out, *P);
      else dispatch_pcg_sep<double, 1>(sh, ctx, sys, x, o, T, st, n_active, out, *P);
    }
  } else if (sys.nrhs == 2) {
    if (mixed) dispatch_pcg<float, 2>(sh, ctx, sys, x, o, T, st, n_active, out);
    else dispatch_pcg<double, 2>(sh, ctx, sys, x, o, T, st, n_active, out);
  } else {
    // the generic drop-in (one scalar right-hand side) runs in FP64 as the reference does
    dispatch_pcg<double, 1>(sh, ctx, sys, x, o, T, st, n_active, out);
  }
  std::vector<ChartResult> res(NC);
  for (int64_t c = 0; c < NC; ++c) {
    const ChartState& cs = out[c];
    if (cs.status == RUV_ERR_TIMEOUT)
      throw Error{RUV_ERR_TIMEOUT, "team solver: a bounded wait for a team's sums ran out (RUV_SPIN_LIMIT)"};
    res[c].status = cs.status;
    res[c].iters = cs.iters;
    res[c].refinements = cs.refinements;
    res[c].rel_res = cs.bnorm > 1e-300 ? std::sqrt(cs.rr) / cs.bnorm : std::sqrt(cs.rr);
  }
  return res;
}


// ===================================================================== no-alloc CG
// A variant of the FP64 PCG behind ruv_cg_solve for callers that cannot allocate device
// memory: its scratch (the CG vectors, the inverse diagonal, tile partials, tile table and
// solver state) lives in one file-scope __device__ array of fixed size instead of the
// context workspace, the caller's device buffers hold the system and the solution, and
// the host loop issues plain launches (no CUDA graph, no pinned staging).
namespace {

constexpr int64_t kNoAllocMaxRows = RUV_NOALLOC_MAX_ROWS;
constexpr int kNoAllocTile = 256;
constexpr int64_t kNoAllocMaxTiles = (kNoAllocMaxRows + kNoAllocTile - 1) / kNoAllocTile;

struct NoAllocScratch {
  double r[kNoAllocMaxRows], z[kNoAllocMaxRows], p[kNoAllocMaxRows], q[kNoAllocMaxRows];
  double dinv[kNoAllocMaxRows], diag[kNoAllocMaxRows];
  double part[3 * kNoAllocMaxTiles];
  int64_t tab[2 * kNoAllocMaxTiles];
  int64_t chart_tile[2];
  int32_t tchart[kNoAllocMaxTiles];
  ChartState st;
  int32_t n_active;
  int32_t bad;
  int32_t nonfinite;
};

// The allocation-free solve's scratch (about 12.6 MB).  A __device__ array belongs to the
// module instance of this file, and every CUDA context that loads the module gets its own
// copy, mapped when the module loads (under CUDA's default lazy loading: the first launch or
// symbol query in that context) and held until the context ends.  Host code may not use the
// symbol's name as a device pointer; the entry point resolves the address in the current
// context on every call (a host-side lookup once the module is loaded), so a context other
// than the device's primary one, or a context created again after cudaDeviceReset, never
// sees an address of another context.
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

__global__ void k_na_check_ptr(int32_t n, const int32_t* __restrict__ row_ptr, int32_t* __restrict__ bad) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && row_ptr[0] != 0) atomicExch(bad, 1);
  if (i < n && row_ptr[i + 1] < row_ptr[i]) atomicExch(bad, 1);
}

// Column check, diagonal extraction (first entry on the diagonal, as CsrMatrix::row_get)
// and the single-chart tile table.
__global__ void k_na_setup(int32_t n, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ cols,
                           const double* __restrict__ vals, NoAllocScratch* __restrict__ S) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    double d = 0.0;
    bool found = false;
    for (int32_t k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
      const int32_t c = cols[k];
      if (c < 0 || c >= n) atomicExch(&S->bad, 2);
      if (c == i && !found) {
        d = vals[k];
        found = true;
      }
    }
    S->diag[i] = d;
  }
  const int64_t n_tiles = (n + kNoAllocTile - 1) / kNoAllocTile;
  if (i < n_tiles) {
    S->tab[2 * i] = i * kNoAllocTile;
    S->tab[2 * i + 1] = min((int64_t)n, (i + 1) * kNoAllocTile);
    S->tchart[i] = 0;
  }
  if (i == 0) {
    S->chart_tile[0] = 0;
    S->chart_tile[1] = n_tiles;
  }
}

__global__ void k_na_nonfinite(int32_t n, const double* __restrict__ x, int32_t* __restrict__ flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !isfinite(x[i])) atomicExch(flag, 1);
}

void na_message(char* msg, int32_t len, const char* text) {
  if (msg && len > 0) {
    std::snprintf(msg, (size_t)len, "%s", text);
  }
}

template <int LPR, int U>
void na_iterations(cudaStream_t s, NoAllocScratch* S, Tiles T, const int32_t* row_ptr, const int32_t* cols,
                   const double* vals, double* x, int jac, int none, int64_t max_iter) {
  k_spmv_pq_k<double, 1, LPR, U, false><<<(unsigned)T.n, kTileThreads, 0, s>>>(T, &S->st, row_ptr, cols, nullptr, nullptr,
                                                                              vals, S->p, S->q, S->part, NoStep());
  ChartStep f;
  f.precond_none = none;
  f.max_iter = max_iter;
  f.st = &S->st;
  f.n_active = &S->n_active;
  f.kind = kStepAlpha;
  k_chart_step<1><<<1, kChartThreads, 0, s>>>(T, f, S->part);
  k_update<double, 1><<<(unsigned)T.n, kTileThreads, 0, s>>>(T, &S->st, S->dinv, jac, x, S->r, S->z, S->p, S->q, S->part, NoStep());
  f.kind = kStepBeta;
  k_chart_step<2><<<1, kChartThreads, 0, s>>>(T, f, S->part);
  k_direction<double, 1><<<(unsigned)T.n, kTileThreads, 0, s>>>(T, &S->st, S->z, S->p);
}

}  // namespace
}  // namespace ruv

extern "C" ruv_status ruv_cg_solve_noalloc(int32_t n, const int32_t* row_ptr, const int32_t* cols, const double* vals,
                                           const double* b, double* x, int64_t max_iter, double tol, ruv_precond pc,
                                           int64_t* iters_out, void* stream, char* msg, int32_t msg_len) {
  using namespace ruv;
  if (n <= 0 || !row_ptr || !cols || !vals || !b || !x) {
    na_message(msg, msg_len, "empty system or null device pointer");
    return RUV_ERR_BAD_INPUT;
  }
  if ((int64_t)n > kNoAllocMaxRows) {
    char buf[160];
    std::snprintf(buf, sizeof(buf), "n = %d exceeds the no-alloc scratch maximum of %lld rows (RUV_NOALLOC_MAX_ROWS)",
                  (int)n, (long long)kNoAllocMaxRows);
    na_message(msg, msg_len, buf);
    return RUV_ERR_BAD_INPUT;
  }
  if (pc != RUV_PRECOND_NONE && pc != RUV_PRECOND_JACOBI) {
    na_message(msg, msg_len, "the no-alloc solve supports PRECOND_NONE and PRECOND_JACOBI");
    return RUV_ERR_BAD_INPUT;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    na_message(msg, msg_len, "no current CUDA device");
    return RUV_ERR_NO_DEVICE;
  }
  // The scratch's address in the current context (see g_noalloc_scratch).
  NoAllocScratch* S = nullptr;
  {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr) {
      cudaGetLastError();
      na_message(msg, msg_len, "cudaGetSymbolAddress of the no-alloc scratch failed");
      return RUV_ERR_NO_DEVICE;
    }
    S = static_cast<NoAllocScratch*>(ptr);
  }
  auto launch_fail = [&](const char* what) {
    cudaGetLastError();
    na_message(msg, msg_len, what);
    return RUV_ERR_LAUNCH;
  };
  // flags that must start at zero on every call (the scratch keeps the last call's contents)
  if (cudaMemsetAsync(&S->n_active, 0, 3 * sizeof(int32_t), s) != cudaSuccess) return launch_fail("memset");
  const unsigned grid_n = div_up((int64_t)n + 1, 256);
  k_na_check_ptr<<<grid_n, 256, 0, s>>>(n, row_ptr, &S->bad);
  int32_t flags[3] = {0, 0, 0};
  if (cudaMemcpyAsync(flags, &S->n_active, sizeof(flags), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return launch_fail("row pointer check failed to run");
  if (flags[1]) {
    na_message(msg, msg_len, "row_ptr[0] != 0 or row_ptr not monotone");
    return RUV_ERR_BAD_INPUT;
  }
  k_na_setup<<<grid_n, 256, 0, s>>>(n, row_ptr, cols, vals, S);
  int32_t nnz = 0;
  if (cudaMemcpyAsync(flags, &S->n_active, sizeof(flags), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpyAsync(&nnz, row_ptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return launch_fail("set-up kernel failed");
  if (flags[1]) {
    na_message(msg, msg_len, "column index out of range");
    return RUV_ERR_BAD_INPUT;
  }
  const int jac = pc == RUV_PRECOND_JACOBI ? 1 : 0, none = pc == RUV_PRECOND_NONE ? 1 : 0;
  const int64_t n_tiles = (n + kNoAllocTile - 1) / kNoAllocTile;
  Tiles T{S->tab, S->tchart, S->chart_tile, n_tiles};
  k_dinv<double><<<div_up(n, kTileThreads), kTileThreads, 0, s>>>(n, S->diag, S->dinv);
  k_init<double, 1><<<(unsigned)n_tiles, kTileThreads, 0, s>>>(T, b, S->diag, S->dinv, jac, x, nullptr, S->r, S->z, S->p,
                                                               S->part, nullptr, nullptr);
  k_chart_init<<<1, kChartThreads, 0, s>>>(T, &S->st, S->part, tol, none, &S->n_active);
  const double avg = (double)nnz / (double)n;
  const int lpr = avg <= 5 ? 4 : avg <= 12 ? 8 : avg <= 24 ? 16 : 32;
  int64_t launched = 0;
  for (;;) {
    int32_t active = 0;
    if (cudaMemcpyAsync(&active, &S->n_active, sizeof(int32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return launch_fail("CG iteration failed");
    if (active <= 0 || launched >= max_iter + kCheckEvery) break;
    for (int k = 0; k < kCheckEvery; ++k) {
      if (lpr == 4) na_iterations<4, 2>(s, S, T, row_ptr, cols, vals, x, jac, none, max_iter);
      else if (lpr == 8) na_iterations<8, 4>(s, S, T, row_ptr, cols, vals, x, jac, none, max_iter);
      else if (lpr == 16) na_iterations<16, 1>(s, S, T, row_ptr, cols, vals, x, jac, none, max_iter);
      else na_iterations<32, 1>(s, S, T, row_ptr, cols, vals, x, jac, none, max_iter);
    }
    if (cudaGetLastError() != cudaSuccess) return launch_fail("CG kernel launch failed");
    launched += kCheckEvery;
  }
  ChartState st;
  k_na_nonfinite<<<div_up(n, 256), 256, 0, s>>>(n, x, &S->nonfinite);
  if (cudaMemcpyAsync(&st, &S->st, sizeof(st), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpyAsync(flags, &S->n_active, sizeof(flags), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return launch_fail("reading the solver state failed");
  if (iters_out) *iters_out = st.iters;
  if (st.status != RUV_OK) {
    na_message(msg, msg_len, st.status == RUV_ERR_NOT_CONVERGED ? "CG did not converge within max_iter" : "CG breakdown");
    return (ruv_status)st.status;
  }
  if (flags[2]) {
    na_message(msg, msg_len, "non-finite solution");
    return RUV_ERR_BREAKDOWN;
  }
  na_message(msg, msg_len, "");
  return RUV_OK;
}
