// Team solver: the whole conjugate-gradient loop of a chart, preconditioner included, in one
// kernel run by a team of CTAs (a thread-block cluster).  See team.cu.
#pragma once

#include "pcg.cuh"

namespace ruv {

constexpr int kTeamMaxLevels = 16;

// One level of the AMG hierarchy as the team kernel walks it (level 0: the system operator).
struct TeamLevel {
  const int64_t* chart_row;
  const int32_t *rp, *cols;
  const uint16_t* c16;
  const int32_t* cbase;
  int kind;  // column stream: 0 wide, 1 chart-relative, 2 row-relative
  const float *vals, *dinv;
  const int64_t *poff, *roff;
  const int32_t *pc, *rc, *agg;
  const float *pv, *rv;
  float *b, *x, *y, *t;
  int smoothed;
  int a_lanes, r_lanes, p_lanes;  // log2 of the fewest lanes per row of A, of R and of P
};
struct TeamAmg {
  const int32_t* final_lvl;
  const int64_t* fac_off;
  const float* fac;
  float alpha_c, omega;
  TeamLevel lv[kTeamMaxLevels];
};

// An IC(0) factor: rows by dependency level per chart for both sweeps (ic0.cu).  With to_orig
// the factor's rows are positions of the colour ordering.
struct TeamIc0 {
  const int32_t *frows, *flev, *fnl, *brows, *blev, *bnl;
  const int64_t *lptr, *tptr;
  const int32_t *lc, *tc;
  const void *lv, *tv, *inv;  // inv: 1 / pivot of each row
  void *y, *zp;
  const int32_t* to_orig;
  int64_t width;  // rows of the largest chart over its levels: how many rows a sweep has at a time
};

// What a separate preconditioner offers the team kernel (kind 0: nothing, it is applied by its
// own launches).
struct TeamPrecond {
  int kind = 0;  // 1: AMG V-cycle, 2: IC(0)
  TeamAmg amg{};
  TeamIc0 ic0{};
};

// The loop's arrays (those of pcg.cu) and controls.
template <class S>
struct TeamLoop {
  const S* vals;
  const S* dinv;
  S *x, *r, *z, *p, *q;  // x: the FP32 increment (mixed) or the solution
  double* x64;
  float *r32, *z32;  // FP64 loop: the FP32 preconditioner's vectors
  const float* vals_lo;
  const float2* rsum;
  const float* bdf;
  float* xdf;
  ChartState* st;
  int* n_active;
  int64_t max_iter;
  double delta;
  int jacobi;  // plain loop: 1 Jacobi, 0 none
  int64_t spin_limit = 0;  // tries of a wait for the team's sums (set by team_solve)
};

// Whether the kernels below may be used: not under RUV_TEAM=0 or a knob that picks a kernel of the
// launch-per-step loop (RUV_LPR, RUV_SPMV_TMA, RUV_AMG_STAGE).
bool teams_on(const Ctx& ctx);

// Solves every chart that a team is the faster way for and marks it done in loop.st (status
// RUV_ERR_TIMEOUT where a bounded wait ran out); returns the number of charts left.
template <class S, int NR>
int64_t team_solve(Ctx& ctx, const DevSystem& sys, TeamLoop<S> loop, const TeamPrecond* pc);

}  // namespace ruv
