// Team solver: one thread-block cluster runs the whole preconditioned conjugate-gradient loop of a
// chart -- SpMV, updates, reductions, refreshes, the AMG V-cycle or the IC(0) sweeps, convergence --
// in one kernel, for every chart up to a size.
//
// What bounds a small chart is not bytes but steps: an iteration of the launch-per-step loop
// (pcg.cu) is 5 to 36 kernels of 2 to 10 us each, whatever the chart's size, and every chart of a
// batch waits for the slowest.  Here a step ends at a cluster barrier (0.2-0.3 us measured for 2
// to 16 CTAs, against 1.4-1.7 us for a barrier over 152 CTAs and about 3 us with a reduction
// behind it), dot products cross the cluster through distributed shared memory, each chart stops
// when it converges, and no graph is built.  The charts in flight also stay in L2 from step to
// step, where the lockstep loop streams the whole batch from HBM in every kernel.
//
// A team is 1 to 16 CTAs of 512 threads (one row per thread where the chart is small enough); the
// rule is in team_solve), each with a contiguous share of the chart's rows, consecutive rows on
// consecutive threads.  Vectors live in global memory (they are the launch loop's own arrays) and
// are L1- or L2-resident; the cluster barrier's release/acquire orders them.  Scalars are formed by
// one lane per CTA from the same partial sums in the same order, so every CTA of a team decides
// alike and results do not depend on timing.  (FP64 adds have 64 clocks of latency and 1.6 results
// per clock and SM here: a reduction's last steps and the scalar divisions stay in one warp, and the
// divisions go to the integer pipe, fp64rn.cuh.)
#include "team_dev.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <functional>

namespace ruv {
namespace {

constexpr int kTeamThreads = 512;
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kTeamMaxCtas = 16;
struct TeamShared {
  ChartState st;                    // lane 0's scalars (the same bits in every CTA of the team)
  double part[2][2][kTeamWarps];    // [buffer][value][warp]
  double slot[2][2][kTeamMaxCtas];  // [buffer][value][CTA of the team]
  uint64_t slot_bar[2];             // completes when a buffer's slots have arrived
  double rz, alpha, beta;
  float alpha32, beta32;  // what FP32 vectors take of them
  double due, due2;       // the residual norm at which something is due, and its square_of
  int flag;
  uint64_t left[kTeamMaxCtas];  // per CTA of the team: kStaying, or the barrier it left before and how (team_leave)
  int32_t lvl_row[kTeamMaxLevels];  // the chart's first row and row count per level
  int32_t lvl_n[kTeamMaxLevels];
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
// v into CTA `rank`'s copy of *p, counted on its copy of *bar when it arrives
__device__ __forceinline__ void st_async(const double* p, const uint64_t* bar, uint32_t rank, double v) {
  uint32_t d, m;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(smem_addr(bar)), "r"(rank));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(d),
               "l"(__double_as_longlong(v)), "r"(m)
               : "memory");
}

// v into CTA `rank`'s copy of *p
__device__ __forceinline__ void st_cluster(const uint64_t* p, uint32_t rank, uint64_t v) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(d), "l"(v) : "memory");
}

struct Team {
  int ctas, rank, threads, id;  // id: this thread's number in the team
  int buf;
  uint32_t phase[2];
  mutable uint32_t bars;  // cluster barriers passed: the same number in every CTA at the same barrier
  // every thread of the team; global and shared writes before it are visible after it
  __device__ __forceinline__ void bar() const {
    if (ctas == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
      ++bars;
    }
  }
  // the same where a one-CTA team is already past a block barrier (team_reduce)
  __device__ __forceinline__ void publish() const {
    if (ctas > 1) bar();
  }
};

// tries of the wait for a team's partial sums (each of them suspends for a while by itself): a few
// seconds, far above the longest step (RUV_SPIN_LIMIT overrides; 0: every wait runs out at once)
constexpr int64_t kTeamSpin = int64_t(1) << 22;

enum : int { kGo = 0, kRefresh = 1, kStop = 2, kLost = 3 };

// The end of a team's kernel, for every CTA and however it got here; whether any wait of the team ran
// out.  A CTA whose wait for the others' sums ran out cannot know which way they go on, so it comes
// here while they may still be on their way -- and they need it: a cluster barrier counts every
// CTA, and shared memory that a peer may still write has to stay.  So it meets their barriers from here,
// one after another wherever theirs are in the code, until all have come: it sends no more sums, so the
// wait of each peer's next reduction runs out too, or that peer has ended with this one's last sums.
// A CTA announces itself, before its next barrier, by that barrier's number, and an announcement
// counts from that barrier on: an early look at a later one would send one CTA out ahead of the others.
constexpr uint32_t kStaying = 0, kLeft = 1, kLeftLost = 2;
__device__ __forceinline__ bool team_leave(const Team& tm, TeamShared& sh, bool lost) {
  if (tm.ctas == 1) return false;
  if ((int)threadIdx.x < tm.ctas)
    st_cluster(&sh.left[tm.rank], threadIdx.x, ((uint64_t)(tm.bars + 1) << 32) | (lost ? kLeftLost : kLeft));
  bool all, any;
  do {
    tm.bar();
    all = true;
    any = false;
    for (int k = 0; k < tm.ctas; ++k) {
      const uint64_t u = *const_cast<volatile uint64_t*>(&sh.left[k]);
      all = all && (uint32_t)u != kStaying && (int32_t)(tm.bars - (uint32_t)(u >> 32)) >= 0;
      any = any || (uint32_t)u == kLeftLost;
    }
  } while (!all);
  if (any)  // asynchronous stores of sums that nobody waited for land within a microsecond or so
    for (const long long t0 = clock64(); clock64() - t0 < (1 << 18);) {
    }
  return any;
}

// Sum of every thread's v over the team in a fixed order -- in T within a warp (of FP32 rows at most 32 a
// thread's share, below the launch loop's tile of 1,024), in FP64 from there -- then fn(totals) in one lane of every CTA;
// its return value comes back to every thread (kLost: the wait for the sums ran out).  The CTAs' sums travel as asynchronous stores into
// each peer's shared memory, counted by an mbarrier there, so nothing waits for global stores in
// flight: a cluster barrier took 1,470 clocks behind a step's stores where it takes 600 alone.  No
// thread gets past this before every thread of the team has reached it; it publishes no global
// memory in a team of several CTAs (Team::publish does).
template <int NV, class T, class Fn>
__device__ __forceinline__ int team_reduce(Team& tm, TeamShared& sh, int64_t limit, const T (&v)[NV], Fn fn) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, buf = tm.buf;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const T w = warp_sum(v[k]);
    if (lane == 0) sh.part[buf][k][wid] = (double)w;
  }
  __syncthreads();
  if (wid == 0) {
    // each value in a half of the warp: one chain of FP64 additions for both
    static_assert(NV <= 2 && kTeamWarps == 16 && kTeamMaxCtas == 16, "a value's terms are half a warp's lanes");
    const int value = NV == 2 ? lane >> 4 : 0, term = lane & 15;
    bool ok = true;
    double t = sh.part[buf][value][term];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (tm.ctas > 1) {
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&sh.slot_bar[buf])),
                     "r"((uint32_t)(8 * NV * tm.ctas))
                     : "memory");
      if (term < tm.ctas && lane < 16 * NV)
        st_async(&sh.slot[buf][value][tm.rank], &sh.slot_bar[buf], term, t);
      ok = mbar_wait(&sh.slot_bar[buf], tm.phase[buf], limit);
      ok = __all_sync(0xffffffffu, ok);
      t = term < tm.ctas ? sh.slot[buf][value][term] : 0.0;
      for (int o = tm.ctas >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    double tot[NV];
    tot[0] = t;
    if constexpr (NV == 2) tot[1] = __shfl_sync(0xffffffffu, t, 16);
    if (lane == 0) sh.flag = ok ? fn(tot) : (int)kLost;
  }
  __syncthreads();
  tm.phase[buf] ^= 1;
  tm.buf ^= 1;
  return sh.flag;
}

// A step over rows [r0 + q, r0 + end) of a level, q from place's on: for each, s = sum_e w(e) get(col(e,
// row)) by 2^ll lanes, then fin(row, early, s) in the row's first lane, where early(row) was loaded
// beside the gathers.  Offsets and entries do not change, so the first row's are loaded before the
// barrier in front of the step is waited for.  Trip counts are uniform in a warp.
struct Place {
  int32_t q, end, step;
  int sub, ll;
};
template <int NR, class Ptr, class Col, class W, class G, class Early, class Fin, class Bar>
__device__ __forceinline__ void level_step(const Place& at, int32_t r0, Ptr ptr, Col col, W w, G get, Early early, Fin fin,
                                           Bar bar) {
  using Vf = V<float, NR>;
  const int lanes = 1 << at.ll, off = at.q & ((32 >> at.ll) - 1);
  int32_t lo, hi, j[8];
  float a[8];
  auto entries = [&](int32_t e0, int32_t i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int32_t e = e0 + k * lanes;
      const bool in = e < hi;
      a[k] = in ? w(e) : 0.0f;
      j[k] = in ? col(e, i) : -1;
    }
  };
  auto head = [&](int32_t q) {
    const bool valid = q < at.end;
    lo = valid ? (int32_t)__ldg(ptr + r0 + q) : 0;
    hi = valid ? (int32_t)__ldg(ptr + r0 + q + 1) : 0;
    entries(lo + at.sub, r0 + q);
  };
  head(at.q);
  bar();
  for (int32_t g = at.q - off; g < at.end; g += at.step) {
    const int32_t q = g + off, i = r0 + q;
    if (q != at.q) head(q);
    decltype(early(0)) x;
    Vf v[8], s;
    if (q < at.end) x = early(i);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j[k] >= 0) v[k] = get(j[k]);
#pragma unroll
    for (int c = 0; c < NR; ++c) s.c[c] = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j[k] >= 0)
#pragma unroll
        for (int c = 0; c < NR; ++c) s.c[c] += a[k] * v[k].c[c];
    for (int32_t e0 = lo + at.sub + 8 * lanes; e0 < hi; e0 += 8 * lanes) {
      entries(e0, i);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (j[k] >= 0) v[k] = get(j[k]);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (j[k] >= 0)
#pragma unroll
          for (int c = 0; c < NR; ++c) s.c[c] += a[k] * v[k].c[c];
    }
    for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < NR; ++c) s.c[c] += __shfl_xor_sync(0xffffffffu, s.c[c], o);
    if (q < at.end && at.sub == 0) fin(i, x, s);
  }
}
// The n rows of a level over the team (alone: over its first CTA), by the operator's fewest lanes per
// row (from its row length), more while threads would idle, up to eight.
__device__ __forceinline__ Place place_of(const Team& tm, int32_t n, int fewest, bool alone) {
  const int32_t threads = alone ? kTeamThreads : tm.threads;
  int ll = fewest;
  while (ll < 3 && ((int64_t)n << (ll + 1)) <= threads) ++ll;
  return Place{tm.id >> ll, n, threads >> ll, tm.id & ((1 << ll) - 1), ll};
}

// The CTA's rows [r0, r1) of the system operator: in shared memory for the whole solve where they fit
// (a step that streams it then waits for its gathers alone), else where they are.  Row offsets and
// entries keep their global numbering.
template <class T>
struct OwnOp {
  int32_t r0, r1;
  const int32_t* rp;
  const T* val;
  const float* val32;  // the V-cycle's values
  const int32_t* c32;
  const uint16_t* c16;
  int kind;
  int32_t cb;
  __device__ __forceinline__ int32_t col(int32_t e, int32_t rb) const { return kind ? rb + (int32_t)c16[e] : c32[e]; }
  __device__ __forceinline__ int32_t base(int32_t i) const { return kind == 2 ? i - kRowRelBias : cb; }
  template <class S, int NR, class Get>
  __device__ __forceinline__ V<S, NR> row(const S* v, int32_t i, Get get) const {
    const int32_t rb = base(i);
    return entries_dot<S, NR>(
        rp[i], rp[i + 1], [&](int32_t e) { return v[e]; }, [&](int32_t e) { return col(e, rb); }, get);
  }
};

// One V(1,1) cycle of the chart (the launch-by-launch cycle is amg.cu vtail): lv[0].x = M^-1 lv[0].b.  The
// pre-smoothed values w D^-1 b of level 0 are there already (in x, or y under a tentative
// prolongator) and published; each restriction forms the next level's.  Levels of few rows (from
// `tail` on) run on the team's first CTA between block barriers.  `last` runs for each level-0 row as
// its value is stored; no barrier follows the last pass.
constexpr int32_t kTeamTail = 512;
template <int NR, class Op, class Last>
__device__ __forceinline__ void team_vcycle(const Team& tm, const TeamShared& sh, const TeamAmg& M, const Op& op, int chart,
                                            int f, int tail, Last last) {
  using Vf = V<float, NR>;
  struct Early {
    Vf a, b;
  };
  const bool first = tm.rank == 0;
  // the barrier in front of a step that reads what level k's steps wrote
  auto bar_after = [&](int k) {
    if (k >= tail) __syncthreads();
    else tm.bar();
  };
  for (int k = 0; k < f; ++k) {
    const TeamLevel& L = M.lv[k];
    const TeamLevel& C = M.lv[k + 1];
    // t = b - A x, x the pre-smoothed values
    const float* xp = L.smoothed ? L.x : L.y;
    if (k == 0) {
      for (int32_t i = op.r0 + (int32_t)threadIdx.x; i < op.r1; i += kTeamThreads) {
        const Vf bi = ldv<float, NR>(L.b, i);
        Vf t = op.template row<float, NR>(op.val32, i, [&](int32_t j) { return ldv<float, NR>(xp, j); });
#pragma unroll
        for (int c = 0; c < NR; ++c) t.c[c] = bi.c[c] - t.c[c];
        stv<float, NR>(L.t, i, t);
      }
    } else if (k < tail || first) {
      const Cols cols{L.cols, L.c16, L.kind, L.kind == 1 ? __ldg(L.cbase + chart) : 0};
      level_step<NR>(
          place_of(tm, sh.lvl_n[k], L.a_lanes, k >= tail), sh.lvl_row[k], L.rp,
          [&](int32_t e, int32_t i) { return cols.at(e, cols.base(i)); }, [&](int32_t e) { return __ldg(L.vals + e); },
          [&](int32_t j) { return ldv<float, NR>(xp, j); }, [&](int32_t i) { return ldv<float, NR>(L.b, i); },
          [&](int32_t i, const Vf& bi, const Vf& s) {
            Vf t;
#pragma unroll
            for (int c = 0; c < NR; ++c) t.c[c] = bi.c[c] - s.c[c];
            stv<float, NR>(L.t, i, t);
          },
          [&]() { bar_after(k); });
    }
    // b_c = R t and the coarse level's pre-smoothed values
    float* xc = C.smoothed && k + 1 < f ? C.x : C.y;
    if (k + 1 < tail || first) {
      level_step<NR>(
          place_of(tm, sh.lvl_n[k + 1], L.r_lanes, k + 1 >= tail), sh.lvl_row[k + 1], L.roff,
          [&](int32_t e, int32_t) { return __ldg(L.rc + e); }, [&](int32_t e) { return __ldg(L.rv + e); },
          [&](int32_t j) { return ldv<float, NR>(L.t, j); }, [&](int32_t i) { return M.omega * __ldg(C.dinv + i); },
          [&](int32_t i, float wd, const Vf& s) {
            stv<float, NR>(C.b, i, s);
            Vf y;
#pragma unroll
            for (int c = 0; c < NR; ++c) y.c[c] = wd * s.c[c];
            stv<float, NR>(xc, i, y);
          },
          [&]() { bar_after(k); });
    } else if (k < tail) {
      tm.bar();  // (the first CTA's step has its barrier inside)
    }
  }
  if (f > 0) {
    if (f < tail) tm.bar();
    else if (first) __syncthreads();
  }
  {  // the last level: the dense inverse (symmetric: row i read along its columns), 8 lanes a row
    const TeamLevel& L = M.lv[f];
    const int32_t r0 = sh.lvl_row[f], m = sh.lvl_n[f];
    if (m > kTeamDirect) {  // aggregation stalled above the dense limit: x = D^-1 b
      if (f < tail || first)
        for (int32_t i = r0 + tm.id; i < r0 + m; i += f < tail ? tm.threads : kTeamThreads) {
          Vf v = ldv<float, NR>(L.b, i);
          const float d = __ldg(L.dinv + i);
#pragma unroll
          for (int c = 0; c < NR; ++c) v.c[c] *= d;
          stv<float, NR>(L.x, i, v);
          if (f == 0) last(i, v);
        }
    } else if (first) {
      const float* Ainv = M.fac + __ldg(M.fac_off + chart);
      const int i = threadIdx.x >> 3, sub = threadIdx.x & 7;  // 64 rows x 8 lanes = one CTA
      Vf s;
#pragma unroll
      for (int c = 0; c < NR; ++c) s.c[c] = 0.0f;
      if (i < m) {
#pragma unroll
        for (int q = 0; q < kTeamDirect / 8; ++q) {
          const int j = sub + 8 * q;
          const float a = j < m ? __ldg(Ainv + i * m + j) : 0.0f;
          const Vf b = ldv<float, NR>(L.b, r0 + (j < m ? j : 0));
#pragma unroll
          for (int c = 0; c < NR; ++c) s.c[c] += a * b.c[c];
        }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < NR; ++c) s.c[c] += __shfl_xor_sync(0xffffffffu, s.c[c], o);
      if (i < m && sub == 0) {
        stv<float, NR>(L.x, r0 + i, s);
        if (f == 0) last(r0 + i, s);
      }
    }
  }
  for (int k = f - 1; k >= 0; --k) {
    const TeamLevel& L = M.lv[k];
    const float* xc = M.lv[k + 1].x;
    const bool mine = k < tail || first;
    const int32_t r0 = sh.lvl_row[k], n = sh.lvl_n[k];
    // (a chain of steps on the first CTA ends with the barrier in front of the first step of all)
    auto bar = [&]() { bar_after(k); };
    if (L.smoothed && mine)  // y = x + P x_c
      level_step<NR>(
          k == 0 ? Place{op.r0 - r0 + (int32_t)threadIdx.x, op.r1 - r0, kTeamThreads, 0, 0}
                 : place_of(tm, n, L.p_lanes, k >= tail),
          r0, L.poff, [&](int32_t e, int32_t) { return __ldg(L.pc + e); }, [&](int32_t e) { return __ldg(L.pv + e); },
          [&](int32_t j) { return ldv<float, NR>(xc, j); }, [&](int32_t i) { return ldv<float, NR>(L.x, i); },
          [&](int32_t i, Vf y, const Vf& s) {
#pragma unroll
            for (int c = 0; c < NR; ++c) y.c[c] += s.c[c];
            stv<float, NR>(L.y, i, y);
          },
          bar);
    // x = y + w D^-1 (b - A y); a tentative prolongator's y_j is the pre-smoothed value (kept in y) plus
    // alpha_c x_c[agg[j]], formed on the fly
    auto yval = [&](int32_t j) {
      Vf v = ldv<float, NR>(L.y, j);
      if (L.smoothed) return v;
      const Vf c = ldv<float, NR>(xc, __ldg(L.agg + j));
#pragma unroll
      for (int q = 0; q < NR; ++q) v.c[q] += M.alpha_c * c.c[q];
      return v;
    };
    auto early = [&](int32_t i) { return Early{ldv<float, NR>(L.b, i), yval(i)}; };
    auto fin = [&](int32_t i, const Early& x, const Vf& s) {
      const float wd = M.omega * __ldg(L.dinv + i);
      Vf z;
#pragma unroll
      for (int c = 0; c < NR; ++c) z.c[c] = x.b.c[c] + wd * (x.a.c[c] - s.c[c]);
      stv<float, NR>(L.x, i, z);
      if (k == 0) last(i, z);
    };
    if (k == 0) {
      tm.bar();
      for (int32_t i = op.r0 + (int32_t)threadIdx.x; i < op.r1; i += kTeamThreads) {
        const Early x = early(i);
        fin(i, x, op.template row<float, NR>(op.val32, i, yval));
      }
    } else if (mine) {
      const Cols cols{L.cols, L.c16, L.kind, L.kind == 1 ? __ldg(L.cbase + chart) : 0};
      level_step<NR>(
          place_of(tm, n, L.a_lanes, k >= tail), r0, L.rp,
          [&](int32_t e, int32_t i) { return cols.at(e, cols.base(i)); }, [&](int32_t e) { return __ldg(L.vals + e); }, yval,
          early, fin, bar);
    }
  }
}

// One triangular sweep of the chart, level by level (ic0.cu k_sweep): a row's index, entries and
// pivot are loaded a level ahead, so a level is one round of gathers, the chain of its subtractions
// and three FP64 operations for the quotient (rinv: the pivots' reciprocals).
template <class S, int NR>
struct SweepRow {
  int32_t i, b, d;  // row, first entry, the pivot's entry
  S a[4], pivot, rinv;
  int32_t j[4];
  __device__ __forceinline__ void load(int32_t idx, const int32_t* rows, const int64_t* ptr, const int32_t* col,
                                       const S* val, const S* inv) {
    i = __ldg(rows + idx);
    b = (int32_t)__ldg(ptr + i);
    d = (int32_t)__ldg(ptr + i + 1) - 1;
    pivot = __ldg(val + d);
    if constexpr (sizeof(S) == 8) rinv = __ldg(inv + i);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = b + k < d ? __ldg(val + b + k) : S(0);
      j[k] = b + k < d ? __ldg(col + b + k) : -1;
    }
  }
  template <class In, class Out>
  __device__ __forceinline__ void solve(const int32_t* col, const S* val, In in, const S* out, Out put) const {
    V<S, NR> s = in(i);
    V<S, NR> o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j[k] >= 0) o[k] = ldv<S, NR>(out, j[k]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j[k] >= 0)
#pragma unroll
        for (int c = 0; c < NR; ++c) s.c[c] -= a[k] * o[k].c[c];
    for (int32_t e = b + 4; e < d; ++e) {
      const S w = __ldg(val + e);
      const V<S, NR> g = ldv<S, NR>(out, __ldg(col + e));
#pragma unroll
      for (int c = 0; c < NR; ++c) s.c[c] -= w * g.c[c];
    }
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      if constexpr (sizeof(S) == 8) s.c[c] = div_by(s.c[c], pivot, rinv);
      else s.c[c] /= pivot;
    }
    put(i, s);
  }
};
template <class S, int NR, class In, class Out>
__device__ __forceinline__ void team_sweep(const Team& tm, const int32_t* rows, const int32_t* lvl, int nl,
                                           const int64_t* ptr, const int32_t* col, const S* val, const S* inv, In in,
                                           const S* out, Out put) {
  int32_t lo = __ldg(lvl), hi = __ldg(lvl + 1);
  SweepRow<S, NR> row;
  if (lo + tm.id < hi) row.load(lo + tm.id, rows, ptr, col, val, inv);
  for (int l = 0; l < nl; ++l) {
    const int32_t next = l + 1 < nl ? __ldg(lvl + l + 2) : hi;
    if (lo + tm.id < hi) {
      row.solve(col, val, in, out, put);
      for (int32_t idx = lo + tm.id + tm.threads; idx < hi; idx += tm.threads) {
        row.load(idx, rows, ptr, col, val, inv);
        row.solve(col, val, in, out, put);
      }
    }
    lo = hi;
    hi = next;
    if (lo + tm.id < hi) row.load(lo + tm.id, rows, ptr, col, val, inv);
    tm.bar();
  }
}

struct TeamSys {
  const int32_t* order;  // chart of each team of this launch
  const int64_t* chart_row;
  const int32_t *rp, *cols;
  const uint16_t* c16;
  const int32_t* cbase;
  int kind;
  int store_bytes;  // dynamic shared memory for a CTA's rows of the operator
};

// CTAs on an SM: the FP32 loop without a preconditioner of its own runs at 64 registers a thread, the others
// at 128.  Three of them spill (bytes a thread, stores / loads: k_team<float,2,0> 92 / 172, <float,2,1> 120 / 156,
// <double,2,2> 160 / 160; the rest 48 and less), and what is spilled comes back from L2, past an L1 that every
// cluster barrier empties.
template <class S, int PCK>
constexpr int team_per_sm() {
  return std::is_same<S, float>::value && PCK == 0 ? 2 : 1;
}

// PCK: 0 none or Jacobi, 1 AMG, 2 IC(0).
template <class S, int NR, int PCK>
__global__ void __launch_bounds__(kTeamThreads, team_per_sm<S, PCK>())
    k_team(const __grid_constant__ TeamSys A, const __grid_constant__ TeamLoop<S> P,
           const __grid_constant__ TeamAmg M, const __grid_constant__ TeamIc0 I) {
  constexpr bool mixed = std::is_same<S, float>::value;
  using Vs = V<S, NR>;
  __shared__ TeamShared sh;
  Team tm;
  tm.ctas = (int)cluster_size();
  tm.rank = (int)cluster_rank();
  tm.threads = tm.ctas * kTeamThreads;
  tm.id = tm.rank * kTeamThreads + (int)threadIdx.x;
  tm.buf = 0;
  tm.phase[0] = tm.phase[1] = 0;
  tm.bars = 0;
  const int chart = A.order[cluster_id()];
  auto set_due = [&](double norm) {
    sh.due = mixed ? fmax(norm, sh.st.tol_abs) : sh.st.tol_abs;  // (FP64: a tolerance below zero is met by nothing)
    sh.due2 = square_of(sh.due);
  };
  if (threadIdx.x < kTeamMaxCtas) sh.left[threadIdx.x] = kStaying;
  if (threadIdx.x == 0) {
    sh.st = P.st[chart];
    set_due(mixed ? P.delta * sh.st.r_ref : 0.0);
    sh.rz = sh.st.rz;
    for (int k = 0; k < 2; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh.slot_bar[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (sh.st.state != kActive) return;  // (the whole team)
  if (tm.ctas > 1) tm.bar();           // the whole team runs before anyone writes a peer's memory
  const int32_t r0 = (int32_t)A.chart_row[chart], r1 = (int32_t)A.chart_row[chart + 1];
  // this CTA's rows, and their part of the operator
  constexpr bool copies = PCK == 1 && !mixed;  // FP32 cycle under the FP64 loop
  const int32_t R0 = r0 + (int32_t)((int64_t)(r1 - r0) * tm.rank / tm.ctas);
  const int32_t R1 = r0 + (int32_t)((int64_t)(r1 - r0) * (tm.rank + 1) / tm.ctas);
  OwnOp<S> op{R0, R1, A.rp, P.vals, PCK == 1 ? M.lv[0].vals : nullptr, A.cols, A.c16, A.kind,
              A.kind == 1 ? A.cbase[chart] : 0};
  {
    extern __shared__ __align__(16) unsigned char store[];
    const int32_t e0 = A.rp[R0], ne = A.rp[R1] - e0;
    const int64_t need = (int64_t)ne * (int)(sizeof(S) + (copies ? 4 : 0) + (A.kind ? 2 : 4)) + 4 * (int64_t)(R1 - R0 + 1);
    if (need <= (int64_t)A.store_bytes) {
      S* v = reinterpret_cast<S*>(store);
      float* v32 = reinterpret_cast<float*>(v + ne);
      int32_t* rp = reinterpret_cast<int32_t*>(v32 + (copies ? ne : 0));
      int32_t* c32 = rp + (R1 - R0 + 1);
      uint16_t* c16 = reinterpret_cast<uint16_t*>(c32);
      for (int32_t k = threadIdx.x; k <= R1 - R0; k += kTeamThreads) rp[k] = A.rp[R0 + k];
      for (int32_t k = threadIdx.x; k < ne; k += kTeamThreads) {
        v[k] = P.vals[e0 + k];
        if (copies) v32[k] = M.lv[0].vals[e0 + k];
        if (A.kind) c16[k] = A.c16[e0 + k];
        else c32[k] = A.cols[e0 + k];
      }
      __syncthreads();
      op.rp = rp - R0;
      op.val = v - e0;
      op.val32 = copies ? v32 - e0 : reinterpret_cast<const float*>(v) - e0;
      op.c32 = c32 - e0;
      op.c16 = c16 - e0;
    }
  }
  int f = 0, tail = kTeamMaxLevels;
  if constexpr (PCK == 1) {
    f = M.final_lvl[chart];
    if ((int)threadIdx.x <= f) {
      const int64_t a = M.lv[threadIdx.x].chart_row[chart], b = M.lv[threadIdx.x].chart_row[chart + 1];
      sh.lvl_row[threadIdx.x] = (int32_t)a;
      sh.lvl_n[threadIdx.x] = (int32_t)(b - a);
    }
    __syncthreads();
    for (int k = f; k > 0; --k)
      if (sh.lvl_n[k] <= kTeamTail) tail = k;
  }
  // a row's r has its final value for the V-cycle: level 0's right-hand side and pre-smoothed values
  auto put_r = [&](int32_t i, const Vs& r) {
    if constexpr (PCK == 1) {
      const float wd = M.omega * __ldg(M.lv[0].dinv + i);
      V<float, NR> t, x;
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        t.c[c] = (float)r.c[c];
        x.c[c] = wd * t.c[c];
      }
      if (copies) stv<float, NR>(P.r32, i, t);
      stv<float, NR>(M.lv[0].smoothed ? M.lv[0].x : M.lv[0].y, i, x);
    }
  };

  // z = M^-1 r and the sums r.z, z.q of a separate preconditioner, then fn
  auto apply = [&](auto fn) -> int {
    S acc[2] = {S(0), S(0)};
    auto dots = [&](int32_t i, const Vs& zv) {
      const Vs rv = ldv<S, NR>(P.r, i), qv = ldv<S, NR>(P.q, i);
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        acc[0] += rv.c[c] * zv.c[c];
        acc[1] += zv.c[c] * qv.c[c];
      }
    };
    if constexpr (PCK == 1) {
      team_vcycle<NR>(tm, sh, M, op, chart, f, tail, [&](int32_t i, const V<float, NR>& z) {
        Vs zv;
#pragma unroll
        for (int c = 0; c < NR; ++c) zv.c[c] = (S)z.c[c];
        dots(i, zv);
      });
    } else if constexpr (PCK == 2) {
      const S* lv = static_cast<const S*>(I.lv);
      const S* tv = static_cast<const S*>(I.tv);
      S* y = static_cast<S*>(I.y);
      S* zp = I.to_orig ? static_cast<S*>(I.zp) : P.z;
      const int32_t* to = I.to_orig;
      team_sweep<S, NR>(
          tm, I.frows, I.flev + r0 + chart, I.fnl[chart], I.lptr, I.lc, lv, static_cast<const S*>(I.inv),
          [&](int32_t i) { return ldv<S, NR>(P.r, to ? __ldg(to + i) : i); }, y,
          [&](int32_t i, const Vs& v) { stv<S, NR>(y, i, v); });
      team_sweep<S, NR>(
          tm, I.brows, I.blev + r0 + chart, I.bnl[chart], I.tptr, I.tc, tv, static_cast<const S*>(I.inv),
          [&](int32_t i) { return ldv<S, NR>(y, i); }, zp, [&](int32_t i, const Vs& v) {
            stv<S, NR>(zp, i, v);
            if (to) stv<S, NR>(P.z, __ldg(to + i), v);
          });
      for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) dots(i, ldv<S, NR>(P.z, i));
    }
    const int flag = team_reduce<2, S>(tm, sh, P.spin_limit, acc, fn);
    if (PCK == 1) tm.publish();  // z (the sweeps' last barrier has published theirs)
    return flag;
  };
  auto zrow = [&](int32_t i) -> Vs {
    Vs z;
    if constexpr (PCK == 0) {
      z = ldv<S, NR>(P.r, i);
      const S di = P.jacobi ? __ldg(P.dinv + i) : S(1);
#pragma unroll
      for (int c = 0; c < NR; ++c) z.c[c] *= di;
    } else if constexpr (copies) {
      const V<float, NR> t = ldv<float, NR>(P.z32, i);
#pragma unroll
      for (int c = 0; c < NR; ++c) z.c[c] = (S)t.c[c];
    } else {
      z = ldv<S, NR>(P.z, i);
    }
    return z;
  };

  int flag = kGo;
  if constexpr (PCK != 0) {
    if constexpr (PCK == 1)
      for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) put_r(i, ldv<S, NR>(P.r, i));
    tm.bar();
    flag = apply([&](const double (&t)[2]) {
      sh.rz = t[0];
      return (int)kGo;
    });
    for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) stv<S, NR>(P.p, i, zrow(i));
    tm.bar();
  }
  while (flag < kStop) {
    // q = A p, p.q
    S pq[1] = {S(0)};
    for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) {
      const Vs pi = ldv<S, NR>(P.p, i);
      const Vs s = op.template row<S, NR>(op.val, i, [&](int32_t j) { return ldv<S, NR>(P.p, j); });
      stv<S, NR>(P.q, i, s);
#pragma unroll
      for (int c = 0; c < NR; ++c) pq[0] += pi.c[c] * s.c[c];
    }
    flag = team_reduce<1, S>(tm, sh, P.spin_limit, pq, [&](const double (&t)[1]) {
      if (fabs(t[0]) <= 1e-300 || !isfinite(t[0])) {  // solver.rs:505-508
        sh.st.status = RUV_ERR_BREAKDOWN;
        return (int)kStop;
      }
      sh.alpha = div_rn(sh.rz, t[0]);
      sh.alpha32 = (float)sh.alpha;
      return (int)kGo;
    });
    if (flag >= kStop) break;
    // x += alpha p, r -= alpha q; r.r and (plain loop) r.z
    const S alpha = mixed ? (S)sh.alpha32 : (S)sh.alpha;
    S rr[2] = {S(0), S(0)};
    for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) {
      Vs xv = ldv<S, NR>(P.x, i), rv = ldv<S, NR>(P.r, i);
      const Vs pv = ldv<S, NR>(P.p, i), qv = ldv<S, NR>(P.q, i);
      const S di = PCK == 0 && P.jacobi ? __ldg(P.dinv + i) : S(1);
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        xv.c[c] += alpha * pv.c[c];
        rv.c[c] -= alpha * qv.c[c];
        rr[0] += rv.c[c] * rv.c[c];
        if (PCK == 0) rr[1] += rv.c[c] * (rv.c[c] * di);
      }
      stv<S, NR>(P.x, i, xv);
      stv<S, NR>(P.r, i, rv);
      put_r(i, rv);
    }
    auto new_beta = [&](double rznew) {
      sh.beta = div_rn(rznew, sh.rz);
      sh.beta32 = (float)sh.beta;
      sh.rz = rznew;
    };
    flag = team_reduce<2, S>(tm, sh, P.spin_limit, rr, [&](const double (&t)[2]) {
      sh.st.iters += 1;
      const bool due = at_most(t[0], sh.due, sh.due2);
      if constexpr (mixed) {
        // the FP32 residual only schedules true-residual refreshes
        if (due || !isfinite(t[0]) || sh.st.iters >= P.max_iter) return (int)kRefresh;
      } else {
        sh.st.rr = t[0];
        if (due) {
          sh.st.status = RUV_OK;
          return (int)kStop;
        }
        if (PCK != 0 && !isfinite(t[0])) {
          sh.st.status = RUV_ERR_BREAKDOWN;
          return (int)kStop;
        }
        if (sh.st.iters >= P.max_iter) {
          sh.st.status = RUV_ERR_NOT_CONVERGED;
          return (int)kStop;
        }
      }
      if (PCK == 0) new_beta(P.jacobi ? t[1] : t[0]);
      return (int)kGo;
    });
    if (flag >= kStop) break;
    bool fresh = false;
    if constexpr (mixed) {
      if (flag == kRefresh) {
        fresh = true;
        // fold the FP32 increment into the double-float solution, then r = b - A x (pcg.cu
        // k_fold, k_true_residual)
        for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) {
          DF<NR> xv = lddf<NR>(P.xdf, i);
          const V<float, NR> dv = ldv<float, NR>(P.x, i);
          V<float, NR> zero;
#pragma unroll
          for (int c = 0; c < NR; ++c) {
            float s2, e2;
            two_sum(xv.h[c], dv.c[c], s2, e2);
            e2 += xv.l[c];
            xv.h[c] = s2 + e2;
            xv.l[c] = e2 - (xv.h[c] - s2);
            zero.c[c] = 0.0f;
          }
          stdf<NR>(P.xdf, i, xv);
          stv<float, NR>(P.x, i, zero);
        }
        tm.bar();
        const float rsc = sh.st.rscale;
        float acc[2] = {0.0f, 0.0f};
        for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) {
          const int32_t lo = op.rp[i], hi = op.rp[i + 1], rb = op.base(i);
          const DF<NR> xi = lddf<NR>(P.xdf, i);
          float Sh[NR], Sl[NR];
#pragma unroll
          for (int c = 0; c < NR; ++c) Sh[c] = Sl[c] = 0.0f;
          for (int32_t e0 = lo; e0 < hi; e0 += 4) {  // four neighbours in flight
            float ah[4], al[4];
            DF<NR> xj[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (e0 + q < hi) {
                ah[q] = (float)op.val[e0 + q];
                al[q] = __ldg(P.vals_lo + e0 + q);
                xj[q] = lddf<NR>(P.xdf, op.col(e0 + q, rb));
              }
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (e0 + q < hi)
#pragma unroll
                for (int c = 0; c < NR; ++c) {
                  float dh, dl;
                  two_sum(xj[q].h[c], -xi.h[c], dh, dl);
                  dl += xj[q].l[c] - xi.l[c];
                  df_fma(ah[q], al[q], dh, dl, Sh[c], Sl[c]);
                }
          }
          const float2 rs = __ldg(P.rsum + i);
          const DF<NR> bv = lddf<NR>(P.bdf, i);
          const float di = PCK == 0 && P.jacobi ? __ldg(P.dinv + i) : 1.0f;
          V<float, NR> rv;
#pragma unroll
          for (int c = 0; c < NR; ++c) {
            float th = 0.0f, tl = 0.0f;  // A x = rs x_i + S
            df_fma(rs.x, rs.y, xi.h[c], xi.l[c], th, tl);
            float ah2, ae2;
            two_sum(th, Sh[c], ah2, ae2);
            const float axl = tl + Sl[c] + ae2;
            float uh, ue;  // r = b - A x
            two_sum(bv.h[c], -ah2, uh, ue);
            ue += bv.l[c] - axl;
            rv.c[c] = uh + ue;
            const float t = rv.c[c] * rsc;
            acc[0] += t * t;
            acc[1] += t * (rv.c[c] * di * rsc);
          }
          stv<float, NR>(P.r, i, rv);
          put_r(i, rv);
        }
        flag = team_reduce<2, float>(tm, sh, P.spin_limit, acc, [&](const double (&t)[2]) {
          const double inv = 1.0 / ((double)rsc * (double)rsc);
          sh.st.refinements += 1;
          sh.st.rr = t[0] * inv;
          const double rn = sqrt(sh.st.rr);
          if (rn <= sh.st.tol_abs) {
            sh.st.status = RUV_OK;
            return (int)kStop;
          }
          if (!isfinite(rn)) {
            sh.st.status = RUV_ERR_BREAKDOWN;
            return (int)kStop;
          }
          if (sh.st.iters >= P.max_iter) {
            sh.st.status = RUV_ERR_NOT_CONVERGED;
            return (int)kStop;
          }
          sh.st.r_ref = rn;
          set_due(P.delta * rn);
          if constexpr (PCK == 0 && mixed) new_beta((P.jacobi ? t[1] : t[0]) * inv);
          return (int)kGo;
        });
        if (flag >= kStop) break;
      }
    }
    if constexpr (PCK != 0) {
      tm.publish();  // r, for the rows other CTAs own
      flag = apply([&](const double (&t)[2]) {
        // flexible (Polak-Ribiere) for the V-cycle using r_new - r_old = -alpha q, Fletcher-Reeves
        // for IC(0) and right after a refresh (pcg.cu k_chart_beta_pc)
        double beta = div_rn(PCK == 1 && !fresh ? -sh.alpha * t[1] : t[0], sh.rz);
        if (!isfinite(beta)) beta = 0.0;
        sh.beta = beta;
        sh.beta32 = (float)beta;
        sh.rz = t[0];
        return (int)kGo;
      });
      if (flag >= kStop) break;
    }
    // p = z + beta p
    const S beta = mixed ? (S)sh.beta32 : (S)sh.beta;
    for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) {
      const Vs zv = zrow(i);
      Vs pv = ldv<S, NR>(P.p, i);
#pragma unroll
      for (int c = 0; c < NR; ++c) pv.c[c] = zv.c[c] + beta * pv.c[c];
      stv<S, NR>(P.p, i, pv);
    }
    tm.bar();
  }
  if constexpr (mixed) {  // fold what is pending; the FP64 solution is hi + lo
    for (int32_t i = R0 + (int32_t)threadIdx.x; i < R1; i += kTeamThreads) {
      DF<NR> xv = lddf<NR>(P.xdf, i);
      const V<float, NR> dv = ldv<float, NR>(P.x, i);
      V<float, NR> zero;
      V<double, NR> x;
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        float s2, e2;
        two_sum(xv.h[c], dv.c[c], s2, e2);
        e2 += xv.l[c];
        xv.h[c] = s2 + e2;
        xv.l[c] = e2 - (xv.h[c] - s2);
        zero.c[c] = 0.0f;
        x.c[c] = (double)xv.h[c] + (double)xv.l[c];
      }
      stdf<NR>(P.xdf, i, xv);
      stv<float, NR>(P.x, i, zero);
      stv<double, NR>(P.x64, i, x);
    }
  }
  const bool lost = team_leave(tm, sh, flag == kLost);
  if (tm.id == 0) {
    if (lost) sh.st.status = RUV_ERR_TIMEOUT;
    sh.st.state = kDone;
    sh.st.refresh = 0;
    P.st[chart] = sh.st;
    atomicSub(P.n_active, 1);
  }
}

// ---------------------------------------------------------------- which charts, and how many CTAs
// CTAs of a team for `want` CTAs' worth of work.
int team_ctas(int64_t want) {
  int c = 1;
  while (c < want && c < kTeamMaxCtas) c *= 2;
  return c;
}

// Bytes of a row of the operator in shared memory.
template <class S, int PCK>
double store_row(double per_row, bool narrow) {
  return per_row * (double)(sizeof(S) + (PCK == 1 && sizeof(S) == 8 ? 4 : 0) + (narrow ? 2 : 4)) + 4.0;
}

template <class S, int NR, int PCK>
void launch_team(cudaStream_t s, int ctas, int64_t n, int64_t rows, double per_row, TeamSys A, const TeamLoop<S>& P,
                 const TeamPrecond* pc) {
  auto k = k_team<S, NR, PCK>;
  // room for the largest chart's share of the operator (a CTA with more reads it from global memory),
  // as long as the CTAs that the registers allow on an SM still fit
  const int64_t want = (int64_t)(1.1 * store_row<S, PCK>(per_row, A.kind != 0) * (double)((rows + ctas - 1) / ctas)) + 1024;
  const int64_t most = (team_per_sm<S, PCK>() == 2 ? 104 : 200) * 1024;
  A.store_bytes = want <= most ? (int)((want + 15) & ~(int64_t)15) : 0;
  RUV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  if (ctas > 8) RUV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n * ctas));
  cfg.blockDim = dim3(kTeamThreads);
  cfg.dynamicSmemBytes = (size_t)A.store_bytes;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  static const TeamAmg no_amg{};
  static const TeamIc0 no_ic0{};
  RUV_CUDA(cudaLaunchKernelEx(&cfg, k, A, P, PCK == 1 ? pc->amg : no_amg, PCK == 2 ? pc->ic0 : no_ic0));
  count_launches(1);
}

}  // namespace

bool teams_on(const Ctx& ctx) {
  const char* e = std::getenv("RUV_TEAM");
  return !((e && e[0] == '0') || std::getenv("RUV_SPMV_TMA") || std::getenv("RUV_AMG_STAGE") || ctx.shape_forced);
}

void Ctx::team_streams(int n) {
  if (!team_go) RUV_CUDA(cudaEventCreateWithFlags(&team_go, cudaEventDisableTiming));
  for (int k = 0; k < n; ++k) {
    if (!team_done[k]) RUV_CUDA(cudaEventCreateWithFlags(&team_done[k], cudaEventDisableTiming));
    if (!team_stream[k]) RUV_CUDA(cudaStreamCreateWithFlags(&team_stream[k], cudaStreamNonBlocking));
  }
}

template <class S, int NR>
int64_t team_solve(Ctx& ctx, const DevSystem& sys, TeamLoop<S> loop, const TeamPrecond* pc) {
  const int64_t NC = sys.n_charts;
  const int kind = pc ? pc->kind : 0;
  constexpr bool mixed = std::is_same<S, float>::value;
  auto rows_of = [&](int64_t c) { return sys.h_chart_row[c + 1] - sys.h_chart_row[c]; };
  int64_t left = 0, largest = 0;
  for (int64_t c = 0; c < NC; ++c) largest = std::max(largest, rows_of(c));
  const char* le = std::getenv("RUV_SPIN_LIMIT");
  loop.spin_limit = le ? std::max<int64_t>(0, std::atoll(le)) : kTeamSpin;
  const char* re = std::getenv("RUV_TEAM_ROWS");
  // The largest chart a team of 16 SMs takes, where both ways were measured (ms, team / launch loop):
  // mixed Jacobi 47,500 rows 20.5 / 27.3, 66,600 31.1 / 33.3, 88,800 44.7 / 42.3; FP64 Jacobi, two columns,
  // 16,400 rows 11.3 / 14.8, 21,900 15.5 / 17.0, 25,000 20.4 / 18.0; V-cycle 32,000 rows mixed 5.8 / 6.4, FP64
  // 6.2 / 6.6, 89,000 mixed 11.9 / 9.4; colour-ordered IC(0) 14,400 rows 7.0 / 35.
  // One column: rows of at most 8 entries cost the loop one lane each, and the line lies at about as many
  // entries (7.5 a row, 25,000 rows 15.7 / 15.8, 30,000 16.6 / 16.2, 40,000 20.1 / 16.5; 5 a row, 40,000 rows
  // 13.9 / 14.0, 47,000 20.5 / 18.8), longer rows eight lanes and more (10 a row, 40,000 rows 21.3 / 23.4, 47,000
  // 24.1 / 23.2).  A team gives a row one thread whatever its length, so long rows lower every limit: Jacobi 47
  // entries a row, 40,000 rows 28.4 / 30.9; 94, 20,000 rows 11.0 / 11.8, 25,000 15.8 / 14.1, 40,000 29.8 / 21.1;
  // 187, 10,000 rows 6.0 / 6.5, 15,000 9.3 / 9.0.  V-cycle 47, 10,000 rows 6.6 / 7.2; 94, 5,000 rows 10.9 / 11.4,
  // 10,000 15.7 / 14.1, 30,000 24.0 / 16.8.  IC(0) 24, 40,000 rows 240 / 249; 47, 40,000 rows 475 / 459.
  const double per_row = sys.n_rows > 0 ? std::max(1.0, (double)sys.nnz / (double)sys.n_rows) : 1.0;
  const int64_t by_rows = kind == 1   ? (mixed ? 40000 : 32000)
                          : kind == 2 ? (mixed ? 90000 : 40000)
                          : mixed     ? 75000
                          : NR == 2   ? 23000
                                      : 43000;
  const double entries = kind == 1 ? 5e5 : kind == 2 ? 1.5e6 : !mixed && NR == 1 && per_row <= 8.0 ? 2e5 : 2e6;
  const int64_t most = re ? std::atoll(re) : std::min(by_rows, (int64_t)(entries / per_row));
  // a V-cycle is a chain of small steps, and a chart left to the other loop makes them all again: all
  // charts by teams, or none.  Teams hold 512 rows in flight on an SM where the launch loop's kernels
  // stream, so a batch of many rows is the other loop's, and the sooner the larger its charts are, whose
  // teams of 16 SMs then wait for each other (ms, team / loop, at a largest chart and rows in all).  AMG-SA mixed: 8,000
  // 646,000 8.1 / 8.5; 10,000 517,000 6.9 / 7.2, 609,000 8.2 / 7.9; 14,500 375,000 6.7 / 7.0, 555,000 8.9 / 8.3; 18,500
  // 335,000 6.3 / 6.9, 446,000 8.0 / 7.5; 24,000 404,000 7.8 / 7.7, 518,000 9.0 / 8.0.  AMG-SA FP64: 4,000 635,000 8.9 / 9.5;
  // 5,900 466,000 7.3 / 7.6; 8,000 212,000 4.7 / 5.5, 440,000 7.7 / 7.4; 10,000 167,000 4.9 / 5.1, 320,000 7.2 / 6.5; 23,500
  // 231,000 6.3 / 6.8, 348,000 8.3 / 7.8.  Tentative prolongators, cheaper cycles and more of them: mixed 14,900 691,000
  // 10.4 / 11.4, 19,400 446,000 8.5 / 9.1, 588,000 11.5 / 10.4; FP64 10,000 254,000 6.7 / 8.4, 517,000 11.4 / 11.5, 23,500 333,000
  // 9.1 / 10.2, 583,000 15.1 / 13.2.
  bool none = !teams_on(ctx) || (pc && kind == 0);
  if (kind == 1) {
    const bool sa = pc->amg.lv[0].smoothed != 0;
    const int64_t line = sa ? (mixed ? 10000 : 6000) : (mixed ? 16000 : 10000);
    const int64_t rows = largest <= line ? (sa || mixed ? 600000 : 500000)
                         : sa            ? (mixed ? 400000 : 250000)
                                         : (mixed ? 450000 : 350000);
    none = none || largest > most || sys.n_rows > rows;
  }
  // IC(0): a team of one CTA an SM has its chart's levels for itself, where the loop's sweeps hold several charts
  // an SM and end with the longest.  So batches whose charts wait for each other's SMs are the loop's: by
  // `waves`, the time of all teams over the longest chart's, a chart's taken as rows^1.25 (team / loop ms at waves.  Natural
  // order mixed: 1 5.9 / 8.9, 1.3 9.4 / 12.1, 1.5 4.2 / 4.5, 1.95 13.1 / 12.5, 2.6 56.8 / 40.7, 20,000 charts 108 / 44; FP64: 1 15.6 / 18.4,
  // 1.3 19.1 / 18.9, 1.5 7.5 / 6.8, 1.95 27.4 / 19.6, 20,000 charts 216 / 79.  Colours, whose levels are wide and few, teams of
  // one CTA mixed: 6 4.6 / 5.5, 26 16.7 / 16.8, 39 9.2 / 9.0; FP64: 5 22.0 / 25.1, 6 6.7 / 6.5, 26 25.6 / 21.9; of two mixed: 1.5 32.7 / 39.2, 1.8
  // 49.8 / 48.0; FP64: 1.5 44.9 / 51.6, 1.7 55.7 / 53.5; of four mixed: 1.2 44.8 / 41.2, 1.5 64.9 / 73.8, 1.75 83 / 80; FP64: 1 67 / 82,
  // 1.2 59.7 / 53.6, 1.5 93 / 91; of eight: 1.5 120 / 171 mixed, 161 / 208 FP64, 2.9 194 / 192 and 273 / 226; of sixteen
  // 2.2 122 / 270, 162 / 332).
  if (kind == 2 && !re && !none) {
    const bool colours = pc->ic0.to_orig != nullptr;
    const int ctas = team_ctas(std::max<int64_t>(1, pc->ic0.width / 256));
    const size_t slots = (size_t)std::max(1, ctx.sm_count / ctas);
    std::vector<double> cost;
    for (int64_t c = 0; c < NC; ++c)
      if (rows_of(c) > 0 && rows_of(c) <= most) cost.push_back(std::pow((double)rows_of(c), 1.25));
    std::sort(cost.begin(), cost.end(), std::greater<double>());
    double waves = 1.0, sum = 0.0;
    for (double c : cost) sum += c;
    if (cost.size() > slots) waves = std::max(sum / (double)slots, cost[slots - 1] + cost[slots]) / cost[0];
    none = waves > (!colours    ? (mixed ? 1.6 : 1.25)
                    : ctas == 1 ? (mixed ? 20.0 : 5.5)
                    : ctas == 2 ? (mixed ? 1.7 : 1.55)
                    : ctas == 4 ? (mixed ? 1.5 : 1.1)
                                : (mixed ? 2.8 : 2.1));
  }
  // Rows per CTA: as few as let every team run at once.  An FP32 step of one CTA of 512 threads costs
  // little more for two rows a thread, and its block barrier tens of clocks where a cluster's takes
  // over a thousand; FP64 rows are bound by the SM's FP64 pipe and spread out earlier.
  const char* pe = std::getenv("RUV_TEAM_PER");
  int64_t per = mixed ? (kind == 1 ? 512 : 1024) : 256;
  const int64_t slots = (mixed && kind == 0 ? 2 : 1) * (int64_t)ctx.sm_count, per_most = mixed ? 2048 : 1024;
  if (pe) {
    per = std::max(64, std::atoi(pe));
  } else if (kind != 2) {
    for (; per < per_most; per *= 2) {
      int64_t ctas = 0;
      for (int64_t c = 0; c < NC; ++c) ctas += rows_of(c) > 0 ? team_ctas((rows_of(c) + per - 1) / per) : 0;
      if (ctas <= slots) break;
    }
  }
  // charts by team size, the largest first within each
  std::vector<int32_t> cls[5];
  for (int64_t c = 0; c < NC; ++c) {
    const int64_t rows = rows_of(c);
    if (rows == 0) continue;
    if (none || rows > most) {
      ++left;
      continue;
    }
    const int64_t want = kind == 2 ? std::max<int64_t>(1, pc->ic0.width / 256) : (rows + per - 1) / per;
    cls[__builtin_ctz(team_ctas(want))].push_back((int32_t)c);
  }
  std::vector<int32_t> order;
  int64_t first[6] = {0};
  for (int k = 0; k < 5; ++k) {
    std::sort(cls[k].begin(), cls[k].end(), [&](int32_t a, int32_t b) {
      const int64_t na = sys.h_chart_row[a + 1] - sys.h_chart_row[a], nb = sys.h_chart_row[b + 1] - sys.h_chart_row[b];
      return na != nb ? na > nb : a < b;
    });
    order.insert(order.end(), cls[k].begin(), cls[k].end());
    first[k + 1] = (int64_t)order.size();
  }
  if (order.empty()) return left;
  cudaStream_t s = ctx.stream;
  int32_t* d_order = ctx.ws.get<int32_t>("team.order", (int64_t)order.size());
  void* h_order = ctx.team_pinned.get(sizeof(int32_t) * order.size());  // (every solve ends with a synchronisation)
  std::copy(order.begin(), order.end(), static_cast<int32_t*>(h_order));
  RUV_CUDA(cudaMemcpyAsync(d_order, h_order, sizeof(int32_t) * order.size(), cudaMemcpyHostToDevice, s));
  const int nw = !sys.cols16 ? 0 : sys.rowrel16 ? 2 : 1;
  // one launch per team size, side by side: each on a stream of its own between two events
  struct Join {
    Ctx& ctx;
    int used = 0;
    ~Join() {
      for (int k = 0; k < used; ++k) {
        cudaEventRecord(ctx.team_done[k], ctx.team_stream[k]);
        cudaStreamWaitEvent(ctx.stream, ctx.team_done[k], 0);
      }
    }
  } join{ctx};
  cudaStream_t main = ctx.stream;
  int classes = 0;
  for (int k = 0; k < 5; ++k) classes += first[k + 1] > first[k];
  if (classes > 1) {
    ctx.team_streams(classes - 1);
    RUV_CUDA(cudaEventRecord(ctx.team_go, main));
    for (int k = 0; k < classes - 1; ++k) RUV_CUDA(cudaStreamWaitEvent(ctx.team_stream[k], ctx.team_go, 0));
  }
  for (int k = 4; k >= 0; --k) {
    const int64_t n = first[k + 1] - first[k];
    if (n == 0) continue;
    cudaStream_t s = --classes == 0 ? main : ctx.team_stream[join.used++];
    const TeamSys A{d_order + first[k], sys.chart_row, sys.row_ptr, sys.cols, sys.cols16, sys.cbase, nw, 0};
    const int64_t rows = rows_of(order[first[k]]);  // the class's largest
    if (kind == 1) launch_team<S, NR, 1>(s, 1 << k, n, rows, per_row, A, loop, pc);
    else if (kind == 2) launch_team<S, NR, 2>(s, 1 << k, n, rows, per_row, A, loop, pc);
    else launch_team<S, NR, 0>(s, 1 << k, n, rows, per_row, A, loop, pc);
  }
  RUV_LAUNCH_CHECK();
  return left;
}

template int64_t team_solve<float, 2>(Ctx&, const DevSystem&, TeamLoop<float>, const TeamPrecond*);
template int64_t team_solve<double, 2>(Ctx&, const DevSystem&, TeamLoop<double>, const TeamPrecond*);
template int64_t team_solve<double, 1>(Ctx&, const DevSystem&, TeamLoop<double>, const TeamPrecond*);

}  // namespace ruv
