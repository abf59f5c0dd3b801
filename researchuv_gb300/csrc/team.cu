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
// rule is in team_size.  Rows go round-robin over the team in blocks of 512, so consecutive threads
// read consecutive rows.  Vectors live in global memory (they are the launch loop's own arrays) and
// are L1- or L2-resident; the cluster barrier's release/acquire orders them.  Scalars are formed by
// one lane per CTA from the same partial sums in the same order, so every CTA of a team decides
// alike and results do not depend on timing.  (FP64 adds have 64 clocks of latency and 1.6 results
// per clock and SM here: a reduction's last steps and the scalar divisions stay in one warp.)
#include "team.cuh"

#include <algorithm>
#include <cstdlib>

namespace ruv {
namespace {

constexpr int kTeamThreads = 512;
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kTeamMaxCtas = 16;
constexpr float kTeamOmega = 2.0f / 3.0f;  // the V-cycle's Jacobi weight (amg.cu kOmega)
constexpr int kTeamDirect = 64;            // rows solved by the dense inverse (amg.cu kDirect)

struct TeamShared {
  ChartState st;                    // lane 0's scalars (the same bits in every CTA of the team)
  double part[2][2][kTeamWarps];    // [buffer][value][warp], as S
  unsigned long long slot[2][2][kTeamMaxCtas];  // [buffer][value][CTA of the team]: a double or a Pair
  uint64_t slot_bar[2];             // completes when a buffer's slots have arrived
  // the scalars, as a double or (mixed loop) a Pair, and what the vectors take of them
  unsigned long long s_rz, s_alpha;
  double alpha, beta;
  float alpha32, beta32;
  double due, due2;  // the residual norm at which something is due, and its square_of
  float due2f;
  int flag;
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
__device__ __forceinline__ void st_async(const unsigned long long* p, const uint64_t* bar, uint32_t rank,
                                         unsigned long long v) {
  uint32_t d, m;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(smem_addr(bar)), "r"(rank));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(d),
               "l"(v), "r"(m)
               : "memory");
}

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

struct Team {
  int ctas, rank, threads, id;  // id: this thread's number in the team
  int buf;
  uint32_t phase[2];
  // every thread of the team; global and shared writes before it are visible after it
  __device__ __forceinline__ void bar() const {
    if (ctas == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
    }
  }
  // the same where a one-CTA team is already past a block barrier (team_reduce)
  __device__ __forceinline__ void publish() const {
    if (ctas > 1) bar();
  }
};

// tries of the wait for a team's partial sums (each of them suspends for a while by itself): a few
// seconds, far above the longest step
constexpr int64_t kTeamSpin = int64_t(1) << 22;

enum : int { kGo = 0, kRefresh = 1, kStop = 2, kLost = 3 };

// Sum of every thread's v over the team in a fixed order, then fn(totals) in one lane of every CTA;
// its return value comes back to every thread.  The CTAs' sums travel as asynchronous stores into
// each peer's shared memory, counted by an mbarrier there, so nothing waits for global stores in
// flight: a cluster barrier took 1,470 clocks behind a step's stores where it takes 600 alone.  No
// thread gets past this before every thread of the team has reached it; it publishes no global
// memory in a team of several CTAs (Team::publish does).
template <int NV, class T, class Fn>
__device__ __forceinline__ int team_reduce(Team& tm, TeamShared& sh, const T (&v)[NV], Fn fn) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, buf = tm.buf;
  T* part = reinterpret_cast<T*>(sh.part[buf]);
  T w[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) w[k] = warp_sum(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) part[k * kTeamWarps + wid] = w[k];
  __syncthreads();
  using Sc = typename ScalarOf<T>::type;
  if (wid == 0) {
    Sc tot[NV];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      T t = part[k * kTeamWarps + (lane & (kTeamWarps - 1))];
#pragma unroll
      for (int o = kTeamWarps / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if constexpr (sizeof(T) == 4) tot[k] = pair_of(t);
      else tot[k] = t;
    }
    if (tm.ctas > 1) {
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&sh.slot_bar[buf])),
                     "r"((uint32_t)(8 * NV * tm.ctas))
                     : "memory");
      if (lane < tm.ctas)
#pragma unroll
        for (int k = 0; k < NV; ++k) st_async(&sh.slot[buf][k][tm.rank], &sh.slot_bar[buf], lane, sc_bits(tot[k]));
      ok = mbar_wait(&sh.slot_bar[buf], tm.phase[buf], kTeamSpin);
      ok = __all_sync(0xffffffffu, ok);
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        Sc t = lane < tm.ctas ? sc_of_bits(Sc{}, sh.slot[buf][k][lane]) : sc_zero(Sc{});
        for (int o = tm.ctas >> 1; o > 0; o >>= 1) t = sc_add(t, sc_shfl(t, o));
        tot[k] = t;
      }
    }
    if (lane == 0) sh.flag = ok ? fn(tot) : (int)kLost;
  }
  __syncthreads();
  tm.phase[buf] ^= 1;
  tm.buf ^= 1;
  return sh.flag;
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

// sum_e vals[e] get(col(e)) of one row, eight entries in flight (a mesh Laplacian's row in one
// sweep), entry order.
template <class S, int NR, class Get>
__device__ __forceinline__ V<S, NR> row_dot(const int32_t* rp, const Cols& cols, const S* vals, int32_t i, Get get) {
  const int32_t lo = __ldg(rp + i), hi = __ldg(rp + i + 1), rb = cols.base(i);
  V<S, NR> s;
#pragma unroll
  for (int c = 0; c < NR; ++c) s.c[c] = S(0);
  for (int32_t e0 = lo; e0 < hi; e0 += 8) {
    S a[8];
    int32_t j[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in = e0 + k < hi;
      a[k] = in ? __ldg(vals + e0 + k) : S(0);
      j[k] = in ? cols.at(e0 + k, rb) : -1;
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

// For each of the n rows from row r0 on: s = sum_e w(e) get(col(e, row)), by 2^ll lanes, then
// fin(row, s) in the row's first lane.  Trip counts are uniform, so every lane is in the shuffles.
template <int NR, class Ptr, class Col, class W, class G, class Fin>
__device__ __forceinline__ void level_rows(const Team& tm, int32_t r0, int32_t n, int ll, Ptr ptr, Col col, W w, G get,
                                           Fin fin) {
  const int lanes = 1 << ll, sub = tm.id & (lanes - 1), step = tm.threads >> ll;
  for (int32_t base = 0; base < n; base += step) {
    const int32_t q = base + (tm.id >> ll), i = r0 + q;
    const bool valid = q < n;
    const int32_t lo = valid ? (int32_t)__ldg(ptr + i) : 0, hi = valid ? (int32_t)__ldg(ptr + i + 1) : 0;
    V<float, NR> s;
#pragma unroll
    for (int c = 0; c < NR; ++c) s.c[c] = 0.0f;
    for (int32_t e0 = lo + sub; e0 < hi; e0 += 8 * lanes) {
      float a[8];
      int32_t j[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int32_t e = e0 + k * lanes;
        const bool in = e < hi;
        a[k] = in ? w(e) : 0.0f;
        j[k] = in ? col(e, i) : -1;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (j[k] >= 0) {
          const V<float, NR> g = get(j[k]);
#pragma unroll
          for (int c = 0; c < NR; ++c) s.c[c] += a[k] * g.c[c];
        }
    }
    for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < NR; ++c) s.c[c] += __shfl_xor_sync(0xffffffffu, s.c[c], o);
    if (sub == 0 && valid) fin(i, s);
  }
}

// log2 of the lanes per row for n rows on the team: the operator's fewest (from its row length),
// more while threads would idle, up to eight.
__device__ __forceinline__ int lanes_of(const Team& tm, int32_t n, int fewest) {
  int ll = fewest;
  while (ll < 3 && ((int64_t)n << (ll + 1)) <= tm.threads) ++ll;
  return ll;
}

// One V(1,1) cycle of the chart (the launch-by-launch cycle is amg.cu vtail): lv[0].x = M^-1 lv[0].b.
// `last` runs for each level-0 row as its value is stored; no barrier follows the last pass.
template <int NR, class Last>
__device__ __forceinline__ void team_vcycle(const Team& tm, const TeamShared& sh, const TeamAmg& M, int chart, int f,
                                            Last last) {
  using Vf = V<float, NR>;
  for (int k = 0; k < f; ++k) {
    const TeamLevel& L = M.lv[k];
    const Cols cols{L.cols, L.c16, L.kind, L.kind == 1 ? __ldg(L.cbase + chart) : 0};
    const int32_t n = sh.lvl_n[k];
    // t = b - A (w D^-1 b), the pre-smoothed neighbours formed on the fly
    level_rows<NR>(
        tm, sh.lvl_row[k], n, lanes_of(tm, n, L.a_lanes), L.rp,
        [&](int32_t e, int32_t i) { return cols.at(e, cols.base(i)); }, [&](int32_t e) { return __ldg(L.vals + e); },
        [&](int32_t j) {
          Vf v = ldv<float, NR>(L.b, j);
          const float wd = kTeamOmega * __ldg(L.dinv + j);
#pragma unroll
          for (int c = 0; c < NR; ++c) v.c[c] *= wd;
          return v;
        },
        [&](int32_t i, const Vf& s) {
          const Vf bi = ldv<float, NR>(L.b, i);
          Vf xi, ti;
          const float wd = kTeamOmega * __ldg(L.dinv + i);
#pragma unroll
          for (int c = 0; c < NR; ++c) {
            xi.c[c] = wd * bi.c[c];
            ti.c[c] = bi.c[c] - s.c[c];
          }
          if (L.smoothed) stv<float, NR>(L.x, i, xi);
          stv<float, NR>(L.t, i, ti);
        });
    tm.bar();
    // b_c = R t
    const int32_t nc = sh.lvl_n[k + 1];
    level_rows<NR>(
        tm, sh.lvl_row[k + 1], nc, lanes_of(tm, nc, L.r_lanes), L.roff,
        [&](int32_t e, int32_t) { return __ldg(L.rc + e); }, [&](int32_t e) { return __ldg(L.rv + e); },
        [&](int32_t j) { return ldv<float, NR>(L.t, j); },
        [&](int32_t i, const Vf& s) { stv<float, NR>(M.lv[k + 1].b, i, s); });
    tm.bar();
  }
  {  // the last level: the dense inverse (symmetric: row i read along its columns), 8 lanes a row
    const TeamLevel& L = M.lv[f];
    const int32_t r0 = sh.lvl_row[f], m = sh.lvl_n[f];
    if (m > kTeamDirect) {  // aggregation stalled above the dense limit: x = D^-1 b
      for (int32_t i = r0 + tm.id; i < r0 + m; i += tm.threads) {
        Vf v = ldv<float, NR>(L.b, i);
        const float d = __ldg(L.dinv + i);
#pragma unroll
        for (int c = 0; c < NR; ++c) v.c[c] *= d;
        stv<float, NR>(L.x, i, v);
        if (f == 0) last(i, v);
      }
    } else if (tm.rank == 0) {
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
    tm.bar();
    const TeamLevel& L = M.lv[k];
    const float* xc = M.lv[k + 1].x;
    const Cols cols{L.cols, L.c16, L.kind, L.kind == 1 ? __ldg(L.cbase + chart) : 0};
    const int32_t r0 = sh.lvl_row[k], n = sh.lvl_n[k];
    const int la = lanes_of(tm, n, L.a_lanes);
    auto col = [&](int32_t e, int32_t i) { return cols.at(e, cols.base(i)); };
    auto w = [&](int32_t e) { return __ldg(L.vals + e); };
    auto smooth = [&](auto yval) {  // x = y + w D^-1 (b - A y)
      level_rows<NR>(tm, r0, n, la, L.rp, col, w, yval, [&](int32_t i, const Vf& s) {
        const Vf bi = ldv<float, NR>(L.b, i), yi = yval(i);
        Vf xi;
        const float wd = kTeamOmega * __ldg(L.dinv + i);
#pragma unroll
        for (int c = 0; c < NR; ++c) xi.c[c] = yi.c[c] + wd * (bi.c[c] - s.c[c]);
        stv<float, NR>(L.x, i, xi);
        if (k == 0) last(i, xi);
      });
    };
    if (L.smoothed) {
      level_rows<NR>(
          tm, r0, n, lanes_of(tm, n, L.p_lanes), L.poff, [&](int32_t e, int32_t) { return __ldg(L.pc + e); },
          [&](int32_t e) { return __ldg(L.pv + e); }, [&](int32_t j) { return ldv<float, NR>(xc, j); },
          [&](int32_t i, const Vf& s) {
            Vf y = ldv<float, NR>(L.x, i);
#pragma unroll
            for (int c = 0; c < NR; ++c) y.c[c] += s.c[c];
            stv<float, NR>(L.y, i, y);
          });
      tm.bar();
      smooth([&](int32_t j) { return ldv<float, NR>(L.y, j); });
    } else {  // tentative: y_j = w D^-1_j b_j + alpha_c x_c[agg[j]] formed on the fly
      smooth([&](int32_t j) {
        Vf v = ldv<float, NR>(L.b, j);
        const float wd = kTeamOmega * __ldg(L.dinv + j);
        const Vf c = ldv<float, NR>(xc, __ldg(L.agg + j));
#pragma unroll
        for (int q = 0; q < NR; ++q) v.c[q] = wd * v.c[q] + M.alpha_c * c.c[q];
        return v;
      });
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
  const float* vals32;
};

// PCK: 0 none or Jacobi, 1 AMG, 2 IC(0).
template <class S, int NR, int PCK>
__global__ void __launch_bounds__(kTeamThreads, std::is_same<S, double>::value ? 1 : 2)
    k_team(const __grid_constant__ TeamSys A, const __grid_constant__ TeamLoop<S> P,
           const __grid_constant__ TeamAmg M, const __grid_constant__ TeamIc0 I) {
  constexpr bool mixed = std::is_same<S, float>::value;
  using Vs = V<S, NR>;
  using Sc = typename ScalarOf<S>::type;
  __shared__ TeamShared sh;
  Team tm;
  tm.ctas = (int)cluster_size();
  tm.rank = (int)cluster_rank();
  tm.threads = tm.ctas * kTeamThreads;
  tm.id = tm.rank * kTeamThreads + (int)threadIdx.x;
  tm.buf = 0;
  tm.phase[0] = tm.phase[1] = 0;
  const int chart = A.order[cluster_id()];
  auto set_due = [&](double norm) {
    sh.due = fmax(norm, sh.st.tol_abs);
    if constexpr (mixed) sh.due2f = square_of(0.0f, sh.due);
    else sh.due2 = square_of(0.0, sh.due);
  };
  if (threadIdx.x == 0) {
    sh.st = P.st[chart];
    set_due(mixed ? P.delta * sh.st.r_ref : 0.0);
    sh.s_rz = sc_bits(sc_from(Sc{}, sh.st.rz));
    for (int k = 0; k < 2; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh.slot_bar[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (sh.st.state != kActive) return;  // (the whole team)
  if (tm.ctas > 1) tm.bar();           // the whole team runs before anyone writes a peer's memory
  const int32_t r0 = (int32_t)A.chart_row[chart], r1 = (int32_t)A.chart_row[chart + 1];
  const Cols cols{A.cols, A.c16, A.kind, A.kind == 1 ? A.cbase[chart] : 0};
  int f = 0;
  if constexpr (PCK == 1) {
    f = M.final_lvl[chart];
    if ((int)threadIdx.x <= f) {
      const int64_t a = M.lv[threadIdx.x].chart_row[chart], b = M.lv[threadIdx.x].chart_row[chart + 1];
      sh.lvl_row[threadIdx.x] = (int32_t)a;
      sh.lvl_n[threadIdx.x] = (int32_t)(b - a);
    }
    __syncthreads();
  }
  constexpr bool copies = PCK == 1 && !mixed;  // FP32 cycle under the FP64 loop

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
      team_vcycle<NR>(tm, sh, M, chart, f, [&](int32_t i, const V<float, NR>& z) {
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
      for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) dots(i, ldv<S, NR>(P.z, i));
    }
    const int flag = team_reduce<2, S>(tm, sh, acc, fn);
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
    if constexpr (copies) {
      for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
        const Vs r = ldv<S, NR>(P.r, i);
        V<float, NR> t;
#pragma unroll
        for (int c = 0; c < NR; ++c) t.c[c] = (float)r.c[c];
        stv<float, NR>(P.r32, i, t);
      }
    }
    tm.bar();
    flag = apply([&](const Sc (&t)[2]) {
      sh.s_rz = sc_bits(t[0]);
      return (int)kGo;
    });
    for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) stv<S, NR>(P.p, i, zrow(i));
    tm.bar();
  }
  while (flag < kStop) {
    // q = A p, p.q
    S pq[1] = {S(0)};
    for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
      const Vs s = row_dot<S, NR>(A.rp, cols, P.vals, i, [&](int32_t j) { return ldv<S, NR>(P.p, j); });
      const Vs pi = ldv<S, NR>(P.p, i);
      stv<S, NR>(P.q, i, s);
#pragma unroll
      for (int c = 0; c < NR; ++c) pq[0] += pi.c[c] * s.c[c];
    }
    flag = team_reduce<1, S>(tm, sh, pq, [&](const Sc (&t)[1]) {
      if (vanishes(t[0]) || !isfinite(sc_hi(t[0]))) {  // solver.rs:505-508
        sh.st.status = RUV_ERR_BREAKDOWN;
        return (int)kStop;
      }
      const Sc alpha = sc_div(sc_of_bits(Sc{}, sh.s_rz), t[0]);
      sh.s_alpha = sc_bits(alpha);
      if constexpr (mixed) sh.alpha32 = alpha.h;
      else sh.alpha = alpha;
      return (int)kGo;
    });
    if (flag >= kStop) break;
    // x += alpha p, r -= alpha q; r.r and (plain loop) r.z
    const S alpha = mixed ? (S)sh.alpha32 : (S)sh.alpha;
    S rr[2] = {S(0), S(0)};
    for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
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
      if constexpr (copies) {
        V<float, NR> t;
#pragma unroll
        for (int c = 0; c < NR; ++c) t.c[c] = (float)rv.c[c];
        stv<float, NR>(P.r32, i, t);
      }
    }
    auto new_beta = [&](Sc rznew) {
      const Sc beta = sc_div(rznew, sc_of_bits(Sc{}, sh.s_rz));
      if constexpr (mixed) sh.beta32 = beta.h;
      else sh.beta = beta;
      sh.s_rz = sc_bits(rznew);
    };
    flag = team_reduce<2, S>(tm, sh, rr, [&](const Sc (&t)[2]) {
      sh.st.iters += 1;
      bool due;
      if constexpr (mixed) due = at_most(t[0].h, sh.due, sh.due2f);
      else due = at_most(t[0], sh.due, sh.due2);
      if constexpr (mixed) {
        // the FP32 residual only schedules true-residual refreshes
        if (due || !isfinite(sc_hi(t[0])) || sh.st.iters >= P.max_iter) return (int)kRefresh;
      } else {
        sh.st.rr = sc_f64(t[0]);
        if (due) {
          sh.st.status = RUV_OK;
          return (int)kStop;
        }
        if (PCK != 0 && !isfinite(sc_hi(t[0]))) {
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
        for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
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
        for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
          const int32_t lo = __ldg(A.rp + i), hi = __ldg(A.rp + i + 1), rb = cols.base(i);
          const DF<NR> xi = lddf<NR>(P.xdf, i);
          float Sh[NR], Sl[NR];
#pragma unroll
          for (int c = 0; c < NR; ++c) Sh[c] = Sl[c] = 0.0f;
#pragma unroll 4
          for (int32_t e = lo; e < hi; ++e) {
            const float ah = __ldg(P.vals + e), al = __ldg(P.vals_lo + e);
            const DF<NR> xj = lddf<NR>(P.xdf, cols.at(e, rb));
#pragma unroll
            for (int c = 0; c < NR; ++c) {
              float dh, dl;
              two_sum(xj.h[c], -xi.h[c], dh, dl);
              dl += xj.l[c] - xi.l[c];
              df_fma(ah, al, dh, dl, Sh[c], Sl[c]);
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
        }
        flag = team_reduce<2, float>(tm, sh, acc, [&](const Pair (&t)[2]) {
          const double inv = 1.0 / ((double)rsc * (double)rsc);
          sh.st.refinements += 1;
          sh.st.rr = t[0].f64() * inv;
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
          if constexpr (PCK == 0 && mixed) new_beta(pair_of((P.jacobi ? t[1] : t[0]).f64() * inv));
          return (int)kGo;
        });
        if (flag >= kStop) break;
      }
    }
    if constexpr (PCK != 0) {
      tm.publish();  // r, for the rows other CTAs own
      flag = apply([&](const Sc (&t)[2]) {
        // flexible (Polak-Ribiere) for the V-cycle using r_new - r_old = -alpha q, Fletcher-Reeves
        // for IC(0) and right after a refresh (pcg.cu k_chart_beta_pc)
        Sc beta = sc_div(PCK == 1 && !fresh ? sc_neg_mul(sc_of_bits(Sc{}, sh.s_alpha), t[1]) : t[0],
                         sc_of_bits(Sc{}, sh.s_rz));
        if (!isfinite(sc_hi(beta))) beta = sc_zero(beta);
        if constexpr (mixed) sh.beta32 = beta.h;
        else sh.beta = beta;
        sh.s_rz = sc_bits(t[0]);
        return (int)kGo;
      });
      if (flag >= kStop) break;
    }
    // p = z + beta p
    const S beta = mixed ? (S)sh.beta32 : (S)sh.beta;
    for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
      const Vs zv = zrow(i);
      Vs pv = ldv<S, NR>(P.p, i);
#pragma unroll
      for (int c = 0; c < NR; ++c) pv.c[c] = zv.c[c] + beta * pv.c[c];
      stv<S, NR>(P.p, i, pv);
    }
    tm.bar();
  }
  if constexpr (mixed) {  // fold what is pending; the FP64 solution is hi + lo
    for (int32_t i = r0 + tm.id; i < r1; i += tm.threads) {
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
  if (tm.id == 0) {
    if (flag == kLost) sh.st.status = RUV_ERR_TIMEOUT;
    sh.st.state = kDone;
    sh.st.refresh = 0;
    P.st[chart] = sh.st;
    atomicSub(P.n_active, 1);
  }
  if (tm.ctas > 1) tm.bar();  // no CTA leaves while a peer may still write its shared memory
}

// ---------------------------------------------------------------- which charts, and how many CTAs
// CTAs of a chart's team (0: left to the launch-per-step loop).
int team_size(int64_t rows, bool mixed, int kind, int64_t width) {
  // one CTA while a step fits it: its block barrier costs tens of clocks, a cluster's over a
  // thousand; FP64 rows are bound by the SM's FP64 pipe instead and spread out earlier
  const int64_t per = mixed ? 1024 : 256;
  int64_t want = (rows + per - 1) / per;
  if (kind == 2) want = std::max<int64_t>(1, width / 256);
  const int64_t lim = mixed ? 131072 : 40000;
  if (rows > lim) return 0;
  int c = 1;
  while (c < want && c < kTeamMaxCtas) c *= 2;
  return c;
}

template <class S, int NR, int PCK>
void launch_team(cudaStream_t s, int ctas, int64_t n, const TeamSys& A, const TeamLoop<S>& P, const TeamPrecond* pc) {
  auto k = k_team<S, NR, PCK>;
  if (ctas > 8) RUV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n * ctas));
  cfg.blockDim = dim3(kTeamThreads);
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

void Ctx::team_streams(int n) {
  if (!team_go) RUV_CUDA(cudaEventCreateWithFlags(&team_go, cudaEventDisableTiming));
  for (int k = 0; k < n; ++k) {
    if (!team_done[k]) RUV_CUDA(cudaEventCreateWithFlags(&team_done[k], cudaEventDisableTiming));
    if (!team_stream[k]) RUV_CUDA(cudaStreamCreateWithFlags(&team_stream[k], cudaStreamNonBlocking));
  }
}

template <class S, int NR>
int64_t team_solve(Ctx& ctx, const DevSystem& sys, const TeamLoop<S>& loop, const TeamPrecond* pc) {
  const int64_t NC = sys.n_charts;
  // RUV_TEAM=0, or a knob that picks a kernel of the launch-per-step loop: that loop for all
  const char* e = std::getenv("RUV_TEAM");
  const bool off = (e && e[0] == '0') || std::getenv("RUV_SPMV_TMA") || std::getenv("RUV_AMG_STAGE") || ctx.shape_forced;
  const int kind = pc ? pc->kind : 0;
  int64_t left = 0, largest = 0;
  for (int64_t c = 0; c < NC; ++c) largest = std::max(largest, sys.h_chart_row[c + 1] - sys.h_chart_row[c]);
  // a V-cycle is a chain of a dozen small steps: by teams only where one CTA holds every chart
  const bool none = off || (pc && kind == 0) || (kind == 1 && largest > 1024);
  // charts by team size, the largest first within each
  std::vector<int32_t> cls[5];
  for (int64_t c = 0; c < NC; ++c) {
    const int64_t rows = sys.h_chart_row[c + 1] - sys.h_chart_row[c];
    if (rows == 0) continue;
    const int ctas = none ? 0
                     : team_size(rows, std::is_same<S, float>::value, kind, pc && kind == 2 ? pc->ic0.width : 0);
    if (ctas == 0) {
      ++left;
      continue;
    }
    cls[__builtin_ctz(ctas)].push_back((int32_t)c);
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
    const TeamSys A{d_order + first[k], sys.chart_row, sys.row_ptr, sys.cols, sys.cols16, sys.cbase, nw, sys.vals32};
    if (kind == 1) launch_team<S, NR, 1>(s, 1 << k, n, A, loop, pc);
    else if (kind == 2) launch_team<S, NR, 2>(s, 1 << k, n, A, loop, pc);
    else launch_team<S, NR, 0>(s, 1 << k, n, A, loop, pc);
  }
  RUV_LAUNCH_CHECK();
  return left;
}

template int64_t team_solve<float, 2>(Ctx&, const DevSystem&, const TeamLoop<float>&, const TeamPrecond*);
template int64_t team_solve<double, 2>(Ctx&, const DevSystem&, const TeamLoop<double>&, const TeamPrecond*);
template int64_t team_solve<double, 1>(Ctx&, const DevSystem&, const TeamLoop<double>&, const TeamPrecond*);

}  // namespace ruv
