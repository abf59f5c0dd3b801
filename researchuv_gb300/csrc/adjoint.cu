// Differentiation of the batched LSCM unfold with respect to the 3-D vertex positions, and
// the distortion metrics of a UV layout (unwrap/src/metrics.rs:59-141).
//
// The differentiated map is the solve the reference runs (unwrap/src/lscm.rs:594-719) with
// the pins held at their targets: for every chart, A(p) uv = b(p), where A is the weighted
// Laplacian over free vertices with coefficients c_ij = w_ij / max(|p_j - p_i|^2, EPS),
// w_ij the sum of the clamped corner cotangents opposite edge ij, and b collects
// c_ij * pin_j over pinned neighbours.  For a loss with gradient g = dL/duv (free rows):
//   lam = A^-1 g                       (the same SPD operator and preconditioner)
//   dL/dc_ij = -(lam_i - lam_j) . (uv_i - uv_j)     (lam = 0 on pinned vertices)
//   dL/dw_ij = dL/dc_ij / max(d2, EPS);  dL/dd2 = -dL/dc_ij w_ij / d2^2 (when d2 > EPS)
//   dL/dcot  = dL/dw of the edge the corner faces (0 where the cotangent was clamped)
//   dcot / dp from cot = (a1 . a2) / |a1 x a2| at the corner.
// The assembly is recomputed in the backward pass (the reverse pass reads the recomputed
// cotangents, incidence records and edge coefficients, nothing stored by the forward solve).
// Position gradients are accumulated with FP64 atomics.
//
// The distortion loss sum_t area_t (s1/s2 - 1)^2 (area_t the 3-D area, s1 >= s2 the
// singular values of the UV Jacobian F = U P^-1 of metrics.rs:95-128, formed stably) is
// differentiated per triangle in reverse mode, FP64.  Triangles whose three vertices are all pinned are left
// out of the loss: their UVs are set by the pin rule, not by the solve, and the rule can
// place all three on one side of the border rectangle (the corner triangles of a grid chart),
// where s2 = 0 and the term is unbounded.
#include <cmath>

#include "system.cuh"

namespace ruv {
namespace {

constexpr int kAdjThreads = 256;

// ---------------------------------------------------------------- distortion term
// The distortion term of one triangle (metrics.rs:95-128): 0.5 |n| (s1 / max(s2, 1e-30) - 1)^2,
// or a skip (degenerate normal or tangent-frame determinant; those triangles add nothing); with
// `grad` also its gradient g in the 15 coordinates (p: 9, u: 6).
//
// The gradient is the reverse pass over the invariants of the edges e1, e2: m = |e1|^2, c = e1.e2,
// l1 = max(|e1|, 1e-30) and |n|, in which the frame's inverse is i00 = l1 / m, i01 = -c l1 / (m |n|),
// i10 = 0, i11 = l1 / |n|.  It takes about as many operations as the term itself, where forward-mode
// dual numbers (three seeds, five passes) took twenty times that, all on the SM's FP64 pipe: 1.38 ms for
// 227,000 triangles, of 12.3 ms for the loss and its gradient on 64 charts, which now take 11.1.
__device__ __forceinline__ bool tri_distortion(const double (&p)[9], const double (&u)[6], double& out, bool grad,
                                               double (&g)[15]) {
  const double e1x = p[3] - p[0], e1y = p[4] - p[1], e1z = p[5] - p[2];
  const double e2x = p[6] - p[0], e2y = p[7] - p[1], e2z = p[8] - p[2];
  const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
  const double ln = sqrt(nx * nx + ny * ny + nz * nz);
  if (ln < 1e-30) return false;
  const double ux = nx / ln, uy = ny / ln, uz = nz / ln;
  const double m = e1x * e1x + e1y * e1y + e1z * e1z, c = e1x * e2x + e1y * e2y + e1z * e2z;
  const double le = sqrt(m);
  const bool clamped = !(le > 1e-30);
  const double l1 = clamped ? 1e-30 : le;
  const double t1x = e1x / l1, t1y = e1y / l1, t1z = e1z / l1;
  const double t2x = uy * t1z - uz * t1y, t2y = uz * t1x - ux * t1z, t2z = ux * t1y - uy * t1x;
  const double e1t1 = e1x * t1x + e1y * t1y + e1z * t1z;
  const double e2t1 = e2x * t1x + e2y * t1y + e2z * t1z;
  const double e1t2 = e1x * t2x + e1y * t2y + e1z * t2z;
  const double e2t2 = e2x * t2x + e2y * t2y + e2z * t2z;
  const double det = e1t1 * e2t2 - e2t1 * e1t2;
  if (fabs(det) < 1e-30) return false;
  const double i00 = e2t2 / det, i01 = -e2t1 / det, i10 = -e1t2 / det, i11 = e1t1 / det;
  const double d1u = u[2] - u[0], d1v = u[3] - u[1], d2u = u[4] - u[0], d2v = u[5] - u[1];
  const double f00 = d1u * i00 + d2u * i10, f01 = d1u * i01 + d2u * i11;
  const double f10 = d1v * i00 + d2v * i10, f11 = d1v * i01 + d2v * i11;
  // singular values of F: s1 = (|(f00 + f11, f10 - f01)| + |(f00 - f11, f10 + f01)|) / 2 and
  // s2 = |det F| / s1 -- the same values as svd2 (metrics.rs:59-70), formed without its
  // 0.5 tr - disc cancellation, which loses (s1/s2)^2 ulps on anisotropic triangles
  const double p0 = f00 + f11, p1 = f10 - f01, q0 = f00 - f11, q1 = f10 + f01;
  const double P = sqrt(p0 * p0 + p1 * p1), Q = sqrt(q0 * q0 + q1 * q1);
  const double s1 = 0.5 * (P + Q);
  const double dF = f00 * f11 - f01 * f10;
  const double s2 = s1 > 0.0 ? fabs(dF) / s1 : 0.0;
  const double sc = s2 > 1e-30 ? s2 : 1e-30;
  const double r = s1 / sc - 1.0;
  out = 0.5 * (ln * (r * r));
  if (!grad) return true;
  // r, s2, s1
  const double gr = ln * r;
  double gs1 = gr / sc, gdF = 0.0;
  if (s2 > 1e-30) {  // (then s1 > 0)
    const double gs2 = -gr * s1 / (s2 * s2);
    gdF = (dF < 0.0 ? -gs2 : gs2) / s1;
    gs1 -= gs2 * s2 / s1;
  }
  // F (where P or Q is 0 the one-sided slope is unbounded; taken as 0)
  const double hp = P > 0.0 ? 0.5 * gs1 / P : 0.0, hq = Q > 0.0 ? 0.5 * gs1 / Q : 0.0;
  const double gp0 = hp * p0, gp1 = hp * p1, gq0 = hq * q0, gq1 = hq * q1;
  const double g00 = gp0 + gq0 + gdF * f11, g11 = gp0 - gq0 + gdF * f00;
  const double g10 = gp1 + gq1 - gdF * f01, g01 = gq1 - gp1 - gdF * f10;
  // UVs
  const double gd1u = g00 * i00 + g01 * i01, gd1v = g10 * i00 + g11 * i01, gd2u = g01 * i11, gd2v = g11 * i11;
  g[9] = -(gd1u + gd2u);
  g[10] = -(gd1v + gd2v);
  g[11] = gd1u;
  g[12] = gd1v;
  g[13] = gd2u;
  g[14] = gd2v;
  // the frame's inverse, then m, c, l1 and |n|
  const double gi00 = g00 * d1u + g10 * d1v, gi01 = g01 * d1u + g11 * d1v, gi11 = g01 * d2u + g11 * d2v;
  const double w0 = gi00 * i00, w1 = gi01 * i01, w2 = gi11 * i11;
  const double gm = -(w0 + w1) / m + (clamped ? 0.0 : 0.5 * (w0 + w1 + w2) / m);  // (l1's share: dl1 / dm = l1 / 2m)
  const double gc = -gi01 * l1 / (m * ln);
  const double gl = 0.5 * r * r - (w1 + w2) / ln;
  // edges
  const double gnx = gl * ux, gny = gl * uy, gnz = gl * uz;
  const double a1x = 2.0 * gm * e1x + gc * e2x + (e2y * gnz - e2z * gny);
  const double a1y = 2.0 * gm * e1y + gc * e2y + (e2z * gnx - e2x * gnz);
  const double a1z = 2.0 * gm * e1z + gc * e2z + (e2x * gny - e2y * gnx);
  const double a2x = gc * e1x + (gny * e1z - gnz * e1y);
  const double a2y = gc * e1y + (gnz * e1x - gnx * e1z);
  const double a2z = gc * e1z + (gnx * e1y - gny * e1x);
  g[0] = -(a1x + a2x);
  g[1] = -(a1y + a2y);
  g[2] = -(a1z + a2z);
  g[3] = a1x;
  g[4] = a1y;
  g[5] = a1z;
  g[6] = a2x;
  g[7] = a2y;
  g[8] = a2z;
  return true;
}

__device__ __forceinline__ int64_t chart_of(const int64_t* off, int64_t n, int64_t i) {
  int64_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (off[mid] <= i) lo = mid; else hi = mid;
  }
  return lo;
}

// Loss per triangle (loss_t) and, with gradients wanted, d loss / d(p, uv) accumulated.
__global__ void __launch_bounds__(kAdjThreads) k_distortion(const int64_t* __restrict__ tri_off,
                                                            const int64_t* __restrict__ vert_off, int64_t n_charts,
                                                            int64_t n_tris, const int32_t* __restrict__ tris,
                                                            const uint8_t* __restrict__ pinned,
                                                            const double* __restrict__ p3, const double* __restrict__ uv,
                                                            double* __restrict__ loss_t, double* duv, double* dp3) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tris) return;
  const int64_t c = chart_of(tri_off, n_charts, t);
  const int64_t v0 = vert_off[c];
  int64_t v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = v0 + tris[3 * t + k];
  if (pinned[v[0]] && pinned[v[1]] && pinned[v[2]]) {
    loss_t[t] = 0.0;
    return;
  }
  double p[9], u[6], g[15], val = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int j = 0; j < 3; ++j) p[3 * k + j] = p3[3 * v[k] + j];
    u[2 * k] = uv[2 * v[k]];
    u[2 * k + 1] = uv[2 * v[k] + 1];
  }
  const bool grad = duv != nullptr || dp3 != nullptr;
  if (tri_distortion(p, u, val, grad, g) && grad) {
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (dp3) atomicAdd(&dp3[3 * v[q / 3] + q % 3], g[q]);
#pragma unroll
    for (int q = 0; q < 6; ++q)
      if (duv) atomicAdd(&duv[2 * v[q / 2] + q % 2], g[9 + q]);
  }
  loss_t[t] = val;
}

// Per-chart sums of a per-triangle array (one CTA per chart, fixed order: deterministic).
__global__ void __launch_bounds__(kAdjThreads) k_chart_sum(const int64_t* __restrict__ tri_off, const double* __restrict__ a,
                                                           double* __restrict__ out) {
  __shared__ double sh[32];
  const int64_t c = blockIdx.x;
  double s[1] = {0.0};
  for (int64_t t = tri_off[c] + threadIdx.x; t < tri_off[c + 1]; t += blockDim.x) s[0] += a[t];
  block_sum<1>(s, sh);
  if (threadIdx.x == 0) out[c] = s[0];
}

// ---------------------------------------------------------------- metrics (metrics.rs:73-141)
// Every operation rounded on its own (no FMA contraction) in the reference's order, so each
// per-triangle value equals the reference's bit for bit; the per-chart sums run in triangle
// order.
__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sb(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ml(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double rmax(double a, double b) {  // Rust f64::max
  if (a != a) return b;
  if (b != b) return a;
  return a > b ? a : b;
}
__device__ __forceinline__ double dot3(const double* a, const double* b) {
  return ad(ad(ml(a[0], b[0]), ml(a[1], b[1])), ml(a[2], b[2]));
}
__device__ __forceinline__ void cross3(const double* a, const double* b, double* o) {
  o[0] = sb(ml(a[1], b[2]), ml(a[2], b[1]));
  o[1] = sb(ml(a[2], b[0]), ml(a[0], b[2]));
  o[2] = sb(ml(a[0], b[1]), ml(a[1], b[0]));
}
__device__ __forceinline__ double tri_signed(double au, double av, double bu, double bv, double cu, double cv) {
  return sb(ml(sb(bu, au), sb(cv, av)), ml(sb(cu, au), sb(bv, av)));  // metrics.rs:32-35
}

// Per triangle: conformal ratio (or -1 when skipped), area ratio, flip flag, signed UV area.
__global__ void __launch_bounds__(kAdjThreads) k_tri_metrics(const int64_t* __restrict__ tri_off,
                                                             const int64_t* __restrict__ vert_off, int64_t n_charts,
                                                             int64_t n_tris, const int32_t* __restrict__ tris,
                                                             const double* __restrict__ p3, const double* __restrict__ uv,
                                                             double4* __restrict__ m) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tris) return;
  const int64_t c = chart_of(tri_off, n_charts, t);
  const int64_t v0 = vert_off[c];
  const int64_t a = v0 + tris[3 * t], b = v0 + tris[3 * t + 1], d = v0 + tris[3 * t + 2];
  double e1[3], e2[3], n[3];
  for (int k = 0; k < 3; ++k) {
    e1[k] = sb(p3[3 * b + k], p3[3 * a + k]);
    e2[k] = sb(p3[3 * d + k], p3[3 * a + k]);
  }
  cross3(e1, e2, n);
  const double ln = sqrt(dot3(n, n));
  const double sgn = tri_signed(uv[2 * a], uv[2 * a + 1], uv[2 * b], uv[2 * b + 1], uv[2 * d], uv[2 * d + 1]);
  double4 r = make_double4(-1.0, -1.0, 0.0, sgn);
  if (ln >= 1e-30) {
    double nu[3], t1[3], t2[3];
    const double l1 = rmax(sqrt(dot3(e1, e1)), 1e-30);
    for (int k = 0; k < 3; ++k) {
      nu[k] = dv(n[k], ln);
      t1[k] = dv(e1[k], l1);
    }
    cross3(nu, t1, t2);
    const double e1t1 = dot3(e1, t1), e2t1 = dot3(e2, t1), e1t2 = dot3(e1, t2), e2t2 = dot3(e2, t2);
    const double det = sb(ml(e1t1, e2t2), ml(e2t1, e1t2));
    if (fabs(det) < 1e-30) {
      r.z = 1.0;
    } else {
      const double i00 = dv(e2t2, det), i01 = dv(-e2t1, det), i10 = dv(-e1t2, det), i11 = dv(e1t1, det);
      const double d1u = sb(uv[2 * b], uv[2 * a]), d1v = sb(uv[2 * b + 1], uv[2 * a + 1]);
      const double d2u = sb(uv[2 * d], uv[2 * a]), d2v = sb(uv[2 * d + 1], uv[2 * a + 1]);
      const double f00 = ad(ml(d1u, i00), ml(d2u, i10)), f01 = ad(ml(d1u, i01), ml(d2u, i11));
      const double f10 = ad(ml(d1v, i00), ml(d2v, i10)), f11 = ad(ml(d1v, i01), ml(d2v, i11));
      const double aa = ad(ml(f00, f00), ml(f10, f10)), bb = ad(ml(f00, f01), ml(f10, f11));
      const double cc = ad(ml(f01, f01), ml(f11, f11));
      const double tr = ad(aa, cc), dd = ml(0.5, sb(aa, cc));
      const double disc = sqrt(rmax(ad(ml(dd, dd), ml(bb, bb)), 0.0));
      const double lam1 = ad(ml(0.5, tr), disc), lam2 = rmax(sb(ml(0.5, tr), disc), 0.0);
      const double s1 = sqrt(rmax(lam1, 0.0)), s2 = sqrt(lam2);
      r.x = dv(s1, rmax(s2, 1e-30));
      r.y = dv(ml(0.5, fabs(sb(ml(d1u, d2v), ml(d2u, d1v)))), ml(0.5, ln));
    }
  }
  m[t] = r;
}

// Per chart (one CTA): [conformal mean, conformal max, area ratio mean, flips, folds].
//
// The three sums run in triangle order, one rounded addition at a time (the reference's bits), so
// the longest chart's chain of dependent FP64 additions bounds the kernel.  Each sum has a lane of
// its own in one of the first three warps, fed from shared memory; the other warps stage the next
// chunk and take the maximum and the counts, which no order changes.  A skipped triangle adds -0,
// which changes no bit of a sum.  folds needs the sign of the whole area sum, so both signs are
// counted on the way.  (One thread per chart walking global memory took 8.6 ms on 256 charts of up
// to 20,000 triangles, 430 ns a triangle.)
constexpr int kMetThreads = 256;
constexpr int kMetSumWarps = 3;
constexpr int kMetChunk = 640;  // four staged triangles per staging thread and chunk
__global__ void __launch_bounds__(kMetThreads) k_chart_metrics(const int64_t* __restrict__ tri_off,
                                                               const double4* __restrict__ m, double* __restrict__ out) {
  __shared__ __align__(16) double buf[2][kMetSumWarps][kMetChunk];
  __shared__ double sums[kMetSumWarps];
  __shared__ double wmax[kMetThreads / 32];
  __shared__ int counts[4];  // triangles measured, flips, signed areas <= 0, >= 0
  const int64_t c = blockIdx.x, t0 = tri_off[c], t1 = tri_off[c + 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x < 4) counts[threadIdx.x] = 0;
  double cm = 0.0;
  int cnt = 0, flips = 0, le = 0, ge = 0;
  auto stage = [&](int64_t base, int to, int first, int step) {
    const int n = (int)(t1 - base < kMetChunk ? t1 - base : kMetChunk);
    for (int i = first; i < kMetChunk; i += step) {
      double x = -0.0, y = -0.0, w = -0.0;
      if (i < n) {
        const double4 r = m[base + i];
        if (r.x >= 0.0) {
          x = r.x;
          y = r.y;
          cm = rmax(cm, r.x);
          ++cnt;
        }
        w = r.w;
        flips += r.z != 0.0;
        le += r.w <= 0.0;
        ge += r.w >= 0.0;
      }
      buf[to][0][i] = x;
      buf[to][1][i] = y;
      buf[to][2][i] = w;
    }
  };
  stage(t0, 0, threadIdx.x, kMetThreads);
  __syncthreads();
  double s = 0.0;
  int cur = 0;
  for (int64_t base = t0; base < t1; base += kMetChunk, cur ^= 1) {
    if (wid >= kMetSumWarps) {
      if (base + kMetChunk < t1)
        stage(base + kMetChunk, cur ^ 1, threadIdx.x - 32 * kMetSumWarps, kMetThreads - 32 * kMetSumWarps);
    } else if (lane == 0) {
      const double2* v = reinterpret_cast<const double2*>(buf[cur][wid]);
      const int n = (int)(t1 - base < kMetChunk ? t1 - base : kMetChunk);
      for (int i = 0; i < (n + 7) / 8; ++i) {  // (past n the chunk holds -0)
        const double2 a = v[4 * i], b = v[4 * i + 1], d = v[4 * i + 2], e = v[4 * i + 3];
        s = ad(ad(ad(ad(ad(ad(ad(ad(s, a.x), a.y), b.x), b.y), d.x), d.y), e.x), e.y);
      }
    }
    __syncthreads();
  }
  if (wid < kMetSumWarps && lane == 0) sums[wid] = s;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cm = rmax(cm, __shfl_xor_sync(0xffffffffu, cm, o));
  const int q[4] = {cnt, flips, le, ge};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int total = __reduce_add_sync(0xffffffffu, q[k]);
    if (lane == 0 && total) atomicAdd(&counts[k], total);
  }
  if (lane == 0) wmax[wid] = cm;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 0; w < kMetThreads / 32; ++w) cm = rmax(cm, wmax[w]);
  const double nd = (double)(counts[0] > 1 ? counts[0] : 1);
  out[5 * c] = dv(sums[0], nd);
  out[5 * c + 1] = cm;
  out[5 * c + 2] = dv(sums[1], nd);
  out[5 * c + 3] = (double)counts[1];
  // a triangle folds when its signed area times the sign of the whole is not above zero
  out[5 * c + 4] = (double)(sums[2] < 0.0 ? counts[3] : counts[2]);
}

// The same sums with a thread per chart, for batches of many short charts: there the FP64 pipe bounds the
// kernel above, whose additions are one lane of a warp instruction each (20 clocks of an SM), and 32
// charts share an instruction here, but the longest chart's walk through global memory bounds it.  The line by
// triangles in all over the longest chart's (ms a call, this / above): 300 charts of 197 longest ones 0.099 / 0.083, 1,000 of 470
// 0.251 / 0.193, 3,000 of 1,200 2.19 / 1.85, 3,000 of 1,428 0.410 / 0.425, 3,000 of 2,023 0.153 / 0.189, 30,000 of
// 20,423 0.79 / 1.29.
constexpr int64_t kMetEach = 1400;
__global__ void k_chart_metrics_each(int64_t n_charts, const int64_t* __restrict__ tri_off,
                                     const double4* __restrict__ m, double* __restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_charts) return;
  double cs = 0.0, cm = 0.0, as = 0.0, sg = 0.0;
  int64_t cnt = 0, flips = 0, le = 0, ge = 0;
  for (int64_t t = tri_off[c]; t < tri_off[c + 1]; ++t) {
    const double4 r = m[t];
    if (r.x >= 0.0) {
      cs = ad(cs, r.x);
      cm = rmax(cm, r.x);
      as = ad(as, r.y);
      ++cnt;
    }
    flips += r.z != 0.0;
    le += r.w <= 0.0;
    ge += r.w >= 0.0;
    sg = ad(sg, r.w);
  }
  const double nd = (double)(cnt > 1 ? cnt : 1);
  out[5 * c] = dv(cs, nd);
  out[5 * c + 1] = cm;
  out[5 * c + 2] = dv(as, nd);
  out[5 * c + 3] = (double)flips;
  out[5 * c + 4] = (double)(sg < 0.0 ? ge : le);
}

// ---------------------------------------------------------------- rectangularize (metrics.rs:147-227)
constexpr int kRectAngles = 72;
constexpr int kRectThreads = 512;

__device__ __forceinline__ void warp_minmax4(double (&v)[4]) {  // min, max, min, max
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v[0] = fmin(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
    v[1] = fmax(v[1], __shfl_xor_sync(0xffffffffu, v[1], o));
    v[2] = fmin(v[2], __shfl_xor_sync(0xffffffffu, v[2], o));
    v[3] = fmax(v[3], __shfl_xor_sync(0xffffffffu, v[3], o));
  }
}

// One CTA per chart.  The border points are listed first (a chart of n vertices has about
// sqrt(n) of them), then the 72-angle ladder runs over that list (each warp a set of angles; min /
// max are exact in any order, so is the list's), the first angle of least score is kept, and the
// whole chart is rotated, normalised to [0,1]^2 and its border points snapped to the nearest
// rectangle side.  (The ladder over every vertex with its border flag took 3.5 ms on 256 charts
// of up to 10,000 vertices.)  The angle table (cos, sin) comes from the host's libm, as the reference's
// does; every product and sum is rounded on its own (no FMA), so the result is bit-identical.
__global__ void __launch_bounds__(kRectThreads) k_rectangularize(const int64_t* __restrict__ vert_off,
                                                                 const double* __restrict__ uv,
                                                                 const uint8_t* __restrict__ border,
                                                                 const double* __restrict__ cs, int32_t* __restrict__ list,
                                                                 double* __restrict__ q, double* __restrict__ ext) {
  __shared__ double score[kRectAngles];
  __shared__ double red[4][kRectThreads / 32];
  __shared__ double rot[2];
  __shared__ int n_border;
  const int64_t c = blockIdx.x;
  const int64_t v0 = vert_off[c], v1 = vert_off[c + 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = kRectThreads / 32;
  if (v1 <= v0) return;
  if (threadIdx.x == 0) n_border = 0;
  __syncthreads();
  for (int64_t base = v0; base < v1; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const bool on = i < v1 && border[i];
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    int at = 0;
    if (lane == 0 && mask) at = atomicAdd(&n_border, __popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (on) list[v0 + at + __popc(mask & ((1u << lane) - 1u))] = (int32_t)(i - v0);
  }
  __syncthreads();
  const int nb = n_border;
  const bool has_border = nb > 0;
  double cth = 1.0, sth = 0.0;
  if (has_border) {
    for (int k = wid; k < kRectAngles; k += nw) {
      const double co = cs[2 * k], si = cs[2 * k + 1];
      double v[4] = {INFINITY, -INFINITY, INFINITY, -INFINITY};
      for (int b = lane; b < nb; b += 32) {
        const int64_t i = v0 + list[v0 + b];
        const double pu = uv[2 * i], pv = uv[2 * i + 1];
        const double qu = ad(ml(co, pu), ml(si, pv));
        const double qv = ad(ml(-si, pu), ml(co, pv));
        v[0] = fmin(v[0], qu);
        v[1] = fmax(v[1], qu);
        v[2] = fmin(v[2], qv);
        v[3] = fmax(v[3], qv);
      }
      warp_minmax4(v);
      if (lane == 0) {
        const double e0 = sb(v[1], v[0]), e1 = sb(v[3], v[2]);
        score[k] = sqrt(ad(ml(e0, ad(e0, 1e-30)), ml(e1, ad(e1, 1e-30))));
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int best = 0;  // the first angle of least score (later ties do not replace it)
      for (int k = 1; k < kRectAngles; ++k)
        if (score[k] < score[best]) best = k;
      rot[0] = cs[2 * best];
      rot[1] = cs[2 * best + 1];
    }
    __syncthreads();
    cth = rot[0];
    sth = rot[1];
  }
  // rotate and take the bounding box
  double v[4] = {INFINITY, -INFINITY, INFINITY, -INFINITY};
  for (int64_t i = v0 + threadIdx.x; i < v1; i += blockDim.x) {
    const double pu = uv[2 * i], pv = uv[2 * i + 1];
    double qu = pu, qv = pv;
    if (has_border) {
      qu = ad(ml(cth, pu), ml(sth, pv));
      qv = ad(ml(-sth, pu), ml(cth, pv));
    }
    q[2 * i] = qu;
    q[2 * i + 1] = qv;
    v[0] = fmin(v[0], qu);
    v[1] = fmax(v[1], qu);
    v[2] = fmin(v[2], qv);
    v[3] = fmax(v[3], qv);
  }
  warp_minmax4(v);
  if (lane == 0)
    for (int k = 0; k < 4; ++k) red[k][wid] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    double m[4] = {red[0][0], red[1][0], red[2][0], red[3][0]};
    for (int w = 1; w < nw; ++w) {
      m[0] = fmin(m[0], red[0][w]);
      m[1] = fmax(m[1], red[1][w]);
      m[2] = fmin(m[2], red[2][w]);
      m[3] = fmax(m[3], red[3][w]);
    }
    red[0][0] = m[0];
    red[2][0] = m[2];
    red[1][0] = sb(m[1], m[0]);  // extents
    red[3][0] = sb(m[3], m[2]);
    ext[2 * c] = red[1][0];
    ext[2 * c + 1] = red[3][0];
  }
  __syncthreads();
  const double mu = red[0][0], mv = red[2][0], eu = rmax(red[1][0], 1e-30), ev = rmax(red[3][0], 1e-30);
  for (int64_t i = v0 + threadIdx.x; i < v1; i += blockDim.x) {
    double pu = dv(sb(q[2 * i], mu), eu), pv = dv(sb(q[2 * i + 1], mv), ev);
    if (has_border && border[i]) {  // verticalize: snap onto the nearest side
      const double dx = fmin(pu, sb(1.0, pu)), dy = fmin(pv, sb(1.0, pv));
      if (dx <= dy) pu = pu < 0.5 ? 0.0 : 1.0;
      else pv = pv < 0.5 ? 0.0 : 1.0;
    }
    q[2 * i] = pu;
    q[2 * i + 1] = pv;
  }
}

// ---------------------------------------------------------------- reverse pass of the assembly
// g (vertex-ordered, 2 per vertex) -> per free row.
__global__ void k_gather_rows(int64_t n_rows, const int32_t* __restrict__ row_vert, const double* __restrict__ gv,
                              double* __restrict__ grow) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_rows) return;
  const int64_t v = row_vert[r];
  grow[2 * r] = gv[2 * v];
  grow[2 * r + 1] = gv[2 * v + 1];
}

// One free vertex v: for each kept edge (v, nb) that v owns (nb pinned, or v < nb), the
// coefficient's adjoint; its edge-length part goes to p_v and p_nb, its weight part to the
// corners facing the edge (corner_g).
__global__ void k_edge_adjoint(int64_t n_verts, const uint8_t* __restrict__ pinned, const int64_t* __restrict__ row_of,
                               const int64_t* __restrict__ rec_off, const int2* __restrict__ rec,
                               const double* __restrict__ coef, const double* __restrict__ cot,
                               const double* __restrict__ p3, const double* __restrict__ pin_uv,
                               const double* __restrict__ x, const double* __restrict__ lam, double* __restrict__ corner_g,
                               double* dp3) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_verts || pinned[v]) return;
  const int64_t r1 = rec_off[v + 1];
  const int64_t rv = row_of[v];
  const double xu = x[2 * rv], xv = x[2 * rv + 1], lu = lam[2 * rv], lv = lam[2 * rv + 1];
  for (int64_t i = rec_off[v]; i < r1;) {
    const int32_t nb = rec[i].x;
    int64_t j = i;
    double w = 0.0;
    for (; j < r1 && rec[j].x == nb; ++j) w += cot[rec[j].y];
    const double c = coef[i];
    const bool own = pinned[nb] || v < nb;
    if (own && c >= 0.0) {
      double nu, nv, mu = 0.0, mv = 0.0;
      if (pinned[nb]) {
        nu = pin_uv[2 * nb];
        nv = pin_uv[2 * nb + 1];
      } else {
        const int64_t rn = row_of[nb];
        nu = x[2 * rn];
        nv = x[2 * rn + 1];
        mu = lam[2 * rn];
        mv = lam[2 * rn + 1];
      }
      const double gc = -((lu - mu) * (xu - nu) + (lv - mv) * (xv - nv));
      const double dx = p3[3 * nb] - p3[3 * v], dy = p3[3 * nb + 1] - p3[3 * v + 1], dz = p3[3 * nb + 2] - p3[3 * v + 2];
      const double d2 = dx * dx + dy * dy + dz * dz;
      double gw;
      if (d2 > kEpsDegenerate) {
        gw = gc / d2;
        const double gd2 = -gc * w / (d2 * d2);
        atomicAdd(&dp3[3 * nb], 2.0 * gd2 * dx);
        atomicAdd(&dp3[3 * nb + 1], 2.0 * gd2 * dy);
        atomicAdd(&dp3[3 * nb + 2], 2.0 * gd2 * dz);
        atomicAdd(&dp3[3 * v], -2.0 * gd2 * dx);
        atomicAdd(&dp3[3 * v + 1], -2.0 * gd2 * dy);
        atomicAdd(&dp3[3 * v + 2], -2.0 * gd2 * dz);
      } else {
        gw = gc / kEpsDegenerate;
      }
      for (int64_t k = i; k < j; ++k) corner_g[rec[k].y] = gw;
    }
    i = j;
  }
}

// One triangle: the cotangent adjoint of each corner that was not clamped.
__global__ void k_cot_adjoint(int64_t n_tris, const int32_t* __restrict__ tri_g, const double* __restrict__ p3,
                              const double* __restrict__ cot, const double* __restrict__ corner_g, double* dp3) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tris) return;
  int64_t vi[3];
  double p[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    vi[k] = tri_g[3 * t + k];
#pragma unroll
    for (int j = 0; j < 3; ++j) p[k][j] = p3[3 * vi[k] + j];
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double g = corner_g[3 * t + m];
    const double ct = cot[3 * t + m];
    if (g == 0.0 || !(ct > 0.0)) continue;
    const int o = m, e1 = (m + 2) % 3, e0 = (m + 1) % 3;
    double a1[3], a2[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      a1[j] = p[e1][j] - p[o][j];
      a2[j] = p[e0][j] - p[o][j];
    }
    const double n[3] = {a1[1] * a2[2] - a1[2] * a2[1], a1[2] * a2[0] - a1[0] * a2[2], a1[0] * a2[1] - a1[1] * a2[0]};
    const double C = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (!(C > 0.0)) continue;
    const double nh[3] = {n[0] / C, n[1] / C, n[2] / C};
    // d cot / d a1 = (a2 - cot (a2 x nh)) / C;  d cot / d a2 = (a1 - cot (nh x a1)) / C
    const double a2n[3] = {a2[1] * nh[2] - a2[2] * nh[1], a2[2] * nh[0] - a2[0] * nh[2], a2[0] * nh[1] - a2[1] * nh[0]};
    const double na1[3] = {nh[1] * a1[2] - nh[2] * a1[1], nh[2] * a1[0] - nh[0] * a1[2], nh[0] * a1[1] - nh[1] * a1[0]};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double g1 = g * (a2[j] - ct * a2n[j]) / C;
      const double g2 = g * (a1[j] - ct * na1[j]) / C;
      atomicAdd(&dp3[3 * vi[e1] + j], g1);
      atomicAdd(&dp3[3 * vi[e0] + j], g2);
      atomicAdd(&dp3[3 * vi[o] + j], -(g1 + g2));
    }
  }
}

}  // namespace

void lscm_backward(Ctx& ctx, DevBatch& bt, const DevSystem& sys, const double* x, const double* g_vert,
                   const SolveOpts& o, double* dp3, std::vector<ChartResult>& res) {
  cudaStream_t s = ctx.stream;
  Workspace& ws = ctx.ws;
  const int64_t NR = sys.n_rows, NV = bt.n_verts, NT = bt.n_tris;
  double* grow = ws.get<double>("adj.g", std::max<int64_t>(2 * NR, 1));
  double* lam = ws.get<double>("adj.lam", std::max<int64_t>(2 * NR, 1));
  if (NR > 0) {
    k_gather_rows<<<div_up(NR, kAdjThreads), kAdjThreads, 0, s>>>(NR, bt.row_vert, g_vert, grow);
    count_launches(1);
    RUV_LAUNCH_CHECK();
  }
  DevSystem adj = sys;  // same operator, right-hand side g
  adj.b = grow;
  res = pcg_solve(ctx, adj, lam, o);
  double* corner_g = ws.get<double>("adj.corner_g", std::max<int64_t>(3 * NT, 1));
  RUV_CUDA(cudaMemsetAsync(corner_g, 0, sizeof(double) * std::max<int64_t>(3 * NT, 1), s));
  RUV_CUDA(cudaMemsetAsync(dp3, 0, sizeof(double) * std::max<int64_t>(3 * NV, 1), s));
  if (NV > 0) {
    k_edge_adjoint<<<div_up(NV, kAdjThreads), kAdjThreads, 0, s>>>(NV, bt.pinned, bt.row_of, bt.rec_off, bt.rec, bt.coef,
                                                                    bt.cot, bt.p3, bt.pin_uv, x, lam, corner_g, dp3);
    count_launches(1);
  }
  if (NT > 0) {
    k_cot_adjoint<<<div_up(NT, kAdjThreads), kAdjThreads, 0, s>>>(NT, bt.tri_g, bt.p3, bt.cot, corner_g, dp3);
    count_launches(1);
  }
  RUV_LAUNCH_CHECK();
}

void distortion_loss(Ctx& ctx, const DevBatch& bt, const double* uv, double* duv, double* dp3, std::vector<double>& loss) {
  cudaStream_t s = ctx.stream;
  const int64_t NT = bt.n_tris, NC = bt.n_charts;
  double* lt = ctx.ws.get<double>("dist.loss_t", std::max<int64_t>(NT, 1));
  double* lc = ctx.ws.get<double>("dist.loss_c", std::max<int64_t>(NC, 1));
  if (NT > 0) {
    k_distortion<<<div_up(NT, kAdjThreads), kAdjThreads, 0, s>>>(bt.tri_off, bt.vert_off, NC, NT, bt.tris, bt.pinned,
                                                                  bt.p3, uv, lt, duv, dp3);
    count_launches(1);
  }
  if (NC > 0) {
    k_chart_sum<<<(unsigned)NC, kAdjThreads, 0, s>>>(bt.tri_off, lt, lc);
    count_launches(1);
  }
  RUV_LAUNCH_CHECK();
  loss.resize(NC);
  if (NC > 0) RUV_CUDA(cudaMemcpyAsync(loss.data(), lc, sizeof(double) * NC, cudaMemcpyDeviceToHost, s));
  RUV_CUDA(cudaStreamSynchronize(s));
}

void rectangularize(Ctx& ctx, const DevBatch& bt, const double* uv, const uint8_t* border, double* q, double* ext) {
  cudaStream_t s = ctx.stream;
  // the angle ladder of metrics.rs:166-171 with the host's libm (np.linspace(0, pi, 72))
  std::vector<double> h(2 * kRectAngles);
  for (int k = 0; k < kRectAngles; ++k) {
    const double ang = 3.141592653589793 * (double)k / (double)(kRectAngles - 1);
    h[2 * k] = std::cos(ang);
    h[2 * k + 1] = std::sin(ang);
  }
  double* cs = ctx.ws.get<double>("rect.cs", 2 * kRectAngles);
  RUV_CUDA(cudaMemcpyAsync(cs, h.data(), sizeof(double) * 2 * kRectAngles, cudaMemcpyHostToDevice, s));
  if (bt.n_charts > 0) {
    int32_t* list = ctx.ws.get<int32_t>("rect.list", std::max<int64_t>(bt.n_verts, 1));
    k_rectangularize<<<(unsigned)bt.n_charts, kRectThreads, 0, s>>>(bt.vert_off, uv, border, cs, list, q, ext);
    count_launches(1);
  }
  RUV_LAUNCH_CHECK();
  RUV_CUDA(cudaStreamSynchronize(s));  // `h` goes out of scope
}

void chart_metrics(Ctx& ctx, const DevBatch& bt, const double* uv, std::vector<double>& out5) {
  cudaStream_t s = ctx.stream;
  const int64_t NT = bt.n_tris, NC = bt.n_charts;
  double4* m = ctx.ws.get<double4>("met.tri", std::max<int64_t>(NT, 1));
  double* o = ctx.ws.get<double>("met.out", std::max<int64_t>(5 * NC, 1));
  if (NT > 0) {
    k_tri_metrics<<<div_up(NT, kAdjThreads), kAdjThreads, 0, s>>>(bt.tri_off, bt.vert_off, NC, NT, bt.tris, bt.p3, uv, m);
    count_launches(1);
  }
  if (NC > 0) {
    int64_t longest = 0;
    for (int64_t c = 0; c < NC; ++c) longest = std::max(longest, bt.h_tri_off[c + 1] - bt.h_tri_off[c]);
    if (NT > kMetEach * longest)
      k_chart_metrics_each<<<div_up(NC, 64), 64, 0, s>>>(NC, bt.tri_off, m, o);
    else
      k_chart_metrics<<<(unsigned)NC, kMetThreads, 0, s>>>(bt.tri_off, m, o);
    count_launches(1);
  }
  RUV_LAUNCH_CHECK();
  out5.resize(5 * NC);
  if (NC > 0) RUV_CUDA(cudaMemcpyAsync(out5.data(), o, sizeof(double) * 5 * NC, cudaMemcpyDeviceToHost, s));
  RUV_CUDA(cudaStreamSynchronize(s));
}

}  // namespace ruv
