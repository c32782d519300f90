// bsg_wishart.cuh -- the FP64 Omega | beta draw run by one warp at the end
// of a sweep: Marsaglia-Tsang gamma variates, warp-parallel Cholesky, and
// the Bartlett construction.
#pragma once

#include "bsg_device.cuh"

namespace bsg {

// ----------------------------------------------------- FP64 Wishart tail --
// Marsaglia & Tsang (2000) gamma(a, 1); a < 1 through the U^(1/a) boost.
// Attempt t of slot uses counter (slot*64 + t, 0, sweep, chain<<8|GAMMA).
// The squeeze u < 1 - 0.0331 x^4 lies inside the acceptance region, so it
// accepts exactly the attempts the log test would; it spares the two FP64
// logarithms in most attempts.  F64: the normal of each attempt in FP64
// (the FP64 chain) instead of the FP32 inversion.
template <bool F64 = false>
static __device__ double gamma_mt(double a, uint32_t slot, uint32_t sweep,
                                  uint32_t c3, uint32_t k0, uint32_t k1,
                                  int *err) {
  const bool boost = a < 1.0;
  const double aa = boost ? a + 1.0 : a;
  const double dd = aa - 1.0 / 3.0, c = 1.0 / sqrt(9.0 * dd);
  for (int t = 0; t < kGammaMax; ++t) {
    const uint4 r = philox1(make_uint4(slot * 64u + (uint32_t)t, 0u, sweep, c3),
                            k0, k1);
    const double x = F64 ? normal_of_d(r.x) : (double)normal_of(r.x);
    const double cx = c * x;
    if (!(cx > -1.0)) continue;
    const double v3 = (1.0 + cx) * (1.0 + cx) * (1.0 + cx);
    const double u = u_of_d(r.y), x2 = x * x;
    if (u < 1.0 - 0.0331 * x2 * x2 ||
        log(u) < 0.5 * x * x + dd * (1.0 - v3 + 3.0 * log1p(cx)))
      return dd * v3 * (boost ? pow(u_of_d(r.z), 1.0 / a) : 1.0);
  }
  *err |= kErrGammaCap;
  return dd;
}

// The Bartlett variates of a sweep, which do not depend on S: lane i < P
// draws sqrt(chi^2(df - i)) into wd[i], lane q < P(P-1)/2 the normal of
// the q-th strictly lower entry (row-major) into wd[kMaxP + q].  Run off the
// Omega draw's dependency chain: by a warp of colour 1 before its wait (FP64
// chains: by the last colour-0 block).  Returns the lane's error bits.  F64:
// normals in FP64 (the FP64 chain).
template <bool F64 = false>
static __device__ int wishart_draws(const ChainDev &ch, const DatasetDev &d,
                                    long long sweep, int lane, double *wd) {
  const int P = d.P;
  const uint32_t cid = ch.chain_id << 8, sw = (uint32_t)sweep;
  int err = 0;
  const double df = (double)d.V + (double)ch.df_offset;
  if (lane < P)
    wd[lane] = sqrt(2.0 * gamma_mt<F64>(0.5 * (df - lane), (uint32_t)lane, sw,
                                        cid | kTagGamma, ch.key0, ch.key1, &err));
  if (lane < P * (P - 1) / 2) {
    const uint4 r = philox1(make_uint4((uint32_t)(lane >> 2), 0u, sw, cid | kTagWNorm),
                            ch.key0, ch.key1);
    wd[kMaxP + lane] = F64 ? normal_of_d(pick4(r, lane & 3))
                           : (double)normal_of(pick4(r, lane & 3));
  }
  return err;
}

// 1 / sqrt(d) in FP64 from the single-precision value (relative error e of
// some 2^-22) by one third-order step, which leaves e^3: four dependent FP64
// operations, each about 80 cycles here; rounds within an ulp or so.  (d, a
// pivot of S + I, is hardly ever outside a float's range.)
static __device__ __forceinline__ double rsqrt_step(double d) {
  if (!(d > 1e-30 && d < 1e30)) return rsqrt(d);
  const double y = (double)rsqrt_approx((float)d);
  const double e = fma(-(d * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// Omega | beta ~ Wishart(df, (S + I)^-1) by the Bartlett construction of
// rwishart2 (cholesky.cpp:245-286), FP64, one warp.  The reference forms
// chol((S + I)^-1) by chol -> invert -> chol (covar.cpp:286-291,
// covarGPU.cu:1099-1104); the same factor is reached here with a fraction
// of the dependent work: with the reverse (upper) Cholesky S + I = U U',
// the inverse is U^-T U^-1 and U^-T is lower triangular with a positive
// diagonal, so chol((S + I)^-1) = U^-T (the Cholesky factor is unique),
// and B = U^-T T comes from forward substitution without forming U^-T.
//
// What counts is the depth of the chain, as nothing else of the sweep can go
// on: lane q owns entry q of the packed lower triangle (P = 8: q + 32 too) in
// registers, and P is a template argument, so that no index is computed at run
// time (with run-time P and the matrices in shared memory it took 4.3 to 5.0 us
// for P = 3; the sweep of the 20^3 study went from 19.7 to 17.8 us by this and
// the kept sums' place after the block's arrival).
template <int P>
static __device__ void wishart_warp(const ChainDev &ch, const double *tot, int supplied,
                                    const Supplied &sup, int lane) {
  constexpr int NP = P * (P + 1) / 2, NE = (NP + 31) / 32;
  __shared__ double U[P][P], B[P][P], piv;  // U[k][j]: U' by rows
  int ei[NE], ej[NE];
  double a[NE], t[NE];
#pragma unroll
  for (int u = 0; u < NE; ++u) {
    const int q = lane + 32 * u;
    int r = 0;
#pragma unroll
    for (int k = 1; k < P; ++k) r += q >= k * (k + 1) / 2;
    ei[u] = q < NP ? r : -1;
    ej[u] = q - r * (r + 1) / 2;
    // S + I, and the Bartlett factor T: sqrt(chi^2) on the diagonal, normals
    // below it (drawn by colour 1's last warp before its wait, or supplied)
    a[u] = t[u] = 0.0;
    if (q < NP) {
      const bool dg = ei[u] == ej[u];
      const int w = ei[u] * (ei[u] - 1) / 2 + ej[u];
      a[u] = tot[q] + (dg ? 1.0 : 0.0);
      t[u] = supplied ? (dg ? sqrt(sup.chi2[ei[u]]) : sup.wnorm[w])
                      : __ldcg(ch.wdraw + (dg ? ei[u] : kMaxP + w));
      if (q == NP - 1) piv = a[u];
    }
  }
  __syncwarp();
  // S + I = U U' with U upper, last pivot first
  bool ok = true;
  double rd[P];  // 1 / U[k][k]
#pragma unroll
  for (int k = P - 1; k >= 0; --k) {
    const double dk = piv;
    ok = ok && (dk > 0.0);
    rd[k] = rsqrt_step(dk);
#pragma unroll
    for (int u = 0; u < NE; ++u)
      if (ei[u] == k) U[k][ej[u]] = a[u] * rd[k];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < NE; ++u)
      if (ei[u] >= 0 && ei[u] < k) {
        a[u] -= U[k][ei[u]] * U[k][ej[u]];
        if (k > 0 && ei[u] == k - 1 && ej[u] == k - 1) piv = a[u];
      }
    __syncwarp();
  }
  int err = 0;
  if (ok) {
    // B = U^-T T by forward substitution U' B = T, right-looking; B is lower
    // triangular like T
#pragma unroll
    for (int i = 0; i < P; ++i) {
#pragma unroll
      for (int u = 0; u < NE; ++u)
        if (ei[u] == i) B[i][ej[u]] = t[u] * rd[i];
      __syncwarp();
#pragma unroll
      for (int u = 0; u < NE; ++u)
        if (ei[u] > i && ej[u] <= i) t[u] -= U[ei[u]][i] * B[i][ej[u]];
    }
    bool fin = true;
    double om[NE];
#pragma unroll
    for (int u = 0; u < NE; ++u) {  // Omega = B B'
      om[u] = 0.0;
      if (ei[u] >= 0) {
#pragma unroll
        for (int k = 0; k < P; ++k)
          if (k <= ej[u]) om[u] += B[ei[u]][k] * B[ej[u]][k];
        fin = fin && isfinite(om[u]);
      }
    }
    fin = __all_sync(0xffffffffu, fin);
    if (fin) {
#pragma unroll
      for (int u = 0; u < NE; ++u)
        if (ei[u] >= 0) {
          const int lo = ei[u] * P + ej[u], up = ej[u] * P + ei[u];
          ch.omega_d[lo] = ch.omega_d[up] = om[u];
          ch.omega_f[lo] = ch.omega_f[up] = (float)om[u];
        }
    } else {
      err |= kErrNaN;
    }
  } else {
    err |= kErrWishart;
  }
  if (lane == 0 && err) {
    atomicOr(ch.status, err);
    atomicOr(ch.any_status, err);
  }
}

// What else ends a sweep and does not wait for Omega, run by another warp
// beside wishart_warp: the column means, beta_WM, the counters.
static __device__ void sweep_end_warp(const ChainDev &ch, const DatasetDev &d,
                                      const double *tot, long long sweep, bool kept,
                                      int supplied, int lane) {
  const uint32_t cid = ch.chain_id << 8, sw = (uint32_t)sweep;
  if (lane < d.P) ch.colmean[lane] = (float)(tot[kMaxPairs + lane] / (double)d.V);
  if (lane == 0) {
    // beta_WM | Z, beta ~ N(var * sum_v WM_v sum_i (Z_iv - x_i' beta_v),
    // var = 1 / (N sum_v WM_v^2)) (updateBetaGPU, covarGPU.cu:680-720)
    float bw = *ch.wm_beta;
    if (ch.wm_update && !supplied) {
      const double var = 1.0 / ((double)d.N * d.wm2);
      const uint4 r = philox1(make_uint4(0u, 0u, sw, cid | kTagWm), ch.key0, ch.key1);
      const double z = (double)normal_of(pick4(r, 0));
      const float nb = (float)(var * tot[kWmOff] + sqrt(var) * z);
      if (isfinite(nb)) {
        bw = nb;
        *ch.wm_beta = nb;
      } else {
        atomicOr(ch.status, kErrNaN);
        atomicOr(ch.any_status, kErrNaN);
      }
    }
    if (kept) {
      *ch.wm_sum += (double)bw;  // MWM of mcmc.cpp:636
      *ch.nkept += 1;
    }
    ch.sweep[1] = sweep + 1;
    ch.done[1] = 0u;
  }
}

}  // namespace bsg
