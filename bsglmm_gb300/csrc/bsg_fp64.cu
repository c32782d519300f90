// bsg_fp64.cu -- the colour kernel of FP64 chains: the whole sweep in double
// precision on the sampler's Philox counters (latent draws, X'Z, the
// conditional precision and its Cholesky, the coefficient draw, the Omega
// pair sums, the Bartlett variates and the posterior sums).  A chain in this
// mode is the GPU form of the FP64 oracle chain (the C restatement of
// covar.cpp:121-325 and mcmc.cpp:584-651 on the same counters), fast enough
// to run the long reference chains that the FP32 sampler's maps are
// measured against at the brain-sized studies, where the CPU would take
// days.  One thread per voxel, subjects in order, or (few voxels, many
// subjects) four lanes per voxel.
//
// What bounds it is the FP64 pipe (two lanes per clock and SM: a warp's
// operation takes 16 cycles), so the latent draw is written for FP64
// operations: about 55 + 2 P per subject and voxel.  With CUDA's normcdf and
// normcdfinv, which it used before, an update took some 330 of them, 2,120
// instructions in all, since the lanes of a warp go down both branches of each.
#include "../../include/bsglmm_gb300.h"
#include "bsg_mills_table.h"
#include "bsg_wishart.cuh"

namespace bsg {
namespace {

constexpr int kF64Chunk = 512;  // subjects of the design staged per pass
constexpr int kF64Unroll = 2;   // subjects drawn side by side
constexpr long long kATailBits = 0x4014000000000000ll;  // kATail = 5.0
constexpr int kATailHi = 0x40140000;                    // its high word
static_assert(kATail == 5.0f, "the bits above");
constexpr uint32_t kFarHi = 0xC0428000u;  // high word of -37.0

// The tables of the draw, in shared memory (lanes index them apart).
struct DrawTables {
  double mills[kMillsCoef][kMillsRows];
  double exp2[64];
  double centre[kMillsRows];  // row / 8
};

__device__ void load_tables(DrawTables &tb, int tid, int nthreads) {
  for (int t = tid; t < kMillsRows * kMillsCoef; t += nthreads)
    tb.mills[t % kMillsCoef][t / kMillsCoef] = kMillsTable[t];
  for (int t = tid; t < 64; t += nthreads) tb.exp2[t] = kExp2Table[t];
  for (int t = tid; t < kMillsRows; t += nthreads) tb.centre[t] = 0.125 * t;
}

// Mills ratio (1 - Phi(x)) / phi(x) for x = row / 8 + h, |h| <= 1/16 (and a
// little over: rows are picked in FP32).
__device__ __forceinline__ double mills(uint32_t row, double h, const DrawTables &tb) {
  double c = tb.mills[kMillsCoef - 1][row];
#pragma unroll
  for (int i = kMillsCoef - 2; i >= 0; --i) c = fma(c, h, tb.mills[i][row]);
  return c;
}

// The row of x: the nearest multiple of 1/8.  Beyond the table (x > 11.06) the
// last one, with h = 0: there Q(x) < 1e-28 only ever meets u >= 2^-33.
__device__ __forceinline__ uint32_t mills_row(float x) {
  return min((uint32_t)__float2int_rn(x * 8.f), (uint32_t)kMillsRows - 1u);
}
constexpr float kMillsEnd = 11.0625f;

// exp(y + dy) for |y| <= 700 and a tiny dy (-0.0: none) by a table of 2^(j/64)
// and a polynomial of degree 5 (Tang 1989).  n log(2)/64 is exact in its
// leading part for the |n| < 2^17 that occur.
__device__ __forceinline__ double exp_tab(double y, double dy, const DrawTables &tb) {
  const double m = fma(y, 9.23324826168936568e+01, 0x1.8p52);
  const int n = __double2loint(m);
  const double k = m - 0x1.8p52;
  const double r = fma(k, -2.98158582698529328e-12, fma(k, -0x1.62e42fee00000p-7, y)) + dy;
  double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  q = fma(q, r, 1.0 / 6.0);
  q = fma(q, r, 0.5);
  q = fma(q, r, 1.0);
  const double t = tb.exp2[n & 63];
  const double e = fma(t, q * r, t);
  return __hiloint2double(__double2hiint(e) + ((n >> 6) << 20), __double2loint(e));
}

__device__ __forceinline__ double flip_sign_d(double x, bool flip) {
  return __hiloint2double(__double2hiint(x) ^ (flip ? (int)0x80000000 : 0), __double2loint(x));
}

// N(0,1) truncated to (a, +inf), -37 < a <= kATail (beyond, what it returns is
// replaced), by inversion of u(k) in FP64:
// t = Phi^-1(Phi(a) + u Q(a)).  With T = Q(|a|) the upper tail of t is
// p = T (1 - u) for a >= 0 and (1 - u) - T (1 - u) for a < 0; there, where
// the lower tail p = u + T (1 - u) is below 1/2, it is taken instead, so that
// the small side keeps its relative precision.  x = Q^-1(p) starts from the
// FP32 sampler's inversion (relative error d of 1e-6) and takes one step of
// the series of Q(x + d) = p to third order, which leaves d^4:
//   F = (Q(x) - p) / phi(x) = R(x) - p sqrt(2 pi) exp(x^2 / 2),
//   d = F + x F^2 / 2 + (2 x^2 + 1) F^3 / 6.
__device__ __forceinline__ double tn_lower_inv_d(double a, uint32_t k, const DrawTables &tb) {
  constexpr double kSqrt2Pi = 2.50662827463100069;
  // u = (k + 1/2) 2^-32 exactly, from the double 2^52 + k; so is 1 - u
  const double u = fma(__hiloint2double(0x43300000, (int)k), 0x1p-32, -0x1p20 + 0x1p-33);
  const double uc = 1.0 - u;
  const bool neg = __double2hiint(a) < 0;
  const double ax = fabs(a);
  // FP32: which tail, and the starting point
  const float fa = (float)ax;
  const float fu = u_of(k), fuc = u_of(~k), fT = phi_tail(fa);
  const float ftuc = __fmul_rn(fT, fuc), fq = fmaf(fT, fuc, fu);
  const bool lo = neg && fq < 0.5f;
  const float x0 = -ndtri_lower(lo ? fq : (neg ? __fsub_rn(fuc, ftuc) : ftuc));
  // T sqrt(2 pi) = R(|a|) exp(-a^2 / 2), a^2 with its rounding error
  const double a2 = ax * ax, a2l = fma(ax, ax, -a2);
  const uint32_t ra = mills_row(fa);
  const double ha = fa > kMillsEnd ? 0.0 : ax - tb.centre[ra];
  const double T = mills(ra, ha, tb) * exp_tab(-0.5 * a2, -0.5 * a2l, tb);
  const double A = lo ? u : (neg ? uc : 0.0);
  const double p = fma(flip_sign_d(uc, neg && !lo), T, A * kSqrt2Pi);
  const double x = (double)x0, xx = x * x;  // exact
  const uint32_t rx = mills_row(x0);
  const double hx = (double)(x0 > kMillsEnd ? 0.f : x0 - 0.125f * (float)rx);  // exact
  const double F = fma(-p, exp_tab(0.5 * xx, -0.0, tb), mills(rx, hx, tb));
  double d = fma(F, fma(xx, 1.0 / 3.0, 1.0 / 6.0), 0.5 * x);
  d = fma(F, d, 1.0);
  return flip_sign_d(fma(F, d, x), lo);
}

// The same for a <= -37: 1 - Q(a) is below 1e-299 and only ever meets u >=
// 2^-33, while a^2 / 2 would leave exp_tab's range.
__device__ __noinline__ double tn_lower_far_d(uint32_t k) { return normal_of_d(k); }

// a > kATail: the Robert (1995) exponential-proposal rejection of
// tn_lower_tail in FP64, on the same counters and attempt order.
__device__ __noinline__ double tn_lower_tail_d(double a, uint32_t i, uint32_t v,
                                               uint32_t sweep, uint32_t c3,
                                               uint32_t key0, uint32_t key1, int *ok) {
  const double as = 0.5 * (a + sqrt(a * a + 4.0));
  for (int q = 0; q < kTailMax / 2; ++q) {
    const uint4 r = philox1(make_uint4(i * 8u + (uint32_t)q, v, sweep, c3), key0, key1);
    double x = a - log(u_of_d(r.x)) / as, d = x - as;
    if (log(u_of_d(r.y)) < -0.5 * d * d) return x;
    x = a - log(u_of_d(r.z)) / as;
    d = x - as;
    if (log(u_of_d(r.w)) < -0.5 * d * d) return x;
  }
  *ok = 0;
  return a;
}

// Abramowitz & Stegun 26.2.17 in FP64, as the reference's CPU compute_prb
// evaluates it (covar.cpp:327-348).
__device__ double prob_sdnorm_d(double x) {
  const double b1 = 0.319381530, b2 = -0.356563782, b3 = 1.781477937;
  const double b4 = -1.821255978, b5 = 1.330274429, p = 0.2316419;
  const double c = 0.39894228;
  const double t = 1.0 / (1.0 + p * fabs(x));
  const double tail = c * exp(-x * x / 2.0) * t *
                      (t * (t * (t * (t * b5 + b4) + b3) + b2) + b1);
  return x >= 0.0 ? 1.0 - tail : tail;
}

// Sum of one value over the blocks' partials (value-major), in a fixed
// order: lane l takes the blocks l, l + 32, ...; then the lanes are
// combined.  One warp.
__device__ double sum_rows(const double *base, int nrow, int lane) {
  double s = 0.0;
  for (int r = lane; r < nrow; r += 32) s += __ldcg(base + r);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// LPV lanes per voxel, each taking every LPV-th group of four subjects.  A
// warp alone issues an FP64 operation every 80 cycles or so (18,848 voxels on
// one lane each put two warps on an SM: FP64 pipe 38 % busy), and four or five
// fill the pipe; see f64_lanes for the rule.
template <int P, int LPV>
__global__ void __launch_bounds__(kF64Threads)
    fp64_colour_kernel(const DatasetDev *__restrict__ dsv, ChainDev *__restrict__ chv,
                       const BlockMap *__restrict__ map, int colour) {
  constexpr int NT = P * (P + 1) / 2;
  __shared__ DrawTables tb;
  __shared__ double Xs[kF64Chunk * P];
  __shared__ double Om[P * P], Xtx[P * P];
  __shared__ double red[kF64Threads / 32][kFusedVals];
  __shared__ double tot[kFusedVals];
  __shared__ int is_last;

  const BlockMap bm = map[blockIdx.x];
  ChainDev &ch = chv[bm.chain];
  const DatasetDev &d = dsv[bm.dataset];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nc = d.n[colour];
  const int lane_v = tid % LPV;  // this lane's share of the subjects
  const int j = bm.start + tid / LPV;
  const bool active = j < nc;
  const int N = d.N, Vp = d.Vp;
  const long long sweep_ll = ch.sweep[colour];
  const uint32_t sweep = (uint32_t)sweep_ll, cid = ch.chain_id << 8;
  const bool kept =
      sweep_ll > ch.burnin && (sweep_ll % (ch.thin > 0 ? ch.thin : 1)) == 0;
  const double *b64 = ch.beta64;

  double beta[P], acc[P], bwm = 0.0;
  int v = 0, sc = 0;
  if (active) {
    sc = d.nb[colour][j];
    v = d.vidx[colour][j];
    bwm = (double)*ch.wm_beta * (d.wm ? (double)d.wm[v] : 1.0);
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    beta[p] = active ? b64[(size_t)p * Vp + sc] : 0.0;
    acc[p] = 0.0;
  }
  int ok = 1;
  const uint32_t *yb = d.ybits[colour];
  load_tables(tb, tid, blockDim.x);

  // ---- latent Z_iv for every subject, accumulated into X'(Z - b_WM WM)
  // (updateZ, covar.cpp:302-325, and the b of Spat_Coefff, covar.cpp:142-150)
  for (int i0 = 0; i0 < N; i0 += kF64Chunk) {
    const int cn = min(kF64Chunk, N - i0);
    __syncthreads();
    for (int t = tid; t < P * cn; t += blockDim.x) {
      const int p = t / cn, ii = t - p * cn;
      Xs[ii * P + p] = (double)d.covar[(size_t)p * N + i0 + ii];
    }
    __syncthreads();
    if (!active) continue;
    auto yload = [&](int ii) -> uint32_t {
      return ii < cn ? __ldg(yb + (size_t)((i0 + ii) >> 5) * nc + j) : 0u;
    };
    uint32_t ynext = yload(4 * lane_v);
    for (int ii0 = 4 * lane_v; ii0 < cn; ii0 += 4 * LPV) {
      const uint32_t yw = ynext;
      ynext = yload(ii0 + 4 * LPV);
      const uint4 r = philox1(make_uint4((uint32_t)((i0 + ii0) >> 2), (uint32_t)v, sweep,
                                         cid | kTagZ), ch.key0, ch.key1);
      // kF64Unroll subjects at a time (their draws are independent and hide
      // each other's latency); the last group may be short
#pragma unroll
      for (int h = 0; h < 4; h += kF64Unroll) {
        const int ii = ii0 + h, i = i0 + ii;  // i0 is a multiple of 32
        if (ii >= cn) break;
        double mu[kF64Unroll], t[kF64Unroll], a[kF64Unroll];
        bool y[kF64Unroll];
        bool far = false;
#pragma unroll
        for (int q = 0; q < kF64Unroll; ++q) {
          const int iq = min(ii + q, cn - 1);  // (a short group repeats its last)
          mu[q] = bwm;
#pragma unroll
          for (int p = 0; p < P; ++p) mu[q] += beta[p] * Xs[iq * P + p];
          y[q] = (yw >> ((i + q) & 31)) & 1u;
          a[q] = flip_sign_d(mu[q], y[q]);
          t[q] = tn_lower_inv_d(a[q], pick4(r, h + q), tb);
          // a > kATail or a <= -37, by the high words (a NaN counts as far)
          const int hi = __double2hiint(a[q]);
          far = far || hi >= kATailHi || (uint32_t)hi >= kFarHi;
        }
        if (far) {
#pragma unroll
          for (int q = 0; q < kF64Unroll; ++q) {
            if (ii + q >= cn) continue;
            if (__double_as_longlong(a[q]) > kATailBits)
              t[q] = tn_lower_tail_d(a[q], (uint32_t)(i + q), (uint32_t)v, sweep,
                                     cid | kTagZTail, ch.key0, ch.key1, &ok);
            else if ((uint32_t)__double2hiint(a[q]) >= kFarHi)
              t[q] = tn_lower_far_d(pick4(r, h + q));
          }
        }
#pragma unroll
        for (int q = 0; q < kF64Unroll; ++q) {
          if (ii + q < cn) {
            const double zr = mu[q] + flip_sign_d(t[q], !y[q]) - bwm;  // Z - b_WM WM
#pragma unroll
            for (int p = 0; p < P; ++p) acc[p] += Xs[(ii + q) * P + p] * zr;
          }
        }
      }
    }
  }
#pragma unroll
  for (int o = LPV / 2; o > 0; o >>= 1)
#pragma unroll
    for (int p = 0; p < P; ++p) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], o);

  // ---- beta_v | rest (Spat_Coefff, covar.cpp:142-180), production form
  for (int t = tid; t < P * P; t += blockDim.x) {
    Om[t] = ch.omega_d[t];
    Xtx[t] = (double)d.xtx[t];
  }
  __syncthreads();
  int err = ok ? 0 : kErrTnCap;
  double bnew[P], pv[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) pv[q] = 0.0;
  if (active && lane_v == 0) {
    double sumV[P];
#pragma unroll
    for (int p = 0; p < P; ++p) sumV[p] = 0.0;
    for (int t = 1; t <= 6; ++t) {
      const int sn = d.nb[colour][(size_t)t * nc + j];
#pragma unroll
      for (int p = 0; p < P; ++p) sumV[p] += b64[(size_t)p * Vp + sn];
    }
    const unsigned nbm = d.nbm[colour][j];
    const double nnb = (double)__popc(nbm);
    double b[P], Q[NT], e[P];
#pragma unroll
    for (int a = 0; a < P; ++a) {
      double s = acc[a];
#pragma unroll
      for (int q = 0; q < P; ++q) s += Om[q + a * P] * sumV[q];
      b[a] = s;
#pragma unroll
      for (int q = 0; q <= a; ++q) Q[tri(a, q)] = Xtx[q + a * P] + nnb * Om[q + a * P];
    }
    const bool okc = chol_packed<P>(Q);
#pragma unroll
    for (int p0 = 0; p0 < P; p0 += 4) {
      const uint4 rb = philox1(
          make_uint4((uint32_t)(p0 >> 2), (uint32_t)v, sweep, cid | kTagBeta), ch.key0,
          ch.key1);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (p0 + q < P) e[p0 + q] = normal_of_d(pick4(rb, q));
    }
    // Q = G G': beta = G^-T (G^-1 b + e), mean Q^-1 b and covariance Q^-1
    solve_lower<P>(Q, b);
#pragma unroll
    for (int p = 0; p < P; ++p) bnew[p] = b[p] + e[p];
    solve_upper<P>(Q, bnew);
    bool fin = true;
#pragma unroll
    for (int p = 0; p < P; ++p) fin = fin && isfinite(bnew[p]);
    if (okc && fin) {
#pragma unroll
      for (int p = 0; p < P; ++p) {
        ch.beta64[(size_t)p * Vp + sc] = bnew[p];
        ch.beta[(size_t)p * Vp + sc] = (float)bnew[p];
      }
    } else {
#pragma unroll
      for (int p = 0; p < P; ++p) bnew[p] = beta[p];
    }
    err |= (okc ? 0 : kErrChol) | ((okc && !fin) ? kErrNaN : 0);

    // ---- posterior running sums of the kept sweep (mcmc.cpp:637-645)
    if (kept) {
#pragma unroll
      for (int p = 0; p < P; ++p) {
        ch.acc_sum[(size_t)p * d.V + v] += bnew[p];
        ch.acc_sq[(size_t)p * d.V + v] += bnew[p] * bnew[p];
      }
#pragma unroll
      for (int g2 = 0; g2 < P; ++g2)
        if (g2 < d.S) ch.prb_sum[(size_t)g2 * d.V + v] += prob_sdnorm_d(bnew[g2] + bwm);
    }

    // ---- Omega pair products of the voxel's edges (colour 1 sees every
    // in-mask edge once), with the reference's indicator (covar.cpp:235-253)
    if (colour == 1) {
      for (int t = 0; t < 6; ++t) {
        const int sn = d.nb[1][(size_t)(t + 1) * nc + j];
        const bool fwd = t & 1;
        const bool nin = (nbm >> t) & 1u;
        double dd[P];
        bool ind[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const double bn = b64[(size_t)p * Vp + sn];
          dd[p] = bnew[p] - bn;
          ind[p] = fwd ? (bn != 0.0) : (nin && bnew[p] != 0.0);
        }
#pragma unroll
        for (int r2 = 0; r2 < P; ++r2)
          if (ind[r2]) {
#pragma unroll
            for (int c2 = 0; c2 <= r2; ++c2) pv[tri(r2, c2)] += dd[r2] * dd[c2];
          }
      }
    }
  } else {
#pragma unroll
    for (int p = 0; p < P; ++p) bnew[p] = 0.0;  // no column-sum share
  }
  if (err) {
    atomicOr(ch.status, err);
    atomicOr(ch.any_status, err);
  }

  // ---- block partials (FP64 warp trees), the last block of each colour
  // sums them in block order; colour 0's also draws the Bartlett variates,
  // colour 1's draws Omega
  constexpr int kColOff = kMaxPairs;
  constexpr int NV = NT + P;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    if (colour == 0 && q < NT) continue;
    double val = q < NT ? pv[q] : bnew[q - NT];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
    if (lane == 0) red[warp][q < NT ? q : kColOff + (q - NT)] = val;
  }
  __syncthreads();
  const int nwarp = kF64Threads / 32;
  constexpr int kVox = kF64Threads / LPV;  // voxels per block
  const int lb = bm.start / kVox;
  const int nblk = max(1, (nc + kVox - 1) / kVox);
  if (colour == 0) {
    if (tid < P) {
      double s = 0.0;
      for (int w = 0; w < nwarp; ++w) s += red[w][kColOff + tid];
      ch.partials0[(size_t)tid * ch.pstride0 + lb] = s;
      __threadfence();
    }
    __syncthreads();
    if (tid == 0) is_last = atomicAdd(ch.done, 1u) == (unsigned)(nblk - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int m = warp; m < P; m += nwarp) {
      const double s = sum_rows(ch.partials0 + (size_t)m * ch.pstride0, nblk, lane);
      if (lane == 0) ch.tot0[m] = s;
    }
    if (warp == nwarp - 1) {
      const int e = __reduce_or_sync(0xffffffffu,
                                     wishart_draws<true>(ch, d, sweep_ll, lane, ch.wdraw));
      if (e && lane == 0) {
        atomicOr(ch.status, e);
        atomicOr(ch.any_status, e);
      }
    }
    __syncthreads();
    if (tid == 0) {
      ch.sweep[0] = sweep_ll + 1;
      ch.done[0] = 0u;
      __threadfence();
    }
    return;
  }
  if (tid < NV) {
    const int q = tid < NT ? tid : kColOff + (tid - NT);
    double s = 0.0;
    for (int w = 0; w < nwarp; ++w) s += red[w][q];
    ch.partials1[(size_t)q * ch.pstride1 + lb] = s;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) is_last = atomicAdd(ch.done + 1, 1u) == (unsigned)(nblk - 1);
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  for (int m = warp; m < NV; m += nwarp) {
    const int q = m < NT ? m : kColOff + (m - NT);
    double s = sum_rows(ch.partials1 + (size_t)q * ch.pstride1, nblk, lane);
    if (q >= kColOff) s += __ldcg(ch.tot0 + (q - kColOff));
    if (lane == 0) tot[q] = s;
  }
  __syncthreads();
  if (warp == 0) wishart_warp<P>(ch, tot, 0, Supplied{}, lane);
  if (warp == 1) sweep_end_warp(ch, d, tot, sweep_ll, kept, 0, lane);
}

// Self-check of the latent draw: t[i] = tn_lower_inv_d(a[i], k[i]).
__global__ void draw64_selftest_kernel(int64_t n, const double *a, const uint32_t *k,
                                       double *t) {
  __shared__ DrawTables tb;
  load_tables(tb, threadIdx.x, blockDim.x);
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) t[i] = tn_lower_inv_d(a[i], k[i], tb);
}

// Self-check of div_by against the division, bit for bit, over mantissas of all kinds
// and exponents within 2^40, and of rsqrt_step: its largest relative error, in
// units of 2^-53, from the remainder 1 - d y^2 taken to twice the precision.
__global__ void quotient_selftest_kernel(int64_t n, uint32_t k0, uint32_t k1,
                                         unsigned long long *out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint4 r = philox1(make_uint4((uint32_t)i, (uint32_t)(i >> 32), 2u, 0xA5u), k0, k1);
  auto mant = [](uint32_t w, int kind) -> uint32_t {  // random, or next to a power of two
    const uint32_t m = w & 0x7fffffu;
    return kind == 0 ? m & 7u : kind == 1 ? 0x7fffffu - (m & 7u) : m;
  };
  auto expo = [](uint32_t w) -> uint32_t { return 127u - 40u + (w >> 24) % 81u; };
  const float x = __uint_as_float((r.x & 0x80000000u) | expo(r.y << 1) << 23 |
                                  mant(r.x, (int)(r.z & 7u)));
  const float g = __uint_as_float(expo(r.y >> 9 << 24 | r.y) << 23 |
                                  mant(r.y, (int)(r.z >> 3 & 7u)));
  if (__float_as_uint(div_by(x, g, 1.f / g)) != __float_as_uint(x / g)) atomicAdd(out, 1ull);
  const double d = __hiloint2double((int)((1023u - 60u + (r.z >> 8) % 121u) << 20 |
                                          (r.w & 0xfffffu)), (int)(r.x * 2654435761u ^ r.w));
  const double y = rsqrt_step(d), y2 = y * y, lo = fma(y, y, -y2);
  const double e = 0.5 * (fma(-d, y2, 1.0) - d * lo);
  atomicMax(out + 1, (unsigned long long)(fabs(e) * 0x1p53 * 1000.0));
}

}  // namespace

cudaError_t launch_fp64(int P, int lanes, const DatasetDev *ds, ChainDev *ch,
                        const BlockMap *map, int nblocks, int colour, cudaStream_t st) {
  if (nblocks <= 0) return cudaSuccess;
  switch (P) {
#define BSG_F64(PP)                                                                    \
  case PP:                                                                             \
    if (lanes == 1)                                                                    \
      fp64_colour_kernel<PP, 1><<<nblocks, kF64Threads, 0, st>>>(ds, ch, map, colour); \
    else                                                                               \
      fp64_colour_kernel<PP, kF64Lanes>                                                \
          <<<nblocks, kF64Threads, 0, st>>>(ds, ch, map, colour);                      \
    break;
    BSG_F64(1)
    BSG_F64(2)
    BSG_F64(3)
    BSG_F64(4)
    BSG_F64(5)
    BSG_F64(6)
    BSG_F64(7)
    BSG_F64(8)
#undef BSG_F64
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace bsg

extern "C" bsg_status bsg_selftest_draw64(int32_t device, int64_t n, const double *a,
                                          const uint32_t *k, double *t) {
  if (n < 1 || n > (1 << 26) || !a || !k || !t) return BSG_ERR_INVALID;
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) return BSG_ERR_NO_DEVICE;
  if (cudaSetDevice(device) != cudaSuccess) return BSG_ERR_INVALID;
  double *buf = nullptr;  // a, t, k
  if (cudaMalloc(&buf, (size_t)n * 20) != cudaSuccess) return BSG_ERR_CUDA;
  uint32_t *dk = (uint32_t *)(buf + 2 * n);
  cudaError_t e = cudaMemcpy(buf, a, (size_t)n * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dk, k, (size_t)n * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    bsg::draw64_selftest_kernel<<<(unsigned)((n + 127) / 128), 128>>>(n, buf, dk, buf + n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(t, buf + n, (size_t)n * 8, cudaMemcpyDeviceToHost);
  cudaFree(buf);
  return e == cudaSuccess ? BSG_OK : BSG_ERR_CUDA;
}

extern "C" bsg_status bsg_selftest_quotients(int32_t device, int64_t n, uint64_t seed,
                                             int64_t *mismatches, double *rsqrt_error) {
  if (n < 1 || n > (1ll << 36) || !mismatches || !rsqrt_error) return BSG_ERR_INVALID;
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) return BSG_ERR_NO_DEVICE;
  if (cudaSetDevice(device) != cudaSuccess) return BSG_ERR_INVALID;
  unsigned long long *out = nullptr, h[2] = {0, 0};
  if (cudaMalloc(&out, sizeof(h)) != cudaSuccess) return BSG_ERR_CUDA;
  cudaError_t e = cudaMemset(out, 0, sizeof(h));
  if (e == cudaSuccess) {
    bsg::quotient_selftest_kernel<<<(unsigned)((n + 255) / 256), 256>>>(
        n, (uint32_t)seed, (uint32_t)(seed >> 32), out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(out);
  if (e != cudaSuccess) return BSG_ERR_CUDA;
  *mismatches = (int64_t)h[0];
  *rsqrt_error = (double)h[1] / 1000.0;
  return BSG_OK;
}
