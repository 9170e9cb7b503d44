// Fisher matrices of the batched plans, pespace/inference/fisher.py:27-162:
// F_ij = 4 df Re sum_{det, c, f} conj(dh_i) dh_j / S_c(f).  FP64 plans take
// the derivatives of the A/E/T model with respect to the 11 parameters by
// forward-mode dual numbers in FP64 at every live bin (the same per-bin model
// as the FP64 plan; IMRPhenomHM: the six modes' links summed per detector);
// mixed IMRPhenomD plans by FP32 duals with the model's structure
// (k_fisher_fast below), mixed IMRPhenomHM plans as the FP64 ones.
// A block of 64 threads evaluates 64 bins of one detector, stores
// sqrt(w) dh in shared memory, and its threads then form the 66 pair sums of
// those bins; per-block partials are summed in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "pes_ff.cuh"
#include "pes_freq.cuh"
#include "pes_plan.cuh"

namespace pes {

constexpr int kFisherThreads = 64;
constexpr int kFisherBlocks = 48;  // blocks per sample, grid-stride over the live bins
constexpr int kPairs = 66;         // a <= b of 11 parameters
using FisherScalar = Dual<11>;

__device__ __forceinline__ void pair_of(int p, int& a, int& b) {
  a = 0;
  while (p >= 11 - a) {
    p -= 11 - a;
    ++a;
  }
  b = a + p;
}

// hmb: the samples' IMRPhenomHM mode coefficients (IMRPhenomHM plans: the
// six modes' links summed per detector, antenna.py:446-458), else null.
__global__ void __launch_bounds__(kFisherThreads) k_fisher_bins(PlanDev P,
                                                                const SampleBlock<FisherScalar>* __restrict__ blocks,
                                                                const PhenomHMCoef<FisherScalar>* __restrict__ hmb,
                                                                double* __restrict__ partial) {
  using T = FisherScalar;
  __shared__ SampleBlock<T> sb;
  __shared__ double dh[kFisherThreads][3][22];  // sqrt(w) dRe h / dtheta_a, then sqrt(w) dIm h / dtheta_a
  const int s = blockIdx.y, t = threadIdx.x;
  {
    const int n8 = sizeof(SampleBlock<T>) / 8;
    const double* src = reinterpret_cast<const double*>(&blocks[s]);
    double* dst = reinterpret_cast<double*>(&sb);
    for (int j = t; j < n8; j += kFisherThreads) dst[j] = src[j];
  }
  __syncthreads();
  int pa[2], pb[2];
  bool own[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int p = t + k * kFisherThreads;
    own[k] = p < kPairs;
    pair_of(own[k] ? p : 0, pa[k], pb[k]);
  }
  double acc[2] = {0.0, 0.0};
  if (sb.status == kSampleOk) {
    for (int64_t base = (int64_t)blockIdx.x * kFisherThreads; base < sb.kcut;
         base += (int64_t)gridDim.x * kFisherThreads) {
      const int64_t i = base + t;
      const bool live = i < sb.kcut;
      const double f = (double)(P.k0 + (live ? i : 0)) * P.f_step;
      Cx<T> hp, hc, ts;
      T tft;
      if (live) {
        dsincos((-2.0 * kPi * f) * sb.tc, &ts.im, &ts.re);
        if (!hmb) {
          T Mf = sb.wf.Msec * f;
          T amp, psi, tf;
          phenomd_eval<T>(sb.wf, Mf, amp, psi, tf);
          T sn, cs;
          dsincos(psi, &sn, &cs);
          T ap = sb.wf.pfac * amp, ac = sb.wf.cfac * amp;
          hp = cx(ap * cs, -(ap * sn));
          hc = cx(-(ac * sn), -(ac * cs));
          hp = cmul(hp, ts);
          hc = cmul(hc, ts);
          tft = tf + sb.tc;
        }
      }
      for (int d = 0; d < P.n_det; ++d) {
        if (live) {
          Cx<T> L[6], C[3];
          if (hmb) {
#pragma unroll
            for (int l = 0; l < 6; ++l) L[l] = cx(lift<T>(0.0), lift<T>(0.0));
#pragma unroll 1
            for (int k = 0; k < kHMModes; ++k) {
              Cx<T> mhp, mhc, Lk[6];
              T mtft;
              if (!hm_mode_container<T>(sb, hmb[s], k, f, ts, mhp, mhc, mtft)) continue;
              single_links<T>(P.orbit[d], f, mhp, mhc, mtft, sb.pol, Lk);
#pragma unroll
              for (int l = 0; l < 6; ++l) L[l] = L[l] + Lk[l];
            }
          } else {
            single_links<T>(P.orbit[d], f, hp, hc, tft, sb.pol, L);
          }
          const TdiFactor dp = P.tdi[d * P.nbins + i];
          tdi_channels<T>(cx(dp.dre, dp.dim), cx(dp.pre, dp.pim), 1, L, C);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double sw = sqrt(P.w[((size_t)d * 3 + c) * P.nbins + i]);  // zero off the channel mask
#pragma unroll
            for (int a = 0; a < 11; ++a) {
              dh[t][c][a] = sw * C[c].re.d[a];
              dh[t][c][11 + a] = sw * C[c].im.d[a];
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int a = 0; a < 22; ++a) dh[t][c][a] = 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (!own[k]) continue;
          const int a = pa[k], b = pb[k];
          double x = 0.0;
          for (int u = 0; u < kFisherThreads; ++u)
#pragma unroll
            for (int c = 0; c < 3; ++c) x += dh[u][c][a] * dh[u][c][b] + dh[u][c][11 + a] * dh[u][c][11 + b];
          acc[k] += x;
        }
        __syncthreads();
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (own[k]) partial[((size_t)s * gridDim.x + blockIdx.x) * kPairs + t + k * kFisherThreads] = acc[k];
}

__global__ void k_fisher_final(const SampleBlock<FisherScalar>* __restrict__ blocks, int64_t B, int nblk,
                               double scale, const double* __restrict__ partial, double* __restrict__ fisher,
                               int32_t* __restrict__ status) {
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (tid >= B * kPairs) return;
  const int64_t s = tid / kPairs;
  const int p = (int)(tid % kPairs);
  int a, b;
  pair_of(p, a, b);
  const bool ok = blocks[s].status == kSampleOk;
  double x = 0.0;
  for (int k = 0; k < nblk; ++k) x += partial[((size_t)s * nblk + k) * kPairs + p];
  const double v = ok ? scale * x : NAN;
  fisher[s * 121 + a * 11 + b] = v;
  fisher[s * 121 + b * 11 + a] = v;
  if (status && p == 0) status[s] = blocks[s].status;
}

// Fisher matrices of mixed IMRPhenomD plans in FP32, by the structure of the
// model: h_c = A Y_c(T, lambda, sin beta, psi, cos iota) exp(-i phase), T = t(f) + t_c,
// phase = Psi + 2 pi f (k.x0(T, lambda, sin beta) + t_c), with A, Psi, t(f)
// depending on the mass and spin parameters only.  Its derivatives are
//   dh/dtheta = (d(A Y)/dtheta - i A Y dphase/dtheta) exp(-i phase),
// and the phase factor cancels in conj(dh_a) dh_b, so the Fisher needs no
// phase values.  The waveform's part per bin (A, t(f) and the tangents of A, Psi
// and t(f), in float-float) is linear in the tangents of the model's coefficients: Horner
// sums over tabulated powers of f, each sample's coefficients rescaled to them.
// The response per unit amplitude takes FP32 duals over (T, lambda, sin beta,
// psi, cos iota); ln D_L and phi_c are analytic (dh = -h and 2 i h).
//
// Four warps evaluate 128 bins of one detector and store sqrt(w) times the 11
// complex derivatives in shared memory; a fifth sums the 66 pairs over the
// previous 128 (two buffers; FP32 within the 128 bins in their
// order, FP64 across).  A lane takes up to three pairs of one row, so that it
// loads 4 complex numbers for 6 products (a thread per pair loaded 12 values for
// 6, three of four warps waiting).  Float-float dual numbers through the
// waveform, and FP64 square roots and conversions of the weights per bin, took
// most of the time before: 100 samples on 125 410 bins 5.21 -> 2.04 ms, and 1.88 ms with
// two groups of 128 bins per block, whose warps fetch the same code; 1.98 ms with A's
// tangents in float-float too (about 5 500 FP32 operations per bin and detector, most of
// them in the response).
constexpr int kFastThreads = 128;  // bins per group
constexpr int kFastGroups = 2;     // groups per block
constexpr int kFastBins = kFastThreads * kFastGroups;
constexpr int kFastBlock = kFastBins + 32 * kFastGroups;  // and a summing warp per group
constexpr int kFastRows = 152 * kFastGroups;              // small calls: partial sums of the whole call
using FR = DualS<5>;                           // T, lambda, sin beta, psi, cos iota

// Per bin, for the FP32 frequency that the response takes too: f, f^{1/3} | 1/f,
// ln(f)/3 | f^{-5/3}, f^{-1/4} (hi, lo pairs) and f^{-7/6}.
__global__ void k_fisher_grid(PlanDev P, float4* __restrict__ rows, float2* __restrict__ p76) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.nbins) return;
  const double f = (double)(float)((double)(P.k0 + i) * P.f_step);
  const double u = cbrt(f);
  auto row = [](double a, double b) {
    const FF x = ff_from(a), y = ff_from(b);
    return make_float4(x.hi, x.lo, y.hi, y.lo);
  };
  rows[i] = row(f, u);
  rows[P.nbins + i] = row(1.0 / f, log(f) / 3.0);
  rows[2 * P.nbins + i] = row(1.0 / (f * u * u), 1.0 / sqrt(sqrt(f)));
  const FF g = ff_from(1.0 / (f * sqrt(u)));
  p76[i] = make_float2(g.hi, g.lo);
}

// A bin's TDI factors and the square roots of its weights over the amplitudes'
// scale (zero off the channel mask) in FP32: [n_det][nbins] rows (D, P), (A, E, T, 0).
__global__ void k_fisher_weights(PlanDev P, double inv_scale2, float4* __restrict__ wt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int d = blockIdx.y;
  if (i >= P.nbins) return;
  const TdiFactor t = P.tdi[(size_t)d * P.nbins + i];
  const double* w = P.w + (size_t)d * 3 * P.nbins + i;
  float4* o = wt + (size_t)d * 2 * P.nbins + i;
  o[0] = make_float4((float)t.dre, (float)t.dim, (float)t.pre, (float)t.pim);
  o[P.nbins] = make_float4((float)sqrt(w[0] * inv_scale2), (float)sqrt(w[P.nbins] * inv_scale2),
                           (float)sqrt(w[2 * P.nbins] * inv_scale2), 0.0f);
}

struct FisherSample {
  // phase tangents, [term][ln Mc, q, chi_1, chi_2] as hi, lo pairs
  float2 pin[12][4], lg0[4], lg1[4], pint[4][4], pm[5][4];
  // t(f): inspiral (j - 5) pin_j / (6 pi), lg / (6 pi); intermediate; merger-ringdown
  float2 rin[12], rl0, rl1, ri[3], rm[4];  // rm: pm1, pm2, 0.75 pm3, pm4 fd, over 2 pi
  float2 drin[12][4], drl0[4], drl1[4], dri[3][4], drm[4][4];
  float2 f5, ifd, fd, fd2, pm4, df5[4], dfd[4];
  // amplitude: a0 scaled; Ahat and its tangents (intermediate in (f - fc) / hw)
  float2 a0, ai[8], ei[5], fc, ihw, gm, wf, w2, fr, gx;
  float2 dlna0[4], dai[8][4], dei[5][4], dlngm[4], dw[4], dfr[4], dgx[4];
  float fj1, fj2, fa1, fa2;
  Polar<FR> pol;
  FR pfac, cfac;
  float tc;
  int32_t status, kcut;
};

// grid B: warp 0 the phase (a lane per tangent) and the polarisation, warp 1 the amplitude.
__global__ void __launch_bounds__(64) k_fisher_prep(double scale, const SampleBlock<FisherScalar>* __restrict__ blocks,
                                                    FisherSample* __restrict__ out) {
  const int s = blockIdx.x, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  FisherSample& o = out[s];
  const SampleBlock<FisherScalar>& b = blocks[s];
  if (b.status != kSampleOk) {  // uniform
    if (threadIdx.x == 0) {
      o.status = b.status;
      o.kcut = 0;
    }
    return;
  }
  auto ff2 = [](double x) {
    const FF q = ff_from(x);
    return make_float2(q.hi, q.lo);
  };
  if (wid == 0 && lane >= 8) {
    constexpr int npol = (int)(sizeof(Polar<FisherScalar>) / sizeof(FisherScalar));
    static_assert(sizeof(Polar<FR>) / sizeof(FR) == npol, "polarisation block must be an array of scalars");
    const FisherScalar* ps = reinterpret_cast<const FisherScalar*>(&b.pol);
    FR* pd = reinterpret_cast<FR*>(&o.pol);
    for (int k = lane - 8; k < npol; k += 24) {
      pd[k].v = (float)ps[k].v;
      pd[k].d[0] = 0.0f;
      pd[k].d[1] = (float)ps[k].d[6];  // lambda
      pd[k].d[2] = (float)ps[k].d[7];  // sin beta
      pd[k].d[3] = (float)ps[k].d[8];  // psi
      pd[k].d[4] = 0.0f;
    }
    if (lane == 31) {
      o.pfac.v = (float)b.wf.pfac.v;
      o.cfac.v = (float)b.wf.cfac.v;
#pragma unroll
      for (int a = 0; a < 4; ++a) o.pfac.d[a] = o.cfac.d[a] = 0.0f;
      o.pfac.d[4] = (float)b.wf.pfac.d[5];  // cos iota
      o.cfac.d[4] = (float)b.wf.cfac.d[5];
      o.tc = (float)b.tc.v;
    }
    return;
  }
  if (lane >= 4) return;
  // this lane's tangent of the coefficients, rescaled to f in Hz
  using S = Dual<1>;
  PhenomDCoef<S> c;
  {
    const FisherScalar* src = reinterpret_cast<const FisherScalar*>(&b.wf);
    S* dst = reinterpret_cast<S*>(&c);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(c) / sizeof(S)); ++k) {
      dst[k].v = src[k].v;
      dst[k].d[0] = src[k].d[lane];
    }
  }
  FreqCoef<S> fc;
  const double iM = 1.0 / c.Msec.v;
  constexpr double i2p = 1.0 / (2.0 * kPi), i6p = 1.0 / (6.0 * kPi);
  if (wid == 0) {
    freq_coef<S, kPhasePart>(c, fc);
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      const double r = (j - 5) * i6p;
      o.pin[j][lane] = ff2(fc.pin[j].d[0]);
      o.drin[j][lane] = ff2(r * fc.pin[j].d[0]);
      if (lane == 0) o.rin[j] = ff2(r * fc.pin[j].v);
    }
    o.lg0[lane] = ff2(fc.lg0.d[0]);
    o.lg1[lane] = ff2(fc.lg1.d[0]);
    o.drl0[lane] = ff2(i6p * fc.lg0.d[0]);
    o.drl1[lane] = ff2(i6p * fc.lg1.d[0]);
#pragma unroll
    for (int j = 0; j < 4; ++j) o.pint[j][lane] = ff2((j == 3 ? 3.0 : 1.0) * fc.pint[j].d[0]);
    const S m4 = fc.pm[4] * fc.fd;
    const double rm[4] = {1.0, -1.0, 0.75, 1.0};
#pragma unroll
    for (int j = 0; j < 5; ++j) o.pm[j][lane] = ff2(fc.pm[j].d[0]);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double r = (j == 1 ? -3.0 : 1.0) * i2p;
      o.dri[j][lane] = ff2(r * fc.pint[1 + j].d[0]);
      if (lane == 0) o.ri[j] = ff2(r * fc.pint[1 + j].v);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const S x = j == 3 ? m4 : fc.pm[1 + j];
      o.drm[j][lane] = ff2(rm[j] * i2p * x.d[0]);
      if (lane == 0) o.rm[j] = ff2(rm[j] * i2p * x.v);
    }
    o.df5[lane] = ff2(fc.f5.d[0]);
    o.dfd[lane] = ff2(fc.fd.d[0]);
    if (lane == 0) {
      o.rl0 = ff2(i6p * fc.lg0.v);
      o.rl1 = ff2(i6p * fc.lg1.v);
      o.f5 = ff2(fc.f5.v);
      o.ifd = ff2(1.0 / fc.fd.v);
      o.fd = ff2(fc.fd.v);
      o.fd2 = ff2(fc.fd.v * fc.fd.v);
      o.pm4 = ff2(fc.pm[4].v);
      o.fj1 = (float)(kPhiJoinIns * iM);
      o.fj2 = (float)(0.5 * (c.fRD.v * iM));
      o.status = kSampleOk;
      o.kcut = (int32_t)b.kcut;
    }
    return;
  }
  freq_coef<S, kAmpPart>(c, fc);
  // the intermediate quartic about the middle of its range
  const double f1 = kAmpJoinIns * iM, f2 = c.fpeak.v * iM, hw = 0.5 * (f2 - f1), mid = 0.5 * (f1 + f2);
  {
    S e[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) e[j] = fc.dl[j];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int j = 3; j >= k; --j) e[j] = e[j] + e[j + 1] * mid;
    double pw = 1.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      o.dei[j][lane] = ff2(e[j].d[0] * pw);
      if (lane == 0) o.ei[j] = ff2(e[j].v * pw);
      pw *= hw;
    }
  }
  o.dlna0[lane] = ff2(fc.a0.d[0] / fc.a0.v);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    o.dai[j][lane] = ff2(fc.ai[j].d[0]);
    if (lane == 0) o.ai[j] = ff2(fc.ai[j].v);
  }
  o.dlngm[lane] = ff2(fc.gm.d[0] / fc.gm.v);
  o.dw[lane] = ff2(fc.w.d[0]);
  o.dfr[lane] = ff2(fc.fr.d[0]);
  o.dgx[lane] = ff2(fc.gx.d[0]);
  if (lane == 0) {
    o.a0 = ff2(fc.a0.v * scale);
    o.fc = ff2(mid);
    o.ihw = ff2(1.0 / hw);
    o.gm = ff2(fc.gm.v);
    o.wf = ff2(fc.w.v);
    o.w2 = ff2(fc.w.v * fc.w.v);
    o.fr = ff2(fc.fr.v);
    o.gx = ff2(fc.gx.v);
    o.fa1 = (float)f1;
    o.fa2 = (float)f2;
  }
}

__device__ __forceinline__ FF ff_load(const float2& a) { return ff_make(a.x, a.y); }

// The waveform's part of a bin: amplitude, t(f), and the tangents over ln Mc, q, chi_1, chi_2.
struct WaveTangents {
  float A, tf;
  float dA[4], ps[4], dt[4];
};
__device__ __forceinline__ void wave_tangents(const FisherSample& sb, const float4* __restrict__ rows,
                                              const float2* __restrict__ p76, int64_t n, int64_t i, WaveTangents& o) {
  float (&ps)[4] = o.ps, (&dt)[4] = o.dt;
  const float4 r0 = rows[i], r1 = rows[n + i], r2 = rows[2 * n + i];
  const FF ff = ff_make(r0.x, r0.y), uu = ff_make(r0.z, r0.w), jj = ff_make(r1.x, r1.y), ll = ff_make(r1.z, r1.w);
  const float f = ff.hi;
  // ---- phase tangents, t(f) and its tangents
  FF tf;
  if (f < sb.fj1) {
    const FF iu5 = ff_make(r2.x, r2.y);
    FF R = ff_load(sb.rin[11]);
#pragma unroll
    for (int j = 10; j >= 0; --j) R = ff_mad(R, uu, ff_load(sb.rin[j]));
    const FF ul = uu * ff_addf(ll, 1.0f);
    const FF l1 = ff_mad(ff_load(sb.rl1), ul, ff_load(sb.rl0));
    tf = ff_mad(R, iu5, l1);
    tf = jj * ff_fast_two_sum(tf.hi, tf.lo);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      FF p = ff_load(sb.pin[11][k]);
      FF r = ff_load(sb.drin[11][k]);
#pragma unroll
      for (int j = 10; j >= 0; --j) {
        p = ff_mad(p, uu, ff_load(sb.pin[j][k]));
        r = ff_mad(r, uu, ff_load(sb.drin[j][k]));
      }
      const FF l = ff_mad(ff_load(sb.lg1[k]), uu, ff_load(sb.lg0[k])) * ll;
      p = ff_mad(p, iu5, l);
      ps[k] = p.hi + p.lo;
      r = ff_mad(r, iu5, ff_mad(ff_load(sb.drl1[k]), ul, ff_load(sb.drl0[k])));
      dt[k] = (jj * ff_fast_two_sum(r.hi, r.lo)).hi;
    }
  } else if (f < sb.fj2) {
    const FF j3 = (jj * jj) * jj;
    const FF j4 = j3 * jj;
    tf = ff_mad(ff_load(sb.ri[1]), j4, ff_load(sb.ri[0]));
    tf = ff_mad(ff_load(sb.ri[2]), jj, tf);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      FF p = ff_mad(ff_load(sb.pint[1][k]), ff, ff_load(sb.pint[0][k]));
      p = ff_mad(ff_load(sb.pint[2][k]), j3, p);
      p = ff_mad(ff_load(sb.pint[3][k]), ll, p);
      ps[k] = p.hi + p.lo;
      const FF r = ff_mad(ff_load(sb.dri[2][k]), jj, ff_mad(ff_load(sb.dri[1][k]), j4, ff_load(sb.dri[0][k])));
      dt[k] = r.hi + r.lo;
    }
  } else {
    const FF q = ff_make(r2.z, r2.w), fq = ff * q;
    const FF xx = ff - ff_load(sb.f5);
    const FF rd = ff_make(1.0f, 0.0f) / (xx * xx + ff_load(sb.fd2));
    const FF fd = ff_load(sb.fd), m4 = -(ff_load(sb.pm4) * rd), rm4 = ff_mulf(ff_load(sb.rm[3]) * rd, 2.0f) * rd;
    const FF at = datan(xx * ff_load(sb.ifd));
    tf = ff_mad(ff_load(sb.rm[1]), jj * jj, ff_load(sb.rm[0]));
    tf = ff_mad(ff_load(sb.rm[2]), q, tf);
    tf = ff_mad(ff_load(sb.rm[3]), rd, tf);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      FF p = ff_mad(ff_load(sb.pm[1][k]), ff, ff_load(sb.pm[0][k]));
      p = ff_mad(ff_load(sb.pm[2][k]), jj, p);
      p = ff_mad(ff_load(sb.pm[3][k]), fq, p);
      p = ff_mad(ff_load(sb.pm[4][k]), at, p);
      const FF d5 = ff_load(sb.df5[k]), dd = ff_load(sb.dfd[k]);
      p = ff_mad(m4, ff_dot2(d5, fd, xx, dd), p);
      ps[k] = p.hi + p.lo;
      FF r = ff_mad(ff_load(sb.drm[1][k]), jj * jj, ff_load(sb.drm[0][k]));
      r = ff_mad(ff_load(sb.drm[2][k]), q, r);
      r = ff_mad(ff_load(sb.drm[3][k]), rd, r);
      r = ff_mad(rm4, ff_dot2(xx, d5, -fd, dd), r);  // rm[3] times the tangent of rd
      dt[k] = r.hi + r.lo;
    }
  }
  tf = ff_fast_two_sum(tf.hi, tf.lo);
  o.tf = tf.hi;
  // ---- amplitude, the tangents of its logarithm
  FF ah, da[4];
  if (f < sb.fa1) {
    FF p = ff_load(sb.ai[7]);
#pragma unroll
    for (int j = 6; j >= 0; --j) p = ff_mad(p, uu, ff_load(sb.ai[j]));
    ah = ff_addf(ff_fast_two_sum(p.hi, p.lo) * (uu * uu), 1.0f);
    const FF g = uu * uu / ah;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      FF r = ff_load(sb.dai[7][k]);
#pragma unroll
      for (int j = 6; j >= 0; --j) r = ff_mad(r, uu, ff_load(sb.dai[j][k]));
      da[k] = ff_mad(r, g, ff_load(sb.dlna0[k]));
    }
  } else if (f < sb.fa2) {
    const FF xx = (ff - ff_load(sb.fc)) * ff_load(sb.ihw);
    ah = ff_load(sb.ei[4]);
#pragma unroll
    for (int j = 3; j >= 0; --j) ah = ff_mad(ah, xx, ff_load(sb.ei[j]));
    ah = ff_fast_two_sum(ah.hi, ah.lo);
    const FF g = ff_make(1.0f, 0.0f) / ah;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      FF r = ff_load(sb.dei[4][k]);
#pragma unroll
      for (int j = 3; j >= 0; --j) r = ff_mad(r, xx, ff_load(sb.dei[j][k]));
      da[k] = ff_mad(r, g, ff_load(sb.dlna0[k]));
    }
  } else {
    const FF xx = ff - ff_load(sb.fr);
    const FF den = xx * xx + ff_load(sb.w2), gx = ff_load(sb.gx), w = ff_load(sb.wf);
    const FF rw2 = ff_make(2.0f, 0.0f) / den;
    ah = ff_load(sb.gm) / den * dexp(-(gx * xx));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const FF dr = ff_load(sb.dfr[k]);
      const FF c = ff_load(sb.dlna0[k]) + ff_load(sb.dlngm[k]);
      da[k] = ff_mad(rw2, ff_dot2(xx, dr, -w, ff_load(sb.dw[k])), ff_add_lazy(c, ff_dot2(gx, dr, -ff_load(sb.dgx[k]), xx)));
    }
  }
  const FF A = ff_load(sb.a0) * ff_load(p76[i]) * ah;
  o.A = A.hi;
#pragma unroll
  for (int k = 0; k < 4; ++k) o.dA[k] = (A * ff_fast_two_sum(da[k].hi, da[k].lo)).hi;
}

// The summing warp's share: rows of the upper triangle in pieces of up to three pairs, one per lane.
__device__ __forceinline__ void pairs_of(int lane, int& a, int& b, int& count) {
  a = 0;
  for (int piece = lane; a < 11; ++a) {
    const int pieces = (11 - a + 2) / 3;
    if (piece < pieces) {
      b = a + 3 * piece;
      count = min(3, 11 - b);
      return;
    }
    piece -= pieces;
  }
  a = b = count = 0;
}

constexpr size_t fisher_smem() { return 2 * sizeof(float2) * kFastBins * 3 * 11; }

// grid (blocks, B), grid-stride over pairs of groups of 128 live bins.
__global__ void __launch_bounds__(kFastBlock, 1) k_fisher_fast(PlanDev P, const FisherSample* __restrict__ samples,
                                                               const float4* __restrict__ rows,
                                                               const float2* __restrict__ p76,
                                                               const float4* __restrict__ wt,
                                                               double* __restrict__ partial) {
  extern __shared__ float2 dh_buf[];  // [2][bin][channel][11]: sqrt(w) dh / dtheta_a
  __shared__ FisherSample sb;
  __shared__ OrbitF orb[PES_MAX_DETECTORS];
  const int s = blockIdx.y, t = threadIdx.x;
  const int64_t n = P.nbins;
  {
    const int* src = reinterpret_cast<const int*>(&samples[s]);
    int* dst = reinterpret_cast<int*>(&sb);
    for (int k = t; k < (int)(sizeof(FisherSample) / 4); k += kFastBlock) dst[k] = src[k];
    if (t < P.n_det) orb[t] = orbit_f(P.orbit[t]);
  }
  __syncthreads();
  const int kcut = sb.status == kSampleOk ? sb.kcut : 0;
  const bool summing = t >= kFastBins;
  const int grp = summing ? (t - kFastBins) >> 5 : t / kFastThreads;
  int pa = 0, pb = 0, np = 0;
  if (summing) pairs_of(t & 31, pa, pb, np);
  double acc[3] = {0.0, 0.0, 0.0};
  WaveTangents wv;
  int step = 0;  // (group, detector) pairs evaluated so far
  const int first = blockIdx.x * kFastBins, stride = gridDim.x * kFastBins;
  const int steps = first < kcut ? (kcut - first + stride - 1) / stride * P.n_det : 0;
  for (; step <= steps; ++step) {
    float2* buf = dh_buf + (size_t)(step & 1) * (kFastBins * 33);
    if (!summing && step < steps) {
      const int d = step % P.n_det;
      const int i = first + step / P.n_det * stride + t;
      float2* dst = buf + t * 33;
      if (i < kcut) {
        const float f = rows[i].x;
        if (d == 0) wave_tangents(sb, rows, p76, n, i, wv);
        const float4 td = wt[(size_t)d * 2 * n + i], sw3 = wt[((size_t)d * 2 + 1) * n + i];
        Cx<FR> Y[3];
        FR kx0;
        {
          FR T = lift<FR>(0.0);
          T.v = wv.tf + sb.tc;
          T.d[0] = 1.0f;
          const FR zero = lift<FR>(0.0);
          Cx<FR> L[6];
          single_links_impl<true, FR>(orb[d], f, cx(sb.pfac, zero), cx(zero, -sb.cfac), T, sb.pol, L, &kx0);
          tdi_channels_t<true, FR>(cx(lift<FR>(td.x), lift<FR>(td.y)), cx(lift<FR>(td.z), lift<FR>(td.w)), 1, L, Y);
        }
        const float A = wv.A, tp = 6.283185307179586f * f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float sw = c == 0 ? sw3.x : (c == 1 ? sw3.y : sw3.z);
          const FR& Yr = Y[c].re;
          const FR& Yi = Y[c].im;
          const float ar = A * Yr.v, ai = A * Yi.v;  // A Y
          float ur[11], ui[11];
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // ln Mc, q, chi_1, chi_2
            const float dA = wv.dA[k], dt = wv.dt[k];
            const float ph = wv.ps[k] + tp * kx0.d[0] * dt;
            ur[k] = dA * Yr.v + A * Yr.d[0] * dt + ai * ph;
            ui[k] = dA * Yi.v + A * Yi.d[0] * dt - ar * ph;
          }
          ur[4] = -ar;  // ln D_L: dh = -h
          ui[4] = -ai;
          ur[5] = A * Yr.d[4];  // cos iota
          ui[5] = A * Yi.d[4];
          ur[6] = A * Yr.d[1] + ai * tp * kx0.d[1];  // lambda
          ui[6] = A * Yi.d[1] - ar * tp * kx0.d[1];
          ur[7] = A * Yr.d[2] + ai * tp * kx0.d[2];  // sin beta
          ui[7] = A * Yi.d[2] - ar * tp * kx0.d[2];
          ur[8] = A * Yr.d[3];  // psi
          ui[8] = A * Yi.d[3];
          ur[9] = -2.0f * ai;  // phi_c: dh = 2 i h
          ui[9] = 2.0f * ar;
          const float pt = tp * (kx0.d[0] + 1.0f);  // t_c
          ur[10] = A * Yr.d[0] + ai * pt;
          ui[10] = A * Yi.d[0] - ar * pt;
#pragma unroll
          for (int a = 0; a < 11; ++a) dst[c * 11 + a] = make_float2(sw * ur[a], sw * ui[a]);
        }
      } else {
        for (int a = 0; a < 33; ++a) dst[a] = make_float2(0.0f, 0.0f);
      }
    }
    if (summing && step > 0) {
      const float2* src = dh_buf + (size_t)((step & 1) ^ 1) * (kFastBins * 33) + grp * (kFastThreads * 33);
      float x[3] = {0.0f, 0.0f, 0.0f};
      const int b1 = min(pb + 1, 10), b2 = min(pb + 2, 10);
#pragma unroll 4
      for (int u = 0; u < kFastThreads * 3; ++u) {
        const float2* q = src + u * 11;
        const float2 va = q[pa], v0 = q[pb], v1 = q[b1], v2 = q[b2];
        x[0] = fmaf(va.x, v0.x, fmaf(va.y, v0.y, x[0]));
        x[1] = fmaf(va.x, v1.x, fmaf(va.y, v1.y, x[1]));
        x[2] = fmaf(va.x, v2.x, fmaf(va.y, v2.y, x[2]));
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) acc[k] += (double)x[k];
    }
    __syncthreads();
  }
  if (summing)
    for (int k = 0; k < np; ++k)
      partial[((size_t)s * gridDim.x * kFastGroups + blockIdx.x * kFastGroups + grp) * kPairs + (pa * 11 - pa * (pa - 1) / 2 + (pb + k - pa))] = acc[k];
}

// The first call's buffers and tables (fisher_blocks last: it marks them complete).
// The tables are filled on a stream of their own: later calls may come on another
// stream, and the caller's may be capturing a graph.
static int fisher_create(PesPlan* p, bool fast) {
  const int64_t M = p->desc.max_batch, n = p->desc.nbins, nd = p->desc.n_det;
  const int64_t rows = std::max<int64_t>(M * kFisherBlocks, kFastRows + M * (int64_t)kFastGroups);
  PES_CHECK_CUDA(cudaMalloc(&p->fisher_partial, sizeof(double) * rows * kPairs));
  if (fast) {
    PES_CHECK_CUDA(cudaMalloc(&p->fisher_samples, sizeof(FisherSample) * M));
    PES_CHECK_CUDA(cudaMalloc(&p->fisher_rows, sizeof(float4) * n * (3 + 2 * nd)));
    PES_CHECK_CUDA(cudaMalloc(&p->fisher_p76, sizeof(float2) * n));
    PES_CHECK_CUDA(cudaFuncSetAttribute(k_fisher_fast, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fisher_smem()));
    cudaStream_t own;
    PES_CHECK_CUDA(cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking));
    k_fisher_grid<<<ceil_div(n, 128), 128, 0, own>>>(p->dev, p->fisher_rows, p->fisher_p76);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(own);
    cudaStreamDestroy(own);
    PES_CHECK_CUDA(e);
  }
  PES_CHECK_CUDA(cudaMalloc(&p->fisher_blocks, sizeof(SampleBlock<FisherScalar>) * M));
  return PES_OK;
}

}  // namespace pes

using namespace pes;

extern "C" int pes_fisher_batch(PesPlan* p, const double* theta, int64_t B, double* fisher, int32_t* status,
                                void* stream) {
  PES_REQUIRE(p, "pes_fisher_batch: null plan");
  PES_REQUIRE(B >= 0 && B <= p->desc.max_batch, "pes_fisher_batch: batch size %lld outside [0, max_batch=%d]",
              (long long)B, p->desc.max_batch);
  PES_REQUIRE(B == 0 || (theta && fisher), "pes_fisher_batch: null theta or fisher");
  const unsigned need = (1u << p->desc.n_det) - 1u;
  PES_REQUIRE((p->data_set_mask & need) == need, "pes_fisher_batch: PSD not set for every detector (pes_plan_set_data)");
  if (B == 0) return PES_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool hm = p->desc.approximant == PES_APPROX_PHENOMHM, fast = p->mixed && !hm;
  const int64_t n = p->desc.nbins, nd = p->desc.n_det;
  // partial sums per sample: kFisherBlocks, more in calls that would leave SMs idle
  const int64_t nrow = !fast ? (int64_t)kFisherBlocks
                             : std::min<int64_t>(ceil_div(n, kFastThreads),
                                                 std::max<int64_t>(kFisherBlocks, ceil_div(kFastRows, B)));
  const int64_t nblk = !fast ? nrow : ceil_div(nrow, kFastGroups) * (int64_t)kFastGroups;
  if (!p->fisher_blocks) {
    const int rc = fisher_create(p, fast);
    if (rc != PES_OK) {  // a later call begins again
      cudaFree(p->fisher_partial);
      cudaFree(p->fisher_samples);
      cudaFree(p->fisher_rows);
      cudaFree(p->fisher_p76);
      p->fisher_partial = nullptr;
      p->fisher_samples = nullptr;
      p->fisher_rows = nullptr;
      p->fisher_p76 = nullptr;
      return rc;
    }
  }
  auto* blocks = reinterpret_cast<SampleBlock<FisherScalar>*>(p->fisher_blocks);
  k_setup<FisherScalar><<<setup_blocks(B), 64, 0, st>>>(p->dev, theta, B, 0, blocks, hm_blocks<FisherScalar>(p));
  PES_CHECK_LAUNCH();
  if (fast) {  // mixed IMRPhenomD plans: FP32 structured derivatives
    auto* samples = reinterpret_cast<FisherSample*>(p->fisher_samples);
    float4* wt = p->fisher_rows + 3 * n;
    const float scale = (float)(kPc / (kMRSun * kMTSun));
    const double inv_scale2 = 1.0 / ((double)scale * (double)scale);
    k_fisher_weights<<<dim3(ceil_div(n, 128), (unsigned)nd), 128, 0, st>>>(p->dev, inv_scale2, wt);
    PES_CHECK_LAUNCH();
    k_fisher_prep<<<(unsigned)B, 64, 0, st>>>(scale, blocks, samples);
    PES_CHECK_LAUNCH();
    k_fisher_fast<<<dim3((unsigned)(nblk / kFastGroups), (unsigned)B), kFastBlock, fisher_smem(), st>>>(
        p->dev, samples, p->fisher_rows, p->fisher_p76, wt, p->fisher_partial);
  } else {  // FP64 plans and IMRPhenomHM: FP64 dual numbers through the whole model
    k_fisher_bins<<<dim3(kFisherBlocks, (unsigned)B), kFisherThreads, 0, st>>>(
        p->dev, blocks, hm ? hm_blocks<FisherScalar>(p) : nullptr, p->fisher_partial);
  }
  PES_CHECK_LAUNCH();
  k_fisher_final<<<(unsigned)ceil_div(B * kPairs, 128), 128, 0, st>>>(blocks, B, (int)nblk, 4.0 * p->dev.df,
                                                                       p->fisher_partial, fisher, status);
  PES_CHECK_LAUNCH();
  return PES_OK;
}
