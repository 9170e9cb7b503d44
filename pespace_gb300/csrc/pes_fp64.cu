// The dense FP64 path of IMRPhenomD plans: lnL and its 11-parameter gradient
// with every live bin evaluated in FP64.
//
// GB300 issues one FP64 instruction of a warp over 64 cycles (1/64 of the FP32
// rate), so the number of FP64 instructions per bin is the time; loads, integer
// work, table look-ups and even register spills hide behind them.  Per bin:
//
//  * powers and logarithms of f come from a table of the grid (plan set-up) and
//    the sample's coefficients are rescaled to them, so that the model needs no
//    cube root, logarithm, square root or division per bin in the inspiral;
//  * the arms' components along the polarisation axes and the node delays are
//    trigonometric polynomials of the orbital angle (of degree 2 for
//    heliocentric constellations, of degree 1 for geocentric ones), their
//    coefficients a 9-point transform per sample and detector; the third arm
//    and node are minus the sum of the others (465 -> 424 FP64 instructions per
//    bin against patterns of degree 4 for every arm);
//  * the constellation centre's delay joins the waveform's phase and t_c in one
//    sine and cosine, reduced in two parts and read from a 256-entry table with
//    short Taylor polynomials;
//  * sin(x)/x by its Taylor series, as long as the bin's largest argument needs;
//  * the gradient is the hand-written adjoint of that evaluation (one pass
//    whatever the number of parameters); the mass and spin parameters enter
//    linearly through the model's coefficients, so the pass accumulates the
//    adjoints of the coefficients over the bins and the tangents multiply their
//    sums once per sample (their set-up runs beside the dense pass).
//
// Measured: lnL and gradient of 12 samples on LISA + TianQin (2^20 s) 10.6 -> 0.97 ms
// against three passes of Dual<4> through the plain model; lnL of 37 samples on
// 65 471 bins 1.42 -> 0.88 ms (0.67 to 0.88 ms with the draws' live bins).  The FP64 pipe is active 88% of the cycles of
// either pass (424 and about 800 FP64 instructions per bin and detector).
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "pes_freq.cuh"
#include "pes_plan.cuh"

namespace pes {

constexpr int k64Threads = 128;
// Bins per thread: 4, or 1 for calls of up to k64SmallBlocks blocks of 128 bins.
// One warp per SM partition already saturates its FP64 pipe, so a call of
// fewer blocks than the chip holds takes as long as one thread's bins
// (one sample of 31 452 bins: 87 us at 4); larger calls share a block's
// prologue and the reduction of the gradient's accumulators over more bins.
constexpr int k64BinsPerThread = 4;
constexpr int k64SmallBlocks = 152 * 4 * 2;
// Block partials.  lnL needs one double per block, the gradient k64Acc; a gradient
// of many samples runs in chunks of them, so that its workspace is the larger of
// what k64GradRows blocks take (6.7 MB: 54 times the 304 gradient blocks that the
// chip holds, so that the chunks' last waves do not matter) and of k64RowDoubles
// doubles per block of the whole batch (51 made 10.9 GB of 4096 samples on
// 3 354 437 bins).
constexpr int64_t k64GradRows = 16384;
constexpr int k64RowDoubles = 5;

// ------------------------------------------------------------------ tables
// Per bin, seven rows of nbins: f, f^{1/3}, f^{-5/3} (rounded once: the phase's leading
// terms multiply its error by 1e5), ln(f)/3, 1/f, f^{-1/4}, f^{-7/6}.
enum { kGf, kGu, kGiu5, kGlf3, kGif, kGq, kGp76, kGridRows };
__global__ void k_grid64(PlanDev P, double* __restrict__ grid, double2* __restrict__ trig) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < kTrig) {
    double s, c;
    sincospi(2.0 * (double)i / kTrig, &s, &c);
    trig[i] = make_double2(s, c);
  }
  if (i >= P.nbins) return;
  const double f = (double)(P.k0 + i) * P.f_step;
  const double u = cbrt(f);
  grid[kGf * P.nbins + i] = f;
  grid[kGu * P.nbins + i] = u;
  {
    const DD c = dd_cbrt({f, 0.0});
    grid[kGiu5 * P.nbins + i] = dd_div(c, dd_mul({f, 0.0}, {f, 0.0})).h;
  }
  grid[kGlf3 * P.nbins + i] = log(f) / 3.0;
  grid[kGif * P.nbins + i] = 1.0 / f;
  grid[kGq * P.nbins + i] = 1.0 / sqrt(sqrt(f));
  grid[kGp76 * P.nbins + i] = 1.0 / (f * sqrt(u));
}

// The per-sample block of the dense pass.
struct Dense64Block {
  FreqCoef<double> c;
  double rin[12];                // (j-5) pin_j / (6 pi)
  double ifd, fd2, w2;           // 1/fd, fd^2, w^2
  double fj1, fj2, fa1, fa2;     // joins in Hz: phase 0.018, fRD/2; amplitude 0.014, fpeak
  double pfac, cfac, cosi, tc;
  int64_t kcut;
  int32_t status;
  int32_t pad;
};

constexpr int kLeadTerms = 5;  // pin[0..4], the first scalars of FreqCoef (pin[1] = 0)

// The set-up of one sample per block (grid B): warps 0 and 1 the two parts of
// the coefficient block (phenomd_setup) and then of its rescaled form, a warp per
// detector the response's polynomials beside them (in turn on one SM partition
// the chains took 38 + 40 us).
__global__ void __launch_bounds__(32 * (2 + PES_MAX_DETECTORS))
k_setup64(PlanDev P, const double* __restrict__ theta, SampleBlock<double>* __restrict__ blocks,
          Dense64Block* __restrict__ out, RespTab* __restrict__ resp) {
  __shared__ double rows[2][kFCount][3];
  __shared__ double2 w9[9];  // cos, sin of 2 pi m / 9
  __shared__ double v[PES_MAX_DETECTORS][27][6];  // [detector][set * 9 + angle]: n.p, n.q of two arms, y of two nodes
  const int s = blockIdx.x, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SampleBlock<double>& b = blocks[s];
  const double* th = theta + 11 * (int64_t)s;
  double raw[11];
#pragma unroll
  for (int j = 0; j < 11; ++j) raw[j] = th[j];
  Dense64Block& o = out[s];
  if (!theta_in_domain(raw)) {  // uniform per block
    if (threadIdx.x == 0) {
      b.status = o.status = kSampleOutOfDomain;
      b.kcut = o.kcut = 0;
      b.fcut = 0.0;
    }
    return;
  }
  nine_angles(w9);
  __syncthreads();
  if (wid < 2) {
    if (lane < kSetupLanes) {
      constexpr unsigned mask = (1u << kSetupLanes) - 1u;
      if (wid == 0)
        setup_part<double, kPhasePart, false>(P, raw, 0, lane, mask, rows[0], b, nullptr);
      else
        setup_part<double, kAmpPart, false>(P, raw, 0, lane, mask, rows[1], b, nullptr);
    }
  } else {
    response_tables(P, th, wid - 2, lane, v[wid - 2], w9, resp[(size_t)s * P.n_det + wid - 2]);
  }
  __syncthreads();
  if (lane != 0 || wid > 2) return;
  if (wid == 2) {
    // the leading phase terms' coefficients, rounded once (their phases reach 1e5 rad), beside the others
    const DD icu = dd_div({1.0, 0.0}, dd_cbrt({b.wf.Msec, 0.0})), icu2 = dd_mul(icu, icu), icu3 = dd_mul(icu2, icu);
    const double lead[kLeadTerms] = {dd_mul(dd_mul(icu3, icu2), {b.wf.pin[0], 0.0}).h, 0.0, dd_mul(icu3, {b.wf.pin[2], 0.0}).h,
                                     dd_mul(icu2, {b.wf.pin[3], 0.0}).h, dd_mul(icu, {b.wf.pin[4], 0.0}).h};
#pragma unroll
    for (int j = 0; j < kLeadTerms; ++j) {
      o.c.pin[j] = lead[j];
      o.rin[j] = lead[j] * ((j - 5) / (6.0 * kPi));
    }
    return;
  }
  const double iM = 1.0 / b.wf.Msec;
  FreqCoef<double> c;
  if (wid == 0) {
    freq_coef<double, kPhasePart>(b.wf, c);
    double* dst = reinterpret_cast<double*>(&o.c);
    const double* src = reinterpret_cast<const double*>(&c);
#pragma unroll
    for (int k = kLeadTerms; k < (int)(offsetof(FreqCoef<double>, a0) / sizeof(double)); ++k) dst[k] = src[k];
#pragma unroll
    for (int j = kLeadTerms; j < 12; ++j) o.rin[j] = c.pin[j] * ((j - 5) / (6.0 * kPi));
    o.ifd = 1.0 / c.fd;
    o.fd2 = c.fd * c.fd;
    o.fj1 = kPhiJoinIns * iM;
    o.fj2 = 0.5 * (b.wf.fRD * iM);
  } else {
    freq_coef<double, kAmpPart>(b.wf, c);
    double* dst = reinterpret_cast<double*>(&o.c);
    const double* src = reinterpret_cast<const double*>(&c);
#pragma unroll
    for (int k = (int)(offsetof(FreqCoef<double>, a0) / sizeof(double)); k < kFreqScalars; ++k) dst[k] = src[k];
    o.w2 = c.w * c.w;
    o.fa1 = kAmpJoinIns * iM;
    o.fa2 = b.wf.fpeak * iM;
    o.pfac = b.wf.pfac;
    o.cfac = b.wf.cfac;
    o.cosi = raw[5];
    o.tc = raw[10];
    o.status = b.status;
    o.kcut = b.kcut;
  }
}

// ------------------------------------------------------------------ the dense pass
// Accumulators of the gradient pass: the lnL sum; direct parameters; the
// adjoints of the FreqCoef scalars in their order.
enum { kAccR, kAccLnD, kAccCosi, kAccLam, kAccSb, kAccPsi, kAccPhic, kAccTc, kAccCoef };
constexpr int k64Acc = kAccCoef + kFreqScalars;

// One bin of one sample: sum over detectors of sum_c |d - h|^2 w; kGrad: its adjoints into acc.
template <bool kGrad>
__device__ __forceinline__ double bin64(const PlanDev& P, const Dense64Block& b, const RespTab* __restrict__ resp,
                                        const double2* __restrict__ tab, const double* __restrict__ grid, int64_t i,
                                        double* acc) {
  const int64_t n = P.nbins;
  const FreqCoef<double>& c = b.c;
  const double f = grid[kGf * n + i], u = grid[kGu * n + i], lf3 = grid[kGlf3 * n + i], jf = grid[kGif * n + i];
  // ---- phase and t(f)
  const int preg = f < b.fj1 ? 0 : (f < b.fj2 ? 1 : 2);
  double psi, tf, at = 0.0, rden = 0.0, q14 = 0.0, x5 = 0.0;
  if (preg == 0) {
    const double iu5 = grid[kGiu5 * n + i];
    double p = c.pin[11], r = b.rin[11];
#pragma unroll
    for (int j = 10; j >= 0; --j) {
      p = fma(p, u, c.pin[j]);
      if (j != 5) r = fma(r, u, b.rin[j]); else r *= u;
    }
    const double l1 = c.lg1 * u;
    psi = fma(p, iu5, (c.lg0 + l1) * lf3);
    tf = jf * fma(r, iu5, fma(l1, lf3 + 1.0, c.lg0) * (1.0 / (6.0 * kPi)));
  } else if (preg == 1) {
    const double jf2 = jf * jf, jf3 = jf2 * jf;
    psi = fma(c.pint[1], f, fma(c.pint[2], jf3, fma(c.pint[3], 3.0 * lf3, c.pint[0])));
    tf = fma(jf, fma(-3.0 * c.pint[2], jf3, c.pint[3]), c.pint[1]) * (1.0 / (2.0 * kPi));
  } else {
    q14 = grid[kGq * n + i];
    x5 = f - c.f5;
    rden = rcp64(fma(x5, x5, b.fd2));
    at = atan64(tab, x5 * b.ifd);
    psi = fma(c.pm[1], f, fma(c.pm[2], jf, fma(c.pm[3], f * q14, fma(c.pm[4], at, c.pm[0]))));
    tf = fma(-c.pm[2] * jf, jf, fma(0.75 * c.pm[3], q14, fma(c.pm[4] * c.fd, rden, c.pm[1]))) * (1.0 / (2.0 * kPi));
  }
  // ---- amplitude
  const int areg = f < b.fa1 ? 0 : (f < b.fa2 ? 1 : 2);
  double ah, rw = 0.0, xr = 0.0;
  if (areg == 0) {
    double p = c.ai[7];
#pragma unroll
    for (int j = 6; j >= 0; --j) p = fma(p, u, c.ai[j]);
    ah = fma(u * u, p, 1.0);
  } else if (areg == 1) {
    ah = fma(f, fma(f, fma(f, fma(f, c.dl[4], c.dl[3]), c.dl[2]), c.dl[1]), c.dl[0]);
  } else {
    xr = f - c.fr;
    rw = rcp64(fma(xr, xr, b.w2));
    ah = c.gm * rw * exp(-(c.gx * xr));
  }
  const double a0p = c.a0 * grid[kGp76 * n + i], A = a0p * ah;
  // ---- phase 2 pi f t_c, rounded as the plain formula's argument is, whole turns removed
  const double w2 = (2.0 * kPi) * f;
  const double ptc = turns64(w2 * b.tc);
  const double T = tf + b.tc, pif = kPi * f;
  double sum = 0.0;
  double reS = 0.0, imS = 0.0, RT = 0.0;  // adjoints of A (over A), of the phase and of T
  for (int d = 0; d < P.n_det; ++d) {
    const RespTab& R = resp[d];
    const PesOrbit& ob = P.orbit[d];
    // ---- harmonics of the orbital angle, arm components and delays
    double c1, s1, ca, sa;
    if (ob.kind == 0) {
      sincos64(tab, fma(ob.omega_revolution, T, ob.revolution_initial), &sa, &ca);
      c1 = ca;
      s1 = sa;
    } else {
      sincos64(tab, fma(ob.omega_revolution, T, ob.revolution_initial), &sa, &ca);
      sincos64(tab, fma(ob.omega_rotation, T, ob.rotation_initial), &s1, &c1);
    }
    double c2 = 0.0, s2 = 0.0;
    if (ob.kind == 0) {
      c2 = fma(c1, c1, -(s1 * s1));
      s2 = 2.0 * (s1 * c1);
    }
    auto poly = [&](const double* Y) {
      double v = fma(Y[1], c1, Y[2] * s1);
      if (ob.kind == 0) v += fma(Y[3], c2, fma(Y[4], s2, Y[0]));
      return v;
    };
    const double kx0 = fma(R.k0[0][0], ca, R.k0[0][1] * sa);
    // ---- e^{-i Phi} P(f) A
    double sn, cs;
    sincos64(tab, fma(w2, kx0, psi) + ptc, &sn, &cs);
    const TdiFactor tdi = P.tdi[(size_t)d * n + i];
    const double qr = fma(tdi.pre, cs, tdi.pim * sn), qi = fma(tdi.pim, cs, -(tdi.pre * sn));
    const double hqr = A * qr, hqi = A * qi;
    // ---- links per unit of that factor: l = sinc(x+-) b, b = a (gi - i gr) E
    const double a = pif * ob.arm_sec;
    const int tier = sinc_tier(2.0 * a);
    double th[3];
#pragma unroll
    for (int k = 0; k < 2; ++k) th[k] = pif * poly(R.y[0][k]);
    th[2] = -(th[0] + th[1]);
    double np[3], nq[3];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      np[k] = poly(R.np[0][k]);
      nq[k] = poly(R.nq[0][k]);
    }
    np[2] = np[0] + np[1];  // (its sign drops out of the patterns)
    nq[2] = nq[0] + nq[1];
    const double pfa2 = b.pfac * a, cfa2 = -2.0 * (b.cfac * a);
    double gr[3], gi[3], er[3], ei[3], br[3], bi[3], sp[3], sm[3], dsp[3], dsm[3], Fp[3], Fx[3];
    double lr[6], li[6];
#pragma unroll
    for (int pr = 0; pr < 3; ++pr) {
      const int k2 = (pr + 1) % 3;
      Fp[pr] = fma(np[pr], np[pr], -(nq[pr] * nq[pr]));
      Fx[pr] = np[pr] * nq[pr];  // half of Fx
      gr[pr] = pfa2 * Fp[pr];
      gi[pr] = cfa2 * Fx[pr];
      double es, ec;
      sincos64(tab, a - th[(pr + 2) % 3], &es, &ec);  // a + th[pr] + th[k2]
      er[pr] = ec;
      ei[pr] = -es;
      br[pr] = fma(gi[pr], ec, -(gr[pr] * es));
      bi[pr] = -fma(gi[pr], es, gr[pr] * ec);
      const double dl = th[k2] - th[pr];
      sinc64<kGrad>(tab, tier, a + dl, &sp[pr], &dsp[pr]);
      sinc64<kGrad>(tab, tier, a - dl, &sm[pr], &dsm[pr]);
      lr[2 * pr] = sp[pr] * br[pr];
      li[2 * pr] = sp[pr] * bi[pr];
      lr[2 * pr + 1] = sm[pr] * br[pr];
      li[2 * pr + 1] = sm[pr] * bi[pr];
    }
    // ---- TDI: X = (l13 - l12) + D (l31 - l21) and cyclic, A/E/T
    const double Dr = tdi.dre, Di = tdi.dim;
    double Xr[3], Xi[3];
    {
      const int p0[3] = {5, 1, 3}, p1[3] = {0, 2, 4}, q0[3] = {4, 0, 2}, q1[3] = {1, 3, 5};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double vr = lr[q0[k]] - lr[q1[k]], vi = li[q0[k]] - li[q1[k]];
        Xr[k] = (lr[p0[k]] - lr[p1[k]]) + fma(Dr, vr, -(Di * vi));
        Xi[k] = (li[p0[k]] - li[p1[k]]) + fma(Dr, vi, Di * vr);
      }
    }
    constexpr double r2 = 0.70710678118654752, r6 = 0.40824829046386302, r3 = 0.57735026918962576;
    double Yr[3], Yi[3];
    {
      const double tr = Xr[0] + Xr[2], ti = Xi[0] + Xi[2];
      Yr[0] = r2 * (Xr[2] - Xr[0]);
      Yi[0] = r2 * (Xi[2] - Xi[0]);
      Yr[1] = r6 * fma(-2.0, Xr[1], tr);
      Yi[1] = r6 * fma(-2.0, Xi[1], ti);
      Yr[2] = r3 * (tr + Xr[1]);
      Yi[2] = r3 * (ti + Xi[1]);
    }
    // ---- residual
    double Cr[3], Ci[3];  // adjoints of Y_c (cotangents: dR = Re sum C dY)
    double s0 = 0.0, s1_ = 0.0;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      if (!((P.chan_mask >> ch) & 1)) {
        if (kGrad) Cr[ch] = Ci[ch] = 0.0;
        continue;
      }
      const size_t off = ((size_t)d * 3 + ch) * n + i;
      const double w = P.w[off];
      const double2 dv = P.data[off];
      const double rr = dv.x - fma(hqr, Yr[ch], -(hqi * Yi[ch]));
      const double ri = dv.y - fma(hqr, Yi[ch], hqi * Yr[ch]);
      sum = fma(w, fma(rr, rr, ri * ri), sum);
      if (kGrad) {
        const double pr_ = -2.0 * w * rr, pi_ = 2.0 * w * ri;  // -2 w conj(d - h)
        // per unit amplitude: rho Q
        const double xr = fma(pr_, qr, -(pi_ * qi)), xi = fma(pr_, qi, pi_ * qr);
        s0 += fma(xr, Yr[ch], -(xi * Yi[ch]));
        s1_ += fma(xr, Yi[ch], xi * Yr[ch]);
        Cr[ch] = A * xr;
        Ci[ch] = A * xi;
      }
    }
    if (!kGrad) continue;
    reS += s0;
    const double iS = A * s1_;
    imS += iS;
    // ---- adjoint of TDI
    double Ar[3], Ai[3];  // of X, Y, Z
    {
      const double xr = r2 * Cr[0], xi = r2 * Ci[0], er_ = r6 * Cr[1], ei_ = r6 * Ci[1], tr = r3 * Cr[2], ti = r3 * Ci[2];
      const double etr = er_ + tr, eti = ei_ + ti;
      Ar[0] = etr - xr;
      Ai[0] = eti - xi;
      Ar[1] = fma(-2.0, er_, tr);
      Ai[1] = fma(-2.0, ei_, ti);
      Ar[2] = etr + xr;
      Ai[2] = eti + xi;
    }
    double DAr[3], DAi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      DAr[k] = fma(Dr, Ar[k], -(Di * Ai[k]));
      DAi[k] = fma(Dr, Ai[k], Di * Ar[k]);
    }
    // links 12, 21, 23, 32, 31, 13
    const double Lr[6] = {DAr[1] - Ar[0], Ar[1] - DAr[0], DAr[2] - Ar[1], Ar[2] - DAr[1], DAr[0] - Ar[2], Ar[0] - DAr[2]};
    const double Li[6] = {DAi[1] - Ai[0], Ai[1] - DAi[0], DAi[2] - Ai[1], Ai[2] - DAi[1], DAi[0] - Ai[2], Ai[0] - DAi[2]};
    // ---- adjoint of the links
    double tha[3] = {0.0, 0.0, 0.0}, Fpa[3], Fxa[3];
    double pfa = 0.0, cfa = 0.0;
#pragma unroll
    for (int pr = 0; pr < 3; ++pr) {
      const int k2 = (pr + 1) % 3;
      const double xp = (fma(Lr[2 * pr], br[pr], -(Li[2 * pr] * bi[pr]))) * dsp[pr];
      const double xm = (fma(Lr[2 * pr + 1], br[pr], -(Li[2 * pr + 1] * bi[pr]))) * dsm[pr];
      const double bar = fma(sp[pr], Lr[2 * pr], sm[pr] * Lr[2 * pr + 1]);
      const double bai = fma(sp[pr], Li[2 * pr], sm[pr] * Li[2 * pr + 1]);
      const double kr = fma(bar, er[pr], -(bai * ei[pr])), ki = fma(bar, ei[pr], bai * er[pr]);
      const double arg = fma(ki, gi[pr], -(kr * gr[pr]));
      const double dx = xp - xm;
      tha[k2] += arg + dx;
      tha[pr] += arg - dx;
      // db = (dgi - i dgr) E
      const double gra = a * ki, gia = a * kr;
      Fpa[pr] = b.pfac * gra;
      Fxa[pr] = -(b.cfac * gia);
      pfa = fma(gra, Fp[pr], pfa);
      cfa = fma(-2.0 * gia, Fx[pr], cfa);
    }
    // ---- adjoints of n.p, n.q and of the delays; the third of each is minus the others' sum
    double pa[3], qa[3];
#pragma unroll
    for (int pr = 0; pr < 3; ++pr) {
      const double fp2 = 2.0 * Fpa[pr], fx2 = 2.0 * Fxa[pr];
      pa[pr] = fma(fp2, np[pr], fx2 * nq[pr]);
      qa[pr] = fma(fx2, np[pr], -(fp2 * nq[pr]));
    }
    const double pa2[2] = {pa[0] + pa[2], pa[1] + pa[2]}, qa2[2] = {qa[0] + qa[2], qa[1] + qa[2]};
    const double ya[2] = {pif * (tha[0] - tha[2]), pif * (tha[1] - tha[2])};
    const double iSw = iS * w2;
    // ---- T: derivative of the polynomials with the orbital angle
    {
      double v = 0.0;
      const double c2d = 2.0 * c2, s2d = 2.0 * s2;
      auto dpoly = [&](const double* Y) {
        double x = fma(Y[2], c1, -(Y[1] * s1));
        if (ob.kind == 0) x = fma(Y[4], c2d, fma(-Y[3], s2d, x));
        return x;
      };
#pragma unroll
      for (int k = 0; k < 2; ++k)
        v = fma(pa2[k], dpoly(R.np[0][k]), fma(qa2[k], dpoly(R.nq[0][k]), fma(ya[k], dpoly(R.y[0][k]), v)));
      const double om = ob.kind == 0 ? ob.omega_revolution : ob.omega_rotation;
      const double dk = fma(R.k0[0][1], ca, -(R.k0[0][0] * sa));
      RT = fma(om, v, RT);
      RT = fma(iSw, ob.omega_revolution * dk, RT);
    }
    // ---- sky position, polarisation, inclination
#pragma unroll
    for (int st = 1; st < 3; ++st) {
      double v = iSw * fma(R.k0[st][0], ca, R.k0[st][1] * sa);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        v = fma(pa2[k], poly(R.np[st][k]), fma(qa2[k], poly(R.nq[st][k]), fma(ya[k], poly(R.y[st][k]), v)));
      acc[st == 1 ? kAccLam : kAccSb] += v;
    }
    {
      // dF+/dpsi = 2 Fx, dFx/dpsi = -2 F+ (Fx here halved)
      double v = 0.0;
#pragma unroll
      for (int pr = 0; pr < 3; ++pr) v += fma(2.0 * Fpa[pr], Fx[pr], -(Fxa[pr] * Fp[pr]));
      acc[kAccPsi] = fma(2.0, v, acc[kAccPsi]);
    }
    acc[kAccCosi] += fma(b.cosi, pfa, cfa);
  }
  if (!kGrad) return sum;
  // ---- waveform: adjoints of its coefficients
  const double rA = a0p * reS;  // dR / dAhat
  acc[kAccR] += sum;
  acc[kAccLnD] -= A * reS;
  acc[kAccPhic] -= 2.0 * imS;
  acc[kAccTc] += fma(w2, imS, RT);
  double* W = acc + kAccCoef;
#define PES_W(field) W[offsetof(FreqCoef<double>, field) / sizeof(double)]
  const double g2 = RT * (1.0 / (2.0 * kPi));
  if (preg == 0) {
    const double g = (RT * (1.0 / (6.0 * kPi))) * jf;
    double bj = grid[kGiu5 * n + i];
    double* wp = &PES_W(pin);
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      if (j != 1) wp[j] = fma(bj, j == 5 ? imS : fma(g, (double)(j - 5), imS), wp[j]);
      if (j < 11) bj *= u;
    }
    const double l = imS * lf3;
    PES_W(lg0) += l + g;
    PES_W(lg1) = fma(u, fma(g, lf3 + 1.0, l), PES_W(lg1));
  } else if (preg == 1) {
    const double jf2 = jf * jf, jf3 = jf2 * jf;
    double* wp = &PES_W(pint);
    wp[0] += imS;
    wp[1] += fma(imS, f, g2);
    wp[2] = fma(jf3, fma(-3.0 * g2, jf, imS), wp[2]);
    wp[3] += fma(3.0 * imS, lf3, g2 * jf);
  } else {
    double* wp = &PES_W(pm);
    wp[0] += imS;
    wp[1] += fma(imS, f, g2);
    wp[2] = fma(jf, fma(-g2, jf, imS), wp[2]);
    wp[3] = fma(q14, fma(imS, f, 0.75 * g2), wp[3]);
    wp[4] += fma(imS, at, g2 * (c.fd * rden));
    const double pr_ = c.pm[4] * rden;
    PES_W(f5) = fma(pr_ * c.fd, fma(2.0 * g2 * x5, rden, -imS), PES_W(f5));
    PES_W(fd) = fma(pr_, fma(g2, fma(-2.0 * b.fd2, rden, 1.0), -(imS * x5)), PES_W(fd));
  }
  PES_W(a0) = fma(rA, ah, PES_W(a0));
  if (areg == 0) {
    double bj = rA * u * u;
    double* wp = &PES_W(ai);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      wp[j] += bj;
      if (j < 7) bj *= u;
    }
  } else if (areg == 1) {
    double bj = rA;
    double* wp = &PES_W(dl);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      wp[j] += bj;
      if (j < 4) bj *= f;
    }
  } else {
    const double h = rA * ah;
    PES_W(gm) += h;
    PES_W(w) = fma(h, -2.0 * c.w * rw, PES_W(w));
    PES_W(fr) = fma(h, fma(2.0 * xr, rw, c.gx), PES_W(fr));
    PES_W(gx) = fma(-h, xr, PES_W(gx));
  }
#undef PES_W
  return sum;
}

template <bool kGrad>
constexpr size_t dense64_smem() {
  return kGrad ? sizeof(double) * (k64Threads / 32) * k64Acc * 33 : 0;
}

// grid (blocks of k64Threads * bpt bins, B); partial [B][nblk][1 or k64Acc], written by blocks with a live bin.
template <bool kGrad>
__global__ void __launch_bounds__(k64Threads) k_dense64(PlanDev P, const Dense64Block* __restrict__ blocks,
                                                        const RespTab* __restrict__ resp,
                                                        const double* __restrict__ grid,
                                                        const double2* __restrict__ trig, int nblk, int bpt,
                                                        double* __restrict__ partial) {
  extern __shared__ double red64[];
  __shared__ Dense64Block sb;
  __shared__ RespTab rt[PES_MAX_DETECTORS];
  __shared__ double2 tab[kTrig];
  const int s = blockIdx.y;
  const int64_t base = (int64_t)blockIdx.x * (k64Threads * bpt);
  if (blocks[s].status != kSampleOk || base >= blocks[s].kcut) return;  // uniform; the finaliser skips such blocks
  {
    const double* src = reinterpret_cast<const double*>(&blocks[s]);
    double* dst = reinterpret_cast<double*>(&sb);
    for (int j = threadIdx.x; j < (int)(sizeof(Dense64Block) / 8); j += k64Threads) dst[j] = src[j];
    src = reinterpret_cast<const double*>(resp + (size_t)s * P.n_det);
    dst = reinterpret_cast<double*>(rt);
    for (int j = threadIdx.x; j < (int)(sizeof(RespTab) / 8) * P.n_det; j += k64Threads) dst[j] = src[j];
    for (int j = threadIdx.x; j < kTrig; j += k64Threads) tab[j] = trig[j];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if constexpr (!kGrad) {
    double acc = 0.0;
#pragma unroll 1
    for (int j = 0; j < bpt; ++j) {
      const int64_t i = base + (int64_t)j * k64Threads + threadIdx.x;
      if (i < sb.kcut) acc += bin64<false>(P, sb, rt, tab, grid, i, nullptr);
    }
    __shared__ double red[k64Threads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) red[wid] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double x = 0.0;
#pragma unroll
      for (int k = 0; k < k64Threads / 32; ++k) x += red[k];
      partial[(size_t)s * nblk + blockIdx.x] = x;
    }
  } else {
    double acc[k64Acc];
#pragma unroll
    for (int k = 0; k < k64Acc; ++k) acc[k] = 0.0;
#pragma unroll 1
    for (int j = 0; j < bpt; ++j) {
      const int64_t i = base + (int64_t)j * k64Threads + threadIdx.x;
      if (i < sb.kcut) bin64<true>(P, sb, rt, tab, grid, i, acc);
    }
    // each warp's accumulators through shared memory (rows of 33): a lane sums a row
    double* m = red64 + (size_t)wid * k64Acc * 33;
#pragma unroll
    for (int k = 0; k < k64Acc; ++k) m[k * 33 + lane] = acc[k];
    __syncwarp();
    for (int k = lane; k < k64Acc; k += 32) {
      double x = 0.0;
#pragma unroll 8
      for (int l = 0; l < 32; ++l) x += m[k * 33 + l];
      m[k * 33] = x;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < k64Acc; k += k64Threads) {
      double x = 0.0;
#pragma unroll
      for (int w = 0; w < k64Threads / 32; ++w) x += red64[((size_t)w * k64Acc + k) * 33];
      partial[((size_t)s * nblk + blockIdx.x) * k64Acc + k] = x;
    }
  }
}

// One warp per sample: block partials in a fixed order.  kGrad: the tangents of
// the coefficients times their adjoints.
template <bool kGrad>
__global__ void __launch_bounds__(64) k_final64(PlanDev P, const Dense64Block* __restrict__ blocks, int64_t B, int nblk,
                                                int bpt, const double* __restrict__ partial,
                                                const SampleBlock<Dual<4>>* __restrict__ tan,
                                                double* __restrict__ lnl, double* __restrict__ grad,
                                                int32_t* __restrict__ status) {
  const int64_t s = blockIdx.x * 2 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (s >= B) return;
  const Dense64Block& b = blocks[s];
  if (b.status != kSampleOk) {
    if (lane == 0) {
      lnl[s] = -INFINITY;
      if (status) status[s] = b.status;
    }
    if (kGrad && lane < 11) grad[11 * s + lane] = 0.0;
    return;
  }
  const int live = (int)((b.kcut + k64Threads * bpt - 1) / (k64Threads * bpt));
  const double scale = -2.0 * P.df;
  constexpr int NV = kGrad ? k64Acc : 1;
  auto total = [&](int k) {
    double x = 0.0;
    for (int j = lane; j < live; j += 32) x += partial[((size_t)s * nblk + j) * NV + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  const double sum = total(kAccR);
  if (lane == 0) {
    const double v = scale * (sum + P.suffix[b.kcut]);
    lnl[s] = v;
    if (status) status[s] = isfinite(v) ? kSampleOk : kSampleNonFinite;
  }
  if constexpr (kGrad) {
    __shared__ double tot[2][k64Acc];
    double* t = tot[threadIdx.x >> 5];
    // a lane per accumulator (coalesced), blocks in order
    for (int k = lane; k < k64Acc; k += 32) {
      double x = 0.0;
      for (int j = 0; j < live; ++j) x += partial[((size_t)s * nblk + j) * NV + k];
      t[k] = x;
    }
    __syncwarp();
    if (lane < 4) {  // ln Mc, q, chi_1, chi_2: this lane's tangent of every coefficient
      using S = Dual<1>;
      PhenomDCoef<S> c;
      {
        const Dual<4>* src = reinterpret_cast<const Dual<4>*>(&tan[s].wf);
        S* dst = reinterpret_cast<S*>(&c);
#pragma unroll
        for (int k = 0; k < (int)(sizeof(c) / sizeof(S)); ++k) {
          dst[k].v = src[k].v;
          dst[k].d[0] = src[k].d[lane];
        }
      }
      FreqCoef<S> fc;
      freq_coef<S>(c, fc);
      const S* x = reinterpret_cast<const S*>(&fc);
      double g = 0.0;
#pragma unroll
      for (int k = 0; k < kFreqScalars; ++k) {
        double wk = t[kAccCoef + k];
        if (k == (int)(offsetof(FreqCoef<double>, a0) / sizeof(double))) wk /= b.c.a0;
        if (k == (int)(offsetof(FreqCoef<double>, gm) / sizeof(double))) wk /= b.c.gm;
        g += wk * x[k].d[0];
      }
      grad[11 * s + lane] = scale * g;
    } else if (lane < 11) {
      const int from[7] = {kAccLnD, kAccCosi, kAccLam, kAccSb, kAccPsi, kAccPhic, kAccTc};
      double g = 0.0;
#pragma unroll
      for (int k = 0; k < 7; ++k)
        if (lane == 4 + k) g = t[from[k]];
      grad[11 * s + lane] = scale * g;
    }
  }
}

// Coefficient blocks with the tangents of the mass and spin parameters, one
// thread per sample in the plain order of the formulae: the tangents of the
// intermediate amplitude's coefficients are ill-conditioned (1e-9 of some
// gradients), and this order is the one its results are known by.  It runs
// beside the dense pass, which does not read it; calls of a few samples wait for it
// (one sample on 7 839 bins: 255 us, lnL alone 90 us).
__global__ void k_tangents64(PlanDev P, const double* __restrict__ theta, int64_t B,
                             SampleBlock<Dual<4>>* __restrict__ blocks) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= B) return;
  double raw[11];
  for (int j = 0; j < 11; ++j) raw[j] = theta[11 * s + j];
  if (!theta_in_domain(raw)) return;
  using T = Dual<4>;
  T th[11];
  for (int j = 0; j < 11; ++j) th[j] = Seed<T>::make(raw[j], j < 4 ? j : -1);
  phenomd_setup_serial<T, 3>(th, P.f_ref, nullptr, 0, 1, 0u, blocks[s].wf);
}

// ------------------------------------------------------------------ host side
struct Fp64Buffers {
  double* grid = nullptr;
  double2* trig = nullptr;
  Dense64Block* blocks = nullptr;
  RespTab* resp = nullptr;
  double* partial = nullptr;
  int64_t grad_rows = 0;  // blocks of a gradient chunk that `partial` holds
  SampleBlock<Dual<4>>* tan = nullptr;
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};

int fp64_create(PesPlan* p) {
  Fp64Buffers* b = new Fp64Buffers();
  p->fp64 = b;
  const int64_t n = p->desc.nbins, B = p->desc.max_batch;
  // block partials: of the largest batch at 4 bins per thread, or of a small call at 1
  const int64_t nblk = ceil_div(n, k64Threads * k64BinsPerThread), rows = std::max<int64_t>(B * nblk, k64SmallBlocks);
  b->grad_rows = std::max(std::min(rows, k64GradRows), std::max(nblk, B * nblk * k64RowDoubles / k64Acc));
  const int64_t partial = std::max(rows, b->grad_rows * k64Acc);
  cudaError_t e = cudaMalloc(&b->grid, sizeof(double) * kGridRows * n);
  if (e == cudaSuccess) e = cudaMalloc(&b->trig, sizeof(double2) * kTrig);
  if (e == cudaSuccess) e = cudaMalloc(&b->blocks, sizeof(Dense64Block) * B);
  if (e == cudaSuccess) e = cudaMalloc(&b->resp, sizeof(RespTab) * B * p->desc.n_det);
  if (e == cudaSuccess) e = cudaMalloc(&b->partial, sizeof(double) * partial);
  if (e == cudaSuccess) e = cudaMalloc(&b->tan, sizeof(SampleBlock<Dual<4>>) * B);
  if (e != cudaSuccess) {
    set_error("pes_plan_create: cudaMalloc failed: %s", cudaGetErrorString(e));
    return PES_ENOMEM;
  }
  PES_CHECK_CUDA(cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking));
  PES_CHECK_CUDA(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming));
  PES_CHECK_CUDA(cudaEventCreateWithFlags(&b->join, cudaEventDisableTiming));
  PES_CHECK_CUDA(cudaFuncSetAttribute(k_dense64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)dense64_smem<true>()));
  k_grid64<<<ceil_div(n < kTrig ? kTrig : n, 128), 128>>>(p->dev, b->grid, b->trig);
  PES_CHECK_LAUNCH();
  PES_CHECK_CUDA(cudaStreamSynchronize(nullptr));
  return PES_OK;
}

void fp64_destroy(PesPlan* p) {
  Fp64Buffers* b = p->fp64;
  if (!b) return;
  if (b->side) {
    cudaStreamSynchronize(b->side);
    cudaStreamDestroy(b->side);
  }
  if (b->fork) cudaEventDestroy(b->fork);
  if (b->join) cudaEventDestroy(b->join);
  cudaFree(b->grid);
  cudaFree(b->trig);
  cudaFree(b->blocks);
  cudaFree(b->resp);
  cudaFree(b->partial);
  cudaFree(b->tan);
  delete b;
  p->fp64 = nullptr;
}

int fp64_lnl(PesPlan* p, const double* theta, int64_t B, double* lnl, double* grad, int32_t* status, cudaStream_t st) {
  Fp64Buffers* b = p->fp64;
  SampleBlock<double>* sb = reinterpret_cast<SampleBlock<double>*>(p->blocks);
  if (grad) {
    PES_CHECK_CUDA(cudaEventRecord(b->fork, st));
    PES_CHECK_CUDA(cudaStreamWaitEvent(b->side, b->fork, 0));
    ProfScope ps(p, kKSetup, b->side);
    k_tangents64<<<ceil_div(B, kPerSampleThreads), kPerSampleThreads, 0, b->side>>>(p->dev, theta, B, b->tan);
  }
  PES_CHECK_LAUNCH();
  if (grad) PES_CHECK_CUDA(cudaEventRecord(b->join, b->side));
  {
    ProfScope ps(p, kKSetup, st);
    k_setup64<<<(unsigned)B, 32 * (2 + p->desc.n_det), 0, st>>>(p->dev, theta, sb, b->blocks, b->resp);
  }
  PES_CHECK_LAUNCH();
  const int64_t n = p->desc.nbins;
  const int bpt = B * (int64_t)ceil_div(n, k64Threads) <= k64SmallBlocks ? 1 : k64BinsPerThread;
  const int nblk = (int)ceil_div(n, k64Threads * bpt);
  if (!grad) {
    {
      ProfScope ps(p, kKDenseFp64, st);
      k_dense64<false><<<dim3(nblk, (unsigned)B), k64Threads, 0, st>>>(p->dev, b->blocks, b->resp, b->grid, b->trig, nblk,
                                                                       bpt, b->partial);
    }
    PES_CHECK_LAUNCH();
    {
      ProfScope ps(p, kKFinalize, st);
      k_final64<false><<<ceil_div(B, 2), 64, 0, st>>>(p->dev, b->blocks, B, nblk, bpt, b->partial, nullptr, lnl, nullptr,
                                                     status);
    }
    PES_CHECK_LAUNCH();
    return PES_OK;
  }
  // in chunks of the samples whose partials the workspace holds
  const int64_t most = std::min<int64_t>(B, b->grad_rows / nblk);
  for (int64_t s0 = 0; s0 < B; s0 += most) {
    const int64_t Bc = std::min(most, B - s0);
    {
      ProfScope ps(p, kKDenseFp64, st);
      k_dense64<true><<<dim3(nblk, (unsigned)Bc), k64Threads, dense64_smem<true>(), st>>>(
          p->dev, b->blocks + s0, b->resp + s0 * p->desc.n_det, b->grid, b->trig, nblk, bpt, b->partial);
    }
    PES_CHECK_LAUNCH();
    if (s0 == 0) PES_CHECK_CUDA(cudaStreamWaitEvent(st, b->join, 0));
    {
      ProfScope ps(p, kKFinalize, st);
      k_final64<true><<<ceil_div(Bc, 2), 64, 0, st>>>(p->dev, b->blocks + s0, Bc, nblk, bpt, b->partial, b->tan + s0,
                                                     lnl + s0, grad + 11 * s0, status ? status + s0 : nullptr);
    }
    PES_CHECK_LAUNCH();
  }
  return PES_OK;
}

}  // namespace pes
