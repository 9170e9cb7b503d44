// Granular drop-in entry points: one per reference plugin method (orbit
// vectors, single-link response, TDI combination, Whittle likelihood) plus the
// IMRPhenomD / IMRPhenomHM waveform producers.  FP64 throughout, one thread per frequency.
#include <cmath>
#include <cstdarg>
#include <cstddef>
#include <cstdio>
#include <mutex>

#include "pes_abi_common.cuh"
#include "pes_freq.cuh"
#include "pes_physics.cuh"

namespace pes {

static thread_local char g_error[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

// ------------------------------------------------------------------ kernels
__global__ void k_orbit_vectors(PesOrbit o, const double* __restrict__ t, int64_t n, double* __restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double nn[3][3], xx[3][3];
  constellation<double>(o, t[i], nn, xx);
  double* o18 = out + 18 * i;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      o18[3 * a + j] = nn[a][j];
      o18[9 + 3 * a + j] = xx[a][j];
    }
}

// The response's trigonometric polynomials in the orbital angle, [1, c1, s1, c2,
// s2], of one source and detector (the value part of RespTab, from the orbit's
// closed form on the host): the arms of links 12 and 23 along the polarisation
// axes, the delays k.(x - x0) of nodes 1 and 2, and k.x0.
struct LinkArg {
  double np[2][5], nq[2][5], y[2][5], k0[2];
  double om[2], ph[2];  // revolution, rotation: rate and initial angle
  double arm_sec, tc;
  int32_t helio;
  int32_t finite;  // every number above is
};

static void link_arg(const PesOrbit& ob, double lam, double beta, double psi, double tc, LinkArg& o) {
  const double sl = std::sin(lam), cl = std::cos(lam), sb = std::sin(beta), cb = std::cos(beta);
  const double sp = std::sin(psi), cp = std::cos(psi);
  const double p[3] = {sl * cp - cl * sb * sp, -cl * cp - sl * sb * sp, cb * sp};
  const double q[3] = {-sl * sp - cl * sb * cp, cl * sp - sl * sb * cp, cb * cp};
  const double k[3] = {-(cb * cl), -(cb * sl), -sb};
  double x[3][3][5] = {};  // [node][axis][term]
  const double r = ob.r_sec;
  for (int n = 0; n < 3; ++n) {
    if (ob.kind == 0) {
      const double ck = ob.ck[n], sk = ob.sk[n];
      x[n][0][0] = -1.5 * r * ck;
      x[n][0][3] = 0.5 * r * ck;
      x[n][0][4] = 0.5 * r * sk;
      x[n][1][0] = -1.5 * r * sk;
      x[n][1][3] = -0.5 * r * sk;
      x[n][1][4] = 0.5 * r * ck;
      x[n][2][1] = -1.7320508075688772 * r * ck;
      x[n][2][2] = -1.7320508075688772 * r * sk;
    } else {
      // angle + 2 pi n / 3: cos = c1 a - s1 b, sin = s1 a + c1 b
      const double a = n == 0 ? 1.0 : -0.5, b = n == 0 ? 0.0 : (n == 1 ? 0.86602540378443865 : -0.86602540378443865);
      const double S[3] = {ob.sbeta_ref * ob.clam_ref, ob.sbeta_ref * ob.slam_ref, -ob.cbeta_ref};
      const double K[3] = {ob.slam_ref, -ob.clam_ref, 0.0};
      for (int j = 0; j < 3; ++j) {
        x[n][j][1] = r * (S[j] * b + K[j] * a);
        x[n][j][2] = r * (S[j] * a - K[j] * b);
      }
    }
  }
  const double iL = 1.0 / ob.arm_sec;
  for (int n = 0; n < 2; ++n)
    for (int t = 0; t < 5; ++t) {
      double np = 0.0, nq = 0.0, y = 0.0;
      for (int j = 0; j < 3; ++j) {
        const double a = (x[n + 1][j][t] - x[n][j][t]) * iL;
        np += a * p[j];
        nq += a * q[j];
        y += k[j] * x[n][j][t];
      }
      o.np[n][t] = np;
      o.nq[n][t] = nq;
      o.y[n][t] = y;
    }
  o.k0[0] = k[0] * kAUsec;
  o.k0[1] = k[1] * kAUsec;
  o.om[0] = ob.omega_revolution;
  o.om[1] = ob.omega_rotation;
  o.ph[0] = ob.revolution_initial;
  o.ph[1] = ob.rotation_initial;
  o.arm_sec = ob.arm_sec;
  o.tc = tc;
  o.helio = ob.kind == 0;
  o.finite = 1;
  const double* v = reinterpret_cast<const double*>(&o);
  for (size_t k = 0; k < offsetof(LinkArg, helio) / sizeof(double); ++k) o.finite &= std::isfinite(v[k]);
}

constexpr int kLinkThreads = 128;

// Six links of every bin, the modes summed.  FP64-bound: about 215 FP64
// instructions per mode (the plain formulae with the library's sines took 514).
__global__ void __launch_bounds__(kLinkThreads) k_response_links(const __grid_constant__ LinkArg a, const double* __restrict__ freqs,
                                                        int64_t n, int nmodes, const double2* __restrict__ hp,
                                                        const double2* __restrict__ hc, const double* __restrict__ tf,
                                                        double2* __restrict__ links) {
  __shared__ double2 tab[kTrig];
  fill_trig(tab);
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kLinkThreads + threadIdx.x;
  if (i < n) {
    const double f = freqs[i], pif = kPi * f, w2 = 2.0 * kPi * f, aL = pif * a.arm_sec;
    const int tier = sinc_tier(2.0 * fabs(aL));
    // 2 pi f t_c, rounded as the plain formula's argument is, whole turns removed
    const double ptc = turns64(w2 * a.tc);
    double ar[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, ai[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
    for (int m = 0; m < nmodes; ++m) {
      const double2 h1 = hp[m * n + i], h2 = hc[m * n + i];
      const double t = tf[m * n + i];
      const double T = t + a.tc;
      // above its cut a mode is zero, and so are its links (of finite angles and times)
      if (h1.x == 0.0 && h1.y == 0.0 && h2.x == 0.0 && h2.y == 0.0 && a.finite && isfinite(T) && isfinite(f)) continue;
      double ca, sa, c1, s1, c2 = 0.0, s2 = 0.0;
      sincos64(tab, fma(a.om[0], T, a.ph[0]), &sa, &ca);
      c1 = ca;
      s1 = sa;
      if (a.helio) {
        c2 = fma(c1, c1, -(s1 * s1));
        s2 = 2.0 * (s1 * c1);
      } else {
        sincos64(tab, fma(a.om[1], T, a.ph[1]), &s1, &c1);
      }
      auto poly = [&](const double* Y) {
        double v = fma(Y[1], c1, Y[2] * s1);
        if (a.helio) v += fma(Y[3], c2, fma(Y[4], s2, Y[0]));
        return v;
      };
      // -i a e^{-2 pi i f (t_c + k.x0)} times the polarisations
      double sn, cs;
      sincos64(tab, fma(w2, fma(a.k0[0], ca, a.k0[1] * sa), ptc), &sn, &cs);
      sn *= aL;
      cs *= aL;
      const double pr_ = fma(h1.y, cs, -(h1.x * sn)), pi_ = -fma(h1.x, cs, h1.y * sn);
      const double xr = 2.0 * fma(h2.y, cs, -(h2.x * sn)), xi = -2.0 * fma(h2.x, cs, h2.y * sn);
      double th[3], np[3], nq[3];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        th[k] = pif * poly(a.y[k]);
        np[k] = poly(a.np[k]);
        nq[k] = poly(a.nq[k]);
      }
      th[2] = -(th[0] + th[1]);
      np[2] = np[0] + np[1];  // (its sign drops out of the patterns)
      nq[2] = nq[0] + nq[1];
#pragma unroll
      for (int pr = 0; pr < 3; ++pr) {
        const int k2 = (pr + 1) % 3;
        const double Fp = fma(np[pr], np[pr], -(nq[pr] * nq[pr])), Fx = np[pr] * nq[pr];  // half of Fx
        const double gr = fma(Fp, pr_, Fx * xr), gi = fma(Fp, pi_, Fx * xi);
        double es, ec;
        sincos64(tab, aL - th[(pr + 2) % 3], &es, &ec);  // a + th[pr] + th[k2]
        const double br = fma(gr, ec, gi * es), bi = fma(gi, ec, -(gr * es));
        const double dl = th[k2] - th[pr];
        double sp, sm, d;
        sinc64<false>(tab, tier, aL + dl, &sp, &d);
        sinc64<false>(tab, tier, aL - dl, &sm, &d);
        ar[2 * pr] = fma(sp, br, ar[2 * pr]);
        ai[2 * pr] = fma(sp, bi, ai[2 * pr]);
        ar[2 * pr + 1] = fma(sm, br, ar[2 * pr + 1]);
        ai[2 * pr + 1] = fma(sm, bi, ai[2 * pr + 1]);
      }
    }
#pragma unroll
    for (int l = 0; l < 6; ++l) links[l * n + i] = make_double2(ar[l], ai[l]);
  }
}

// Michelson TDI of the six links.  FP64-bound: 80 FP64 instructions per bin (the plain
// formulae with the library's sine and cosine took 140, 27 us on 125 410 bins): the A/E/T
// norms join the generation prefactor, which is (1 - D^2) or (1 - D^2)(1 - D^4).
constexpr int kTdiThreads = 128;
__global__ void __launch_bounds__(kTdiThreads) k_tdi(const double* __restrict__ freqs, int64_t n, double arm, int gen20,
                                                     int orth, const double2* __restrict__ links,
                                                     double2* __restrict__ out) {
  __shared__ double2 tab[kTrig];
  fill_trig(tab);
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kTdiThreads + threadIdx.x;
  if (i >= n) return;
  double Dr, Di;
  sincos64(tab, -2.0 * kPi * freqs[i] * arm, &Di, &Dr);
  const double d2r = fma(Dr, Dr, -(Di * Di)), d2i = 2.0 * (Dr * Di);
  double pr = 1.0 - d2r, pi = -d2i;
  if (gen20) {
    const double qr = 1.0 - fma(d2r, d2r, -(d2i * d2i)), qi = -2.0 * (d2r * d2i);
    const double t = fma(pr, qr, -(pi * qi));
    pi = fma(pr, qi, pi * qr);
    pr = t;
  }
  double2 L[6];
#pragma unroll
  for (int l = 0; l < 6; ++l) L[l] = links[l * n + i];
  // L: 0=12 1=21 2=23 3=32 4=31 5=13; X = (l13 - l12) + D (l31 - l21) and cyclic
  double xr[3], xi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 a = L[(5 + 2 * k) % 6], b = L[2 * k], c = L[(4 + 2 * k) % 6], d = L[2 * k + 1];
    const double vr = c.x - d.x, vi = c.y - d.y;
    xr[k] = fma(Dr, vr, fma(-Di, vi, a.x - b.x));
    xi[k] = fma(Dr, vi, fma(Di, vr, a.y - b.y));
  }
  if (orth) {
    const double sr = xr[0] + xr[2], si = xi[0] + xi[2], ar = xr[2] - xr[0], ai = xi[2] - xi[0];
    const double yr = xr[1], yi = xi[1];
    xr[0] = ar;
    xi[0] = ai;
    xr[1] = fma(-2.0, yr, sr);
    xi[1] = fma(-2.0, yi, si);
    xr[2] = sr + yr;
    xi[2] = si + yi;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double w = c == 0 ? 0.70710678118654752 : (c == 1 ? 0.40824829046386302 : 0.57735026918962576);
    const double gr = orth ? pr * w : pr, gi = orth ? pi * w : pi;
    out[c * n + i] = make_double2(fma(gr, xr[c], -(gi * xi[c])), fma(gr, xi[c], gi * xr[c]));
  }
}

constexpr int kWhittleThreads = 256;
constexpr int kWhittleMaxBlocks = 1024;

__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    r = (l < (int)(blockDim.x >> 5)) ? sh[l] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  return r;  // valid in thread 0
}

// pass 1: each block sums a fixed, contiguous range of bins
__global__ void k_whittle_partial(const double2* __restrict__ d, const double2* __restrict__ h,
                                  const double* __restrict__ S, int nchan, int64_t n, int64_t per_block,
                                  double* __restrict__ partial) {
  __shared__ double sh[32];
  const int64_t lo = blockIdx.x * per_block;
  const int64_t hi = min(n, lo + per_block);
  double acc = 0.0;
  for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    double ip = 0.0;
    for (int c = 0; c < nchan; ++c) {
      double2 a = d[c * n + i], b = h[c * n + i];
      double rr = a.x - b.x, ri = a.y - b.y;
      ip += (rr * rr + ri * ri) / S[c * n + i];
    }
    acc += ip;
  }
  double r = block_sum(acc, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

// pass 2: one block sums the partials in a fixed order
__global__ void k_whittle_final(const double* __restrict__ partial, int nblk, double scale, double* __restrict__ out) {
  __shared__ double sh[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < nblk; i += blockDim.x) acc += partial[i];
  double r = block_sum(acc, sh);
  if (threadIdx.x == 0) out[0] = scale * r;
}

// Scratch of the allocation-free Whittle entry point: one partial sum per block
// of k_whittle_partial (at most kWhittleMaxBlocks).  8 KB that every device
// which loads this library keeps until the process exits.
constexpr int kNoAllocPartials = kWhittleMaxBlocks;
static __device__ __align__(256) double g_whittle_scratch[kNoAllocPartials];

// Device address of g_whittle_scratch for each device, looked up on the first
// call made with that device current.
constexpr int kMaxDevices = 64;
static std::mutex g_scratch_mu;
static double* g_scratch_ptr[kMaxDevices] = {};

static int whittle_scratch(double** out) {
  int dev = -1;
  PES_CHECK_CUDA(cudaGetDevice(&dev));
  PES_REQUIRE(dev >= 0 && dev < kMaxDevices, "pes_whittle_lnl_noalloc: device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (g_scratch_ptr[dev] == nullptr) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_whittle_scratch);
    if (e != cudaSuccess) {
      set_error("pes_whittle_lnl_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                cudaGetErrorString(e));
      return PES_ECUDA;
    }
    g_scratch_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_scratch_ptr[dev];
  return PES_OK;
}

// IMRPhenomD / IMRPhenomHM modes on an array of frequencies.  The parameters are
// the host's, so the host sets the sample up (a few microseconds; a set-up by
// one warp of every block was a serial FP64 chain of 45 us and half of the work
// of six modes on 150 000 bins) and passes each mode's coefficients, rescaled
// to frequencies in Hz, as kernel arguments.  A thread takes one bin of every
// mode: the powers and the logarithm of f are shared by the modes, and in the
// inspiral a mode is two polynomials, a sine and a cosine.  Bound by the FP64
// pipe: about 90 FP64 instructions per mode and 90 per bin; six modes go to two
// threads, since the bins below the cut alone leave some SM partitions a warp
// more than others.  (bilby's call on one detector, 125 410 bins: 519 -> 212 us
// with the response below; six modes on three detectors, 149 850 bins: 4.70 -> 1.32 ms.)
struct WaveMode {
  // phase: inspiral f^{-5/3} sum pin_j f^{j/3} + (lg0 + lg1 f^{1/3}) ln(f)/3 below fj1;
  // it0 + it1 f + it2 x^{-3} + it3 ln x, x = ap f + bp, to fj2;
  // mr0 + mr1 f + mr2 / f + mr3 f^{3/4} + mr4 atan((f - f5) / fd) above
  double pin[12], rin[12], lg0, lg1;  // rin_j = (j - 5) pin_j / (6 pi)
  double it0, it1, it2, it3, ap, bp;
  double mr0, mr1, mr2, mr3, mr4, f5, fd, ifd;
  double fj1, fj2;
  // amplitude: a0 f^{-7/6} (1 + sum ai_j f^{(j+2)/3}) below fa; a1 y^{-7/6} Ahat(y)
  // at the mapped frequency y = sum y_j (f - fa)^j to fb; a2 f^{-7/6} Ahat(R f) above
  double a0, a1, a2, ai[8], dl[5], y1, y2, y3, fa, fb, fpk, R;
  double gm, w2, fr, gx, ymax;
  // post-Newtonian ratio (b1 v + b2 v^2 + b3 v^3) / (1 + h2 v^2 + 2 pi v^3), v = cv f^{1/3}
  // below fa, va (2 - exp(1 - f / fa))^{1/3} above
  double b1, b2, b3, h2, cv, va, ifa;
  double P, C;                        // hp = P h, hc = i C h
};
constexpr int kWaveThreads = 128;
template <int kModes>
struct WaveArg {
  WaveMode md[kModes];
};

static void wave_mode(const PhenomDCoef<double>& c, const HMMode<double>& md, const PhenomHMCoef<double>* h, int k,
                      WaveMode& o) {
  const double M = c.Msec, iM = 1.0 / M;
  const double m = (double)kHMlmHost[k][1], hm = 0.5 * m, qt = md.qt;
  // inspiral at 2 f / m: powers of tm M (the leading phase terms reach 1e5 rad: their
  // coefficients are rounded once)
  const DD tm = dd_div({2.0, 0.0}, {m, 0.0}), Mt = dd_mul(tm, {M, 0.0}), cu = dd_cbrt(Mt), one = {1.0, 0.0};
  const DD icu = dd_div(one, cu), icu2 = dd_mul(icu, icu);
  DD pw = dd_mul(dd_mul(icu2, icu2), icu);
  for (int j = 0; j < 12; ++j) {
    o.pin[j] = dd_mul(pw, {hm * c.pin[j], 0.0}).h;
    pw = dd_mul(pw, cu);
  }
  const double lcu = std::log(cu.h);
  o.lg0 = hm * c.lg0;
  o.lg1 = hm * c.lg1 * cu.h;
  o.pin[5] += o.lg0 * lcu + qt;
  o.pin[6] += o.lg1 * lcu;
  for (int j = 0; j < 12; ++j) o.rin[j] = o.pin[j] * ((j - 5) / (6.0 * kPi));
  // intermediate: 22 phase at x = ap f + bp
  const double ia = 1.0 / md.aP;
  o.ap = md.aP;
  o.bp = md.bP * iM;
  o.it0 = (c.pint[0] + c.pint[3] * std::log(M) + c.pint[1] * md.bP) * ia + md.cI0 + qt;
  o.it1 = (c.pint[1] + md.cI1) * M;
  o.it2 = c.pint[2] * (iM * iM * iM) * ia;
  o.it3 = c.pint[3] * ia;
  // merger-ringdown: at Rholm f
  const double R = md.Rholm, iR = 1.0 / R, RM = R * M, q = std::sqrt(std::sqrt(RM));
  o.mr0 = c.pm[0] * iR + md.cR0 + qt;
  o.mr1 = (c.pm[1] + md.cR1) * M;
  o.mr2 = c.pm[2] * iR / RM;
  o.mr3 = c.pm[3] * (q * q * q) * iR;
  o.mr4 = c.pm[4] * iR;
  o.f5 = c.pm[5] / RM;
  o.fd = md.fDMeff / RM;
  o.ifd = RM / md.fDMeff;
  o.fj1 = md.fiP * iM;
  o.fj2 = md.frP * iM;
  // amplitude
  auto p76 = [](double x) { return 1.0 / (x * std::sqrt(std::cbrt(x))); };
  o.a0 = c.amp_scale * p76(Mt.h);
  o.a1 = c.amp_scale * p76(M);
  o.a2 = c.amp_scale * p76(RM);
  double s = cu.h * cu.h;
  for (int j = 0; j < 8; ++j) {
    o.ai[j] = c.ai[j] * s;
    s *= cu.h;
  }
  s = 1.0;
  for (int j = 0; j < 5; ++j) {
    o.dl[j] = md.dl[j] * s;
    s *= M;
  }
  o.fa = md.fiA * iM;
  o.fb = md.frA * iM;
  o.ifa = M / md.fiA;
  o.R = R;
  {
    const double t = 2.0 / m, H = o.fb - o.fa, A = t * o.fa, B = R * o.fb;
    // the cubic Hermite blend in powers of f - fa
    o.y1 = t;
    o.y2 = k == 0 ? 0.0 : (3.0 * (B - A) - H * (2.0 * t + R)) / (H * H);
    o.y3 = k == 0 ? 0.0 : (2.0 * (A - B) + H * (t + R)) / (H * H * H);
  }
  o.fpk = md.fpeak * iM;
  const double w = md.g3fDMeff * iM;
  o.gm = c.g1 * w * iM;
  o.w2 = w * w;
  o.fr = c.fRD * iM;
  o.gx = c.g2 / w;
  o.ymax = kMfCut * iM;
  o.b1 = o.b2 = o.b3 = o.h2 = o.cv = o.va = 0.0;
  if (k > 0) {
    const double r2 = std::sqrt(2.0), r23 = std::sqrt(2.0 / 3.0), r57 = 0.84515425472851657;
    const double a2 = 0.75 * 1.0350983390135313 * h->dlt * r23;
    if (k == 1) {
      o.b1 = r2 / 3.0 * h->dlt;
      o.b2 = -r2 / 2.0 * (h->chia + h->dlt * h->chis);
      o.b3 = o.b1 * (-17.0 / 28.0 + (5.0 / 7.0) * h->eta);
    } else if (k == 2) {
      o.b1 = a2;
      o.b3 = a2 * (-4.0 + 2.0 * h->eta);
    } else if (k == 3) {
      o.b2 = r57 / 3.0 * (1.0 - 3.0 * h->eta);
    } else if (k == 4) {
      o.b2 = 8.0 / 9.0 * r57 / r2 * (1.0 - 3.0 * h->eta);
    } else {
      o.b3 = 9.0 / (4.0 * 8.3666002653407556) * r23 * h->dlt * (1.0 - 2.0 * h->eta);
    }
    o.h2 = -107.0 / 42.0 + (55.0 / 42.0) * h->eta;
    o.cv = std::cbrt(md.tpm * M);
    o.va = std::cbrt(md.tpm * md.fiA);
  }
  o.P = md.P;
  o.C = md.C;
}

// y^{-7/6} and y^{1/3}
__device__ __forceinline__ double pow76(double y, double* u) {
  *u = cbrt(y);
  return rcp64(y) * rsqrt(*u);
}
__device__ __forceinline__ double wave_mrd(const WaveMode& c, double y) {
  const double x = y - c.fr;
  return c.gm * rcp64(fma(x, x, c.w2)) * exp(-(c.gx * x));
}

template <int kModes>
__global__ void __launch_bounds__(kWaveThreads) k_wave(const __grid_constant__ WaveArg<kModes> arg, double f_cut,
                                              const double* __restrict__ freqs, int64_t n, double2* __restrict__ hp,
                                              double2* __restrict__ hc, double* __restrict__ tf) {
  __shared__ double2 tab[kTrig];
  fill_trig(tab);
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kWaveThreads + threadIdx.x;
  if (i < n) {
    const double f = freqs[i];
    const bool in = !(f > f_cut);
    double u = 0.0, jf = 0.0, lf3 = 0.0, iu5 = 0.0, iu5l = 0.0, p76 = 0.0;
    if (in) {
      u = cbrt(f);
      jf = rcp64(f);
      lf3 = log(f) * (1.0 / 3.0);
      p76 = jf * rsqrt(u);
      // u^{-5} = u / f^2 as a pair: the phase's leading terms multiply its error by 1e5
      const double q = jf * jf, eq = fma(jf, jf, -q), ej = fma(-f, jf, 1.0);
      const double u2 = u * u, e2 = fma(u, u, -u2), u3 = u2 * u, e3 = fma(u2, u, -u3);
      const double du = ((f - u3) - fma(e2, u, e3)) * jf * (1.0 / 3.0);  // relative error of u
      iu5 = q * u;
      iu5l = fma(eq, u, fma(q, u, -iu5)) + iu5 * fma(2.0, ej, du);
    }
#pragma unroll 1
    for (int k = blockIdx.y; k < kModes; k += gridDim.y) {
      const WaveMode& c = arg.md[k];
      const int64_t o = (int64_t)k * n + i;
      // ---- amplitude (NaN frequencies stay: they are not above the cut)
      double A, y = 0.0, v = c.cv * u;
      if (in) {
        if (f < c.fa || (k > 0 && f == c.fa)) {
          double p = c.ai[7];
#pragma unroll
          for (int j = 6; j >= 0; --j) p = fma(p, u, c.ai[j]);
          A = c.a0 * p76 * fma(u * u, p, 1.0);
        } else {
          if (f < c.fb || k == 0) {
            const double x = f - c.fa;
            double uy = u, py = p76;
            y = f;
            if (k > 0) {
              y = fma(x, fma(x, fma(x, c.y3, c.y2), c.y1), c.y1 * c.fa);
              py = pow76(y, &uy);
            }
            const double ah = y >= c.fpk ? wave_mrd(c, y)
                                         : fma(y, fma(y, fma(y, fma(y, c.dl[4], c.dl[3]), c.dl[2]), c.dl[1]), c.dl[0]);
            A = c.a1 * py * ah;
          } else {
            y = c.R * f;
            A = c.a2 * p76 * wave_mrd(c, y);
          }
          if (k > 0) v = c.va * cbrt(2.0 - exp(1.0 - f * c.ifa));
        }
        if (k > 0) {
          const double v2 = v * v;
          A *= v * fma(v, fma(v, c.b3, c.b2), c.b1) * rcp64(fma(v2, fma(2.0 * kPi, v, c.h2), 1.0));
        }
      }
      if (!in || y > c.ymax) {
        hp[o] = make_double2(0.0, 0.0);
        hc[o] = make_double2(0.0, 0.0);
        tf[o] = 0.0;
        continue;
      }
      // ---- phase and t(f)
      double psi, t;
      if (f < c.fj1) {
        double p = c.pin[11], r = c.rin[11];
#pragma unroll
        for (int j = 10; j >= 0; --j) {
          p = fma(p, u, c.pin[j]);
          if (j != 5) r = fma(r, u, c.rin[j]); else r *= u;
        }
        const double l1 = c.lg1 * u;
        psi = fma(p, iu5, fma(p, iu5l, (c.lg0 + l1) * lf3));
        t = jf * fma(r, iu5, fma(l1, lf3 + 1.0, c.lg0) * (1.0 / (6.0 * kPi)));
      } else if (f < c.fj2) {
        double jx = jf, l = 3.0 * lf3;
        if (k > 0) {
          const double x = fma(c.ap, f, c.bp);
          jx = rcp64(x);
          l = log(x);
        }
        const double j3 = jx * jx * jx;
        psi = fma(c.it1, f, fma(c.it2, j3, fma(c.it3, l, c.it0)));
        t = fma(c.ap * jx, fma(-3.0 * c.it2, j3, c.it3), c.it1) * (1.0 / (2.0 * kPi));
      } else {
        const double q = rsqrt(sqrt(f)), x = f - c.f5, rd = rcp64(fma(x, x, c.fd * c.fd));
        psi = fma(c.mr1, f, fma(c.mr2, jf, fma(c.mr3, f * q, fma(c.mr4, atan64(tab, x * c.ifd), c.mr0))));
        t = fma(-c.mr2 * jf, jf, fma(0.75 * c.mr3, q, fma(c.mr4 * c.fd, rd, c.mr1))) * (1.0 / (2.0 * kPi));
      }
      double sn, cs;
      sincos64(tab, psi, &sn, &cs);
      // h = A e^{-i Psi}; hp = P h, hc = i C h
      const double ap = c.P * A, ac = c.C * A;
      hp[o] = make_double2(ap * cs, -(ap * sn));
      hc[o] = make_double2(ac * sn, ac * cs);
      tf[o] = t;
    }
  }
}

// The sample's coefficients on the host and the launch.
template <int kModes>
static int launch_wave(const double* theta, const double* freqs, int64_t n, double f_ref, double f_cut, double* hp,
                       double* hc, double* tf, cudaStream_t st) {
  PhenomDCoef<double> c;
  double rows[kFCount][3];
  phenomd_setup<double, 3>(theta, f_ref, rows, 0, 1, 0u, c);
  PhenomHMCoef<double> h;
  phenomhm_common<double>(theta, c, h);
  WaveArg<kModes> arg;
  for (int k = 0; k < kModes; ++k) {
    phenomhm_mode<double, 3>(theta, c, k, h.md[k]);
    wave_mode(c, h.md[k], &h, k, arg.md[k]);
  }
  if (kModes == 1) {  // IMRPhenomD's own polarisation factors
    arg.md[0].P = c.pfac;
    arg.md[0].C = -c.cfac;
  }
  k_wave<kModes><<<dim3(ceil_div(n, kWaveThreads), kModes > 1 ? 2 : 1), kWaveThreads, 0, st>>>(
      arg, f_cut, freqs, n, reinterpret_cast<double2*>(hp), reinterpret_cast<double2*>(hc), tf);
  PES_CHECK_LAUNCH();
  return PES_OK;
}

}  // namespace pes

using namespace pes;

// ------------------------------------------------------------------ C ABI
// ------------------------------------------------------------------ PN t(f)
// Post-Newtonian time-frequency map of the reference's lalsimulation interface
// (pespace/waveform/interface_lalsim.py:297-482): aligned-spin TaylorF2 phase
// Psi(x) = sum_k (a_k + b_k ln(pi x)) x^((k-5)/3), x = M f, and
// t(f) = -M/(2 pi) (Psi'(x) - Psi'(x_ISCO)) below x_ISCO = 6^-3/2 / pi, 0 above.
// The coefficient table is the published expansion the reference uses (its
// 4PN spin-orbit term carries pi^2, interface_lalsim.py:435-444).
constexpr double kPnXIsco = 0.021658244478713225;  // M f at the ISCO, 1 / (6^(3/2) pi)

struct PnCoef {
  double a[9];      // a_0..a_8 (a_5 = 0)
  double b5, b6, b8;
  double msec;      // total mass [s]
  double d_isco;    // Psi'(x_ISCO)
};

__device__ double pn_dpsi(const PnCoef& c, double x) {
  // Psi'(x) = sum_k (k-5)/3 a_k x^((k-8)/3) + b5/x + b6 x^(-2/3) (ln(pi x)/3 + 1) + b8 (ln(pi x) + 1):
  // Horner in w = x^(-1/3) for the power terms (exponents -8/3 .. 0)
  const double w = 1.0 / cbrt(x);
  double p = (-5.0 / 3.0) * c.a[0];
  p = p * w + (-4.0 / 3.0) * c.a[1];
  p = p * w + (-1.0) * c.a[2];
  p = p * w + (-2.0 / 3.0) * c.a[3];
  p = p * w + (-1.0 / 3.0) * c.a[4];
  p = p * w;                              // k = 5: no power term
  p = p * w + (1.0 / 3.0) * c.a[6];
  p = p * w + (2.0 / 3.0) * c.a[7];
  p = p * w + c.a[8];
  const double lp = log(kPi * x);
  const double w2 = w * w;
  return p + c.b5 * w2 * w + c.b6 * w2 * (lp * (1.0 / 3.0) + 1.0) + c.b8 * (lp + 1.0);
}

__device__ void pn_coefficients(double m1, double m2, double chi1, double chi2, PnCoef& c) {
  const double mt = m1 + m2;
  const double eta = m1 * m2 / (mt * mt), e2 = eta * eta, e3 = e2 * eta;
  const double dl = sqrt(fmax(0.0, 1.0 - 4.0 * eta));
  const double xa = 0.5 * (chi1 - chi2), xs = 0.5 * (chi1 + chi2);
  const double pi = kPi, pi2 = kPi * kPi, pi13 = cbrt(kPi), pi23 = pi13 * pi13;
  const double pfac = -3.0 / (128.0 * eta);
  const double c2 = 3715.0 / 756.0 + 55.0 / 9.0 * eta;
  const double c3 = -16.0 * pi + 113.0 / 3.0 * dl * xa + (113.0 / 3.0 - 76.0 / 3.0 * eta) * xs;
  const double c4 = 15293365.0 / 508032.0 + 27145.0 / 504.0 * eta + 3085.0 / 72.0 * e2 +
                    (-405.0 / 8.0 + 200.0 * eta) * xa * xa - 405.0 / 4.0 * dl * xa * xs +
                    (-405.0 / 8.0 + 5.0 / 2.0 * eta) * xs * xs;
  const double c5l = (38645.0 / 756.0 - 65.0 / 9.0 * eta) * pi + (-732985.0 / 2268.0 - 140.0 / 9.0 * eta) * dl * xa +
                     (-732985.0 / 2268.0 + 24260.0 / 81.0 * eta + 340.0 / 9.0 * e2) * xs;
  const double c6 = 11583231236531.0 / 4694215680.0 - 640.0 / 3.0 * pi2 - 6848.0 / 21.0 * kEulerGamma +
                    (-15737765635.0 / 3048192.0 + 2255.0 / 12.0 * pi2) * eta + 76055.0 / 1728.0 * e2 -
                    127825.0 / 1296.0 * e3 - 0.69314718055994531 * 13696.0 / 21.0 + 2270.0 / 3.0 * pi * dl * xa +
                    (2270.0 / 3.0 - 520.0 * eta) * pi * xs + (75515.0 / 144.0 - 8225.0 / 18.0 * eta) * dl * xs * xa +
                    (75515.0 / 288.0 - 263245.0 / 252.0 * eta - 480.0 * e2) * xa * xa +
                    (75515.0 / 288.0 - 232415.0 / 504.0 * eta + 1255.0 / 9.0 * e2) * xs * xs;
  const double c7 =
      (77096675.0 / 254016.0 + 378515.0 / 1512.0 * eta - 74045.0 / 756.0 * e2) * pi +
      (-25150083775.0 / 3048192.0 + 26804935.0 / 6048.0 * eta - 1985.0 / 48.0 * e2) * dl * xa +
      (-25150083775.0 / 3048192.0 + 10566655595.0 / 762048.0 * eta - 1042165.0 / 3024.0 * e2 + 5345.0 / 36.0 * e3) * xs -
      1140.0 * pi * dl * xa * xs + (-570.0 + 2240.0 * eta) * pi * xa * xa + (-570.0 + 40.0 * eta) * pi * xs * xs +
      (14585.0 / 8.0 - 215.0 / 2.0 * eta) * dl * xa * xs * xs + (14585.0 / 8.0 - 7270.0 * eta + 80.0 * e2) * xa * xa * xs +
      (14585.0 / 24.0 - 2380.0 * eta) * dl * xa * xa * xa +
      (14585.0 / 24.0 - 475.0 / 6.0 * eta + 100.0 / 3.0 * e2) * xs * xs * xs;
  const double c8 = (233915.0 / 168.0 - 99185.0 / 252.0 * eta) * dl * xa +
                    (233915.0 / 168.0 - 3970375.0 / 2268.0 * eta + 19655.0 / 189.0 * e2) * xs;
  c.a[0] = pfac / (pi * pi23);
  c.a[1] = 0.0;
  c.a[2] = pfac * c2 / pi;
  c.a[3] = pfac * c3 / pi23;
  c.a[4] = pfac * c4 / pi13;
  c.a[5] = 0.0;
  c.a[6] = pfac * c6 * pi13;
  c.a[7] = pfac * c7 * pi23;
  c.a[8] = pfac * c8 * pi2;
  c.b5 = pfac * c5l;
  c.b6 = pfac * (-6848.0 / 63.0) * pi13;
  c.b8 = -c.a[8];
  c.msec = mt * kMTSun;
  c.d_isco = pn_dpsi(c, kPnXIsco);
}

// grid (ceil(n / 256), B): thread 0 of each block sets up the sample's coefficients
__global__ void k_pn_tf(const double* __restrict__ params, int64_t n, const double* __restrict__ freqs,
                        double* __restrict__ tf) {
  __shared__ PnCoef c;
  const int64_t b = blockIdx.y;
  if (threadIdx.x == 0) {
    const double* q = params + 4 * b;
    pn_coefficients(q[0], q[1], q[2], q[3], c);
  }
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = freqs[i] * c.msec;
  tf[b * n + i] = (x < kPnXIsco && x > 0.0) ? -c.msec / (2.0 * kPi) * (pn_dpsi(c, x) - c.d_isco) : 0.0;
}

// ------------------------------------------------ time-domain Michelson TDI
// TDMichelsonConstantEqualArm.update_tdi_response (pespace/detector/tdi.py:
// 1460-1600): every output sample i combines the six single-link series at
// the undelayed sample i + added and, for each delay k = 0..max_delay-1, the
// linear interpolation left + (right - left) * frac_k between samples
// i + shift_k and i + shift_k + 1 (utils.py:83-100).  The shifts, fractions and
// `added` are the reference's expressions on Python floats (tdi.py:1449-1454,
// 1469-1491), evaluated on the host by td_layout.  The arithmetic keeps the
// reference's order with no contraction (explicit round-to-nearest adds and
// multiplies), so the result is bit-identical to a left-to-right evaluation.
//
// Each block stages the window [i0, i0 + kTdTile + added + 1) of its six link
// series in shared memory with coalesced loads, and beside it the differences
// right - left of neighbouring samples: every delay that reads a sample pair
// reuses its difference (the same subtraction of the same operands), which
// takes 6 instead of 6 max_delay FP64 subtractions per output sample.  Per
// output sample the unique traffic is 6 x 8 B read and 3 x 8 B written, but
// the reference's operation order leaves about 145 unfused FP64 operations,
// so the FP64 pipe (1/64 of the FP32 rate) binds, not HBM.  A window beyond
// kTdMaxWindow samples (added > 1535, e.g. sub-0.04 s sampling) reads
// through the L1 and subtracts per delay instead.

struct TdLayout {
  int max_delay;
  int64_t added;
  int64_t shift[7];
  double frac[7];
  double rs2, rs6, rs3;  // sqrt(2), sqrt(6), sqrt(3), correctly rounded
};

constexpr int kTdThreads = 256;
constexpr int kTdTile = 512;
constexpr int kTdMaxWindow = 2048;  // values and differences: 12 x 2048 x 8 B = 192 KB of shared memory

// Python's float // and % (CPython's divmod: floor of (a - fmod(a, b)) / b,
// rounded to the nearest integer when it lands within half of one).
static void py_divmod(double a, double b, double* floordiv, double* mod) {
  double m = std::fmod(a, b);
  double div = (a - m) / b;
  if (m != 0.0) {
    if ((b < 0) != (m < 0)) {
      m += b;
      div -= 1.0;
    }
  } else {
    m = std::copysign(0.0, b);
  }
  double fd;
  if (div != 0.0) {
    fd = std::floor(div);
    if (div - fd > 0.5) fd += 1.0;
  } else {
    fd = std::copysign(0.0, a / b);
  }
  *floordiv = fd;
  *mod = m;
}

static void td_layout(double arm, double dt, int gen20, TdLayout& lay) {
  lay.max_delay = gen20 ? 7 : 3;
  double q, r;
  py_divmod(lay.max_delay * arm, dt, &q, &r);
  lay.added = (int64_t)(q + 1.0);  // int(max_num_delay * armlength // delta_time + 1)
  for (int k = 0; k < 7; ++k) {
    lay.shift[k] = 0;
    lay.frac[k] = 0.0;
  }
  for (int k = 0; k < lay.max_delay; ++k) {
    const int nd = k + 1;
    py_divmod(nd * arm, dt, &q, &r);
    lay.frac[k] = 1.0 - r / dt;  // 1 - (num_delay * armlength % delta_time) / delta_time
    py_divmod((lay.max_delay - nd) * arm, dt, &q, &r);
    lay.shift[k] = (int64_t)q;  // (max_num_delay - num_delay) * armlength // delta_time
  }
  lay.rs2 = std::sqrt(2.0);
  lay.rs6 = std::sqrt(6.0);
  lay.rs3 = std::sqrt(3.0);
}

// grid (ceil(n / kTdTile), B); links [B][6][n_ext] in the order link12, link21,
// link23, link32, link31, link13; out [B][3][n].
template <int kMaxDelay, bool kStaged>
__global__ void __launch_bounds__(kTdThreads) k_td_tdi(TdLayout lay, const double* __restrict__ links, int64_t n_ext,
                                                       int64_t n, int orth, double* __restrict__ out) {
  extern __shared__ double td_win[];  // [6][win] values, then [6][win] differences
  const double* src = links + (int64_t)blockIdx.y * 6 * n_ext;
  double* dst = out + (int64_t)blockIdx.y * 3 * n;
  const int64_t i0 = (int64_t)blockIdx.x * kTdTile;
  const int64_t win = kTdTile + lay.added + 1;
  double* td_dif = td_win + 6 * win;
  if (kStaged) {
    const int64_t avail = n_ext - i0;
#pragma unroll 1
    for (int l = 0; l < 6; ++l) {
      const double* s = src + (int64_t)l * n_ext + i0;
      double* w = td_win + l * win;
#pragma unroll 4
      for (int64_t j = threadIdx.x; j < win; j += kTdThreads) w[j] = j < avail ? __ldg(s + j) : 0.0;
    }
    __syncthreads();
#pragma unroll 1
    for (int l = 0; l < 6; ++l) {
      const double* w = td_win + l * win;
      double* df = td_dif + l * win;
#pragma unroll 4
      for (int64_t j = threadIdx.x; j + 1 < win; j += kTdThreads) df[j] = __dsub_rn(w[j + 1], w[j]);
    }
    __syncthreads();
  }
  // X = sum of the "plus" terms, then minus the "minus" terms, in the order of
  // tdi.py:1506-1591 (k = -1: the undelayed sample); Y and Z are the cyclic
  // relabelling 1 -> 2 -> 3 -> 1, i.e. link index l -> (l + 2) mod 6.
  constexpr int kTerms = kMaxDelay + 1;
  constexpr int xp[8] = {5, 4, 0, 1, 0, 1, 5, 4};
  constexpr int xm[8] = {0, 1, 5, 4, 5, 4, 0, 1};
#pragma unroll 1
  for (int r = 0; r < kTdTile / kTdThreads; ++r) {
    const int64_t t = threadIdx.x + r * kTdThreads;
    const int64_t i = i0 + t;
    if (i >= n) break;
    auto at = [&](int l, int64_t off) -> double {
      return kStaged ? td_win[l * win + t + off] : __ldg(src + (int64_t)l * n_ext + i + off);
    };
    auto term = [&](int l, int k) -> double {
      if (k < 0) return at(l, lay.added);
      const double left = at(l, lay.shift[k]);
      const double dif = kStaged ? td_dif[l * win + t + lay.shift[k]] : __dsub_rn(at(l, lay.shift[k] + 1), left);
      return __dadd_rn(left, __dmul_rn(dif, lay.frac[k]));
    };
    double ch[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double acc = term((xp[0] + 2 * c) % 6, -1);
#pragma unroll
      for (int j = 1; j < kTerms; ++j) acc = __dadd_rn(acc, term((xp[j] + 2 * c) % 6, j - 1));
#pragma unroll
      for (int j = 0; j < kTerms; ++j) acc = __dsub_rn(acc, term((xm[j] + 2 * c) % 6, j - 1));
      ch[c] = acc;
    }
    if (orth) {
      const double X = ch[0], Y = ch[1], Z = ch[2];
      dst[i] = __ddiv_rn(__dsub_rn(Z, X), lay.rs2);
      dst[n + i] = __ddiv_rn(__dadd_rn(__dsub_rn(X, __dmul_rn(2.0, Y)), Z), lay.rs6);
      dst[2 * n + i] = __ddiv_rn(__dadd_rn(__dadd_rn(X, Y), Z), lay.rs3);
    } else {
      dst[i] = ch[0];
      dst[n + i] = ch[1];
      dst[2 * n + i] = ch[2];
    }
  }
}

template <int kMaxDelay>
static int launch_td_tdi(const TdLayout& lay, const double* links, int64_t B, int64_t n_ext, int64_t n, int orth,
                         double* out, cudaStream_t st) {
  const dim3 grid((unsigned)((n + kTdTile - 1) / kTdTile), (unsigned)B);
  const int64_t win = kTdTile + lay.added + 1;
  if (win <= kTdMaxWindow) {
    const size_t smem = (size_t)12 * win * sizeof(double);
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k_td_tdi<kMaxDelay, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem);
      if (e != cudaSuccess) {
        set_error("pes_td_tdi_combination: %s", cudaGetErrorString(e));
        return PES_ECUDA;
      }
    }
    k_td_tdi<kMaxDelay, true><<<grid, kTdThreads, smem, st>>>(lay, links, n_ext, n, orth, out);
  } else {
    k_td_tdi<kMaxDelay, false><<<grid, kTdThreads, 0, st>>>(lay, links, n_ext, n, orth, out);
  }
  PES_CHECK_LAUNCH();
  return PES_OK;
}

// Float-float variant (pes_td_tdi_combination_mixed): the same combination on
// the FP32 pipe.  Each block scales its window by a power of two (its largest
// exponent to 2^0, exact) and splits every double into a float-float pair from
// the bits alone (integer operations: the FP64 pipe is not used on the way
// in).  Every delay that a channel applies to one link it applies with the
// opposite sign to another, to links 13 and 12 (difference P) or 31 and 21 (Q)
// for X and cyclically for Y and Z:
//   X = P + D1 Q - D2 P - D3 Q  [- D4 P - D5 Q + D6 P + D7 Q, TDI 2.0],
// so a block forms the six differences (and those of neighbouring samples)
// once per window sample and a channel interpolates 3 or 7 terms instead of 6
// or 14.  Each channel goes back to a double from the
// bits and one FP64 add.  Scaled magnitudes below 2^-126 (2^-126 of the
// window's largest link sample), and the tails of those below 2^-103, flush to
// zero; a NaN or an infinity among the inputs gives NaN in the outputs that
// read it.
//
// Issue slots bind (84% of cycles; FMA pipe 47%, ALU 52%): about 430 operations of the
// sums, 200 of the window and 60 of the way out per sample.  8 388 609 samples, TDI 2.0, A/E/T: 682 us with
// 14 interpolated terms per channel and loads link by link, 476 us with the
// differences, 338 us with all of a block's loads in flight (1.8 TB/s).
struct TdLayoutFF {
  int max_delay;
  int64_t added;
  int64_t shift[7];
  float2 frac[7];      // the weights as float-float pairs
  float2 rs2, rs6, rs3;  // 1/sqrt(2), 1/sqrt(6), 1/sqrt(3) as float-float pairs
};

static float2 ff_pair(double x) {
  const float h = (float)x;
  return make_float2(h, (float)(x - (double)h));
}

static void td_layout_ff(const TdLayout& lay, TdLayoutFF& out) {
  out.max_delay = lay.max_delay;
  out.added = lay.added;
  for (int k = 0; k < 7; ++k) {
    out.shift[k] = lay.shift[k];
    out.frac[k] = ff_pair(lay.frac[k]);
  }
  out.rs2 = ff_pair(1.0 / std::sqrt(2.0));
  out.rs6 = ff_pair(1.0 / std::sqrt(6.0));
  out.rs3 = ff_pair(1.0 / std::sqrt(3.0));
}

// The scaling of a block's window, x -> x * 2^-scale: limits on the high word
// of |x| and the exponent's shift.
struct TdScale {
  unsigned rebias;        // (896 + scale) << 23
  unsigned head0, tail0;  // high words from which x * 2^-scale is at least 2^-126 (and x normal), 2^-103
};
__device__ __forceinline__ TdScale td_scale(int scale) {
  TdScale s;
  s.rebias = (unsigned)(896 + scale) << 23;
  s.head0 = (unsigned)max(1, 1023 - 126 + scale) << 20;
  s.tail0 = (unsigned)max(1, 1023 - 103 + scale) << 20;
  return s;
}

// x * 2^-scale as a float-float pair: head = sign, exponent and the top 23
// fraction bits (the exponent's low 9 bits, shifted modulo 2^32); tail = the
// other 29 fraction bits over 2^29, rounded to 24 significant bits, times the
// head's power of two over 2^23.
__device__ __forceinline__ FF td_split(double x, const TdScale& s) {
  const unsigned H = (unsigned)__double2hiint(x), L = (unsigned)__double2loint(x);
  const unsigned a = H & 0x7fffffffu, sign = H & 0x80000000u;
  unsigned hb = (__funnelshift_l(L, H, 3) - s.rebias) | sign;
  const float pw = __uint_as_float((hb & 0xff800000u) - (23u << 23));  // +-2^(e - 23)
  float lo = (__uint2float_rn(L & 0x1fffffffu) * 1.862645149230957e-09f) * pw;
  lo = a < s.tail0 ? 0.0f : lo;
  hb = a < s.head0 ? 0u : hb;
  hb = a >= 0x7ff00000u ? 0x7fc00000u : hb;
  return ff_make(__uint_as_float(hb), lo);
}

// global to shared memory, 8 bytes (bytes = 0: zeros)
__device__ __forceinline__ void td_copy8(void* smem, const void* gmem, int bytes) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(a), "l"(gmem), "r"(bytes) : "memory");
}

// A channel's running sum: heads added exactly (two_sum), the errors and tails
// in lo, folded into the head after each delay.
struct TdSum {
  float hi, lo;
  __device__ __forceinline__ void add(float h, float l) {
    const FF s = ff_two_sum(hi, h);
    hi = s.hi;
    lo = (lo + s.lo) + l;
  }
  __device__ __forceinline__ void renorm() {
    const FF s = ff_fast_two_sum(hi, lo);
    hi = s.hi;
    lo = s.lo;
  }
  // + d * f
  __device__ __forceinline__ void fma(const FF& d, float fh, float fl) {
    const float p = d.hi * fh;
    add(p, fmaf(d.lo, fh, fmaf(d.hi, fl, fmaf(d.hi, fh, -p))));
  }
};

// float f * 2^scale as a double, from the bits
__device__ __forceinline__ double td_widen(float f, int scale) {
  const unsigned u = __float_as_uint(f);
  const int ef = (int)((u >> 23) & 0xFF);
  if (ef == 0xFF) return __longlong_as_double(0x7ff8000000000000ll);
  const int ed = ef - 127 + 1023 + scale;
  if (ef == 0 || ed <= 0) return 0.0;
  if (ed >= 0x7FF) return __longlong_as_double((long long)(((unsigned long long)(u >> 31) << 63) | 0x7ff0000000000000ull));
  const unsigned long long sign = (unsigned long long)(u & 0x80000000u) << 32;
  return __longlong_as_double((long long)(sign | ((unsigned long long)ed << 52) |
                                          ((unsigned long long)(u & 0x7FFFFFu) << 29)));
}

template <int kMaxDelay>
__global__ void __launch_bounds__(kTdThreads) k_td_tdi_ff(TdLayoutFF lay, const double* __restrict__ links,
                                                          int64_t n_ext, int64_t n, int orth,
                                                          double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char td_raw[];
  const int win = kTdTile + (int)lay.added + 1;  // at most kTdMaxWindow
  FF* val = reinterpret_cast<FF*>(td_raw);  // [6][win]: the doubles first, then their float-float pairs
  FF* dif = val + 6 * win;                  // [6][win]: right - left
  double* raw = reinterpret_cast<double*>(td_raw);
  __shared__ int wmax[kTdThreads / 32];
  const double* src = links + (int64_t)blockIdx.y * 6 * n_ext;
  double* dst = out + (int64_t)blockIdx.y * 3 * n;
  const int64_t i0 = (int64_t)blockIdx.x * kTdTile;
  const int avail = (int)min((int64_t)win, n_ext - i0);
  // all of a thread's loads in flight at once (in turn per link, they took a
  // third of the block's time)
#pragma unroll 1
  for (int j = threadIdx.x; j < win; j += kTdThreads) {
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      const bool in = j < avail;
      td_copy8(raw + l * win + j, src + l * n_ext + i0 + (in ? j : 0), in ? 8 : 0);
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  int emax = 0;  // largest finite biased exponent in the window (each thread's own slots)
#pragma unroll 1
  for (int j = threadIdx.x; j < win; j += kTdThreads) {
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      const int E = (__double2hiint(raw[l * win + j]) >> 20) & 0x7FF;
      if (E != 0x7FF) emax = max(emax, E);
    }
  }
  emax = __reduce_max_sync(0xffffffffu, emax);
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = emax;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kTdThreads / 32; ++w) emax = max(emax, wmax[w]);
  const int scale = emax - 1023;  // the window's largest magnitude maps into [1, 2)
  const TdScale sc = td_scale(scale);
  // each thread rewrites the slots it loaded: the six links become, for channel
  // c, the differences P (slot 2c) and Q (slot 2c + 1), in place
#pragma unroll 1
  for (int j = threadIdx.x; j < win; j += kTdThreads) {
    FF l[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) l[k] = td_split(raw[k * win + j], sc);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      val[2 * c * win + j] = l[(5 + 2 * c) % 6] - l[2 * c];
      val[(2 * c + 1) * win + j] = l[(4 + 2 * c) % 6] - l[2 * c + 1];
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int j = threadIdx.x; j + 1 < win; j += kTdThreads) {
#pragma unroll
    for (int l = 0; l < 6; ++l) dif[l * win + j] = val[l * win + j + 1] - val[l * win + j];
  }
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < kTdTile / kTdThreads; ++r) {
    const int t = threadIdx.x + r * kTdThreads;
    const int64_t i = i0 + t;
    if (i >= n) break;
    FF ch[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const FF v0 = val[2 * c * win + t + (int)lay.added];
      TdSum acc;
      acc.hi = v0.hi;
      acc.lo = v0.lo;
#pragma unroll
      for (int k = 0; k < kMaxDelay; ++k) {
        const int o = (2 * c + 1 - (k & 1)) * win + t + (int)lay.shift[k];
        const FF v = val[o], d = dif[o];
        const float2 f = lay.frac[k];
        if (k == 0 || k > 4) {
          acc.add(v.hi, v.lo);
          acc.fma(d, f.x, f.y);
        } else {
          acc.add(-v.hi, -v.lo);
          acc.fma(d, -f.x, -f.y);
        }
        acc.renorm();
      }
      ch[c] = ff_two_sum(acc.hi, acc.lo);
    }
    FF o3[3];
    if (orth) {
      const FF X = ch[0], Y = ch[1], Z = ch[2];
      o3[0] = (Z - X) * ff_make(lay.rs2.x, lay.rs2.y);
      o3[1] = (X - ff_mulf(Y, 2.0f) + Z) * ff_make(lay.rs6.x, lay.rs6.y);
      o3[2] = (X + Y + Z) * ff_make(lay.rs3.x, lay.rs3.y);
    } else {
      o3[0] = ch[0];
      o3[1] = ch[1];
      o3[2] = ch[2];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) dst[(int64_t)c * n + i] = __dadd_rn(td_widen(o3[c].hi, scale), td_widen(o3[c].lo, scale));
  }
}

template <int kMaxDelay>
static int launch_td_tdi_ff(const TdLayout& lay, const double* links, int64_t B, int64_t n_ext, int64_t n, int orth,
                            double* out, cudaStream_t st) {
  TdLayoutFF lf;
  td_layout_ff(lay, lf);
  const dim3 grid((unsigned)((n + kTdTile - 1) / kTdTile), (unsigned)B);
  const int64_t win = kTdTile + lay.added + 1;
  const size_t smem = (size_t)12 * win * sizeof(FF);  // [6][win] values + [6][win] differences, float pairs
  if (win > kTdMaxWindow) {
    set_error("pes_td_tdi_combination_mixed: the longest delay (%lld samples) exceeds %d",
              (long long)lay.added, kTdMaxWindow - kTdTile - 1);
    return PES_EINVAL;
  }
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_td_tdi_ff<kMaxDelay>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) {
      set_error("pes_td_tdi_combination_mixed: %s", cudaGetErrorString(e));
      return PES_ECUDA;
    }
  }
  k_td_tdi_ff<kMaxDelay><<<grid, kTdThreads, smem, st>>>(lf, links, n_ext, n, orth, out);
  PES_CHECK_LAUNCH();
  return PES_OK;
}

extern "C" {

const char* pes_last_error(void) { return pes::g_error; }
int pes_version(void) { return 1; }

int pes_orbit_vectors(const PesOrbit* orbit, const double* time, int64_t n, double* out, void* stream) {
  PES_REQUIRE(orbit && (n == 0 || (time && out)), "pes_orbit_vectors: null pointer");
  PES_REQUIRE(n >= 0, "pes_orbit_vectors: n < 0");
  PES_REQUIRE(orbit->kind == 0 || orbit->kind == 1, "pes_orbit_vectors: unknown orbit kind %d", orbit->kind);
  if (n == 0) return PES_OK;
  k_orbit_vectors<<<ceil_div(n, 128), 128, 0, as_stream(stream)>>>(*orbit, time, n, out);
  PES_CHECK_LAUNCH();
  return PES_OK;
}

int pes_polarization(double lam, double beta, double psi, double* plus9, double* cross9, double* k3) {
  PES_REQUIRE(plus9 && cross9 && k3, "pes_polarization: null pointer");
  Polar<double> p;
  make_polar<double>(lam, ::sin(beta), ::cos(beta), psi, p);
  const int ii[6] = {0, 0, 0, 1, 1, 2}, jj[6] = {0, 1, 2, 1, 2, 2};
  for (int m = 0; m < 6; ++m) {
    plus9[3 * ii[m] + jj[m]] = plus9[3 * jj[m] + ii[m]] = p.P[m];
    cross9[3 * ii[m] + jj[m]] = cross9[3 * jj[m] + ii[m]] = p.X[m];
  }
  for (int j = 0; j < 3; ++j) k3[j] = p.k[j];
  return PES_OK;
}

int pes_response_links(const PesOrbit* orbit, const double* freqs, int64_t n, int32_t n_modes, const double* hp,
                       const double* hc, const double* tf, double lam, double beta, double psi, double tc,
                       double* links, void* stream) {
  PES_REQUIRE(orbit, "pes_response_links: null orbit");
  PES_REQUIRE(n >= 0 && n_modes >= 1, "pes_response_links: bad sizes n=%lld modes=%d", (long long)n, n_modes);
  PES_REQUIRE(orbit->kind == 0 || orbit->kind == 1, "pes_response_links: unknown orbit kind %d", orbit->kind);
  if (n == 0) return PES_OK;
  PES_REQUIRE(freqs && hp && hc && tf && links, "pes_response_links: null pointer");
  LinkArg arg;
  link_arg(*orbit, lam, beta, psi, tc, arg);
  k_response_links<<<ceil_div(n, kLinkThreads), kLinkThreads, 0, as_stream(stream)>>>(
      arg, freqs, n, n_modes, reinterpret_cast<const double2*>(hp), reinterpret_cast<const double2*>(hc), tf,
      reinterpret_cast<double2*>(links));
  PES_CHECK_LAUNCH();
  return PES_OK;
}

int pes_tdi_combination(const double* freqs, int64_t n, double arm_sec, int32_t generation, int32_t orthogonal,
                        const double* links, double* out, void* stream) {
  PES_REQUIRE(generation == 15 || generation == 20, "pes_tdi_combination: unsupported generation %d", generation);
  PES_REQUIRE(n >= 0, "pes_tdi_combination: n < 0");
  if (n == 0) return PES_OK;
  PES_REQUIRE(freqs && links && out, "pes_tdi_combination: null pointer");
  k_tdi<<<ceil_div(n, kTdiThreads), kTdiThreads, 0, as_stream(stream)>>>(freqs, n, arm_sec, generation == 20, orthogonal != 0,
                                                          reinterpret_cast<const double2*>(links),
                                                          reinterpret_cast<double2*>(out));
  PES_CHECK_LAUNCH();
  return PES_OK;
}

int64_t pes_whittle_workspace_len(int64_t n) {
  if (n <= 0) return 1;
  // one bin per thread up to 1024 blocks (four per thread left most SMs a block or none:
  // 20 us on 125 410 bins)
  int64_t blocks = (n + kWhittleThreads - 1) / kWhittleThreads;
  return blocks < kWhittleMaxBlocks ? blocks : kWhittleMaxBlocks;
}

int pes_whittle_lnl(const double* data, const double* response, const double* psd, int32_t n_chan, int64_t n,
                    double df, double* workspace, int64_t workspace_len, double* out, void* stream) {
  PES_REQUIRE(n_chan >= 1 && n_chan <= 3, "pes_whittle_lnl: n_chan must be 1..3, got %d", n_chan);
  PES_REQUIRE(n >= 0, "pes_whittle_lnl: n < 0");
  PES_REQUIRE(out, "pes_whittle_lnl: null out");
  const int64_t nblk = pes_whittle_workspace_len(n);
  PES_REQUIRE(workspace && workspace_len >= nblk, "pes_whittle_lnl: workspace needs %lld doubles",
              (long long)nblk);
  cudaStream_t st = as_stream(stream);
  if (n == 0) {
    PES_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(double), st));
    return PES_OK;
  }
  PES_REQUIRE(data && response && psd, "pes_whittle_lnl: null pointer");
  const int64_t per_block = (n + nblk - 1) / nblk;
  k_whittle_partial<<<(unsigned)nblk, kWhittleThreads, 0, st>>>(reinterpret_cast<const double2*>(data),
                                                                 reinterpret_cast<const double2*>(response), psd,
                                                                 n_chan, n, per_block, workspace);
  PES_CHECK_LAUNCH();
  k_whittle_final<<<1, kWhittleThreads, 0, st>>>(workspace, (int)nblk, -2.0 * df, out);
  PES_CHECK_LAUNCH();
  return PES_OK;
}

int pes_whittle_lnl_noalloc(const double* data, const double* response, const double* psd, int32_t n_chan,
                            int64_t n, double df, double* out, void* stream) {
  PES_REQUIRE(n_chan >= 1 && n_chan <= 3, "pes_whittle_lnl_noalloc: n_chan must be 1..3, got %d", n_chan);
  PES_REQUIRE(n >= 0 && n <= PES_WHITTLE_NOALLOC_MAX_BINS,
              "pes_whittle_lnl_noalloc: n = %lld outside [0, %lld]", (long long)n,
              (long long)PES_WHITTLE_NOALLOC_MAX_BINS);
  PES_REQUIRE(out, "pes_whittle_lnl_noalloc: null out");
  const int64_t nblk = pes_whittle_workspace_len(n);
  PES_REQUIRE(nblk <= kNoAllocPartials, "pes_whittle_lnl_noalloc: %lld partial sums exceed the %d-entry scratch",
              (long long)nblk, kNoAllocPartials);
  double* scratch = nullptr;
  int rc = whittle_scratch(&scratch);
  if (rc != PES_OK) return rc;
  cudaStream_t st = as_stream(stream);
  if (n == 0) {
    PES_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(double), st));
    return PES_OK;
  }
  PES_REQUIRE(data && response && psd, "pes_whittle_lnl_noalloc: null pointer");
  // every partial the final pass reads is written by the first pass, so the
  // scratch needs no clearing between calls
  const int64_t per_block = (n + nblk - 1) / nblk;
  k_whittle_partial<<<(unsigned)nblk, kWhittleThreads, 0, st>>>(reinterpret_cast<const double2*>(data),
                                                                 reinterpret_cast<const double2*>(response), psd,
                                                                 n_chan, n, per_block, scratch);
  PES_CHECK_LAUNCH();
  k_whittle_final<<<1, kWhittleThreads, 0, st>>>(scratch, (int)nblk, -2.0 * df, out);
  PES_CHECK_LAUNCH();
  return PES_OK;
}

int pes_phenomd(const double* theta, const double* freqs, int64_t n, double f_ref, double f_cut_hz, double* hp,
                double* hc, double* tf, void* stream) {
  PES_REQUIRE(theta, "pes_phenomd: null theta");
  PES_REQUIRE(n >= 0, "pes_phenomd: n < 0");
  if (n == 0) return PES_OK;
  PES_REQUIRE(freqs && hp && hc && tf, "pes_phenomd: null pointer");
  return launch_wave<1>(theta, freqs, n, f_ref, f_cut_hz, hp, hc, tf, as_stream(stream));
}

int pes_phenomhm(const double* theta, const double* freqs, int64_t n, double f_ref, double f_cut_hz, double* hp,
                 double* hc, double* tf, void* stream) {
  PES_REQUIRE(theta, "pes_phenomhm: null theta");
  PES_REQUIRE(n >= 0, "pes_phenomhm: n < 0");
  if (n == 0) return PES_OK;
  PES_REQUIRE(freqs && hp && hc && tf, "pes_phenomhm: null pointer");
  return launch_wave<kHMModes>(theta, freqs, n, f_ref, f_cut_hz, hp, hc, tf, as_stream(stream));
}

int pes_pn_tf(const double* params, int64_t B, const double* freqs, int64_t n, double* tf, void* stream) {
  PES_REQUIRE(B >= 0 && n >= 0, "pes_pn_tf: negative size (B = %lld, n = %lld)", (long long)B, (long long)n);
  PES_REQUIRE(B <= 65535, "pes_pn_tf: at most 65535 parameter sets per call, got %lld", (long long)B);
  if (B == 0 || n == 0) return PES_OK;
  PES_REQUIRE(params && freqs && tf, "pes_pn_tf: null pointer");
  k_pn_tf<<<dim3(ceil_div(n, 256), (unsigned)B), 256, 0, as_stream(stream)>>>(params, n, freqs, tf);
  PES_CHECK_LAUNCH();
  return PES_OK;
}

int pes_td_tdi_layout(double arm_sec, double delta_time, int32_t generation, int64_t* added, int32_t* max_delay,
                      int64_t* shifts, double* fracs) {
  PES_REQUIRE(generation == 15 || generation == 20, "pes_td_tdi_layout: unsupported generation %d", generation);
  PES_REQUIRE(std::isfinite(arm_sec) && arm_sec > 0.0 && std::isfinite(delta_time) && delta_time > 0.0,
              "pes_td_tdi_layout: arm length and sampling step must be finite and > 0 (%g, %g)", arm_sec,
              delta_time);
  PES_REQUIRE(added && max_delay && shifts && fracs, "pes_td_tdi_layout: null pointer");
  PES_REQUIRE(7.0 * arm_sec / delta_time < 1e9, "pes_td_tdi_layout: delay of %g samples too long",
              7.0 * arm_sec / delta_time);
  TdLayout lay;
  td_layout(arm_sec, delta_time, generation == 20, lay);
  *added = lay.added;
  *max_delay = lay.max_delay;
  for (int k = 0; k < lay.max_delay; ++k) {
    shifts[k] = lay.shift[k];
    fracs[k] = lay.frac[k];
  }
  return PES_OK;
}

int pes_td_tdi_combination(const double* links, int64_t B, int64_t n_ext, int64_t n, double arm_sec,
                           double delta_time, int32_t generation, int32_t orthogonal, double* out, void* stream) {
  PES_REQUIRE(generation == 15 || generation == 20, "pes_td_tdi_combination: unsupported generation %d",
              generation);
  PES_REQUIRE(std::isfinite(arm_sec) && arm_sec > 0.0 && std::isfinite(delta_time) && delta_time > 0.0,
              "pes_td_tdi_combination: arm length and sampling step must be finite and > 0 (%g, %g)", arm_sec,
              delta_time);
  PES_REQUIRE(B >= 0 && B <= 65535 && n >= 0 && n_ext >= 0,
              "pes_td_tdi_combination: bad sizes (B = %lld, n = %lld, n_ext = %lld)", (long long)B, (long long)n,
              (long long)n_ext);
  PES_REQUIRE(n <= (int64_t)kTdTile * 0x7FFFFFFF, "pes_td_tdi_combination: %lld samples exceed the launch grid",
              (long long)n);
  PES_REQUIRE(7.0 * arm_sec / delta_time < 1e9, "pes_td_tdi_combination: delay of %g samples too long",
              7.0 * arm_sec / delta_time);
  TdLayout lay;
  td_layout(arm_sec, delta_time, generation == 20, lay);
  for (int k = 0; k < lay.max_delay; ++k)  // every read stays in [i, i + added]
    PES_REQUIRE(lay.shift[k] >= 0 && lay.shift[k] + 1 <= lay.added,
                "pes_td_tdi_combination: delay layout out of range (shift %lld, added %lld)",
                (long long)lay.shift[k], (long long)lay.added);
  PES_REQUIRE(n_ext >= n + lay.added,
              "pes_td_tdi_combination: %lld link samples for %lld outputs, need n + %lld (the longest delay)",
              (long long)n_ext, (long long)n, (long long)lay.added);
  if (B == 0 || n == 0) return PES_OK;
  PES_REQUIRE(links && out, "pes_td_tdi_combination: null pointer");
  const cudaStream_t st = as_stream(stream);
  return generation == 20 ? launch_td_tdi<7>(lay, links, B, n_ext, n, orthogonal != 0, out, st)
                          : launch_td_tdi<3>(lay, links, B, n_ext, n, orthogonal != 0, out, st);
}

int pes_td_tdi_combination_mixed(const double* links, int64_t B, int64_t n_ext, int64_t n, double arm_sec,
                                 double delta_time, int32_t generation, int32_t orthogonal, double* out,
                                 void* stream) {
  PES_REQUIRE(generation == 15 || generation == 20, "pes_td_tdi_combination_mixed: unsupported generation %d",
              generation);
  PES_REQUIRE(std::isfinite(arm_sec) && arm_sec > 0.0 && std::isfinite(delta_time) && delta_time > 0.0,
              "pes_td_tdi_combination_mixed: arm length and sampling step must be finite and > 0 (%g, %g)",
              arm_sec, delta_time);
  PES_REQUIRE(B >= 0 && B <= 65535 && n >= 0 && n_ext >= 0,
              "pes_td_tdi_combination_mixed: bad sizes (B = %lld, n = %lld, n_ext = %lld)", (long long)B,
              (long long)n, (long long)n_ext);
  PES_REQUIRE(n <= (int64_t)kTdTile * 0x7FFFFFFF, "pes_td_tdi_combination_mixed: %lld samples exceed the launch grid",
              (long long)n);
  PES_REQUIRE(7.0 * arm_sec / delta_time < 1e9, "pes_td_tdi_combination_mixed: delay of %g samples too long",
              7.0 * arm_sec / delta_time);
  TdLayout lay;
  td_layout(arm_sec, delta_time, generation == 20, lay);
  for (int k = 0; k < lay.max_delay; ++k)  // every read stays in [i, i + added]
    PES_REQUIRE(lay.shift[k] >= 0 && lay.shift[k] + 1 <= lay.added,
                "pes_td_tdi_combination_mixed: delay layout out of range (shift %lld, added %lld)",
                (long long)lay.shift[k], (long long)lay.added);
  PES_REQUIRE(n_ext >= n + lay.added,
              "pes_td_tdi_combination_mixed: %lld link samples for %lld outputs, need n + %lld (the longest delay)",
              (long long)n_ext, (long long)n, (long long)lay.added);
  PES_REQUIRE(kTdTile + lay.added + 1 <= kTdMaxWindow,
              "pes_td_tdi_combination_mixed: the longest delay (%lld samples) exceeds %d", (long long)lay.added,
              kTdMaxWindow - kTdTile - 1);
  if (B == 0 || n == 0) return PES_OK;
  PES_REQUIRE(links && out, "pes_td_tdi_combination_mixed: null pointer");
  const cudaStream_t st = as_stream(stream);
  return generation == 20 ? launch_td_tdi_ff<7>(lay, links, B, n_ext, n, orthogonal != 0, out, st)
                          : launch_td_tdi_ff<3>(lay, links, B, n_ext, n, orthogonal != 0, out, st);
}

}  // extern "C"
