// Forms of the model shared by the FP64 dense pass, the mixed Fisher pass and
// the plugins: FP64 functions of few operations, IMRPhenomD's coefficients rescaled to frequencies in Hz, and the response's
// trigonometric polynomials in the orbital angle.
#pragma once

#include "pes_plan.cuh"

namespace pes {

// ------------------------------------------------------------------ functions
constexpr int kTrig = 256;  // entries of the sine/cosine table
constexpr double k64Magic = 6755399441055744.0;             // 1.5 * 2^52: (x + M) - M rounds to an integer
constexpr double k64TwoPi = 6.283185307179586;              // 2 pi, head
constexpr double k64TwoPiLo = 2.4492935982947064e-16;       // 2 pi - head
constexpr double k64InvTwoPi = 0.15915494309189535;

// |x| from 2^45 on (also infinities and NaN): past what sincos64 reduces
__device__ __forceinline__ bool far64(double x) { return (__double2hiint(x) & 0x7fffffff) >= 0x42c00000; }
// sin and cos of such arguments (phases of light sources decades before they merge): the library's.
static __device__ __noinline__ double2 sincos64_far(double x) {
  double2 r;
  sincos(x, &r.x, &r.y);
  return r;
}

// sin and cos: x = k 2 pi / 256 + r, |r| <= pi / 256, table of the first, Taylor
// polynomials of the second (truncation below 1e-19), angle sum.  The rounding to k by
// k64Magic holds below 2^51 steps: |x| < 2^45.
__device__ __forceinline__ void sincos64(const double2* __restrict__ tab, double x, double* s, double* c) {
  if (far64(x)) {
    const double2 v = sincos64_far(x);
    *s = v.x;
    *c = v.y;
    return;
  }
  const double t = fma(x, k64InvTwoPi * kTrig, k64Magic);
  const int k = __double2loint(t) & (kTrig - 1);
  const double kf = t - k64Magic;
  double r = fma(-kf, k64TwoPi / kTrig, x);
  r = fma(-kf, k64TwoPiLo / kTrig, r);
  const double z = r * r;
  const double sr = fma(r * z, fma(z, 1.0 / 120.0, -1.0 / 6.0), r);
  const double cm = z * fma(z, fma(z, -1.0 / 720.0, 1.0 / 24.0), -0.5);
  const double2 e = tab[k];
  *s = e.x + fma(e.x, cm, e.y * sr);
  *c = e.y + fma(e.y, cm, -(e.x * sr));
}

// x less its whole turns (x itself where far64)
__device__ __forceinline__ double turns64(double x) {
  if (far64(x)) return x;
  const double kf = fma(x, k64InvTwoPi, k64Magic) - k64Magic;
  return fma(-kf, k64TwoPiLo, fma(-kf, k64TwoPi, x));
}

// 1 / x for normal positive x: the hardware estimate and two Newton steps
__device__ __forceinline__ double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  r = fma(r, fma(-x, r, 1.0), r);
  return r;
}

// atan(x): the nearest multiple phi of 2 pi / 256 by the FP32 function (not an
// FP64 instruction), then tan(atan x - phi) = (x cos phi - sin phi) / (cos phi
// + x sin phi), at most 0.013, and four terms of its arctangent series
// (truncation below 1e-18).
__device__ __forceinline__ double atan64(const double2* __restrict__ tab, double x) {
  const int k = __float2int_rn(atanf((float)x) * (float)(kTrig * k64InvTwoPi));
  const double2 e = tab[k & (kTrig - 1)];
  const double t = fma(x, e.y, -e.x) * rcp64(fma(x, e.x, e.y)), z = t * t;
  const double p = fma(z, fma(z, -1.0 / 7.0, 0.2), -1.0 / 3.0);
  const double kd = __hiloint2double(0x43380000 + (k >> 31), k) - k64Magic;  // (double)k
  return fma(kd, k64TwoPi / kTrig, fma(t * z, p, t));
}

// sin(x)/x and d/dx sin(x)/x: N terms of the Taylor series in z = x^2
template <int N>
__device__ __forceinline__ double sinc_taylor_n(double z) {
  constexpr double c[13] = {1.0, -0.16666666666666666, 0.008333333333333333, -0.0001984126984126984,
                            2.7557319223985893e-06, -2.505210838544172e-08, 1.6059043836821613e-10,
                            -7.647163731819816e-13, 2.8114572543455206e-15, -8.22063524662433e-18,
                            1.9572941063391263e-20, -3.868170170630684e-23, 6.446950284384474e-26};
  double p = c[N - 1];
#pragma unroll
  for (int k = N - 2; k >= 0; --k) p = fma(p, z, c[k]);
  return p;
}
template <int N>
__device__ __forceinline__ double dsinc_taylor_n(double z) {  // times x
  constexpr double c[12] = {-0.3333333333333333, 0.03333333333333333, -0.0011904761904761906, 2.2045855379188714e-05,
                            -2.505210838544172e-07, 1.9270852604185937e-09, -1.0706029224547743e-11,
                            4.498331606952833e-14, -1.4797143443923793e-16, 3.9145882126782523e-19,
                            -8.509974375387505e-22, 1.5472680682522736e-24};
  double p = c[N - 1];
#pragma unroll
  for (int k = N - 2; k >= 0; --k) p = fma(p, z, c[k]);
  return p;
}
// the series' length for arguments up to amax: truncation below 1e-17 each
// (0.25: z^6/13!; 0.7: z^8/17!; 2: z^13/27!); 3: sin(x)/x itself
__device__ __forceinline__ int sinc_tier(double amax) { return amax <= 0.25 ? 0 : (amax <= 0.7 ? 1 : (amax <= 2.0 ? 2 : 3)); }
template <bool kGrad>
__device__ __forceinline__ void sinc64(const double2* __restrict__ tab, int tier, double x, double* s, double* ds) {
  const double z = x * x;
  if (tier == 0) {
    *s = sinc_taylor_n<6>(z);
    if (kGrad) *ds = dsinc_taylor_n<6>(z) * x;
  } else if (tier == 1) {
    *s = sinc_taylor_n<8>(z);
    if (kGrad) *ds = dsinc_taylor_n<8>(z) * x;
  } else if (tier == 2 || z <= 4.0) {
    *s = sinc_taylor_n<13>(z);
    if (kGrad) *ds = dsinc_taylor_n<12>(z) * x;
  } else {
    double sn, cs;
    sincos64(tab, x, &sn, &cs);
    const double ix = 1.0 / x;
    *s = sn * ix;
    if (kGrad) *ds = (cs - *s) * ix;
  }
}

// The table in shared memory from its first quadrant (the caller's barrier follows).
__device__ __forceinline__ void fill_trig(double2* tab) {
  if (threadIdx.x < kTrig / 4) {
    double s, c;
    sincospi(2.0 * (double)threadIdx.x / kTrig, &s, &c);
    tab[threadIdx.x] = make_double2(s, c);
    tab[threadIdx.x + kTrig / 4] = make_double2(c, -s);
    tab[threadIdx.x + kTrig / 2] = make_double2(-s, -c);
    tab[threadIdx.x + 3 * kTrig / 4] = make_double2(-c, s);
  }
}

// Products and quotients of pairs hi + lo.
struct DD {
  double h, l;
};
PES_HD DD dd_two(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
PES_HD DD dd_mul(const DD& a, const DD& b) {
  const double p = a.h * b.h;
  return dd_two(p, ::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
PES_HD DD dd_div(const DD& a, const DD& b) {
  const double q = a.h / b.h;
  const double p = q * b.h, e = ::fma(q, b.h, -p);
  return dd_two(q, (((a.h - p) - e) + a.l - q * b.l) / b.h);
}
PES_HD DD dd_cbrt(const DD& a) {
  const double c = ::cbrt(a.h);
  const DD c3 = dd_mul(dd_mul({c, 0.0}, {c, 0.0}), {c, 0.0});
  return dd_two(c, ((a.h - c3.h) + (a.l - c3.l)) / (3.0 * c * c));
}

// IMRPhenomD's coefficients for frequencies in Hz (PhenomDCoef times powers of
// the total mass), so that a bin's tabulated powers of f multiply them.
template <class T>
struct FreqCoef {
  T pin[12];            // Psi_ins = f^{-5/3} sum pin_j f^{j/3} + (lg0 + lg1 f^{1/3}) ln(f)/3
  T lg0, lg1;
  T pint[4];            // Psi_int = pint0 + pint1 f + pint2 f^{-3} + pint3 ln f
  T pm[5], f5, fd;      // Psi_mrd = pm0 + pm1 f + pm2/f + pm3 f^{3/4} + pm4 atan((f - f5)/fd)
  T a0;                 // A = a0 f^{-7/6} Ahat
  T ai[8];              // Ahat_ins = 1 + sum ai_j f^{(j+2)/3}
  T dl[5];              // Ahat_int = sum dl_j f^j
  T gm, w, fr, gx;      // Ahat_mrd = gm / ((f - fr)^2 + w^2) exp(-gx (f - fr))
};
constexpr int kFreqScalars = (int)(sizeof(FreqCoef<double>) / sizeof(double));

// kRole: kPhasePart (pin .. fd) and/or kAmpPart (a0 .. gx)
template <class T, int kRole = 3>
PES_HD void freq_coef(const PhenomDCoef<T>& c, FreqCoef<T>& o) {
  const T M = c.Msec, cu = dcbrt(M), icu = 1.0 / cu, iM = icu * icu * icu;
  if constexpr ((kRole & kAmpPart) != 0) {
    o.a0 = c.amp_scale * (iM / dsqrt(cu));
    T pw = cu * cu;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o.ai[j] = c.ai[j] * pw;
      pw = pw * cu;
    }
    pw = lift<T>(1.0);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      o.dl[j] = c.dl[j] * pw;
      pw = pw * M;
    }
    o.w = c.g3fDM * iM;
    o.gm = c.g1 * (o.w * iM);
    o.fr = c.fRD * iM;
    o.gx = c.g2 / o.w;
  }
  if constexpr ((kRole & kPhasePart) == 0) return;
  const T icu2 = icu * icu;
  T pw = iM * icu2;  // cu^(j-5)
#pragma unroll
  for (int j = 0; j < 12; ++j) {
    o.pin[j] = c.pin[j] * pw;
    pw = pw * cu;
  }
  const T lcu = dlog(cu);
  o.lg0 = c.lg0;
  o.lg1 = c.lg1 * cu;
  o.pin[5] = o.pin[5] + o.lg0 * lcu;
  o.pin[6] = o.pin[6] + o.lg1 * lcu;
  o.pint[0] = c.pint[0] + c.pint[3] * (3.0 * lcu);
  o.pint[1] = c.pint[1] * M;
  o.pint[2] = c.pint[2] * (iM * iM * iM);
  o.pint[3] = c.pint[3];
  o.pm[0] = c.pm[0];
  o.pm[1] = c.pm[1] * M;
  o.pm[2] = c.pm[2] * iM;
  const T q = dsqrt(dsqrt(M));
  o.pm[3] = c.pm[3] * (q * q * q);
  o.pm[4] = c.pm[4];
  o.f5 = c.pm[5] * iM;
  o.fd = c.fDM * iM;
}

// Per sample and detector, the response's trigonometric polynomials in the
// orbital angle, [1, c1, s1, c2, s2]: the arms n (links 12 and 23; link 31 is
// minus their sum) along the polarisation axes p and q, F+ = (n.p)^2 - (n.q)^2,
// Fx = 2 (n.p)(n.q); the node delays y_k = k.(x_k - x0) of nodes 1 and 2 (they
// sum to zero); k.x0 = k0[0] cos alpha + k0[1] sin alpha; each for the value and
// for its derivatives with respect to lambda and sin beta.  Geocentric: the
// terms c1, s1 of the rotation angle, alpha of k.x0 apart.
struct RespTab {
  double np[3][2][5], nq[3][2][5];  // [value, d/dlambda, d/dsinbeta][arm]
  double y[3][2][5];
  double k0[3][2];
};
// One warp: detector d's polynomials at the parameters th (set * 9 + angle per
// lane, then the Fourier sums); v: the warp's scratch, w9: the nine angles.
static __device__ void response_tables(const PlanDev& P, const double* __restrict__ th, int d, int lane, double (*v)[6],
                                const double2* w9, RespTab& r) {
  const PesOrbit& ob = P.orbit[d];
  // 9 equispaced angles x (value, d/dlambda, d/dsinbeta)
  if (lane < 27) {
    const int set = lane / 9, m = lane % 9;
    const double cm = w9[m].x, sm = w9[m].y;
    // polarisation vectors p, q and the propagation vector, and this set's derivative of them
    double sl, cl, sp, cp;
    dsincos(th[6], &sl, &cl);
    dsincos(th[8], &sp, &cp);
    const double sb = th[7], cb = sqrt((1.0 - sb) * (1.0 + sb)), dcb = -sb / cb;
    const double p[3] = {sl * cp - cl * sb * sp, -cl * cp - sl * sb * sp, cb * sp};
    const double q[3] = {-sl * sp - cl * sb * cp, cl * sp - sl * sb * cp, cb * cp};
    double dp[3] = {0.0, 0.0, 0.0}, dq[3] = {0.0, 0.0, 0.0}, k[3];
    if (set == 0) {
      k[0] = -(cb * cl);
      k[1] = -(cb * sl);
      k[2] = -sb;
    } else if (set == 1) {
      dp[0] = -p[1];
      dp[1] = p[0];
      dp[2] = 0.0;
      dq[0] = -q[1];
      dq[1] = q[0];
      dq[2] = 0.0;
      k[0] = cb * sl;
      k[1] = -(cb * cl);
      k[2] = 0.0;
    } else {
      dp[0] = -cl * sp;
      dp[1] = -sl * sp;
      dp[2] = dcb * sp;
      dq[0] = -cl * cp;
      dq[1] = -sl * cp;
      dq[2] = dcb * cp;
      k[0] = -(dcb * cl);
      k[1] = -(dcb * sl);
      k[2] = -1.0;
    }
    double xd[3][3];
    if (ob.kind == 0) {
      const double sc = sm * cm, s2 = sm * sm, c2 = cm * cm;
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        xd[n][0] = ob.r_sec * (sc * ob.sk[n] - (1.0 + s2) * ob.ck[n]);
        xd[n][1] = ob.r_sec * (sc * ob.ck[n] - (1.0 + c2) * ob.sk[n]);
        xd[n][2] = ob.r_sec * (-1.7320508075688772 * (cm * ob.ck[n] + sm * ob.sk[n]));
      }
    } else {
      const double c3 = -0.5, s3 = 0.86602540378443865;
      const double ck[3] = {cm, cm * c3 - sm * s3, cm * c3 + sm * s3};
      const double sk[3] = {sm, sm * c3 + cm * s3, sm * c3 - cm * s3};
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        xd[n][0] = ob.r_sec * (ob.sbeta_ref * ob.clam_ref * sk[n] + ob.slam_ref * ck[n]);
        xd[n][1] = ob.r_sec * (ob.sbeta_ref * ob.slam_ref * sk[n] - ob.clam_ref * ck[n]);
        xd[n][2] = ob.r_sec * (-ob.cbeta_ref * sk[n]);
      }
    }
    const double iL = 1.0 / ob.arm_sec;
    double* o6 = v[lane];
#pragma unroll
    for (int pr = 0; pr < 2; ++pr) {  // arms of links 12, 23
      double np = 0.0, nq = 0.0, y = 0.0;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double n = (xd[pr + 1][j] - xd[pr][j]) * iL;
        np += n * (set == 0 ? p[j] : dp[j]);
        nq += n * (set == 0 ? q[j] : dq[j]);
        y += k[j] * xd[pr][j];
      }
      o6[pr] = np;
      o6[2 + pr] = nq;
      o6[4 + pr] = y;
    }
    if (m == 0) {
      r.k0[set][0] = k[0] * kAUsec;
      r.k0[set][1] = k[1] * kAUsec;
    }
  }
  __syncwarp();
  // Fourier coefficients (2/9 sum v cos(m alpha), sin) of the six functions, degree 2, of each set
  for (int t = lane; t < 3 * 30; t += 32) {
    const int set = t / 30, q = t % 30 / 5, h = t % 5;
    const int m = (h + 1) / 2;
    double acc = 0.0;
#pragma unroll
    for (int a = 0; a < 9; ++a) {
      const double2 e = w9[(m * a) % 9];
      const double w = h == 0 ? 1.0 : ((h & 1) ? e.x : e.y);
      acc += v[set * 9 + a][q] * w;
    }
    acc *= h == 0 ? 1.0 / 9.0 : 2.0 / 9.0;
    if (q < 2)
      r.np[set][q][h] = acc;
    else if (q < 4)
      r.nq[set][q - 2][h] = acc;
    else
      r.y[set][q - 4][h] = acc;
  }
}

// cos, sin of 2 pi m / 9, m = threadIdx.x < 9, into w9 (a barrier before its use is the caller's)
__device__ __forceinline__ void nine_angles(double2* w9) {
  if (threadIdx.x < 9) {
    constexpr double c9[9] = {1.0, 0.766044443118978, 0.17364817766693036, -0.5, -0.9396926207859084,
                              -0.9396926207859084, -0.5, 0.17364817766693036, 0.766044443118978};
    constexpr double s9[9] = {0.0, 0.6427876096865394, 0.984807753012208, 0.8660254037844386, 0.3420201433256687,
                              -0.3420201433256687, -0.8660254037844386, -0.984807753012208, -0.6427876096865394};
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (q == threadIdx.x) w9[q] = make_double2(c9[q], s9[q]);
  }
}

}  // namespace pes
