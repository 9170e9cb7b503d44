// Host check of the float-float forms of the re-evaluation and of the <h|h> sums
// (pespace_gb300/csrc/pes_ff.cuh) against long double: unrenormalised
// multiply-adds and dot products, alone and in a chain, and the tabulated sine and
// cosine.  Prints the largest errors, one "name value" pair per line.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../pespace_gb300/csrc/pes_ff.cuh"

using namespace pes;

static long double ld(const FF& x) { return (long double)x.hi + (long double)x.lo; }

int main() {
  std::mt19937_64 rng(2027);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  auto any = [&] { return ff_from((U(rng) < 0.5 ? -1.0 : 1.0) * std::pow(10.0, -4.0 + 8.0 * U(rng))); };
  double e_mad = 0, e_dot = 0, e_chain = 0, e_tab[3] = {0, 0, 0};
  float4 tab[kFfTrig];
  const long double two_pi = 6.283185307179586476925286766559L;
  for (int k = 0; k < kFfTrig; ++k) {
    const long double a = two_pi * k / kFfTrig;
    const float s = (float)sinl(a), c = (float)cosl(a);
    tab[k] = make_float4(s, (float)(sinl(a) - s), c, (float)(cosl(a) - c));
  }
  const double range[3] = {1e3, 1e4, 262144.0};
  for (int it = 0; it < 400000; ++it) {
    const FF a = any(), b = any(), c = any(), d = any();
    e_mad = std::fmax(e_mad, (double)(fabsl(ld(ff_mad(a, b, c)) - (ld(a) * ld(b) + ld(c))) / (fabsl(ld(a) * ld(b)) + fabsl(ld(c)))));
    e_dot = std::fmax(e_dot, (double)(fabsl(ld(ff_dot2(a, b, c, d)) - (ld(a) * ld(b) + ld(c) * ld(d))) /
                                      (fabsl(ld(a) * ld(b)) + fabsl(ld(c) * ld(d)))));
    // a polynomial of twelve terms, against its sum of magnitudes
    const FF u = ff_from(0.05 + U(rng));
    FF lazy = any();
    long double want = ld(lazy), mag = fabsl(want);
    for (int j = 0; j < 11; ++j) {
      const FF t = any();
      lazy = ff_mad(lazy, u, t);
      want = want * ld(u) + ld(t);
      mag = mag * fabsl(ld(u)) + fabsl(ld(t));
    }
    e_chain = std::fmax(e_chain, (double)(fabsl(ld(lazy) - want) / mag));
    for (int r = 0; r < 3; ++r) {
      const FF x = ff_from((2.0 * U(rng) - 1.0) * range[r]);
      FF s, c2;
      ff_sincos_tab(tab, x, &s, &c2);
      e_tab[r] = std::fmax(e_tab[r], std::fmax((double)fabsl(ld(s) - sinl(ld(x))), (double)fabsl(ld(c2) - cosl(ld(x)))));
    }
  }
  std::printf("mad %.3e\ndot2 %.3e\nchain %.3e\ntab_1e3 %.3e\ntab_1e4 %.3e\ntab_2e18 %.3e\n", e_mad, e_dot,
              e_chain, e_tab[0], e_tab[1], e_tab[2]);
  return 0;
}
