"""The fixed-point transforms of the nonlinear pass
(falcon-dns_gb300/csrc/falcon_fixed.h) on the host with g++: whole inverse
(DIT) and forward (DIF) transforms of the plans of make_line_plan and of
grids of 3 Nm points, stage by stage as the kernel runs them (block scale
from the largest value of the stage before, padded places, tables of
fft_tables_host), against a long-double DFT.  Tolerance: a stage adds at most
2 units rms (2 products with constants) of 2^-61 of its bound to values that
fill the bound to 2^-6 or better in rms (3 bits of growth margin, 3 of peak
over rms), so 5 stages stay below sqrt(5) 2 2^-55 < 2^-52.8 of the norm; the
twiddles' cos/sin add 2^-54.  Inputs: random, all of the largest magnitude
with random signs, and one mode (for which one output holds everything).
Also the products of grid values, the doubles' conversion and the choice of
the length."""
import os
import subprocess

import pytest

from conftest import PKG

HARNESS = r'''
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "falcon_fixed.h"
#include "falcon_internal.h"
using namespace falcon;
typedef long double L;
typedef std::complex<L> C;
static const L PI = 3.141592653589793238462643383279502884L;
static unsigned long long rng = 88172645463325252ULL;
static unsigned long long rnd() { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }

struct Tables { std::vector<int4> tw; std::vector<unsigned> pos; std::vector<uint16_t> tab; };
static Tables tables(const FftPlan& f) {  // fft_tables_host with long-double angles
  Tables t;
  const int P = f.P;
  t.tw.resize(fx_table_size(f) + 1);
  auto root = [&](long long n, int N) {
    const L a = 2 * PI * (L)(n % N) / N;
    return fx_twiddle(2 * llrintl(cosl(a) * 0x1p61L), -2 * llrintl(sinl(a) * 0x1p61L));
  };
  for (int i = 0; i < P; ++i) {
    unsigned at = 0;
    for (int s = f.nrad - 1, x = i; s >= 0; x /= f.rad[s--]) at += (unsigned)(x % f.rad[s] * f.span[s]);
    t.tab.push_back((uint16_t)at);
  }
  for (int i = 0; i < P; ++i) t.pos.push_back(t.tab[fft_position(f, i)]);
  if (f.pfa) return t;
  const int inner = f.rad[f.nrad - 1];
  for (int s = f.nrad - 2, m = inner; s >= 0; --s) {
    const int p = f.rad[s];
    for (int q = 1; q < p; ++q)
      for (int k = 0; k < m; ++k) t.tw[m - inner + (q - 1) * m + k] = root((long long)q * k, m * p);
    m *= p;
  }
  int at = P;
  for (int s = 0; s < f.nrad; ++s)
    for (int j = 0, n = fx_root_size(f, f.rad[s]); j < n; ++j) t.tw[at++] = root(j, n);
  return t;
}
static void stage(const FftPlan& f, const Tables& t, int s, longlong2* b, int m, bool dif, int d, FxMax& o) {
  const int p = f.rad[s], inner = f.rad[f.nrad - 1];
  const int4* tw = t.tw.data() + (m - inner);
  const int4* root = t.tw.data() + f.P;
  for (int i = 0; i < s; ++i) root += fx_root_size(f, f.rad[i]);
#define K(q)                                                                                                        \
  case q:                                                                                                           \
    for (int lane = 0; lane < 3; ++lane)                                                                            \
      if (f.pfa) fx_stage<q, false>(b, t.tab.data(), f.span[s], f.P, m, tw, lane, 3, dif, d, o);                    \
      else fx_stage<q, true>(b, t.tab.data(), f.span[s], f.P, m, tw, lane, 3, dif, d, o);                           \
    return;
  switch (p) {
    K(2) K(3) K(4) K(5) K(6) K(7) K(8)
    default: fx_stage_any(b, f.P, p, m, tw, root, 0, 1, dif, d, o);
  }
}
int main() {
  int bad = 0, checked = 0;
  double worst = 0;
  std::vector<FftPlan> plans;
  for (int nm : {1, 2, 3, 5, 7, 8, 14, 21, 33, 42, 44, 61, 85, 100, 143, 170, 209, 341, 342, 512}) {
    FftPlan f;
    if (make_line_plan(nm, kMaxPadded, &f) || f.P < 3 * nm || f.rad[0] * f.span[0] > 0xffff) { std::printf("PLAN %d\n", nm); ++bad; continue; }
    plans.push_back(f);
    if (make_fft_plan(3 * nm, &f)) ++bad;
    bool wide = false;  // radices 11-31 of prime-factor plans run on the tensor cores
    for (int i = 0; i < f.nrad; ++i) wide = wide || (f.pfa && f.rad[i] > 7);
    if (!wide) plans.push_back(f);
  }
  for (const FftPlan& f : plans) {
    const int P = f.P;
    const Tables t = tables(f);
    auto place = [&](int n) {  // grid point n in the plan's order
      if (!f.pfa) return (int)t.tab[n];
      int at = 0, span = P;
      for (int i = 0; i < f.nrad; ++i) { span /= f.rad[i]; at += (n % f.rad[i]) * span; }
      return at;
    };
    std::vector<C> w(P);
    for (int k = 0; k < P; ++k) w[k] = std::polar(1.0L, -2 * PI * (L)k / P);
    for (int dif = 0; dif < 2; ++dif)
      for (int mode = 0; mode < 3; ++mode) {
        std::vector<longlong2> b(f.rad[0] * f.span[0]);
        std::vector<C> z(P);
        for (int k = 0; k < P; ++k) {
          long long x = (long long)(rnd() >> 4) - (1LL << 59), y = (long long)(rnd() >> 4) - (1LL << 59);
          if (mode == 1) { x = (rnd() & 1) ? (1LL << 60) - 1 : 1 - (1LL << 60); y = (rnd() & 1) ? (1LL << 60) - 1 : 1 - (1LL << 60); }
          if (mode == 2 && k != P / 3) x = y = 0;
          b[dif ? place(k) : (int)t.pos[k]] = fx_make(x, y);
          z[k] = C((L)x, (L)y);
        }
        int E = 0, bits = 60, m = dif ? P : 1;
        for (int i = 0; i < f.nrad; ++i) {
          const int s = dif ? i : f.nrad - 1 - i, p = f.rad[s], d = bits + fx_growth(p) - 61;
          if (dif) m /= p;
          FxMax o{0, 0};
          stage(f, t, s, b.data(), m, dif, d, o);
          if (!dif) m *= p;
          E += d;
          bits = fx_bits(o.x | o.y);
          if (bits > 61) { std::printf("RANGE %d %d\n", P, bits); ++bad; }
        }
        L err = 0, nrm = 0;
        for (int n = 0; n < P; ++n) {
          C ref = 0;
          for (int k = 0; k < P; ++k) ref += z[k] * w[(long long)k * n % P];
          const longlong2 v = b[dif ? (int)t.pos[n] : place(n)];
          err += std::norm(C((L)v.x, (L)v.y) * ldexpl(1.0L, E) - ref);
          nrm += std::norm(ref);
        }
        const double e = (double)sqrtl(err / nrm);
        worst = std::max(worst, e);
        ++checked;
        if (!(e < 0x1p-52 * 0.83)) { std::printf("ERR P %d pfa %d dif %d mode %d: %g\n", P, f.pfa, dif, mode, e); ++bad; }
      }
  }
  for (int i = 0; i < 200000; ++i) {  // grid products: within 2 units; conversions: exact
    const long long a = (long long)rnd() >> (2 + rnd() % 40), b = (long long)rnd() >> (2 + rnd() % 40);
    const __int128 ab = (__int128)a * b;
    const L off = (L)fx_mulhi(a, b) - (L)(double)0 - ldexpl((L)(long long)(ab >> 64), 0) - ldexpl((L)(unsigned long long)ab, -64);
    if (fabsl(off) > 2) { std::printf("MULHI %lld %lld %Lg\n", a, b, off); ++bad; }
    const unsigned long long bits = (rnd() >> 12) | ((1 + rnd() % 2046) << 52);
    double v;
    memcpy(&v, &bits, 8);
    const int top = (int)((bits >> 52) & 0x7ff) + (int)(rnd() % 70);
    const L want = floorl(ldexpl((L)v, 59 - (top - 1022)));
    if ((L)fx_mag_of(bits, top) != want) { std::printf("MAG %a %d\n", v, top); ++bad; }
  }
  std::printf("worst %g\n%d %d\n", worst, checked, bad);
  return 0;
}
'''


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixedfft")
    (d / "h.cpp").write_text("#include <cstring>\n" + HARNESS)
    exe = d / "h"
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(PKG, "csrc"), "-I" + cuda_inc, str(d / "h.cpp"),
                    "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout


def test_fixed_point_transforms_against_the_dft(harness):
    checked, bad = (int(x) for x in harness.strip().splitlines()[-1].split())
    assert bad == 0, harness
    assert checked > 150
