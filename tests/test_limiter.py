"""The FP64 flux limiter of the scalar stage (csrc/elmm_temperature.cuh,
kappa_limiter), its source compiled for the host: the product with 1/3 and its
correction give the quotient by three, and the limiter what it gives with the
division, bit for bit: over random ratios of every magnitude, quotients that
are exact or next to a rounding boundary, and infinities and NaN."""
import os
import subprocess

from conftest import ROOT

HARNESS = r'''
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>
#define __device__
#define __forceinline__ inline
using std::fma; using std::fmax; using std::fmin;
%s
static double plain(double r) { return fmax(0.0, fmin(2.0 * r, fmin(2.0, (1.0 + 2.0 * r) / 3.0))); }
static bool same(double a, double b) { return a == b || (std::isnan(a) && std::isnan(b)); }
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double bits(uint64_t u) { double d; std::memcpy(&d, &u, 8); return d; }
int main() {
  long bad = 0;
  auto check = [&](double r) {
    bad += !same(kappa_limiter<double>(r), plain(r));
    // the quotient alone, where 2 r and 2 would hide it
    const double x = 1.0 + 2.0 * r, q = x * (1.0 / 3.0), t = fma(fma(-3.0, q, x), 1.0 / 3.0, q);
    if (std::isfinite(x)) bad += !same(t, x / 3.0);
  };
  for (int n = 0; n < 4000000; n++) {
    check(bits((rnd() & 0x000fffffffffffffull) | ((uint64_t)(1023 - 60 + rnd() %% 1000) << 52) | (rnd() << 63)));  // any size
    check((double)(int64_t)(rnd() >> 12) * 0x1p-51 - 1.0);                                                 // [-1, 1)
    const double q = bits((rnd() & 0x000fffffffffffffull) | (1023ull << 52));                                // 3 q and its neighbours
    check((3 * q - 1) / 2);
    check((std::nextafter(3 * q, 9.0) - 1) / 2);
    check((std::nextafter(3 * q, 0.0) - 1) / 2);
  }
  const double inf = std::numeric_limits<double>::infinity();
  for (double r : {0.0, -0.0, -0.5, 0.25, 1.0, 2.5, inf, -inf, std::nan(""), 1e308, -1e308, 1e-320})
    bad += !same(kappa_limiter<double>(r), plain(r));
  printf("%%ld\n", bad);
  return bad != 0;
}
'''


def test_limiter_rounds_as_the_division(tmp_path):
    text = open(os.path.join(ROOT, "gpu_elmm_b200", "csrc", "elmm_temperature.cuh")).read()
    i = text.index("template <typename T>\n__device__ __forceinline__ T kappa_limiter(T r) {")
    src = tmp_path / "limiter.cpp"
    src.write_text(HARNESS % text[i:text.index("\n}\n", i) + 3])
    exe = str(tmp_path / "limiter")
    subprocess.run(["g++", "-O2", "-march=native", "-ffp-contract=off", "-std=c++17", str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
