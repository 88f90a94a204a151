"""x^y from the exponent's table (csrc/powtab.hpp) against the C library's long double: accuracy
over the range it serves, and the ends of that range, where x^y overflows or becomes subnormal
and pow takes over.  A host probe compiled here; the device compiles the same function."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cfloat>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "powtab.hpp"
static PowTab t;
// distance from x^y in units of the last place of its double (subnormal ones' is 2^-1074)
static double ulps(double x, double y) {
  const double v = tpow(&t, x);
  const long double r = powl((long double)x, (long double)y);
  const double rd = (double)r;
  if (std::isinf(rd) || v == rd) return v == rd ? 0.0 : 1e300;
  if (!std::isfinite(v)) return 1e300;
  return (double)(fabsl(v - r) / (long double)(std::nextafter(rd, INFINITY) - rd));
}
int main(int, char** argv) {
  const double y = atof(argv[1]);
  if (!pow_table(y, t)) return 2;
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> mant(1.0, 2.0);
  std::uniform_int_distribution<int> near(-8, 7), all(-1022, 1023);
  double a = 0.0, b = 0.0;
  for (int n = 0; n < 400000; n++) a = std::fmax(a, ulps(std::ldexp(mant(g), near(g)), y));
  for (int n = 0; n < 100000; n++) b = std::fmax(b, ulps(std::ldexp(mant(g), all(g)), y));
  // both sides of every power of two, among them each end of the table's range
  for (int k = -1022; k <= 1023; k++)
    for (double x : {std::ldexp(1.0, k), std::nextafter(std::ldexp(1.0, k), 0.0),
                     std::nextafter(std::ldexp(1.0, k), INFINITY), std::ldexp(1.75, k)})
      b = std::fmax(b, ulps(x, y));
  const bool special = tpow(&t, 0.0) == 0.0 && std::isinf(tpow(&t, INFINITY)) &&
                       std::isnan(tpow(&t, NAN)) && std::isfinite(tpow(&t, 4.9e-324));
  std::printf("%.4f %.4f %d\n", a, b, special);
  return 0;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("powtab")
    (d / "probe.cpp").write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "cpfft_gb300", "csrc"), str(d / "probe.cpp"), "-o",
                    str(d / "probe")], check=True, capture_output=True)
    return str(d / "probe")


@pytest.mark.parametrize("y", [0.05, 0.5, 1.5, 2.25, 4.48, 7.5, 7.99, 8.0])
def test_power_table(probe, y):
    r = subprocess.run([probe, repr(y)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    inner, ends, special = r.stdout.split()
    # half an ulp of the last rounding, and its second-order terms: the correction's own roundings
    # (|u| y 2^-53 of the value each, 2^-6 at most) and the series' seventh term (below 2^-58)
    assert float(inner) <= 0.6
    # pow's bound and one unit more where the rounding error of w is itself subnormal
    assert float(ends) <= 2.0
    assert special == "1"


def test_power_table_refuses_other_exponents(tmp_path):
    src = tmp_path / "probe.cpp"
    src.write_text('#include <initializer_list>\n#include "powtab.hpp"\nint main() { static PowTab t; int n = 0;\n'
                   '  for (double y : {0.0, -1.0, 8.0000001, (double)NAN, (double)INFINITY}) n += pow_table(y, t);\n'
                   '  return n; }\n')
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "cpfft_gb300", "csrc"), str(src),
                    "-o", str(tmp_path / "probe")], check=True, capture_output=True)
    assert subprocess.run([str(tmp_path / "probe")]).returncode == 0
