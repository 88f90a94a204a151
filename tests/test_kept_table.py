"""Device tables kept from their first use (csrc/kept.hpp, f2disp's cosine table): a table whose
allocation or upload fails isn't kept, and the next call makes it again.  A host probe with fakes
of the failing calls."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "kept.hpp"
static int allocs, fills, frees;
static double mem[4];
int main() {
  double* slot = nullptr;
  auto call = [&](int alloc_rc, int fill_rc) {
    return keep_filled(slot, [&](double*& p) { allocs++; if (!alloc_rc) p = mem; return alloc_rc; },
                       [&](double* p) { fills++; if (!fill_rc) p[0] = 42.0; return fill_rc; },
                       [&](double* p) { frees += p == mem; });
  };
  const int a = call(-4, 0), none_a = slot == nullptr;   // no memory
  const int b = call(0, -3), none_b = slot == nullptr;   // the upload fails
  const int c = call(0, 0), kept = slot == mem && mem[0] == 42.0;
  const int d = call(-9, -9);                            // there already: nothing is called
  std::printf("%d %d %d %d %d %d %d %d %d %d\n", a, none_a, b, none_b, c, kept, d, allocs, fills, frees);
}
"""


def test_kept_table(tmp_path):
    (tmp_path / "probe.cpp").write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "cpfft_gb300", "csrc"),
                    str(tmp_path / "probe.cpp"), "-o", str(tmp_path / "probe")], check=True)
    r = subprocess.run([str(tmp_path / "probe")], capture_output=True, text=True)
    assert r.stdout.split() == ["-4", "1", "-3", "1", "0", "1", "0", "3", "2", "1"]
