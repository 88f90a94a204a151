"""Page preparation of the caller's output buffers (csrc/prefault.hpp) at every size and
alignment around its 4 MiB threshold: a host probe compiled here with the division checks of
-fsanitize=undefined."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include <cstring>
#include "prefault.hpp"
int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), M4 = 4u << 20, len = 24u << 20;
  const size_t sizes[] = {0, 1, page, M4 - 1, M4, M4 + 1, M4 + page - 1, M4 + page, M4 + 2 * page,
                          2 * M4 - 1, 2 * M4, 2 * M4 + 3, 17u << 20};
  const size_t offsets[] = {0, 1, 8, page - 8, page - 1};
  Prefault none({{nullptr, 64u << 20}});
  none.join();
  int n = 0;
  for (size_t size : sizes)
    for (size_t off : offsets) {
      char* m = (char*)mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
      if (m == MAP_FAILED) return 2;
      char* b = m + off;
      if (size) { b[0] = 7; b[size - 1] = 9; }
      {
        Prefault pf({{b, size}});
        pf.join();
        pf.join();
      }
      if (size && (b[size - 1] != 9 || (size > 1 && b[0] != 7))) return 3;  // contents are kept
      for (size_t i = 1; i + 1 < size; i += page / 2)
        if (b[i] != 0) return 4;
      munmap(m, len);
      n++;
    }
  std::printf("%d\n", n);
  return 0;
}
"""


def test_prefault_sizes_and_alignments(tmp_path):
    src = tmp_path / "probe.cpp"
    src.write_text(PROBE)
    exe = tmp_path / "probe"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined",
                    "-fsanitize-undefined-trap-on-error", "-pthread",
                    "-I", os.path.join(ROOT, "cpfft_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "65", (r.returncode, r.stdout)
