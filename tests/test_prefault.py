"""Page preparation of the caller's output buffers (csrc/prefault.hpp): every size and alignment
around its 4 MiB threshold, and buffers handed over again, whose pages are there already.  Host
probes compiled here with the division checks of -fsanitize=undefined."""
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


REUSE = r"""
#include <cstdio>
#include <cstring>
#include "prefault.hpp"
static char* map(size_t len) {
  return (char*)mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
}
int main() {
  const size_t len = 24u << 20;
  char* m = map(len);
  size_t t[5];
  { Prefault pf({{m, len}}); t[0] = pf.threads(); }          // untouched pages: prepared
  { Prefault pf({{m, len}}); t[1] = pf.threads(); }          // handed over again
  char* h = map(len);
  std::memset(h, 1, len / 2);
  { Prefault pf({{h, len}}); t[2] = pf.threads(); }          // the second half is missing
  char* e = map(len);
  std::memset(e, 1, len - (2u << 20));
  { Prefault pf({{e, len}}); t[3] = pf.threads(); }          // only the end is missing
  { Prefault pf({{m + 9, len - 9}, {h, len}}); t[4] = pf.threads(); }
  std::printf("%zu %zu %zu %zu %zu\n", t[0], t[1], t[2], t[3], t[4]);
  return 0;
}
"""


def run(tmp_path, source):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined",
                    "-fsanitize-undefined-trap-on-error", "-pthread",
                    "-I", os.path.join(ROOT, "cpfft_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)
    return r.stdout.split()


def test_prefault_sizes_and_alignments(tmp_path):
    assert run(tmp_path, PROBE) == ["65"]


def test_prefault_leaves_present_pages_alone(tmp_path):
    assert run(tmp_path, REUSE) == ["4", "0", "4", "4", "0"]
