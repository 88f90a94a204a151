// prefault.hpp -- pages of the caller's large output buffers, prepared while the GPU works.
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <initializer_list>
#include <thread>
#include <utility>
#include <vector>

// Pages of large host output buffers made present by helper threads while the GPU works: a
// device-to-host copy into untouched pages faults them one by one (151 MB: 5.5 ms against
// 0.8 ms into present pages; two to four threads prepare them in 1.8 ms).  Contents are
// kept; a buffer the call cannot prepare is left to the copy, and so is one whose pages are
// there already (a host that hands over the same array every step, or a pinned one): starting
// the threads for it took the FP64 operator at 64^3 from 0.64 to 0.69 ms.
class Prefault {
  std::vector<std::thread> th_;

  // eight pages spread over [a0, a1), its first and last among them, are all present
  static bool present(size_t a0, size_t a1, size_t page) {
    const size_t n = (a1 - a0) / page, samples = 8;
    for (size_t k = 0; k < samples; k++) {
      unsigned char here = 0;
      if (mincore((void*)(a0 + (n - 1) * k / (samples - 1) * page), page, &here) != 0 || !(here & 1))
        return false;
    }
    return true;
  }

 public:
  Prefault(std::initializer_list<std::pair<void*, size_t>> bufs) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    for (const auto& b : bufs) {
      const size_t a0 = ((size_t)b.first + page - 1) / page * page;
      const size_t a1 = ((size_t)b.first + b.second) / page * page;
      if (!b.first || a1 < a0 + (4u << 20)) continue;  // whole pages: less than a share for one thread
      if (present(a0, a1, page)) continue;
      const size_t nt = std::min<size_t>(4, (a1 - a0) >> 22), part = (a1 - a0) / (nt * page) * page;
      for (size_t k = 0; k < nt && part; k++) {
        const size_t p0 = a0 + k * part, p1 = k + 1 == nt ? a1 : p0 + part;
        try {
          th_.emplace_back([p0, p1] { madvise((void*)p0, p1 - p0, 23 /* MADV_POPULATE_WRITE */); });
        } catch (...) {  // no thread to be had: the copy faults the pages itself
          return;
        }
      }
    }
  }
  void join() {
    for (auto& t : th_) t.join();
    th_.clear();
  }
  size_t threads() const { return th_.size(); }
  ~Prefault() { join(); }
};
