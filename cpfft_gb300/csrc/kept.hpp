// kept.hpp -- a device table that its owner keeps from its first use on.
#pragma once

// Fills `slot` on the first call: `alloc(p)` allocates the table, `fill(p)` uploads it and waits.
// The slot takes the table only then; after a failure (non-zero return) it stays empty, so that the
// next call makes the table again instead of reading one that was never written.
template <typename T, typename Alloc, typename Fill, typename Release>
int keep_filled(T*& slot, Alloc&& alloc, Fill&& fill, Release&& release) {
  if (slot) return 0;
  T* p = nullptr;
  int rc = alloc(p);
  if (rc) return rc;
  if ((rc = fill(p))) {
    release(p);
    return rc;
  }
  slot = p;
  return 0;
}
