// Host memory that a copy from the device is about to fill.
#pragma once
#include <cstddef>

namespace eif {

// Makes every page of [p, p + bytes) resident and writable without changing it: one byte of every
// 4 KB is written back as it is, in one atomic operation (a plain read would first map the zero
// page, and a store of its own could undo another thread's write). By 4 KB whatever the system's
// page size: a virtual machine's larger pages may lie on smaller ones of its host (steps of the
// 64 KB that sysconf gives: 6.7 ms for a run of 384 x 768 that is averaged, 4.6 with these).
inline void fault_in_pages(void *p, size_t bytes) {
  unsigned char *q = static_cast<unsigned char *>(p);
  for (size_t k = 0; k < bytes; k += 4096) __atomic_fetch_or(q + k, (unsigned char)0, __ATOMIC_RELAXED);
  if (bytes) __atomic_fetch_or(q + bytes - 1, (unsigned char)0, __ATOMIC_RELAXED);
}

}  // namespace eif
