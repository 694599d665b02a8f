// afl_host.h -- host memory of the downloads.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <exception>
#include <thread>

#include <sys/mman.h>
#include <unistd.h>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace afl {

// Faults in the pages of a buffer that a device-to-host copy is about to fill.
// A caller's fresh buffer has none, and the copy takes the faults one by one in
// its own thread: a 128^3 field (16.8 MB) took 4.9 ms into a fresh buffer and
// 0.9 ms into a used one, a 256^3 field 28-35 and 7 ms.  Asking the kernel for
// whole ranges first (MADV_POPULATE_WRITE, which keeps their contents) makes that
// 3.2 and 12-14 ms.  Two threads from 8 MB and four from 64 MB: on recycled
// memory they take 0.5 and 3.3 ms of it, eight 1.0 and 8.6 ms.  Below 256 KB a
// few faults are cheaper than the call.  Buffers whose sampled pages are present
// are left alone.  Only speed depends on any of this: errors (an older kernel, a
// mapping that cannot be populated) are ignored.
inline void prefault(void *buf, size_t bytes) {
  if (!buf || bytes < (size_t(256) << 10)) return;
  const uintptr_t page = static_cast<uintptr_t>(sysconf(_SC_PAGESIZE));
  const uintptr_t lo = (reinterpret_cast<uintptr_t>(buf) + page - 1) / page * page;
  const uintptr_t hi = (reinterpret_cast<uintptr_t>(buf) + bytes) / page * page;
  if (hi <= lo) return;
  bool present = true;
  for (int s = 0; s < 8 && present; ++s) {
    const uintptr_t at = lo + (hi - lo - page) / page * s / 7 * page;
    unsigned char v = 0;
    if (mincore(reinterpret_cast<void *>(at), page, &v) != 0) return;
    present = (v & 1) != 0;
  }
  if (present) return;
  const int parts = bytes >= (size_t(64) << 20) ? 4 : bytes >= (size_t(8) << 20) ? 2 : 1;
  const uintptr_t huge = uintptr_t(2) << 20;
  const uintptr_t step = parts == 1 ? hi - lo : ((hi - lo) / parts + huge - 1) / huge * huge;
  auto part = [=](int n) {
    const uintptr_t a = lo + step * n, b = std::min(hi, a + step);
    if (a < b) madvise(reinterpret_cast<void *>(a), b - a, MADV_POPULATE_WRITE);
  };
  std::thread others[3];
  int started = 1;
  try {
    for (; started < parts; ++started) others[started - 1] = std::thread(part, started);
  } catch (const std::exception &) {  // no thread or no memory for one: the copy faults the rest
  }
  part(0);
  for (int n = 1; n < started; ++n) others[n - 1].join();
}

}  // namespace afl
