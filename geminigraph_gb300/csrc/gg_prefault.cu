// Pages of a caller's result arrays, made ready while the device works.
#include <sys/mman.h>
#include <unistd.h>

#include <thread>

#include "gg_common.cuh"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14; older kernels refuse it and nothing changes
#endif

namespace gg {

// Below SMALL an array comes from the allocator's own heap as a rule, whose
// pages are there; up to INLINE the pages take the calling thread 31 us a MB
// (a thread would cost 50 - 80 us); above, up to THREADS threads share them:
// 154 MB take 4.7 / 2.6 / 1.8 / 3.2 ms with 1 / 2 / 4 / 8 threads.
constexpr size_t SMALL = 64 << 10, INLINE = 1 << 20, PER_THREAD = 2 << 20;
constexpr int THREADS = 4, SAMPLES = 9;

static size_t page_size() {
  static const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  return page;
}

// Whether the range's pages are there, by SAMPLES of them: an array that the
// allocator hands out again needs no thread (35 us of a call that takes 500
// us).  A wrong answer either way costs time only.
static bool present(const Prefault::Range &r) {
  if (!r.p || !r.n) return true;
  for (int i = 0; i < SAMPLES; i++) {
    unsigned char in = 0;
    const uintptr_t at = ((uintptr_t)r.p + (r.n - 1) / (SAMPLES - 1) * i) / page_size() * page_size();
    if (mincore((void *)at, 1, &in) != 0 || !(in & 1)) return false;
  }
  return true;
}

static void populate(const Prefault::Range &r, int part, int parts) {
  if (!r.p || !r.n) return;
  const size_t page = page_size();
  const uintptr_t base = (uintptr_t)r.p;
  const uintptr_t lo = (base + r.n / parts * part) / page * page;
  const uintptr_t hi = part + 1 == parts ? base + r.n : base + r.n / parts * (part + 1);
  // a refusal (an older kernel, pinned or foreign memory) is no error: the
  // copy that follows does what it did
  (void)madvise((void *)lo, hi - lo, MADV_POPULATE_WRITE);
}

Prefault::Prefault(void *a, size_t na, void *b, size_t nb) {
  const Range r0{a, a ? na : 0}, r1{b, b ? nb : 0};
  const size_t total = r0.n + r1.n;
  if (total < SMALL || (present(r0) && present(r1))) return;
  auto share = [r0, r1](int part, int parts) {
    populate(r0, part, parts);
    populate(r1, part, parts);
  };
  if (total <= INLINE) {
    share(0, 1);
    return;
  }
  const int parts = total / PER_THREAD >= THREADS ? THREADS : total / PER_THREAD < 1 ? 1 : (int)(total / PER_THREAD);
  try {
    // the first thread starts the others, so that the caller goes on to its launches
    main_ = std::thread([share, parts] {
      std::thread more[THREADS];
      int i = 1;
      try {
        for (; i < parts; i++) more[i] = std::thread(share, i, parts);
      } catch (...) {  // no more threads: their shares are this one's
      }
      share(0, parts);
      for (int j = i; j < parts; j++) share(j, parts);
      for (int j = 1; j < i; j++) more[j].join();
    });
  } catch (...) {  // no thread: the copy finds the pages as they are
  }
}

void Prefault::wait() {
  if (main_.joinable()) main_.join();
}

}  // namespace gg
