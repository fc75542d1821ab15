// Graph build internals shared by the in-core build (gg_store.cu) and the
// partitioned build (gg_partition.cu).  Not part of the C ABI.
#ifndef GG_BUILD_CUH
#define GG_BUILD_CUH

#include <vector>

#include "gg_common.cuh"

namespace gg {

// Bits of the largest vertex id (at least 1): keys pack (major << b) | minor.
int bits_for(uint32_t V);

// The 32-bit values of a sort: read from `in` (null: keys only), moved
// between b0 and b1 (b0 may be `in`; `in` is only read when it is neither),
// the last pass writing to `last` when it is set.
struct SortValues {
  uint32_t *in = nullptr, *b0 = nullptr, *b1 = nullptr, *last = nullptr;
};

// The digits of a sort on key bits [lo_bit, hi_bit): of about equal width, at
// most 8 bits, so no pass sorts on a narrow remainder.  Where the two halves
// of the bits take as many passes apart as together, no digit spans them.
constexpr int RS_THREADS = 512;
constexpr int RS_BINS = 256;
constexpr int RS_MAX_PASSES = 8;
struct RsPlan {
  int passes;
  int shift[RS_MAX_PASSES];
  int bits[RS_MAX_PASSES];
  uint32_t mask[RS_MAX_PASSES];
};
inline int rs_passes(int bits) { return (bits + 7) / 8; }
inline bool rs_halves(int bits) { return bits % 2 == 0 && 2 * rs_passes(bits / 2) == rs_passes(bits); }
inline RsPlan rs_plan(int lo_bit, int hi_bit) {
  RsPlan p;
  p.passes = 0;
  const int halves = rs_halves(hi_bit - lo_bit) ? 2 : 1, width = (hi_bit - lo_bit) / halves;
  for (int h = 0; h < halves; h++)
    for (int i = 0, n = rs_passes(width), at = h * width; i < n && p.passes < RS_MAX_PASSES; i++) {
      const int bits = ((h + 1) * width - at + n - i - 1) / (n - i);
      p.shift[p.passes] = lo_bit + at;
      p.mask[p.passes] = (1u << bits) - 1u;
      p.bits[p.passes++] = bits;
      at += bits;
    }
  return p;
}

// Whether the first digits of b's sort are a's.
inline bool rs_leads(const RsPlan &a, const RsPlan &b) {
  bool same = a.passes <= b.passes;
  for (int p = 0; same && p < a.passes; p++) same = a.shift[p] == b.shift[p] && a.bits[p] == b.bits[p];
  return same;
}

// Digit counts of every pass while the keys are at hand, per block in shared
// memory (all RS_THREADS threads call rs_count_begin and _end).  The passes are
// unrolled, so that shifts and masks are operands from the constant bank: read
// by index, one pass's after the other's, they took 0.61 ms for 134 M keys of
// 46 bits, and 1.25 ms in the kernel that makes the keys (0.51 without
// counting); unrolled, 0.57 there.  Two copies of the counters by lane are no
// faster, 4 and 8 slower (0.86).
typedef uint32_t RsCounters[RS_MAX_PASSES][RS_BINS];
__device__ __forceinline__ void rs_count_begin(RsCounters &h) {
  for (int i = threadIdx.x; i < RS_MAX_PASSES * RS_BINS; i += RS_THREADS) (&h[0][0])[i] = 0;
  __syncthreads();
}
__device__ __forceinline__ void rs_count(RsCounters &h, const RsPlan &plan, uint64_t k) {
#pragma unroll
  for (int p = 0; p < RS_MAX_PASSES; p++)
    if (p < plan.passes) atomicAdd(&h[p][(uint32_t)(k >> plan.shift[p]) & plan.mask[p]], 1u);
}
__device__ __forceinline__ void rs_count_end(const RsCounters &h, const RsPlan &plan, uint32_t *hist) {
  __syncthreads();
  for (int i = threadIdx.x; i < plan.passes * RS_BINS; i += RS_THREADS)
    if ((&h[0][0])[i]) atomicAdd(hist + i, (&h[0][0])[i]);
}

// What the head of a sort's scratch holds: nothing yet; the digit counts of
// rs_plan(lo_bit, hi_bit) (added to scratch after radix_clear); or the places
// that an earlier sort of the same keys made for its first passes, which are
// this one's (rs_leads).
enum RsCounts { RS_NONE, RS_COUNTED, RS_PLACED };
int radix_clear(gg_graph *g, void *scratch, size_t n);

// Stable LSD radix sort of n < 2^32 keys (and values) on the key bits
// [lo_bit, hi_bit), ping-ponging the keys between k0 (the input) and k1;
// *kres / *vres name the buffers holding the result.  scratch: device memory
// of radix_scratch_bytes(n), 16-byte aligned.  Waits for the stream.
size_t radix_scratch_bytes(size_t n);
int radix_sort(gg_graph *g, void *scratch, uint64_t *k0, uint64_t *k1, const SortValues &v, size_t n, int lo_bit,
               int hi_bit, uint64_t **kres, uint32_t **vres, RsCounts have = RS_NONE);

// Neighbour / weight storage in device memory, or in mapped pinned host memory.
int adj_alloc(gg_graph *g, bool host, void **p, size_t bytes);

// Degrees, the deg > 0 bitmap and the bins of a direction whose offsets are written.
int finish_dir(gg_graph *g, Dir *d);

// The in-core build from E records in device memory.
int build_from_device_records(gg_graph *g, const uint32_t *rec, uint64_t E);

// Largest force_partitions the build options accept.
constexpr int32_t OC_MAX_FORCED = 256;

// In-core or partitioned, and for the partitioned build its range and group
// capacities (entries), from the device-memory budget.
int build_plan(gg_graph *g, uint64_t E, bool rec_on_device, const gg_build_options *opt, bool *partitioned,
               uint64_t *cap, uint64_t *gcap);

// Builds both directions from E records readable by the device at rec.
int build_records(gg_graph *g, const uint32_t *rec, uint64_t E, bool partitioned, uint64_t cap, uint64_t gcap,
                  gg_build_options *opt);

// Device buffers freed together when the build returns.
struct DevScratch {
  std::vector<void *> p;
  DevScratch() = default;
  DevScratch(const DevScratch &) = delete;
  DevScratch &operator=(const DevScratch &) = delete;
  ~DevScratch() {
    for (void *q : p) cudaFree(q);
  }
  // The sort buffers of n entries in one allocation (a cudaMalloc and its
  // cudaFree cost about 0.15 ms together at these sizes).
  int sort_buffers(size_t n, bool values, uint64_t **k0, uint64_t **k1, uint32_t **v0, uint32_t **v1, void **scratch) {
    const size_t keys = (sizeof(uint64_t) * n + 255) / 256 * 256;
    const size_t vals = values ? (sizeof(uint32_t) * n + 255) / 256 * 256 : 0;
    char *q = nullptr;
    GG_TRY(get(&q, 2 * keys + 2 * vals + radix_scratch_bytes(n)));
    *k0 = (uint64_t *)q;
    *k1 = (uint64_t *)(q + keys);
    *v0 = values ? (uint32_t *)(q + 2 * keys) : nullptr;
    *v1 = values ? (uint32_t *)(q + 2 * keys + vals) : nullptr;
    *scratch = q + 2 * keys + 2 * vals;
    return GG_OK;
  }
  template <typename T>
  int get(T **out, size_t count) {
    void *q = nullptr;
    GG_CUDA(cudaMalloc(&q, count ? count * sizeof(T) : 16));
    p.push_back(q);
    *out = (T *)q;
    return GG_OK;
  }
};

}  // namespace gg

#endif
