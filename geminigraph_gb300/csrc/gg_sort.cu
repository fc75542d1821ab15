// Stable LSD radix sort of 64-bit keys with optional 32-bit values: the graph
// build's and the hot-source layout's sort.
//
// Bound: HBM.  A pass reads and writes every key and value once (24 B per
// entry with values), so it is one kernel: the digit counts of all passes
// come from one read of the keys up front (rs_histogram), and a tile learns
// where its digits go by looking back over the tiles before it (each tile
// publishes its counts, then its running totals) instead of from a count
// pass and a scan.  Keys and values are reordered by digit in shared memory
// and leave as runs of consecutive addresses (6144 entries over at most 256
// digits: 24 entries, 192 bytes on average), where a scatter straight from
// registers writes one 8-byte piece per lane.
// Measured on GB300, graph of 134 M weighted records (V 8.4 M), both
// directions: 54.8 ms with a count kernel, a scan and a register scatter per
// pass (3.35 ms a scatter, 960 GB/s), 18.5 ms with these passes (1.13 ms
// each, 2.9 TB/s; the ranking's ballots and block barriers are what is left).
// With the counts taken where the keys are made, and the CSC's from the CSR's
// sort, 18.6 ms for 19.7 on the same box.
// 256 to 1024 threads with 8 to 20 keys each: 18.5 to 22 ms; ranking by
// __match_any_sync: 21.4 ms.
#include "gg_build.cuh"
#include "gg_common.cuh"
#include "gg_scan.cuh"

namespace gg {

constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 12;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
// Polls of one predecessor's word before a tile gives up (about a second):
// tiles are numbered in the order they start and publish their counts before
// they wait, so a wait ends unless a device fault stopped an earlier tile.
constexpr unsigned RS_SPIN = 1u << 20;

// Digit counts of every pass, one read of the keys (a graph build's are taken
// where the keys are made).
__global__ void __launch_bounds__(RS_THREADS)
    rs_histogram(const uint64_t *__restrict__ keys, size_t n, RsPlan plan, uint32_t *__restrict__ hist) {
  __shared__ RsCounters h;
  rs_count_begin(h);
  for (size_t i = (size_t)blockIdx.x * RS_THREADS + threadIdx.x; i < n; i += (size_t)gridDim.x * RS_THREADS)
    rs_count(h, plan, keys[i]);
  rs_count_end(h, plan, hist);
}

// hist[p][d] -> the position where digit d of pass p starts.
__global__ void __launch_bounds__(SCAN_THREADS) rs_bases(uint32_t *hist, int passes) {
  for (int p = 0; p < passes; p++) {
    uint32_t excl;
    const uint32_t x = hist[p * RS_BINS + threadIdx.x];
    block_exclusive_scan<uint32_t>(x, &excl);
    hist[p * RS_BINS + threadIdx.x] = excl;
  }
}

// The look-back word of (tile, digit): the count in the upper 56 bits, in the
// lower 8 bits 2 * pass + 1 (the tile's own count) or 2 * pass + 2 (the
// count of this and all earlier tiles); other tags are words of earlier passes.
__device__ __forceinline__ unsigned long long rs_peek(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void rs_publish(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <bool VALS>
constexpr size_t rs_smem() {
  return sizeof(uint64_t) * RS_TILE + (VALS ? sizeof(uint32_t) * RS_TILE : 0);
}

// One pass.  Warp w ranks keys [w * 384, +384) of the tile in order (round
// r, lane): lanes of equal digit find each other by one ballot per digit
// bit, and a warp-private count (in the space the reordered keys take later)
// holds the rounds before.  Keys past n are all ones and rank last.
template <bool VALS>
__global__ void __launch_bounds__(RS_THREADS, 2)
    rs_pass(const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint64_t *__restrict__ kout,
            uint32_t *__restrict__ vout, size_t n, int pass, int shift, int bits, const uint32_t *__restrict__ base,
            unsigned long long *look, unsigned *ticket, unsigned *err) {
  extern __shared__ uint64_t s_keys[];
  uint32_t *s_vals = reinterpret_cast<uint32_t *>(s_keys + RS_TILE);
  uint32_t(*whist)[RS_BINS] = reinterpret_cast<uint32_t(*)[RS_BINS]>(s_keys);
  __shared__ uint32_t s_excl[RS_BINS], s_out[RS_BINS];
  __shared__ uint32_t s_scan[RS_BINS / 32];
  __shared__ uint32_t s_tile, s_bad;
  const unsigned w = threadIdx.x >> 5, lane = lane_id();
  if (threadIdx.x == 0) {
    s_tile = atomicAdd(ticket, 1u);
    s_bad = 0;
  }
  for (int i = threadIdx.x; i < RS_WARPS * RS_BINS; i += RS_THREADS) (&whist[0][0])[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const size_t tile0 = (size_t)tile * RS_TILE;
  const uint32_t tile_n = n - tile0 < RS_TILE ? (uint32_t)(n - tile0) : RS_TILE;
  const uint32_t mine = w * (32 * RS_ITEMS) + lane;
  const uint32_t mask = (1u << bits) - 1u;
  uint64_t key[RS_ITEMS];
  uint32_t rank[RS_ITEMS];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; r++) key[r] = mine + 32 * r < tile_n ? kin[tile0 + mine + 32 * r] : ~0ull;
#pragma unroll
  for (int r = 0; r < RS_ITEMS; r++) {
    const uint32_t d = (uint32_t)(key[r] >> shift) & mask;
    unsigned peers = GG_FULL;
#pragma unroll
    for (int b = 0; b < 8; b++) {
      if (b >= bits) break;
      const unsigned one = __ballot_sync(GG_FULL, (d >> b) & 1u);
      peers &= (d >> b) & 1u ? one : ~one;
    }
    const uint32_t before = whist[w][d];
    __syncwarp();
    if (lane == (unsigned)(__ffs(peers) - 1)) whist[w][d] = before + __popc(peers);
    __syncwarp();
    rank[r] = before + __popc(peers & lanemask_lt());
  }
  __syncthreads();
  // thread d: counts of digit d before each warp, the tile's count, its place
  uint32_t total = 0;
  if (threadIdx.x < RS_BINS) {
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ww++) {
      const uint32_t t = whist[ww][threadIdx.x];
      whist[ww][threadIdx.x] = total;
      total += t;
    }
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(GG_FULL, incl, o);
      if (lane >= (unsigned)o) incl += y;
    }
    if (lane == 31) s_scan[w] = incl;
    s_excl[threadIdx.x] = incl - total;
    if (threadIdx.x == mask) total -= RS_TILE - tile_n;  // the keys past n
    const unsigned long long tag = 2 * pass + (tile == 0 ? 2 : 1);
    rs_publish(look + (size_t)tile * RS_BINS + threadIdx.x, ((unsigned long long)total << 8) | tag);
  }
  __syncthreads();
  if (threadIdx.x < RS_BINS) {
    uint32_t lower = 0;
    for (unsigned i = 0; i < w; i++) lower += s_scan[i];
    s_excl[threadIdx.x] += lower;
  }
  __syncthreads();
  uint32_t val[VALS ? RS_ITEMS : 1];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; r++) {
    if (VALS) val[r] = mine + 32 * r < tile_n ? vin[tile0 + mine + 32 * r] : 0u;
    const uint32_t d = (uint32_t)(key[r] >> shift) & mask;
    rank[r] += s_excl[d] + whist[w][d];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_ITEMS; r++) {
    s_keys[rank[r]] = key[r];
    if (VALS) s_vals[rank[r]] = val[r];
  }
  // digit d of the earlier tiles
  if (threadIdx.x < RS_BINS) {
    unsigned long long sum = 0;
    bool bad = false;
    for (uint32_t t = tile; t-- > 0 && !bad;) {
      const unsigned long long *p = look + (size_t)t * RS_BINS + threadIdx.x;
      unsigned long long v = rs_peek(p);
      for (unsigned spin = 0; (v & 255u) != 2 * pass + 1 && (v & 255u) != 2 * pass + 2; v = rs_peek(p))
        if (++spin > RS_SPIN) {
          bad = true;
          break;
        }
      sum += v >> 8;
      if ((v & 255u) == 2 * pass + 2) break;
    }
    if (tile > 0)
      rs_publish(look + (size_t)tile * RS_BINS + threadIdx.x, ((sum + total) << 8) | (2 * pass + 2));
    if (bad) s_bad = 1;
    // entry i of the reordered tile goes to s_out[its digit] + i
    s_out[threadIdx.x] = base[threadIdx.x] + (uint32_t)sum - s_excl[threadIdx.x];
  }
  __syncthreads();
  if (s_bad) {
    if (threadIdx.x == 0) atomicOr(err, 1u);
    return;
  }
  for (uint32_t i = threadIdx.x; i < tile_n; i += RS_THREADS) {
    const uint64_t k = s_keys[i];
    const uint32_t at = s_out[(uint32_t)(k >> shift) & mask] + i;
    if (at < n) {
      kout[at] = k;
      if (VALS) vout[at] = s_vals[i];
    }
  }
}

static size_t rs_tiles(size_t n) { return (n + RS_TILE - 1) / RS_TILE; }
// Head of the scratch: digit counts of every pass, a ticket per pass, the error word.
constexpr size_t RS_HEAD = sizeof(uint32_t) * (RS_MAX_PASSES * RS_BINS + RS_MAX_PASSES + 8);
static_assert(RS_HEAD % 16 == 0, "the look-back words follow the head");
size_t radix_scratch_bytes(size_t n) { return RS_HEAD + sizeof(unsigned long long) * RS_BINS * rs_tiles(n); }

int radix_clear(gg_graph *g, void *scratch, size_t n) {
  GG_CUDA(cudaMemsetAsync(scratch, 0, radix_scratch_bytes(n), g->stream));
  return GG_OK;
}

int radix_sort(gg_graph *g, void *scratch, uint64_t *k0, uint64_t *k1, const SortValues &v, size_t n, int lo_bit,
               int hi_bit, uint64_t **kres, uint32_t **vres, RsCounts have) {
  *kres = k0;
  *vres = v.in;
  if (n > 1 && rs_passes(hi_bit - lo_bit) > RS_MAX_PASSES) {
    set_error("radix sort of %d key bits", hi_bit - lo_bit);
    return GG_ERR_INVALID;
  }
  RsPlan plan = rs_plan(lo_bit, hi_bit);
  if (n <= 1) plan.passes = 0;
  if (plan.passes == 0) {
    if (v.in && v.last && n) {
      GG_CUDA(cudaMemcpyAsync(v.last, v.in, sizeof(uint32_t) * n, cudaMemcpyDefault, g->stream));
      *vres = v.last;
    }
    return GG_OK;
  }
  uint32_t *hist = (uint32_t *)scratch;
  unsigned *ticket = hist + RS_MAX_PASSES * RS_BINS;
  unsigned *err = ticket + RS_MAX_PASSES;
  unsigned long long *look = (unsigned long long *)((char *)scratch + RS_HEAD);
  const size_t tiles = rs_tiles(n);
  if (have == RS_PLACED) {
    GG_CUDA(cudaMemsetAsync(ticket, 0, radix_scratch_bytes(n) - ((char *)ticket - (char *)scratch), g->stream));
  } else {
    if (have == RS_NONE) {
      GG_TRY(radix_clear(g, scratch, n));
      rs_histogram<<<grid_for(n, RS_THREADS, g->num_sms, 4), RS_THREADS, 0, g->stream>>>(k0, n, plan, hist);
    }
    rs_bases<<<1, SCAN_THREADS, 0, g->stream>>>(hist, plan.passes);
  }
  GG_CUDA(cudaGetLastError());
  if (v.in)
    GG_CUDA(cudaFuncSetAttribute(rs_pass<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rs_smem<true>()));
  else
    GG_CUDA(cudaFuncSetAttribute(rs_pass<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rs_smem<false>()));
  uint64_t *ka = k0, *kb = k1;
  uint32_t *va = v.in;
  for (int p = 0; p < plan.passes; p++) {
    if (v.in) {
      uint32_t *vb = v.last && p == plan.passes - 1 ? v.last : va == v.b1 ? v.b0 : v.b1;
      rs_pass<true><<<(unsigned)tiles, RS_THREADS, rs_smem<true>(), g->stream>>>(
          ka, va, kb, vb, n, p, plan.shift[p], plan.bits[p], hist + p * RS_BINS, look, ticket + p, err);
      va = vb;
    } else {
      rs_pass<false><<<(unsigned)tiles, RS_THREADS, rs_smem<false>(), g->stream>>>(
          ka, nullptr, kb, nullptr, n, p, plan.shift[p], plan.bits[p], hist + p * RS_BINS, look, ticket + p, err);
    }
    GG_CUDA(cudaGetLastError());
    uint64_t *tk = ka;
    ka = kb;
    kb = tk;
  }
  unsigned bad = 0;
  GG_CUDA(cudaMemcpyAsync(&bad, err, sizeof(bad), cudaMemcpyDeviceToHost, g->stream));
  GG_CUDA(cudaStreamSynchronize(g->stream));
  if (bad) {
    set_error("radix sort: a tile waited too long for an earlier one");
    return GG_ERR_CUDA;
  }
  *kres = ka;
  *vres = va;
  return GG_OK;
}

}  // namespace gg
