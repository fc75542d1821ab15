// Graph store: edge list -> CSR (out) + CSC (in) on the device.
//
// Replaces Graph::load_directed (core/graph.hpp:771-1339) and
// Graph::load_undirected_from_directed (core/graph.hpp:349-757).  The
// reference makes five passes over the file with MPI self-shuffles and racing
// fetch_add fills; here the CSR is one stable LSD radix sort of packed 64-bit
// (src << b | dst) keys on the device (b = bits of V-1), the CSC a stable sort
// of the CSR's order on dst alone, each followed by a boundary pass that
// writes the offsets.  Lists come out sorted
// by neighbour id with duplicate edges in record order, so the build is
// deterministic.  Degrees are offset differences; symmetric graphs sort the
// records plus their reverses once and alias CSC = CSR (core/graph.hpp:733-738);
// their degree therefore counts both endpoints (core/graph.hpp:393-399).
#include <errno.h>
#include <fcntl.h>
#include <math.h>
#include <stdarg.h>
#include <string.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <chrono>
#include <thread>
#include <vector>

#include "gg_build.cuh"
#include "gg_common.cuh"
#include "gg_gen.h"
#include "gg_scan.cuh"

namespace gg {

// ------------------------------------------------------------------ errors
static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int cuda_status(cudaError_t e, const char *what) {
  set_error("CUDA error %d (%s) in %s", (int)e, cudaGetErrorString(e), what);
  if (e == cudaErrorMemoryAllocation) return GG_ERR_NOMEM;
  return GG_ERR_CUDA;
}

size_t scan_scratch_elems(size_t n) { return scan_scratch_elems_impl(n) + 1; }

// ------------------------------------------------------------------ workspace
int ws_get(gg_graph *g, WsSlot slot, size_t bytes, void **out) {
  Workspace &w = g->ws;
  if (bytes == 0) bytes = 16;
  if (w.bytes[slot] < bytes) {
    if (w.ptr[slot]) GG_CUDA(cudaFree(w.ptr[slot]));
    w.ptr[slot] = nullptr;
    w.bytes[slot] = 0;
    GG_CUDA(cudaMalloc(&w.ptr[slot], bytes));
    w.bytes[slot] = bytes;
  }
  *out = w.ptr[slot];
  return GG_OK;
}

int ws_free_all(gg_graph *g) {
  Workspace &w = g->ws;
  for (int i = 0; i < WS_NSLOTS; i++) {
    if (w.ptr[i]) cudaFree(w.ptr[i]);
    w.ptr[i] = nullptr;
    w.bytes[i] = 0;
  }
  if (w.ctr) cudaFree(w.ctr);
  if (w.ctr_host) cudaFreeHost(w.ctr_host);
  if (w.stage) cudaFreeHost(w.stage);
  w.ctr = nullptr;
  w.ctr_host = nullptr;
  w.stage = nullptr;
  return GG_OK;
}

__global__ void copy_words_to_mapped(const uint32_t *__restrict__ src, uint32_t *dst, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

int read_small(gg_graph *g, void *dst, const void *src, size_t bytes) {
  if (!g->ws.stage || bytes > STAGE_BYTES_HOST || (bytes & 3) || ((uintptr_t)src & 3)) {
    GG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, g->stream));
    GG_CUDA(cudaStreamSynchronize(g->stream));
    return GG_OK;
  }
  copy_words_to_mapped<<<1, 256, 0, g->stream>>>((const uint32_t *)src, (uint32_t *)g->ws.stage, bytes / 4);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaStreamSynchronize(g->stream));
  memcpy(dst, g->ws.stage, bytes);
  return GG_OK;
}

int counters_reset(gg_graph *g) {
  GG_CUDA(cudaMemsetAsync(g->ws.ctr, 0, sizeof(Counters), g->stream));
  return GG_OK;
}

int counters_read(gg_graph *g, Counters *out) { return read_small(g, out, g->ws.ctr, sizeof(Counters)); }

int Trace::reserve_events(size_t n) {
  if (!st || !st->call_ms) return GG_OK;
  while (g->evpool.size() < ev.size() + n) {
    cudaEvent_t e;
    GG_CUDA(cudaEventCreate(&e));
    g->evpool.push_back(e);
  }
  return GG_OK;
}

// Inside a stream capture the record is made an external event node, which
// records the event when the graph runs (so that it can be timed); the flag
// is refused outside a capture.
int Trace::record(cudaEvent_t e) {
  if (capturing)
    GG_CUDA(cudaEventRecordWithFlags(e, g->stream, cudaEventRecordExternal));
  else
    GG_CUDA(cudaEventRecord(e, g->stream));
  return GG_OK;
}

int Trace::kbegin() {
  if (!timing()) return GG_OK;
  GG_TRY(reserve_events(2));
  cudaEvent_t e0 = g->evpool[ev.size()];
  ev.push_back(e0);
  ev_call.push_back(st->calls - 1);
  if (!replay) GG_TRY(record(e0));
  return GG_OK;
}

int Trace::kend() {
  if (!timing() || ev.size() % 2 == 0) return GG_OK;
  cudaEvent_t e1 = g->evpool[ev.size()];
  ev.push_back(e1);
  if (!replay) GG_TRY(record(e1));
  return GG_OK;
}

int Trace::collect() {
  if (!st || !st->call_ms) return GG_OK;
  for (size_t i = 0; i + 1 < ev.size(); i += 2) {
    float ms = 0;
    GG_CUDA(cudaEventSynchronize(ev[i + 1]));
    GG_CUDA(cudaEventElapsedTime(&ms, ev[i], ev[i + 1]));
    st->call_ms[ev_call[i / 2]] += ms;
  }
  ev.clear();
  ev_call.clear();
  return GG_OK;
}

// GG_CHECK builds: the run's bounds checks, read once it has finished.
int check_status(gg_graph *g) {
#if defined(GG_CHECK)
  static const char *const files[] = {"gg_engine.cuh", "gg_common.cuh", "gg_batched.cu", "gg_bc_batched.cu",
                                      "gg_store.cu",   "gg_bfs_pr.cu",  "gg_cc_sssp_bc.cu", "gg_partition.cu"};
  unsigned h[4] = {0, 0, 0, 0};
  GG_CUDA(cudaMemcpy(h, g->check_err, sizeof(h), cudaMemcpyDeviceToHost));
  if (h[0]) {
    const char *file = "?";
    for (const char *f : files)
      if (site_file_hash(f) == (h[0] >> 16)) file = f;
    GG_CUDA(cudaMemset(g->check_err, 0, sizeof(h)));
    set_error("device bounds check failed at %s:%u: index or vertex id %llu out of range (%u failures)", file,
              h[0] & 0xffffu, ((unsigned long long)h[2] << 32) | h[1], h[3]);
    return GG_ERR_CHECK;
  }
#else
  (void)g;
#endif
  return GG_OK;
}

int timed_begin(gg_graph *g) {
  GG_CUDA(cudaEventRecord(g->ev0, g->stream));
  return GG_OK;
}

int timed_end(gg_graph *g, gg_run_stats *st, int launches) {
  GG_CUDA(cudaEventRecord(g->ev1, g->stream));
  GG_CUDA(cudaEventSynchronize(g->ev1));
  return timed_read(g, st, launches);
}

int timed_read(gg_graph *g, gg_run_stats *st, int launches) {
  GG_TRY(check_status(g));
  float ms = 0;
  GG_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
  if (st) {
    st->device_ms = ms;
    st->kernel_launches = launches;
  }
  return GG_OK;
}

// ------------------------------------------------------------------ build kernels
// mode 0: key (src,dst); 2: both (src,dst) and (dst,src), records then reverses.
// The digit counts of their sort on the way: a pass of its own over 134 M keys
// took 0.61 ms beside the 0.51 ms of making them; both 0.57 ms here.
__global__ void __launch_bounds__(RS_THREADS)
    make_keys(const uint32_t *__restrict__ rec, size_t E, int words, int mode, int bits, uint32_t V,
              uint64_t *__restrict__ keys, uint32_t *__restrict__ vals, unsigned *err, RsPlan plan, uint32_t *hist) {
  __shared__ RsCounters h;
  rs_count_begin(h);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t s = rec[i * words], d = rec[i * words + 1];
    uint32_t wb = words == 3 ? rec[i * words + 2] : 0u;
    if (s >= V || d >= V) {
      atomicOr(err, 1u);
      s = 0;
      d = 0;
    }
    uint64_t fwd = ((uint64_t)s << bits) | d, rev = ((uint64_t)d << bits) | s;
    keys[i] = fwd;
    rs_count(h, plan, fwd);
    if (mode == 2) {
      keys[E + i] = rev;
      rs_count(h, plan, rev);
    }
    if (vals) {
      vals[i] = wb;
      if (mode == 2) vals[E + i] = wb;
    }
  }
  rs_count_end(h, plan, hist);
}

// off[v] = first position whose major id is >= v, for v in [0, V], and nbr =
// the minor ids, from n sorted keys.  The major id is a key's upper part
// (low_major: its low `bits` bits; bits above both ids are ignored).  The
// vertices between two keys' majors
// (and after the last) share one offset: up to GAP_INLINE of them are written
// by the key's own thread, longer runs go to the gap list in pieces for
// fill_gaps (a hot-source numbering ends with all vertices without a list: 30
// M of them took one thread 150 ms at R-MAT 26).  A full list falls back to
// the thread.
constexpr uint32_t GAP_INLINE = 64, GAP_PIECE = 1u << 16, GAP_CAP = 1u << 16;
struct Gap {
  uint64_t value, from, to;  // off[from .. to) = value
};
__device__ __forceinline__ void write_gap(uint64_t *off, uint64_t from, uint64_t to, uint64_t value, Gap *gaps,
                                          unsigned *ngaps) {
  if (to - from > GAP_INLINE) {
    const uint32_t pieces = (uint32_t)((to - from + GAP_PIECE - 1) / GAP_PIECE);
    const uint32_t at = atomicAdd(ngaps, pieces);
    if (at < GAP_CAP && GAP_CAP - at >= pieces) {
      for (uint32_t i = 0; i < pieces; i++, from += GAP_PIECE)
        gaps[at + i] = Gap{value, from, from + GAP_PIECE < to ? from + GAP_PIECE : to};
      return;
    }
    for (uint32_t i = at; i < GAP_CAP && i - at < pieces; i++) gaps[i] = Gap{0, 0, 0};
  }
  for (; from < to; from++) off[from] = value;
}
__global__ void offsets_from_keys(const uint64_t *__restrict__ keys, size_t n, int bits, bool low_major, uint32_t V,
                                  uint64_t *__restrict__ off, uint32_t *__restrict__ nbr, Gap *gaps,
                                  unsigned *ngaps) {
  const uint64_t mask = (1ull << bits) - 1;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    const uint64_t low = k & mask, high = (k >> bits) & mask;
    const uint64_t maj = low_major ? low : high;
    nbr[i] = (uint32_t)(low_major ? high : low);
    uint64_t next = 0;  // first vertex without an offset yet
    if (i) next = ((low_major ? keys[i - 1] : keys[i - 1] >> bits) & mask) + 1;
    if (next <= maj) write_gap(off, next, maj + 1, i, gaps, ngaps);
    if (i == n - 1) write_gap(off, maj + 1, (uint64_t)V + 1, n, gaps, ngaps);
  }
}
__global__ void fill_gaps(uint64_t *__restrict__ off, const Gap *__restrict__ gaps, const unsigned *ngaps) {
  const uint32_t n = *ngaps < GAP_CAP ? *ngaps : GAP_CAP;
  for (uint32_t g = blockIdx.x; g < n; g += gridDim.x) {
    const Gap p = gaps[g];
    for (uint64_t v = p.from + threadIdx.x; v < p.to; v += blockDim.x) off[v] = p.value;
  }
}

// Bitmap of the vertices with deg > 0 (one warp per 32-bit word).
__global__ void nonzero_bitmap(const uint32_t *__restrict__ deg, uint32_t V, uint32_t *__restrict__ nz,
                               size_t words) {
  size_t nthreads = words * 32;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nthreads; i += (size_t)gridDim.x * blockDim.x) {
    bool p = i < V && deg[i] > 0;
    unsigned b = __ballot_sync(GG_FULL, p);
    if ((threadIdx.x & 31) == 0) nz[i >> 5] = b;
  }
}

__global__ void degrees_from_offsets(const uint64_t *__restrict__ off, uint32_t V, uint32_t *__restrict__ deg) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x)
    deg[v] = (uint32_t)(off[v + 1] - off[v]);
}

// 1 where lo < deg[i].
struct DegAbove {
  const uint32_t *deg;
  uint32_t lo;
  __device__ __forceinline__ uint32_t operator()(size_t i) const { return deg[i] > lo ? 1u : 0u; }
};

__global__ void compact_by_pos(const uint32_t *__restrict__ deg, uint32_t V, uint32_t lo,
                               const uint32_t *__restrict__ pos, uint32_t *__restrict__ out) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x)
    if (deg[v] > lo) out[pos[v]] = (uint32_t)v;
}

// Heavy vertices among a vertex list (1 each), and their HEAVY_CHUNK chunks.
struct HeavyCount {
  const uint32_t *list;
  const uint32_t *deg;
  uint32_t chunk;  // 0: count the vertices
  __device__ __forceinline__ uint32_t operator()(size_t i) const {
    const uint32_t d = deg[list[i]];
    return d <= HEAVY_DEG ? 0u : chunk ? (d + chunk - 1) / chunk : 1u;
  }
};

// Long lists are cut at absolute multiples of the chunk size in the adjacency
// array (so every chunk's 16-byte windows are aligned): a list [b, e) covers
// blocks b/chunk .. (e-1)/chunk.
struct AlignedChunkCount {
  const uint32_t *list;
  const uint64_t *off;
  uint32_t chunk;
  __device__ __forceinline__ uint32_t operator()(size_t i) const {
    const uint32_t v = list[i];
    const uint64_t b = off[v], e = off[v + 1];
    return e > b ? (uint32_t)((e - 1) / chunk - b / chunk + 1) : 0u;
  }
};

// The heavy ones among the long-list vertices; pos, first: the scans of
// HeavyCount over the list (vertices, chunks).
__global__ void pick_heavy(const uint32_t *__restrict__ big, uint32_t nbig, const uint32_t *__restrict__ deg,
                           const uint32_t *__restrict__ pos, const uint32_t *__restrict__ first,
                           uint32_t *__restrict__ heavy, uint32_t *__restrict__ heavy_chunk) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nbig; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t v = big[i], h = pos[i];
    if (deg[v] > HEAVY_DEG) {
      heavy[h] = v;
      heavy_chunk[h] = first[i];
    }
    if (i == nbig - 1) heavy_chunk[pos[nbig]] = first[nbig];
  }
}

__global__ void fill_chunk_owner(const uint32_t *__restrict__ heavy_chunk, uint32_t nheavy,
                                 uint32_t *__restrict__ owner) {
  for (size_t h = (size_t)blockIdx.x * blockDim.x + threadIdx.x; h < nheavy; h += (size_t)gridDim.x * blockDim.x)
    for (uint32_t c = heavy_chunk[h]; c < heavy_chunk[h + 1]; c++) owner[c] = (uint32_t)h;
}

__global__ void gen_rmat_kernel(uint32_t *__restrict__ rec, uint64_t E, uint32_t scale, uint64_t key, int weighted) {
  int words = weighted ? 3 : 2;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t s, d;
    gg_rmat_edge(key, scale, e, &s, &d);
    rec[e * words] = s;
    rec[e * words + 1] = d;
    if (weighted) rec[e * words + 2] = __float_as_uint(gg_gen_weight(key, e));
  }
}

__global__ void gen_grid_kernel(uint32_t *__restrict__ rec, uint64_t E, uint32_t n, uint64_t key, int weighted) {
  int words = weighted ? 3 : 2;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t s, d;
    gg_grid_edge(n, e, &s, &d);
    rec[e * words] = s;
    rec[e * words + 1] = d;
    if (weighted) rec[e * words + 2] = __float_as_uint(gg_gen_weight(key, e));
  }
}

int bits_for(uint32_t V) {
  int b = 1;
  while (b < 32 && ((uint64_t)1 << b) < V) b++;
  return b;
}

static void free_sell(gg_graph *g, Dir *d);
static int sell_or_plain(gg_graph *g, Dir *d);
static void hot_bins(const gg_graph *g, Dir *d);
static int ranks_build(gg_graph *g);

// Degree bins of one direction (see Dir): the long lists (deg > light) with
// their aligned chunks, and the heavy ones among them for the BFS pulls.
// Two allocations hold all of them (bins_mem once the number of long lists
// is known, owner_mem once the chunk counts are).
static int build_bins(gg_graph *g, Dir *d) {
  const uint32_t V = g->V;
  cudaStream_t s = g->stream;
  DevScratch tmp;
  uint32_t *pos = nullptr, *scratch = nullptr;
  GG_TRY(tmp.get(&pos, (size_t)V + 1 + scan_scratch_elems(V)));
  scratch = pos + V + 1;
  GG_CUDA((exclusive_scan<uint32_t, DegAbove>(DegAbove{d->deg, d->light}, V, pos, scratch, s, nullptr)));
  uint32_t n = 0;
  GG_CUDA(cudaMemcpyAsync(&n, pos + V, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  if (n == 0) return GG_OK;
  GG_CUDA(cudaMalloc(&d->bins_mem, sizeof(uint32_t) * (2 * (size_t)n + 1)));
  d->nbig = n;
  d->big = d->bins_mem;
  d->big_chunk = d->big + n;
  g->graph_bytes += sizeof(uint32_t) * (2 * (size_t)n + 1);
  compact_by_pos<<<grid_for(V, 256, g->num_sms, 16), 256, 0, s>>>(d->deg, V, d->light, pos, d->big);
  GG_CUDA(cudaGetLastError());
  uint32_t *hpos = nullptr, *hfirst = nullptr, *sc = nullptr;
  GG_TRY(tmp.get(&hpos, 2 * ((size_t)n + 1) + scan_scratch_elems(n)));
  hfirst = hpos + n + 1;
  sc = hfirst + n + 1;
  GG_CUDA((exclusive_scan<uint32_t, AlignedChunkCount>(AlignedChunkCount{d->big, d->off, d->chunk}, n, d->big_chunk,
                                                       sc, s, nullptr)));
  GG_CUDA((exclusive_scan<uint32_t, HeavyCount>(HeavyCount{d->big, d->deg, 0}, n, hpos, sc, s, nullptr)));
  GG_CUDA((exclusive_scan<uint32_t, HeavyCount>(HeavyCount{d->big, d->deg, HEAVY_CHUNK}, n, hfirst, sc, s, nullptr)));
  uint32_t tot[3] = {0, 0, 0};
  GG_CUDA(cudaMemcpyAsync(&tot[0], d->big_chunk + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaMemcpyAsync(&tot[1], hpos + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaMemcpyAsync(&tot[2], hfirst + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  const size_t words = (size_t)tot[0] + tot[2] + 2 * (size_t)tot[1] + 1;
  GG_CUDA(cudaMalloc(&d->owner_mem, sizeof(uint32_t) * words));
  g->graph_bytes += sizeof(uint32_t) * words;
  d->owner_words = words;
  d->nbigchunks = tot[0];
  d->nheavy = tot[1];
  d->nchunks = tot[2];
  d->big_owner = d->owner_mem;
  d->chunk_owner = d->big_owner + tot[0];
  d->heavy = d->chunk_owner + tot[2];
  d->heavy_chunk = d->heavy + tot[1];
  fill_chunk_owner<<<grid_for(n, 128, g->num_sms, 8), 128, 0, s>>>(d->big_chunk, n, d->big_owner);
  pick_heavy<<<grid_for(n, 256, g->num_sms, 8), 256, 0, s>>>(d->big, n, d->deg, hpos, hfirst, d->heavy,
                                                            d->heavy_chunk);
  if (tot[1]) fill_chunk_owner<<<grid_for(tot[1], 128, g->num_sms, 8), 128, 0, s>>>(d->heavy_chunk, tot[1],
                                                                                  d->chunk_owner);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaStreamSynchronize(s));
  return GG_OK;
}

static void free_bins(gg_graph *g, Dir *d) {
  if (d->bins_mem) g->graph_bytes -= sizeof(uint32_t) * (2 * (size_t)d->nbig + 1);
  g->graph_bytes -= sizeof(uint32_t) * d->owner_words;
  if (d->bins_mem) cudaFree(d->bins_mem);
  if (d->owner_mem) cudaFree(d->owner_mem);
  d->bins_mem = d->owner_mem = nullptr;
  d->owner_words = 0;
  d->heavy = d->heavy_chunk = d->chunk_owner = d->big = d->big_chunk = d->big_owner = nullptr;
  d->nheavy = d->nchunks = d->nbig = d->nbigchunks = 0;
}

// Rebuilds both directions' degree bins for a light-list bound and a pull
// chunk size (the autotuner's two knobs).
int rebuild_bins(gg_graph *g, uint32_t light, uint32_t chunk, uint32_t vec) {
  if (light < 1 || light > HEAVY_DEG || (chunk != 128 && chunk != 256 && chunk != 512) || vec > 3) {
    set_error("light list bound must be 1..%u, the pull chunk 128, 256 or 512 and the vector flags 0..3",
              HEAVY_DEG);
    return GG_ERR_INVALID;
  }
  g->out.vec = g->in.vec = g->pr.vec = vec;
  GG_CUDA(cudaSetDevice(g->device));
  GG_CUDA(cudaStreamSynchronize(g->stream));
  const bool alias = g->in.nbr == g->out.nbr;
  free_bins(g, &g->out);
  g->out.light = light;
  g->out.chunk = chunk;
  GG_TRY(build_bins(g, &g->out));
  if (alias) {
    g->in = g->out;
  } else {
    free_bins(g, &g->in);
    g->in.light = light;
    g->in.chunk = chunk;
    GG_TRY(build_bins(g, &g->in));
  }
  g->bins_set = 1;
  Dir *hot[3] = {g->pr_ready ? &g->pr : nullptr, g->pr_out_ready ? &g->pr_out : nullptr,
                 g->ps_ready ? &g->ps : nullptr};
  for (Dir *d : hot) {
    if (!d) continue;
    const bool rows = d->sell_desc != nullptr;
    free_sell(g, d);
    free_bins(g, d);
    hot_bins(g, d);
    GG_TRY(build_bins(g, d));
    if (rows) GG_TRY(sell_or_plain(g, d));
  }
  return GG_OK;
}

// Neighbour / weight storage: device memory, or mapped pinned host memory
// when the graph keeps its adjacency on the host (the kernels dereference
// the same pointer over NVLink-C2C; unified addressing makes the host and
// device addresses of a mapped allocation equal).
int adj_alloc(gg_graph *g, bool host, void **p, size_t bytes) {
  *p = nullptr;
  if (!host) {
    GG_CUDA(cudaMalloc(p, bytes));
    g->graph_bytes += bytes;
    return GG_OK;
  }
  GG_CUDA(cudaHostAlloc(p, bytes, cudaHostAllocMapped));
  void *dp = nullptr;
  cudaError_t e = cudaHostGetDevicePointer(&dp, *p, 0);
  if (e != cudaSuccess || dp != *p) {
    cudaFreeHost(*p);
    *p = nullptr;
    if (e != cudaSuccess) return cuda_status(e, "mapped adjacency");
    set_error("mapped host adjacency needs unified addressing");
    return GG_ERR_CUDA;
  }
  g->host_bytes += bytes;
  return GG_OK;
}

static void adj_release(bool host, void *p) {
  if (!p) return;
  if (host)
    cudaFreeHost(p);
  else
    cudaFree(p);
}

// Degrees (offset differences), the deg > 0 bitmap and the degree bins of a
// direction whose offsets are written.
int finish_dir(gg_graph *g, Dir *d) {
  const uint32_t V = g->V;
  d->nv = V;
  d->ne = g->nadj;
  d->err = g->check_err;
  degrees_from_offsets<<<grid_for(V, 256, g->num_sms, 16), 256, 0, g->stream>>>(d->off, V, d->deg);
  GG_CUDA(cudaGetLastError());
  size_t words = bitmap_words32(V);
  GG_CUDA(cudaMalloc(&d->nz, sizeof(uint32_t) * words));
  g->graph_bytes += sizeof(uint32_t) * words;
  nonzero_bitmap<<<grid_for(words * 32, 256, g->num_sms, 16), 256, 0, g->stream>>>(d->deg, V, d->nz, words);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaStreamSynchronize(g->stream));
  return build_bins(g, d);
}

// One direction from its n sorted keys (see offsets_from_keys): offsets,
// neighbours, degrees and bins.  The weights, if any, are in place.
static int emit_dir(gg_graph *g, const uint64_t *keys, size_t n, int bits, bool low_major, Dir *d, bool host) {
  uint32_t V = g->V;
  GG_CUDA(cudaMalloc(&d->off, sizeof(uint64_t) * ((size_t)V + 1)));
  // padded to a multiple of 64 entries: chunked pulls load whole aligned
  // 16-byte windows that may run past the last list
  const size_t npad = (n + 64) / 64 * 64;
  GG_TRY(adj_alloc(g, host, (void **)&d->nbr, sizeof(uint32_t) * npad));
  GG_CUDA(cudaMemsetAsync(d->nbr + n, 0, sizeof(uint32_t) * (npad - n), g->stream));
  GG_CUDA(cudaMalloc(&d->deg, sizeof(uint32_t) * ((size_t)V + 1)));
  g->graph_bytes += sizeof(uint64_t) * ((size_t)V + 1) + sizeof(uint32_t) * ((size_t)V + 1);
  if (n == 0) {
    GG_CUDA(cudaMemsetAsync(d->off, 0, sizeof(uint64_t) * ((size_t)V + 1), g->stream));
  } else {
    DevScratch tmp;
    char *blob = nullptr;
    GG_TRY(tmp.get(&blob, 16 + sizeof(Gap) * GAP_CAP));
    unsigned *ngaps = (unsigned *)blob;
    Gap *gaps = (Gap *)(blob + 16);
    GG_CUDA(cudaMemsetAsync(ngaps, 0, sizeof(unsigned), g->stream));
    offsets_from_keys<<<grid_for(n, 256, g->num_sms, 16), 256, 0, g->stream>>>(keys, n, bits, low_major, V, d->off,
                                                                               d->nbr, gaps, ngaps);
    fill_gaps<<<(unsigned)g->num_sms * 4, 256, 0, g->stream>>>(d->off, gaps, ngaps);
    GG_CUDA(cudaGetLastError());
  }
  return finish_dir(g, d);
}

// Sorts keys (and weights, values vin moved between b0 and b1) on the key
// bits [0, hi_bit) and emits the direction.  The last pass writes the
// weights where they stay, in device memory; host adjacency takes a copy.
static int sort_dir(gg_graph *g, void *scratch, uint64_t *ka, uint64_t *kb, uint32_t *vin, uint32_t *b0, uint32_t *b1,
                    size_t n, int bits, bool low_major, Dir *d, bool host, uint64_t **ks, uint32_t **vs,
                    RsCounts have = RS_NONE) {
  if (vin) GG_TRY(adj_alloc(g, host, (void **)&d->w, sizeof(float) * (n ? n : 1)));
  SortValues v{vin, b0, b1, host ? nullptr : (uint32_t *)d->w};
  GG_TRY(radix_sort(g, scratch, ka, kb, v, n, 0, low_major ? bits : 2 * bits, ks, vs, have));
  if (vin && host && n) GG_CUDA(cudaMemcpyAsync(d->w, *vs, sizeof(float) * n, cudaMemcpyDefault, g->stream));
  return emit_dir(g, *ks, n, bits, low_major, d, host);
}

static void free_dir(Dir *d, bool adj_host) {
  if (d->off) cudaFree(d->off);
  adj_release(adj_host, d->nbr);
  adj_release(adj_host, d->w);
  if (d->deg) cudaFree(d->deg);
  if (d->nz) cudaFree(d->nz);
  if (d->bins_mem) cudaFree(d->bins_mem);
  if (d->owner_mem) cudaFree(d->owner_mem);
  *d = Dir();
}

// ---------------------------------------------------------------- PageRank layout
// PageRank gathers source state once per edge; a source is gathered as
// often as its out-degree.  Renumbering vertices by descending out-degree
// packs the most gathered values into few cache lines (on R-MAT graphs the
// top 2^20 sources of scale 26 draw ~70% of the gathers), and sorting each
// in-list by the new numbers puts a hub's hottest in-neighbours side by side
// in one warp's loads.  The renumbered incoming adjacency is built once by
// the same radix sort as the load; ranks map back to vertex order on output.
// Sort key of a vertex: its out-degree to an eighth of its power of two
// (exact below 16; descending), then its in-degree (exact below 2048;
// descending), then its id.  How often a source is gathered decides where it
// lies to within 12%, and runs of vertices that are alike in that lie by list
// length, which is what pull_rows needs of 32 consecutive rows.
constexpr int RANK_BITS = 20;
__device__ __forceinline__ uint32_t out_class(uint32_t d) {
  if (d < 16) return d;
  const uint32_t e = 31 - __clz(d);
  return 16 + (e - 4) * 8 + ((d >> (e - 3)) & 7u);  // at most 239
}
__device__ __forceinline__ uint32_t in_class(uint32_t d) {
  if (d < 2048) return d;
  const uint32_t e = 31 - __clz(d);
  return 2048 + (e - 11) * 64 + ((d >> (e - 6)) & 63u);  // at most 3391
}
__global__ void degree_rank_keys(const uint32_t *__restrict__ out_deg, const uint32_t *__restrict__ in_deg, uint32_t V,
                                 int bits, uint64_t *__restrict__ keys) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x) {
    const uint32_t k = ((255u - out_class(out_deg[v])) << 12) | (4095u - in_class(in_deg[v]));
    keys[v] = ((uint64_t)k << bits) | v;
  }
}

// keys: the V sorted degree keys, vertex id in the low `bits` bits.
__global__ void rank_tables(const uint64_t *__restrict__ keys, uint32_t V, int bits,
                            const uint32_t *__restrict__ out_deg, uint32_t *__restrict__ id_of_rank,
                            uint32_t *__restrict__ rank_of, uint32_t *__restrict__ od) {
  const uint64_t mask = (1ull << bits) - 1;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < V; r += (size_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)(keys[r] & mask);
    id_of_rank[r] = v;
    rank_of[v] = (uint32_t)r;
    od[r] = out_deg[v];
  }
}

// Classes of equal width over the weights' range [wmin, wmin + range]
// (bits = 0: none), for lists ordered by weight.
constexpr int WEIGHT_BITS = 6;
struct WeightClass {
  int bits = 0;
  float wmin = 0.0f, inv = 0.0f;  // inv: classes per unit of weight
  __device__ __forceinline__ uint32_t of(float w) const {
    const float x = __fmul_rn(__fsub_rn(w, wmin), inv);  // monotone in w
    const float top = (float)((1 << bits) - 1);
    return x >= top ? (1u << bits) - 1u : x > 0.0f ? (uint32_t)x : 0u;
  }
};

// Entry p of the lists taken in the order list_of[0], list_of[1], ... (null:
// 0, 1, ...), list r at first[r]: keys[p] = (r << bits) | rank_of[its
// neighbour] (rank_of null: the neighbour), vals[p] = its weight.  Tiles of
// consecutive p, each thread finding its list by binary search in the tile's
// slice of `first` in shared memory, so reads of long lists and all writes
// are coalesced.  Lists from nlist on are empty.
constexpr int EX_THREADS = 256;
constexpr int EX_TILE = 2048;
__global__ void __launch_bounds__(EX_THREADS)
    expand_keys(Dir d, const uint64_t *__restrict__ first, uint32_t nlist, const uint32_t *__restrict__ list_of,
                const uint32_t *__restrict__ rank_of, size_t n, int bits, uint64_t *__restrict__ keys,
                uint32_t *__restrict__ vals, WeightClass wc) {
  __shared__ uint64_t s_first[EX_TILE + 1];
  __shared__ uint64_t s_off[EX_TILE + 1];
  __shared__ uint32_t s_lo, s_hi;
  const size_t ntiles = (n + EX_TILE - 1) / EX_TILE;
  for (size_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint64_t p0 = tile * EX_TILE, p1 = p0 + EX_TILE < n ? p0 + EX_TILE : n;
    if (threadIdx.x < 64) {
      // the lists holding the tile's first and last entry: the last r with first[r] <= x
      const uint64_t x = threadIdx.x < 32 ? p0 : p1 - 1;
      const uint32_t r = warp_upper_bound(first, 0u, nlist, x) - 1;
      if (lane_id() == 0) (threadIdx.x < 32 ? s_lo : s_hi) = r;
    }
    __syncthreads();
    const uint32_t lo = s_lo, cnt = s_hi - s_lo + 1;
    const bool staged = cnt <= EX_TILE;
    if (staged)
      for (uint32_t i = threadIdx.x; i < cnt; i += EX_THREADS) {
        s_first[i] = first[lo + i];
        s_off[i] = d.off[list_of ? list_of[lo + i] : lo + i];
      }
    __syncthreads();
#pragma unroll 4
    for (uint64_t p = p0 + threadIdx.x; p < p1; p += EX_THREADS) {
      uint32_t a = 0, b = cnt - 1;
      while (a < b) {
        const uint32_t mid = a + (b - a + 1) / 2;
        if ((staged ? s_first[mid] : first[lo + mid]) <= p)
          a = mid;
        else
          b = mid - 1;
      }
      const uint64_t k = staged ? s_off[a] + (p - s_first[a])
                                : d.off[list_of ? list_of[lo + a] : lo + a] + (p - first[lo + a]);
      const uint32_t u = nbr_at(d, k, GG_SITE);
      uint64_t key = ((uint64_t)(lo + a) << bits) | (rank_of ? rank_of[u] : u);
      if (vals) {
        const float w = d.w[k];
        vals[p] = __float_as_uint(w);
        if (wc.bits) key |= (uint64_t)wc.of(w) << (2 * bits);
      }
      keys[p] = key;
    }
    __syncthreads();
  }
}

// Steps of every slice (the longest light list over four), and whether any
// of its vertices has a list.
__global__ void sell_widths(const uint32_t *__restrict__ deg, uint32_t V, uint32_t light, uint32_t nslices,
                            uint32_t *__restrict__ steps, uint32_t *__restrict__ full) {
  const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
  const unsigned lane = lane_id();
  for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) / 32; s < nslices; s += nwarps) {
    const size_t v = (size_t)s * 32 + lane;
    const uint32_t d = v < V ? deg[v] : 0u;
    const uint32_t m = __reduce_max_sync(GG_FULL, d <= light ? d : 0u);
    const bool any = __any_sync(GG_FULL, d > 0);
    if (lane == 0) {
      steps[s] = (m + 3) / 4;
      full[s] = any;
    }
  }
}

// Descriptors (slices with lists first, both in slice order) and the
// column-major entries.  first, place: the scans of steps and full.
__global__ void sell_fill(Dir d, uint32_t V, uint32_t nslices, uint32_t nfull, const uint32_t *__restrict__ first,
                          const uint32_t *__restrict__ place, uint4 *__restrict__ desc, uint4 *__restrict__ col,
                          float4 *__restrict__ wcol) {
  const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
  const unsigned lane = lane_id();
  for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) / 32; s < nslices; s += nwarps) {
    const uint32_t t0 = first[s], steps = first[s + 1] - t0, p = place[s];
    if (lane == 0) desc[place[s + 1] > p ? p : nfull + (s - p)] = make_uint4(s, t0, steps, 0);
    const size_t v = (size_t)s * 32 + lane;
    uint64_t b = 0;
    uint32_t n = 0;
    if (v < V) {
      b = d.off[v];
      n = d.deg[v] <= d.light ? d.deg[v] : 0u;
    }
    for (uint32_t t = 0; t < steps; t++) {
      uint32_t u[4];
      float w[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const bool in = 4 * t + j < n;
        u[j] = in ? nbr_at(d, b + 4 * t + j, GG_SITE) : V;
        w[j] = in && wcol ? d.w[b + 4 * t + j] : 0.0f;
      }
      const size_t at = (size_t)(t0 + t) * 32 + lane;
      col[at] = make_uint4(u[0], u[1], u[2], u[3]);
      if (wcol) wcol[at] = make_float4(w[0], w[1], w[2], w[3]);
    }
  }
}

static void free_sell(gg_graph *g, Dir *d) {
  if (d->sell_desc) g->graph_bytes -= sizeof(uint4) * d->nslices;
  if (d->sell_col) g->graph_bytes -= sizeof(uint4) * 32 * d->sell_steps * (d->sell_w ? 2 : 1);
  if (d->sell_desc) cudaFree(d->sell_desc);
  if (d->sell_col) cudaFree(d->sell_col);
  d->sell_desc = d->sell_col = nullptr;
  d->sell_w = nullptr;
  d->nslices = d->nfull = 0;
  d->sell_steps = 0;
}

// The rows of a hot-source direction (see pull_rows) from its lists and bins.
static int build_sell(gg_graph *g, Dir *d) {
  cudaStream_t s = g->stream;
  const uint32_t V = g->V, ns = (uint32_t)(((size_t)V + 31) / 32);
  DevScratch tmp;
  uint32_t *steps = nullptr;
  GG_TRY(tmp.get(&steps, 4 * ((size_t)ns + 1) + scan_scratch_elems(ns)));
  uint32_t *full = steps + ns + 1, *first = full + ns + 1, *place = first + ns + 1, *scratch = place + ns + 1;
  const unsigned grid = grid_for((size_t)ns * 32, 256, g->num_sms, 8);
  sell_widths<<<grid, 256, 0, s>>>(d->deg, V, d->light, ns, steps, full);
  GG_CUDA(cudaGetLastError());
  GG_CUDA((exclusive_scan<uint32_t, ArrayIn<uint32_t>>(ArrayIn<uint32_t>{steps}, ns, first, scratch, s, nullptr)));
  GG_CUDA((exclusive_scan<uint32_t, ArrayIn<uint32_t>>(ArrayIn<uint32_t>{full}, ns, place, scratch, s, nullptr)));
  uint32_t tot[2] = {0, 0};
  GG_CUDA(cudaMemcpyAsync(&tot[0], first + ns, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaMemcpyAsync(&tot[1], place + ns, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  const size_t entries = 32 * (size_t)tot[0];
  uint4 *col = nullptr;
  GG_CUDA(cudaMalloc(&col, sizeof(uint4) * (entries ? entries : 1) * (d->w ? 2 : 1)));
  d->sell_col = col;
  d->sell_w = d->w ? reinterpret_cast<float4 *>(col + entries) : nullptr;
  d->sell_steps = tot[0];
  d->nslices = ns;
  d->nfull = tot[1];
  g->graph_bytes += sizeof(uint4) * entries * (d->w ? 2 : 1);
  uint4 *desc = nullptr;
  GG_CUDA(cudaMalloc(&desc, sizeof(uint4) * ns));
  g->graph_bytes += sizeof(uint4) * ns;
  d->sell_desc = desc;
  sell_fill<<<grid, 256, 0, s>>>(*d, V, ns, d->nfull, first, place, desc, col, d->sell_w);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaStreamSynchronize(s));
  return GG_OK;
}

// A direction without room for its rows is pulled through its lists, as a
// plain one.
static int sell_or_plain(gg_graph *g, Dir *d) {
  const int r = build_sell(g, d);
  if (r == GG_OK) return r;
  free_sell(g, d);
  if (r != GG_ERR_NOMEM) return r;
  cudaGetLastError();
  return GG_OK;
}

// Light bound and chunk size of a hot-source direction unless
// gg_graph_set_bins chose them.  A light list is one lane's serial walk, about
// 0.1 us per entry, so the bound grows with the graph (entries / 2^16, a power
// of two in 32..1024): the longest walk stays below the time the whole pull
// takes.  Measured, PageRank of 20 iterations with bounds 32 / 128 / 512 /
// 1024: R-MAT 18 506 / 454 / 546 / 889 us, R-MAT 20 1297 / 1029 / 1041 / 1396
// us, R-MAT 26 98 / 73 / 69 / 67 ms.
static void hot_bins(const gg_graph *g, Dir *d) {
  if (g->bins_set) {
    d->light = g->out.light;
    d->chunk = g->out.chunk;
    return;
  }
  uint32_t l = 32;
  while (l < 1024 && (g->nadj >> 16) >= 2 * (uint64_t)l) l *= 2;
  d->light = l;
  d->chunk = 512;
}

// Frees a renumbered direction and its device bytes.
static void free_hot_dir(gg_graph *g, Dir *d) {
  const size_t V = g->V;
  free_sell(g, d);
  free_bins(g, d);
  const size_t npad = (g->nadj + 64) / 64 * 64;
  g->graph_bytes -= sizeof(uint64_t) * (V + 1) + sizeof(uint32_t) * (npad + V + 1) +
                    sizeof(uint32_t) * bitmap_words32(g->V) + (d->w ? sizeof(float) * (g->nadj ? g->nadj : 1) : 0);
  if (d->off) cudaFree(d->off);
  if (d->nbr) cudaFree(d->nbr);
  if (d->w) cudaFree(d->w);
  if (d->deg) cudaFree(d->deg);
  if (d->nz) cudaFree(d->nz);
  *d = Dir();
}

void pr_layout_free(gg_graph *g) {
  if (!g->ranks_ready) return;
  cudaStreamSynchronize(g->stream);
  if (g->pr_ready) free_hot_dir(g, &g->pr);
  if (g->pr_out_ready) free_hot_dir(g, &g->pr_out);
  if (g->ps_ready) free_hot_dir(g, &g->ps);
  g->pr_ready = g->pr_out_ready = g->ps_ready = false;
  g->graph_bytes -= sizeof(uint32_t) * 3 * (size_t)g->V;
  cudaFree(g->pr_rank_of);
  g->pr_rank_of = g->pr_id_of_rank = g->pr_od = nullptr;
  g->ranks_ready = false;
}

// The transpose of src's lists taken in rank order, in the hot-source
// numbering: list r' holds the ranks r of the lists that hold r', ascending
// (wc: by weight class, then ascending).  The expansion walks the lists in
// ascending rank, so one stable sort on the other end's rank alone orders
// both (half the passes of a sort on the pair).  Weights are carried along;
// duplicate edges keep src's order.
static int transpose_dir(gg_graph *g, const Dir &src, Dir *dst, WeightClass wc = WeightClass()) {
  const size_t n = g->nadj;
  const int bits = bits_for(g->V);
  DevScratch tmp;
  uint64_t *first = nullptr, *scan = nullptr;
  uint64_t *k0 = nullptr, *k1 = nullptr, *ks = nullptr;
  uint32_t *v0 = nullptr, *v1 = nullptr, *vs = nullptr;
  void *scratch = nullptr;
  GG_TRY(tmp.get(&first, (size_t)g->V + 1 + scan_scratch_elems(g->V)));
  scan = first + g->V + 1;
  GG_TRY(tmp.sort_buffers(n, g->weighted != 0, &k0, &k1, &v0, &v1, &scratch));
  GG_CUDA((exclusive_scan<unsigned long long, QueueDegreeIn>(QueueDegreeIn{g->pr_id_of_rank, src.deg}, g->V,
                                                             (unsigned long long *)first, (unsigned long long *)scan,
                                                             g->stream, nullptr)));
  if (n) {
    expand_keys<<<grid_for((n + EX_TILE - 1) / EX_TILE * EX_THREADS, EX_THREADS, g->num_sms, 6), EX_THREADS, 0,
                  g->stream>>>(src, first, g->V, g->pr_id_of_rank, g->pr_rank_of, n, bits, k0, v0, wc);
    GG_CUDA(cudaGetLastError());
  }
  *dst = Dir();
  dst->vec = src.vec;
  hot_bins(g, dst);
  uint64_t *ka = k0;
  uint32_t *va = v0;
  if (wc.bits) {
    const SortValues v{v0, v0, v1, nullptr};
    GG_TRY(radix_sort(g, scratch, k0, k1, v, n, 2 * bits, 2 * bits + wc.bits, &ka, &va));
  }
  return sort_dir(g, scratch, ka, ka == k0 ? k1 : k0, va, va, va == v0 ? v1 : v0, n, bits, true, dst, false, &ks, &vs);
}

// The outgoing adjacency in the hot-source numbering.
int hot_out_build(gg_graph *g) {
  if (g->pr_out_ready) return GG_OK;
  GG_TRY(ranks_build(g));
  const int s = transpose_dir(g, g->in, &g->pr_out);
  if (s != GG_OK) {
    free_hot_dir(g, &g->pr_out);
    return s;
  }
  g->pr_out_ready = true;
  return GG_OK;
}

// The renumbered outgoing adjacency's rows, for pulls over it (BC's
// backward sweep).
int hot_out_rows(gg_graph *g) {
  GG_TRY(hot_out_build(g));
  return g->pr_out.sell_desc ? GG_OK : sell_or_plain(g, &g->pr_out);
}

// The vertices ranked by degree_rank_keys: the numbering's three tables.
static int ranks_build(gg_graph *g) {
  if (g->ranks_ready) return GG_OK;
  GG_CUDA(cudaSetDevice(g->device));
  const uint32_t V = g->V;
  const int bits = bits_for(V);
  DevScratch tmp;
  uint64_t *k0 = nullptr, *k1 = nullptr, *ks = nullptr;
  uint32_t *v0 = nullptr, *v1 = nullptr, *vs = nullptr;
  void *scratch = nullptr;
  GG_TRY(tmp.sort_buffers(V, false, &k0, &k1, &v0, &v1, &scratch));
  degree_rank_keys<<<grid_for(V, 256, g->num_sms, 16), 256, 0, g->stream>>>(g->out.deg, g->in.deg, V, bits, k0);
  GG_CUDA(cudaGetLastError());
  // the keys start in id order and the sort is stable: the class bits suffice
  GG_TRY(radix_sort(g, scratch, k0, k1, SortValues(), V, bits, bits + RANK_BITS, &ks, &vs));
  uint32_t *tables = nullptr;
  GG_CUDA(cudaMalloc(&tables, sizeof(uint32_t) * 3 * (size_t)V));
  g->pr_rank_of = tables;
  g->pr_id_of_rank = tables + V;
  g->pr_od = tables + 2 * (size_t)V;
  g->graph_bytes += sizeof(uint32_t) * 3 * (size_t)V;
  g->ranks_ready = true;
  rank_tables<<<grid_for(V, 256, g->num_sms, 16), 256, 0, g->stream>>>(ks, V, bits, g->out.deg, g->pr_id_of_rank,
                                                                      g->pr_rank_of, g->pr_od);
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaStreamSynchronize(g->stream));
  return GG_OK;
}

// The incoming adjacency renumbered, with its rows.
int pr_layout_build(gg_graph *g) {
  if (g->pr_ready) return GG_OK;
  GG_TRY(ranks_build(g));
  const int s = transpose_dir(g, g->out, &g->pr);
  if (s != GG_OK) {
    free_hot_dir(g, &g->pr);
    return s;
  }
  g->pr_ready = true;
  return sell_or_plain(g, &g->pr);
}

// Least and largest weight (NaN weights left out), as ordered integers.
__device__ __forceinline__ uint32_t float_order(float x) {
  const uint32_t u = __float_as_uint(x);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__global__ void weight_range(const float *__restrict__ w, size_t n, uint32_t *range) {
  uint32_t lo = 0xffffffffu, hi = 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float x = w[i];
    if (x != x) continue;
    const uint32_t o = float_order(x);
    lo = o < lo ? o : lo;
    hi = o > hi ? o : hi;
  }
  lo = __reduce_min_sync(GG_FULL, lo);
  hi = __reduce_max_sync(GG_FULL, hi);
  if (lane_id() == 0) {
    if (lo != 0xffffffffu) atomicMin(range, lo);
    if (hi) atomicMax(range + 1, hi);
  }
}
static float float_of_order(uint32_t o) {
  const uint32_t u = o & 0x80000000u ? o & 0x7fffffffu : ~o;
  float f;
  memcpy(&f, &u, sizeof f);
  return f;
}

// SSSP's layout: the incoming adjacency renumbered, each list by ascending
// weight class (64 classes of equal width), with its rows, and for a directed
// graph the outgoing adjacency.  A dense call relaxes only what an active
// source can improve: with the active sources' least distance, a list's walk
// ends where that distance plus the next weight reaches the vertex's own.  On
// R-MAT graphs with weights in [0, 1) a hub settles near the least active
// distance, so most of its list is never gathered.  R-MAT 24, 268 M entries:
// 11.1 ms walking every list, 5.7 ms so; the class pass adds 2.4 ms to the
// layout's build.
int sssp_layout_build(gg_graph *g) {
  GG_TRY(ranks_build(g));
  if (!g->ps_ready) {
    WeightClass wc;
    g->ps_width = INFINITY;
    g->ps_wmin = -INFINITY;
    if (g->nadj && 2 * bits_for(g->V) + WEIGHT_BITS <= 64) {
      DevScratch tmp;
      uint32_t *dev = nullptr, h[2] = {0xffffffffu, 0u};
      GG_TRY(tmp.get(&dev, 2));
      GG_CUDA(cudaMemcpyAsync(dev, h, sizeof(h), cudaMemcpyHostToDevice, g->stream));
      weight_range<<<grid_for(g->nadj, 256, g->num_sms, 8), 256, 0, g->stream>>>(g->in.w, g->nadj, dev);
      GG_CUDA(cudaGetLastError());
      GG_CUDA(cudaMemcpyAsync(h, dev, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
      GG_CUDA(cudaStreamSynchronize(g->stream));
      const float lo = float_of_order(h[0]), hi = float_of_order(h[1]), range = hi - lo;
      if (h[0] <= h[1] && isfinite(lo) && isfinite(hi) && isfinite(range)) {
        g->ps_wmin = lo;
        wc.wmin = lo;
        const float classes = (float)(1 << WEIGHT_BITS);
        if (range > 0.0f && isfinite(classes / range)) {
          wc.bits = WEIGHT_BITS;
          wc.inv = classes / range;
          // a class's width and the rounding of its bounds (see WeightClass)
          g->ps_width = range / classes * 1.001f + 1e-6f * fmaxf(fabsf(lo), fabsf(hi));
        }
      }
    }
    const int s = transpose_dir(g, g->out, &g->ps, wc);
    if (s != GG_OK) {
      free_hot_dir(g, &g->ps);
      return s;
    }
    g->ps_ready = true;
    GG_TRY(sell_or_plain(g, &g->ps));
  }
  return g->symmetric ? GG_OK : hot_out_build(g);
}

void graph_destroy(gg_graph *g) {
  if (!g) return;
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  pools_destroy(g);
  for (cudaGraphExec_t &x : g->pr_exec) {
    if (x) cudaGraphExecDestroy(x);
    x = nullptr;
  }
  pr_layout_free(g);
  bool alias = g->in.nbr == g->out.nbr;
  free_dir(&g->out, g->adj_host);
  if (!alias) free_dir(&g->in, g->adj_host);
  ws_free_all(g);
  if (g->ev0) cudaEventDestroy(g->ev0);
  if (g->ev1) cudaEventDestroy(g->ev1);
  if (g->fork) cudaEventDestroy(g->fork);
  if (g->join) cudaEventDestroy(g->join);
  if (g->side) {
    cudaStreamSynchronize(g->side);
    cudaStreamDestroy(g->side);
  }
  for (cudaEvent_t e : g->evpool) cudaEventDestroy(e);
  if (g->check_err) cudaFree(g->check_err);
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
}

static int graph_create(int device, uint32_t V, int weighted, int symmetric, gg_graph **out) {
  if (V == 0) {
    set_error("vertices must be > 0");
    return GG_ERR_INVALID;
  }
  int ndev = 0;
  GG_CUDA(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) {
    set_error("device %d out of range (%d devices)", device, ndev);
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(device));
  gg_graph *g = new gg_graph();
  g->device = device;
  g->V = V;
  g->weighted = weighted ? 1 : 0;
  g->symmetric = symmetric ? 1 : 0;
  cudaError_t e = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&g->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&g->ev1);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&g->side, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->join, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaMalloc(&g->check_err, 4 * sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemset(g->check_err, 0, 4 * sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMalloc(&g->ws.ctr, sizeof(Counters));
  if (e == cudaSuccess) e = cudaMallocHost(&g->ws.ctr_host, sizeof(Counters));
  if (e == cudaSuccess) e = cudaHostAlloc(&g->ws.stage, STAGE_BYTES_HOST, cudaHostAllocMapped);
  if (e != cudaSuccess) {
    graph_destroy(g);
    return cuda_status(e, "graph create");
  }
  *out = g;
  return GG_OK;
}

// Builds CSR/CSC from E records in device memory (4-byte aligned).
int build_from_device_records(gg_graph *g, const uint32_t *rec, uint64_t E) {
  int words = g->weighted ? 3 : 2;
  g->E = E;
  size_t n = g->symmetric ? 2 * E : E;
  g->nadj = n;
  if (n >= 0xFFFFFFFFull) {
    set_error("%llu adjacency entries per direction: the device sort supports < 2^32",
              (unsigned long long)n);
    return GG_ERR_TOO_LARGE;
  }
  const int bits = bits_for(g->V);
  const bool host = g->adj_host != 0;
  DevScratch tmp;
  uint64_t *k0 = nullptr, *k1 = nullptr, *ks = nullptr;
  uint32_t *v0 = nullptr, *v1 = nullptr, *vs = nullptr;
  void *scratch = nullptr;
  unsigned *err = nullptr;
  GG_TRY(tmp.sort_buffers(n, g->weighted != 0, &k0, &k1, &v0, &v1, &scratch));
  GG_TRY(tmp.get(&err, 1));
  GG_CUDA(cudaMemsetAsync(err, 0, sizeof(unsigned), g->stream));
  if (E) {
    GG_TRY(radix_clear(g, scratch, n));
    const RsPlan plan = rs_plan(0, 2 * bits);
    make_keys<<<grid_for(E, RS_THREADS, g->num_sms, 4), RS_THREADS, 0, g->stream>>>(
        rec, E, words, g->symmetric ? 2 : 0, bits, g->V, k0, v0, err, plan, (uint32_t *)scratch);
    GG_CUDA(cudaGetLastError());
    unsigned herr = 0;
    GG_CUDA(cudaMemcpyAsync(&herr, err, sizeof(unsigned), cudaMemcpyDeviceToHost, g->stream));
    GG_CUDA(cudaStreamSynchronize(g->stream));
    if (herr) {
      set_error("an edge names a vertex id >= vertices (%u)", g->V);
      return GG_ERR_RANGE;
    }
  }
  GG_TRY(sort_dir(g, scratch, k0, k1, v0, v0, v1, n, bits, false, &g->out, host, &ks, &vs,
                  E ? RS_COUNTED : RS_NONE));
  if (g->symmetric) {
    g->in = g->out;
  } else {
    // the CSC from the CSR's order (source, destination, record): a stable
    // sort on the destination bits alone gives (destination, source, record);
    // where no digit of that sort spans both ids, the destination's places are
    // in the scratch already (0.33 ms of counting at 134 M keys)
    uint32_t *b0 = vs == v1 ? v1 : v0, *b1 = vs == v1 ? v0 : v1;
    GG_TRY(sort_dir(g, scratch, ks, ks == k0 ? k1 : k0, vs, b0, b1, n, bits, true, &g->in, host, &ks, &vs,
                    n > 1 && rs_leads(rs_plan(0, bits), rs_plan(0, 2 * bits)) ? RS_PLACED : RS_NONE));
  }
  GG_CUDA(cudaStreamSynchronize(g->stream));
  return GG_OK;
}

static uint64_t unit_of(int weighted) { return weighted ? 12 : 8; }

}  // namespace gg

using namespace gg;

extern "C" {

const char *gg_last_error(void) { return g_err; }

int gg_host_alloc(uint64_t bytes, void **out) {
  if (!out) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaMallocHost(out, bytes ? bytes : 1));
  return GG_OK;
}

// core/graph.hpp:253-307 with one partition: the file is the array's bytes,
// vertex 0 first.  `array` may be host or device memory.
static bool is_device_ptr(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

int gg_dump_vertex_array(const void *array, uint64_t elem_size, uint32_t vertices, const char *path) {
  if (!array || !path || elem_size == 0) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  const uint64_t bytes = elem_size * vertices;
  std::vector<char> stage;
  const char *src = (const char *)array;
  if (is_device_ptr(array)) {
    stage.resize(bytes);
    GG_CUDA(cudaMemcpy(stage.data(), array, bytes, cudaMemcpyDeviceToHost));
    src = stage.data();
  }
  FILE *f = fopen(path, "wb");
  if (!f) {
    set_error("cannot open %s for writing", path);
    return GG_ERR_IO;
  }
  const size_t n = fwrite(src, 1, bytes, f);
  const int rc = fclose(f);
  if (n != bytes || rc != 0) {
    set_error("short write to %s", path);
    return GG_ERR_IO;
  }
  return GG_OK;
}

int gg_restore_vertex_array(void *array, uint64_t elem_size, uint32_t vertices, const char *path) {
  if (!array || !path || elem_size == 0) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  const uint64_t bytes = elem_size * vertices;
  FILE *f = fopen(path, "rb");
  if (!f) {
    set_error("cannot open %s", path);
    return GG_ERR_IO;
  }
  fseek(f, 0, SEEK_END);
  const long len = ftell(f);
  fseek(f, 0, SEEK_SET);
  if (len < 0 || (uint64_t)len != bytes) {
    fclose(f);
    set_error("%s holds %ld bytes, the array %llu", path, len, (unsigned long long)bytes);
    return GG_ERR_INVALID;
  }
  std::vector<char> stage;
  const bool dev = is_device_ptr(array);
  char *dst = (char *)array;
  if (dev) {
    stage.resize(bytes);
    dst = stage.data();
  }
  const size_t n = fread(dst, 1, bytes, f);
  fclose(f);
  if (n != bytes) {
    set_error("short read from %s", path);
    return GG_ERR_IO;
  }
  if (dev) GG_CUDA(cudaMemcpy(array, stage.data(), bytes, cudaMemcpyHostToDevice));
  return GG_OK;
}

int gg_host_free(void *p) {
  if (p) GG_CUDA(cudaFreeHost(p));
  return GG_OK;
}

int gg_graph_from_device_records(const void *d_records, uint64_t bytes, uint32_t vertices, int weighted,
                                 int symmetric, int device, gg_graph **out) {
  if (!out || (!d_records && bytes >= unit_of(weighted))) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  if ((uintptr_t)d_records % 4) {
    set_error("device records must be 4-byte aligned");
    return GG_ERR_INVALID;
  }
  gg_graph *g = nullptr;
  GG_TRY(graph_create(device, vertices, weighted, symmetric, &g));
  const uint64_t E = bytes / unit_of(weighted);
  bool part = false;
  uint64_t cap = 0, gcap = 0;
  int s = build_plan(g, E, true, nullptr, &part, &cap, &gcap);
  if (s == GG_OK) s = build_records(g, (const uint32_t *)d_records, E, part, cap, gcap, nullptr);
  if (s != GG_OK) {
    graph_destroy(g);
    return s;
  }
  *out = g;
  return GG_OK;
}

// Device-readable view of host records for the partitioned build: device
// or pinned memory as it is, anything else registered for the call.
struct RecordsView {
  const uint32_t *dev = nullptr;
  void *registered = nullptr;
  void *staged = nullptr;  // pinned copy when the range cannot be registered
  RecordsView() = default;
  RecordsView(const RecordsView &) = delete;
  RecordsView &operator=(const RecordsView &) = delete;
  ~RecordsView() {
    if (registered) cudaHostUnregister(registered);
    if (staged) cudaFreeHost(staged);
  }
};

static int records_view(const void *records, uint64_t bytes, RecordsView *rv) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, records) != cudaSuccess) {
    cudaGetLastError();
    a.type = cudaMemoryTypeUnregistered;
  }
  if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) {
    rv->dev = (const uint32_t *)records;
    return GG_OK;
  }
  if (a.type == cudaMemoryTypeHost && a.devicePointer) {
    rv->dev = (const uint32_t *)a.devicePointer;
    return GG_OK;
  }
  void *p = const_cast<void *>(records);
  cudaError_t e = cudaHostRegister(p, bytes, cudaHostRegisterMapped | cudaHostRegisterReadOnly);
  if (e != cudaSuccess) {
    cudaGetLastError();
    e = cudaHostRegister(p, bytes, cudaHostRegisterMapped);
  }
  void *dp = nullptr;
  if (e == cudaSuccess) {
    rv->registered = p;
    GG_CUDA(cudaHostGetDevicePointer(&dp, p, 0));
  } else {
    // e.g. the range shares pages with memory registered elsewhere
    cudaGetLastError();
    GG_CUDA(cudaHostAlloc(&rv->staged, bytes, cudaHostAllocMapped));
    memcpy(rv->staged, records, bytes);
    GG_CUDA(cudaHostGetDevicePointer(&dp, rv->staged, 0));
  }
  rv->dev = (const uint32_t *)dp;
  return GG_OK;
}

static double wall_ms_since(const std::chrono::steady_clock::time_point &t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

static int graph_create_opts(int device, uint32_t V, int weighted, int symmetric, const gg_build_options *opt,
                             gg_graph **out) {
  GG_TRY(graph_create(device, V, weighted, symmetric, out));
  if (opt && opt->adjacency_host) {
    (*out)->adj_host = 1;
    (*out)->pr_layout = 0;
  }
  if (opt && (opt->force_partitions < 0 || opt->force_partitions > OC_MAX_FORCED)) {
    graph_destroy(*out);
    *out = nullptr;
    set_error("force_partitions must be in [0, %d]", OC_MAX_FORCED);
    return GG_ERR_INVALID;
  }
  return GG_OK;
}

int gg_graph_from_records_ex(const void *records, uint64_t bytes, uint32_t vertices, int weighted, int symmetric,
                             int device, gg_build_options *opt, gg_graph **out) {
  const auto t0 = std::chrono::steady_clock::now();
  uint64_t unit = unit_of(weighted);
  uint64_t E = bytes / unit;
  if (!out || (!records && E)) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  if ((uintptr_t)records % 4) {
    set_error("records must be 4-byte aligned");
    return GG_ERR_INVALID;
  }
  gg_graph *g = nullptr;
  GG_TRY(graph_create_opts(device, vertices, weighted, symmetric, opt, &g));
  bool part = false;
  uint64_t cap = 0, gcap = 0;
  int s = build_plan(g, E, false, opt, &part, &cap, &gcap);
  if (s == GG_OK && !part) {
    void *d = nullptr;
    cudaError_t e = cudaMalloc(&d, E * unit ? E * unit : 16);
    if (e == cudaSuccess && E) e = cudaMemcpy(d, records, E * unit, cudaMemcpyDefault);
    s = e == cudaSuccess ? build_records(g, (const uint32_t *)d, E, false, 0, 0, opt) : cuda_status(e, "copy records");
    if (d) cudaFree(d);
  } else if (s == GG_OK) {
    RecordsView rv;
    s = E ? records_view(records, E * unit, &rv) : GG_OK;
    if (s == GG_OK) s = build_records(g, rv.dev, E, true, cap, gcap, opt);
    cudaStreamSynchronize(g->stream);
  }
  if (s != GG_OK) {
    graph_destroy(g);
    return s;
  }
  if (opt) opt->build_ms = wall_ms_since(t0);
  *out = g;
  return GG_OK;
}

int gg_graph_from_records(const void *records, uint64_t bytes, uint32_t vertices, int weighted, int symmetric,
                          int device, gg_graph **out) {
  return gg_graph_from_records_ex(records, bytes, vertices, weighted, symmetric, device, nullptr, out);
}

// Reads [0, bytes) of fd into dst with several threads.
static int read_parallel(int fd, char *dst, uint64_t bytes, const char *path) {
  const int T = 8;
  const uint64_t per = (bytes / T + 4095) / 4096 * 4096;
  std::vector<std::thread> th;
  std::vector<int> bad(T, 0);
  for (int t = 0; t < T; t++) {
    const uint64_t a = per * t, b = std::min<uint64_t>(bytes, per * (t + 1));
    if (a >= b) break;
    th.emplace_back([=, &bad]() {
      uint64_t off = a;
      while (off < b) {
        const size_t want = (size_t)std::min<uint64_t>(b - off, (uint64_t)1 << 30);
        ssize_t r = pread(fd, dst + off, want, (off_t)off);
        if (r <= 0) {
          bad[t] = 1;
          return;
        }
        off += (uint64_t)r;
      }
    });
  }
  for (auto &x : th) x.join();
  for (int t = 0; t < T; t++)
    if (bad[t]) {
      set_error("read error on %s", path);
      return GG_ERR_IO;
    }
  return GG_OK;
}

int gg_graph_load(const char *path, uint32_t vertices, int weighted, int symmetric, int device, gg_graph **out) {
  return gg_graph_load_ex(path, vertices, weighted, symmetric, device, nullptr, out);
}

int gg_graph_load_ex(const char *path, uint32_t vertices, int weighted, int symmetric, int device,
                     gg_build_options *opt, gg_graph **out) {
  const auto t0 = std::chrono::steady_clock::now();
  if (!path || !out) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  int fd = open(path, O_RDONLY);
  if (fd < 0) {
    set_error("cannot open %s: %s", path, strerror(errno));
    return GG_ERR_IO;
  }
  struct stat st;
  if (fstat(fd, &st) != 0) {
    set_error("cannot stat %s: %s", path, strerror(errno));
    close(fd);
    return GG_ERR_IO;
  }
  uint64_t unit = unit_of(weighted);
  uint64_t E = (uint64_t)st.st_size / unit;
  uint64_t total = E * unit;
  gg_graph *g = nullptr;
  int s = graph_create_opts(device, vertices, weighted, symmetric, opt, &g);
  if (s != GG_OK) {
    close(fd);
    return s;
  }
  bool part = false;
  uint64_t cap = 0, gcap = 0;
  s = build_plan(g, E, false, opt, &part, &cap, &gcap);
  if (s == GG_OK && part) {
    // records stay in mapped pinned host memory, read by the build kernels
    char *h = nullptr;
    cudaError_t e = cudaHostAlloc((void **)&h, total ? total : 16, cudaHostAllocMapped);
    if (e != cudaSuccess) s = cuda_status(e, "pinned records");
    if (s == GG_OK) s = read_parallel(fd, h, total, path);
    close(fd);
    void *dp = nullptr;
    if (s == GG_OK) {
      e = cudaHostGetDevicePointer(&dp, h, 0);
      if (e != cudaSuccess) s = cuda_status(e, "pinned records");
    }
    if (s == GG_OK) s = build_records(g, (const uint32_t *)dp, E, true, cap, gcap, opt);
    cudaStreamSynchronize(g->stream);
    if (h) cudaFreeHost(h);
    if (s != GG_OK) {
      graph_destroy(g);
      return s;
    }
    if (opt) opt->build_ms = wall_ms_since(t0);
    *out = g;
    return GG_OK;
  }
  if (s != GG_OK) {
    close(fd);
    graph_destroy(g);
    return s;
  }
  // stream the file through two pinned chunks
  const size_t CH = (size_t)64 << 20;
  char *pin[2] = {nullptr, nullptr};
  cudaEvent_t done[2] = {nullptr, nullptr};
  char *d = nullptr;
  cudaError_t e = cudaMalloc((void **)&d, total ? total : 16);
  for (int i = 0; i < 2 && e == cudaSuccess; i++) {
    e = cudaMallocHost((void **)&pin[i], CH);
    if (e == cudaSuccess) e = cudaEventCreate(&done[i]);
  }
  if (e != cudaSuccess) s = cuda_status(e, "load buffers");
  uint64_t off = 0;
  int k = 0;
  while (s == GG_OK && off < total) {
    size_t want = (size_t)((total - off) < CH ? (total - off) : CH);
    e = cudaEventSynchronize(done[k]);
    if (e != cudaSuccess) {
      s = cuda_status(e, "load");
      break;
    }
    size_t got = 0;
    while (got < want) {
      ssize_t r = pread(fd, pin[k] + got, want - got, (off_t)(off + got));
      if (r <= 0) {
        set_error("read error on %s at %llu", path, (unsigned long long)(off + got));
        s = GG_ERR_IO;
        break;
      }
      got += (size_t)r;
    }
    if (s != GG_OK) break;
    e = cudaMemcpyAsync(d + off, pin[k], want, cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) e = cudaEventRecord(done[k], g->stream);
    if (e != cudaSuccess) {
      s = cuda_status(e, "load copy");
      break;
    }
    off += want;
    k ^= 1;
  }
  close(fd);
  cudaStreamSynchronize(g->stream);
  for (int i = 0; i < 2; i++) {
    if (pin[i]) cudaFreeHost(pin[i]);
    if (done[i]) cudaEventDestroy(done[i]);
  }
  if (s == GG_OK) s = build_records(g, (const uint32_t *)d, E, false, 0, 0, opt);
  if (d) cudaFree(d);
  if (s != GG_OK) {
    graph_destroy(g);
    return s;
  }
  if (opt) opt->build_ms = wall_ms_since(t0);
  *out = g;
  return GG_OK;
}

uint64_t gg_generate_count(int kind, uint32_t p1, uint32_t p2) {
  if (kind == 0) return p1 > 31 ? 0 : ((uint64_t)1 << p1) * p2;
  if (kind == 1) return gg_grid_count(p1);
  return 0;
}

int gg_generate_records(int kind, uint32_t p1, uint32_t p2, uint64_t seed, int weighted, void *records,
                        int threads) {
  uint64_t E = gg_generate_count(kind, p1, p2);
  if ((kind != 0 && kind != 1) || (kind == 0 && (p1 < 1 || p1 > 31)) || (!records && E)) {
    set_error("bad generator arguments");
    return GG_ERR_INVALID;
  }
  if (threads <= 0) threads = (int)std::thread::hardware_concurrency();
  if (threads <= 0) threads = 1;
  uint64_t key = gg_gen_key(seed);
  int words = weighted ? 3 : 2;
  uint32_t *rec = (uint32_t *)records;
  auto work = [&](uint64_t a, uint64_t b) {
    for (uint64_t e = a; e < b; e++) {
      uint32_t s, d;
      if (kind == 0)
        gg_rmat_edge(key, p1, e, &s, &d);
      else
        gg_grid_edge(p1, e, &s, &d);
      rec[e * words] = s;
      rec[e * words + 1] = d;
      if (weighted) {
        float w = gg_gen_weight(key, e);
        memcpy(&rec[e * words + 2], &w, 4);
      }
    }
  };
  std::vector<std::thread> pool;
  uint64_t chunk = (E + threads - 1) / threads;
  for (int t = 0; t < threads; t++) {
    uint64_t a = (uint64_t)t * chunk, b = a + chunk < E ? a + chunk : E;
    if (a >= b) break;
    pool.emplace_back(work, a, b);
  }
  for (auto &th : pool) th.join();
  return GG_OK;
}

int gg_graph_generate(int kind, uint32_t p1, uint32_t p2, uint64_t seed, int weighted, int symmetric, int device,
                      gg_graph **out) {
  return gg_graph_generate_ex(kind, p1, p2, seed, weighted, symmetric, device, nullptr, out);
}

int gg_graph_generate_ex(int kind, uint32_t p1, uint32_t p2, uint64_t seed, int weighted, int symmetric, int device,
                         gg_build_options *opt, gg_graph **out) {
  const auto t0 = std::chrono::steady_clock::now();
  uint64_t E = gg_generate_count(kind, p1, p2);
  uint32_t V;
  if (kind == 0 && p1 >= 1 && p1 <= 31) {
    V = 1u << p1;
  } else if (kind == 1 && p1 >= 1 && (uint64_t)p1 * p1 < 0xFFFFFFFFull) {
    V = p1 * p1;
  } else {
    set_error("bad generator arguments");
    return GG_ERR_INVALID;
  }
  if (!out) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  gg_graph *g = nullptr;
  GG_TRY(graph_create_opts(device, V, weighted, symmetric, opt, &g));
  uint32_t *d = nullptr;
  int words = weighted ? 3 : 2;
  cudaError_t e = cudaMalloc(&d, E ? E * words * 4 : 16);
  uint64_t key = gg_gen_key(seed);
  if (e == cudaSuccess && E) {
    unsigned blocks = grid_for(E, 256, g->num_sms, 32);
    if (kind == 0)
      gen_rmat_kernel<<<blocks, 256, 0, g->stream>>>(d, E, p1, key, weighted);
    else
      gen_grid_kernel<<<blocks, 256, 0, g->stream>>>(d, E, p1, key, weighted);
    e = cudaGetLastError();
  }
  bool part = false;
  uint64_t cap = 0, gcap = 0;
  int s = e == cudaSuccess ? build_plan(g, E, true, opt, &part, &cap, &gcap) : cuda_status(e, "generate");
  if (s == GG_OK) s = build_records(g, d, E, part, cap, gcap, opt);
  if (d) cudaFree(d);
  if (s != GG_OK) {
    graph_destroy(g);
    return s;
  }
  if (opt) opt->build_ms = wall_ms_since(t0);
  *out = g;
  return GG_OK;
}

int gg_graph_free(gg_graph *g) {
  graph_destroy(g);
  return GG_OK;
}

int gg_graph_info_get(const gg_graph *g, gg_graph_info *info) {
  if (!g || !info) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  info->vertices = g->V;
  info->edges = g->E;
  info->adj_entries = g->nadj;
  info->weighted = g->weighted;
  info->symmetric = g->symmetric;
  info->transposed = g->transposed;
  info->device = g->device;
  uint64_t ws_bytes = 0;
  for (int i = 0; i < WS_NSLOTS; i++) ws_bytes += g->ws.bytes[i];
  info->device_bytes = g->graph_bytes + ws_bytes;
  info->host_bytes = g->host_bytes;
  return GG_OK;
}

int gg_graph_transpose(gg_graph *g) {
  if (!g) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  pr_layout_free(g);
  Dir t = g->out;
  g->out = g->in;
  g->in = t;
  g->transposed ^= 1;
  return GG_OK;
}

int gg_graph_device_view(const gg_graph *g, int incoming, gg_device_adj *out) {
  if (!g || !out) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  const Dir &d = incoming ? g->in : g->out;
  out->offsets = d.off;
  out->neighbours = d.nbr;
  out->weights = d.w;
  out->degree = d.deg;
  out->vertices = g->V;
  out->entries = g->nadj;
  out->edges = g->E;
  out->device = g->device;
  return GG_OK;
}

int gg_graph_adjacency(const gg_graph *g, int incoming, uint64_t *offsets, uint32_t *neighbours, float *weights,
                       uint32_t *degree) {
  if (!g) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(g->device));
  const Dir &d = incoming ? g->in : g->out;
  if (offsets) GG_CUDA(cudaMemcpy(offsets, d.off, sizeof(uint64_t) * ((size_t)g->V + 1), cudaMemcpyDeviceToHost));
  if (neighbours && g->nadj)
    GG_CUDA(cudaMemcpy(neighbours, d.nbr, sizeof(uint32_t) * g->nadj, cudaMemcpyDefault));
  if (weights && g->weighted && g->nadj)
    GG_CUDA(cudaMemcpy(weights, d.w, sizeof(float) * g->nadj, cudaMemcpyDefault));
  if (degree) GG_CUDA(cudaMemcpy(degree, d.deg, sizeof(uint32_t) * g->V, cudaMemcpyDeviceToHost));
  return GG_OK;
}

int gg_is_sparse(uint64_t active_edges, uint64_t edges) { return active_edges < edges / 20 ? 1 : 0; }

const void *gg_result_device_ptr(const gg_graph *g, int which) {
  if (!g || which < 0 || which > 1) return nullptr;
  return g->result[which];
}

}  // extern "C"
