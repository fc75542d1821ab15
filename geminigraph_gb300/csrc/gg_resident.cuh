// Runs that stay on the device: one cooperative launch carries out many
// process_edges calls, a grid-wide barrier between their steps (1.2 us on
// GB300 from 8 to 600 blocks; a launch and a wait of the host take 9 us, and a
// host-driven call six to eight launches).  Used for whole traversals of
// graphs whose calls are shorter than that, and on large graphs for runs of
// consecutive small sparse calls.
//
// Every block keeps the run's state (queue length, switch value, which buffer
// is which) in registers and derives the next call's from the step's tally
// after the barrier, so all blocks agree on every branch.  Tallies rotate over
// three slots: step s adds to slot s % 3 and clears slot (s + 1) % 3, which
// was last read before the barrier before last.
#ifndef GG_RESIDENT_CUH
#define GG_RESIDENT_CUH

#include "gg_engine.cuh"

namespace gg {

constexpr int RES_THREADS = 256;
constexpr int RES_BLOCKS = 4;            // per SM, at most
constexpr uint32_t RES_CALLS = 1536;     // calls of one launch (trace rows)
constexpr uint32_t RES_HUB = 128;        // queued vertices with longer lists are cut into chunks of this
// On a graph too large for whole runs a call stays on the device up to this
// queue length and number of active edges.
constexpr uint32_t RES_MAX_QUEUE = 65536;
constexpr unsigned long long RES_MAX_AE = 1ull << 20;

struct ResRow {  // one call, written to host memory
  unsigned long long ae;
  uint32_t activated, mode;
};

// Where a run stands between two calls.
struct ResState {
  unsigned long long ae = 0;  // active_edges of the next call
  uint32_t n_act = 0;         // its active vertices
  uint32_t n = 0, hubs = 0;   // queue entries from the front, hubs from the back (qvalid)
  uint32_t calls = 0;         // calls made by this launch
  uint32_t role = 0;          // which state array is the one to read
  uint32_t q = 0, bm = 0;     // queue and bitmap of the active set
  uint32_t qvalid = 0;        // the queue holds the active set (else the bitmap does)
  uint32_t step = 0;          // the next step's tally slot (clear)
};

// What the host reads after a launch, in mapped host memory.
struct ResOut {
  ResState st;
  alignas(16) ResRow row[RES_CALLS];
};
static_assert(sizeof(ResRow) == 16, "rows move as 16-byte words");
constexpr size_t RES_OUT_BYTES = (sizeof(ResOut) + 255) / 256 * 256;
static_assert(RES_OUT_BYTES < STAGE_BYTES_HOST, "the run's rows fit the staging buffer");
constexpr size_t RES_RESULT_BYTES = STAGE_BYTES_HOST - RES_OUT_BYTES;  // small results go there too

struct ResTally {
  unsigned long long app, happ;  // queue and hub appends: count | out-degree sum << 32
  Counters c;                    // pulls; aux: a step's own result
};

// Appends v to the queue: one atomic per group of lanes that arrive together.
// Returns the place.
__device__ __forceinline__ uint32_t res_place(uint32_t od, unsigned long long *count) {
  const unsigned am = __activemask(), lane = lane_id();
  const int leader = __ffs(am) - 1;
  const unsigned sum = __reduce_add_sync(am, od);
  unsigned long long base = 0;
  if ((int)lane == leader)
    base = atomicAdd(count, (unsigned long long)__popc(am) | ((unsigned long long)sum << 32));
  return (uint32_t)__shfl_sync(am, (uint32_t)base, leader) + __popc(am & ((1u << lane) - 1u));
}
// Hubs from the back, q[cap - 1 - i].  Lanes may be divergent.
__device__ __forceinline__ void res_append(uint32_t v, uint32_t od, uint32_t *q, size_t cap, ResTally *slot) {
  if (od > RES_HUB)
    q[cap - 1 - res_place(od, &slot->happ)] = v;
  else
    q[res_place(od, &slot->app)] = v;
}

// A block's appends of one step, gathered in shared memory and placed with
// one atomic: a grid's call appends a thousand vertices from as many warps,
// and as many atomics on one counter take longer (10 us) than the call.
struct ResStage {
  static constexpr uint32_t CAP = 1024;
  uint32_t v[CAP];
  uint32_t n, sum, full, base;  // full: entries in place when a group did not fit any more
};
// Lanes may be divergent.
__device__ __forceinline__ void res_stage(uint32_t v, uint32_t od, ResStage &s, uint32_t *q, size_t cap,
                                          ResTally *slot) {
  if (od > RES_HUB) {
    q[cap - 1 - res_place(od, &slot->happ)] = v;
    return;
  }
  const unsigned am = __activemask(), lane = lane_id();
  const int leader = __ffs(am) - 1;
  const unsigned sum = __reduce_add_sync(am, od);
  uint32_t base = 0;
  if ((int)lane == leader) {
    base = atomicAdd(&s.n, (uint32_t)__popc(am));
    if (base + __popc(am) <= ResStage::CAP)
      atomicAdd(&s.sum, sum);
    else
      atomicMin(&s.full, base);  // these and all later groups go to the queue themselves
  }
  base = __shfl_sync(am, base, leader);
  if (base + __popc(am) <= ResStage::CAP)
    s.v[base + __popc(am & ((1u << lane) - 1u))] = v;
  else
    q[res_place(od, &slot->app)] = v;
}
// Once per block before its first step, and at the end of each step that
// stages; all threads call.
__device__ __forceinline__ void res_stage_init(ResStage &s) {
  if (threadIdx.x == 0) {
    s.n = 0;
    s.sum = 0;
    s.full = ResStage::CAP;
  }
}
__device__ __forceinline__ void res_stage_flush(ResStage &s, uint32_t *q, ResTally *slot) {
  __syncthreads();
  const uint32_t n = s.n < s.full ? s.n : s.full;
  if (n == 0) return;  // uniform
  if (threadIdx.x == 0)
    s.base = (uint32_t)atomicAdd(&slot->app, (unsigned long long)n | ((unsigned long long)s.sum << 32));
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += RES_THREADS) q[s.base + i] = s.v[i];
  res_stage_init(s);  // read again after the grid's barrier only
}

// f(src, k) for every out-edge k of every queued vertex, head(src) once per
// vertex.  Short lists: a group of lanes per vertex, about as many lanes as
// the lists have entries (ae in all), fewer where there are not enough
// threads; hubs: a warp per chunk of RES_HUB entries.
template <class Head, class Edge>
__device__ __forceinline__ void res_expand(const Dir &d, const uint32_t *q, uint32_t n, uint32_t hubs,
                                           unsigned long long ae, size_t cap, Head head, Edge f) {
  const size_t nthreads = (size_t)gridDim.x * RES_THREADS, tid = (size_t)blockIdx.x * RES_THREADS + threadIdx.x;
  const unsigned lane = lane_id();
  const unsigned long long total_n = (unsigned long long)n + hubs;
  const uint32_t group = ae > 16 * total_n && (size_t)n * 32 <= nthreads  ? 32u
                         : ae > 4 * total_n && (size_t)n * 8 <= nthreads ? 8u
                                                                         : 4u;
  const uint32_t sub = (uint32_t)(tid % group);
  for (size_t i = tid / group; i < n; i += nthreads / group) {
    const uint32_t src = q[i];
    const unsigned long long b = d.off[src], e = d.off[src + 1];
    const auto m = head(src, sub == 0);
    for (unsigned long long k = b + sub; k < e; k += group) f(m, src, k);
  }
  __syncwarp();
  const uint32_t nwarps = (uint32_t)(nthreads / 32), warp = (uint32_t)(tid / 32);
  for (size_t base = 0; base < hubs; base += 32) {
    uint32_t src = 0, chunks = 0;
    unsigned long long b = 0, e = 0;
    if (base + lane < hubs) {
      src = q[cap - 1 - (base + lane)];
      b = d.off[src];
      e = d.off[src + 1];
      chunks = (uint32_t)((e - b + RES_HUB - 1) / RES_HUB);
    }
    uint32_t incl = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(GG_FULL, incl, o);
      if (lane >= (unsigned)o) incl += y;
    }
    const uint32_t total = __shfl_sync(GG_FULL, incl, 31);
    for (uint32_t c = warp; c < total; c += nwarps) {
      const int j = __ffs(__ballot_sync(GG_FULL, incl > c)) - 1;
      const uint32_t part = c - __shfl_sync(GG_FULL, incl - chunks, j);
      const uint32_t sj = __shfl_sync(GG_FULL, src, j);
      const unsigned long long bj = __shfl_sync(GG_FULL, b, j), ej = __shfl_sync(GG_FULL, e, j);
      const auto m = head(sj, lane == 0 && part == 0);
      const unsigned long long k0 = bj + (unsigned long long)part * RES_HUB;
#pragma unroll
      for (uint32_t i = 0; i < RES_HUB; i += 32)
        if (k0 + i + lane < ej) f(m, sj, k0 + i + lane);
      __syncwarp();
    }
  }
}

// The queue of the bits of bm (hubs apart); a warp per 32 words.
__device__ __forceinline__ void res_queue_from_bitmap(const uint32_t *bm, size_t words, const uint32_t *out_deg,
                                                      uint32_t *q, size_t cap, ResTally *slot) {
  const uint32_t nwarps = gridDim.x * (RES_THREADS / 32), warp = (blockIdx.x * RES_THREADS + threadIdx.x) / 32;
  const unsigned lane = lane_id();
  for (size_t g = warp; g * 32 < words; g += nwarps) {
    const uint32_t w = g * 32 + lane < words ? bm[g * 32 + lane] : 0u;
    for (unsigned any = __ballot_sync(GG_FULL, w != 0); any; any &= any - 1) {
      const int j = __ffs(any) - 1;
      const uint32_t wj = __shfl_sync(GG_FULL, w, j);
      if ((wj >> lane) & 1u) {
        const uint32_t v = (uint32_t)((g * 32 + j) * 32 + lane);
        res_append(v, out_deg[v], q, cap, slot);
      }
      __syncwarp();
    }
  }
}

// The queue without its degree-0 vertices and with its hubs, as the
// host-driven kernels take it.
__device__ __forceinline__ void res_plain_queue(const uint32_t *q, uint32_t n, uint32_t hubs, size_t cap,
                                                const uint32_t *out_deg, uint32_t *to, ResTally *slot) {
  const size_t nthreads = (size_t)gridDim.x * RES_THREADS, total = (size_t)n + hubs;
  for (size_t i = (size_t)blockIdx.x * RES_THREADS + threadIdx.x; i < (total + 31) / 32 * 32; i += nthreads) {
    const uint32_t v = i < n ? q[i] : i < total ? q[cap - 1 - (i - n)] : 0u;
    const bool keep = i < total && out_deg[v] > 0;
    const unsigned b = __ballot_sync(GG_FULL, keep);
    unsigned long long base = 0;
    if (b && lane_id() == 0) base = atomicAdd(&slot->app, (unsigned long long)__popc(b));
    const uint32_t at = (uint32_t)__shfl_sync(GG_FULL, base, 0);
    if (keep) to[at + __popc(b & lanemask_lt())] = v;
  }
}

// A tally slot after the barrier (written by atomics of other SMs).
__device__ __forceinline__ unsigned long long res_read(const unsigned long long *p) {
  return *(const volatile unsigned long long *)p;
}
__device__ __forceinline__ uint32_t res_read(const uint32_t *p) { return *(const volatile uint32_t *)p; }

__device__ __forceinline__ void res_clear(ResTally *slot) {
  if (blockIdx.x == 0 && threadIdx.x < sizeof(ResTally) / 4) ((uint32_t *)slot)[threadIdx.x] = 0u;
}

// The end of a launch: its state and rows to the host (not as the calls end:
// a barrier waits for the stores before it, and these take the host's link).
__device__ __forceinline__ void res_report(const ResState &st, const ResRow *rows, ResOut *out) {
  if (blockIdx.x != 0) return;
  __syncthreads();
  const uint4 *from = reinterpret_cast<const uint4 *>(rows);
  uint4 *to = reinterpret_cast<uint4 *>(out->row);
  for (uint32_t i = threadIdx.x; i < st.calls; i += RES_THREADS) to[i] = from[i];
  if (threadIdx.x == 0) out->st = st;
}

// Up to this many entries a dense SSSP call of a whole run pushes (R-MAT
// graphs of 2^16 / 2^18 / 2^20 entries: 279 / 451 / 1322 us pushing, 325 / 333
// / 463 us pulling: the hubs' atomics).
constexpr unsigned long long RES_PUSH_ALL = 1ull << 17;

// Tally slots, call rows and a word in the graph's workspace.  Every launch
// leaves the slot that the next one's first step uses clear (ResState::step,
// kept in g->res_step), so they are set to zero only when they are new.
inline int res_buffers(gg_graph *g, ResTally **slots, ResRow **rows, uint32_t **word) {
  char *blob = nullptr;
  const size_t head = (3 * sizeof(ResTally) + 16 + 255) / 256 * 256;
  GG_TRY(ws(g, WS_RES, head + sizeof(ResRow) * RES_CALLS, &blob));
  if (g->res_step < 0) {
    GG_CUDA(cudaMemsetAsync(blob, 0, head, g->stream));
    g->res_step = 0;
  }
  *slots = (ResTally *)blob;
  *word = (uint32_t *)(blob + 3 * sizeof(ResTally));
  *rows = (ResRow *)(blob + head);
  return GG_OK;
}

// A resident kernel's cooperative launch, recorded as the timed region's end;
// waits for it.  `in` is its starting state among the arguments; the final
// one is in g->ws.stage.
inline int res_launch(gg_graph *g, const void *kernel, unsigned blocks, void **args, ResState *in, Launch *L) {
  in->step = (uint32_t)g->res_step;
  g->res_step = -1;  // unless the launch ends
  GG_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(RES_THREADS), args, 0, g->stream));
  L->launches += 1;
  GG_CUDA(cudaEventRecord(g->ev1, g->stream));
  GG_CUDA(cudaEventSynchronize(g->ev1));
  g->res_step = (int)((const ResOut *)g->ws.stage)->st.step;
  return GG_OK;
}
// The launch's calls as trace rows.
inline void res_trace(const gg_graph *g, Trace &tr) {
  const ResOut *o = (const ResOut *)g->ws.stage;
  for (uint32_t r = 0; r < o->st.calls; r++) tr.add((int)o->row[r].mode, o->row[r].ae, o->row[r].activated);
}
// Blocks of a run.  The barrier costs the same for 8 as for 600; fewer suit
// graphs with little work per call, tiny ones and those of low degree, whose
// frontiers stay narrow (SSSP with one block per SM and with four: 400 x 400
// grid 3.4 and 4.7 ms, 1024 x 1024 grid 21.9 and 16.0; R-MAT 16 533 and 446 us).
inline unsigned res_blocks(const gg_graph *g) {
  const bool narrow = g->nadj <= (1ull << 15) || (g->nadj <= 6ull * g->V && g->nadj <= (1ull << 20));
  return (unsigned)g->num_sms * (narrow ? 1 : RES_BLOCKS);
}

}  // namespace gg

#endif
