// BFS (toolkits/bfs.cpp) and PageRank (toolkits/pagerank.cpp) on the
// device engine, plus the process_vertices reduction of the switch.
#include <string.h>

#include "gg_engine.cuh"
#include "gg_resident.cuh"

namespace gg {

// ------------------------------------------------------------------ BFS
// Sparse slot (bfs.cpp:49-59): claim unvisited dst with a CAS on its parent.
struct BfsPush {
  uint32_t *parent;
  uint32_t V;
  static constexpr bool kClaims = true;  // the order of the edges picks the parents (see small pushes)
  // visited bits are set right after a vertex's parent: most already-reached
  // targets are turned away by this L2-resident bitmap, not by a random read
  // of the parent array; parent (then the CAS) stays the authority
  const uint32_t *visited;
  __device__ __forceinline__ bool push(uint32_t src, uint32_t, uint32_t dst, float) const {
    if (visited && bm_test(visited, dst)) return false;
    if (*(volatile uint32_t *)(parent + dst) != V) return false;
    return atomicCAS(parent + dst, V, src) == V;
  }
};

// ------------------------------------------------------------------ small pushes
// Consecutive sparse calls whose frontiers are small (high-diameter graphs
// such as grids, the first and last calls of a power-law BFS) run in one
// cooperative launch (push_small_coop).
//
// The tree's parents depend on how these kernels and push_lb take the edges:
// of several sources that reach a vertex in one call the first to claim it is
// its parent, and on a quiet GPU that is the same one in every run.  Kernels
// that spread the edges wider (gg_resident.cuh's) were 2.6 times as fast on
// 4096 vertices and picked other, equally valid parents for 4% of them;
// callers who compare trees would see that, so the pushes stay as they are,
// code and launch shape.
constexpr int SMALL_THREADS = 256;
constexpr uint32_t SMALL_BATCH = 512;        // calls enqueued per host round trip
constexpr uint32_t SMALL_MAX_QUEUE = 65536;  // largest queue a small call takes
constexpr unsigned long long SMALL_MAX_AE = 1ull << 20;
constexpr uint32_t SMALL_MAX_DEG = 1024;     // largest out-degree in a small call's queue
constexpr int COOP_BLOCKS = 32;              // blocks of a cooperative small run (all resident)

struct SmallRun {
  unsigned long long ae;         // active_edges of the call about to run
  unsigned long long edges_lim;  // edges / 20
  unsigned long long total_ae;   // sum of active_edges over the run's calls
  unsigned int n;                // its queue length
  unsigned int go;               // the next launch runs a call
  unsigned int calls;            // trace rows written in this batch
  unsigned int level;            // activation stamp of the current call (> 0)
  unsigned int ticket;           // blocks finished in the current call
  unsigned int last_activated;   // activated count of the last call
  unsigned int maxdeg;           // largest out-degree in the queue of the call about to run
  Counters next;                 // accumulators of the current call
};

// Queue append from divergent lanes: one atomic per group of lanes that
// reach this point together.
__device__ __forceinline__ void queue_append_any(uint32_t v, uint32_t *q, unsigned *qlen) {
  const unsigned am = __activemask();
  const int leader = __ffs(am) - 1;
  const unsigned lane = lane_id();
  unsigned base = 0;
  if ((int)lane == leader) base = atomicAdd(qlen, (unsigned)__popc(am));
  base = __shfl_sync(am, base, leader);
  q[base + __popc(am & ((1u << lane) - 1u))] = v;
}

// Activation inside a small push call: stamp-deduplicated unless the op's
// slot already lets one thread win (BFS's CAS).  Lanes may be divergent.
template <bool kUnique>
__device__ __forceinline__ void small_activate_t(uint32_t v, Counters *tally, uint32_t *stamp, unsigned level,
                                                 uint32_t *visited, uint32_t *q_out, const uint32_t *out_deg,
                                                 const uint32_t *in_deg, Tally &t) {
  if (!kUnique) {
    if (stamp[v] == level || atomicExch(stamp + v, level) == level) return;
  }
  if (visited) atomicOr(visited + (v >> 5), 1u << (v & 31));
  uint32_t od = out_deg[v];
  t.activated += 1;
  t.edges += od;
  t.maxdeg = od > t.maxdeg ? od : t.maxdeg;
  if (in_deg) t.in_edges += in_deg[v];
  if (od > 0) queue_append_any(v, q_out, &tally->qlen);
}
template <class Op, bool kUnique>
__device__ __forceinline__ void small_call_t(Counters *tally, const uint32_t *__restrict__ q_in,
                                             uint32_t *__restrict__ q_out, const Dir &d, const Op &op,
                                             uint32_t *stamp, uint32_t *visited,
                                             const uint32_t *__restrict__ out_deg,
                                             const uint32_t *__restrict__ in_deg, uint32_t n, unsigned level) {
  const unsigned lane = lane_id();
  Tally t;
  const size_t nround = ((size_t)n + 31) / 32 * 32;
  for (size_t i = (size_t)blockIdx.x * SMALL_THREADS + threadIdx.x; i < nround; i += (size_t)gridDim.x * SMALL_THREADS) {
    const bool valid = i < n;
    uint32_t src = 0;
    unsigned long long b = 0, e = 0;
    if (valid) {
      src = q_in[i];
      b = d.off[src];
      e = d.off[src + 1];
    }
    if (valid && e - b <= LIGHT_DEG) {
      for (unsigned long long k = b; k < e; k++) {
        uint32_t dst = nbr_at(d, k, GG_SITE);
        if (op.push(src, (uint32_t)i, dst, d.w ? d.w[k] : 0.0f))
          small_activate_t<kUnique>(dst, tally, stamp, level, visited, q_out, out_deg, in_deg, t);
      }
    }
    unsigned coop = __ballot_sync(GG_FULL, valid && e - b > LIGHT_DEG);
    while (coop) {
      const unsigned leader = __ffs(coop) - 1;
      coop &= coop - 1;
      const unsigned long long lb = __shfl_sync(GG_FULL, b, leader), le = __shfl_sync(GG_FULL, e, leader);
      const uint32_t lsrc = __shfl_sync(GG_FULL, src, leader);
      const uint32_t li = (uint32_t)__shfl_sync(GG_FULL, (unsigned long long)i, leader);
      for (unsigned long long k = lb + lane; k < le; k += 32) {
        uint32_t dst = nbr_at(d, k, GG_SITE);
        if (op.push(lsrc, li, dst, d.w ? d.w[k] : 0.0f))
          small_activate_t<kUnique>(dst, tally, stamp, level, visited, q_out, out_deg, in_deg, t);
      }
    }
  }
  t.flush(tally);
}

// One cooperative launch: up to max_calls calls, the
// queues alternating (qa -> qb, then qb -> qa, ...), one grid-wide barrier
// per call.  Call c's tally goes to tally[c % 3]; after the barrier every
// block reads it and derives the next call's queue length, switch value and
// whether it runs (identical in all blocks, so all leave the loop together);
// block 0 writes the trace row and clears tally[(c + 1) % 3], which no block
// reads any more (the last reads were before the previous barrier).
template <class Op, bool kUnique>
__global__ void __launch_bounds__(SMALL_THREADS)
    push_small_coop(SmallRun *st, Counters *tally, uint32_t *qa, uint32_t *qb, Dir d, Op op, uint32_t *stamp,
                    uint32_t *visited, const uint32_t *__restrict__ out_deg, const uint32_t *__restrict__ in_deg,
                    unsigned long long *tr_ae, unsigned int *tr_act, unsigned max_calls) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  unsigned n = st->n, level = st->level, go = st->go, maxdeg = st->maxdeg, na = 0;
  unsigned long long ae = st->ae, total = st->total_ae;
  const unsigned long long lim = st->edges_lim;
  unsigned c = 0;
  for (; c < max_calls && go; c++) {
    Counters *cur = tally + (c % 3);
    if (blockIdx.x == 0 && threadIdx.x == 0) memset(tally + ((c + 1) % 3), 0, sizeof(Counters));
    small_call_t<Op, kUnique>(cur, (c & 1) ? qb : qa, (c & 1) ? qa : qb, d, op, stamp, visited, out_deg, in_deg, n,
                              level);
    grid.sync();
    const unsigned long long ne = *(volatile unsigned long long *)&cur->edges;
    na = *(volatile unsigned *)&cur->activated;
    const unsigned nq = *(volatile unsigned *)&cur->qlen;
    const unsigned nm = *(volatile unsigned *)&cur->maxdeg;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      tr_ae[c] = ae;
      tr_act[c] = na;
    }
    total += ae;
    level += 1;
    ae = ne;
    n = nq;
    maxdeg = nm;
    go = (na > 0 && ne < lim && nq <= SMALL_MAX_QUEUE && ne <= SMALL_MAX_AE && nm <= SMALL_MAX_DEG) ? 1u : 0u;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->calls = c;
    st->total_ae = total;
    st->level = level;
    st->ae = ae;
    st->n = n;
    st->last_activated = na;
    st->maxdeg = maxdeg;
    st->go = go;
    __threadfence();
  }
}

// Host and device view of a run: its state, the calls' rows, the tallies.
struct SmallBlob {
  SmallRun st;
  unsigned long long ae[SMALL_BATCH];
  unsigned int act[SMALL_BATCH];
  Counters tally[3];
};
static_assert(sizeof(SmallBlob) < STAGE_BYTES_HOST, "a run is read back in one piece");

static __host__ __device__ __forceinline__ SmallRun small_state(unsigned long long ae, unsigned long long lim, uint32_t n,
                                                                uint32_t go, uint32_t maxdeg) {
  SmallRun st;
  memset(&st, 0, sizeof(st));
  st.ae = ae;
  st.edges_lim = lim;
  st.n = n;
  st.go = go;
  st.maxdeg = maxdeg;
  st.level = 1;
  return st;
}
static __host__ __device__ __forceinline__ bool small_ok(uint32_t nq, unsigned long long ae, uint32_t maxdeg) {
  return ae > 0 && nq <= SMALL_MAX_QUEUE && ae <= SMALL_MAX_AE && maxdeg <= SMALL_MAX_DEG;
}

// A run's starting state, for one that the host begins.
__global__ void small_begin(SmallBlob *blob, SmallRun st) {
  blob->st = st;
  memset(&blob->tally[0], 0, sizeof(Counters));
}

// A traversal's start in one launch: parents, visited, the root's queue and
// the first small run's state (go: the first call is a small sparse one).
__global__ void bfs_begin(uint32_t *parent, uint32_t V, uint32_t *visited, size_t words, uint32_t root, uint32_t *q,
                          const uint32_t *out_deg, SmallBlob *blob, unsigned long long first_lim,
                          unsigned long long lim) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  for (size_t v = tid; v < V; v += stride) parent[v] = v == root ? root : V;
  for (size_t i = tid; i < words; i += stride) visited[i] = i == root >> 5 ? 1u << (root & 31) : 0u;
  if (tid == 0) {
    const uint32_t od = out_deg[root];
    q[0] = root;
    blob->st = small_state(od, lim, 1, od < first_lim && small_ok(1, od, od) ? 1u : 0u, od);
    memset(&blob->tally[0], 0, sizeof(Counters));
  }
}

// ------------------------------------------------------------------ dense runs
// Consecutive dense calls in one cooperative launch (gg_resident.cuh), entered
// with a queue and left with one, in vertex order as queue_from_bitmap's.  Of
// three bitmaps a call reads the frontier's, writes a clean one and cleans the
// third.  Whole BFS with host-launched dense calls and with these: R-MAT 16 /
// 20 / 22 / 24 305 / 344 / 396 / 829 us and 245 / 300 / 348 / 792.
struct DenseArgs {
  Dir out, in;
  uint32_t *parent, *visited;
  const uint32_t *q_in;
  uint32_t *q_out, *bm[3];
  unsigned long long *first;      // per heavy in-list vertex: the first hit
  uint32_t *seg;                  // per block: its part of the queue
  ResTally *slots;
  ResRow *rows;
  ResOut *out_host;
  unsigned long long edges_lim;   // the reference's switch: edges / 20
  unsigned long long pull_lim;    // pull from this many active edges on
  uint32_t V;
};
constexpr int DENSE_BLOCKS = 5;   // per SM

// bfs_walk for graphs with fewer vertices than lanes: a warp per vertex, so
// that no lane walks a list by itself (4096 vertices: 54 us for two calls with
// bfs_walk).  The same order within a list, whatever its length.
__device__ __forceinline__ void bfs_walk_wide(const Dir &d, uint32_t V, const uint32_t *active_in, uint32_t *parent,
                                              const ActOut &act, Tally &t, size_t warp, size_t nwarps) {
  const unsigned lane = lane_id();
  for (size_t v = warp; v < V; v += nwarps) {
    if (bm_test(act.visited, (uint32_t)v) || !bm_test(d.nz, (uint32_t)v)) continue;
    const unsigned long long b = d.off[v], e = d.off[v + 1];
    uint32_t hit = NONE32;
    for (unsigned long long base = b; base < e && hit == NONE32; base += 64) {
      const unsigned long long k = base + lane;
      uint32_t s0 = 0, s1 = 0;
      bool h0 = false, h1 = false;
      if (k < e) s0 = nbr_at(d, k, GG_SITE);
      if (k + 32 < e) s1 = nbr_at(d, k + 32, GG_SITE);
      if (k < e) h0 = bm_test(active_in, s0);
      if (k + 32 < e) h1 = bm_test(active_in, s1);
      const unsigned m0 = __ballot_sync(GG_FULL, h0), m1 = __ballot_sync(GG_FULL, h1);
      if (m0)
        hit = __shfl_sync(GG_FULL, s0, __ffs(m0) - 1);
      else if (m1)
        hit = __shfl_sync(GG_FULL, s1, __ffs(m1) - 1);
    }
    if (lane == 0 && hit != NONE32) {
      const uint32_t od = act.out_deg[v], bit = 1u << (v & 31);
      parent[v] = hit;
      atomicOr(act.active_out + (v >> 5), bit);
      atomicOr(act.visited + (v >> 5), bit);
      t.activated += 1;
      t.edges += od;
      t.maxdeg = od > t.maxdeg ? od : t.maxdeg;
    }
  }
}

// Up to this many vertices: larger graphs' dense calls are long enough to be
// launched one by one, with the walk's registers to themselves (whole call, one
// launch / one by one: R-MAT 26 2.54 / 2.37 ms, R-MAT 24 0.83 / 0.84, R-MAT 20
// 0.27 / 0.33, 8 M vertices uniform 1.05 / 1.08).
constexpr uint32_t DENSE_RUN_MAX = 1u << 24;

// On return st.n is the queue's length, st.hubs the largest out-degree in it.
__global__ void __launch_bounds__(RES_THREADS, DENSE_BLOCKS) bfs_dense_run(DenseArgs p, ResState st) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const uint32_t V = p.V;
  const size_t words = 2 * ((size_t)V / 64 + 1);
  const size_t nthreads = (size_t)gridDim.x * RES_THREADS, tid = (size_t)blockIdx.x * RES_THREADS + threadIdx.x;
  uint32_t step = st.step;
  uint32_t f = 0, clean = 1;
  for (size_t i = tid; i < words; i += nthreads) p.bm[0][i] = p.bm[1][i] = p.bm[2][i] = 0u;
  for (size_t h = tid; h < p.in.nheavy; h += nthreads) p.first[h] = ~0ull;
  grid.sync();
  for (size_t i = tid; i < st.n; i += nthreads) {
    const uint32_t v = p.q_in[i];
    atomicOr(p.bm[0] + (v >> 5), 1u << (v & 31));
  }
  grid.sync();
  st.calls = 0;
  do {
    res_clear(p.slots + (step + 1) % 3);
    ResTally *slot = p.slots + step % 3;
    const uint32_t third = 3 - f - clean;
    for (size_t i = tid; i < words; i += nthreads) p.bm[third][i] = 0u;
    ActOut act;
    act.active_out = p.bm[clean];
    act.visited = p.visited;
    act.out_deg = p.out.deg;
    Tally t;
    const bool wide = V <= nthreads;
    if (wide)
      bfs_walk_wide(p.in, V, p.bm[f], p.parent, act, t, tid / 32, nthreads / 32);
    else
      bfs_walk<2>(p.in, V, p.bm[f], p.parent, act, t, tid / 32, nthreads / 32);
    if (!wide && p.in.nheavy) {
      bfs_heavy_walk(p.in, p.bm[f], p.visited, p.first);
      grid.sync();
      bfs_heavy_take(p.in, p.first, p.parent, act, t);
    }
    t.flush(&slot->c);
    grid.sync();
    const unsigned long long ae = st.ae;
    st.n_act = res_read(&slot->c.activated);
    st.ae = res_read(&slot->c.edges);
    st.hubs = res_read(&slot->c.maxdeg);
    step++;
    f = clean;
    clean = third;
    if (tid == 0) p.rows[st.calls] = ResRow{ae, st.n_act, ae < p.edges_lim ? 0u : 1u};
    st.calls++;
  } while (st.n_act > 0 && st.ae >= p.pull_lim && st.calls < RES_CALLS);
  st.n = 0;
  if (st.n_act > 0) {
    // the queue: a block takes consecutive words, its place is the sum of the
    // counts of the blocks before it
    const size_t per = (words + gridDim.x - 1) / gridDim.x;
    const size_t lo = per * blockIdx.x < words ? per * blockIdx.x : words, hi = lo + per < words ? lo + per : words;
    const uint32_t *bm = p.bm[f], *nz = p.out.nz;
    uint32_t cnt = 0;
    for (size_t i = lo + threadIdx.x; i < hi; i += RES_THREADS) cnt += __popc(bm[i] & nz[i]);
    uint32_t excl;
    const uint32_t own = block_exclusive_scan<uint32_t>(cnt, &excl);
    if (threadIdx.x == 0) p.seg[blockIdx.x] = own;
    grid.sync();
    uint32_t below = 0, all = 0;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += RES_THREADS) {
      const uint32_t x = res_read(p.seg + i);
      all += x;
      if (i < blockIdx.x) below += x;
    }
    uint32_t at = block_exclusive_scan<uint32_t>(below, &excl);
    st.n = block_exclusive_scan<uint32_t>(all, &excl);
    for (size_t base = lo; base < hi; base += RES_THREADS) {
      const size_t i = base + threadIdx.x;
      uint32_t w = i < hi ? bm[i] & nz[i] : 0u;
      const uint32_t tot = block_exclusive_scan<uint32_t>((uint32_t)__popc(w), &excl);
      for (uint32_t o = at + excl; w; w &= w - 1) p.q_out[o++] = (uint32_t)(i * 32 + __ffs(w) - 1);
      at += tot;
    }
  }
  st.step = step % 3;
  res_report(st, p.rows, p.out_host);
}
// parent_slot: the workspace array the parent tree is written to (the
// pipelined calls alternate between two).
static int bfs_run(gg_graph *g, uint32_t root, uint32_t *parent_host, gg_run_stats *st, WsSlot parent_slot = WS_S0) {
  if (root >= g->V) {
    set_error("root %u >= vertices %u", root, g->V);
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(g->device));
  const uint32_t V = g->V;
  const size_t words = bitmap_words32(V);
  uint32_t *parent, *visited, *bm[2], *q[2];
  SmallBlob *blob;
  GG_TRY(ws(g, parent_slot, V, &parent));
  GG_TRY(ws(g, WS_BM0, words, &visited));
  GG_TRY(ws(g, WS_BM1, words, &bm[0]));
  GG_TRY(ws(g, WS_BM2, words, &bm[1]));
  GG_TRY(ws(g, WS_Q0, (size_t)V + 1, &q[0]));
  GG_TRY(ws(g, WS_Q1, (size_t)V + 1, &q[1]));
  GG_TRY(ws(g, WS_SMALL, 1, &blob));
  Launch L(g);
  Trace tr(st, g, "gg_bfs");
  cudaStream_t s = g->stream;
  Counters *ctr = g->ws.ctr;
  const bool coop = L.coop_ok() && g->ws.stage;
  const bool dense_runs = coop && !(st && st->call_ms) && g->V <= DENSE_RUN_MAX;
  // the reference's mode (core/graph.hpp:1503-1509), recorded in the trace;
  // the kernel that runs follows g->bfs_pull_div (any in-neighbour on the
  // frontier is a valid parent, so the levels do not depend on it)
  const unsigned long long lim = g->E / 20, pull_lim = g->E / g->bfs_pull_div;
  // small runs stop at the nearer of the two
  const unsigned long long small_lim = lim < pull_lim ? lim : pull_lim;
  unsigned long long ae = 0;
  uint32_t n_act = 1, nq = 1, md = 0;
  bool qvalid = true;  // q[cur] holds the active vertices with out-degree > 0
  int cur = 0;
  // Carries out the small run whose state is in *blob, as many launches as it takes.
  auto small_run = [&]() -> int {
    static thread_local SmallBlob host;
    SmallRun *sr = &blob->st;
    Counters *tally = blob->tally;
    unsigned long long *tr_ae = blob->ae;
    unsigned *tr_act = blob->act, batch = SMALL_BATCH;
    for (;;) {
      uint32_t *qa = q[cur], *qb = q[cur ^ 1], *stamp = nullptr;
      Dir d = g->out;
      BfsPush op{parent, V, visited};
      const uint32_t *deg = g->out.deg, *in_deg = nullptr;
      void *args[] = {&sr,       &tally, &qa,    &qb,    &d,    &op, &stamp, &visited, (void *)&deg, (void *)&in_deg,
                      &tr_ae, &tr_act, &batch};
      GG_CUDA(cudaLaunchCooperativeKernel((const void *)push_small_coop<BfsPush, true>, dim3(COOP_BLOCKS),
                                          dim3(SMALL_THREADS), args, 0, s));
      L.launches += 1;
      GG_TRY(read_small(g, &host, blob, sizeof(SmallBlob)));
      const SmallRun &h = host.st;
      for (uint32_t r = 0; r < h.calls; r++) tr.add(0, host.ae[r], host.act[r]);
      cur ^= (int)(h.calls & 1);
      if (h.calls) n_act = h.last_activated;
      ae = h.ae;
      nq = h.n;
      md = h.maxdeg;
      if (!h.go) return GG_OK;
      small_begin<<<1, 1, 0, s>>>(blob, small_state(ae, lim, nq, 1, md));  // the batch ended with the run still going
      L.launches += 1;
    }
  };
  Prefault pages(parent_host, sizeof(uint32_t) * V);
  GG_TRY(timed_begin(g));
  bfs_begin<<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(parent, V, visited, words, root, q[0], g->out.deg, blob,
                                                        coop ? small_lim : 0ull, lim);
  L.launches += 1;
  GG_CUDA(cudaGetLastError());
  bool bits = false;       // bm[cur] holds the frontier too
  bool from_pull = false;  // the call before was a pull: the next push is push_lb's (see small pushes)
  if (coop) {
    GG_TRY(small_run());
  } else {
    SmallRun h;
    GG_TRY(read_small(g, &h, &blob->st, sizeof(h)));
    ae = h.ae;
    md = h.maxdeg;
  }
  while (n_act > 0) {
    const bool sparse = ae < lim, push = ae < pull_lim;
    if (coop && sparse && push && qvalid && !from_pull && small_ok(nq, ae, md)) {
      // consecutive small sparse calls run on the device without host round trips
      small_begin<<<1, 1, 0, s>>>(blob, small_state(ae, lim, nq, 1, md));
      L.launches += 1;
      GG_CUDA(cudaGetLastError());
      GG_TRY(small_run());
      bits = false;
      continue;
    }
    if (!push && qvalid && dense_runs) {
      DenseArgs p{};
      p.out = g->out;
      p.in = g->in;
      p.parent = parent;
      p.visited = visited;
      p.q_in = q[cur];
      p.q_out = q[cur ^ 1];
      p.bm[0] = bm[0];
      p.bm[1] = bm[1];
      GG_TRY(ws(g, WS_BM3, words, &p.bm[2]));
      GG_TRY(ws(g, WS_PARTIAL, g->in.nheavy, &p.first));
      GG_TRY(ws(g, WS_QPOS, (size_t)g->num_sms * DENSE_BLOCKS, &p.seg));
      uint32_t *word = nullptr;
      GG_TRY(res_buffers(g, &p.slots, &p.rows, &word));
      p.out_host = (ResOut *)g->ws.stage;
      p.edges_lim = lim;
      p.pull_lim = pull_lim;
      p.V = V;
      ResState in;
      in.ae = ae;
      in.n_act = n_act;
      in.n = nq;
      void *args[] = {&p, &in};
      const unsigned blocks = (unsigned)g->num_sms * DENSE_BLOCKS;
      GG_TRY(res_launch(g, (const void *)bfs_dense_run, blocks, args, &in, &L));
      const ResState out = ((const ResOut *)g->ws.stage)->st;
      res_trace(g, tr);
      ae = out.ae;
      n_act = out.n_act;
      nq = out.n;
      md = out.hubs;
      cur ^= 1;
      bits = false;
      from_pull = true;
      continue;
    }
    if (!push && qvalid && !bits) {  // the frontier is q[cur]
      GG_CUDA(cudaMemsetAsync(bm[cur], 0, words * 4, s));
      if (nq) bitmap_from_queue<<<grid_for(nq, 256, g->num_sms), 256, 0, s>>>(q[cur], nq, bm[cur]);
      L.launches += 1;
    }
    tr.add(sparse ? 0 : 1, ae, 0);
    int nx = cur ^ 1;
    if (push && ae > 0 && !qvalid) GG_TRY(L.queue_from_bitmap(bm[cur], g->out.nz, q[cur], &nq));
    GG_CUDA(cudaMemsetAsync(bm[nx], 0, words * 4, s));
    GG_TRY(counters_reset(g));
    ActOut a;
    a.active_out = bm[nx];
    a.visited = visited;
    a.q_out = push ? q[nx] : nullptr;
    a.qlen = &ctr->qlen;
    a.out_deg = g->out.deg;
    a.queue_nonzero_only = true;
    if (push) {
      if (ae > 0) {
        unsigned long long *P;
        GG_TRY(L.scan_queue_degrees(q[cur], nq, g->out.deg, &P));
        GG_TRY(tr.kbegin());
        push_lb<BfsPush><<<L.push_grid(ae), PUSH_THREADS, 0, s>>>(q[cur], P, nq, ae, g->out, BfsPush{parent, V, visited},
                                                                    a, ctr);
        GG_TRY(tr.kend());
        L.launches += 1;
      }
    } else {
      GG_TRY(tr.kbegin());
      GG_TRY(L.bfs_pull(g->in, bm[cur], parent, a, ctr));
      GG_TRY(tr.kend());
    }
    GG_CUDA(cudaGetLastError());
    Counters c;
    GG_TRY(counters_read(g, &c));
    n_act = c.activated;
    nq = c.qlen;
    md = c.maxdeg;
    qvalid = push;
    bits = true;
    from_pull = !push;
    ae = c.edges;
    tr.set_activated(c.activated);
    cur = nx;
  }
  GG_TRY(timed_end(g, st, L.launches));
  GG_TRY(tr.collect());
  pages.wait();
  if (parent_host) GG_CUDA(cudaMemcpy(parent_host, parent, sizeof(uint32_t) * V, cudaMemcpyDeviceToHost));
  g->result[0] = parent;
  g->result[1] = nullptr;
  return GG_OK;
}

// ------------------------------------------------------------------ PageRank
// toolkits/pagerank.cpp:26-129.  Active = all vertices, so every
// process_edges call is dense (active_edges = edges >= edges/20); the pull
// gathers curr over the CSC and the process_vertices update that follows it
// (pagerank.cpp:77-97) is fused into the same kernel's epilogue.
template <typename T>
struct PrPull {
  using Acc = T;
  const T *curr;
  T *next;
  const uint32_t *out_deg;
  int last;
  uint32_t hot = 0xffffffffu;  // sources below this number are gathered through L1
  int zeros_done = 0;          // both buffers hold the vertices without in-edges
  static constexpr bool kDelta = true;
  static constexpr bool kDense = true;  // curr[V] is 0
  static constexpr bool kCompensated = sizeof(T) == 4;
  __device__ __forceinline__ bool want(uint32_t) const { return true; }
  __host__ __device__ __forceinline__ bool zero_kept() const { return zeros_done; }
  __device__ __forceinline__ T identity(uint32_t) const { return T(0); }
  __device__ __forceinline__ T identity_coop() const { return T(0); }
  __device__ __forceinline__ T gather(const Dir &, unsigned long long, uint32_t u) const {
    return ld_gather(curr, u, hot);
  }
  __host__ __forceinline__ bool gathers_all(uint32_t V) const { return hot >= V; }
  template <bool ALL>
  __device__ __forceinline__ T value(uint32_t u, float) const {
    return ALL ? curr[u] : ld_gather(curr, u, hot);
  }
  __device__ __forceinline__ T combine(T a, T b) const { return a + b; }
  __device__ __forceinline__ T warp_combine(T x) const { return warp_sum(x); }
  __device__ __forceinline__ bool finish(uint32_t v, T sum, uint32_t, Tally &t) const;
};

template <>
__device__ __forceinline__ bool PrPull<double>::finish(uint32_t v, double sum, uint32_t, Tally &t) const {
  const double d = 0.85;
  double nv = __dadd_rn(1.0 - d, __dmul_rn(d, sum));
  if (!last) {
    uint32_t od = out_deg[v];
    if (od > 0) {
      nv = __ddiv_rn(nv, (double)od);
      t.delta += __dmul_rn(fabs(__dadd_rn(nv, -curr[v])), (double)od);
    } else {
      t.delta += fabs(__dadd_rn(nv, -curr[v]));
    }
  }
  next[v] = nv;
  return false;
}

template <>
__device__ __forceinline__ bool PrPull<float>::finish(uint32_t v, float sum, uint32_t, Tally &t) const {
  const float d = 0.85f;
  float nv = __fadd_rn(1.0f - d, __fmul_rn(d, sum));
  if (!last) {
    uint32_t od = out_deg[v];
    if (od > 0) {
      nv = __fdiv_rn(nv, (float)od);
      t.add_delta(fabsf(__fadd_rn(nv, -curr[v])), od);
    } else {
      t.add_delta(fabsf(__fadd_rn(nv, -curr[v])), 1);
    }
  }
  next[v] = nv;
  return false;
}

// curr = 1 / out-degree (1 where it is 0); both buffers are 0 at V, where the
// rows' empty places point.
template <typename T>
__global__ void pr_init(T *curr, T *other, const uint32_t *out_deg, uint32_t V) {
  if (blockIdx.x == 0 && threadIdx.x == 0) curr[V] = other[V] = T(0);
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x) {
    uint32_t od = out_deg[v];
    curr[v] = od > 0 ? T(1) / (T)od : T(1);
  }
}

// Ranks computed in the hot-source numbering back to vertex order.
template <typename T>
__global__ void pr_unrank(const T *__restrict__ by_rank, const uint32_t *__restrict__ rank_of, uint32_t V,
                          T *__restrict__ out) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x)
    out[v] = by_rank[rank_of[v]];
}

// pagerank.cpp:35-97.  With the hot-source layout (the default) the
// iterations run in that numbering: pr_od is the out-degree there, every
// vertex's arithmetic is unchanged, and only the order in which an in-list
// is summed differs from the plain adjacency (by source number).
template <typename T>
static int pr_run(gg_graph *g, int iterations, T *ranks_host, double *deltas_host, gg_run_stats *st) {
  if (iterations < 0) {
    set_error("iterations must be >= 0");
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(g->device));
  if (g->pr_layout) GG_TRY(pr_layout_build(g));
  const bool ranked = g->pr_layout && g->pr_ready;
  const Dir &din = ranked ? g->pr : g->in;
  const uint32_t *od = ranked ? g->pr_od : g->out.deg;
  const uint32_t V = g->V;
  T *buf[2], *out = nullptr;
  Counters *per_iter;
  if (ranked) GG_TRY(ws(g, WS_S0, (size_t)V, &out));
  GG_TRY(ws(g, WS_S2, (size_t)V + 1, &buf[0]));
  GG_TRY(ws(g, WS_S3, (size_t)V + 1, &buf[1]));
  GG_TRY(ws(g, WS_HUBSUM, (size_t)(iterations > 0 ? iterations : 1), &per_iter));
  Launch L(g);
  Trace tr(st, g, "gg_pagerank");
  cudaStream_t s = g->stream;
  const uint32_t hot = ranked ? (uint32_t)(g->l1_hot_bytes / sizeof(T)) : 0xffffffffu;
  T *part = nullptr;
  if (din.nbig) GG_TRY(ws(g, WS_PARTIAL, din.nbigchunks, &part));
  // The run is device work only, so it is captured once as a CUDA graph and
  // replayed while its arguments are unchanged: no launch gaps between the
  // iterations' kernels.
  PrGraphKey key;
  memset(&key, 0, sizeof(key));
  key.din = din;
  key.od = od;
  key.buf0 = buf[0];
  key.buf1 = buf[1];
  key.out = out;
  key.per_iter = per_iter;
  key.partial = part;
  key.V = V;
  key.iterations = iterations;
  key.tsize = (int32_t)sizeof(T);
  key.ranked = ranked;
  key.timing = tr.timing_requested();
  key.hot = hot;
  key.split = g->pull_light_blocks;
  key.side = g->side;
  const int slot = sizeof(T) == 4 ? 0 : 1;  // one cached graph per precision
  cudaGraphExec_t &exec = g->pr_exec[slot];
  const bool replay = exec && memcmp(&key, &g->pr_key[slot], sizeof(key)) == 0;
  int cur = 0;
  // bookkeeping (trace, launch count) always; launches only while capturing
  auto enqueue = [&](bool launch) -> int {
    if (launch) {
      GG_CUDA(cudaMemsetAsync(per_iter, 0, sizeof(Counters) * (iterations > 0 ? iterations : 1), s));
      pr_init<T><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(buf[0], buf[1], od, V);
    }
    L.launches += 1;
    cur = 0;
    // active = all: active_edges = sum of out_degree = adjacency entries
    unsigned long long ae = g->nadj;
    for (int i = 0; i < iterations; i++) {
      tr.add(ae < g->E / 20 ? 0 : 1, ae, V);
      // a vertex without in-edges has one value from iteration 0 on (its
      // delta is 0 then), written to either buffer by iterations 0 and 1;
      // the last iteration writes it undivided
      PrPull<T> op{buf[cur], buf[cur ^ 1], od, i == iterations - 1, hot, i >= 2 && i < iterations - 1};
      GG_TRY(tr.kbegin());
      if (launch)
        GG_TRY(L.pull(din, op, ActOut(), per_iter + i));
      else
        L.launches += Launch::pull_launches(din);
      GG_TRY(tr.kend());
      cur ^= 1;
    }
    if (ranked) {
      if (launch) pr_unrank<T><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(buf[cur], g->pr_rank_of, V, out);
      L.launches += 1;
    }
    if (launch) GG_CUDA(cudaGetLastError());
    return GG_OK;
  };
  if (!replay) {
    if (exec) GG_CUDA(cudaGraphExecDestroy(exec));
    exec = nullptr;
    GG_TRY(tr.reserve_events(2 * (size_t)iterations));
    GG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    tr.capturing = true;
    const int rc = enqueue(true);
    tr.capturing = false;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(s, &graph);
    if (rc == GG_OK && e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (rc != GG_OK) return rc;
    GG_CUDA(e);
    g->pr_key[slot] = key;
  } else {
    tr.replay = true;
    GG_TRY(enqueue(false));
  }
  GG_TRY(timed_begin(g));
  GG_CUDA(cudaGraphLaunch(exec, s));
  Prefault pages(ranks_host, sizeof(T) * V);
  const T *result = ranked ? out : buf[cur];
  GG_TRY(timed_end(g, st, L.launches));
  GG_TRY(tr.collect());
  if (deltas_host && iterations > 0) {
    Counters *hc = new Counters[iterations];
    cudaError_t e = cudaMemcpy(hc, per_iter, sizeof(Counters) * iterations, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) {
      deltas_host[0] = 1.0;  // process_vertices returns 1 per vertex; divided by |V|
      for (int i = 1; i < iterations; i++) deltas_host[i] = hc[i - 1].delta / V;
    }
    delete[] hc;
    GG_CUDA(e);
  }
  pages.wait();
  if (ranks_host) GG_CUDA(cudaMemcpy(ranks_host, result, sizeof(T) * V, cudaMemcpyDeviceToHost));
  g->result[0] = result;
  g->result[1] = nullptr;
  return GG_OK;
}

// ------------------------------------------------------------------ process_vertices
__global__ void active_edges_kernel(const uint32_t *__restrict__ bm, size_t words, const uint32_t *__restrict__ deg,
                                    uint32_t V, Counters *ctr) {
  Tally t;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t w = bm[i];
    while (w) {
      uint32_t b = __ffs(w) - 1;
      w &= w - 1;
      size_t v = i * 32 + b;
      if (v < V) t.edges += deg[v];
    }
  }
  t.flush(ctr);
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_bfs(gg_graph *g, uint32_t root, uint32_t *parent, gg_run_stats *stats) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  return bfs_run(g, root, parent, stats);
}

int gg_graph_set_pr_layout(gg_graph *g, int hot_sources) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  g->pr_layout = hot_sources ? 1 : 0;
  if (!g->pr_layout) pr_layout_free(g);
  return GG_OK;
}

int gg_graph_set_l1_hot(gg_graph *g, uint32_t l1_bytes) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  g->l1_hot_bytes = l1_bytes;
  return GG_OK;
}

int gg_graph_set_dense_push(gg_graph *g, uint32_t divisor) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  g->dense_push_div = divisor;
  g->dense_push_set = 1;
  return GG_OK;
}

int gg_graph_set_bfs_pull(gg_graph *g, uint32_t divisor) {
  if (!g || divisor == 0) {
    set_error("need a graph and a divisor > 0");
    return GG_ERR_INVALID;
  }
  g->bfs_pull_div = divisor;
  return GG_OK;
}

int gg_graph_set_pull_split(gg_graph *g, uint32_t light_blocks) {
  if (!g || light_blocks > 7) {
    set_error("need a graph and 0..7 light blocks per SM");
    return GG_ERR_INVALID;
  }
  g->pull_light_blocks = light_blocks;
  return GG_OK;
}

int gg_bfs_many(gg_graph *g, const uint32_t *roots, int n, uint32_t *const *parents, gg_run_stats *stats) {
  if (!g || !roots || n < 0 || (n && !parents)) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  for (int i = 0; i < n; i++)
    if (roots[i] >= g->V) {
      set_error("root %u >= vertices %u", roots[i], g->V);
      return GG_ERR_INVALID;
    }
  GG_CUDA(cudaSetDevice(g->device));
  if (stats) {
    stats->calls = 0;
    stats->active_edges_total = 0;
    stats->device_ms = 0;
    stats->kernel_launches = 0;
  }
  const WsSlot slot[2] = {WS_S0, WS_PIPE};
  cudaStream_t cs = nullptr;
  cudaEvent_t done[2] = {nullptr, nullptr}, copied[2] = {nullptr, nullptr};
  int status = GG_OK;
  cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  for (int b = 0; b < 2 && e == cudaSuccess; b++) {
    e = cudaEventCreateWithFlags(&done[b], cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&copied[b], cudaEventDisableTiming);
  }
  if (e != cudaSuccess) status = cuda_status(e, "pipeline set-up");
  for (int i = 0; i < n && status == GG_OK; i++) {
    const int b = i & 1;
    // the buffer's previous result must be on the host before it is reused
    if (i >= 2) e = cudaStreamWaitEvent(g->stream, copied[b], 0);
    if (e != cudaSuccess) {
      status = cuda_status(e, "pipeline wait");
      break;
    }
    gg_run_stats one;
    memset(&one, 0, sizeof(one));
    status = bfs_run(g, roots[i], nullptr, &one, slot[b]);
    if (status != GG_OK) break;
    if (stats) {
      stats->calls += one.calls;
      stats->active_edges_total += one.active_edges_total;
      stats->device_ms += one.device_ms;
      stats->kernel_launches += one.kernel_launches;
    }
    uint32_t *dev = nullptr;
    status = ws(g, slot[b], g->V, &dev);
    if (status != GG_OK) break;
    e = cudaEventRecord(done[b], g->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(cs, done[b], 0);
    if (e == cudaSuccess && parents[i])
      e = cudaMemcpyAsync(parents[i], dev, sizeof(uint32_t) * g->V, cudaMemcpyDeviceToHost, cs);
    if (e == cudaSuccess) e = cudaEventRecord(copied[b], cs);
    if (e != cudaSuccess) status = cuda_status(e, "pipeline copy");
  }
  if (cs) {
    const cudaError_t e2 = cudaStreamSynchronize(cs);
    if (status == GG_OK && e2 != cudaSuccess) status = cuda_status(e2, "pipeline copy");
    cudaStreamDestroy(cs);
  }
  for (int b = 0; b < 2; b++) {
    if (done[b]) cudaEventDestroy(done[b]);
    if (copied[b]) cudaEventDestroy(copied[b]);
  }
  return status;
}

int gg_pagerank(gg_graph *g, int iterations, double *ranks, double *deltas, gg_run_stats *stats) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  return pr_run<double>(g, iterations, ranks, deltas, stats);
}

int gg_pagerank_f32(gg_graph *g, int iterations, float *ranks, double *deltas, gg_run_stats *stats) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  return pr_run<float>(g, iterations, ranks, deltas, stats);
}

int gg_active_edges(gg_graph *g, const uint64_t *active_bitmap, uint64_t *active_edges) {
  if (!g || !active_bitmap || !active_edges) {
    set_error("null argument");
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(g->device));
  Trace range(nullptr, g, "process_vertices");
  size_t words = bitmap_words32(g->V);
  uint32_t *bm;
  GG_TRY(ws(g, WS_BM3, words, &bm));
  GG_CUDA(cudaMemcpyAsync(bm, active_bitmap, words * 4, cudaMemcpyHostToDevice, g->stream));
  GG_TRY(counters_reset(g));
  active_edges_kernel<<<grid_for(words, 256, g->num_sms), 256, 0, g->stream>>>(bm, words, g->out.deg, g->V,
                                                                              g->ws.ctr);
  GG_CUDA(cudaGetLastError());
  Counters c;
  GG_TRY(counters_read(g, &c));
  *active_edges = c.edges;
  return GG_OK;
}

}  // extern "C"
