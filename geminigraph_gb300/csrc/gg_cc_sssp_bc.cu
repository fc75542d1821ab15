// CC (toolkits/cc.cpp), SSSP (toolkits/sssp.cpp) and BC (toolkits/bc.cpp,
// compute) on the device engine.
#include <math.h>

#include <vector>

#include "gg_engine.cuh"
#include "gg_resident.cuh"

namespace gg {

// ------------------------------------------------------------------ CC
// Sparse slot (cc.cpp:48-59): msg = label of the source at the start of the
// call (snapshot); a lower msg lowers label[dst] and activates dst.
struct CcPush {
  uint32_t *label;
  const uint32_t *msg;
  __device__ __forceinline__ bool push(uint32_t, uint32_t i, uint32_t dst, float) const {
    uint32_t m = msg[i];
    if (m < *(volatile uint32_t *)(label + dst)) {
      atomicMin(label + dst, m);
      return true;
    }
    return false;
  }
};

// Dense signal + slot (cc.cpp:60-79): msg = min(dst, labels of all
// in-neighbours); read from cur, written to nxt.  (A label never exceeds its
// vertex's id, so the message may start at the label instead of the id.)
// Every label a gather can return is at least the least id with an out-edge
// (floor): a vertex that has it is done, and a list that has shown it is too.
// From the second call on most vertices of a graph with one large component
// have it, the rest find it at their hottest in-neighbours, which lead the
// lists of the hot-source layout.  R-MAT 24 (537 M entries): 4.4 ms walking
// every list in each of three dense calls, 1.15 ms with this and cc_first.
struct CcPull {
  using Acc = uint32_t;
  const uint32_t *cur;
  uint32_t *nxt;
  uint32_t floor = 0;
  uint32_t hot = 0xffffffffu;     // sources below this number are gathered through L1
  __device__ __forceinline__ bool want(uint32_t) const { return true; }
  // no call changes a vertex without in-edges: both buffers hold its label
  __host__ __device__ __forceinline__ bool zero_kept() const { return true; }
  __device__ __forceinline__ uint32_t identity(uint32_t v) const { return cur[v]; }
  __device__ __forceinline__ void begin() {}
  __device__ __forceinline__ bool skip(uint32_t v) const { return cur[v] <= floor; }
  __device__ __forceinline__ bool stop(uint32_t acc, float) const { return acc <= floor; }
  __device__ __forceinline__ uint32_t identity_coop() const { return 0xffffffffu; }
  __device__ __forceinline__ uint32_t gather(const Dir &, unsigned long long, uint32_t u) const {
    return ld_gather(cur, u, hot);
  }
  __host__ __forceinline__ bool gathers_all(uint32_t V) const { return hot >= V; }
  template <bool ALL>
  __device__ __forceinline__ uint32_t value(uint32_t u, float) const {
    return ALL ? cur[u] : ld_gather(cur, u, hot);
  }
  __device__ __forceinline__ uint32_t combine(uint32_t a, uint32_t b) const { return b < a ? b : a; }
  __device__ __forceinline__ uint32_t warp_combine(uint32_t x) const { return warp_min(x); }
  __device__ __forceinline__ bool finish(uint32_t v, uint32_t m, uint32_t, Tally &) const {
    uint32_t c = cur[v];
    if (m < c) {
      nxt[v] = m;
      return true;
    }
    nxt[v] = c;
    return false;
  }
};

// ------------------------------------------------------------------ SSSP
// Lowers *p to v if v is smaller; true if this call lowered it (write_min,
// core/atomic.hpp:35-42).  Non-negative floats order like their int bits;
// negative floats order like the reverse of their unsigned bits, and any
// stored value of the other sign compares correctly in both forms.
__device__ __forceinline__ bool atomic_min_float(float *p, float v) {
  if (!(v < 0.0f)) {
    int old = atomicMin((int *)p, __float_as_int(v));
    return __int_as_float(old) > v;
  }
  unsigned old = atomicMax((unsigned *)p, __float_as_uint(v));
  return __uint_as_float(old) > v;
}

struct SsspPush {
  float *dist;
  const float *msg;
  __device__ __forceinline__ bool push(uint32_t, uint32_t i, uint32_t dst, float w) const {
    float relax = __fadd_rn(msg[i], w);
    if (relax < *(volatile float *)(dist + dst)) return atomic_min_float(dist + dst, relax);
    return false;
  }
};

// sssp.cpp:60-80: the dense signal takes the min over ALL in-edges (its
// active check is commented out, sssp.cpp:64-70); INF = 1e9.
// On SSSP's layout a list is walked by ascending weight class and only as far
// as an active source could still lower the vertex: an inactive source cannot
// (see relax_loop), an active one's candidate is at least fl(lo + w) for the
// active sources' least distance lo and the least weight w of what is left.
struct SsspPull {
  using Acc = float;
  const float *cur;
  float *nxt;
  float wmin = -INFINITY, width = INFINITY;  // of the layout (gg_graph)
  const unsigned *lo_enc = nullptr;          // ~float_order(lo), written by active_min
  float lo = -INFINITY;
  __device__ __forceinline__ void begin() {
    const uint32_t o = ~*lo_enc;
    lo = __uint_as_float(o & 0x80000000u ? o & 0x7fffffffu : ~o);
  }
  __device__ __forceinline__ bool skip(uint32_t v) const { return __fadd_rn(lo, wmin) >= cur[v]; }
  __device__ __forceinline__ bool stop(float acc, float w) const {
    return __fadd_rn(lo, __fsub_rd(w, width)) >= acc;
  }
  uint32_t hot = 0xffffffffu;  // sources below this number are gathered through L1
  __device__ __forceinline__ bool want(uint32_t) const { return true; }
  // no call changes a vertex without in-edges: both buffers hold its distance
  __host__ __device__ __forceinline__ bool zero_kept() const { return true; }
  // the message may start at the distance: only a lower one is written
  __device__ __forceinline__ float identity(uint32_t v) const { return cur[v]; }
  __device__ __forceinline__ float identity_coop() const { return 1e9f; }
  __device__ __forceinline__ float gather(const Dir &d, unsigned long long k, uint32_t u) const {
    return __fadd_rn(ld_gather(cur, u, hot), d.w[k]);
  }
  // the same candidate with the weight read by the kernel
  __device__ __forceinline__ float gather_w(uint32_t u, float w) const { return __fadd_rn(ld_gather(cur, u, hot), w); }
  __host__ __forceinline__ bool gathers_all(uint32_t V) const { return hot >= V; }
  template <bool ALL>
  __device__ __forceinline__ float value(uint32_t u, float w) const {
    return __fadd_rn(ALL ? cur[u] : ld_gather(cur, u, hot), w);
  }
  __device__ __forceinline__ float combine(float a, float b) const { return b < a ? b : a; }
  __device__ __forceinline__ float warp_combine(float x) const { return warp_min(x); }
  __device__ __forceinline__ bool finish(uint32_t v, float m, uint32_t, Tally &) const {
    float c = cur[v];
    if (m < c) {
      nxt[v] = m;
      return true;
    }
    nxt[v] = c;
    return false;
  }
};

// The least distance among the active vertices (queue q, or bitmap bm when q
// is null), as ~float_order in *out (0 before).
__global__ void active_min(const uint32_t *__restrict__ q, uint32_t n, const uint32_t *__restrict__ bm, size_t words,
                           const float *__restrict__ dist, unsigned *out) {
  uint32_t best = 0;
  auto take = [&](uint32_t v) {
    const uint32_t u = __float_as_uint(dist[v]);
    const uint32_t o = ~(u & 0x80000000u ? ~u : u | 0x80000000u);
    best = o > best ? o : best;
  };
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (q) {
    for (size_t i = tid; i < n; i += stride) take(q[i]);
  } else {
    // a warp per 32 words: each word's vertices by the lanes, coalesced
    for (size_t g = tid / 32; g * 32 < words; g += stride / 32) {
      const size_t i = g * 32 + lane_id();
      const uint32_t w = i < words ? bm[i] : 0u;
      for (unsigned any = __ballot_sync(GG_FULL, w != 0); any; any &= any - 1) {
        const int j = __ffs(any) - 1;
        const uint32_t wj = __shfl_sync(GG_FULL, w, j);
        if ((wj >> lane_id()) & 1u) take((uint32_t)((g * 32 + j) * 32 + lane_id()));
      }
    }
  }
  best = __reduce_max_sync(GG_FULL, best);
  if (lane_id() == 0 && best) atomicMax(out, best);
}

// CC's first call, every vertex active with its own id as label: the least
// in-neighbour, the first entry of the (plain) in-list.  v in the numbering
// of the labels, id_of its vertex (null: v itself).
__device__ __forceinline__ void cc_first_walk(const Dir &d, uint32_t V, const uint32_t *id_of, uint32_t *label,
                                              const ActOut &act, Tally &t) {
  const size_t groups = ((size_t)V + 31) / 32, nwarps = (size_t)gridDim.x * (PULL_THREADS / 32);
  for (size_t g = (size_t)blockIdx.x * (PULL_THREADS / 32) + (threadIdx.x >> 5); g < groups; g += nwarps) {
    const uint32_t v = (uint32_t)(g * 32 + lane_id());
    bool a = false;
    if (v < V) {
      const uint32_t id = id_of ? id_of[v] : v;
      const unsigned long long b = d.off[id];
      if (d.off[id + 1] > b) {
        const uint32_t u = nbr_at(d, b, GG_SITE);
        a = u < id;
        if (a) label[v] = u;
      }
    }
    pull_activate(a, v, g, act, t);
  }
}
__global__ void __launch_bounds__(PULL_THREADS)
    cc_first(Dir d, uint32_t V, const uint32_t *__restrict__ id_of, uint32_t *__restrict__ label, ActOut act,
             Counters *ctr) {
  Tally t;
  cc_first_walk(d, V, id_of, label, act, t);
  t.flush(ctr);
}

// The least vertex with an out-edge (V if none), by one block over the
// deg > 0 bitmap.
__device__ __forceinline__ void least_source_block(const uint32_t *__restrict__ nz, size_t words, uint32_t V,
                                                   uint32_t *out) {
  __shared__ uint32_t s_min;
  if (threadIdx.x == 0) s_min = V;
  __syncthreads();
  for (size_t base = 0; base < words; base += blockDim.x) {
    const size_t i = base + threadIdx.x;
    const uint32_t w = i < words ? nz[i] : 0u;
    if (w) atomicMin(&s_min, (uint32_t)(i * 32 + __ffs(w) - 1));
    if (__syncthreads_or(w != 0)) break;
  }
  if (threadIdx.x == 0) *out = s_min;
}
__global__ void __launch_bounds__(1024) least_source(const uint32_t *__restrict__ nz, size_t words, uint32_t V,
                                                     uint32_t *out) {
  least_source_block(nz, words, V, out);
}

// ------------------------------------------------------------------ resident CC / SSSP
// What a resident run needs of the two toolkits.
struct CcRun {
  using T = uint32_t;
  using Pull = CcPull;
  static constexpr bool kWeighted = false;
  // largest graph (entries) run whole: R-MAT 18 / 20 / 22 / 24 (2^27 to 2^29
  // entries the last two) 293 / 323 / 497 / 1153 us from the host, 160 / 189 /
  // 358 / 1235 so
  static constexpr unsigned long long kWhole = 1ull << 28;
  static __device__ __forceinline__ T cand(T msg, float) { return msg; }
  static __device__ __forceinline__ T amin(T *p, T x) { return atomicMin(p, x); }
};
struct SsspRun {
  using T = float;
  using Pull = SsspPull;
  static constexpr bool kWeighted = true;
  // R-MAT 16 / 18 / 20 / 24: 834 / 928 / 1519 / 5740 us from the host, 446 /
  // 601 / 1501 / 12400 so (its pulls have fewer warps than the host's kernels)
  static constexpr unsigned long long kWhole = 1ull << 24;
  static __device__ __forceinline__ T cand(T msg, float w) { return __fadd_rn(msg, w); }
  // write_min, returning the value before (see atomic_min_float)
  static __device__ __forceinline__ T amin(T *p, T x) {
    if (!(x < 0.0f)) return __int_as_float(atomicMin((int *)p, __float_as_int(x)));
    return __uint_as_float(atomicMax((unsigned *)p, __float_as_uint(x)));
  }
};

struct RelaxArgs {
  Dir out, in;                    // the run's numbering; in.sell_desc: pulls can run here
  Dir plain_in;                   // CC's first call
  const uint32_t *plain_nz;
  const uint32_t *id_of, *rank_of;  // null: the run is in vertex order
  uint32_t *q[2], *bm[2];
  void *a[2], *result, *partials;
  ResTally *slots;                // three
  uint32_t *word;                 // one value between the run's start and its first call
  ResRow *rows;                   // the calls' rows while the run goes on
  ResOut *out_host;               // mapped host memory
  void *result_host;              // also the result, when it fits (mapped)
  unsigned long long edges_lim;   // edges / 20
  unsigned long long nadj;
  uint32_t V, push_div, root;
  uint32_t init;                  // 1: start of a traversal; 2: continued by another launch; 0: entered from the host loop
  uint32_t whole;                 // no call is too large
};

// Consecutive calls of the CC / SSSP loop.  Two state arrays: at the start of
// a call every vertex's value is in the one to read (R); slots lower the other
// (W).  Every message is read from R, which no slot of the call writes, so
// all signals precede all slots without a snapshot.  For W to become the next
// call's R, every vertex that R had right and W not is brought up to date
// during the call: those are the active ones (changed in the previous call,
// which wrote what is now R), each by the thread that expands it.  A slot that
// lowers W[dst] below R[dst] is the first of the call to do so exactly if W
// held R's value or more before: it appends dst to the next queue.
template <class Run>
__global__ void __launch_bounds__(RES_THREADS, RES_BLOCKS) relax_run(RelaxArgs p, typename Run::Pull pull, ResState st) {
  using T = typename Run::T;
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const uint32_t V = p.V;
  const size_t cap = (size_t)V + 1;
  const size_t words = 2 * ((size_t)V / 64 + 1);
  const size_t nthreads = (size_t)gridDim.x * RES_THREADS, tid = (size_t)blockIdx.x * RES_THREADS + threadIdx.x;
  const bool first_thread = tid == 0;
  T *a0 = (T *)p.a[0], *a1 = (T *)p.a[1];
  __shared__ ResStage s_stage;
  res_stage_init(s_stage);
  uint32_t step = st.step;
  auto slot = [&]() { return p.slots + step % 3; };
  auto begin_step = [&]() { res_clear(p.slots + (step + 1) % 3); };
  st.calls = 0;
  if (p.init == 1) {
    for (size_t i = tid; i < words; i += nthreads) p.bm[0][i] = p.bm[1][i] = 0u;
    if constexpr (Run::kWeighted) {
      const uint32_t start = p.rank_of ? p.rank_of[p.root] : p.root;
      for (size_t v = tid; v < V; v += nthreads) a0[v] = a1[v] = v == start ? 0.0f : 1e9f;
      st.ae = p.out.deg[start];
      st.n_act = 1;
      st.n = st.ae > RES_HUB ? 0 : 1;
      st.hubs = 1 - st.n;
      st.qvalid = 1;
      if (first_thread) p.q[0][st.n ? 0 : cap - 1] = start;
    } else {
      for (size_t v = tid; v < V; v += nthreads) a0[v] = a1[v] = p.id_of ? p.id_of[v] : (uint32_t)v;
      st.ae = p.nadj;
      st.n_act = V;
      if (blockIdx.x == 0) least_source_block(p.plain_nz, words, V, p.word);
    }
    grid.sync();
    if constexpr (!Run::kWeighted) pull.floor = res_read(p.word);
  } else if (p.init == 0) {
    // the queue with its hubs apart (the host has copied R to W)
    begin_step();
    for (size_t i = tid; i < st.n; i += nthreads) {
      const uint32_t v = p.q[st.q][i];
      res_append(v, p.out.deg[v], p.q[st.q ^ 1], cap, slot());
    }
    grid.sync();
    st.n = (uint32_t)res_read(&slot()->app);
    st.hubs = (uint32_t)res_read(&slot()->happ);
    st.q ^= 1;
    step++;
  }
  bool opening = p.init == 1 && !Run::kWeighted;
  while (st.n_act > 0 && st.calls < RES_CALLS) {
    const bool sparse = st.ae < p.edges_lim;
    const bool push = sparse || (p.push_div && st.ae < p.nadj / p.push_div);
    if (!push && !p.in.sell_desc) break;
    if (!p.whole && (!sparse || st.n + st.hubs > RES_MAX_QUEUE || st.ae > RES_MAX_AE)) break;
    const unsigned long long ae = st.ae;
    const T *R = (const T *)p.a[st.role];
    T *W = (T *)p.a[st.role ^ 1];
    if (push) {
      if (!st.qvalid) {
        begin_step();
        res_queue_from_bitmap(p.bm[st.bm], words, p.out.deg, p.q[st.q], cap, slot());
        grid.sync();
        st.n = (uint32_t)res_read(&slot()->app);
        st.hubs = (uint32_t)res_read(&slot()->happ);
        step++;
      }
      begin_step();
      ResTally *sl = slot();
      uint32_t *qn = p.q[st.q ^ 1];
      res_expand(
          p.out, p.q[st.q], st.n, st.hubs, st.ae, cap,
          [&](uint32_t src, bool lead) {
            const T msg = R[src];
            if (lead) Run::amin(W + src, msg);
            return msg;
          },
          [&](T msg, uint32_t, unsigned long long k) {
            const uint32_t dst = nbr_at(p.out, k, GG_SITE);
            const T x = Run::cand(msg, Run::kWeighted ? p.out.w[k] : 0.0f);
            const T r = R[dst];
            if (x < r) {
              const uint32_t od = p.out.deg[dst];
              if (!(Run::amin(W + dst, x) < r)) res_stage(dst, od, s_stage, qn, cap, sl);
            }
          });
      res_stage_flush(s_stage, qn, sl);
      grid.sync();
      const unsigned long long app = res_read(&sl->app), happ = res_read(&sl->happ);
      step++;
      st.n = (uint32_t)app;
      st.hubs = (uint32_t)happ;
      st.n_act = st.n + st.hubs;
      st.ae = (app >> 32) + (happ >> 32);
      st.q ^= 1;
      st.qvalid = 1;
      st.role ^= 1;
    } else {
      typename Run::Pull op = pull;
      op.cur = R;
      op.nxt = W;
      // the least active distance, which ends the walks of large graphs early;
      // below 2^22 entries finding it takes longer (R-MAT 16 and 18: 446 and
      // 601 us without, 556 and 745 with; R-MAT 20: 1632 and 1501)
      if (Run::kWeighted && p.nadj > (1ull << 22)) {
        begin_step();
        uint32_t best = 0;
        auto take = [&](uint32_t v) {
          const uint32_t u = __float_as_uint((float)R[v]);
          const uint32_t o = ~(u & 0x80000000u ? ~u : u | 0x80000000u);
          best = o > best ? o : best;
        };
        if (st.qvalid) {
          for (size_t i = tid; i < st.n + st.hubs; i += nthreads)
            take(i < st.n ? p.q[st.q][i] : p.q[st.q][cap - 1 - (i - st.n)]);
        } else {
          for (size_t i = tid; i < words * 32; i += nthreads)
            if ((p.bm[st.bm][i >> 5] >> (i & 31)) & 1u) take((uint32_t)i);
        }
        best = __reduce_max_sync(GG_FULL, best);
        if (lane_id() == 0 && best) atomicMax(&slot()->c.aux, best);
        grid.sync();
        if constexpr (Run::kWeighted) op.lo_enc = &slot()->c.aux;
        op.begin();
        step++;
      }
      begin_step();
      ActOut act;
      act.active_out = p.bm[st.bm ^ 1];
      act.out_deg = p.out.deg;
      Tally t;
      if (opening) {
        // label[v] = v: in place, both arrays agree on what it leaves alone
        cc_first_walk(p.plain_in, V, p.id_of, (uint32_t *)W, act, t);
      } else {
        const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps = gridDim.x * (RES_THREADS / 32);
        const bool parts = p.in.nheavy > 0;
        if (!parts) long_lists<typename Run::Pull, true>(p.in, op, act, t, warp, nwarps);
        rows_walk<typename Run::Pull, true, true>(p.in, V, op, act, t, parts ? (T *)p.partials : nullptr, warp, nwarps);
        // the set this call was entered with has no reader any more; the next
        // pull sets its bits there
        for (size_t i = tid; i < words; i += nthreads) p.bm[st.bm][i] = 0u;
        if (parts) {
          grid.sync();
          big_finish<typename Run::Pull, 8, true>(p.in, op, (const T *)p.partials, act, t);
        }
      }
      t.flush(&slot()->c);
      grid.sync();
      st.n_act = res_read(&slot()->c.activated);
      st.ae = res_read(&slot()->c.edges);
      step++;
      st.bm ^= 1;
      st.qvalid = 0;
      st.role ^= 1;
      opening = false;
    }
    if (first_thread) p.rows[st.calls] = ResRow{ae, st.n_act, sparse ? 0u : 1u};
    st.calls++;
  }
  if (st.n_act == 0) {
    const T *R = (const T *)p.a[st.role];
    T *out = (T *)p.result, *host = (T *)p.result_host;
    for (size_t v = tid; v < V; v += nthreads) {
      const T x = R[p.rank_of ? p.rank_of[v] : v];
      if (p.rank_of) out[v] = x;
      if (host) host[v] = x;
    }
  } else if (st.qvalid && st.calls < RES_CALLS) {
    // back to the host loop: its queues hold vertices with out-edges only
    begin_step();
    res_plain_queue(p.q[st.q], st.n, st.hubs, cap, p.out.deg, p.q[st.q ^ 1], slot());
    grid.sync();
    st.n = (uint32_t)res_read(&slot()->app);
    st.hubs = 0;
    st.q ^= 1;
    step++;
  }
  st.step = step % 3;
  res_report(st, p.rows, p.out_host);
}

// A dense call pushes below this fraction of the adjacency.  A pull that ends
// its walks early is the faster form down to fewer active edges: SSSP R-MAT
// 24, divisors 4 / 8 / 16: 7.2 / 5.9 / 5.7 ms, R-MAT 22: 2.9 / 2.3 / 2.2 ms
// (walking every list: 4 was the best).
template <class PullOp>
static uint32_t relax_push_div(const gg_graph *g, const Dir &din) {
  return has_gather_w<PullOp>::value && din.sell_desc && !g->dense_push_set ? 16 : g->dense_push_div;
}

template <class Run>
static int relax_args(gg_graph *g, const Dir &dout, const Dir &din, void *a0, void *a1, uint32_t *const *q,
                      uint32_t *const *bm, RelaxArgs *p) {
  *p = RelaxArgs{};
  p->out = dout;
  p->in = din;
  p->q[0] = q[0];
  p->q[1] = q[1];
  p->bm[0] = bm[0];
  p->bm[1] = bm[1];
  p->a[0] = a0;
  p->a[1] = a1;
  typename Run::T *part = nullptr;
  GG_TRY(ws(g, WS_PARTIAL, din.nbigchunks, &part));
  p->partials = part;
  GG_TRY(res_buffers(g, &p->slots, &p->rows, &p->word));
  p->out_host = (ResOut *)g->ws.stage;
  p->edges_lim = g->E / 20;
  p->nadj = g->nadj;
  p->V = g->V;
  p->push_div = relax_push_div<typename Run::Pull>(g, din);
  return GG_OK;
}

// One launch of relax_run; *st is where it stopped.
template <class Run>
static int relax_launch(gg_graph *g, RelaxArgs &p, typename Run::Pull pull, ResState *st, Launch &L, Trace &tr) {
  ResState in = *st;
  void *args[] = {&p, &pull, &in};
  GG_TRY(res_launch(g, (const void *)relax_run<Run>, p.whole ? res_blocks(g) : (unsigned)g->num_sms, args, &in, &L));
  *st = ((const ResOut *)g->ws.stage)->st;
  res_trace(g, tr);
  return GG_OK;
}

// A whole CC / SSSP traversal on the device; *ran = false where it has to run
// from the host: a large graph (there the calls are long enough to launch one
// by one, with kernels of their own), no rows to pull, gathers by source
// number, or per-call times asked for.
template <class Run>
static int relax_whole(gg_graph *g, const Dir &dout, const Dir &din, const typename Run::Pull &pull, bool ranked,
                       uint32_t root, void *const *a, uint32_t *const *q, uint32_t *const *bm, void *result,
                       size_t result_bytes, Launch &L, Trace &tr, const gg_run_stats *stats, bool *ran, void **dev,
                       const void **host) {
  *ran = false;
  if (g->nadj > Run::kWhole || !din.sell_desc || !pull.gathers_all(g->V) || (stats && stats->call_ms) || !L.coop_ok() ||
      !g->ws.stage)
    return GG_OK;
  RelaxArgs p;
  GG_TRY((relax_args<Run>(g, dout, din, a[0], a[1], q, bm, &p)));
  p.plain_in = g->in;
  p.plain_nz = g->out.nz;
  p.id_of = ranked ? g->pr_id_of_rank : nullptr;
  p.rank_of = ranked ? g->pr_rank_of : nullptr;
  p.result = result;
  p.result_host = result_bytes <= RES_RESULT_BYTES ? (char *)g->ws.stage + RES_OUT_BYTES : nullptr;
  p.root = root;
  p.whole = 1;
  if (!g->dense_push_set) {
    // CC's pulls over rows end at the floor and beat its pushes, which all
    // lower the same hubs (R-MAT 16 / 18, a late dense call: 45 / 184 us
    // pushing, 15 / 18 pulling; at R-MAT 24, 537 M entries, from the host,
    // the vertices that a pull looks at are the greater cost)
    if (!Run::kWeighted) p.push_div = 0;
    if (Run::kWeighted && g->nadj <= RES_PUSH_ALL) p.push_div = 1;
  }
  p.init = 1;
  ResState st;
  do {
    GG_TRY((relax_launch<Run>(g, p, pull, &st, L, tr)));
    p.init = 2;
  } while (st.n_act > 0);
  *ran = true;
  *dev = ranked ? result : a[st.role];
  *host = p.result_host;
  return GG_OK;
}

// Runs the CC / SSSP frontier loop: both toolkits loop while the slots
// activate something, with a message snapshot for push calls and two state
// buffers for pull calls.
template <class Run, typename T, class PushOp, class PullOp>
static int relax_loop(gg_graph *g, const Dir &dout, const Dir &din, const PullOp &pull, T *state0, T *state1,
                      uint32_t *q0, uint32_t *q1, uint32_t *bm0, uint32_t *bm1, uint32_t n_act, uint32_t nq,
                      bool qvalid, unsigned long long ae, Trace &tr, Launch &L, T **result) {
  const uint32_t V = g->V;
  const size_t words = bitmap_words32(V);
  cudaStream_t s = g->stream;
  Counters *ctr = g->ws.ctr;
  T *cur = state0, *nxt = state1;
  uint32_t *q[2] = {q0, q1};
  uint32_t *bm[2] = {bm0, bm1};
  T *msg;
  GG_TRY(ws(g, WS_MSG, (size_t)V + 1, &msg));
  // A pull that ends its walks early is the faster form down to fewer active
  // edges: SSSP R-MAT 24, divisors 4 / 8 / 16: 7.2 / 5.9 / 5.7 ms, R-MAT 22:
  // 2.9 / 2.3 / 2.2 ms (walking every list: 4 was the best).
  const uint32_t push_div = relax_push_div<PullOp>(g, din);
  int c_i = 0;
  while (n_act > 0) {
    bool sparse = ae < g->E / 20;
    if (sparse && qvalid && nq <= RES_MAX_QUEUE && ae <= RES_MAX_AE && ae > 0 && L.coop_ok()) {
      // consecutive small sparse calls run on the device without host round trips
      RelaxArgs p;
      GG_TRY((relax_args<Run>(g, dout, din, cur, nxt, q, bm, &p)));
      ResState st;
      st.ae = ae;
      st.n_act = n_act;
      st.n = nq;
      st.qvalid = 1;
      st.q = (uint32_t)c_i;
      GG_CUDA(cudaMemcpyAsync(nxt, cur, sizeof(T) * V, cudaMemcpyDeviceToDevice, s));
      GG_TRY((relax_launch<Run>(g, p, pull, &st, L, tr)));
      // as many calls as fit one launch: the arrays and the queue are the kernel's still
      while (st.n_act > 0 && st.calls == RES_CALLS) {
        p.init = 2;
        GG_TRY((relax_launch<Run>(g, p, pull, &st, L, tr)));
      }
      ae = st.ae;
      n_act = st.n_act;
      nq = st.n;
      c_i = (int)st.q;
      if (st.role) {
        T *t = cur;
        cur = nxt;
        nxt = t;
      }
      continue;
    }
    tr.add(sparse ? 0 : 1, ae, 0);
    // A dense call may run as a push over the frontier: a source that is
    // not active was relaxed against its current value in the call after it
    // last changed, so it cannot lower any out-neighbour now, and the
    // minimum over the active sources' candidates is the dense call's
    // minimum over all in-edges -- the same values and the same activated
    // set (the snapshot keeps every signal before every slot).
    const bool push = sparse || (push_div && ae < g->nadj / push_div);
    int nx = c_i ^ 1;
    if (push && ae > 0 && !qvalid) GG_TRY(L.queue_from_bitmap(bm[c_i], dout.nz, q[c_i], &nq));
    GG_CUDA(cudaMemsetAsync(bm[nx], 0, words * 4, s));
    GG_TRY(counters_reset(g));
    ActOut a;
    a.active_out = bm[nx];
    a.q_out = push ? q[nx] : nullptr;
    a.qlen = &ctr->qlen;
    a.out_deg = dout.deg;
    a.queue_nonzero_only = true;
    if (push) {
      if (ae > 0) {
        gather_by_queue<T><<<grid_for(nq, 256, g->num_sms), 256, 0, s>>>(q[c_i], nq, cur, msg);
        unsigned long long *P;
        GG_TRY(L.scan_queue_degrees(q[c_i], nq, dout.deg, &P));
        GG_TRY(tr.kbegin());
        push_lb<PushOp><<<L.push_grid(ae), PUSH_THREADS, 0, s>>>(q[c_i], P, nq, ae, dout, PushOp{cur, msg}, a,
                                                                   ctr);
        GG_TRY(tr.kend());
        L.launches += 2;
      }
    } else {
      GG_TRY(tr.kbegin());
      PullOp op = pull;
      op.cur = cur;
      op.nxt = nxt;
      if constexpr (has_gather_w<PullOp>::value) {
        if (din.sell_desc) {
          const size_t work = qvalid ? nq : words;
          active_min<<<grid_for(work, 256, g->num_sms, 8), 256, 0, s>>>(qvalid ? q[c_i] : nullptr, nq, bm[c_i], words,
                                                                       cur, &ctr->aux);
          L.launches += 1;
          op.lo_enc = &ctr->aux;
        }
      }
      GG_TRY(L.pull(din, op, a, ctr));
      GG_TRY(tr.kend());
      T *t = cur;
      cur = nxt;
      nxt = t;
    }
    GG_CUDA(cudaGetLastError());
    Counters c;
    GG_TRY(counters_read(g, &c));
    n_act = c.activated;
    nq = c.qlen;
    qvalid = push;
    ae = c.edges;
    tr.set_activated(c.activated);
    c_i = nx;
  }
  *result = cur;
  return GG_OK;
}

// a[v] = b[v] = src[v]
template <typename T>
__global__ void copy_twice(const T *__restrict__ src, size_t n, T *__restrict__ a, T *__restrict__ b) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const T x = src[v];
    a[v] = x;
    b[v] = x;
  }
}

// out[v] = by_rank[rank_of[v]]
template <typename T>
__global__ void unrank(const T *__restrict__ by_rank, const uint32_t *__restrict__ rank_of, uint32_t V,
                       T *__restrict__ out) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x)
    out[v] = by_rank[rank_of[v]];
}

// The end of a whole run: its time and its result.
static int relax_done(gg_graph *g, gg_run_stats *st, const Launch &L, Prefault &pages, void *user, const void *dev,
                      const void *host, size_t bytes) {
  GG_TRY(timed_read(g, st, L.launches));
  pages.wait();
  if (user && host)
    memcpy(user, host, bytes);
  else if (user)
    GG_CUDA(cudaMemcpy(user, dev, bytes, cudaMemcpyDeviceToHost));
  g->result[0] = dev;
  g->result[1] = nullptr;
  return GG_OK;
}

static int cc_run(gg_graph *g, uint32_t *label_host, gg_run_stats *st) {
  GG_CUDA(cudaSetDevice(g->device));
  const uint32_t V = g->V;
  const size_t words = bitmap_words32(V);
  uint32_t *lab[2], *bm[2], *q[2];
  GG_TRY(ws(g, WS_S0, V, &lab[0]));
  GG_TRY(ws(g, WS_S1, V, &lab[1]));
  GG_TRY(ws(g, WS_BM1, words, &bm[0]));
  GG_TRY(ws(g, WS_BM2, words, &bm[1]));
  GG_TRY(ws(g, WS_Q0, (size_t)V + 1, &q[0]));
  GG_TRY(ws(g, WS_Q1, (size_t)V + 1, &q[1]));
  // On a symmetric graph the hot-source layout (vertices renumbered by
  // descending degree, built once and shared with PageRank) packs the most
  // gathered labels into few cache lines.  Labels stay vertex ids, so the
  // minimum is the reference's; they map back to vertex order at the end.
  if (g->symmetric && g->pr_layout) GG_TRY(pr_layout_build(g));
  const bool ranked = g->symmetric && g->pr_layout && g->pr_ready;
  const Dir &dout = ranked ? g->pr : g->out;
  const Dir &din = ranked ? g->pr : g->in;
  uint32_t *out = nullptr;
  if (ranked) GG_TRY(ws(g, WS_S2, V, &out));
  Launch L(g);
  Trace tr(st, g, "gg_cc");
  cudaStream_t s = g->stream;
  Counters *ctr = g->ws.ctr;
  Prefault pages(label_host, sizeof(uint32_t) * V);
  GG_TRY(timed_begin(g));
  CcPull pull{};
  pull.hot = ranked ? g->l1_hot_bytes / 4 : 0xffffffffu;
  bool whole = false;
  void *dev = nullptr;
  const void *host = nullptr;
  void *const states[2] = {lab[0], lab[1]};
  GG_TRY((relax_whole<CcRun>(g, dout, din, pull, ranked, 0, states, q, bm, out, sizeof(uint32_t) * V, L, tr, st, &whole,
                             &dev, &host)));
  if (whole) return relax_done(g, st, L, pages, label_host, dev, host, sizeof(uint32_t) * V);
  // label[v] = v over active_in = all (cc.cpp:31-37)
  if (ranked)
    copy_twice<uint32_t><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(g->pr_id_of_rank, V, lab[0], lab[1]);
  else
    iota_u32<<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(lab[0], V);
  L.launches += 1;
  GG_CUDA(cudaGetLastError());
  uint32_t *res = nullptr;
  uint32_t n_act = V;
  unsigned long long ae = g->nadj;
  // the first call: dense by the reference's switch (every vertex active)
  tr.add(1, ae, 0);
  GG_CUDA(cudaMemsetAsync(bm[0], 0, words * 4, s));
  GG_TRY(counters_reset(g));
  least_source<<<1, 1024, 0, s>>>(g->out.nz, words, V, &ctr->aux);
  ActOut act;
  act.active_out = bm[0];
  act.out_deg = dout.deg;
  GG_TRY(tr.kbegin());
  cc_first<<<L.pull_grid(), PULL_THREADS, 0, s>>>(g->in, V, ranked ? g->pr_id_of_rank : nullptr, lab[0], act, ctr);
  GG_TRY(tr.kend());
  L.launches += 2;
  GG_CUDA(cudaGetLastError());
  Counters c;
  GG_TRY(counters_read(g, &c));
  tr.set_activated(c.activated);
  pull.floor = c.aux;
  n_act = c.activated;
  ae = c.edges;
  GG_TRY((relax_loop<CcRun, uint32_t, CcPush, CcPull>(g, dout, din, pull, lab[0], lab[1], q[0], q[1], bm[0], bm[1], n_act, 0,
                                               false, ae, tr, L, &res)));
  if (ranked) {
    unrank<uint32_t><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(res, g->pr_rank_of, V, out);
    L.launches += 1;
    GG_CUDA(cudaGetLastError());
    res = out;
  }
  GG_TRY(timed_end(g, st, L.launches));
  GG_TRY(tr.collect());
  pages.wait();
  if (label_host) GG_CUDA(cudaMemcpy(label_host, res, sizeof(uint32_t) * V, cudaMemcpyDeviceToHost));
  g->result[0] = res;
  g->result[1] = nullptr;
  return GG_OK;
}

__global__ void sssp_root(float *dist, float *other, uint32_t root, uint32_t *active, uint32_t *q,
                          const uint32_t *out_deg, Counters *ctr) {
  dist[root] = 0.0f;
  other[root] = 0.0f;
  active[root >> 5] |= 1u << (root & 31);
  q[0] = root;
  ctr->edges = out_deg[root];
  ctr->maxdeg = out_deg[root];
}

static int sssp_run(gg_graph *g, uint32_t root, float *dist_host, gg_run_stats *st) {
  if (!g->weighted) {
    set_error("sssp needs a weighted graph");
    return GG_ERR_UNWEIGHTED;
  }
  if (root >= g->V) {
    set_error("root %u >= vertices %u", root, g->V);
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(g->device));
  const uint32_t V = g->V;
  const size_t words = bitmap_words32(V);
  float *dist[2];
  uint32_t *bm[2], *q[2];
  GG_TRY(ws(g, WS_S0, V, &dist[0]));
  GG_TRY(ws(g, WS_S1, V, &dist[1]));
  GG_TRY(ws(g, WS_BM1, words, &bm[0]));
  GG_TRY(ws(g, WS_BM2, words, &bm[1]));
  GG_TRY(ws(g, WS_Q0, (size_t)V + 1, &q[0]));
  GG_TRY(ws(g, WS_Q1, (size_t)V + 1, &q[1]));
  // Hot-source layout (as PageRank's and CC's): both directions renumbered
  // by descending out-degree, weights carried along.  Every candidate
  // distance d[u] + w is the same sum, and a minimum does not depend on
  // order, so the distances are bit-identical; they map back to vertex order
  // at the end.
  if (g->pr_layout) GG_TRY(sssp_layout_build(g));
  const bool ranked = g->pr_layout && g->ps_ready && (g->symmetric || g->pr_out_ready);
  const Dir &dout = ranked ? (g->symmetric ? g->ps : g->pr_out) : g->out;
  const Dir &din = ranked ? g->ps : g->in;
  uint32_t start = root;
  float *out = nullptr;
  if (ranked) GG_TRY(ws(g, WS_S2, V, &out));
  Launch L(g);
  Trace tr(st, g, "gg_sssp");
  cudaStream_t s = g->stream;
  SsspPull pull{};
  pull.hot = ranked ? g->l1_hot_bytes / 4 : 0xffffffffu;
  pull.wmin = g->ps_wmin;
  pull.width = g->ps_width;
  Prefault pages(dist_host, sizeof(float) * V);
  GG_TRY(timed_begin(g));
  bool whole = false;
  void *dev = nullptr;
  const void *host = nullptr;
  void *const states[2] = {dist[0], dist[1]};
  GG_TRY((relax_whole<SsspRun>(g, dout, din, pull, ranked, root, states, q, bm, out, sizeof(float) * V, L, tr, st, &whole,
                               &dev, &host)));
  if (whole) return relax_done(g, st, L, pages, dist_host, dev, host, sizeof(float) * V);
  if (ranked) GG_CUDA(cudaMemcpy(&start, g->pr_rank_of + root, sizeof(uint32_t), cudaMemcpyDeviceToHost));
  GG_CUDA(cudaMemsetAsync(bm[0], 0, words * 4, s));
  GG_TRY(counters_reset(g));
  fill_kernel<float><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(dist[0], V, 1e9f);
  fill_kernel<float><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(dist[1], V, 1e9f);
  sssp_root<<<1, 1, 0, s>>>(dist[0], dist[1], start, bm[0], q[0], dout.deg, g->ws.ctr);
  L.launches += 3;
  GG_CUDA(cudaGetLastError());
  Counters c;
  GG_TRY(counters_read(g, &c));
  float *res = nullptr;
  GG_TRY((relax_loop<SsspRun, float, SsspPush, SsspPull>(g, dout, din, pull, dist[0], dist[1], q[0], q[1], bm[0], bm[1], 1,
                                                1, true, c.edges, tr, L, &res)));
  if (ranked) {
    unrank<float><<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(res, g->pr_rank_of, V, out);
    L.launches += 1;
    GG_CUDA(cudaGetLastError());
    res = out;
  }
  GG_TRY(timed_end(g, st, L.launches));
  GG_TRY(tr.collect());
  pages.wait();
  if (dist_host) GG_CUDA(cudaMemcpy(dist_host, res, sizeof(float) * V, cudaMemcpyDeviceToHost));
  g->result[0] = res;
  g->result[1] = nullptr;
  return GG_OK;
}

// ------------------------------------------------------------------ BC
// Forward sparse slot (bc.cpp:58-69): unvisited dst gains the source's path
// count; the first contribution (old value 0) activates dst.
struct BcFwdPush {
  double *np;
  const uint32_t *visited;
  __device__ __forceinline__ bool push(uint32_t src, uint32_t, uint32_t dst, float) const {
    if (bm_test(visited, dst)) return false;
    return atomicAdd(np + dst, np[src]) == 0.0;
  }
};

// Forward dense (bc.cpp:70-89): an unvisited vertex sums the path counts of
// its active in-neighbours.
struct BcFwdPull {
  using Acc = double;
  double *np;
  const uint32_t *active_in;
  const uint32_t *visited;
  __device__ __forceinline__ bool want(uint32_t v) const { return !bm_test(visited, v); }
  __host__ __device__ __forceinline__ bool zero_kept() const { return true; }
  __device__ __forceinline__ double identity(uint32_t) const { return 0.0; }
  __device__ __forceinline__ double identity_coop() const { return 0.0; }
  __device__ __forceinline__ double gather(const Dir &, unsigned long long, uint32_t s) const {
    return bm_test_ldg(active_in, s) ? np[s] : 0.0;
  }
  __host__ __forceinline__ bool gathers_all(uint32_t) const { return true; }
  template <bool ALL>
  __device__ __forceinline__ double value(uint32_t s, float) const {
    return bm_test_ldg(active_in, s) ? np[s] : 0.0;
  }
  __device__ __forceinline__ double combine(double a, double b) const { return a + b; }
  __device__ __forceinline__ double warp_combine(double x) const { return warp_sum(x); }
  __device__ __forceinline__ bool finish(uint32_t v, double sum, uint32_t, Tally &) const {
    if (sum > 0.0) {
      np[v] += sum;
      return true;
    }
    return false;
  }
};

// Backward sparse slot (bc.cpp:130-138) on the transposed graph.
struct BcBwdPush {
  double *dep;
  const uint32_t *visited;
  __device__ __forceinline__ bool push(uint32_t src, uint32_t, uint32_t dst, float) const {
    if (!bm_test(visited, dst)) atomicAdd(dep + dst, dep[src]);
    return false;
  }
};

// Backward dense (bc.cpp:139-155): unvisited vertices sum the dependencies
// of their in-neighbours (on the transposed graph) in the current level.
struct BcBwdPull {
  using Acc = double;
  double *dep;
  const uint32_t *level;
  const uint32_t *visited;
  __device__ __forceinline__ bool want(uint32_t v) const { return !bm_test(visited, v); }
  __host__ __device__ __forceinline__ bool zero_kept() const { return true; }
  __device__ __forceinline__ double identity(uint32_t) const { return 0.0; }
  __device__ __forceinline__ double identity_coop() const { return 0.0; }
  __device__ __forceinline__ double gather(const Dir &, unsigned long long, uint32_t s) const {
    return bm_test_ldg(level, s) ? dep[s] : 0.0;
  }
  __host__ __forceinline__ bool gathers_all(uint32_t) const { return true; }
  template <bool ALL>
  __device__ __forceinline__ double value(uint32_t s, float) const {
    return bm_test_ldg(level, s) ? dep[s] : 0.0;
  }
  __device__ __forceinline__ double combine(double a, double b) const { return a + b; }
  __device__ __forceinline__ double warp_combine(double x) const { return warp_sum(x); }
  __device__ __forceinline__ bool finish(uint32_t v, double sum, uint32_t deg, Tally &) const {
    if (deg > 0) dep[v] += sum;
    return false;
  }
};

// Path counts and dependencies 0, the root's count 1; the root is level 0.
// One launch, and the root's number in the layout is read here: as two fills,
// two clears, a copy of that number to the host and a one-thread kernel it
// was 45 us of a 480 us call on 4096 vertices.
__global__ void bc_begin(double *np, double *dep, uint32_t V, uint32_t root, const uint32_t *__restrict__ rank_of,
                         uint32_t *visited, uint32_t *active, size_t words, uint32_t *qlev,
                         const uint32_t *__restrict__ out_deg, const uint32_t *__restrict__ in_deg, Counters *ctr) {
  const uint32_t r = rank_of ? rank_of[root] : root;
  const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  for (size_t v = t0; v < V; v += step) {
    np[v] = v == r ? 1.0 : 0.0;
    dep[v] = 0.0;
  }
  for (size_t w = t0; w < words; w += step) visited[w] = active[w] = w == r >> 5 ? 1u << (r & 31) : 0u;
  if (t0 == 0) {
    qlev[0] = r;
    ctr->edges = out_deg[r];
    ctr->in_edges = in_deg[r];
  }
}

// Between two forward calls: the last call's vertices join visited
// (bc.cpp:91-98), the next call's bitmap and the counters start at 0.  One
// launch instead of a kernel and two clears (9 us of a small graph's call).
__global__ void bc_step(uint32_t *visited, const uint32_t *__restrict__ active, uint32_t *next, size_t words,
                        Counters *ctr) {
  const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (size_t w = t0; w < words; w += (size_t)gridDim.x * blockDim.x) {
    visited[w] |= active[w];
    next[w] = 0u;
  }
  if (t0 == 0) *ctr = Counters{};
}

// process_vertices over one level: visited |= level, inv_num_paths = 1 /
// num_paths, dep += inv (bc.cpp:103-120,157-164); level: also the level's
// bitmap, for a dense call.  The levels hold the vertices that were reached,
// side by side: the FP64 unit takes 16 cycles per warp instruction whether 1
// or 32 lanes divide, and far more for the infinity that 1 / 0 paths gives: a
// division over all vertices cost 45 us at R-MAT 22 (with bc_final's: the
// whole call 1681 us before, 1331 us now).
__global__ void bc_level_apply(const uint32_t *__restrict__ q, uint32_t n, uint32_t *visited, double *dep,
                               const double *__restrict__ np, double *inv, uint32_t *level) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t v = q[i];
    const double x = 1.0 / np[v];
    atomicOr(visited + (v >> 5), 1u << (v & 31));
    if (level) atomicOr(level + (v >> 5), 1u << (v & 31));
    inv[v] = x;
    dep[v] += x;
  }
}

// The results in the graph's own numbering: dependencies = (dep - inv) / inv
// (bc.cpp:170-176) as (dep - inv) * num_paths, which rounds once less, and the
// inverse path counts.  A vertex that was not reached has 1 / 0 paths and
// (dep - inf) / inf, written as such: divisions of infinities over all
// vertices, with the two renumberings after them, took 193 us at R-MAT 22.
// dep_out and inv_out may be dep and np (no renumbering).
__global__ void bc_final(const double *dep, const double *np, const double *__restrict__ inv,
                         const uint32_t *__restrict__ rank_of, uint32_t V, double *dep_out, double *inv_out) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x) {
    const uint32_t r = rank_of ? rank_of[v] : (uint32_t)v;
    const double n = np[r];
    double x = __longlong_as_double(0x7ff0000000000000ll), y = __longlong_as_double(0x7ff8000000000000ll);
    if (n != 0.0) {
      x = inv[r];
      y = (dep[r] - x) * n;
    }
    dep_out[v] = y;
    inv_out[v] = x;
  }
}

static int bc_run(gg_graph *g, uint32_t root, double *dep_host, double *inv_host, gg_run_stats *st) {
  if (root >= g->V) {
    set_error("root %u >= vertices %u", root, g->V);
    return GG_ERR_INVALID;
  }
  GG_CUDA(cudaSetDevice(g->device));
  const uint32_t V = g->V;
  const size_t words = bitmap_words32(V);
  double *np, *dep, *inv;
  uint32_t *visited, *bm[2], *qlev;
  GG_TRY(ws(g, WS_S2, V, &np));
  GG_TRY(ws(g, WS_S3, V, &dep));
  GG_TRY(ws(g, WS_MSG, V, &inv));
  GG_TRY(ws(g, WS_BM0, words, &visited));
  GG_TRY(ws(g, WS_BM1, words, &bm[0]));
  GG_TRY(ws(g, WS_BM2, words, &bm[1]));
  GG_TRY(ws(g, WS_QLEV, (size_t)V + 2, &qlev));
  // Hot-source layout (as SSSP's): both directions renumbered; path counts
  // are exact and dependencies change only in summation order.
  if (g->pr_layout) {
    GG_TRY(pr_layout_build(g));
    if (!g->symmetric) GG_TRY(hot_out_rows(g));
  }
  const bool ranked = g->pr_layout && g->pr_ready && (g->symmetric || g->pr_out_ready);
  const Dir &dout = ranked ? (g->symmetric ? g->pr : g->pr_out) : g->out;
  const Dir &din = ranked ? g->pr : g->in;
  const uint32_t *rank_of = ranked ? g->pr_rank_of : nullptr;
  double *dep_out = dep, *np_out = np;
  if (ranked) {
    GG_TRY(ws(g, WS_S0, V, &dep_out));
    GG_TRY(ws(g, WS_S1, V, &np_out));
  }
  Launch L(g);
  Trace tr(st, g, "gg_bc");
  cudaStream_t s = g->stream;
  Counters *ctr = g->ws.ctr;
  Prefault pages(dep_host, sizeof(double) * V, inv_host, sizeof(double) * V);
  GG_TRY(timed_begin(g));
  GG_TRY(counters_reset(g));
  bc_begin<<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(np, dep, V, root, rank_of, visited, bm[0], words, qlev,
                                                        dout.deg, din.deg, ctr);
  L.launches += 1;
  GG_CUDA(cudaGetLastError());
  Counters c;
  GG_TRY(counters_read(g, &c));
  // level L occupies qlev[lev_off[L], lev_off[L+1]); lev_out/in = degree sums
  std::vector<uint64_t> lev_off{0, 1}, lev_out{c.edges}, lev_in{c.in_edges};
  int cur = 0;
  uint32_t n = 1;
  while (n > 0) {
    size_t L_ = lev_off.size() - 2;
    unsigned long long ae = lev_out[L_];
    bool sparse = ae < g->E / 20;
    tr.add(sparse ? 0 : 1, ae, 0);
    int nx = cur ^ 1;
    bc_step<<<grid_for(words, 256, g->num_sms), 256, 0, s>>>(visited, bm[cur], bm[nx], words, ctr);
    L.launches += 1;
    ActOut a;
    a.active_out = bm[nx];
    a.qlen = &ctr->qlen;
    a.out_deg = dout.deg;
    a.in_deg = din.deg;
    const uint32_t *qin = qlev + lev_off[L_];
    a.q_out = sparse ? qlev + lev_off.back() : nullptr;
    if (sparse) {
      if (ae > 0) {
        unsigned long long *P;
        GG_TRY(L.scan_queue_degrees(qin, n, dout.deg, &P));
        GG_TRY(tr.kbegin());
        push_lb<BcFwdPush><<<L.push_grid(ae), PUSH_THREADS, 0, s>>>(qin, P, n, ae, dout, BcFwdPush{np, visited},
                                                                      a, ctr);
        GG_TRY(tr.kend());
        L.launches += 1;
      }
    } else {
      GG_TRY(tr.kbegin());
      GG_TRY(L.pull(din, BcFwdPull{np, bm[cur], visited}, a, ctr));
      GG_TRY(tr.kend());
    }
    GG_CUDA(cudaGetLastError());
    GG_TRY(counters_read(g, &c));
    tr.set_activated(c.activated);
    n = c.activated;
    if (!sparse && n > 0) {
      uint32_t nl = 0;
      GG_TRY(L.queue_from_bitmap(bm[nx], nullptr, qlev + lev_off.back(), &nl));
    }
    lev_off.push_back(lev_off.back() + n);
    lev_out.push_back(c.edges);
    lev_in.push_back(c.in_edges);
    cur = nx;
  }
  // levels 0..top; level `top` is the empty set the last forward call produced
  const int top = (int)lev_off.size() - 2;
  GG_CUDA(cudaMemsetAsync(visited, 0, words * 4, s));
  // the levels' bitmaps, for dense calls (the forward calls are done with them)
  uint32_t *lvbm = bm[0], *lvbm_next = bm[1];
  auto dense_level = [&](int lev) { return lev_in[lev] >= g->E / 20; };
  if (dense_level(top)) GG_CUDA(cudaMemsetAsync(lvbm, 0, words * 4, s));  // the last level is empty
  // backward on the transposed graph: push over the CSC, pull over the CSR
  const Dir &tout = din, &tin = dout;
  for (int lev = top; lev >= 1; lev--) {
    uint32_t ln = (uint32_t)(lev_off[lev + 1] - lev_off[lev]);
    const uint32_t *ql = qlev + lev_off[lev];
    unsigned long long ae = lev_in[lev];
    bool sparse = !dense_level(lev);
    tr.add(sparse ? 0 : 1, ae, 0);
    if (sparse) {
      if (ae > 0) {
        unsigned long long *P;
        GG_TRY(L.scan_queue_degrees(ql, ln, tout.deg, &P));
        GG_TRY(tr.kbegin());
        push_lb<BcBwdPush><<<L.push_grid(ae), PUSH_THREADS, 0, s>>>(ql, P, ln, ae, tout, BcBwdPush{dep, visited},
                                                                      ActOut(), ctr);
        GG_TRY(tr.kend());
        L.launches += 1;
      }
    } else {
      GG_TRY(tr.kbegin());
      GG_TRY(L.pull(tin, BcBwdPull{dep, lvbm, visited}, ActOut(), ctr));
      GG_TRY(tr.kend());
    }
    uint32_t pn = (uint32_t)(lev_off[lev] - lev_off[lev - 1]);
    uint32_t *mark = lev > 1 && dense_level(lev - 1) ? lvbm_next : nullptr;
    if (mark) GG_CUDA(cudaMemsetAsync(mark, 0, words * 4, s));
    if (pn)
      bc_level_apply<<<grid_for(pn, 256, g->num_sms), 256, 0, s>>>(qlev + lev_off[lev - 1], pn, visited, dep, np, inv,
                                                                   mark);
    L.launches += 1;
    GG_CUDA(cudaGetLastError());
    std::swap(lvbm, lvbm_next);
  }
  bc_final<<<grid_for(V, 256, g->num_sms), 256, 0, s>>>(dep, np, inv, rank_of, V, dep_out, np_out);
  L.launches += 1;
  GG_CUDA(cudaGetLastError());
  GG_TRY(timed_end(g, st, L.launches));
  GG_TRY(tr.collect());
  pages.wait();
  if (dep_host) GG_CUDA(cudaMemcpy(dep_host, dep_out, sizeof(double) * V, cudaMemcpyDeviceToHost));
  if (inv_host) GG_CUDA(cudaMemcpy(inv_host, np_out, sizeof(double) * V, cudaMemcpyDeviceToHost));
  g->result[0] = dep_out;
  g->result[1] = np_out;
  return GG_OK;
}

}  // namespace gg

using namespace gg;

extern "C" {

int gg_cc(gg_graph *g, uint32_t *label, gg_run_stats *stats) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  return cc_run(g, label, stats);
}

int gg_sssp(gg_graph *g, uint32_t root, float *distance, gg_run_stats *stats) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  return sssp_run(g, root, distance, stats);
}

int gg_bc(gg_graph *g, uint32_t root, double *dependencies, double *inv_num_paths, gg_run_stats *stats) {
  if (!g) {
    set_error("null graph");
    return GG_ERR_INVALID;
  }
  return bc_run(g, root, dependencies, inv_num_paths, stats);
}

}  // extern "C"
