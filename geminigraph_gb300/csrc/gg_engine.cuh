// Edge-processing engine: the GB300 form of Graph::process_edges
// (core/graph.hpp:1492-1867) and Graph::process_vertices (:1406-1469).
//
// Reference semantics kept exactly:
//  * switch: sparse iff active_edges < edges / 20 (:1509), active_edges =
//    sum of out_degree over the active set (:1503-1508);
//  * every signal of a call is computed before any slot of the call applies
//    (messages are buffered, :1541-1556 and :1755-1793).  Push kernels read
//    their message from a snapshot taken before the kernel (or from state no
//    slot of the call can write); pull kernels that read a state array the
//    same call writes use two buffers (read one, write the other).
// Fused on the device:
//  * signal + slot: the push kernel computes the slot for each edge of each
//    queued vertex; the pull kernel gathers the in-list (signal) and applies
//    the slot to its own vertex with a plain store (one writer per vertex);
//  * the activation epilogue of every edge kernel sets the active_out bit,
//    appends the vertex to the next queue and adds its out_degree to the
//    next call's active_edges, so the switch of the next call and the
//    process_vertices(active_out) count need no extra pass.
#ifndef GG_ENGINE_CUH
#define GG_ENGINE_CUH

#include <string.h>

#include <cooperative_groups.h>
#include <type_traits>

#include "gg_common.cuh"
#include "gg_scan.cuh"

namespace gg {

constexpr uint32_t NONE32 = 0xffffffffu;

// Ops whose gather adds an edge weight (SSSP) may take the weight from the
// kernel (gather_w): the chunk kernel reads weights coalesced and past L1,
// as it reads neighbour ids, so that L1 keeps the gathered state.
template <class Op, class = void>
struct has_gather_w : std::false_type {};
template <class Op>
struct has_gather_w<Op, std::void_t<decltype(&Op::gather_w)>> : std::true_type {};
constexpr int PUSH_THREADS = 256;
// Ops whose finish adds to the tally's delta (PageRank).
template <class Op, class = void>
struct has_delta : std::false_type {};
template <class Op>
struct has_delta<Op, std::void_t<decltype(Op::kDelta)>> : std::true_type {};
// The end of a pull kernel: what the op and the call tally, once per block.
template <class Op, int THREADS>
__device__ __forceinline__ void pull_flush(Tally &t, bool activates, Counters *ctr) {
  if constexpr (has_delta<Op>::value) t.template flush_delta<THREADS>(ctr);
  if (activates) t.flush(ctr);
}
constexpr int PUSH_TILE = 1024;              // edges per block iteration of push_lb
constexpr int PUSH_STAGE = PUSH_TILE + 1;    // queue entries a tile spans when each has >= 1 edge
constexpr int PULL_THREADS = 256;

// Where an edge kernel records activations.  Only push (sparse) calls append
// to a queue; after a pull (dense) call the next queue, if the next call is
// sparse, is compacted from the bitmap in vertex order (queue_from_bitmap),
// which avoids one same-address atomic per warp of activated vertices.
struct ActOut {
  uint32_t *active_out = nullptr;  // bitmap; null: the call activates nothing
  uint32_t *visited = nullptr;     // also set here when non-null
  uint32_t *q_out = nullptr;       // next queue (push calls); null: none
  unsigned *qlen = nullptr;
  const uint32_t *out_deg = nullptr;
  const uint32_t *in_deg = nullptr;  // optional: also sum in_degree
  bool queue_nonzero_only = false;   // append only vertices with out_degree > 0
};

// Push activation: pred may be true for several lanes naming the same
// vertex; the bitmap decides who appends.  All lanes must call.
__device__ __forceinline__ void push_activate(bool pred, uint32_t v, const ActOut &a, Tally &t) {
  bool fresh = false;
  if (pred) {
    fresh = bm_set_atomic(a.active_out, v);
    if (fresh && a.visited) atomicOr(a.visited + (v >> 5), 1u << (v & 31));
  }
  uint32_t od = fresh ? a.out_deg[v] : 0u;
  if (a.q_out) queue_push(fresh && (!a.queue_nonzero_only || od > 0), v, a.q_out, a.qlen);
  if (fresh) {
    t.activated += 1;
    t.edges += od;
    t.maxdeg = od > t.maxdeg ? od : t.maxdeg;
    if (a.in_deg) t.in_edges += a.in_deg[v];
  }
}

// Pull activation: the warp owns bitmap word g (vertices 32g..32g+31), so the
// word is written with plain stores (SHARED: with an atomic, where other
// warps set bits of the word too).  All lanes must call.
template <bool SHARED = false>
__device__ __forceinline__ void pull_activate(bool act, uint32_t v, size_t g, const ActOut &a, Tally &t) {
  unsigned bits = __ballot_sync(GG_FULL, act);
  if (lane_id() == 0 && bits) {
    if (SHARED)
      atomicOr(a.active_out + g, bits);
    else
      a.active_out[g] = bits;
    if (a.visited) a.visited[g] |= bits;
  }
  if (act) {
    const uint32_t od = a.out_deg[v];
    t.activated += 1;
    t.edges += od;
    t.maxdeg = od > t.maxdeg ? od : t.maxdeg;
    if (a.in_deg) t.in_edges += a.in_deg[v];
  }
}

template <typename T>
__device__ __forceinline__ uint32_t upper_bound_idx(const T *P, uint32_t lo, uint32_t hi, T x) {
  // first index in [lo, hi) with P[i] > x (hi if none)
  while (lo < hi) {
    uint32_t mid = lo + ((hi - lo) >> 1);
    if (P[mid] <= x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Ops whose result depends on which edge comes first (BFS's parents): their
// tiles keep the timing they have, one thread's searches included.
template <class Op, class = void>
struct has_claims : std::false_type {};
template <class Op>
struct has_claims<Op, std::void_t<decltype(Op::kClaims)>> : std::true_type {};

// The queue entry holding edge e0 of the prefix P and one past the entry
// holding edge e1 - 1, by the block's first two warps (one thread's two
// binary searches are 40 dependent loads for a queue of a million).
__device__ __forceinline__ void tile_bounds(const unsigned long long *P, uint32_t n, unsigned long long e0,
                                            unsigned long long e1, uint32_t *s_lo, uint32_t *s_hi) {
  if (threadIdx.x >= 64) return;
  const uint32_t b = warp_upper_bound<unsigned long long>(P, 0, n + 1, threadIdx.x < 32 ? e0 : e1 - 1);
  if (lane_id() == 0) {
    if (threadIdx.x < 32)
      *s_lo = b - 1;
    else
      *s_hi = b;
  }
}

// ---------------------------------------------------------------- push
// Sparse mode (core/graph.hpp:1510-1663): for every queued vertex q[i] and
// every out-edge, op.push(src, i, dst, w) applies the slot and returns
// whether it may activate dst.  Work is split by EDGES: P is the exclusive
// prefix of the queued vertices' degrees (P[n] = total); each block
// iteration takes PUSH_TILE consecutive edges, stages the tile's slice of P
// with the sources and their list offsets in shared memory, and each thread
// finds its edge's source by binary search there.  A hub's list is spread
// over as many blocks as it needs and neighbour loads are coalesced.  A tile
// spanning more than PUSH_STAGE entries (queues holding degree-0 vertices)
// searches P in global memory instead.
template <class Op>
__global__ void __launch_bounds__(PUSH_THREADS)
    push_lb(const uint32_t *__restrict__ q, const unsigned long long *__restrict__ P, uint32_t n,
            unsigned long long total, Dir d, Op op, ActOut act, Counters *ctr) {
  __shared__ unsigned long long s_P[PUSH_STAGE + 1];
  __shared__ unsigned long long s_base[PUSH_STAGE];
  __shared__ uint32_t s_src[PUSH_STAGE];
  __shared__ uint32_t s_lo, s_hi;
  Tally t;
  unsigned long long ntiles = (total + PUSH_TILE - 1) / PUSH_TILE;
  for (unsigned long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    unsigned long long e0 = tile * PUSH_TILE;
    unsigned long long e1 = e0 + PUSH_TILE < total ? e0 + PUSH_TILE : total;
    if constexpr (has_claims<Op>::value) {
      if (threadIdx.x == 0) {
        uint32_t lo = upper_bound_idx<unsigned long long>(P, 0, n + 1, e0) - 1;
        s_lo = lo;
        s_hi = upper_bound_idx<unsigned long long>(P, lo, n + 1, e1 - 1);  // one past the entry holding e1-1
      }
    } else {
      tile_bounds(P, n, e0, e1, &s_lo, &s_hi);
    }
    __syncthreads();
    const uint32_t lo = s_lo, hi = s_hi, cnt = hi - lo;
    const bool staged = cnt <= (uint32_t)PUSH_STAGE;
    if (staged) {
      for (uint32_t i = threadIdx.x; i < cnt; i += PUSH_THREADS) {
        unsigned long long pi = P[lo + i];
        uint32_t src = q[lo + i];
        s_P[i] = pi;
        s_src[i] = src;
        s_base[i] = d.off[src] - pi;
      }
    }
    __syncthreads();
    for (unsigned long long base = e0; base < e1; base += PUSH_THREADS) {
      unsigned long long e = base + threadIdx.x;
      bool pred = false;
      uint32_t dst = 0;
      if (e < e1) {
        uint32_t qi, src;
        unsigned long long k;
        if (staged) {
          uint32_t i = upper_bound_idx<unsigned long long>(s_P, 0, cnt, e) - 1;
          src = s_src[i];
          k = s_base[i] + e;
          qi = lo + i;
        } else {
          qi = upper_bound_idx<unsigned long long>(P, lo, hi, e) - 1;
          src = q[qi];
          k = d.off[src] + (e - P[qi]);
        }
        dst = nbr_at(d, k, GG_SITE);
        float w = d.w ? d.w[k] : 0.0f;
        pred = op.push(src, qi, dst, w);
      }
      if (act.active_out) push_activate(pred, dst, act, t);
    }
    __syncthreads();
  }
  t.flush(ctr);
}

// ---------------------------------------------------------------- pull
// Dense mode (core/graph.hpp:1664-1855), reduction form.  For each vertex v
// with op.want(v): acc = op.identity(v) combined (op.combine) with
// op.gather(d, k, u) (u = the k-th entry) over its in-list, then
// op.finish(v, acc, deg, tally) applies the slot and returns whether v is
// activated.  Op::Acc is the message type; op.identity_coop() is the
// neutral element of combine.  Work is split by the direction's degree bins:
//   pull_light   one warp per 32 consecutive vertices, each lane serially
//                over a list of <= d.light entries (and every deg-0 vertex);
//                the warp owns the bitmap word of its 32 vertices
//   pull_chunks / pull_big_finish(_warps)
//                every longer list cut into d.chunk-edge chunks, one warp
//                per chunk, then a lane (or, without activations, a warp)
//                per vertex combining its chunks
// The chunk kernel runs beside pull_light (second stream); the finish runs
// after both and sets its bitmap bits atomically.
// WIN: each lane reads its list by aligned 32-byte windows (two 16-byte
// loads through L1: eight entries per two load instructions instead of
// eight), the window's entries of [b, e) gathered together and combined in
// list order, so the sums equal the scalar form's bit for bit.  The neighbour
// arrays are padded to a multiple of 64 entries, so a window never leaves
// the array.  Picked per graph by the autotuner (Dir.vec bit 1).
constexpr unsigned LIGHT_WIN = 8;
template <class Op, bool WIN>
__global__ void __launch_bounds__(PULL_THREADS) pull_light(Dir d, uint32_t V, Op op, ActOut act, Counters *ctr) {
  using Acc = typename Op::Acc;
  Tally t;
  size_t nwarps = (size_t)gridDim.x * (PULL_THREADS / 32);
  size_t groups = ((size_t)V + 31) / 32;
  unsigned lane = lane_id();
  for (size_t g = (size_t)blockIdx.x * (PULL_THREADS / 32) + (threadIdx.x >> 5); g < groups; g += nwarps) {
    uint32_t v = (uint32_t)(g * 32 + lane);
    bool todo = v < V && op.want(v);
    unsigned long long b = 0, e = 0;
    if (todo) {
      b = d.off[v];
      e = d.off[v + 1];
    }
    uint32_t deg = (uint32_t)(e - b);
    bool a = false;
    if (todo && deg <= d.light) {
      Acc acc = op.identity(v);
      if constexpr (WIN) {
        for (unsigned long long k = b & ~(unsigned long long)(LIGHT_WIN - 1); k < e; k += LIGHT_WIN) {
          const uint4 w0 = *reinterpret_cast<const uint4 *>(d.nbr + k);
          const uint4 w1 = *reinterpret_cast<const uint4 *>(d.nbr + k + 4);
          const uint32_t u[LIGHT_WIN] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
          Acc gv[LIGHT_WIN];
#pragma unroll
          for (unsigned j = 0; j < LIGHT_WIN; j++)
            gv[j] = k + j >= b && k + j < e ? op.gather(d, k + j, vertex_ok(d, u[j], GG_SITE)) : op.identity_coop();
#pragma unroll
          for (unsigned j = 0; j < LIGHT_WIN; j++)
            if (k + j >= b && k + j < e) acc = op.combine(acc, gv[j]);
        }
      } else {
        // four independent gathers in flight, combined in list order
        unsigned long long k = b;
        for (; k + 4 <= e; k += 4) {
          const uint32_t u0 = nbr_at(d, k, GG_SITE), u1 = nbr_at(d, k + 1, GG_SITE), u2 = nbr_at(d, k + 2, GG_SITE), u3 = nbr_at(d, k + 3, GG_SITE);
          Acc g0 = op.gather(d, k, u0), g1 = op.gather(d, k + 1, u1), g2 = op.gather(d, k + 2, u2),
              g3 = op.gather(d, k + 3, u3);
          acc = op.combine(op.combine(op.combine(op.combine(acc, g0), g1), g2), g3);
        }
        for (; k < e; k++) acc = op.combine(acc, op.gather(d, k, nbr_at(d, k, GG_SITE)));
      }
      a = op.finish(v, acc, deg, t);
    }
    if (act.active_out) pull_activate(a, v, g, act, t);
  }
  pull_flush<Op, PULL_THREADS>(t, act.active_out != nullptr, ctr);
}

// Lists longer than d.light: one warp per d.chunk-edge aligned block of the
// adjacency (d.chunk = 32 * PER_LANE, 128 / 256 / 512), PER_LANE gathers in
// flight per lane; partials[c] = the chunk's combine (lane order, then the
// warp tree).  Two load shapes (d.vec, picked per graph by the autotuner):
//   VEC    lane l loads the block's 16-byte windows l, l + 32, ... with one
//          vector load each (fewer load instructions), read past L1;
//   !VEC   lane l takes entries l, l + 32, ... (a warp's gathers touch
//          consecutive entries, which share cache sectors where an in-list
//          holds runs of consecutive source numbers), read past L1.
template <class Op, int PER_LANE, bool VEC>
__global__ void __launch_bounds__(PULL_THREADS)
    pull_chunks(Dir d, Op op, typename Op::Acc *__restrict__ partials) {
  using Acc = typename Op::Acc;
  constexpr int WIN = PER_LANE / 4;
  const size_t nwarps = (size_t)gridDim.x * (PULL_THREADS / 32);
  const unsigned lane = lane_id();
  for (size_t c = (size_t)blockIdx.x * (PULL_THREADS / 32) + (threadIdx.x >> 5); c < d.nbigchunks; c += nwarps) {
    uint32_t v;
    unsigned long long lo, b, e;
    big_range(d, (uint32_t)c, 32 * PER_LANE, &v, &lo, &b, &e);
    Acc part = op.identity_coop();
    if (op.want(v)) {
      Acc vals[PER_LANE];
      constexpr bool WT = has_gather_w<Op>::value;
      if constexpr (VEC) {
        uint4 w[WIN], wt[WT ? WIN : 1];
#pragma unroll
        for (int i = 0; i < WIN; i++) {
          const unsigned long long p = lo + 4 * (lane + 32 * i);
          const bool in = p < e && p + 4 > b;
          w[i] = in ? ld_once_v4(d.nbr + p) : make_uint4(0, 0, 0, 0);
          if constexpr (WT)
            wt[i] = in ? ld_once_v4(reinterpret_cast<const uint32_t *>(d.w) + p) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int i = 0; i < WIN; i++) {
          const unsigned long long p = lo + 4 * (lane + 32 * i);
          const uint32_t u[4] = {vertex_ok(d, w[i].x, GG_SITE), vertex_ok(d, w[i].y, GG_SITE),
                                 vertex_ok(d, w[i].z, GG_SITE), vertex_ok(d, w[i].w, GG_SITE)};
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const bool in = p + j >= b && p + j < e;
            if constexpr (WT) {
              const uint32_t wb[4] = {wt[i].x, wt[i].y, wt[i].z, wt[i].w};
              vals[4 * i + j] = in ? op.gather_w(u[j], __uint_as_float(wb[j])) : op.identity_coop();
            } else {
              vals[4 * i + j] = in ? op.gather(d, p + j, u[j]) : op.identity_coop();
            }
          }
        }
      } else {
        uint32_t u[PER_LANE];
        float wt[WT ? PER_LANE : 1];
#pragma unroll
        for (int j = 0; j < PER_LANE; j++) {
          const unsigned long long k = b + lane + 32 * j;
          u[j] = k < e ? nbr_once(d, k, GG_SITE) : 0u;
          if constexpr (WT) wt[j] = k < e ? ld_once(d.w + k) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < PER_LANE; j++) {
          const unsigned long long k = b + lane + 32 * j;
          if constexpr (WT)
            vals[j] = k < e ? op.gather_w(u[j], wt[j]) : op.identity_coop();
          else
            vals[j] = k < e ? op.gather(d, k, u[j]) : op.identity_coop();
        }
      }
#pragma unroll
      for (int j = 0; j < PER_LANE; j++) part = op.combine(part, vals[j]);
    }
    part = op.warp_combine(part);
    if (lane == 0) partials[c] = part;
  }
}

// Long-list vertices of a call that activates nothing (PageRank, BC's
// backward sweep): one warp per vertex; the lanes read its chunk partials
// (coalesced, lane-strided), the warp tree combines them, lane 0 applies the
// slot.  Measured against the lane-per-vertex finish below: PageRank R-MAT 20
// 286 -> 326 GTEPS (there the lanes, adding up to 32 partials each in series,
// are latency-bound); calls with activations keep the lane form, which
// records a warp's 32 activations together (SSSP R-MAT 25: 145 against 138).
template <class Op>
__global__ void __launch_bounds__(PULL_THREADS)
    pull_big_finish_warps(Dir d, Op op, const typename Op::Acc *__restrict__ partials, Counters *ctr) {
  using Acc = typename Op::Acc;
  Tally t;
  const size_t nwarps = (size_t)gridDim.x * (PULL_THREADS / 32);
  const unsigned lane = lane_id();
  for (size_t i = (size_t)blockIdx.x * (PULL_THREADS / 32) + (threadIdx.x >> 5); i < d.nbig; i += nwarps) {
    const uint32_t v = d.big[i];
    if (!op.want(v)) continue;
    const uint32_t c0 = d.big_chunk[i], c1 = d.big_chunk[i + 1];
    Acc part = op.identity_coop();
    for (uint32_t c = c0 + lane; c < c1; c += 32) part = op.combine(part, partials[c]);
    part = op.warp_combine(part);
    if (lane == 0) op.finish(v, op.combine(op.identity(v), part), d.deg[v], t);
  }
  pull_flush<Op, PULL_THREADS>(t, false, ctr);
}

// g[0] .. g[N - 1] (N a power of two) combined in pairs: as many operations as
// one after another, a third of the rounding error on long lists.
template <int N, class Op>
__device__ __forceinline__ typename Op::Acc combine_tree(const Op &op, typename Op::Acc *g) {
#pragma unroll
  for (int s = 1; s < N; s *= 2)
#pragma unroll
    for (int j = 0; j < N; j += 2 * s) g[j] = op.combine(g[j], g[j + s]);
  return g[0];
}
// The running result of a list walked a few entries at a time.  Float sums
// (Op::kCompensated) keep the rounding errors of the additions beside the sum
// (Knuth's two-sum): a lane now adds up to 1024 entries itself, where chunks
// of 256 went through trees, and this leaves the ranks' error no larger (20
// iterations, 2-norm against 64 bits, mean of R-MAT graphs of 2^20, 2^22,
// 200003, 20001 and 1001 vertices: 6.15e-8 with the trees, 6.44e-8 without
// the errors kept, 5.95e-8 with; no difference in time).
template <class Op, class = void>
struct Running {
  typename Op::Acc a;
  __device__ __forceinline__ explicit Running(typename Op::Acc x) : a(x) {}
  __device__ __forceinline__ void add(const Op &op, typename Op::Acc x) { a = op.combine(a, x); }
  __device__ __forceinline__ typename Op::Acc value() const { return a; }
};
template <class Op>
struct Running<Op, std::enable_if_t<Op::kCompensated>> {
  float a, lost = 0.0f;
  __device__ __forceinline__ explicit Running(float x) : a(x) {}
  __device__ __forceinline__ void add(const Op &, float x) {
    const float s = __fadd_rn(a, x), b = __fsub_rn(s, a);
    lost = __fadd_rn(lost, __fadd_rn(__fsub_rn(a, __fsub_rn(s, b)), __fsub_rn(x, b)));
    a = s;
  }
  __device__ __forceinline__ float value() const { return __fadd_rn(a, lost); }
};

// One lane per long-list vertex combines its chunk partials in order (a warp
// does it for vertices with more than SERIAL chunks), then applies the slot.
// SPREAD: a warp takes vertices nwarps apart: on a hot-source direction the
// longest lists lead, and 32 of them in one warp are combined one after
// another (R-MAT 20: 32 us of a 75-us iteration).
template <class Op, uint32_t SERIAL, bool SPREAD>
__device__ __forceinline__ void big_finish(const Dir &d, const Op &op, const typename Op::Acc *partials,
                                           const ActOut &act, Tally &t) {
  using Acc = typename Op::Acc;
  const size_t stride = (size_t)gridDim.x * PULL_THREADS;
  const size_t n = SPREAD ? ((size_t)d.nbig + stride - 1) / stride * stride : ((size_t)d.nbig + 31) / 32 * 32;
  const unsigned lane = lane_id();
  const size_t tid = (size_t)blockIdx.x * PULL_THREADS + threadIdx.x;
  const size_t first = SPREAD ? (size_t)lane * (stride / 32) + tid / 32 : tid;
  for (size_t base = 0; base + (SPREAD ? 0 : tid) < n; base += stride) {
    const size_t i = base + first;
    const bool valid = i < d.nbig;
    const uint32_t v = valid ? d.big[i] : 0u;
    const bool todo = valid && op.want(v);
    uint32_t c0 = 0, c1 = 0;
    if (todo) {
      c0 = d.big_chunk[i];
      c1 = d.big_chunk[i + 1];
    }
    Acc acc = op.identity(v);
    if (todo && c1 - c0 <= SERIAL) {
      Running<Op> run(acc);
      for (uint32_t c = c0; c < c1; c++) run.add(op, partials[c]);
      acc = run.value();
    }
    unsigned coop = __ballot_sync(GG_FULL, todo && c1 - c0 > SERIAL);
    while (coop) {
      const unsigned leader = __ffs(coop) - 1;
      coop &= coop - 1;
      const uint32_t lc0 = __shfl_sync(GG_FULL, c0, leader), lc1 = __shfl_sync(GG_FULL, c1, leader);
      Running<Op> run(op.identity_coop());
      for (uint32_t c = lc0 + lane; c < lc1; c += 128) {
        Acc g[4];
#pragma unroll
        for (int j = 0; j < 4; j++) g[j] = c + 32 * j < lc1 ? partials[c + 32 * j] : op.identity_coop();
        run.add(op, combine_tree<4>(op, g));
      }
      const Acc part = op.warp_combine(run.value());
      if (lane == leader) acc = op.combine(acc, part);
    }
    const bool a = todo && op.finish(v, acc, d.deg[v], t);
    if (act.active_out) push_activate(a, v, act, t);
  }
}
template <class Op, uint32_t SERIAL, bool SPREAD>
__global__ void __launch_bounds__(PULL_THREADS)
    pull_big_finish(Dir d, Op op, const typename Op::Acc *partials, ActOut act, Counters *ctr) {
  Tally t;
  big_finish<Op, SERIAL, SPREAD>(d, op, partials, act, t);
  pull_flush<Op, PULL_THREADS>(t, act.active_out != nullptr, ctr);
}

// The reduction pull on a hot-source direction (Dir.sell_desc), one launch
// for every list and a finish for the long ones.
// Rows: the numbering sorts vertices of about equal out-degree by in-degree,
// so 32 consecutive vertices (a slice) have lists of nearly equal length and
// a lane walks its own list without waiting for longer ones.  The light
// lists of a slice are stored column-major, so a warp reads the next four
// entries of its 32 lists with one coalesced 16-byte load per lane, each
// lane adds up its own list (no tree, no partial result: on GB300 an FP64
// add costs a warp 16 cycles whatever the number of lanes that need it), and
// 32 results are finished at once.  The places past a list's end name vertex
// V: a dense op in double (has_dense; its state holds a neutral value there)
// reads them like any other, which takes the length tests from around its
// adds (double PageRank, 117 M edges: 9.9 -> 9.4 ms); the others stop at the
// list's length (in float the extra requests cost more: R-MAT 26 70 against
// 66 ms).
// Long lists: a warp per aligned chunk, lane-strided entries, 8 in flight.
// Slices whose 32 vertices have no list are left out where op.zero_kept()
// says that their values are in place.
// ALL: every gather through L1; else op.load's choice by source number.
// Four blocks of 256 threads per SM: what bounds the kernel is the L1s'
// rate of requests to L2 (at R-MAT 24 74% busy, one request per missing
// gather), and more resident warps lose L1 hits (R-MAT 26: 83 ms for 20
// iterations with six blocks of fewer registers, 67 with four).  The hottest
// 32 K sources' values in shared memory served the gathers that L1 serves
// here: no gain.
// PageRank, 20 iterations, against a lane-serial light kernel with warps
// over chunks beside it and a finish: float R-MAT 20 1.56 -> 1.03 ms, R-MAT
// 26 100 -> 66 ms; double, 7.3 M vertices and 117 M edges, 27.4 -> 8.7 ms.
template <class Op, class = void>
struct has_dense : std::false_type {};
template <class Op>
struct has_dense<Op, std::void_t<decltype(Op::kDense)>> : std::true_type {};
// Ops that can tell when a list need not be walked (on): skip(v) before its
// first entry, stop(acc, w) on the way (acc the result so far, w the weight
// of an entry at or before the next one).  Their identity(v) is the vertex's
// own value, so a list left out finishes with it; begin() runs once per thread
// before the first call of either.
template <class Op, class = void>
struct has_stop : std::false_type {};
template <class Op>
struct has_stop<Op, std::void_t<decltype(&Op::stop)>> : std::true_type {};
constexpr int ROWS_THREADS = 256;
constexpr int ROWS_BLOCKS = 4;  // per SM
constexpr int ROWS_Q = 2;       // columns of four entries in flight per lane
// walk_list: entries [b, e) of vertex v's list by a warp, the combined result
// in all lanes.
template <class Op, bool ALL>
__device__ __forceinline__ typename Op::Acc walk_list(const Dir &d, const Op &op, uint32_t v, unsigned long long b,
                                                      unsigned long long e) {
  using Acc = typename Op::Acc;
  constexpr bool WT = has_gather_w<Op>::value;
  constexpr bool STOP = has_stop<Op>::value;
  constexpr int CH = 8;
  const unsigned lane = lane_id();
  Running<Op> run(STOP ? op.identity(v) : op.identity_coop());
  const uint32_t n = (uint32_t)(e - b);
  for (uint32_t k0 = lane; k0 - lane < n; k0 += 32 * CH) {
    uint32_t u[CH];
    float wt[WT ? CH : 1];
#pragma unroll
    for (int j = 0; j < CH; j++) {
      const uint32_t k = k0 + 32 * j;
      u[j] = k < n ? nbr_once(d, b + k, GG_SITE) : 0u;
      if constexpr (WT) wt[j] = k < n ? ld_once(d.w + b + k) : 0.0f;
    }
    if constexpr (STOP) {
      // lane 0 holds the batch's first entry: with any lane's result
      const Acc best = op.warp_combine(run.value());
      float first = 0.0f;
      if constexpr (WT) first = __shfl_sync(GG_FULL, wt[0], 0);
      if (op.stop(best, first)) break;
    }
    Acc g[CH];
#pragma unroll
    for (int j = 0; j < CH; j++) {
      const uint32_t k = k0 + 32 * j;
      g[j] = k < n ? op.template value<ALL>(u[j], WT ? wt[WT ? j : 0] : 0.0f) : op.identity_coop();
    }
    run.add(op, combine_tree<CH>(op, g));
  }
  return op.warp_combine(run.value());
}

// rows_walk: the part of warp `warp` of `nwarps`; partials null: the long
// lists are somebody else's (SHARED: in the same step).
template <class Op, bool ALL, bool SHARED>
__device__ __forceinline__ void rows_walk(const Dir &d, uint32_t V, const Op &op, const ActOut &act, Tally &t,
                                          typename Op::Acc *partials, uint32_t warp, uint32_t nwarps) {
  using Acc = typename Op::Acc;
  constexpr bool WT = has_gather_w<Op>::value;
  constexpr bool DENSE = has_dense<Op>::value && sizeof(Acc) == 8;
  constexpr bool STOP = has_stop<Op>::value;
  const unsigned lane = lane_id();
  for (uint32_t c = warp; partials && c < d.nbigchunks; c += nwarps) {
    uint32_t v;
    unsigned long long lo, b, e;
    big_range(d, c, d.chunk, &v, &lo, &b, &e);
    bool walk = op.want(v);
    if constexpr (STOP) walk = walk && !op.skip(v);
    const Acc part = walk ? walk_list<Op, ALL>(d, op, v, b, e) : op.identity_coop();
    if (lane == 0) partials[c] = part;
  }
  const uint32_t nsl = op.zero_kept() ? d.nfull : d.nslices;
  uint4 ds = warp < nsl ? d.sell_desc[warp] : make_uint4(0, 0, 0, 0);
  for (uint32_t i = warp; i < nsl; i += nwarps) {
    const uint4 dn = i + nwarps < nsl ? d.sell_desc[i + nwarps] : make_uint4(0, 0, 0, 0);
    const uint32_t v = ds.x * 32 + lane;
    const uint32_t *col = reinterpret_cast<const uint32_t *>(d.sell_col + (size_t)ds.y * 32 + lane);
    const uint32_t *wcol = WT ? reinterpret_cast<const uint32_t *>(d.sell_w + (size_t)ds.y * 32 + lane) : nullptr;
    uint4 c[ROWS_Q], w[WT ? ROWS_Q : 1];
    w[0] = make_uint4(0, 0, 0, 0);
    // the first columns do not wait for the degrees
#pragma unroll
    for (int q = 0; q < ROWS_Q; q++) {
      c[q] = make_uint4(0, 0, 0, 0);
      if (ds.z > q) c[q] = ld_once_v4(col + 128 * q);
      if constexpr (WT) {
        w[q] = make_uint4(0, 0, 0, 0);
        if (ds.z > q) w[q] = ld_once_v4(wcol + 128 * q);
      }
    }
    const uint32_t deg = v < V ? d.deg[v] : 0u;
    const bool todo = v < V && deg <= d.light && op.want(v);
    uint32_t n = todo ? deg : 0u;
    if constexpr (STOP)
      if (n && op.skip(v)) n = 0;
    Running<Op> run(op.identity(v < V ? v : 0u));
    if constexpr (DENSE) {
      uint32_t t4 = 0;
      for (; t4 + ROWS_Q <= ds.z; t4 += ROWS_Q) {
        col += 128 * ROWS_Q;
        Acc g[4 * ROWS_Q];
#pragma unroll
        for (int q = 0; q < ROWS_Q; q++) {
          const uint32_t u[4] = {c[q].x, c[q].y, c[q].z, c[q].w};
#pragma unroll
          for (int j = 0; j < 4; j++) g[4 * q + j] = op.template value<ALL>(u[j], 0.0f);
        }
        // the next columns beside this step's gathers
#pragma unroll
        for (int q = 0; q < ROWS_Q; q++)
          if (t4 + ROWS_Q + q < ds.z) c[q] = ld_once_v4(col + 128 * q);
        run.add(op, combine_tree<4 * ROWS_Q>(op, g));
      }
#pragma unroll
      for (int q = 0; q < ROWS_Q - 1; q++)
        if (t4 + q < ds.z) {
          const uint32_t u[4] = {c[q].x, c[q].y, c[q].z, c[q].w};
          Acc g[4];
#pragma unroll
          for (int j = 0; j < 4; j++) g[j] = op.template value<ALL>(u[j], 0.0f);
          run.add(op, combine_tree<4>(op, g));
        }
    } else {
      for (uint32_t k = 0; k < n; k += 4 * ROWS_Q) {
        if constexpr (STOP) {
          if (op.stop(run.value(), __uint_as_float(w[0].x))) break;
          // where the last entry of this step ends the walk, its successors
          // are not read ahead
          if (WT && k + 4 * ROWS_Q < n && op.stop(run.value(), __uint_as_float(w[WT ? ROWS_Q - 1 : 0].w)))
            n = k + 4 * ROWS_Q;
        }
        col += 128 * ROWS_Q;
        wcol += 128 * ROWS_Q;
        Acc g[4 * ROWS_Q];
#pragma unroll
        for (int q = 0; q < ROWS_Q; q++) {
          const uint32_t u[4] = {c[q].x, c[q].y, c[q].z, c[q].w};
          const uint4 wq = w[WT ? q : 0];
          const uint32_t wb[4] = {wq.x, wq.y, wq.z, wq.w};
#pragma unroll
          for (int j = 0; j < 4; j++)
            g[4 * q + j] = k + 4 * q + j < n ? op.template value<ALL>(vertex_ok(d, u[j], GG_SITE),
                                                                      __uint_as_float(wb[j]))
                                             : op.identity_coop();
        }
        // the next columns beside this step's gathers
#pragma unroll
        for (int q = 0; q < ROWS_Q; q++)
          if (k + 4 * ROWS_Q + 4 * q < n) {
            c[q] = ld_once_v4(col + 128 * q);
            if constexpr (WT) w[q] = ld_once_v4(wcol + 128 * q);
          }
        run.add(op, combine_tree<4 * ROWS_Q>(op, g));
      }
    }
    const bool a = todo && op.finish(v, run.value(), deg, t);
    if (act.active_out) pull_activate<SHARED>(a, v, ds.x, act, t);
    ds = dn;
  }
}
// The long lists by a warp each, finished at once: for graphs whose lists are
// short enough that a barrier and partial results take longer.
template <class Op, bool ALL>
__device__ __forceinline__ void long_lists(const Dir &d, const Op &op, const ActOut &act, Tally &t, uint32_t warp,
                                           uint32_t nwarps) {
  for (uint32_t i = warp; i < d.nbig; i += nwarps) {
    const uint32_t v = d.big[i];
    bool walk = op.want(v);
    if constexpr (has_stop<Op>::value) walk = walk && !op.skip(v);
    const typename Op::Acc part = walk ? walk_list<Op, ALL>(d, op, v, d.off[v], d.off[v + 1]) : op.identity_coop();
    const bool a = lane_id() == 0 && op.want(v) && op.finish(v, op.combine(op.identity(v), part), d.deg[v], t);
    if (act.active_out) push_activate(a, v, act, t);
  }
}
template <class Op, bool ALL>
__global__ void __launch_bounds__(ROWS_THREADS, ROWS_BLOCKS)
    pull_rows(Dir d, uint32_t V, Op op, ActOut act, Counters *ctr, typename Op::Acc *partials) {
  if constexpr (has_stop<Op>::value) op.begin();
  Tally t;
  // consecutive slices and chunks on different SMs
  rows_walk<Op, ALL, false>(d, V, op, act, t, partials, (threadIdx.x >> 5) * gridDim.x + blockIdx.x,
                            gridDim.x * (ROWS_THREADS / 32));
  pull_flush<Op, ROWS_THREADS>(t, act.active_out != nullptr, ctr);
}

// ---------------------------------------------------------------- BFS pull
// toolkits/bfs.cpp:60-76: an unvisited vertex takes the FIRST in-neighbour
// (in CSC order) that is in the active set as its parent.  Every bin keeps
// that order: lanes scan their own list in order; a warp takes the lowest
// lane of the first 32-wide chunk with a hit; heavy chunks record the index
// of their first hit and the finish takes the lowest.
//
// bfs_walk: a warp per 32 consecutive vertices (the word of the bitmaps it
// owns).  What has to be read of a vertex is what bounds it (R-MAT 24: 511 MB
// of offsets, degrees and first entries): vertices that are visited or have
// no in-list cost two bits, the offsets of the others are read one group and
// their bits two groups ahead, degrees only of vertices reached.  A list
// without a hit in its first d.light entries goes on in the same warp, 32
// entries at a time, up to HEAVY_DEG entries (a kernel of a warp per such list
// took 237 us a call at R-MAT 26, nearly all of it finding visited vertices).
// HEAVY lists are bfs_heavy_first's from the start.
// CHUNKS: of 32 entries a warp reads at a time of the longer lists.  Two keep
// more loads in flight, one leaves the kernel 38 registers for 42: bfs_pull_walk
// at R-MAT 26 2.53 / 2.37 ms a BFS with two / one, bfs_dense_run at R-MAT 24 0.83
// / 0.86.
template <int CHUNKS>
__device__ __forceinline__ void bfs_walk(const Dir &d, uint32_t V, const uint32_t *active_in, uint32_t *parent,
                                         const ActOut &act, Tally &t, uint32_t warp, uint32_t nwarps) {
  const uint32_t groups = V / 32 + (V % 32 != 0);  // at most 2^27: g + 2 * nwarps fits
  const unsigned lane = lane_id();
  auto words = [&](uint32_t g, uint32_t &vis, uint32_t &todo) {
    vis = todo = 0;
    if (g < groups) {
      vis = act.visited[g];
      todo = d.nz[g] & ~vis;
    }
  };
  auto bounds = [&](uint32_t g, uint32_t todo, unsigned long long &b, uint32_t &n) {
    b = 0;
    n = 0;
    if ((todo >> lane) & 1u) {
      const size_t v = (size_t)g * 32 + lane;
      b = d.off[v];
      n = (uint32_t)(d.off[v + 1] - b);
    }
  };
  uint32_t vis, todo, vis1, todo1, n;
  unsigned long long b;
  words(warp, vis, todo);
  words(warp + nwarps, vis1, todo1);
  bounds(warp, todo, b, n);
  for (uint32_t g = warp; g < groups; g += nwarps) {
    uint32_t vis2, todo2, n1;
    unsigned long long b1;
    words(g + 2 * nwarps, vis2, todo2);
    bounds(g + nwarps, todo1, b1, n1);
    if (todo) {  // uniform
      uint32_t found = NONE32;
      const uint32_t lim = n > HEAVY_DEG ? 0u : n < d.light ? n : d.light;
      constexpr int STEP = 4;
      for (uint32_t k = 0; k < lim && found == NONE32; k += STEP) {
        uint32_t u[STEP];
#pragma unroll
        for (int j = 0; j < STEP; j++) u[j] = k + j < lim ? nbr_at(d, b + k + j, GG_SITE) : NONE32;
        unsigned hits = 0;
#pragma unroll
        for (int j = 0; j < STEP; j++) hits |= (u[j] != NONE32 && bm_test(active_in, u[j])) ? 1u << j : 0u;
#pragma unroll
        for (int j = STEP - 1; j >= 0; j--)
          if ((hits >> j) & 1u) found = u[j];
      }
      for (unsigned rest = __ballot_sync(GG_FULL, found == NONE32 && n > d.light && n <= HEAVY_DEG); rest;
           rest &= rest - 1) {
        const int j = __ffs(rest) - 1;
        const unsigned long long bj = __shfl_sync(GG_FULL, b, j);
        const uint32_t nj = __shfl_sync(GG_FULL, n, j);
        uint32_t hit = NONE32;
        for (uint32_t k = d.light + lane; k - lane < nj && hit == NONE32; k += 32 * CHUNKS) {
          uint32_t u[CHUNKS];
          bool h[CHUNKS];
#pragma unroll
          for (int c = 0; c < CHUNKS; c++) u[c] = k + 32 * c < nj ? nbr_at(d, bj + k + 32 * c, GG_SITE) : NONE32;
#pragma unroll
          for (int c = 0; c < CHUNKS; c++) h[c] = u[c] != NONE32 && bm_test(active_in, u[c]);
#pragma unroll
          for (int c = 0; c < CHUNKS; c++) {
            const unsigned m = __ballot_sync(GG_FULL, h[c]);
            if (m && hit == NONE32) hit = __shfl_sync(GG_FULL, u[c], __ffs(m) - 1);
          }
        }
        if ((int)lane == j) found = hit;
      }
      const bool a = found != NONE32;
      const unsigned bits = __ballot_sync(GG_FULL, a);
      if (lane == 0 && bits) {
        act.active_out[g] = bits;
        act.visited[g] = vis | bits;
      }
      if (a) {
        const size_t v = (size_t)g * 32 + lane;
        const uint32_t od = act.out_deg[v];
        parent[v] = found;
        t.activated += 1;
        t.edges += od;
        t.maxdeg = od > t.maxdeg ? od : t.maxdeg;
      }
    }
    vis = vis1;
    todo = todo1;
    vis1 = vis2;
    todo1 = todo2;
    b = b1;
    n = n1;
  }
}
// Six blocks of 256 threads per SM (R-MAT 26: 2.35 ms a BFS; eight, with
// spills, 3.25) and four entries a step (eight: 2.60).
constexpr int BFS_BLOCKS = 6;
static __global__ void __launch_bounds__(PULL_THREADS, BFS_BLOCKS)
    bfs_pull_walk(Dir d, uint32_t V, const uint32_t *active_in, uint32_t *parent, ActOut act, Counters *ctr) {
  Tally t;
  bfs_walk<1>(d, V, active_in, parent, act, t, (size_t)blockIdx.x * (PULL_THREADS / 32) + (threadIdx.x >> 5),
           (size_t)gridDim.x * (PULL_THREADS / 32));
  t.flush(ctr);
}

// partials[c] = edge index of the chunk's first active in-neighbour, or ~0.
__device__ __forceinline__ void bfs_heavy_walk(const Dir &d, const uint32_t *active_in, const uint32_t *visited,
                                               unsigned long long *first) {
  // one warp per HEAVY_CHUNK-entry chunk of a list longer than HEAVY_DEG;
  // first[h] = the lowest hit index of heavy vertex h, so a chunk starting
  // past it (or a vertex already visited) is skipped and a scan stops at it
  const size_t nwarps = (size_t)gridDim.x * (PULL_THREADS / 32);
  const unsigned lane = lane_id();
  for (size_t c = (size_t)blockIdx.x * (PULL_THREADS / 32) + (threadIdx.x >> 5); c < d.nchunks; c += nwarps) {
    const uint32_t h = d.chunk_owner[c];
    const uint32_t v = d.heavy[h];
    if (bm_test(visited, v)) continue;
    const unsigned long long b = d.off[v] + (unsigned long long)(c - d.heavy_chunk[h]) * HEAVY_CHUNK;
    const unsigned long long end = d.off[v + 1];
    const unsigned long long e = b + HEAVY_CHUNK < end ? b + HEAVY_CHUNK : end;
    for (unsigned long long base = b; base < e; base += 32) {
      unsigned long long best = 0;
      if (lane == 0) best = *(volatile unsigned long long *)(first + h);
      if (__shfl_sync(GG_FULL, best, 0) < base) break;
      const unsigned long long k = base + lane;
      const bool hit = k < e && bm_test(active_in, nbr_at(d, k, GG_SITE));
      const unsigned bal = __ballot_sync(GG_FULL, hit);
      if (bal) {
        if (lane == 0) atomicMin(first + h, base + (unsigned long long)(__ffs(bal) - 1));
        break;
      }
    }
  }
}

static __global__ void __launch_bounds__(PULL_THREADS)
    bfs_heavy_first(Dir d, const uint32_t *active_in, const uint32_t *visited, unsigned long long *first) {
  bfs_heavy_walk(d, active_in, visited, first);
}

// The heavy vertices' parents; first[] is left as it is needed by the next call.
__device__ __forceinline__ void bfs_heavy_take(const Dir &d, unsigned long long *first, uint32_t *parent,
                                               const ActOut &act, Tally &t) {
  const size_t n = ((size_t)d.nheavy + 31) / 32 * 32;
  for (size_t h = (size_t)blockIdx.x * blockDim.x + threadIdx.x; h < n; h += (size_t)gridDim.x * blockDim.x) {
    bool a = false;
    uint32_t v = 0;
    if (h < d.nheavy) {
      v = d.heavy[h];
      const unsigned long long f = first[h];
      if (f != ~0ull) {
        first[h] = ~0ull;
        if (!bm_test(act.visited, v)) {
          parent[v] = nbr_at(d, f, GG_SITE);
          a = true;
        }
      }
    }
    push_activate(a, v, act, t);
  }
}
static __global__ void __launch_bounds__(PULL_THREADS)
    bfs_heavy_finish(Dir d, unsigned long long *first, uint32_t *parent, ActOut act, Counters *ctr) {
  Tally t;
  bfs_heavy_take(d, first, parent, act, t);
  t.flush(ctr);
}

// ---------------------------------------------------------------- queue from bitmap
// popcount of (bm & mask) per 32-bit word: the scan input of queue_from_bitmap.
struct MaskedPopc {
  const uint32_t *bm;
  const uint32_t *mask;
  __device__ __forceinline__ uint32_t operator()(size_t i) const {
    uint32_t w = bm[i];
    if (mask) w &= mask[i];
    return (uint32_t)__popc(w);
  }
};

// q[pos[i] ...] = the vertices of word i of (bm & mask), ascending.
static __global__ void queue_scatter(const uint32_t *__restrict__ bm, const uint32_t *__restrict__ mask,
                                     size_t words, const uint32_t *__restrict__ pos, uint32_t *__restrict__ q) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t w = bm[i];
    if (mask) w &= mask[i];
    uint32_t p = pos[i];
    while (w) {
      uint32_t b = __ffs(w) - 1;
      w &= w - 1;
      q[p++] = (uint32_t)(i * 32 + b);
    }
  }
}

// ---------------------------------------------------------------- small kernels
// out[i] = src[q[i]]: the message snapshot of a push call's queued vertices.
template <typename T>
static __global__ void gather_by_queue(const uint32_t *__restrict__ q, uint32_t n, const T *__restrict__ src,
                                       T *__restrict__ out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = src[q[i]];
}

template <typename T>
static __global__ void fill_kernel(T *__restrict__ a, size_t n, T v) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    a[i] = v;
}

static __global__ void iota_u32(uint32_t *__restrict__ a, uint32_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    a[i] = (uint32_t)i;
}

// Sets the bits of the n queued vertices.
static __global__ void bitmap_from_queue(const uint32_t *__restrict__ q, uint32_t n, uint32_t *__restrict__ bm) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t v = q[i];
    atomicOr(bm + (v >> 5), 1u << (v & 31));
  }
}

// Bitmap::fill (core/bitmap.hpp:42-52): bits [0, V) set, the rest clear.
static __global__ void bitmap_fill(uint32_t *__restrict__ bm, size_t words, uint32_t V) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) {
    size_t lo = i * 32;
    uint32_t w;
    if (lo + 32 <= V)
      w = 0xffffffffu;
    else if (lo >= V)
      w = 0u;
    else
      w = (1u << (V - lo)) - 1u;
    bm[i] = w;
  }
}

// Launch helpers shared by the toolkits.
struct Launch {
  gg_graph *g;
  int launches = 0;
  explicit Launch(gg_graph *gr) : g(gr) {}
  unsigned pull_grid() const { return grid_for(((size_t)g->V + 31) / 32 * 32, PULL_THREADS, g->num_sms, 8); }
  unsigned push_grid(unsigned long long total) const {
    unsigned long long tiles = (total + PUSH_TILE - 1) / PUSH_TILE;
    unsigned long long cap = (unsigned long long)g->num_sms * 8;
    return (unsigned)(tiles < 1 ? 1 : (tiles > cap ? cap : tiles));
  }
  unsigned heavy_grid(const Dir &d) const {
    return grid_for((size_t)d.nchunks * 32, PULL_THREADS, g->num_sms, 8);
  }
  // Kernels one reduction pull launches.
  static int pull_launches(const Dir &d) { return d.sell_desc ? (d.nbig ? 2 : 1) : d.nbig ? 3 : 1; }
  // The pull of a hot-source direction (pull_rows): no second stream, the
  // long lists' chunks lead in the same launch.
  template <class Op>
  int pull_hot(const Dir &d, const Op &op, const ActOut &act, Counters *ctr) {
    cudaStream_t s = g->stream;
    typename Op::Acc *part = nullptr;
    if (d.nbig) GG_TRY(ws(g, WS_PARTIAL, d.nbigchunks, &part));
    const size_t warps = (size_t)(op.zero_kept() ? d.nfull : d.nslices) + d.nbigchunks;
    const unsigned grid = grid_for(warps * 32, ROWS_THREADS, g->num_sms, ROWS_BLOCKS);
    if (op.gathers_all(g->V))
      pull_rows<Op, true><<<grid, ROWS_THREADS, 0, s>>>(d, g->V, op, act, ctr, part);
    else
      pull_rows<Op, false><<<grid, ROWS_THREADS, 0, s>>>(d, g->V, op, act, ctr, part);
    launches += 1;
    if (d.nbig) {
      pull_big_finish<Op, 8, true><<<grid_for(d.nbig, PULL_THREADS, g->num_sms, 8), PULL_THREADS, 0, s>>>(d, op, part, act,
                                                                                                   ctr);
      launches += 1;
    }
    GG_CUDA(cudaGetLastError());
    return GG_OK;
  }
  // All bins of one dense call: rows, or the light kernel beside the chunks, then the finish.
  template <class Op>
  int pull(const Dir &d, const Op &op, const ActOut &act, Counters *ctr) {
    if (d.sell_desc) return pull_hot(d, op, act, ctr);
    cudaStream_t s = g->stream;
    // light lists on the side stream, beside the chunk kernel (disjoint
    // vertices); the finish, which sets bitmap bits atomically in words the
    // light kernel stores whole, runs after the join
    const bool fork = d.nbig && g->side;
    if (fork) {
      GG_CUDA(cudaEventRecord(g->fork, s));
      GG_CUDA(cudaStreamWaitEvent(g->side, g->fork, 0));
    }
    // split: both kernels resident on every SM at once (8 blocks of 256
    // threads fill an SM), rather than the chunk kernel waiting for the
    // light kernel's blocks to retire
    const uint32_t split = fork && g->pull_light_blocks > 0 && g->pull_light_blocks < 8 ? g->pull_light_blocks : 0;
    unsigned lg = pull_grid();
    if (split) lg = grid_for(((size_t)g->V + 31) / 32 * 32, PULL_THREADS, g->num_sms, (int)split);
    if (d.vec & 2)
      pull_light<Op, true><<<lg, PULL_THREADS, 0, fork ? g->side : s>>>(d, g->V, op, act, ctr);
    else
      pull_light<Op, false><<<lg, PULL_THREADS, 0, fork ? g->side : s>>>(d, g->V, op, act, ctr);
    launches += 1;
    if (fork) GG_CUDA(cudaEventRecord(g->join, g->side));
    if (d.nbig) {
      typename Op::Acc *part = nullptr;
      GG_TRY(ws(g, WS_PARTIAL, d.nbigchunks, &part));
      const unsigned cg = grid_for((size_t)d.nbigchunks * 32, PULL_THREADS, g->num_sms, split ? 8 - (int)split : 8);
      if (d.vec & 1) {
        if (d.chunk == 128)
          pull_chunks<Op, 4, true><<<cg, PULL_THREADS, 0, s>>>(d, op, part);
        else if (d.chunk == 512)
          pull_chunks<Op, 16, true><<<cg, PULL_THREADS, 0, s>>>(d, op, part);
        else
          pull_chunks<Op, 8, true><<<cg, PULL_THREADS, 0, s>>>(d, op, part);
      } else {
        if (d.chunk == 128)
          pull_chunks<Op, 4, false><<<cg, PULL_THREADS, 0, s>>>(d, op, part);
        else if (d.chunk == 512)
          pull_chunks<Op, 16, false><<<cg, PULL_THREADS, 0, s>>>(d, op, part);
        else
          pull_chunks<Op, 8, false><<<cg, PULL_THREADS, 0, s>>>(d, op, part);
      }
      if (fork) GG_CUDA(cudaStreamWaitEvent(s, g->join, 0));
      if (act.active_out)
        pull_big_finish<Op, 32, false><<<grid_for(d.nbig, PULL_THREADS, g->num_sms, 8), PULL_THREADS, 0, s>>>(d, op, part, act,
                                                                                                    ctr);
      else
        pull_big_finish_warps<Op><<<grid_for((size_t)d.nbig * 32, PULL_THREADS, g->num_sms, 8), PULL_THREADS, 0, s>>>(
            d, op, part, ctr);
      launches += 2;
    }
    GG_CUDA(cudaGetLastError());
    return GG_OK;
  }
  int bfs_pull(const Dir &d, const uint32_t *active_in, uint32_t *parent, const ActOut &act, Counters *ctr) {
    cudaStream_t s = g->stream;
    bfs_pull_walk<<<grid_for(((size_t)g->V + 31) / 32 * 32, PULL_THREADS, g->num_sms, BFS_BLOCKS), PULL_THREADS, 0, s>>>(
        d, g->V, active_in, parent, act, ctr);
    launches += 1;
    if (d.nheavy) {
      unsigned long long *first = nullptr;
      GG_TRY(ws(g, WS_PARTIAL, d.nheavy, &first));
      GG_CUDA(cudaMemsetAsync(first, 0xff, sizeof(unsigned long long) * d.nheavy, s));
      bfs_heavy_first<<<heavy_grid(d), PULL_THREADS, 0, s>>>(d, active_in, act.visited, first);
      bfs_heavy_finish<<<grid_for(d.nheavy, PULL_THREADS, g->num_sms, 8), PULL_THREADS, 0, s>>>(d, first, parent,
                                                                                                act, ctr);
      launches += 2;
    }
    GG_CUDA(cudaGetLastError());
    return GG_OK;
  }
  // Ordered queue of the set bits of bm (restricted to mask when non-null);
  // *n receives its length.
  int queue_from_bitmap(const uint32_t *bm, const uint32_t *mask, uint32_t *q, uint32_t *n) {
    size_t words = bitmap_words32(g->V);
    uint32_t *pos = nullptr, *scratch = nullptr;
    GG_TRY(ws(g, WS_QPOS, words + 1, &pos));
    GG_TRY(ws(g, WS_SCAN32, scan_scratch_elems(words), &scratch));
    GG_CUDA((exclusive_scan<uint32_t, MaskedPopc>(MaskedPopc{bm, mask}, words, pos, scratch, g->stream,
                                                  &launches)));
    queue_scatter<<<grid_for(words, 256, g->num_sms, 8), 256, 0, g->stream>>>(bm, mask, words, pos, q);
    launches += 1;
    GG_CUDA(cudaGetLastError());
    return read_small(g, n, pos + words, sizeof(uint32_t));
  }
  // Cooperative launches available (queried once per device).
  bool coop_ok() const {
    int v = 0;
    return cudaDeviceGetAttribute(&v, cudaDevAttrCooperativeLaunch, g->device) == cudaSuccess && v;
  }
  int scan_queue_degrees(const uint32_t *q, uint32_t n, const uint32_t *deg, unsigned long long **P) {
    unsigned long long *p = nullptr, *scratch = nullptr;
    GG_TRY(ws(g, WS_PREFIX, (size_t)g->V + 2, &p));
    GG_TRY(ws(g, WS_SCAN, scan_scratch_elems((size_t)g->V + 1), &scratch));
    GG_CUDA((exclusive_scan<unsigned long long, QueueDegreeIn>(QueueDegreeIn{q, deg}, n, p, scratch, g->stream,
                                                               &launches)));
    *P = p;
    return GG_OK;
  }
};

}  // namespace gg

#endif
