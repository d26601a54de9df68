// GB300 kinetic Delaunay engine: the persistent step kernel and its phases.
//
// One cooperative launch runs a whole kinetic step on the device:
//
//   move      new = old + d (or + v*dt), corners fixed   [DeviceTriangulation::movePoints,
//                                                          include/Device_Triangulation.h:395-410]
//   classify  every edge: orientation of both faces, incircle of the quad;
//             non-Delaunay edges go to a work-list       [delonize / untangle checks,
//                                                          include/Device_Triangulation.h:31-116]
//   stars     only when a face is inverted (the reference's untangle,
//             include/Device_Triangulation.h:422-495, handles only its B/C cases):
//             every vertex works out its own Delaunay star, checks it against its
//             neighbours' and makes it again until all agree, then the mesh is
//             rewritten (star.cuh); nothing is flipped;
//   repair    in its place where few vertices of a large mesh moved, or a few moved far,
//             where few faces turned in a large mesh, on the largest, where sub-steps are
//             asked for, or where stars do not agree (removal_first):
//             (1) revert vertices of non-positive faces to their old positions
//                 until every face is positive;
//             (2) remove the reverted vertices (flip each to degree 3, merge);
//             (3) Lawson to Delaunay;
//             (4) reinsert them at their new positions in parallel rounds
//                 (locate by walking, 1-to-3 / 2-to-4 split, Lawson).
//   lawson    parallel flip rounds over the work-list until it is empty
//             [delonize2, include/Device_Triangulation.h:324-351]: a candidate
//             flips when its hashed priority beats every candidate sharing a
//             face with it, so each round flips an independent set and the
//             highest-priority candidate always flips (no livelock).
//
// Rounds are separated by grid-wide barriers; nothing returns to the host
// between rounds.  Stars from the points' Morton order build the initial triangulation,
// and where they fail the repair's insertion rounds do.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include <unistd.h>

#include "engine.cuh"
#include "star.cuh"

namespace cg = cooperative_groups;

namespace mcl {

constexpr int kThreads = 256;
constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------------------
// Warp-aggregated append to a global work-list: one atomicAdd per warp that
// has items, no block barrier (so warps never wait for each other between
// loop iterations and memory latency overlaps freely).  All 32 lanes of the
// warp must call it together; lanes without items pass k = 0.
template <int K>
__device__ __forceinline__ void warp_push(const int (&mine)[K], int k, int* gl, int* gcount, int gcap,
                                          DevState* st) {
  const int lane = threadIdx.x & 31;
  int x = k;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  const int total = __shfl_sync(kFull, x, 31);
  if (total == 0) return;
  int base = 0;
  if (lane == 31) base = atomicAdd(gcount, total);
  base = __shfl_sync(kFull, base, 31);
  const int off = base + x - k;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    if (j < k) {
      if (off + j < gcap) __stcg(gl + off + j, mine[j]);
      else if (atomicCAS(&st->status, MCL_OK, MCL_ERR_CAPACITY) == MCL_OK) st->site = __LINE__;
    }
  }
}

#define set_error(P, code) flag_error_at(P, code, __LINE__)

// A per-thread count added to a global counter with one atomic per warp (every
// lane calls it): after a pass in which most threads count something, one
// atomic per thread on a single address would queue for tens of microseconds.
template <typename T>
__device__ __forceinline__ void warp_add(T* p, long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(p, (T)v);
}

// A warp's appends to a global list gathered in a shared-memory buffer of
// kWarpBuf entries and written out with one atomicAdd per flush (when the next
// append could overflow it, and at the end of the pass): a pass whose every
// warp appends on most iterations (the classification of a step that moves
// every vertex by a random walk) would otherwise queue thousands of atomics on
// one counter.  `n` is the same in every lane; calls are warp-uniform.
constexpr int kWarpBuf = 128;
struct WarpBuf {
  int* buf;  // this warp's kWarpBuf slots
  int n;
};
__device__ __forceinline__ void wb_flush(WarpBuf& b, int* gl, int* gcount, int gcap, DevState* st) {
  if (b.n == 0) return;
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0) base = atomicAdd(gcount, b.n);
  base = __shfl_sync(kFull, base, 0);
  for (int i = lane; i < b.n; i += 32) {
    if (base + i < gcap) __stcg(gl + base + i, b.buf[i]);
    else if (atomicCAS(&st->status, MCL_OK, MCL_ERR_CAPACITY) == MCL_OK) st->site = __LINE__;
  }
  __syncwarp();  // every lane has read the buffer before it is refilled
  b.n = 0;
}
template <int K>
__device__ __forceinline__ void wb_push(WarpBuf& b, const int (&mine)[K], int k, int* gl, int* gcount, int gcap,
                                        DevState* st) {
  static_assert(32 * K <= kWarpBuf, "one append must fit an empty buffer");
  const int lane = threadIdx.x & 31;
  int x = k;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  const int total = __shfl_sync(kFull, x, 31);
  if (total == 0) return;
  if (b.n + total > kWarpBuf) wb_flush(b, gl, gcount, gcap, st);
  const int off = b.n + x - k;
#pragma unroll
  for (int j = 0; j < K; ++j)
    if (j < k) b.buf[off + j] = mine[j];
  __syncwarp();  // the entries are visible to the lanes of a later flush
  b.n += total;
}

// This thread's position in the spread order used by whole-grid loops over a
// work-list: warp slot w of block b has spread index w * gridDim.x + b, so a
// short list is dealt out one warp per block (across every SM) instead of
// filling the first blocks.  Its item chains are latency-bound, and packed
// onto a few SMs their scattered loads, stores and atomics queue behind each
// other in those SMs' memory pipelines.  A permutation of the global thread
// ids; the warp's first lane has index spread_tid() - lane.
__device__ __forceinline__ int spread_tid() {
  return (int)(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) << 5) + (int)(threadIdx.x & 31);
}

__device__ __forceinline__ bool enqueue_once(const KParams& P, int e, unsigned stamp) {
  return atomicMax(P.qmark + e, stamp) < stamp;
}

// Append v to a global list from divergent code: the threads that reach the
// call together share one atomicAdd (their coalesced group's leader).
__device__ __forceinline__ void push_coalesced(const KParams& P, int* list, int* count, int cap, int v) {
  cg::coalesced_group grp = cg::coalesced_threads();
  int base = 0;
  if (grp.thread_rank() == 0) base = atomicAdd(count, (int)grp.size());
  base = grp.shfl(base, 0);
  const int at = base + (int)grp.thread_rank();
  if (at < cap) __stcg(list + at, v);
  else flag_error(P, MCL_ERR_CAPACITY);
}

// The repair's final Lawson pass starts from every edge its removals and
// splits touched: each is marked (stamp mk in qmark, no return value waited
// for) and appended, with the others of its removal or split, to work-list 0
// after the classification's non-Delaunay edges (one atomicAdd per removal or
// split).  Appends may repeat an edge; before the pass the list is deduplicated
// when it is short, and rebuilt from the marks by a pass over every edge when
// it is long or did not fit (mark_ovf).  mk == 0 marks nothing.
__device__ __forceinline__ void mark_edge(const KParams& P, int e, unsigned mk) {
  if (mk && e >= 0 && e < P.E) atomicMax(P.qmark + e, mk);
}
__device__ __forceinline__ int reserve_marks(const KParams& P, unsigned mk, int cnt) {
  return (mk && P.append_marks) ? atomicAdd(&P.st->wl_count[0], cnt) : -1;
}
__device__ __forceinline__ void append_mark(const KParams& P, int base, int j, int cnt, int e) {
  if (base < 0) return;
  if (base + cnt <= P.E) __stcg(P.wl0 + base + j, e);
  else if (j == 0) P.st->mark_ovf = 1;
}

// Called by every thread of the block (it holds a block barrier).
__device__ void flush_counters(const KParams& P, LocalCounters& lc) {
  // the common counter is reduced over the block (one atomic per block: one
  // per warp on a single address cost microseconds at the end of every step),
  // atomics for the rare ones
  __shared__ unsigned long long part[kThreads / 32];
  __syncthreads();  // one flush may follow another: the sums of the last have been read
  unsigned long long inc = lc.incircle;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) inc += __shfl_down_sync(kFull, inc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    if (t) atomicAdd(&P.st->c[C_INCIRCLE], t);
  }
  if (lc.incircle_fp64) atomicAdd(&P.st->c[C_INCIRCLE_FP64], (unsigned long long)lc.incircle_fp64);
  if (lc.incircle_exact) atomicAdd(&P.st->c[C_INCIRCLE_EXACT], (unsigned long long)lc.incircle_exact);
  if (lc.orient_fp64) atomicAdd(&P.st->c[C_ORIENT_FP64], (unsigned long long)lc.orient_fp64);
  if (lc.orient_exact) atomicAdd(&P.st->c[C_ORIENT_EXACT], (unsigned long long)lc.orient_exact);
  if (lc.sos) atomicAdd(&P.st->c[C_SOS], (unsigned long long)lc.sos);
  if (lc.overflow) {
    atomicAdd(&P.st->c[C_OVERFLOW], 1ull);
    set_error(P, MCL_ERR_PREDICATE);
  }
}

// ---------------------------------------------------------------------------
// New position of v for a fused move: pos_old + displacement (or + v*dt);
// fixed vertices (bounding corners) stay.  pos_old, disp, vel and dt are
// read-only for the whole launch, so they go through the read-only cache.
// Every load is issued before the fixed-vertex test (no load waits on another).
__device__ __forceinline__ float2 moved_pos(const KParams& P, int v) {
  const float2 p = __ldg(P.pos_old + v);
  const bool fixed = __ldg(P.vfix + v) != 0;
  float2 q = p;
  if (P.move_mode == MOVE_DISPLACE) {
    const float2 d = __ldg(P.disp + v);
    q.x = fadd(p.x, d.x);
    q.y = fadd(p.y, d.y);
  } else if (P.move_mode == MOVE_INTEGRATE) {
    const float2 u = __ldg(P.vel + v);
    const float t = __ldg(P.dt + v);
    q.x = fadd(p.x, fmul(u.x, t));
    q.y = fadd(p.y, fmul(u.y, t));
  }
  return fixed ? p : q;
}

// Phase A of a flip round for edge e (already known to be non-Delaunay): claim
// both faces with a priority key, remember the face ids for phase B.
__device__ __forceinline__ void claim_edge_with(const KParams& P, int e, int4 w, unsigned sc) {
  const int fa = min(2 * e, min(w.x, w.y)), fb = min(2 * e + 1, min(w.z, w.w));
  const unsigned long long key = ((unsigned long long)sc << 32) | (unsigned)(~mix32((unsigned)e ^ sc));
  atomicMax(P.claim + fa, key);
  atomicMax(P.claim + fb, key);
  __stcg(P.efa + e, make_int2(fa, fb));
  __stcg(P.cand + e, sc);
}
__device__ __forceinline__ void claim_edge(const KParams& P, int e, unsigned sc) {
  claim_edge_with(P, e, ld_en(P, e), sc);
}

// The vertices of an edge that is not Delaunay or has a non-positive face: if
// the step has a face to untangle, their stars are made anew (star.cuh).  Only
// the step's first classification marks (kFixedPos): the removal path keeps its
// own marks in vmark.
template <bool kMark>
__device__ __forceinline__ void mark_quad(const KParams& P, const int4 q, unsigned stamp) {
  if (!kMark) return;
  __stcg(P.vmark + q.x, (int)stamp);
  __stcg(P.vmark + q.y, (int)stamp);
  if (q.z >= 0) __stcg(P.vmark + q.z, (int)stamp);
  if (q.w >= 0) __stcg(P.vmark + q.w, (int)stamp);
}

// Full predicate ladder for one edge: counts its non-positive faces into `bad`
// and returns true when both faces are positive and the edge is non-Delaunay.
// (An edge that is either marks the vertices of its quad and itself: `cand` is
// the claim's stamp for one, set here for the other.)
template <bool kFixedPos>
__device__ __forceinline__ bool resolve_edge(const KParams& P, int e, unsigned qstamp, unsigned sc, LocalCounters& lc,
                                             int& bad) {
  const int4 q = ld_ev(P, e);
  const float2 a = ldpos_t<kFixedPos>(P, q.x), b = ldpos_t<kFixedPos>(P, q.y);
  const float2 c = q.z >= 0 ? ldpos_t<kFixedPos>(P, q.z) : a;
  const float2 d = q.w >= 0 ? ldpos_t<kFixedPos>(P, q.w) : a;
  const int sa = q.z >= 0 ? orient_v(P, a, b, c, lc) : 1;
  const int sb = q.w >= 0 ? orient_v(P, b, a, d, lc) : 1;
  if (sa <= 0 || sb <= 0) {
    bad += (sa <= 0) + (sb <= 0);
    mark_quad<kFixedPos>(P, q, qstamp);
    __stcg(P.cand + e, sc);
    return false;
  }
  if (q.z < 0 || q.w < 0) return false;
  lc.incircle++;
  if (incircle_sos(a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, q.x, q.y, q.z, q.w, &lc, &lc.overflow) <= 0) return false;
  mark_quad<kFixedPos>(P, q, qstamp);
  return true;
}

// ---------------------------------------------------------------------------
// Phase: (move +) classify every edge.  With a move, a vertex pass writes the
// new positions first (one grid barrier).  Counts non-positive faces;
// non-Delaunay edges of positive faces are queued on work-list 0 and claim
// their faces for the first flip round (stamp sc).
//
// The edge loop evaluates only the FP32 filters: an out-of-line call to the
// FP64 / exact / perturbation stages inside the loop would cost more than the
// whole filter.  Edges the filters cannot decide (a few per million) go to the
// hard list, which is resolved with the full ladder after the barrier; the
// caller must call phase_classify_hard before reading `inverted`.
__device__ __forceinline__ void timeline(const KParams& P, int slot) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && slot < kTimeline) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    P.st->ts[slot] = t;
  }
}

// the latest time any block reached this point
__device__ __forceinline__ void timeline_max(const KParams& P, int slot) {
  if (threadIdx.x == 0 && slot >= 43 && slot < 47) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    atomicMax(&P.st->tsmax[slot - 43], t);
  }
}

// Edges per thread and iteration of the classification pass; vertices per
// thread and iteration of its move pass.
constexpr int kClassifyUnroll = 4;
constexpr int kMoveUnroll = 4;

// The classification streams the edge records through shared memory one
// iteration ahead of their use (cp.async, 16 bytes per record, L2-coherent):
// kEvStages iterations of kClassifyUnroll records per thread.  Each thread
// copies and reads only its own slots, so completion is a cp.async.wait_group
// of the thread itself and no block barrier is involved.  The first
// iteration's records are requested before the move pass, which hides them.
constexpr int kEvStages = 2;
// Behind them the classification's append buffers (non-Delaunay edges, edges of
// a face turned over): kWarpBuf entries per warp each.  One block of shared
// memory, which the star phases use whole for their candidate lists.
constexpr int kEvSlots = kEvStages * kClassifyUnroll * kThreads;
constexpr int kStarSlots = 15;  // candidates per thread in the pool
constexpr int kPool = kStarSlots * 12 * kThreads / 16;
static_assert(kPool >= kEvSlots + 2 * (kThreads / 32) * kWarpBuf / 4, "the staging slots and buffers fit");
__shared__ int4 s_pool[kPool];
__device__ __forceinline__ int4* ev_slot(int stage, int j) {
  return s_pool + (stage * kClassifyUnroll + j) * kThreads + threadIdx.x;
}
__device__ __forceinline__ int* warp_buf(int which) {
  return reinterpret_cast<int*>(s_pool + kEvSlots) + (which * (kThreads / 32) + (threadIdx.x >> 5)) * kWarpBuf;
}

__device__ __forceinline__ void cp_async16(int4* smem, const int4* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Request the records of the classification iteration at `base` into stage
// `st` (one commit group, empty past the end).
__device__ __forceinline__ void stage_edges(const KParams& P, int base, int st) {
#pragma unroll
  for (int j = 0; j < kClassifyUnroll; ++j) {
    const int ei = base + j * blockDim.x + threadIdx.x;
    if (ei < P.E_it) cp_async16(ev_slot(st, j), P.ev + edge_at(P, ei));
  }
  cp_async_commit();
}

// Iterate the outgoing half-edges of v counter-clockwise.
template <typename F>
__device__ bool for_spokes(const KParams& P, int v, F f) {
  const int s0 = ld_i(P.vhe + v);
  if (s0 < 0 || s0 >= 2 * P.E) return false;
  int h = s0;
  for (int k = 0; k < 1024; ++k) {
    f(h);
    h = he_prev(P, h) ^ 1;
    if (h < 0 || h >= 2 * P.E) return false;
    if (h == s0) return true;
  }
  return false;
}

// A step moves few vertices (an aggregation whose walkers froze, a single
// point moved): classify only the edges of their stars and the sides opposite
// them (the edges whose quads hold a moved vertex), each once per launch
// (stamp qstamp in `win`), with the full predicate ladder; work-lists and
// claims as the full pass makes them.  Worth it while the movers touch well
// under all the edges.
constexpr int kSparseEdgesPerMover = 32;

__device__ __forceinline__ void push_one(const KParams& P, int* list, int* count, int e) {
  const int at = atomicAdd(count, 1);
  if (at < P.E) list[at] = e;
  else flag_error(P, MCL_ERR_CAPACITY);
}

template <bool kFixedPos>
__device__ void classify_one(const KParams& P, int e, unsigned qstamp, unsigned sc, LocalCounters& lc, int& bad) {
  if (e < 0 || e >= P.E || atomicMax(P.win + e, qstamp) >= qstamp) return;
  const int4 q = ld_ev(P, e);
  if (q.x < 0) return;
  if (bad_v(P, q.x) || bad_v(P, q.y) || q.z >= P.V || q.w >= P.V) {
    flag_error(P, MCL_ERR_DEGENERATE_INPUT);
    return;
  }
  const int bad0 = bad;
  if (resolve_edge<kFixedPos>(P, e, qstamp, sc, lc, bad) && enqueue_once(P, e, qstamp)) {
    claim_edge(P, e, sc);
    push_one(P, P.wl0, &P.st->wl_count[0], e);
  }
  if (bad != bad0) push_one(P, P.wl1, &P.st->wl_count[1], e);
}

// A warp per mover: all lanes walk the star, sixteen spokes at a time, then lane k takes
// the k-th spoke and lane 16 + k the side opposite, so a mover waits for its records,
// marks, positions and claims once instead of once per edge (48 served meshes of
// 460,000 vertices, 2 % of which move: the launch up to here 126 -> 72 us, the pass 890 ->
// 822).
template <bool kFixedPos>
__device__ void classify_movers(const KParams& P, int nm, unsigned qstamp, unsigned sc, LocalCounters& lc) {
  const int nwarps = (gridDim.x * blockDim.x) >> 5, lane = threadIdx.x & 31;
  int bad = 0;
  for (int i = spread_tid() >> 5; i < nm; i += nwarps) {
    const int s0 = ld_i(P.vhe + ld_i(P.vl0 + i));
    int h = s0, turns = 0;
    bool ok = s0 >= 0 && s0 < 2 * P.E, closed = false;
    while (ok && !closed) {
      int e = -1;
      for (int k = 0; k < 16 && ok && !closed; ++k) {
        const int4 w = ld_en(P, h >> 1);
        const int nx = (h & 1) ? w.z : w.x, pr = (h & 1) ? w.w : w.y;
        if (lane == k) e = h >> 1;
        if (lane == 16 + k) e = nx >> 1;
        h = pr ^ 1;
        ok = h >= 0 && h < 2 * P.E;
        closed = h == s0;
      }
      if (e >= 0) classify_one<kFixedPos>(P, e, qstamp, sc, lc, bad);
      __syncwarp();
      if (++turns == 64 && !closed) ok = false;
    }
    if (!ok && lane == 0) flag_error(P, MCL_ERR_DEGENERATE_INPUT);
  }
  warp_add(&P.st->inverted, bad);
}

// Returns whether only the movers' stars were classified.
template <bool kFixedPos>
__device__ bool phase_classify(cg::grid_group& g, const KParams& P, unsigned qstamp, unsigned sc,
                               LocalCounters& lc) {
  const int stride = gridDim.x * blockDim.x;
  constexpr int U = kClassifyUnroll;
  const int first = blockIdx.x * blockDim.x * U;
  stage_edges(P, first, 0);
  if (P.move_mode != MOVE_NONE) {
    // kMoveUnroll vertices per thread and iteration, every load before any
    // store (the pass is a stream: its loads must overlap)
    // The vertices that actually move are listed (work-list vl0, free until
    // the repair) when the last launch moved few: when they are few, only the
    // edges whose quads hold one of them are classified (every other edge
    // kept the positions of the last step, which left the mesh Delaunay).
    // A launch that moves most vertices after one that did lists nothing
    // (listing them would wait on an append per warp and iteration); the
    // movers are counted either way, for the next launch's choice.
    constexpr int UM = kMoveUnroll;
    const bool listing =
        P.sparse_ok && (long long)ld_i(&P.st->movers_last) * kSparseEdgesPerMover < (long long)P.E_it;
    int moved = 0;
    for (int base = blockIdx.x * blockDim.x * UM; base < P.V_it; base += stride * UM) {
      int v[UM];
      float2 np[UM];
#pragma unroll
      for (int j = 0; j < UM; ++j) {
        const int i = base + j * blockDim.x + threadIdx.x;
        v[j] = i < P.V_it ? vert_at(P, i) : -1;
        if (v[j] >= 0) np[j] = moved_pos(P, v[j]);
      }
      int mv[UM];
      int km = 0;
#pragma unroll
      for (int j = 0; j < UM; ++j)
        if (v[j] >= 0) {
          __stcg(P.pos + v[j], np[j]);
          const float2 po = __ldg(P.pos_old + v[j]);
          if (__float_as_uint(np[j].x) != __float_as_uint(po.x) || __float_as_uint(np[j].y) != __float_as_uint(po.y))
            mv[km++] = v[j];
        }
      moved += km;
      if (listing && __any_sync(kFull, km > 0)) warp_push(mv, km, P.vl0, &P.st->vl_count[0], P.V, P.st);
    }
    warp_add(&P.st->movers_now, moved);
    if (kFixedPos) timeline_max(P, 43);
    g.sync();
    if (kFixedPos) timeline_max(P, 44);
    const int nm = ld_i(&P.st->vl_count[0]);
    if (listing && (long long)nm * kSparseEdgesPerMover < (long long)P.E_it) {
      cp_async_wait<0>();  // the prefetched records are not used
      classify_movers<kFixedPos>(P, nm, qstamp, sc, lc);
      if (kFixedPos) timeline_max(P, 45);
      return true;
    }
  }
  int bad = 0;
  unsigned ninc = 0;
  int def0 = -1, def1 = -1;  // edges deferred to the full ladder after the loop
  WarpBuf wnd{warp_buf(0), 0}, winv{warp_buf(1), 0};
  // kClassifyUnroll edges per thread and iteration, their records and
  // positions loaded before any is evaluated (memory-level parallelism: the
  // pass is latency-bound on the position gathers); edge j of the iteration
  // at base is base + j * blockDim.x + threadIdx.x, so every load stays
  // coalesced across the warp.
  int it = 0;
  for (int base = first; base < P.E_it; base += stride * U, ++it) {
    stage_edges(P, base + stride * U, (it + 1) % kEvStages);
    cp_async_wait<kEvStages - 1>();  // this iteration's records have landed
    int4 q[U];
    int e[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int ei = base + j * blockDim.x + threadIdx.x;
      e[j] = ei < P.E_it ? edge_at(P, ei) : -1;
      q[j] = e[j] >= 0 ? *ev_slot(it % kEvStages, j) : make_int4(-1, -1, -1, -1);
    }
    float2 pa[U], pb[U], pc[U], pd[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int4 r = q[j];
      const bool ok = r.x >= 0 && !(bad_v(P, r.x) || bad_v(P, r.y) || r.z >= P.V || r.w >= P.V);
      if (r.x >= 0 && !ok) {
        flag_error(P, MCL_ERR_DEGENERATE_INPUT);
        q[j].x = -1;
      }
      if (ok) {
        pa[j] = ldpos_t<kFixedPos>(P, r.x);
        pb[j] = ldpos_t<kFixedPos>(P, r.y);
        pc[j] = r.z >= 0 ? ldpos_t<kFixedPos>(P, r.z) : pa[j];
        pd[j] = r.w >= 0 ? ldpos_t<kFixedPos>(P, r.w) : pa[j];
      }
    }
    int mine[U];
    int k = 0;
    int hard[U];
    int kh = 0;
    int inv[U];
    int ki = 0;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int4 r = q[j];
      if (r.x < 0) continue;
      const float2 a = pa[j], b = pb[j], c = pc[j], d = pd[j];
      const int sa = r.z >= 0 ? orient2d_fp32(a.x, a.y, b.x, b.y, c.x, c.y) : 1;
      const int sb = r.w >= 0 ? orient2d_fp32(b.x, b.y, a.x, a.y, d.x, d.y) : 1;
      bool defer = false;
      if (sa == 2 || sb == 2) {
        defer = true;
      } else if (sa <= 0 || sb <= 0) {
        bad += (sa <= 0) + (sb <= 0);
        mark_quad<kFixedPos>(P, r, qstamp);
        __stcg(P.cand + e[j], sc);
        inv[ki++] = e[j];
      } else if (r.z >= 0 && r.w >= 0) {
        ++ninc;
        const int si = incircle_fp32(a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y);
        if (si == 2) {
          defer = true;
        } else if (si > 0) {
          // each edge comes once in this pass and qstamp is the launch's
          // first stamp: the queue mark is a plain store (no atomic waited for)
          __stcg(P.qmark + e[j], qstamp);
          mark_quad<kFixedPos>(P, r, qstamp);
          // once a face has turned over no flip round uses these claims, so a thread
          // that has seen one claims no more (1M random walkers: 85 -> 78 us)
          if (!kFixedPos || bad == 0) claim_edge(P, e[j], sc);
          else __stcg(P.cand + e[j], sc);
          mine[k++] = e[j];
        }
      }
      if (defer) {
        if (def0 < 0) def0 = e[j];
        else if (def1 < 0) def1 = e[j];
        else hard[kh++] = e[j];
      }
    }
    if (__any_sync(kFull, k > 0)) wb_push(wnd, mine, k, P.wl0, &P.st->wl_count[0], P.E, P.st);
    if (__any_sync(kFull, kh > 0)) warp_push(hard, kh, P.hard, &P.st->hard_count, P.E, P.st);
    // edges with a non-positive face: the repair's first send-back pass
    // starts from them (work-list 1 is free until the flip rounds)
    if (__any_sync(kFull, ki > 0)) wb_push(winv, inv, ki, P.wl1, &P.st->wl_count[1], P.E, P.st);
  }
  wb_flush(wnd, P.wl0, &P.st->wl_count[0], P.E, P.st);
  wb_flush(winv, P.wl1, &P.st->wl_count[1], P.E, P.st);
  cp_async_wait<0>();  // nothing left in flight into the staging slots
  // the deferred edges, with the full predicate ladder (out of the loop, so
  // the out-of-line calls do not weigh on the loop above)
  {
    int mine[2];
    int k = 0;
    int inv[2];
    int ki = 0;
    const int defs[2] = {def0, def1};
    for (int j = 0; j < 2; ++j) {
      const int e = defs[j];
      if (e < 0) continue;
      const int bad0 = bad;
      if (resolve_edge<kFixedPos>(P, e, qstamp, sc, lc, bad) && enqueue_once(P, e, qstamp)) {
        claim_edge(P, e, sc);
        mine[k++] = e;
      }
      if (bad != bad0) inv[ki++] = e;
    }
    if (__any_sync(kFull, k > 0)) warp_push(mine, k, P.wl0, &P.st->wl_count[0], P.E, P.st);
    if (__any_sync(kFull, ki > 0)) warp_push(inv, ki, P.wl1, &P.st->wl_count[1], P.E, P.st);
  }
  lc.incircle += ninc;
  warp_add(&P.st->inverted, bad);
  if (kFixedPos) timeline_max(P, 45);
  return false;
}

// Resolve the hard list of phase_classify (after its barrier) with the full
// predicate ladder.  Returns after a barrier when there was anything to do.
template <bool kFixedPos>
__device__ void phase_classify_hard(cg::grid_group& g, const KParams& P, unsigned qstamp, unsigned sc,
                                    LocalCounters& lc) {
  const int n = ld_i(&P.st->hard_count);
  if (n == 0) return;  // uniform: read after the classification barrier
  const int stride = gridDim.x * blockDim.x;
  int bad = 0;
  const int lane = threadIdx.x & 31;
  for (int base = spread_tid() - lane; base < n; base += stride) {
    const int i = base + lane;
    int mine[1];
    int k = 0;
    int inv[1];
    int ki = 0;
    if (i < n) {
      const int e = ld_i(P.hard + i);
      const int bad0 = bad;
      if (resolve_edge<kFixedPos>(P, e, qstamp, sc, lc, bad) && enqueue_once(P, e, qstamp)) {
        claim_edge(P, e, sc);
        mine[k++] = e;
      }
      if (bad != bad0) inv[ki++] = e;
    }
    if (__any_sync(kFull, k > 0)) warp_push(mine, k, P.wl0, &P.st->wl_count[0], P.E, P.st);
    if (__any_sync(kFull, ki > 0)) warp_push(inv, ki, P.wl1, &P.st->wl_count[1], P.E, P.st);
  }
  if (bad) atomicAdd(&P.st->inverted, bad);
  g.sync();
}

__device__ __forceinline__ void timeline_remove(const KParams& P, int slot) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && slot < 64) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    P.st->ts_remove[slot] = t;
  }
}

__device__ __forceinline__ void timeline_insert(const KParams& P, int round, int k) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && round < 16) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    P.st->ts_insert[4 * round + k] = t;
  }
}

// ---------------------------------------------------------------------------
// Lawson flip rounds starting from work-list `src`.  A round is two phases:
//   A  every queued edge that is still non-Delaunay claims its two faces with
//      a hashed priority (atomicMax on the face's smallest half-edge);
//   B  an edge that holds both claims flips and queues its four wing edges;
//      other candidates queue themselves again.
// Winners share no face, so their writes never overlap; the candidate with the
// highest priority always wins both faces, so every round flips at least once.
// If pre_sc != 0 the first round's phase A was done by the classification.
// One flip round over `in[0..n)` by the threads [t0, t0+nt) (a whole grid or a
// single block); `sync` is the matching barrier.
template <bool kFixedPos, typename Sync>
__device__ __forceinline__ int lawson_round(const KParams& P, const int* in, int n, int* out, int* out_count,
                                            unsigned sc, unsigned sq, bool do_phase_a, int t0, int nt,
                                            LocalCounters& lc, Sync sync) {
  if (do_phase_a) {
    for (int i = t0; i < n; i += nt) {
      const int e = ld_i(in + i);
      const int4 q = ld_ev(P, e);
      const int4 w = ld_en(P, e);  // loaded with q: no load waits for the predicate
      if (edge_illegal<kFixedPos>(P, q, lc)) claim_edge_with(P, e, w, sc);
    }
    sync();
  }
  int flips = 0;
  const int lane = threadIdx.x & 31;
  WarpBuf wb{warp_buf(0), 0};
  for (int base = t0 - lane; base < n; base += nt) {
    const int i = base + lane;
    int mine[4];
    int k = 0;
    if (i < n) {
      const int e = ld_i(in + i);
      // Everything a winner needs is loaded together with its claim test: a
      // winner shares no face with another winner, so no flip of this round
      // writes its records, and only its own flip can move vhe[a] off 2e
      // or vhe[b] off 2e+1.
      const unsigned c = (unsigned)ld_i(reinterpret_cast<const int*>(P.cand) + e);
      const int2 f = __ldcg(P.efa + e);
      const int4 q = ld_ev(P, e);
      const int4 w = ld_en(P, e);
      if (c == sc) {
        const unsigned long long key = ((unsigned long long)sc << 32) | (unsigned)(~mix32((unsigned)e ^ sc));
        const unsigned long long ka = __ldcg(P.claim + f.x), kb = __ldcg(P.claim + f.y);
        const int vha = bad_v(P, q.x) ? -1 : ld_i(P.vhe + q.x);
        const int vhb = bad_v(P, q.y) ? -1 : ld_i(P.vhe + q.y);
        if (ka == key && kb == key) {
          if (flip_edge_with(P, e, q, w, vha, vhb)) ++flips;
          const int wing[4] = {w.x >> 1, w.y >> 1, w.z >> 1, w.w >> 1};
          // the four queue marks issued together, their answers used after
          unsigned was[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) was[j] = atomicMax(P.qmark + wing[j], sq);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (was[j] < sq) mine[k++] = wing[j];
        } else if (enqueue_once(P, e, sq)) {
          mine[k++] = e;
        }
      }
    }
    if (__any_sync(kFull, k > 0)) wb_push(wb, mine, k, out, out_count, P.E, P.st);
  }
  wb_flush(wb, out, out_count, P.E, P.st);
  return flips;
}

// Rounds with at most this many queued edges run inside one block (block
// barriers instead of grid barriers); the rest of the grid waits.  No more than the
// block has threads: a second pass over the list waits for the loads of the first
// (20,000 points advected: 1600 edges in one block 18 us, over the grid with two grid
// barriers 8; the step's launch 54 -> 43 us; limits of 32 to 384 the same within 2 us,
// 512 and above 54).
static_assert(kTailItems == kThreads, "an edge per thread");
// Default repair sub-steps per kinetic step (phase_substeps).  Off: on the
// uniform random-walk benchmarks (1M points, sigma = 0.1 x spacing; 512 meshes,
// 8.5M points) 4 and 8 sub-steps leave 25% and 4% of the sent-back vertices
// to removal, but each sub-step costs about as much as the removal and
// reinsertion rounds it saves (latency-bound star walks and flip rounds), so
// the step time does not improve.
constexpr int kSubsteps = 0;

// ---------------------------------------------------------------------------
// Lawson flip rounds starting from work-list `src`.  A round is two phases:
//   A  every queued edge that is still non-Delaunay claims its two faces with
//      a hashed priority (atomicMax on the face's smallest half-edge);
//   B  an edge that holds both claims flips and queues its four wing edges;
//      other candidates queue themselves again.
// Winners share no face, so their writes never overlap; the candidate with the
// highest priority always wins both faces, so every round flips at least once.
// If pre_sc != 0 the first round's phase A was done by the classification.
// With kLast (the launch's final phase) the grid does not wait for a
// single-block tail: the other blocks return at once and block 0 returns
// when the tail is done; only block 0's `stamp` is then current.
template <bool kFixedPos, bool kLast = false>
__device__ void phase_lawson(cg::grid_group& g, const KParams& P, int src, unsigned& stamp,
                             LocalCounters& lc, unsigned pre_sc) {
  const int stride = gridDim.x * blockDim.x;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  int flips = 0;
  for (int round = 0;; ++round) {
    const int n = ld_i(&P.st->wl_count[src]);
    if (n == 0) break;
    if (round >= P.max_rounds) {
      if (gtid == 0) set_error(P, MCL_ERR_NO_CONVERGENCE);
      break;
    }
    if (n <= P.tail_items) {
      // tail: block 0 finishes every remaining round on its own
      if (blockIdx.x == 0) {
        int s2 = src;
        unsigned st2 = stamp;
        for (int r2 = round; r2 < P.max_rounds; ++r2) {
          const int m = ld_i(&P.st->wl_count[s2]);
          if (m == 0) break;
          const int d2 = s2 ^ 1;
          // the first round's phase A may have been done by the classification
          // (then wl_count[d2] is still zero)
          const bool pre = r2 == 0 && pre_sc;
          const unsigned sc = pre ? pre_sc : st2++;
          const unsigned sq = st2++;
          if (threadIdx.x == 0) {
            if (!pre) P.st->wl_count[d2] = 0;
            P.st->c[C_LAWSON_ROUNDS] += 1;
          }
          __syncthreads();
          flips += lawson_round<kFixedPos>(P, s2 ? P.wl1 : P.wl0, m, d2 ? P.wl1 : P.wl0, &P.st->wl_count[d2], sc, sq,
                                           !pre, threadIdx.x, blockDim.x, lc, [] { __syncthreads(); });
          __syncthreads();
          timeline(P, 2 + (r2 < 40 ? r2 : 40));
          s2 = d2;
        }
        if (kLast) stamp = st2;
        else if (threadIdx.x == 0) P.st->tail_stamp = st2;
      }
      if (!kLast) {
        g.sync();
        stamp = (unsigned)ld_i(reinterpret_cast<const int*>(&P.st->tail_stamp));
      }
      break;
    }
    const int dst = src ^ 1;
    const int* in = src ? P.wl1 : P.wl0;
    int* out = dst ? P.wl1 : P.wl0;
    unsigned sc;
    bool phase_a = true;
    if (round == 0 && pre_sc) {
      sc = pre_sc;  // wl_count[dst] is still zero from the end of the last launch or phase
      phase_a = false;
      if (gtid == 0) P.st->c[C_LAWSON_ROUNDS] += 1;
    } else {
      sc = stamp++;
      if (gtid == 0) {
        P.st->wl_count[dst] = 0;
        P.st->c[C_LAWSON_ROUNDS] += 1;
      }
    }
    const unsigned sq = stamp++;
    flips += lawson_round<kFixedPos>(P, in, n, out, &P.st->wl_count[dst], sc, sq, phase_a, spread_tid(), stride, lc,
                                     [&] { g.sync(); });
    g.sync();
    timeline(P, 2 + (round < 40 ? round : 40));
    src = dst;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) flips += __shfl_down_sync(kFull, flips, o);
  if ((threadIdx.x & 31) == 0 && flips) atomicAdd(&P.st->c[C_LAWSON_FLIPS], (unsigned long long)flips);
}


// ---------------------------------------------------------------------------
// Repair (1): revert vertices of non-positive faces until all faces are positive.
__device__ __forceinline__ bool marked(const KParams& P, int v, unsigned fs) {
  return (unsigned)ld_i(P.vmark + v) == fs;
}

__device__ __forceinline__ float2 qpos(const KParams& P, int v, unsigned fs) {
  return marked(P, v, fs) ? P.pos_old[v] : ldpos(P, v);
}

// The list of the vertices the next fixpoint pass checks (their stars):
// pass p writes list p & 1 (vl0 / vl1) with count fix_list[p % 3].
__device__ __forceinline__ void list_for_next_pass(const KParams& P, int v, int pass) {
  push_coalesced(P, (pass & 1) ? P.vl1 : P.vl0, &P.st->fix_list[pass % 3], P.V, v);
}

// Where a fixpoint pass's marks go: appended at once from divergent code
// (MarkNow), or kept by the thread (at most two per work item) for one
// warp-wide buffered append afterwards (MarkLater).  A fresh vertex joins the
// list of every vertex sent back (`hard`) and the next pass's list; a vertex
// listed again joins the next pass's list.
struct MarkNow {
  const KParams& P;
  int pass;
  __device__ void fresh_vertex(int v) const {
    push_coalesced(P, P.hard, &P.st->fix_all, P.E, v);
    list_for_next_pass(P, v, pass);
  }
  __device__ void relist(int v) const { list_for_next_pass(P, v, pass); }
};
struct MarkLater {
  int nv[2], rl[2];
  int kn = 0, kr = 0;
  __device__ void fresh_vertex(int v) { nv[kn++ & 1] = v; }
  __device__ void relist(int v) { rl[kr++ & 1] = v; }
};

// A newly marked vertex records the pass that marked it in vloc (free until
// the insertion rounds) and goes to the sink.
template <typename Sink>
__device__ void mark_vertex(const KParams& P, int v, int& fresh, unsigned fs, int pass, Sink& sink) {
  if (!marked(P, v, fs) && (unsigned)atomicExch(P.vmark + v, (int)fs) != fs) {
    __stcg(P.vloc + v, pass);
    sink.fresh_vertex(v);
    ++fresh;
  }
}

// A non-positive face sends back one vertex per pass: the unmarked free vertex
// that moved farthest (ties: smallest id).  A face whose vertices are all back
// at their old positions is positive (the mesh was valid there), so every pass
// that still sees a bad face marks a vertex and the fixpoint ends.  Sending
// back fewer vertices means fewer removals and reinsertions; the result does
// not depend on the choice (every sent-back vertex is reinserted at its
// target).
// A bad face whose free vertices all turned out marked (by other faces of the
// same pass, after its orientation was read) is checked again next pass
// through the star of one of them.
template <typename Sink>
__device__ void mark_face(const KParams& P, int a, int b, int c, int& fresh, unsigned fs, int pass, Sink& sink) {
  const int t[3] = {a, b, c};
  int pick = -1, any = -1;
  float best = -1.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int v = t[k];
    if (P.vfix[v]) continue;
    if (marked(P, v, fs)) {
      any = v;
      continue;
    }
    const float2 pn = ldpos(P, v), po = P.pos_old[v];
    const float dx = __fsub_rn(pn.x, po.x), dy = __fsub_rn(pn.y, po.y);
    const float m2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
    if (m2 > best || (m2 == best && v < pick)) { best = m2; pick = v; }
  }
  if (pick >= 0) {
    mark_vertex(P, pick, fresh, fs, pass, sink);
  } else if (any >= 0) {
    // vloc of a marked vertex holds a pass of this launch: list it once per pass
    if (atomicExch(P.vloc + any, pass) != pass) sink.relist(any);
    ++fresh;
  }
}

// Returns MCL_OK, an error, or kSentBackMany once more than `most` vertices have been
// marked (listed again ones counted too).
constexpr int kSentBackMany = -1;
__device__ int phase_fixpoint(cg::grid_group& g, const KParams& P, LocalCounters& lc, unsigned fs, long long most) {
  const int stride = gridDim.x * blockDim.x;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  long long all = 0;  // of the passes so far, the same in every thread (fix_all moves on)
  for (int pass = 0; pass < 256; ++pass) {
    // counters are triple-buffered: slot (pass+1)%3 was last read two barriers ago
    const int slot = pass % 3;
    if (gtid == 0) {
      P.st->fix_new[(pass + 1) % 3] = 0;
      P.st->fix_bad[(pass + 1) % 3] = 0;
      P.st->fix_list[(pass + 1) % 3] = 0;
      P.st->c[C_FIX_PASSES] += 1;
    }
    int fresh = 0, bad = 0;
    if (pass == 0) {
      // every face the classification found non-positive, once per edge
      // side (its edges are on work-list 1)
      // (most warps mark on most iterations: the marks go through the
      // warp's append buffers, idle after the classification)
      const int nb = ld_i(&P.st->wl_count[1]);
      const int lane = threadIdx.x & 31;
      WarpBuf whard{warp_buf(0), 0}, wnext{warp_buf(1), 0};
      int* nlist = (pass & 1) ? P.vl1 : P.vl0;
      int* ncount = &P.st->fix_list[pass % 3];
      for (int base = spread_tid() - lane; base < nb; base += stride) {
        const int ii = base + lane;
        MarkLater ml;
        if (ii < nb) {
          const int e = ld_i(P.wl1 + ii);
          const int4 q = ld_ev(P, e);
          if (q.x >= 0 && (bad_v(P, q.x) || bad_v(P, q.y) || q.z >= P.V || q.w >= P.V)) {
            flag_error(P, MCL_ERR_DEGENERATE_INPUT);
          } else if (q.x >= 0) {
            const float2 a = qpos(P, q.x, fs), b = qpos(P, q.y, fs);
            if (q.z >= 0 && orient_v(P, a, b, qpos(P, q.z, fs), lc) <= 0) {
              ++bad;
              mark_face(P, q.x, q.y, q.z, fresh, fs, pass, ml);
            }
            if (q.w >= 0 && orient_v(P, b, a, qpos(P, q.w, fs), lc) <= 0) {
              ++bad;
              mark_face(P, q.y, q.x, q.w, fresh, fs, pass, ml);
            }
          }
        }
        if (__any_sync(kFull, ml.kn > 0)) {
          wb_push(whard, ml.nv, ml.kn, P.hard, &P.st->fix_all, P.E, P.st);
          wb_push(wnext, ml.nv, ml.kn, nlist, ncount, P.V, P.st);
        }
        if (__any_sync(kFull, ml.kr > 0)) wb_push(wnext, ml.rl, ml.kr, nlist, ncount, P.V, P.st);
      }
      wb_flush(whard, P.hard, &P.st->fix_all, P.E, P.st);
      wb_flush(wnext, nlist, ncount, P.V, P.st);
    } else {
      // only a face with a vertex sent back (or listed again) in the last pass
      // can have changed sign: the stars of the last pass's list
      const int nl = ld_i(&P.st->fix_list[(pass - 1) % 3]);
      const int* lst = ((pass - 1) & 1) ? P.vl1 : P.vl0;
      for (int ii = spread_tid(); ii < nl; ii += stride) {
        const int v = ld_i(lst + ii);
        const float2 pv = qpos(P, v, fs);
        const bool ok = for_spokes(P, v, [&](int h) {
          const int d = he_origin(P, h ^ 1), a = he_apex(P, h);
          if (bad_v(P, d) || a < 0 || bad_v(P, a)) return;  // hull side: no face
          if (orient_v(P, pv, qpos(P, d, fs), qpos(P, a, fs), lc) <= 0) {
            ++bad;
            MarkNow now{P, pass};
            mark_face(P, v, d, a, fresh, fs, pass, now);
          }
        });
        if (!ok) flag_error(P, MCL_ERR_DEGENERATE_INPUT);
      }
    }
    warp_add(&P.st->fix_new[slot], fresh);
    warp_add(&P.st->fix_bad[slot], bad);
    g.sync();
    if (pass < 16) timeline_remove(P, 48 + pass);
    const int nfresh = ld_i(&P.st->fix_new[slot]);
    const int nbad = ld_i(&P.st->fix_bad[slot]);
    if (nfresh == 0) return nbad ? MCL_ERR_DEGENERATE_INPUT : MCL_OK;
    all += nfresh;
    if (all > most) return kSentBackMany;
  }
  return MCL_ERR_NO_CONVERGENCE;
}

// ---------------------------------------------------------------------------
// Removal by ear clipping: retriangulate the star polygon of v (its link cycle,
// v left out) with exact orientation tests.  Used when no spoke flip is valid,
// which happens with exactly collinear neighbours (points clamped onto the
// same line of the box, lattices).  A simple polygon always has an ear whose
// closed triangle holds no other polygon vertex, so this always completes.
// The k spoke edges become k-3 diagonals plus the 3 free edges of v.
constexpr int kEarMax = 128;
// Loads per group issued before any of their values is stored: a loop that
// stores each loaded value (to local or shared memory) before the next load
// waits for every load in turn.
constexpr int kGather = 8;

// The star polygon under ear clipping: cyclic links and corner positions.
// Any star up to kEarMax corners: local arrays.
struct LocalPoly {
  int nx_[kEarMax], pv_[kEarMax];
  float2 q_[kEarMax];
  __device__ __forceinline__ int nx(int j) const { return nx_[j]; }
  __device__ __forceinline__ int pv(int j) const { return pv_[j]; }
  __device__ __forceinline__ void set_nx(int j, int x) { nx_[j] = x; }
  __device__ __forceinline__ void set_pv(int j, int x) { pv_[j] = x; }
  __device__ __forceinline__ float2 q(int j) const { return q_[j]; }
  __device__ __forceinline__ void set_q(int j, float2 x) { q_[j] = x; }
};

// Stars of up to kSmallStar corners: links packed four bits each in
// registers and positions in this thread's slots of the classification's
// shared staging array (idle during repair), which the ear search reads
// O(k^2) times.
constexpr int kSmallStar = 16;
struct SmallPoly {
  unsigned long long nx_ = 0, pv_ = 0;
  __device__ __forceinline__ static float2* slot(int j) {
    return reinterpret_cast<float2*>(ev_slot((j >> 3) & 1, (j >> 1) & 3)) + (j & 1);
  }
  __device__ __forceinline__ int nx(int j) const { return (int)((nx_ >> (4 * j)) & 15u); }
  __device__ __forceinline__ int pv(int j) const { return (int)((pv_ >> (4 * j)) & 15u); }
  __device__ __forceinline__ void set_nx(int j, int x) {
    nx_ = (nx_ & ~(15ull << (4 * j))) | ((unsigned long long)x << (4 * j));
  }
  __device__ __forceinline__ void set_pv(int j, int x) {
    pv_ = (pv_ & ~(15ull << (4 * j))) | ((unsigned long long)x << (4 * j));
  }
  __device__ __forceinline__ float2 q(int j) const { return *slot(j); }
  __device__ __forceinline__ void set_q(int j, float2 x) { *slot(j) = x; }
};

// Clip the star polygon of v given its k spokes sp (counter-clockwise), the
// link half-edges lk (lk[i] = next(sp[i]), the side of face i opposite v),
// their origins w and, in poly, their positions; pv is v's position, at which
// its star is valid; bnd is scratch of size k.
//
// Ears by a constant-time test while v stays strictly inside the kernel of the
// remaining polygon (checked at the start: every face of the star positive):
// then the corners are in strictly increasing angle around v, and a convex
// corner b between a and c whose diagonal a -> c has v strictly on its left
// spans an angle below 180 degrees from v; the cone of that angle is convex,
// holds the triangle abc and no other corner, so abc is an ear, and the new
// side a -> c keeps v strictly inside the kernel.  Only when no corner passes
// does the general test run (every other corner checked against the
// triangle, O(k) per candidate); an ear it clips whose diagonal does not have
// v strictly on its left ends the constant-time tests for this star.
template <typename Poly>
__device__ int clip_star(const KParams& P, int v, float2 pv, LocalCounters& lc, unsigned mk, int k, const int* sp,
                         const int* lk, const int* w, Poly& poly, int* bnd) {
  if (k < 3) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
  const int mbase = reserve_marks(P, mk, 2 * k - 3);  // its latency overlaps the clipping
  for (int j = 0; j < k; ++j) {
    poly.set_nx(j, j + 1 == k ? 0 : j + 1);
    poly.set_pv(j, j == 0 ? k - 1 : j - 1);
    bnd[j] = lk[j];
  }
  int remaining = k, j = 0, used = 3;
  // v strictly inside the kernel of the remaining polygon (checked: every
  // side w_i -> w_i+1 has v strictly on its left)
  bool kernel = true;
  for (int i = 0; i < k && kernel; ++i) kernel = orient_v(P, poly.q(i), poly.q(poly.nx(i)), pv, lc) > 0;
  while (remaining > 3) {
    bool found = false;
    if (kernel) {
      for (int t = 0; t < remaining && !found; ++t) {
        const int a = poly.pv(j), b = j, c = poly.nx(j);
        const float2 qa = poly.q(a), qb = poly.q(b), qc = poly.q(c);
        found = orient_v(P, qa, qc, pv, lc) > 0 && orient_v(P, qa, qb, qc, lc) > 0;
        if (!found) j = poly.nx(j);
      }
    }
    for (int t = 0; t < remaining && !found; ++t) {
      const int a = poly.pv(j), b = j, c = poly.nx(j);
      const float2 qa = poly.q(a), qb = poly.q(b), qc = poly.q(c);
      if (orient_v(P, qa, qb, qc, lc) > 0) {
        bool empty = true;
        for (int m = poly.nx(c); m != a && empty; m = poly.nx(m)) {
          const float2 qm = poly.q(m);
          if (orient_v(P, qa, qb, qm, lc) >= 0 && orient_v(P, qb, qc, qm, lc) >= 0 &&
              orient_v(P, qc, qa, qm, lc) >= 0)
            empty = false;
        }
        found = empty;
        if (found && kernel && orient_v(P, qa, qc, pv, lc) <= 0) kernel = false;
      }
      if (!found) j = poly.nx(j);
    }
    if (!found) return MCL_ERR_NO_CONVERGENCE | (__LINE__ << 8);
    const int a = poly.pv(j), b = j, c = poly.nx(j);
    const int g = sp[used++] >> 1;
    const int d0 = 2 * g, d1 = 2 * g + 1;  // d0: w_c -> w_a inside the ear, d1: w_a -> w_c outside
    __stcg(P.ev + g, make_int4(w[c], w[a], w[b], -1));
    __stcg(P.en + g, make_int4(bnd[a], bnd[b], -1, -1));
    he_set_face(P, bnd[a], w[c], bnd[b], d0);
    he_set_face(P, bnd[b], w[a], d0, bnd[a]);
    mark_edge(P, g, mk);
    bnd[a] = d1;
    poly.set_nx(a, c);
    poly.set_pv(c, a);
    --remaining;
    j = c;
  }
  {
    const int a = j, b = poly.nx(a), c = poly.nx(b);
    he_set_face(P, bnd[a], w[c], bnd[b], bnd[c]);
    he_set_face(P, bnd[b], w[a], bnd[c], bnd[a]);
    he_set_face(P, bnd[c], w[b], bnd[a], bnd[b]);
    __stcg(P.vhint + v, bnd[a]);
  }
  for (int i0 = 0; i0 < k; i0 += kGather) {
    // the corners' anchors kGather at a time, loaded before any is rewritten
    // (the corners are distinct, so no store of a group aliases its loads)
    int vh[kGather];
#pragma unroll
    for (int u = 0; u < kGather; ++u) vh[u] = i0 + u < k ? ld_i(P.vhe + w[i0 + u]) : -1;
#pragma unroll
    for (int u = 0; u < kGather; ++u) {
      const int i = i0 + u;
      if (i >= k) continue;
      if (vh[u] == (sp[i] ^ 1)) __stcg(P.vhe + w[i], lk[i]);
      mark_edge(P, lk[i] >> 1, mk);  // the hole's sides face new triangles
    }
  }
  if (mbase >= 0) {
    // the list entries: the sides and the diagonals (the spoke slots sp[3..k)
    // were reused for them); the slots were reserved at the start
    for (int t = 0; t < 2 * k - 3; ++t) append_mark(P, mbase, t, 2 * k - 3, t < k ? lk[t] >> 1 : sp[t - k + 3] >> 1);
  }
  for (int r = 0; r < 3; ++r) {
    const int e = sp[r] >> 1;
    __stcg(P.vfree + 3 * v + r, e);
    __stcg(P.ev + e, make_int4(-1, -1, -1, -1));
    __stcg(P.en + e, make_int4(-1, -1, -1, -1));
  }
  // the neighbour that later point location starts from: the nearest that is
  // not a bounding corner (a corner's half-edges run along the hull, far from
  // v; so do the edges between consecutive hull points)
  int anchor = w[0];
  {
    const float2 p0 = pv;
    float best = INFINITY;
    for (int i0 = 0; i0 < k; i0 += kGather) {
      unsigned char fx[kGather];
#pragma unroll
      for (int u = 0; u < kGather; ++u) fx[u] = i0 + u < k ? P.vfix[w[i0 + u]] : 1;
#pragma unroll
      for (int u = 0; u < kGather; ++u) {
        if (fx[u]) continue;
        const int i = i0 + u;
        const float2 qi = poly.q(i);
        const float dx = __fsub_rn(qi.x, p0.x), dy = __fsub_rn(qi.y, p0.y);
        const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
        if (d2 < best) { best = d2; anchor = w[i]; }
      }
    }
  }
  __stcg(P.vaux + v, anchor);
  __stcg(P.vhe + v, -1);
  return MCL_OK;
}

__device__ int remove_vertex_ears(const KParams& P, int v, LocalCounters& lc, unsigned mk) {
  int sp[kEarMax], lk[kEarMax], w[kEarMax], bnd[kEarMax];
  LocalPoly poly;
  const int s0 = ld_i(P.vhe + v);
  if (bad_h(P, s0)) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
  int k = 0, h = s0;
  do {
    if (k >= kEarMax) return MCL_ERR_CAPACITY | (__LINE__ << 8);
    sp[k] = h;
    lk[k] = he_next(P, h);
    if (bad_h(P, lk[k])) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
    w[k] = he_origin(P, lk[k]);
    if (bad_v(P, w[k])) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
    poly.set_q(k, ldpos(P, w[k]));
    ++k;
    h = he_prev(P, h) ^ 1;
    if (bad_h(P, h)) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
  } while (h != s0);
  return clip_star(P, v, ldpos(P, v), lc, mk, k, sp, lk, w, poly, bnd);
}

// A star walked once per removal round and kept by its thread across the
// round's barriers (claim, verify, remove): the thread handling list entry i
// handles the same entry in all three sub-phases, and a round's winners own
// every face of their stars, so nothing else writes them meanwhile.
constexpr int kStarCache = 32;
struct StarCache {
  int v;                 // cached vertex, -1: none
  int k;                 // its spokes; 0 when more than kStarCache
  int sp[kStarCache];    // spokes, counter-clockwise
  int lk[kStarCache];    // next(sp[i])
  int fm[kStarCache];    // smallest half-edge of face i (its claim slot)
};

// Walk v's star once (one record load per spoke), claiming each face with key.
__device__ bool claim_star(const KParams& P, int v, unsigned long long key, StarCache& sc) {
  sc.v = v;
  sc.k = 0;
  const int s0 = ld_i(P.vhe + v);
  if (bad_h(P, s0)) return false;
  int h = s0, k = 0;
  do {
    const int4 r = ld_en(P, h >> 1);
    const int nxt = (h & 1) ? r.z : r.x, prv = (h & 1) ? r.w : r.y;
    if (bad_h(P, nxt) || bad_h(P, prv)) return false;
    const int f = min(h, min(nxt, prv));
    atomicMax(P.claim + f, key);
    if (k < kStarCache) {
      sc.sp[k] = h;
      sc.lk[k] = nxt;
      sc.fm[k] = f;
    }
    ++k;
    h = prv ^ 1;
  } while (h != s0 && k < 1024);
  if (h != s0) return false;
  sc.k = k <= kStarCache ? k : 0;
  return true;
}

// The positions of corners w[0..k) into poly, kGather loads in flight at a time.
template <typename Poly>
__device__ __forceinline__ void gather_corners(const KParams& P, int k, const int* w, Poly& poly) {
  for (int i0 = 0; i0 < k; i0 += kGather) {
    float2 t[kGather];
#pragma unroll
    for (int u = 0; u < kGather; ++u) t[u] = i0 + u < k ? ldpos(P, w[i0 + u]) : make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < kGather; ++u)
      if (i0 + u < k) poly.set_q(i0 + u, t[u]);
  }
}

// Removal of v from its cached star (sc.k spokes): origins and positions of
// the link loaded together, then the ear clipping.
__device__ int remove_cached(const KParams& P, int v, const StarCache& sc, LocalCounters& lc, unsigned mk) {
  const int k = sc.k;
  int w[kStarCache], bnd[kStarCache];
  // link origins, then their positions, kGather loads in flight at a time (a
  // loop that stores each loaded value before the next load waits for every
  // load in turn)
  for (int i0 = 0; i0 < k; i0 += kGather) {
    int t[kGather];
#pragma unroll
    for (int u = 0; u < kGather; ++u) t[u] = i0 + u < k ? he_origin(P, sc.lk[i0 + u]) : 0;
#pragma unroll
    for (int u = 0; u < kGather; ++u)
      if (i0 + u < k) w[i0 + u] = t[u];
  }
  for (int i = 0; i < k; ++i)
    if (bad_v(P, w[i])) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
  const float2 pv = ldpos(P, v);
  if (k <= kSmallStar) {
    SmallPoly poly;
    gather_corners(P, k, w, poly);
    return clip_star(P, v, pv, lc, mk, k, sc.sp, sc.lk, w, poly, bnd);
  }
  LocalPoly poly;
  gather_corners(P, k, w, poly);
  return clip_star(P, v, pv, lc, mk, k, sc.sp, sc.lk, w, poly, bnd);
}

// ---------------------------------------------------------------------------
// Repair (2): removal of a vertex from a valid triangulation: ear clipping of
// its star polygon, or, for stars above kEarMax spokes, flipping its spokes
// until it has degree 3, then merging its three faces.  Runs in one thread;
// the caller owns every face of the vertex's star.
__device__ int remove_vertex(const KParams& P, int v, LocalCounters& lc, int& flips, unsigned mk) {
  {
    // Ear clipping first: one walk around the star, then local work on the
    // loaded polygon (the spoke flips below walk the star again after every
    // flip, a chain of dependent loads per flip).  Stars of more than
    // kEarMax spokes take the flips.
    const int rc = remove_vertex_ears(P, v, lc, mk);
    if ((rc & 0xff) != MCL_ERR_CAPACITY) {
      ++flips;  // counted as one repair operation
      return rc;
    }
  }
  const float2 pv = ldpos(P, v);
  int nearest = -1;  // the nearest neighbour that is not a bounding corner
  float nearest_d2 = INFINITY;
  for (int guard = 0; guard < 4096; ++guard) {
    const int s0 = ld_i(P.vhe + v);
    if (s0 < 0 || s0 >= 2 * P.E) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
    int deg = 0;
    int h = s0;
    int flipped = -1;
    do {
      ++deg;
      if (guard == 0) {
        const int w = he_origin(P, h ^ 1);
        if (!bad_v(P, w) && !P.vfix[w]) {
          const float2 q = ldpos(P, w);
          const float dx = __fsub_rn(q.x, pv.x), dy = __fsub_rn(q.y, pv.y);
          const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
          if (d2 < nearest_d2) { nearest_d2 = d2; nearest = w; }
        }
      }
      if (flipped < 0) {
        // flipping spoke h = v->w replaces faces (v,w,*) and (w,v,*) by (d,c,a), (c,d,b)
        const int e = h >> 1;
        const int4 q = ld_ev(P, e);
        if (bad_v(P, q.x) || bad_v(P, q.y) || q.z >= P.V || q.w >= P.V) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
        if (q.z >= 0 && q.w >= 0) {
          const float2 a = ldpos(P, q.x), b = ldpos(P, q.y), c = ldpos(P, q.z), d = ldpos(P, q.w);
          if (orient_v(P, d, c, a, lc) > 0 && orient_v(P, c, d, b, lc) > 0) flipped = e;
        }
      }
      h = he_prev(P, h) ^ 1;
      if (h < 0 || h >= 2 * P.E) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
    } while (h != s0 && deg < 1024);
    if (deg >= 1024) return MCL_ERR_CAPACITY | (__LINE__ << 8);
    if (deg == 3) break;
    if (deg < 3) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
    if (flipped < 0) {
      // no spoke flip is valid (exactly collinear neighbours): clip ears
      const int rc = remove_vertex_ears(P, v, lc, mk);
      if (rc != MCL_OK && atomicCAS(&P.st->dbg[0], 0, v + 1) == 0) {
        P.st->dbg[1] = deg;
        int hh = s0;
        for (int k = 0; k < deg && k < 64; ++k) {
          P.st->dbg[2 + k] = he_origin(P, hh ^ 1);
          hh = he_prev(P, hh) ^ 1;
        }
      }
      ++flips;  // counted as one repair operation
      return rc;
    }
    if (!flip_edge(P, flipped)) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
    if (mk) {
      P.st->mark_ovf = 1;  // spoke flips are marked, not appended: rebuild the list from the marks
      const int4 wg = ld_en(P, flipped);  // the flipped edge's four wings
      mark_edge(P, flipped, mk);
      mark_edge(P, wg.x >> 1, mk);
      mark_edge(P, wg.y >> 1, mk);
      mark_edge(P, wg.z >> 1, mk);
      mark_edge(P, wg.w >> 1, mk);
    }
    ++flips;
  }
  // merge the three faces (v,x,y), (v,y,z), (v,z,x) into (x,y,z)
  const int s0 = ld_i(P.vhe + v);
  const int s1 = he_prev(P, s0) ^ 1;
  const int s2 = he_prev(P, s1) ^ 1;
  if ((he_prev(P, s2) ^ 1) != s0) return MCL_ERR_NO_CONVERGENCE | (__LINE__ << 8);
  const int lxy = he_next(P, s0), lyz = he_next(P, s1), lzx = he_next(P, s2);
  if (bad_h(P, s1) || bad_h(P, s2) || bad_h(P, lxy) || bad_h(P, lyz) || bad_h(P, lzx)) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
  const int x = he_origin(P, lxy), y = he_origin(P, lyz), z = he_origin(P, lzx);
  if (bad_v(P, x) || bad_v(P, y) || bad_v(P, z)) return MCL_ERR_DEGENERATE_INPUT | (__LINE__ << 8);
  he_set_face(P, lxy, z, lyz, lzx);
  he_set_face(P, lyz, x, lzx, lxy);
  he_set_face(P, lzx, y, lxy, lyz);
  mark_edge(P, lxy >> 1, mk);
  mark_edge(P, lyz >> 1, mk);
  mark_edge(P, lzx >> 1, mk);
  if (mk) P.st->mark_ovf = 1;
  if (ld_i(P.vhe + x) == (s0 ^ 1)) __stcg(P.vhe + x, lxy);
  if (ld_i(P.vhe + y) == (s1 ^ 1)) __stcg(P.vhe + y, lyz);
  if (ld_i(P.vhe + z) == (s2 ^ 1)) __stcg(P.vhe + z, lzx);
  const int es[3] = {s0 >> 1, s1 >> 1, s2 >> 1};
  for (int k = 0; k < 3; ++k) {
    P.vfree[3 * v + k] = es[k];
    __stcg(P.ev + es[k], make_int4(-1, -1, -1, -1));
    __stcg(P.en + es[k], make_int4(-1, -1, -1, -1));
  }
  P.vhint[v] = lxy;
  // the neighbour that later point location starts from: the nearest of the
  // star it had when its removal began that is not a bounding corner (the
  // last three can be far: consecutive points on the hull)
  P.vaux[v] = nearest >= 0 ? nearest : (!P.vfix[x] ? x : (!P.vfix[y] ? y : z));
  __stcg(P.vhe + v, -1);
  return MCL_OK;
}

__device__ bool phase_remove(cg::grid_group& g, const KParams& P, unsigned& stamp, LocalCounters& lc, unsigned mk) {
  const int stride = gridDim.x * blockDim.x;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, nwarps = stride >> 5, wid = spread_tid() >> 5;
  int src = 0;
  StarCache sc;
  for (int round = 0;; ++round) {
    const int n = ld_i(&P.st->vl_count[src]);
    if (n == 0) return true;
    if (round >= P.max_rounds) {
      if (gtid == 0) set_error(P, MCL_ERR_NO_CONVERGENCE);
      return false;
    }
    const int dst = src ^ 1;
    const int* in = src ? P.vl1 : P.vl0;
    int* out = dst ? P.vl1 : P.vl0;
    const unsigned sk = stamp++;
    if (gtid == 0) {
      P.st->vl_count[dst] = 0;
      P.st->c[C_REMOVE_ROUNDS] += 1;
    }
    // A removal is a long divergent chain (star loads, ear search, writes), so
    // a warp runs its lanes' removals largely one after another: entries are
    // dealt in tiles of T lanes per warp (entry i: warp (i / T) mod warps,
    // lane i mod T), by default as few lanes as let one pass take the list.
    const int T = P.rm_tile > 0 ? min(P.rm_tile, 32) : max(1, min(32, (n + nwarps - 1) / nwarps));
    const int i0 = lane < T ? wid * T + lane : n, di = nwarps * T;
    // claim every face of the star (the thread keeps the last star it walked)
    sc.v = -1;
    for (int i = i0; i < n; i += di) {
      const int v = ld_i(in + i);
      const unsigned long long key = ((unsigned long long)sk << 32) | (unsigned)(~mix32((unsigned)v ^ sk));
      if (!claim_star(P, v, key, sc)) {
        sc.v = -1;
        set_error(P, MCL_ERR_DEGENERATE_INPUT);
      }
    }
    g.sync();
    if (round < 16) timeline_remove(P, 4 * round);
    for (int i = i0; i < n; i += di) {
      const int v = ld_i(in + i);
      const unsigned long long key = ((unsigned long long)sk << 32) | (unsigned)(~mix32((unsigned)v ^ sk));
      bool win = true, ok = true;
      if (sc.v == v && sc.k > 0) {
        // the claims kGather at a time, all loads of a group in flight together
        for (int j0 = 0; j0 < sc.k; j0 += kGather) {
          unsigned long long c[kGather];
#pragma unroll
          for (int u = 0; u < kGather; ++u) c[u] = j0 + u < sc.k ? __ldcg(P.claim + sc.fm[j0 + u]) : key;
#pragma unroll
          for (int u = 0; u < kGather; ++u) win &= c[u] == key;
        }
      } else {
        ok = for_spokes(P, v, [&](int h) {
          if (__ldcg(P.claim + face_min(P, h)) != key) win = false;
        });
      }
      P.vlocf[v] = (ok && win) ? 1 : 0;
      if (!ok) set_error(P, MCL_ERR_DEGENERATE_INPUT);
    }
    g.sync();
    if (round < 16) timeline_remove(P, 4 * round + 1);
    int removed = 0, flips = 0;
    unsigned long long slow = 0;  // the slowest removal of this thread: cycles << 16 | spokes
    WarpBuf wb{warp_buf(0), 0};
    for (int base = wid * T; base < n; base += di) {
      const int i = lane < T ? base + lane : n;
      int mine[1];
      int k = 0;
      if (i < n) {
        const int v = ld_i(in + i);
        if (__ldcg(P.vlocf + v) == 1) {
          int rc;
          const long long t0 = clock64();
          int deg = sc.k;
          if (sc.v == v && sc.k > 0) {
            rc = remove_cached(P, v, sc, lc, mk);
            ++flips;  // counted as one repair operation
          } else {
            rc = remove_vertex(P, v, lc, flips, mk);
            deg = 0;
            if (round < 16) atomicAdd(&P.st->rm_uncached[round], 1ull);
          }
          const unsigned long long dt = (unsigned long long)(clock64() - t0);
          slow = max(slow, (dt << 16) | (unsigned long long)(deg & 0xffff));
          if (rc != MCL_OK) flag_error_at(P, rc & 0xff, 100000 + (rc >> 8));
          else ++removed;
        } else if (ld_i(&P.st->status) == MCL_OK) {
          mine[k++] = v;
        }
      }
      wb_push(wb, mine, k, out, &P.st->vl_count[dst], P.V, P.st);
    }
    wb_flush(wb, out, &P.st->vl_count[dst], P.V, P.st);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) slow = max(slow, __shfl_down_sync(kFull, slow, o));
    if (round < 16 && lane == 0 && slow) atomicMax(&P.st->rm_slow[round], slow);
    warp_add(&P.st->c[C_REMOVED], removed);
    warp_add(&P.st->c[C_REMOVAL_FLIPS], flips);
    g.sync();
    if (round < 16) timeline_remove(P, 4 * round + 2);
    src = dst;
  }
}

// ---------------------------------------------------------------------------
// Point location: visibility walk with exact orientation tests from half-edge h.
// Returns a half-edge of the face containing p; *on is the half-edge p lies on
// (or -1).  Errors are returned as negative MCL codes.  With max_steps > 0 the
// walk stops after that many steps, returns -1 and leaves the face it reached
// in *resume (a parallel round then waits for the longest walk only that long).
// salt != 0: the edge tested first in each face is drawn from a hash of
// (salt, step) (a stochastic walk, which terminates on any triangulation);
// salt == 0: it rotates with the step (enough on a Delaunay triangulation).
__device__ int locate(const KParams& P, float2 p, int h, int* on, LocalCounters& lc, int max_steps = 0,
                      int* resume = nullptr, unsigned salt = 0) {
  *on = -1;
  for (int it = 0; it < P.walk_cap; ++it) {
    if (max_steps > 0 && it == max_steps) {
      *resume = h;
      return -1;
    }
    if (h < 0 || h >= 2 * P.E) return -MCL_ERR_DEGENERATE_INPUT;
    // the face's three corners and its other two half-edges from h's two
    // records (loaded together): origin(next(h)) = origin(twin(h)) and
    // origin(prev(h)) = apex(h)
    const int4 r = ld_ev(P, h >> 1), nn = ld_en(P, h >> 1);
    const bool odd = h & 1;
    const int hs[3] = {h, odd ? nn.z : nn.x, odd ? nn.w : nn.y};
    const int o[3] = {odd ? r.y : r.x, odd ? r.x : r.y, odd ? r.w : r.z};
    for (int k = 0; k < 3; ++k) {
      if (hs[k] < 0 || hs[k] >= 2 * P.E) return -MCL_ERR_DEGENERATE_INPUT;
      if (o[k] < 0 || o[k] >= P.V) return -MCL_ERR_DEGENERATE_INPUT;
    }
    const float2 q[3] = {ldpos(P, o[0]), ldpos(P, o[1]), ldpos(P, o[2])};
    int s[3] = {1, 1, 1};
    int cross = -1;
    const int start = salt ? (int)(mix32(salt + (unsigned)it * 0x9e3779b9u) % 3u) : it % 3;
    // Every edge with p on its far side is a valid step; an edge with a
    // bounding corner is taken only when no other is (stepping through a
    // corner's fan of long hull triangles can take hundreds of steps).
    bool corner_cross = false;
    for (int k = 0; k < 3; ++k) {
      const int i = (start + k) % 3;
      s[i] = orient_v(P, q[i], q[(i + 1) % 3], p, lc);
      if (s[i] < 0) {
        const bool corner = P.vfix[o[i]] || P.vfix[o[(i + 1) % 3]];
        if (cross < 0 || (corner_cross && !corner)) {
          cross = i;
          corner_cross = corner;
        }
        if (!corner) break;
      }
    }
    if (cross >= 0) {
      const int t = hs[cross] ^ 1;
      if (he_apex(P, t) < 0) return -MCL_ERR_DEGENERATE_INPUT;  // outside the bounding square
      h = t;
      continue;
    }
    int zeros = 0, zi = -1;
    for (int i = 0; i < 3; ++i)
      if (s[i] == 0) { ++zeros; zi = i; }
    if (zeros >= 2) return -MCL_ERR_DEGENERATE_INPUT;  // coincides with a vertex
    if (zeros == 1) {
      if (he_apex(P, hs[zi] ^ 1) < 0) return -MCL_ERR_DEGENERATE_INPUT;  // on the bounding square
      *on = hs[zi];
    }
    return h;
  }
  return -(MCL_ERR_NO_CONVERGENCE | (__LINE__ << 8));
}

// 1-to-3 split of the face of half-edge h0 by v with free edges f0, f1, f2.
__device__ void split13(const KParams& P, int v, int h0, const int* f) {
  const int h1 = he_next(P, h0), h2 = he_prev(P, h0);
  const int x0 = he_origin(P, h0), x1 = he_origin(P, h1), x2 = he_origin(P, h2);
  const int f0 = f[0], f1 = f[1], f2 = f[2];
  __stcg(P.ev + f0, make_int4(v, x0, x1, x2));
  __stcg(P.ev + f1, make_int4(v, x1, x2, x0));
  __stcg(P.ev + f2, make_int4(v, x2, x0, x1));
  __stcg(P.en + f0, make_int4(h0, 2 * f1 + 1, 2 * f2, h2));
  __stcg(P.en + f1, make_int4(h1, 2 * f2 + 1, 2 * f0, h0));
  __stcg(P.en + f2, make_int4(h2, 2 * f0 + 1, 2 * f1, h1));
  he_set_face(P, h0, v, 2 * f1 + 1, 2 * f0);
  he_set_face(P, h1, v, 2 * f2 + 1, 2 * f1);
  he_set_face(P, h2, v, 2 * f0 + 1, 2 * f2);
  __stcg(P.vhe + v, 2 * f0);
}

// 2-to-4 split of the edge of half-edge g (v lies on it) with free edges f0..f2.
__device__ void split24(const KParams& P, int v, int g, const int* f) {
  const int h0 = g, h1 = g ^ 1;
  const int n0 = he_next(P, h0), p0 = he_prev(P, h0);
  const int n1 = he_next(P, h1), p1 = he_prev(P, h1);
  const int a = he_origin(P, h0), b = he_origin(P, h1);
  const int c = he_apex(P, h0), d = he_apex(P, h1);
  const int f0 = f[0], f1 = f[1], f2 = f[2];
  // faces: (a,v,c) (v,b,c) (b,v,d) (v,a,d)
  he_set_origin(P, h1, v);
  he_set_face(P, h0, c, 2 * f1, p0);
  he_set_face(P, h1, d, n1, 2 * f2 + 1);
  he_set_face(P, p0, v, h0, 2 * f1);
  he_set_face(P, n0, v, 2 * f1 + 1, 2 * f0);
  he_set_face(P, p1, v, 2 * f0 + 1, 2 * f2);
  he_set_face(P, n1, v, 2 * f2 + 1, h1);
  __stcg(P.ev + f0, make_int4(v, b, c, d));
  __stcg(P.en + f0, make_int4(n0, 2 * f1 + 1, 2 * f2, p1));
  __stcg(P.ev + f1, make_int4(v, c, a, b));
  __stcg(P.en + f1, make_int4(p0, h0, 2 * f0, n0));
  __stcg(P.ev + f2, make_int4(v, d, b, a));
  __stcg(P.en + f2, make_int4(p1, 2 * f0 + 1, h1, n1));
  __stcg(P.vhe + v, 2 * f0);
  if (ld_i(P.vhe + b) == h1) __stcg(P.vhe + b, n0);
}

// Start of the point location of a pending vertex: the hole half-edge recorded
// at its removal when that edge is still live, else the neighbour recorded at
// removal (vaux) and, when that one was removed too, its own recorded
// neighbour, and so on: each hop stays about one spacing from the old
// position, so the walk stays short instead of starting at the bounding square.
__device__ __forceinline__ bool face_has_corner(const KParams& P, int h) {
  const int a = he_origin(P, h), b = he_origin(P, h ^ 1), c = he_apex(P, h);
  return (a >= 0 && P.vfix[a]) || (b >= 0 && P.vfix[b]) || (c >= 0 && P.vfix[c]);
}

// In later rounds of an insertion phase the hint is where the vertex's last
// walk ended (located, or paused): it is taken as it is, or a walk paused in a
// corner's fan would be sent back to its anchor every round and never arrive.
__device__ int insert_start(const KParams& P, int v, bool resume) {
  int h = __ldcg(P.vhint + v);
  const bool hint_ok = h >= 0 && h < 2 * P.E && he_origin(P, h) >= 0 && he_apex(P, h) >= 0;
  if (resume && hint_ok) return h;
  // the live anchor: the neighbour recorded at removal, or its own anchor if
  // that one was removed too
  int x = __ldcg(P.vaux + v), h0 = -1;
  for (int hop = 0; hop < 64 && x >= 0 && x < P.V; ++hop) {
    h0 = ld_i(P.vhe + x);
    if (h0 >= 0 && h0 < 2 * P.E) break;
    h0 = -1;
    x = __ldcg(P.vaux + x);
  }
  // a first start on a bounding corner's fan of long hull triangles makes the
  // walk step along the hull one triangle at a time: prefer a face with no
  // corner.  The hint's edge slot may have been freed by a later removal and
  // reused far away, so it is taken only when it is not farther from the
  // target than the anchor.
  if (hint_ok && !face_has_corner(P, h)) {
    if (h0 < 0) return h;
    const float2 t = ldpos(P, v), ph = ldpos(P, he_origin(P, h)), px = ldpos(P, x);
    const float dh = __fadd_rn(__fmul_rn(ph.x - t.x, ph.x - t.x), __fmul_rn(ph.y - t.y, ph.y - t.y));
    const float dx = __fadd_rn(__fmul_rn(px.x - t.x, px.x - t.x), __fmul_rn(px.y - t.y, px.y - t.y));
    if (dh <= dx) return h;
  }
  if (h0 >= 0) {
    int g = h0;
    for (int k = 0; k < 64; ++k) {
      if (he_apex(P, g) >= 0 && !face_has_corner(P, g)) return g;
      g = he_next(P, g ^ 1);  // next outgoing half-edge of x
      if (g < 0 || g >= 2 * P.E || g == h0) break;
    }
    return hint_ok ? h : h0;
  }
  if (hint_ok) return h;
  // half-edge 0 of the vertex's mesh is never freed: a side of its bounding square
  return P.vroot ? __ldg(P.vroot + v) : 0;
}

// Steps a point location may take in one insertion round before it waits for
// the next round (which starts where it stopped).
constexpr int kWalkSlice = 48;

// With mk != 0 (repair) the rounds only split: the edges each split touches
// are marked with mk for one Lawson pass after the last round (the walks of
// later rounds run on a valid, not yet Delaunay, triangulation; their edge
// order is randomised, so they cannot cycle).  With mk == 0 (the initial
// build) every round ends with Lawson over the edges it touched.
__device__ bool phase_insert(cg::grid_group& g, const KParams& P, unsigned& stamp,
                             LocalCounters& lc, unsigned mk = 0) {
  const int stride = gridDim.x * blockDim.x;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  int src = 0;
  for (int round = 0;; ++round) {
    const int n = ld_i(&P.st->vl_count[src]);
    if (n == 0) return true;
    if (round >= P.max_rounds) {
      if (gtid == 0) set_error(P, MCL_ERR_NO_CONVERGENCE);
      return false;
    }
    const int dst = src ^ 1;
    const int* in = src ? P.vl1 : P.vl0;
    int* out = dst ? P.vl1 : P.vl0;
    const unsigned sk = stamp++;
    const unsigned sq = stamp++;
    if (gtid == 0) {
      P.st->vl_count[dst] = 0;
      if (!mk) P.st->wl_count[0] = 0;  // with mk the list gathers the marks of every round
      P.st->c[C_INSERT_ROUNDS] += 1;
    }
    // locate and claim
    for (int i = spread_tid(); i < n; i += stride) {
      const int v = ld_i(in + i);
      int on = -1;
      int resume = -1;
      // a walk paused in the last round goes on from where it stopped; any
      // other start is the closer of the hint (the face located last round,
      // which can reach far along the hull) and the anchor
      const bool paused = round > 0 && __ldcg(P.vlocf + v) == 4;
      const int h = locate(P, ldpos(P, v), insert_start(P, v, paused), &on, lc, kWalkSlice, &resume,
                           mk ? mix32((unsigned)v ^ sk) | 1u : 0u);
      if (h == -1) {
        // not there yet: go on from here in the next round
        P.vloc[v] = resume;
        P.vlocf[v] = 4;
        continue;
      }
      if (h < 0) {
        flag_error_at(P, (-h) & 0xff, 200000 + ((-h) >> 8));
        P.vlocf[v] = -1;
        continue;
      }
      P.vloc[v] = on >= 0 ? on : h;
      P.vlocf[v] = on >= 0 ? 2 : 0;  // bit 1: on the edge of vloc, bit 0: winner
      const unsigned long long key = ((unsigned long long)sk << 32) | (unsigned)(~mix32((unsigned)v ^ sk));
      if (on >= 0) {
        atomicMax(P.claim + face_min(P, on), key);
        atomicMax(P.claim + face_min(P, on ^ 1), key);
      } else {
        atomicMax(P.claim + face_min(P, h), key);
      }
    }
    g.sync();
    timeline_insert(P, round, 0);
    for (int i = spread_tid(); i < n; i += stride) {
      const int v = ld_i(in + i);
      const int fl = __ldcg(P.vlocf + v);
      if (fl < 0) continue;
      const unsigned long long key = ((unsigned long long)sk << 32) | (unsigned)(~mix32((unsigned)v ^ sk));
      const int h = __ldcg(P.vloc + v);
      bool win = __ldcg(P.claim + face_min(P, h)) == key;
      if (fl & 2) win = win && __ldcg(P.claim + face_min(P, h ^ 1)) == key;
      if (win) P.vlocf[v] = fl | 1;
    }
    g.sync();
    timeline_insert(P, round, 1);
    int inserted = 0;
    WarpBuf wagain{warp_buf(1), 0};
    for (int base = spread_tid() - (int)(threadIdx.x & 31); base < n; base += stride) {
      const int i = base + (int)(threadIdx.x & 31);
      int mine[8];
      int k = 0;
      int again[1];
      int ka = 0;
      if (i < n) {
        const int v = ld_i(in + i);
        const int fl = __ldcg(P.vlocf + v);
        if (fl >= 0 && (fl & 1)) {
          const int f[3] = {__ldcg(P.vfree + 3 * v), __ldcg(P.vfree + 3 * v + 1), __ldcg(P.vfree + 3 * v + 2)};
          int link[4];
          int nl = 0;
          if ((unsigned)f[0] >= (unsigned)P.E || (unsigned)f[1] >= (unsigned)P.E || (unsigned)f[2] >= (unsigned)P.E ||
              bad_h(P, __ldcg(P.vloc + v))) {
            flag_error(P, MCL_ERR_DEGENERATE_INPUT);
          } else if (fl & 2) {
            const int gg = __ldcg(P.vloc + v);
            link[nl++] = he_prev(P, gg);
            link[nl++] = he_next(P, gg);
            link[nl++] = he_prev(P, gg ^ 1);
            link[nl++] = he_next(P, gg ^ 1);
            split24(P, v, gg, f);
          } else {
            const int h = __ldcg(P.vloc + v);
            link[nl++] = h;
            link[nl++] = he_next(P, h);
            link[nl++] = he_prev(P, h);
            split13(P, v, h, f);
          }
          ++inserted;
          for (int j = 0; j < nl; ++j)
            if (bad_h(P, link[j])) { link[j] = 0; flag_error(P, MCL_ERR_DEGENERATE_INPUT); }
          if (mk) {
            // on a triangulation that is not Delaunay the new spokes need not
            // be legal either: the split edge (now v's spoke to a) and f0..f2
            int edges[8];
            int cnt = 0;
            for (int j = 0; j < nl; ++j) edges[cnt++] = link[j] >> 1;
            for (int j = 0; j < 3; ++j) edges[cnt++] = f[j];
            if (fl & 2) edges[cnt++] = __ldcg(P.vloc + v) >> 1;
            const int mbase = reserve_marks(P, mk, cnt);
            for (int j = 0; j < cnt; ++j) {
              mark_edge(P, edges[j], mk);
              append_mark(P, mbase, j, cnt, edges[j]);
            }
          } else {
            for (int j = 0; j < nl; ++j)
              if (enqueue_once(P, link[j] >> 1, sq)) mine[k++] = link[j] >> 1;
            for (int j = 0; j < 3; ++j)
              if (enqueue_once(P, f[j], sq)) mine[k++] = f[j];
          }
        } else if (fl >= 0) {
          __stcg(P.vhint + v, __ldcg(P.vloc + v));
          again[ka++] = v;
        }
      }
      warp_push(mine, k, P.wl0, &P.st->wl_count[0], P.E, P.st);
      wb_push(wagain, again, ka, out, &P.st->vl_count[dst], P.V, P.st);
    }
    wb_flush(wagain, out, &P.st->vl_count[dst], P.V, P.st);
    (void)inserted;
    g.sync();
    timeline_insert(P, round, 2);
    if (!mk) {
      phase_lawson<false>(g, P, 0, stamp, lc, 0);
      g.sync();
    }
    timeline_insert(P, round, 3);
    src = dst;
  }
}

// ---------------------------------------------------------------------------
// End of a launch: publish this launch's counters and status for the host,
// add them to the running totals, and leave the working state clean for the
// next launch (so no reset launch or memset precedes the next step).
// The step counters c of a launch in the public record layout.
__device__ __forceinline__ void publish_counts(const unsigned long long (&c)[C_COUNT], int status, int site,
                                               mcl_step_stats* out) {
  out->inverted_faces = (int64_t)c[C_INVERTED];
  out->reverted_vertices = (int64_t)c[C_REVERTED];
  out->removed_vertices = (int64_t)c[C_REMOVED];
  out->lawson_flips = (int64_t)c[C_LAWSON_FLIPS];
  out->lawson_rounds = (int64_t)c[C_LAWSON_ROUNDS];
  out->removal_flips = (int64_t)c[C_REMOVAL_FLIPS];
  out->insert_rounds = (int64_t)c[C_INSERT_ROUNDS];
  out->incircle_tests = (int64_t)c[C_INCIRCLE];
  out->incircle_fp64 = (int64_t)c[C_INCIRCLE_FP64];
  out->incircle_exact = (int64_t)c[C_INCIRCLE_EXACT];
  out->orient_fp64 = (int64_t)c[C_ORIENT_FP64];
  out->orient_exact = (int64_t)c[C_ORIENT_EXACT];
  out->sos_decisions = (int64_t)c[C_SOS];
  out->status = status;
  out->error_site = site;
  out->failed_launches = status != MCL_OK ? 1 : 0;
  out->substep_vertices = (int64_t)c[C_SUBSTEP_DONE];
}

// By one warp, a counter per lane: a lone thread's reads and writes, each waiting for
// the last, and the copy of the record that followed closed a step with 6 us more.
__device__ void finish_launch(const KParams& P, unsigned stamp) {
  static_assert(C_COUNT <= 32, "a lane per counter");
  DevState* st = P.st;
  const int lane = threadIdx.x & 31;
  // L2-coherent reads: other blocks' atomics and stores are not in this SM's L1
  unsigned long long c = 0, tot = 0;
  if (lane < C_COUNT) {
    c = __ldcg(&st->c[lane]);
    tot = __ldcg(&st->tot[lane]);
  }
  const unsigned long long tm = __ldcg(&st->tsmax[lane & 3]);
  const int status = __ldcg(&st->status), site = __ldcg(&st->site), movers = __ldcg(&st->movers_now);
  const int tried = __ldcg(&st->star_tried), fails = __ldcg(&st->star_fails), hold = __ldcg(&st->star_hold);
  const unsigned long long calls = __ldcg(&st->calls), failed = __ldcg(&st->failed);
  if (lane < C_COUNT) {
    st->last[lane] = c;
    st->tot[lane] = tot + c;
    st->c[lane] = 0;
  }
  const bool repaired = __shfl_sync(kFull, c, C_INVERTED) != 0;
  if (lane < 4) {
    if (!repaired) st->ts[43 + lane] = tm;
    st->tsmax[lane] = 0;
  }
  if (P.stats_out) {  // host-mapped: no copy launch
    unsigned long long all[C_COUNT];
#pragma unroll
    for (int i = 0; i < C_COUNT; ++i) all[i] = __shfl_sync(kFull, c, i);
    if (lane == 0) publish_counts(all, status, site, P.stats_out);
  }
  if (lane != 0) return;
  st->calls = calls + 1;
  if (status != MCL_OK) st->failed = failed + 1;
  st->last_status = status;
  st->last_site = site;
  st->status = 0;
  st->site = 0;
  st->wl_count[0] = st->wl_count[1] = 0;
  st->vl_count[0] = st->vl_count[1] = 0;
  st->inverted = 0;
  st->hard_count = 0;
  for (int i = 0; i < 3; ++i) st->fix_new[i] = st->fix_bad[i] = st->fix_list[i] = 0;
  for (int i = 0; i < 3; ++i) st->star_n[i] = 0;
  st->star_ext = 0;
  st->star_made = 0;
  // Stars that could not be made (one wider than 128, more wide ones than rows) are left
  // out of the next steps, twice as many each time, 32 at most: such a mesh paid for them
  // and for removal on every step (one vertex of 150 neighbours among 1,000,000: 1650 us
  // by removal alone, 2310 with both).
  if (tried == kStarsMade) {
    st->star_hold = st->star_fails = 0;
  } else if (tried == kStarsFailed) {
    st->star_fails = min(fails + 1, 5);
    st->star_hold = 1 << min(fails + 1, 5);
  } else if (tried == kStarsHeld) {
    st->star_hold = hold - 1;
  }
  st->star_tried = 0;
  st->fix_all = 0;
  st->mark_ovf = 0;
  st->movers_last = movers;
  st->movers_now = 0;
  st->epoch = stamp;
}

// ---------------------------------------------------------------------------
// Repair (1b): bring sent-back vertices to their targets in sub-steps, so that
// most of them need no removal.  A Delaunay mesh whose vertex moves on a line
// meets a flip (an incircle event) before any face around the vertex
// degenerates, so moving part of the way, restoring the Delaunay property
// around the vertex and moving on passes the obstruction that sent it back.
// A sub-step moves every pending vertex toward its target (all the way, or
// 9/10 of the way to the first face of its star that would degenerate, times
// 2^-lvl after lvl send-backs in a row); sends back, pass by pass until every
// face is positive, each mover with a non-positive face in its star (lvl + 1);
// runs Lawson rounds over the stars of the movers that stayed; and keeps those
// not yet at their targets pending (lvl 0).  Vertices sent back more than
// kSubstepLevels times in a row, or still pending after P.substeps sub-steps,
// are left on vl0 for removal and reinsertion.  The mesh ends as the Delaunay triangulation of
// the targets either way; this path only saves removals.
//
// In: vl0 = pending vertices at valid positions (pos), targets in `target`,
// vlocf = 0 for each, the mesh Delaunay.  Out: vl0 = vertices left for
// removal (at their last valid positions), the mesh valid and Delaunay.
constexpr int kSubstepLevels = 5;

__device__ void phase_substeps(cg::grid_group& g, const KParams& P, unsigned& stamp, LocalCounters& lc) {
  const int stride = gridDim.x * blockDim.x;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int* const mv[2] = {P.vl2, P.vl2 + P.V};  // movers of a sub-step pass
  int* const rv = P.vl2 + 2 * P.V;          // movers sent back in the current pass
  int* const left = P.vl2 + 3 * P.V;        // past kSubstepLevels halvings
  int src = 0;
  int done = 0;
  for (int s = 0; s < P.substeps; ++s) {
    const int n = ld_i(&P.st->vl_count[src]);
    if (n == 0) break;
    const int dst = src ^ 1;
    const int* in = src ? P.vl1 : P.vl0;
    int* out = dst ? P.vl1 : P.vl0;
    const unsigned qs = stamp++;
    if (gtid == 0) {
      P.st->vl_count[dst] = 0;
      P.st->sub_count[0] = 0;
      P.st->sub_count[1] = 0;
      for (int k = 0; k < 3; ++k) P.st->sub_rev[k] = 0;
      if (s == 0) P.st->sub_count[2] = 0;
      P.st->wl_count[0] = 0;
      P.st->wl_count[1] = 0;
      P.st->c[C_SUBSTEPS] += 1;
    }
    g.sync();
    // (a) move each pending vertex toward its target: all the way when no
    // face of its star degenerates on the way, else 9/10 of the way to the
    // first face that would (the flip that clears it comes before); after
    // lvl consecutive send-backs, 2^-lvl of that
    for (int base = spread_tid() - lane; base < n; base += stride) {
      const int i = base + lane;
      int mine[1];
      int k = 0;
      if (i < n) {
        const int v = ld_i(in + i);
        const float2 p = ldpos(P, v), t = __ldcg(P.target + v);
        const int lvl = ld_i(P.vlocf + v);
        double fmax = 1.0;
        bool blocked = false;
        for_spokes(P, v, [&](int h) {
          const int d = he_origin(P, h ^ 1), a = he_apex(P, h);
          if (bad_v(P, d) || a < 0 || bad_v(P, a)) return;
          const float2 q = ldpos(P, d), r = ldpos(P, a);
          // orientation of (x, q, r) is affine in x: its value at p and at t
          const double o0 = ((double)q.x - p.x) * ((double)r.y - p.y) - ((double)q.y - p.y) * ((double)r.x - p.x);
          const double o1 = ((double)q.x - t.x) * ((double)r.y - t.y) - ((double)q.y - t.y) * ((double)r.x - t.x);
          if (o1 <= 0.0) {
            blocked = true;
            const double f = o0 > 0.0 ? o0 / (o0 - o1) : 0.0;
            fmax = f < fmax ? f : fmax;
          }
        });
        float2 c = t;
        if (blocked || lvl > 0) {
          const float f = (float)((blocked ? 0.9 * fmax : 1.0) * ldexp(1.0, -lvl));
          c.x = fadd(p.x, fmul(fsub(t.x, p.x), f));
          c.y = fadd(p.y, fmul(fsub(t.y, p.y), f));
        }
        __stcg(P.vprev + v, p);
        __stcg(P.pos + v, c);
        mine[k++] = v;
      }
      warp_push(mine, k, mv[0], &P.st->sub_count[0], P.V, P.st);
    }
    g.sync();
    // (b) send back, pass by pass, every mover with a non-positive face in its
    // star: every position is read (detect) before any is restored (apply)
    int cur = 0;
    for (int pass = 0;; ++pass) {
      if (pass == 64) {
        if (gtid == 0) set_error(P, MCL_ERR_NO_CONVERGENCE);
        return;
      }
      const int m = ld_i(&P.st->sub_count[cur]);
      const int nxt = cur ^ 1;
      const int slot = pass % 3;
      for (int base = spread_tid() - lane; base < m; base += stride) {
        const int i = base + lane;
        int stay[1], back[1], pend[1], gone[1];
        int ks = 0, kb = 0, kp = 0, kg = 0;
        if (i < m) {
          const int v = ld_i(mv[cur] + i);
          const float2 pv = ldpos(P, v);
          bool good = true;
          const bool ok = for_spokes(P, v, [&](int h) {
            if (!good) return;
            const int d = he_origin(P, h ^ 1), a = he_apex(P, h);
            if (bad_v(P, d) || a < 0 || bad_v(P, a)) {
              good = false;
              return;
            }
            if (orient_v(P, pv, ldpos(P, d), ldpos(P, a), lc) <= 0) good = false;
          });
          if (!ok) flag_error(P, MCL_ERR_DEGENERATE_INPUT);
          if (good) {
            stay[ks++] = v;
          } else {
            const int lvl = ld_i(P.vlocf + v) + 1;
            __stcg(P.vlocf + v, lvl);
            back[kb++] = v;
            if (lvl > kSubstepLevels) gone[kg++] = v;
            else pend[kp++] = v;
          }
        }
        warp_push(stay, ks, mv[nxt], &P.st->sub_count[nxt], P.V, P.st);
        warp_push(back, kb, rv, &P.st->sub_rev[slot], P.V, P.st);
        warp_push(pend, kp, out, &P.st->vl_count[dst], P.V, P.st);
        warp_push(gone, kg, left, &P.st->sub_count[2], P.V, P.st);
      }
      g.sync();
      const int nrev = ld_i(&P.st->sub_rev[slot]);
      cur = nxt;
      if (nrev == 0) break;
      for (int i = spread_tid(); i < nrev; i += stride) {
        const int v = ld_i(rv + i);
        __stcg(P.pos + v, __ldcg(P.vprev + v));
      }
      if (gtid == 0) {
        P.st->sub_count[nxt ^ 1] = 0;  // the list just read becomes the next survivors' list
        P.st->sub_rev[(pass + 1) % 3] = 0;
      }
      g.sync();
    }
    // (c) movers that stayed: at their targets they are done, else they stay
    // pending (lvl 0); (d) their stars are queued for Lawson rounds
    const int m = ld_i(&P.st->sub_count[cur]);
    for (int base = spread_tid() - lane; base < m; base += stride) {
      const int i = base + lane;
      int pend[1];
      int kp = 0;
      int h0 = -1;
      if (i < m) {
        const int v = ld_i(mv[cur] + i);
        const float2 pv = ldpos(P, v), t = __ldcg(P.target + v);
        if (__float_as_uint(pv.x) == __float_as_uint(t.x) && __float_as_uint(pv.y) == __float_as_uint(t.y)) {
          ++done;
        } else {
          __stcg(P.vlocf + v, 0);
          pend[kp++] = v;
        }
        h0 = ld_i(P.vhe + v);
        if (h0 < 0 || h0 >= 2 * P.E) {
          flag_error(P, MCL_ERR_DEGENERATE_INPUT);
          h0 = -1;
        }
      }
      warp_push(pend, kp, out, &P.st->vl_count[dst], P.V, P.st);
      // the stars in lock step across the warp: spokes and link edges
      int h = h0;
      bool active = h0 >= 0;
      for (int it = 0; it < 1024 && __any_sync(kFull, active); ++it) {
        int mine[2];
        int k = 0;
        if (active) {
          const int es = h >> 1, el = he_next(P, h) >> 1;
          if (enqueue_once(P, es, qs)) mine[k++] = es;
          if (el >= 0 && el < P.E && enqueue_once(P, el, qs)) mine[k++] = el;
          h = he_prev(P, h) ^ 1;
          if (h < 0 || h >= 2 * P.E || h == h0) active = false;
        }
        warp_push(mine, k, P.wl0, &P.st->wl_count[0], P.E, P.st);
      }
    }
    g.sync();
    phase_lawson<false>(g, P, 0, stamp, lc, 0);
    src = dst;
  }
  // left for removal: still pending, and past the halving limit
  const int np = ld_i(&P.st->vl_count[src]);
  const int nl = ld_i(&P.st->sub_count[2]);
  for (int i = gtid; i < np + nl; i += stride) {
    const int v = i < np ? ld_i((src ? P.vl1 : P.vl0) + i) : ld_i(left + (i - np));
    if (src || i >= np) __stcg(P.vl2 + i, v);  // staged through the first mover list
  }
  g.sync();
  if (src || nl) {
    for (int i = gtid; i < np + nl; i += stride)
      if (src || i >= np) __stcg(P.vl0 + i, ld_i(P.vl2 + i));
  }
  if (gtid == 0) P.st->vl_count[0] = np + nl;
  warp_add(&P.st->c[C_SUBSTEP_DONE], done);
  g.sync();
}

// The removal path's first part, for a step whose classification found inverted faces:
// the vertices to send back, marked with fs.  The mesh is as it was when it returns.
__device__ __noinline__ int send_back(cg::grid_group g, const KParams P, unsigned fs, long long most) {
  LocalCounters lc = {0, 0, 0, 0, 0, 0, 0};
  KParams Q = P;
  Q.move_mode = MOVE_NONE;  // positions were moved by the classification
  const int rc = phase_fixpoint(g, Q, lc, fs, most);
  flush_counters(P, lc);
  return rc;
}

// The rest of it: remove the vertices sent back (fs), reinsert them at the new positions,
// Lawson.  Out of line, so k_step's hot loops keep their registers; keeps its own
// counters and returns the next free stamp.
__device__ __noinline__ unsigned repair_step(cg::grid_group g, const KParams P, unsigned stamp, unsigned q0,
                                             unsigned fs) {
  LocalCounters lc = {0, 0, 0, 0, 0, 0, 0};
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  KParams Q = P;
  Q.move_mode = MOVE_NONE;
  // Edges to pass through Lawson at the end carry the mark mk: the
  // classification's non-Delaunay edges (queued with q0), then every edge a
  // removal or a split touches.  Any other edge is Delaunay: its quad keeps
  // the positions it was classified with (every sent-back vertex is removed,
  // and each edge whose quad held one is a spoke, gone, or a side of its
  // hole, marked).
  unsigned mk = q0;
  bool ok = true;
  g.sync();
  timeline(P, 43);
  // removal list: reverted vertices that actually moved.  Few: from the
  // list of every vertex sent back (on `hard`); many: by a pass over the
  // vertices, whose id order keeps neighbouring removals in one warp
  // (the mark order scatters them).
  const int stride = gridDim.x * blockDim.x;
  const int nall = ld_i(&P.st->fix_all);
  const bool few = (long long)nall * 64 < (long long)P.V_it;
  if (gtid == 0) { P.st->vl_count[0] = 0; P.st->vl_count[1] = 0; }
  g.sync();
  const int nsb = few ? nall : P.V_it;
  WarpBuf wrev{warp_buf(0), 0};
  for (int base = (few ? spread_tid() - (int)(threadIdx.x & 31) : blockIdx.x * blockDim.x); base < nsb;
       base += stride) {
    const int vi = base + (few ? (int)(threadIdx.x & 31) : (int)threadIdx.x);
    const int v = vi < nsb ? (few ? ld_i(P.hard + vi) : vert_at(P, vi)) : 0;
    int mine[1];
    int k = 0;
    if (vi < nsb && marked(Q, v, fs) && !P.vfix[v]) {
      const float2 pn = ldpos(Q, v), po = P.pos_old[v];
      if (__float_as_uint(pn.x) != __float_as_uint(po.x) || __float_as_uint(pn.y) != __float_as_uint(po.y)) {
        __stcg(P.target + v, pn);
        __stcg(P.pos + v, po);
        __stcg(P.vlocf + v, 0);  // sub-step level
        mine[k++] = v;
      }
    }
    wb_push(wrev, mine, k, P.vl0, &P.st->vl_count[0], P.V, P.st);
  }
  wb_flush(wrev, P.vl0, &P.st->vl_count[0], P.V, P.st);
  g.sync();
  const int nrev = ld_i(&P.st->vl_count[0]);
  if (gtid == 0) P.st->c[C_REVERTED] += (unsigned long long)nrev;
  if (nrev > 0 && P.substeps > 0) {
    // (1b) Delaunay over every edge with the sent-back vertices at their old
    // positions, then sub-steps toward their targets; the mesh is then
    // Delaunay, so only what removal and reinsertion touch is marked
    if (gtid == 0) { P.st->wl_count[0] = 0; P.st->wl_count[1] = 0; P.st->inverted = 0; P.st->hard_count = 0; }
    g.sync();
    const unsigned qa = stamp++;
    const unsigned sc0 = stamp++;
    phase_classify<false>(g, Q, qa, sc0, lc);
    g.sync();
    phase_classify_hard<false>(g, Q, qa, sc0, lc);
    phase_lawson<false>(g, Q, 0, stamp, lc, sc0);
    g.sync();
    timeline_insert(P, 15, 0);
    phase_substeps(g, Q, stamp, lc);
    timeline_insert(P, 15, 1);
    mk = stamp++;
    // the mesh is Delaunay again: the final Lawson list starts empty
    if (gtid == 0) { P.st->wl_count[0] = 0; P.st->wl_count[1] = 0; }
    g.sync();
  }
  const int nrem = ld_i(&P.st->vl_count[0]);
  // few removals: their marks are appended to a list (no pass over every
  // edge afterwards); many: the list is rebuilt from the marks
  Q.append_marks = (long long)nrem * 64 < (long long)P.E_it ? 1 : 0;
  if (!Q.append_marks && gtid == 0) P.st->mark_ovf = 1;
  if (nrem > 0) {
    // (2) remove what is left, marking each hole's sides and diagonals
    ok = phase_remove(g, Q, stamp, lc, mk);
    g.sync();
    timeline(P, 44);
    // (3) reinsert at the new positions: splits only, their edges marked
    if (gtid == 0) { P.st->vl_count[0] = 0; P.st->vl_count[1] = 0; }
    g.sync();
    // the removed vertices: from the list of every vertex sent back when
    // few (and the sub-steps' classification did not reuse its buffer),
    // else by a pass over the vertices
    const bool from_list = few && !(nrev > 0 && P.substeps > 0);
    const int nscan = from_list ? nall : P.V_it;
    WarpBuf wins{warp_buf(0), 0};
    for (int base = (from_list ? spread_tid() - (int)(threadIdx.x & 31) : blockIdx.x * blockDim.x); base < nscan;
         base += stride) {
      const int vi = base + (from_list ? (int)(threadIdx.x & 31) : (int)threadIdx.x);
      const int v = vi < nscan ? (from_list ? ld_i(P.hard + vi) : vert_at(P, vi)) : 0;
      int mine[1];
      int k = 0;
      if (vi < nscan && ld_i(P.vhe + v) < 0 && marked(Q, v, fs)) {
        __stcg(P.pos + v, __ldcg(P.target + v));
        mine[k++] = v;
      }
      wb_push(wins, mine, k, P.vl0, &P.st->vl_count[0], P.V, P.st);
    }
    wb_flush(wins, P.vl0, &P.st->vl_count[0], P.V, P.st);
    g.sync();
    if (ok) ok = phase_insert(g, Q, stamp, lc, mk);
    g.sync();
  } else {
    timeline(P, 44);
  }
  timeline(P, 45);
  // (4) one Lawson pass from every marked edge: work-list 0 holds the
  // classification's non-Delaunay edges and the appended marks, repeats
  // included; deduplicated into work-list 1 when short, else rebuilt from
  // the marks over every edge
  if (ok) {
    const int nw = ld_i(&P.st->wl_count[0]);
    const bool rebuild = ld_i(&P.st->mark_ovf) || (long long)nw * 4 >= (long long)P.E_it;
    g.sync();  // every thread has read the count and the flag
    if (rebuild) {
      if (gtid == 0) { P.st->wl_count[0] = 0; P.st->wl_count[1] = 0; }
      g.sync();
      WarpBuf wb{warp_buf(0), 0};
      for (int base = blockIdx.x * blockDim.x; base < P.E_it; base += stride) {
        const int ei = base + threadIdx.x;
        const int e = ei < P.E_it ? edge_at(P, ei) : -1;
        int mine[1];
        int k = 0;
        if (e >= 0 && (unsigned)ld_i(reinterpret_cast<const int*>(P.qmark) + e) == mk) mine[k++] = e;
        if (__any_sync(kFull, k > 0)) wb_push(wb, mine, k, P.wl0, &P.st->wl_count[0], P.E, P.st);
      }
      wb_flush(wb, P.wl0, &P.st->wl_count[0], P.E, P.st);
      g.sync();
      phase_lawson<false>(g, Q, 0, stamp, lc, 0);
    } else {
      const unsigned du = stamp++;  // first sight of an edge in this pass (cand is free until the flip rounds)
      if (gtid == 0) P.st->wl_count[1] = 0;
      g.sync();
      WarpBuf wb{warp_buf(0), 0};
      for (int base = spread_tid() - (int)(threadIdx.x & 31); base < nw; base += stride) {
        const int i = base + (int)(threadIdx.x & 31);
        int mine[1];
        int k = 0;
        if (i < nw) {
          const int e = ld_i(P.wl0 + i);
          if (e >= 0 && e < P.E && atomicMax(P.cand + e, du) < du) mine[k++] = e;
        }
        if (__any_sync(kFull, k > 0)) wb_push(wb, mine, k, P.wl1, &P.st->wl_count[1], P.E, P.st);
      }
      wb_flush(wb, P.wl1, &P.st->wl_count[1], P.E, P.st);
      if (gtid == 0) P.st->wl_count[0] = 0;
      g.sync();
      phase_lawson<false>(g, Q, 1, stamp, lc, 0);
    }
    g.sync();
  }
  timeline(P, 46);
  flush_counters(P, lc);
  return stamp;
}

// ---------------------------------------------------------------------------
// Untangling by stars (star.cuh) inside the step's launch.

// A vertex's candidates in this thread's slots of the shared pool (idle after
// the classification): a place and an id each, twelve bytes.
struct SharedCand {
  MCL_HD int cap() const { return kStarSlots; }
  __device__ __forceinline__ static float2* at(int i) {
    return reinterpret_cast<float2*>(s_pool) + i * kThreads + threadIdx.x;
  }
  __device__ __forceinline__ static int* who(int i) {
    return reinterpret_cast<int*>(s_pool) + (2 * kStarSlots + i) * kThreads + threadIdx.x;
  }
  __device__ __forceinline__ Cand get(int i) const {
    const float2 q = *at(i);
    return Cand{q.x, q.y, *who(i)};
  }
  __device__ __forceinline__ void set(int i, Cand c) {
    *at(i) = make_float2(c.x, c.y);
    *who(i) = c.id;
  }
};

// The same for any number of candidates, in local memory: the vertices that
// neither the pool's slots nor a warp can take.
__device__ __noinline__ int star_wide(const KParams& P, int v, bool keep, unsigned bad, bool again,
                                      LocalCounters* lc) {
  LocalCand L;
  return again ? star_from_stars(P, v, L, *lc) : star_from_mesh(P, v, keep, bad, L, *lc);
}
__device__ __forceinline__ bool star_alone(const KParams& P, int v, bool keep, unsigned bad, bool again,
                                           LocalCounters& lc) {
  LocalCounters m = {0, 0, 0, 0, 0, 0, 0};
  const int rc = star_wide(P, v, keep, bad, again, &m);
  star_count(lc, m);
  return rc == kStarOk;
}

// ---- one warp per vertex, one candidate (or neighbour) per lane ----------------
// A lone thread takes tens of microseconds over a star (a thousand dependent
// instructions); a warp takes a few.  Each returns false, having written nothing,
// where the thread's form has to decide: wide or open stars, candidates on (nearly)
// one ray, anything malformed.

// The star from candidate x of each lane that has one; ext: the overflow row v has (-1:
// none).
__device__ __forceinline__ bool warp_star(const KParams& P, int v, MeshBase mb, int x, bool valid, int ext,
                                          LocalCounters& lc) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float2 pv = P.pos[v];
  // the warp's slots: the first two records' places in its own threads' columns
  // (SharedCand), 256 bytes each, so that no other warp's candidates are touched
  auto slot = [&](int i) {
    return reinterpret_cast<float4*>(SharedCand::at(i >> 4) - threadIdx.x + (threadIdx.x & ~31)) + (i & 15);
  };
  auto at = [&](int i) {
    const float4 q = *slot(i);
    return Cand{q.x, q.y, __float_as_int(q.w)};
  };
  unsigned alive = 0;
  int p = 0, s = 0;
  auto beside = [&] {
    const unsigned below = alive & lt, above = alive & ~lt & ~(1u << lane);
    p = 31 - __clz(below ? below : alive);
    s = __ffs(above ? above : alive) - 1;
  };
  Cand c;
  unsigned live = __ballot_sync(kFull, valid);
  if (valid) valid = __ffs(__match_any_sync(live, x)) - 1 == lane;  // one lane per vertex
  bool open = true;
  for (int pass = 0; pass < 2 && open; ++pass) {
    if (pass) {
      // the fan does not close: the corners join (none of them is in a lane yet,
      // or the lane that has it stays)
      const unsigned free = ~__ballot_sync(kFull, valid);
      if (__popc(free) < 4) return false;
      const int k = __popc(free & lt);
      if ((free >> lane & 1u) && k < 4) {
        x = mb.v0 + k;
        valid = true;
      }
      live = __ballot_sync(kFull, valid);
      if (valid) valid = __ffs(__match_any_sync(live, x)) - 1 == lane;
    }
    c = valid ? star_cand(pv, x, P.pos[x]) : Cand{0.f, 0.f, -1};
    float key = valid ? star_key(c, 0.f) : 0.f;
    if (__any_sync(kFull, !(key >= 0.f))) return false;
    live = __ballot_sync(kFull, valid);
    if (__popc(live) < 3) continue;
    key -= __shfl_sync(kFull, key, __ffs(live) - 1);
    if (key < 0.f) key += 4.f;
    // place in the angular order, by the keys alone where no two are close
    int rank = 0;
    bool close = false;
    for (unsigned m = live; m; m &= m - 1) {
      const int j = __ffs(m) - 1;
      const float d = __shfl_sync(kFull, key, j) - key;
      rank += d < 0.f ? 1 : 0;
      close |= fabsf(d) < kStarSameKey && j != lane;
    }
    close = __any_sync(kFull, valid && close);
    // else by the exact test; of two on one ray the farther leaves
    while (close) {
      rank = 0;
      bool out = false, same = false;
      for (unsigned m = live; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const float kj = __shfl_sync(kFull, key, j);
        bool before = kj < key;
        const bool near = valid && j != lane && fabsf(kj - key) < kStarSameKey;
        if (__any_sync(kFull, near)) {
          Cand u;
          u.x = __shfl_sync(kFull, c.x, j);
          u.y = __shfl_sync(kFull, c.y, j);
          u.id = __shfl_sync(kFull, c.id, j);
          if (near) {
            int r = star_cross(u, c);
            if (r == 2) {
              LocalCounters t = {0, 0, 0, 0, 0, 0, 0};
              r = star_cross_exact(P.pos, v, u.id, c.id, &t);
              star_count(lc, t);
              if (r == 0) {
                const int nearer = star_nearer(P.pos, v, u.id, c.id);
                same |= nearer < 0;
                out |= nearer == 0;
              }
            }
            before = r > 0;
          }
          __syncwarp();
        }
        rank += before ? 1 : 0;
      }
      if (__any_sync(kFull, same)) return false;
      if (!__any_sync(kFull, out)) break;
      valid = valid && !out;
      live = __ballot_sync(kFull, valid);
    }
    const int n = __popc(live);
    __syncwarp();
    if (valid) *slot(rank) = make_float4(c.x, c.y, 0.f, __int_as_float(c.id));
    __syncwarp();
    alive = n == 32 ? kFull : (1u << n) - 1u;
    c = at(lane < n ? lane : 0);
    // every lane tests its candidate against the two beside it; of a run of neighbours
    // that would drop every other one does, from the first, so what drops is redundant
    // among those that stay
    for (int turn = 0; turn < 64 && __popc(alive) > 3; ++turn) {
      const bool in = alive >> lane & 1u;
      beside();
      int r = 0;
      if (in) {
        const Cand a = at(p), b = at(s);
        r = star_cross(a, b);
        if (r == 1) {
          lc.incircle++;
          r = star_outside(a, b, c);
        }
        if (r == 2) {
          LocalCounters t = {0, 0, 0, 0, 0, 0, 0};
          r = star_cross_exact(P.pos, v, a.id, b.id, &t);
          if (r > 0) r = star_outside_exact(P.pos, v, a.id, b.id, c.id, &t);
          star_count(lc, t);
        }
      }
      __syncwarp();
      const unsigned d = __ballot_sync(kFull, in && r > 0);
      if (!d) break;
      const unsigned keep = alive & ~d;
      if (!keep) {
        alive &= alive - 1u;
        continue;
      }
      // those of the run before this lane: from the last that stays, around the end
      const unsigned from = ~((2u << (31 - __clz(keep & lt ? keep & lt : keep))) - 1u);
      const int ahead = keep & lt ? __popc(d & lt & from) : __popc(d & (lt | from));
      alive &= ~__ballot_sync(kFull, (d >> lane & 1u) && (ahead & 1) == 0);
    }
    beside();
    bool gap = false;
    if (alive >> lane & 1u) {
      const Cand b = at(s);
      int r = star_cross(c, b);
      if (r == 2) {
        LocalCounters t = {0, 0, 0, 0, 0, 0, 0};
        r = star_cross_exact(P.pos, v, c.id, b.id, &t);
        star_count(lc, t);
      }
      gap = r <= 0;
    }
    open = __any_sync(kFull, gap);
    if (open) {  // what has dropped stays redundant when the corners join
      valid = alive >> lane & 1u;
      x = c.id;
    }
  }
  const int k = __popc(alive);
  if (open || k < 3) return false;
  const bool in = alive >> lane & 1u;
  const int i = __popc(alive & lt);
  int* row = P.srow + (size_t)v * kRow;
  if (k > kRowInline) {
    int e = ext;
    if (lane == 0 && e < 0) e = atomicAdd(&P.st->star_ext, 1);
    e = __shfl_sync(kFull, e, 0);
    if (e >= star_ext_rows(P.V)) return false;
    if (in) __stcg(P.sext + (size_t)e * kExtRow + i, c.id);
    if (lane == 0) __stcg(reinterpret_cast<int4*>(row), make_int4(k | kRowExt, e, -1, -1));
    return true;
  }
  const int own = __reduce_or_sync(kFull, in && star_owned(v, c.id, mb.v0 + 4) ? 1u << i : 0u);
  if (in) __stcg(row + 1 + i, c.id);
  if (lane == 0) __stcg(row, k | own << kRowOwn);
  return true;
}

__device__ __forceinline__ bool warp_from_mesh(const KParams& P, int v, bool keep, unsigned bad, LocalCounters& lc) {
  const int lane = threadIdx.x & 31, HE = 2 * P.E;
  const MeshBase mb = star_base(P, v);
  const int s0 = P.vhe[v];
  if ((unsigned)s0 >= (unsigned)HE) return false;
  int h = s0, k = 0, mine = 0;
  do {  // the ring: every lane walks, lane k keeps the k-th side
    const int4 r = P.en[h >> 1];
    const int nx = (h & 1) ? r.z : r.x, pr = (h & 1) ? r.w : r.y;
    if ((unsigned)nx >= (unsigned)HE || (unsigned)pr >= (unsigned)HE) return false;
    if (lane == k) mine = nx;
    ++k;
    h = pr ^ 1;
  } while (h != s0 && k < 16);
  if (h != s0 || k > kRowInline) return false;
  int x = -1, o = -1;
  bool fine = true;
  if (lane < k) {
    const int4 e = P.ev[mine >> 1];
    const bool across = !keep && P.cand[mine >> 1] == bad;
    x = (mine & 1) ? e.y : e.x;
    o = (mine & 1) ? e.z : e.w;
    fine = x >= mb.v0 && x < mb.v1 && o < mb.v1 && x != v;
    if (!across || o < mb.v0 || o == v) o = -1;
  }
  if (!__all_sync(kFull, fine)) return false;
  if (keep) {
    const int own = __reduce_or_sync(kFull, lane < k && star_owned(v, x, mb.v0 + 4) ? 1u << lane : 0u);
    int* row = P.srow + (size_t)v * kRow;
    if (lane < k) __stcg(row + 1 + lane, x);
    if (lane == 0) __stcg(row, k | own << kRowOwn);
  } else {
    const int far = __shfl_sync(kFull, o, lane & 15);
    if (lane >= 16) x = far;
    if (!warp_star(P, v, mb, x, x >= 0, -1, lc)) return false;
  }
  if (lane == 0) __stcg(P.sinbox + (size_t)kInbox * v, 0);
  return true;
}

__device__ __forceinline__ bool warp_from_stars(const KParams& P, int v, LocalCounters& lc) {
  const int lane = threadIdx.x & 31;
  const MeshBase mb = star_base(P, v);
  const int* row = P.srow + (size_t)v * kRow;
  int* box = P.sinbox + (size_t)kInbox * v;
  const int h = row[0], n = h & kRowCount, m = min(box[0], kInbox - 1), ext = h & kRowExt ? row[1] : -1;
  if ((h & kRowOpen) || n + m > 32 || ext >= star_ext_rows(P.V)) return false;
  const int* at = ext >= 0 ? star_ext(P, ext) : row + 1;
  const int x = lane < n ? at[lane] : (lane < n + m ? box[1 + lane - n] : -1);
  const bool valid = lane < n + m;
  if (!__all_sync(kFull, !valid || (x >= mb.v0 && x < mb.v1 && x != v))) return false;
  if (!warp_star(P, v, mb, x, valid, ext, lc)) return false;
  if (lane == 0) __stcg(box, 0);
  return true;
}

// A first star of v with no mesh to start from, one candidate per lane: up to
// kOrderCell points, evenly spread, of v's cell and of each of the eight around it,
// and the two points on each side of v in the order.  Where the warp cannot make a
// star of them they are left as v's neighbours and inbox for the thread's form.
// What they miss the checks bring in: uniform sets of 1,000 to 100,000 points need 8
// to 11 rounds, of which the first takes three quarters of the vertices and the third
// 1 in 70 (two points per cell: 9 in 10 and 1 in 20; the ten points next to v in the
// order alone: more than 64 rounds).
__device__ __forceinline__ bool warp_from_order(const KParams& P, int v, LocalCounters& lc) {
  const int lane = threadIdx.x & 31;
  const MeshBase mb = star_base(P, v);
  const int lo = mb.v0 + 4, hi = mb.v1 - 1;
  const float2 pv = P.pos[v];
  const int bits = __reduce_min_sync(kFull, lane < kOrderNear ? order_cell(P, v, lane, lo, hi) : 32);
  int bound = 0;
  if (bits < 32 && lane < 18) {  // lanes c, c + 9: where cell c begins and ends
    const int c = lane % 9;
    const unsigned x = ((unsigned)(int)pv.x >> bits) + (unsigned)(c % 3 - 1);
    const unsigned y = ((unsigned)(int)pv.y >> bits) + (unsigned)(c / 3 - 1);
    const unsigned long long k = morton_cell(x << bits, y << bits);
    bound = order_bisect(P, lane < 9 ? k : k + (1ull << (2 * bits)), lo, hi);
  }
  __syncwarp();
  const int c = lane / kOrderCell, t = lane % kOrderCell;
  const int a = __shfl_sync(kFull, bound, c < 9 ? c : 0), b = __shfl_sync(kFull, bound, c < 9 ? c + 9 : 0);
  int x = -1;
  if (lane < 9 * kOrderCell) {
    const int m = b - a, take = min(m, kOrderCell);
    if (t < take) x = a + (int)((long long)t * m / take);
  } else if (lane < 31) {
    x = v + (lane < 29 ? lane - 29 : lane - 28);
  }
  const bool valid = x >= lo && x <= hi && x != v;
  int* box = P.sinbox + (size_t)kInbox * v;
  if (warp_star(P, v, mb, x, valid, -1, lc)) {
    if (lane == 0) __stcg(box, 0);
    return true;
  }
  const unsigned live = __ballot_sync(kFull, valid);
  const int at = __popc(live & ((1u << lane) - 1u)), n = min(__popc(live), kRowInline);
  int* row = P.srow + (size_t)v * kRow;
  if (valid && at < kRowInline) __stcg(row + 1 + at, x);
  if (valid && at >= kRowInline && at < kRowInline + kInbox - 1) __stcg(box + 1 + at - kRowInline, x);
  if (lane == 0) {
    __stcg(row, n | kRowOpen);
    __stcg(box, min(__popc(live) - n, kInbox - 1));
  }
  __threadfence_block();
  __syncwarp();
  return false;
}

// star_check and star_commit, an entry per lane.
template <typename Mark>
__device__ __forceinline__ int warp_check(const KParams& P, int v, int c4, bool all, Mark mark, int* inner,
                                          unsigned long long* ranks) {
  const int lane = threadIdx.x & 31;
  const int* row = P.srow + (size_t)v * kRow;
  const int h = row[0], n = h & kRowCount;
  *inner = 0;
  *ranks = 0;
  const int ext = h & kRowExt ? row[1] : -1;
  if (n > 32 || n < 3 || ext >= star_ext_rows(P.V)) {
    int own = 0;
    if (lane == 0) own = star_check(P, v, c4, all, mark, inner, ranks);
    __syncwarp();
    return own;  // lane 0's counts, and only its
  }
  const int* at = ext >= 0 ? star_ext(P, ext) : row + 1;
  const int w = lane < n ? at[lane] : -1;
  const int bf = __shfl_sync(kFull, w, lane ? lane - 1 : n - 1), af = __shfl_sync(kFull, w, lane + 1 < n ? lane + 1 : 0);
  const int own = __popc(__ballot_sync(kFull, lane < n && star_owned(v, w, c4)));
  int r = 0, in = 0;
  if (lane < n) {
    const int4* theirs = reinterpret_cast<const int4*>(P.srow + (size_t)w * kRow);
    r = star_check_entry(P, v, w, bf, af, c4, all, theirs[0], theirs[1], mark);
    in = w >= c4 ? (star_owned(v, w, c4) ? 1 : -1) : 0;
  }
  __syncwarp();
  const bool bad = __any_sync(kFull, r < 0) || (h & kRowOpen);
  const unsigned q = (unsigned)min(r < 0 ? 0 : r, 15);
  const unsigned lo = __reduce_or_sync(kFull, lane < 8 ? q << (4 * lane) : 0u);
  const unsigned hi = __reduce_or_sync(kFull, lane >= 8 && lane < 15 ? q << (4 * (lane - 8)) : 0u);
  in = __reduce_add_sync(kFull, in);
  if (lane == 0) {
    if (bad) mark(v);
    *inner = in;
    *ranks = (unsigned long long)hi << 32 | lo;
    return own;
  }
  return 0;
}

__device__ __forceinline__ bool warp_commit(const KParams& P, int v) {
  const int lane = threadIdx.x & 31;
  const int* row = P.srow + (size_t)v * kRow;
  const int hd = row[0], n = hd & kRowCount;
  bool fine = true;
  if ((hd & kRowExt) || n > kRowInline) {
    if (lane == 0) fine = star_commit(P, v);
  } else {
    const MeshBase mb = star_base(P, v);
    const int w = lane < n ? row[1 + lane] : -1;
    const int prev = lane ? lane - 1 : n - 1, next = lane + 1 < n ? lane + 1 : 0;
    const int bf = __shfl_sync(kFull, w, prev), af = __shfl_sync(kFull, w, next);
    const int mine = __popc((unsigned)hd >> kRowOwn & ((1u << min(lane, 15)) - 1u));
    int h = 0;
    if (lane < n) h = star_spoke(P, mb, v, w, lane, star_edge0(P, mb, v), mine, false, P.srank[v]);
    __syncwarp();
    const int hb = __shfl_sync(kFull, h, prev), ha = __shfl_sync(kFull, h, next);
    if (!__all_sync(kFull, (unsigned)h < (unsigned)(2 * P.E))) return false;
    if (lane < n) fine = star_put(P, mb, v, w, bf, af, h, hb, ha);
    if (lane == 0) __stcg(P.vhe + v, h);
  }
  return __all_sync(kFull, fine);
}

// v and the vertices of its row get the stamp: their checks may come out
// differently once v's row changes.
__device__ __forceinline__ void warp_touch(const KParams& P, int v, unsigned stamp) {
  const int lane = threadIdx.x & 31;
  const int* row = P.srow + (size_t)v * kRow;
  const int h = ld_i(row);
  int n = h & kRowCount;
  const int* at = row + 1;
  if (h & kRowExt) {
    const int e = ld_i(row + 1);
    at = star_ext(P, e >= 0 && e < star_ext_rows(P.V) ? e : 0);
    n = min(n, kExtRow);
  } else {
    n = min(n, kRowInline);
  }
  for (int i = lane; i < n; i += 32) {
    const int w = ld_i(at + i);
    if ((unsigned)w < (unsigned)P.V) __stcg(P.vaux + w, (int)stamp);
  }
  if (lane == 0) __stcg(P.vaux + v, (int)stamp);
}

// Sums of per-thread values over the block, in every thread.
template <int N>
__device__ __forceinline__ void block_sum(int (&x)[N]) {
  __shared__ int part[N][kThreads / 32];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int y = __reduce_add_sync(kFull, x[k]);
    if ((threadIdx.x & 31) == 0) part[k][threadIdx.x >> 5] = y;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    int y = 0;
    for (int w = 0; w < kThreads / 32; ++w) y += part[k][w];
    x[k] = y;
  }
}

// A vertex whose star disagrees joins the round's list once.  Threads that
// arrive together share one atomicAdd.
constexpr int kStarGivenUp = 1 << 30;
__device__ __forceinline__ void star_list(const KParams& P, int u, unsigned cs, int* list, int* count) {
  if (atomicMax(P.smark + u, cs) >= cs) return;
  cg::coalesced_group grp = cg::coalesced_threads();
  int base = 0;
  if (grp.thread_rank() == 0) base = atomicAdd(count, (int)grp.size());
  const int at = grp.shfl(base, 0) + (int)grp.thread_rank();
  if (at < P.V) __stcg(list + at, u);
}

// Stars or removal?  The stars' time goes with the mesh (every vertex is copied, checked
// and written), removal's with the edges that are not Delaunay and the faces turned, in
// rounds that a larger mesh fills better.  Removal goes first where
//  - few vertices moved (`sparse`: only their stars were classified) and the mesh has
//    more than kStarSparse vertices: 460,000 vertices of which 2 % move, stars 1117 us a
//    pass, removal 800; 200,000 and below, stars 0.6 to 0.9 of removal at any number of
//    movers;
//  - few vertices moved (a sixteenth, or an eighth of more than kStarFar), and far: each has
//    turned more than two faces (six of their sides), fewer in larger meshes.  A star finds
//    its way one neighbour a round, removal walks.  us by stars and by removal: 50,000
//    vertices, 150 movers by 3 x spacing 959 and 518; 512 meshes of 300, 460 movers by 3 x
//    730 and 470; 175,000 vertices, 500 movers by 1.5 x 1362 and 498; 64 meshes of 3,000,
//    600 movers by 1 x 486 and 410; but 1,000 vertices, 50 movers by 3 x 324 and 420;
//  - up to six sevenths moved, and far: most of the faces with a moved corner turned.  The
//    line is on turned sides a face, the faces with a mover counted as 1 - (1 - movers)^3 of
//    two a vertex; it rises with the movers, as removal then walks among more holes, and
//    falls as the mesh grows.  us by stars and by removal: 195,000 vertices, 25 % by 2 x
//    spacing 2230 and 1640, 45 % by 2 x 2490 and 2000, 70 % by 3 x 4340 and 2830, but 70 % by
//    1 x 1590 and 2280, all by 2 x 2980 and 4450; 64 meshes of 3,000, 10 % by 2 x 1460 and
//    943; 600,000, 45 % by 2 x 5580 and 3680; 50,000, 45 % by 3 x 1950 and 1590, by 2 x 1314
//    and 1490.  20,000 vertices are within 14 % of removal by 3 x and further, and gain below;
//  - the mesh has more than kStarMost vertices.  Uniform points, sigma = 0.1 x spacing,
//    stars and removal in ms: 1M 1.23 and 1.67, 2M 2.12 and 2.15, 2.5M 2.58 and 2.48, 3M
//    3.12 and 2.92, 4M 4.06 and 3.29, 8.5M 8.34 and 6.05;
//  - between 670,000 and kStarMost vertices, when all move and few of the edges are open
//    (not Delaunay).  Counted twice where hardly a face has turned, as then the stars
//    agree after a round or two (a random walk), and as a third where most vertices
//    stayed.  us by stars and by removal:
//      vertices  open edges  turned   stars  removal
//       700,000       3,400      50     477      390
//       500,000       2,500      50     348      446
//     1,000,000       4,800      40     580      489
//     1,000,000      16,200   3,000    1056      829
//     1,000,000     109,000  32,000    1400     1422
//     1,000,000      22,900     150     734      932   a walk of 0.01 x spacing
//     2,000,000      10,400     320     992      615
//     2,000,000     119,600  31,000    1891     1407
//     2,000,000     592,600 158,000    2454     2767   a walk of 0.15 x spacing
//    Over 135 such steps of 500,000 to 2.5M vertices a step is within 10 % of removal, but
//    one of 700,000 vertices (14 %), and where stars are the faster they are taken, but for
//    a swarm in one place (1M vertices, 1,400 faces: 678 by stars, 814).
constexpr int kStarSparse = 200000;
constexpr int kStarNear = 4096;
constexpr int kStarFar = 100000;
constexpr int kStarMost = 2500000;
constexpr int kStarDense = 850000;   // open edges allowed: 0.28 a vertex above this
constexpr int kStarTurned = 670000;  // the least vertices where a handful of turned faces goes to removal
__device__ __forceinline__ bool removal_first(const KParams& P, int turned, bool sparse) {
  if (P.V_it > kStarMost || (sparse && P.V_it > kStarSparse)) return true;
  if (P.V_it <= kStarNear) return false;
  const long long movers = P.move_mode == MOVE_NONE ? P.V_it : ld_i(&P.st->movers_now);
  const bool wide = P.V_it > kStarFar, few = 16 * movers < P.V_it || (wide && 8 * movers < P.V_it);
  if (few && turned > (wide ? 3 : P.V_it > kStarFar / 3 ? 5 : 6) * movers) return true;
  if (!few && P.V_it > kStarFar / 3 && 7 * movers < 6ll * P.V_it) {
    const float m = (float)movers / (float)P.V_it, still = (1.f - m) * (1.f - m) * (1.f - m);
    const float far = !wide ? 2.f + 0.9f * m : P.V_it <= 5 * kStarFar / 2 ? 1.6f + 1.2f * m : 1.f + 1.6f * m;
    if ((float)turned > far * (1.f - still) * (float)P.V_it) return true;
  }
  if (P.V_it <= kStarTurned) return false;
  const long long n = ld_i(&P.st->wl_count[0]);
  if (turned < 128 && 128 * n < P.V_it) return true;
  const float open = 4 * movers < P.V_it ? 0.333f * (float)n : (32ll * turned < n ? 2.f : 1.f) * (float)n;
  return open < 0.28f * (float)(P.V_it - kStarDense);
}
// Removal is given up for stars while vertices are still being sent back, when they are
// more than twice the turned faces' sides and this: where neighbours move together, far
// beyond their spacing, each vertex sent back turns the next face over until most of the
// mesh is on its way back (20,000 points in a Taylor-Green flow, three spacings a step:
// one face turned, 16,000 vertices; from 100,000 points the send-back did not end).
constexpr int kSentBack = 1024;

// The vertices of the block's run marked with cs, in order, onto a list.
__device__ __forceinline__ void star_marked(const KParams& P, unsigned cs, int i0, int i1, int* list, int* count) {
  const int lane = threadIdx.x & 31;
  WarpBuf wb{warp_buf(0), 0};
  for (int base = i0 + (int)(threadIdx.x & ~31); base < i1; base += kThreads) {
    const int i = base + lane;
    const int v = i < i1 ? vert_at(P, i) : 0;
    const int mine[1] = {v};
    const int k = i < i1 && (unsigned)ld_i(reinterpret_cast<const int*>(P.smark) + v) == cs ? 1 : 0;
    if (__any_sync(kFull, k)) wb_push(wb, mine, k, list, count, P.V, P.st);
  }
  wb_flush(wb, list, count, P.V, P.st);
}

// A build most of whose stars still disagree after this many rounds is left to
// insertion: the order said too little about who is near whom.
constexpr int kStarSettling = 12;
// So is one with a vertex that many others still tell of themselves after a few rounds: it
// takes in kInbox - 1 of them a round, a lone thread's 100 us each, and more than 128
// neighbours are no star.  Points on a circle around one, a whole build in us by insertion
// alone, with the stars to their end, and so: 80 points 1050, 1680, 1050; 130 1180, 3750,
// 1110; 1,000 1790, 5820, 1780.  (From 40 after two rounds on: 910, 1040 and 1510, but
// 100,000 points of a Cauchy distribution 7.5 ms for 5.8.)
constexpr int kStarWideRounds = 3;
constexpr int kStarTold = 48;

// Vertices (or list entries) per warp of the launch up to which a warp takes one
// vertex at a time; above it a thread does.
constexpr int kWarpStars = 8;

// Each block takes a run of consecutive vertices (their rows and positions meet
// in its L1).  Returns false, with the mesh untouched, when the stars cannot be
// made to agree.  A count is read by all threads after a barrier and next written
// two barriers later, so all take the same branches; bit 30 of the next count says
// that a star could not be made.
// kBuild: there is no mesh yet, the first stars come from the Morton order.
// A vertex that this launch has marked (from q0 on: by the classification, or by a
// send-back given up) makes its first star anew, any other keeps its ring.
template <bool kBuild>
__device__ __forceinline__ bool star_step(cg::grid_group& g, const KParams& P, unsigned& stamp, unsigned q0,
                                          unsigned sc0, LocalCounters& lc) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = stride >> 5, gwarp = spread_tid() >> 5;
  const int per = (P.V_it + (int)gridDim.x - 1) / (int)gridDim.x;
  const int i0 = min(P.V_it, (int)blockIdx.x * per), i1 = min(P.V_it, i0 + per);
  const bool few = P.V_it <= kWarpStars * nwarps;
  int* const cnt = P.st->star_n;
  int* const lists[2] = {P.vl0, P.vl1};
  int made = 0;
  bool fine = true;
  __syncthreads();  // the pool's last readers are done
  if (kBuild) {
    for (int v = i0 + warp; v < i1; v += kThreads / 32) {
      if (P.vfix[v]) continue;
      if (!warp_from_order(P, v, lc) && lane == 0) fine = star_alone(P, v, false, 0, true, lc) && fine;
      __syncwarp();
    }
  } else if (few) {
    for (int i = i0 + warp; i < i1; i += kThreads / 32) {
      const int v = vert_at(P, i);
      if (P.vfix[v]) continue;
      const bool keep = (unsigned)ld_i(P.vmark + v) < q0;
      if (lane == 0) made += keep ? 0 : 1;
      if (!warp_from_mesh(P, v, keep, sc0, lc) && lane == 0) fine = star_alone(P, v, keep, sc0, false, lc) && fine;
      __syncwarp();
    }
  } else {
    for (int base = i0 + warp * 32; base < i1; base += kThreads) {
      const int v = base + lane < i1 ? vert_at(P, base + lane) : -1;
      const bool keep = v >= 0 && (unsigned)ld_i(P.vmark + v) < q0;
      int rc = kStarOk;
      if (v >= 0 && !P.vfix[v]) {
        SharedCand L;
        made += keep ? 0 : 1;
        rc = star_from_mesh(P, v, keep, sc0, L, lc);
      }
      fine = fine && rc != kStarDegenerate;
      // those with more candidates than the slots, by the whole warp
      for (unsigned m = __ballot_sync(kFull, rc == kStarFull); m; m &= m - 1) {
        const int j = __ffs(m) - 1, u = __shfl_sync(kFull, v, j);
        const bool k = __shfl_sync(kFull, (int)keep, j) != 0;
        if (!warp_from_mesh(P, u, k, sc0, lc) && lane == 0) fine = star_alone(P, u, k, sc0, false, lc) && fine;
        __syncwarp();
      }
    }
  }
  __syncwarp();
  warp_add(&P.st->star_made, made);
  if (!fine) atomicOr(cnt, kStarGivenUp);
  g.sync();
  timeline(P, 43);
  int slot = 0, rounds = 0;
  int sums[4];
  bool both = false;     // both ends of an edge look for each other
  unsigned touched = 0;  // stamp of the vertices whose check may have changed (0: all)
  for (;;) {
    // every edge against its owner's row; own edges counted per vertex and block
    unsigned cs = stamp++;
    if (gtid == 0) cnt[(slot + 1) % 3] = 0;
    sums[0] = sums[1] = sums[2] = sums[3] = 0;
    auto mark = [&](int u) {
      sums[3] = 1;
      __stcg(P.smark + u, cs);
    };
    for (int i = i0 + (few ? warp : (int)threadIdx.x); i < i1; i += few ? kThreads / 32 : kThreads) {
      const int v = vert_at(P, i);
      int own = 0;
      if (!P.vfix[v]) {
        const int v0 = star_base(P, v).v0;
        int inner;
        unsigned long long ranks;
        // after a round of few vertices only those whose rows met theirs have
        // changed; the others keep what the last check found
        const bool old = touched && (unsigned)ld_i(P.vaux + v) != touched;
        if (old) {
          const int w = ld_i(P.vlocf + v);
          own = w & 0xffff;
          inner = (w >> 16) - 128;
        } else {
          own = few ? warp_check(P, v, v0 + 4, both, mark, &inner, &ranks)
                    : star_check(P, v, v0 + 4, both, mark, &inner, &ranks);
        }
        if (!few || lane == 0) {
          if (!old) {
            __stcg(P.srank + v, ranks);
            __stcg(P.vlocf + v, own | (inner + 128) << 16);
          }
          sums[1] += own - 3 - (v == v0 + 4 ? 1 : 0);
          sums[2] += inner;
        }
      } else if (!few || lane == 0) {
        __stcg(P.vlocf + v, 0);
      }
      if (!few || lane == 0) sums[0] += own;
    }
    __syncwarp();
    block_sum(sums);
    if (threadIdx.x < 4) {
      int x = sums[0];
#pragma unroll
      for (int k = 1; k < 4; ++k) x = threadIdx.x == k ? sums[k] : x;
      __stcg(P.sblk + 4 * blockIdx.x + threadIdx.x, x);
    }
    g.sync();
    if (ld_i(cnt + slot % 3) & kStarGivenUp) return false;
    // own edges of the blocks before this one; the balance over all of them
    sums[0] = sums[1] = sums[2] = sums[3] = 0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads) {
      const int4 q = __ldcg(reinterpret_cast<const int4*>(P.sblk) + b);
      if (b < (int)blockIdx.x) sums[0] += q.x;
      sums[1] += q.y;
      sums[2] += q.z;
      sums[3] += q.w;
    }
    block_sum(sums);
    if (sums[3] == 0) {
      if (sums[1] == 0 && sums[2] == 0) break;
      // an owner holds a vertex that does not hold it: look from both ends
      if (both) return false;
      both = true;
      touched = 0;
      ++slot;
      g.sync();  // the sums have been read
      continue;
    }
    star_marked(P, cs, i0, i1, lists[slot & 1], cnt + slot % 3);
    g.sync();
    int n = ld_i(cnt + slot % 3);
    // the stars that disagree, again, until their neighbourhoods agree: few are made
    // by a warp each, many by a thread each
    const unsigned ts = stamp++;
    bool all_few = true;
    while (n > 0) {
      if (++rounds > kStarRounds) return false;
      const bool many = n > kWarpStars * nwarps;
      const int* list = lists[slot & 1];
      fine = true;
      if (many) {
        all_few = false;
        for (int base = gwarp * 32; base < n; base += stride) {
          const int v = base + lane < n ? ld_i(list + base + lane) : -1;
          int rc = kStarOk;
          if (v >= 0) {
            if (kBuild && rounds > kStarWideRounds) fine = fine && ld_i(P.sinbox + (size_t)kInbox * v) < kStarTold;
            SharedCand L;
            rc = star_from_stars(P, v, L, lc);
          }
          fine = fine && rc != kStarDegenerate;
          for (unsigned m = __ballot_sync(kFull, rc == kStarFull); m; m &= m - 1) {
            const int u = __shfl_sync(kFull, v, __ffs(m) - 1);
            if (!warp_from_stars(P, u, lc) && lane == 0) fine = star_alone(P, u, false, 0, true, lc) && fine;
            __syncwarp();
          }
        }
      } else {
        for (int i = gwarp; i < n; i += nwarps) {
          const int v = ld_i(list + i);
          if (kBuild && rounds > kStarWideRounds) fine = fine && ld_i(P.sinbox + (size_t)kInbox * v) < kStarTold;
          warp_touch(P, v, ts);
          if (!warp_from_stars(P, v, lc) && lane == 0) fine = star_alone(P, v, false, 0, true, lc) && fine;
          __syncwarp();
          warp_touch(P, v, ts);
        }
      }
      if (!fine) atomicOr(cnt + (slot + 1) % 3, kStarGivenUp);
      g.sync();
      if (rounds <= 40) timeline(P, 1 + rounds);
      ++slot;
      if (2 * n > P.V_it) {  // most were made: the next full check does as well
        if (kBuild && rounds > kStarSettling) return false;
        break;
      }
      cs = stamp++;
      int* next = lists[slot & 1];
      int* count = cnt + slot % 3;
      if (gtid == 0) cnt[(slot + 1) % 3] = 0;
      int inner;
      unsigned long long ranks;
      if (many) {
        // before anything joins: an append to a count that holds the bit is taken for a
        // list that is full, an error of the step (star_list leaves such an entry out)
        if (ld_i(count) & kStarGivenUp) return false;
        auto again = [&](int u) { __stcg(P.smark + u, cs); };
        for (int i = spread_tid(); i < n; i += stride) {
          const int v = ld_i(list + i);
          star_check(P, v, star_base(P, v).v0 + 4, true, again, &inner, &ranks);
        }
        __syncwarp();
        g.sync();
        star_marked(P, cs, i0, i1, next, count);
      } else {
        auto again = [&](int u) { star_list(P, u, cs, next, count); };
        for (int i = gwarp; i < n; i += nwarps) {
          const int v = ld_i(list + i);
          warp_check(P, v, star_base(P, v).v0 + 4, true, again, &inner, &ranks);
        }
        __syncwarp();
      }
      g.sync();
      n = ld_i(count);
      if (n >= kStarGivenUp) return false;
      if (n == 0) ++slot;
    }
    touched = all_few ? ts : 0;
  }
  timeline(P, 44);
  int carry = sums[0];
  __shared__ int wsum[kThreads / 32];
  for (int base = i0; base < i1; base += kThreads) {
    const int i = base + threadIdx.x;
    const int v = i < i1 ? vert_at(P, i) : 0;
    const int own = i < i1 ? ld_i(P.vlocf + v) & 0xffff : 0;
    int x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) before += wsum[w];
      all += wsum[w];
    }
    if (i < i1) __stcg(P.sbase + v, carry + before + x - own);
    carry += all;
  }
  g.sync();
  timeline(P, 45);
  for (int i = i0 + (few ? warp : (int)threadIdx.x); i < i1; i += few ? kThreads / 32 : kThreads) {
    const int v = vert_at(P, i);
    if (P.vfix[v]) continue;
    if (!(few ? warp_commit(P, v) : star_commit(P, v))) set_error(P, MCL_ERR_DEGENERATE_INPUT);
  }
  if (gtid == 0) {
    const unsigned long long m = (unsigned long long)ld_i(&P.st->star_made);
    P.st->c[C_REVERTED] += m;
    P.st->c[C_REMOVED] += m;
    P.st->c[C_INSERT_ROUNDS] += (unsigned long long)rounds + 1;
  }
  timeline(P, 46);
  return true;
}

// One kinetic step in one persistent launch: (move +) classify; if a face is
// inverted, untangle by stars, or, where that cannot be, by removal; else Lawson
// rounds to the Delaunay triangulation.
__global__ void __launch_bounds__(kThreads, 3) k_step(const __grid_constant__ KParams P) {
  cg::grid_group g = cg::this_grid();
  LocalCounters lc = {0, 0, 0, 0, 0, 0, 0};
  unsigned stamp = ld_i(reinterpret_cast<const int*>(&P.st->epoch));
  timeline(P, 0);
  const unsigned q0 = stamp++;
  __shared__ unsigned s_q0;
  if (threadIdx.x == 0) s_q0 = q0;
  const unsigned sc0 = stamp++;
  const bool sparse = phase_classify<true>(g, P, q0, sc0, lc);
  g.sync();
  phase_classify_hard<true>(g, P, q0, sc0, lc);
  timeline(P, 1);
  const int inverted = ld_i(&P.st->inverted), hold = ld_i(&P.st->star_hold);
  if (inverted == 0) {
    phase_lawson<true, true>(g, P, 0, stamp, lc, sc0);
  } else {
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (first) P.st->c[C_INVERTED] += (unsigned long long)inverted;
    // no stars where sub-steps are asked for, on a mesh that is not its square's, and for
    // a while after they could not be made
    const bool never = P.substeps > 0 || !P.square, held = hold > 0;
    if (first && held) P.st->star_tried = kStarsHeld;
    // A send-back, unless stars go first; stars, if it is given up; and a send-back to its
    // end, if they cannot be made.  One call of each: with two, removal and the stars both
    // lost registers (512 meshes of 8.5M vertices 8.2 -> 8.6 ms, 1M random walkers 1233 ->
    // 1252 us).
    bool stars = !(never || held || removal_first(P, inverted, sparse)), done = false;
    long long most = never ? LLONG_MAX : 2ll * inverted + kSentBack;
    unsigned fs = stamp++;
    int rc = kSentBackMany;
    for (;;) {
      if (!stars) {
        rc = send_back(g, P, fs, most);
        if (rc == MCL_OK || most == LLONG_MAX) break;
        g.sync();  // its counts have been read; the next barrier is the stars'
        if (first) {
          for (int i = 0; i < 3; ++i) P.st->fix_new[i] = P.st->fix_bad[i] = P.st->fix_list[i] = 0;
          P.st->fix_all = 0;
        }
      }
      // Nothing lives over these calls that the stars need: the counters are flushed and
      // the stamps read again.
      flush_counters(P, lc);
      lc = LocalCounters{0, 0, 0, 0, 0, 0, 0};
      const unsigned q = s_q0;
      stamp = q + 3;  // q, q + 1 and fs are taken
      done = star_step<false>(g, P, stamp, q, q + 1, lc);
      if (blockIdx.x == 0 && threadIdx.x == 0) P.st->star_tried = done ? kStarsMade : kStarsFailed;
      if (done) break;
      stars = false;
      most = LLONG_MAX;
      fs = stamp++;
    }
    if (!done) {
      if (rc == MCL_OK) stamp = repair_step(g, P, stamp, s_q0, fs);
      else if (blockIdx.x == 0 && threadIdx.x == 0) set_error(P, rc);
    }
  }
  flush_counters(P, lc);
  // No closing grid barrier: each block leaves when its own work is done and
  // the last one to leave publishes the launch.  The block barrier orders its
  // threads' counter updates before thread 0's fence, and the fence (which is
  // cumulative) orders them before the block's arrival.
  __syncthreads();
  if (threadIdx.x < 32) {
    int last = 0;
    if (threadIdx.x == 0) {
      atomicMax(&P.st->stamp_max, stamp);
      __threadfence();
      last = atomicAdd(&P.st->arrived, 1u) == gridDim.x - 1 ? 1 : 0;
    }
    if (__shfl_sync(kFull, last, 0)) {
      __threadfence();
      finish_launch(P, __ldcg(&P.st->stamp_max));
      if (threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        P.st->ts[kTimeline - 1] = t;
        P.st->arrived = 0;
        P.st->stamp_max = 0;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Stable radix sort of the points by Morton key, eight bits a pass, in one
// cooperative launch: a digit on which all keys agree is left out, so a set of n
// points one apart takes log2(n) / 8 passes.  Per pass each warp counts the digits of
// its run, a warp per digit sums them over the blocks, and each warp walks its run
// again in order (lanes with one digit find each other by match).  Bound by the three
// grid barriers and the two walks of a pass: 1,000,000 points on 20 bits of key 94 us,
// barrier and scoreboard stalls on top, 12 % of the issue slots used.
//
// Equal keys are counted: their order is the caller's to decide.
struct SortArgs {
  const float2* in;
  ulonglong2* rec[2];  // n each: key, point
  int* hist;           // 256 per block, then 256
  float2* out[2];      // four corners, then the points in order
  unsigned long long* key;  // their keys, from 4
  DevState* st;        // sort_mask, sort_ties
  int n;
};
constexpr int kSortWarps = kThreads / 32;

__global__ void __launch_bounds__(kThreads, 3) k_sort_points(const __grid_constant__ SortArgs A) {
  cg::grid_group g = cg::this_grid();
  __shared__ int cnt[kSortWarps][256];
  __shared__ int wsum[kSortWarps];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, B = gridDim.x;
  const int gtid = blockIdx.x * kThreads + t, stride = B * kThreads;
  const unsigned lt = (1u << lane) - 1u;
  const int per = (A.n + B * kSortWarps - 1) / (B * kSortWarps);  // a warp's run
  const int w0 = blockIdx.x * kSortWarps + warp;
  const int i0 = (int)min((long long)A.n, (long long)w0 * per), i1 = min(A.n, i0 + per);
  auto key = [&](int which, int i) {
    return __ldcg(reinterpret_cast<const unsigned long long*>(A.rec[which] + i));
  };
  unsigned long long mask = 0;
  if (A.n) {
    const float2 p0 = A.in[0];
    const unsigned long long k0 = morton_key(p0.x, p0.y);
    for (int i = gtid; i < A.n; i += stride) {
      const float2 p = A.in[i];
      const unsigned long long k = morton_key(p.x, p.y);
      mask |= k ^ k0;
      __stcg(A.rec[0] + i, make_ulonglong2(k, (unsigned long long)__float_as_uint(p.x) |
                                                  (unsigned long long)__float_as_uint(p.y) << 32));
    }
  }
  const unsigned mlo = __reduce_or_sync(kFull, (unsigned)mask), mhi = __reduce_or_sync(kFull, (unsigned)(mask >> 32));
  if (lane == 0 && (mlo | mhi)) atomicOr(&A.st->sort_mask, (unsigned long long)mhi << 32 | mlo);
  g.sync();
  mask = __ldcg(&A.st->sort_mask);
  int* const tot = A.hist + 256 * B;
  int src = 0;
  for (int shift = mask ? __ffsll((long long)mask) - 1 : 64; shift < 64; shift += 8) {
    if (((mask >> shift) & 255u) == 0) continue;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) cnt[w][t] = 0;
    __syncthreads();
    for (int base = i0; base < i1; base += 32) {
      const bool in = base + lane < i1;
      const int d = in ? (int)(key(src, base + lane) >> shift & 255u) : 256;
      const unsigned peers = __match_any_sync(kFull, d);
      if (in && (peers & lt) == 0) cnt[warp][d] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    int sum = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const int c = cnt[w][t];
      cnt[w][t] = sum;
      sum += c;
    }
    __stcg(A.hist + t * B + blockIdx.x, sum);
    g.sync();
    for (int bin = w0; bin < 256; bin += B * kSortWarps) {
      int carry = 0;
      for (int b = 0; b < B; b += 32) {
        const int x = b + lane < B ? __ldcg(A.hist + bin * B + b + lane) : 0;
        int s = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(kFull, s, o);
          if (lane >= o) s += y;
        }
        if (b + lane < B) __stcg(A.hist + bin * B + b + lane, carry + s - x);
        carry += __shfl_sync(kFull, s, 31);
      }
      if (lane == 0) __stcg(tot + bin, carry);
    }
    g.sync();
    const int mine = __ldcg(tot + t);
    int s = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, s, o);
      if (lane >= o) s += y;
    }
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    int first = s - mine + __ldcg(A.hist + t * B + blockIdx.x);
    for (int w = 0; w < warp; ++w) first += wsum[w];
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) cnt[w][t] += first;
    __syncthreads();
    for (int base = i0; base < i1; base += 32) {
      const bool in = base + lane < i1;
      ulonglong2 r = make_ulonglong2(0, 0);
      if (in) r = __ldcg(A.rec[src] + base + lane);
      const int d = in ? (int)(r.x >> shift & 255u) : 256;
      const unsigned peers = __match_any_sync(kFull, d);
      int at = 0;
      if (in) at = cnt[warp][d] + __popc(peers & lt);
      __syncwarp();
      if (in && (peers & lt) == 0) cnt[warp][d] += __popc(peers);
      __syncwarp();
      if (in) __stcg(A.rec[src ^ 1] + at, r);
    }
    g.sync();
    src ^= 1;
  }
  int ties = 0;
  for (int i = gtid; i < A.n; i += stride) {
    const ulonglong2 r = __ldcg(A.rec[src] + i);
    const float2 p = make_float2(__uint_as_float((unsigned)r.y), __uint_as_float((unsigned)(r.y >> 32)));
    if (i && key(src, i - 1) == r.x) ++ties;
    A.out[0][4 + i] = p;
    A.out[1][4 + i] = p;
    A.key[4 + i] = r.x;
  }
  if (gtid < 4) {
    const float2 c = make_float2(gtid == 0 || gtid == 3 ? -kSquare : kSquare, gtid < 2 ? -kSquare : kSquare);
    A.out[0][gtid] = c;
    A.out[1][gtid] = c;
  }
  ties = __reduce_add_sync(kFull, ties);
  if (lane == 0 && ties) atomicAdd(&A.st->sort_ties, ties);
}

// What insertion starts from: the square of two triangles (the reference's seed,
// include/Host_Triangulation.h:107-137), every vertex pending, and its three edges.
__constant__ const int kSeed[10][4] = {{2, 0, 0, 2},  {9, 1, -1, -1}, {4, 1, 0, 0},  {1, 2, -1, -1}, {0, 2, 0, 1},
                                       {6, 0, 1, 3},  {8, 2, 1, 0},   {3, 3, -1, -1}, {5, 3, 1, 2},  {7, 0, -1, -1}};
__device__ __forceinline__ void phase_seed(const KParams& P) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (int e = gtid; e < P.E; e += stride) {
    int4 v = make_int4(-1, -1, -1, -1), n = v;
    if (e < 5) {
      const int *a = kSeed[2 * e], *b = kSeed[2 * e + 1];
      int pa = 0, pb = 0;
      for (int h = 0; h < 10; ++h) {
        pa = kSeed[h][0] == 2 * e ? h : pa;
        pb = kSeed[h][0] == 2 * e + 1 ? h : pb;
      }
      v = make_int4(a[1], b[1], a[2] >= 0 ? a[3] : -1, b[2] >= 0 ? b[3] : -1);
      n = make_int4(a[0], pa, b[0], pb);
    }
    __stcg(P.ev + e, v);
    __stcg(P.en + e, n);
  }
  for (int v = gtid; v < P.V; v += stride) {
    __stcg(P.vhe + v, v < 4 ? (v < 2 ? 2 * v : 2 * v + 2) : -1);
    __stcg(P.vhint + v, 0);
    __stcg(P.vaux + v, -1);
    if (v >= 4) __stcg(P.vl0 + v - 4, v);
    for (int k = 0; k < 3; ++k) __stcg(P.vfree + 3 * v + k, v < 4 ? -1 : 5 + 3 * (v - 4) + k);
  }
  if (gtid == 0) {
    P.st->vl_count[0] = P.V - 4;
    P.st->vl_count[1] = 0;
  }
}

// The initial triangulation of the sorted points: by stars, or, where they do not come
// to agree (coincident points, an order that says little), by parallel insertion
// rounds from the bounding square.  Points on equal keys are left to the host's sort
// first (`sorted`), and many of them to insertion: their order is arbitrary.
// Bound by the first stars (a warp each, 31 candidates: about 3000 issue slots) and, on
// small sets, by the rounds' latency, 15 to 20 us each.  Insertion -> stars, GB300:
// 10,000 points 2430 -> 332 us, 100,000 points 3.6 ms -> 880 us, 1,000,000 points
// 9.1 -> 5.7 ms.
constexpr int kBuildTies = 8;  // one in this many
__global__ void __launch_bounds__(kThreads, 3) k_build(const __grid_constant__ KParams P, int sorted) {
  cg::grid_group g = cg::this_grid();
  const int ties = ld_i(&P.st->sort_ties);
  if (!sorted && ties) return;
  timeline(P, 0);
  LocalCounters lc = {0, 0, 0, 0, 0, 0, 0};
  unsigned stamp = ld_i(reinterpret_cast<const int*>(&P.st->epoch));
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  if (sorted) {
    for (int v = gtid; v < P.V; v += gridDim.x * blockDim.x)
      __stcg(P.skey + v, morton_key(P.pos[v].x, P.pos[v].y));
    g.sync();
  }
  if (P.V <= 4 || ties > P.V / kBuildTies || !star_step<true>(g, P, stamp, 0, 0, lc)) {
    g.sync();
    phase_seed(P);
    g.sync();
    phase_insert(g, P, stamp, lc);
  }
  flush_counters(P, lc);
  g.sync();
  if (gtid < 32) finish_launch(P, stamp);
}

// ---------------------------------------------------------------------------
// Host side.
static thread_local std::string g_last_error;

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

}  // namespace mcl

void mcl_set_last_error(const std::string& msg) { mcl::g_last_error = msg; }

namespace mcl {

int cuda_fail(cudaError_t e, const char* what) {
  return fail(e == cudaErrorMemoryAllocation ? MCL_ERR_OUT_OF_MEMORY : MCL_ERR_CUDA,
              std::string(what) + ": " + cudaGetErrorString(e));
}

#define CK(call)                                   \
  do {                                             \
    cudaError_t _e = (call);                       \
    if (_e != cudaSuccess) return cuda_fail(_e, #call); \
  } while (0)

void free_mesh(mcl_mesh* m) {
  if (!m) return;
  void* ptrs[] = {m->slab, m->cebase, m->vprev, m->vl2, m->vcomp, m->vroot, m->cbase, m->table, m->smark, m->smove,
                  m->fnew, m->act_dev, m->bg_cell, m->bg_src, m->bg_rank, m->bg_bucket, m->bg_pos, m->bg_count,
                  m->bg_start, m->bg_local, m->bg_pre, m->bg_par, m->aos_tmp};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  if (m->dstage2) cudaFree(m->dstage2);
  if (m->stats_dev) cudaFree(m->stats_dev);
  if (m->copy_stream) {
    cudaStreamSynchronize(m->copy_stream);
    cudaStreamDestroy(m->copy_stream);
    for (int i = 0; i < 2; ++i) {
      cudaEventDestroy(m->ev_copied[i]);
      cudaEventDestroy(m->ev_used[i]);
    }
  }
  if (m->st_host) {
    if (m->counts_host) cudaHostUnregister(m->st_host);
    std::free(m->st_host);
  }
  if (m->act_host) cudaFreeHost(m->act_host);
  if (m->bg_par_host) cudaFreeHost(m->bg_par_host);
  delete[] m->comp_host;
  delete[] m->act_list;
  delete[] m->dirty;
  delete m;
}

const float2* valid_positions(const mcl_mesh* m) { return m->valid_cur ? m->pos[m->cur] : m->pos[m->cur ^ 1]; }

ActV act_of(const mcl_mesh* m) {
  ActV a;
  a.n = m->nact;
  a.V_it = m->nact ? m->act_V : (int)m->V;
  a.pre = m->nact ? m->act_dev + 2 * m->ncomp + 1 : nullptr;
  a.v0 = m->nact ? m->act_dev + 3 * m->ncomp + 2 : nullptr;
  return a;
}

int alloc_mesh(int64_t V, int64_t E, mcl_mesh** out) {
  if (V < 4 || E < 5 || V > (1ll << 30) || E > (1ll << 29))
    return fail(MCL_ERR_INVALID_ARGUMENT, "mesh size out of range");
  int dev = 0;
  CK(cudaGetDevice(&dev));
  mcl_mesh* m = new mcl_mesh();
  std::memset(m, 0, sizeof(*m));
  m->device = dev;
  m->V = V;
  m->E = E;
  m->T = 2 * (V - 4) + 2;
  m->cur = 0;
  m->valid_cur = true;
  // one allocation, each array on 256 bytes; those that start as zeros lie together, and
  // those that start as -1
  size_t at = 0;
  std::vector<std::pair<void**, size_t>> parts;
  auto A = [&](void** p, size_t bytes) {
    parts.emplace_back(p, at);
    at += (bytes + 255) / 256 * 256;
  };
  A((void**)&m->pos[0], 8 * V);
  A((void**)&m->pos[1], 8 * V);
  A((void**)&m->ev, 16 * E);
  A((void**)&m->en, 16 * E);
  A((void**)&m->vhe, 4 * V);
  A((void**)&m->vfix, V);
  A((void**)&m->efa, std::max(8 * E, 4 * kInbox * V));
  A((void**)&m->hard, 4 * E);
  A((void**)&m->wl[0], 4 * E);
  A((void**)&m->wl[1], 4 * E);
  A((void**)&m->vl[0], 4 * V);
  A((void**)&m->vl[1], 4 * V);
  A((void**)&m->vfree, 12 * V);
  A((void**)&m->vloc, 4 * V);
  A((void**)&m->vlocf, 4 * V);
  A((void**)&m->target, 8 * V);
  A((void**)&m->dstage, 8 * V);
  const size_t ones = at;
  A((void**)&m->vaux, 4 * V);
  A((void**)&m->vhint, 4 * V);
  const size_t zeros = at + 4 * star_mark_at(V);  // the marks end the star scratch
  A((void**)&m->star, 4 * star_ints(V));
  A((void**)&m->cand, 4 * E);
  A((void**)&m->win, 4 * E);
  A((void**)&m->qmark, 4 * E);
  A((void**)&m->claim, 8 * 2 * E);
  A((void**)&m->vmark, 4 * V);
  A((void**)&m->scratch, kScratchBytes);
  A((void**)&m->st, sizeof(DevState));
  cudaError_t e = cudaMalloc((void**)&m->slab, at);
  if (e == cudaSuccess)
    for (const auto& [p, off] : parts) *p = m->slab + off;
  // the mirror of the device state, behind it the counts that queries write and a step's
  // record: pages of the host's, pinned in place
  if (e == cudaSuccess) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), 
                 bytes = (sizeof(DevState) + 8 * kCountSlots + sizeof(mcl_step_stats) + page - 1) / page * page;
    m->st_host = static_cast<DevState*>(std::aligned_alloc(page, bytes));
    e = m->st_host ? cudaHostRegister(m->st_host, bytes, cudaHostRegisterMapped) : cudaErrorMemoryAllocation;
  }
  if (e == cudaSuccess) m->counts_host = reinterpret_cast<unsigned long long*>(m->st_host + 1);
  if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&m->counts_dev, m->counts_host, 0);
  static_assert(sizeof(DevState) % 8 == 0, "what follows the state in the mirror's pages");
  if (e == cudaSuccess) {
    m->stats_host = reinterpret_cast<mcl_step_stats*>(m->counts_host + kCountSlots);
    m->stats_map = reinterpret_cast<mcl_step_stats*>(m->counts_dev + kCountSlots);
  }
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    free_mesh(m);
    return cuda_fail(e, "cudaMalloc(mesh)");
  }
  e = cudaMemsetAsync(m->slab + zeros, 0, at - zeros, 0);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->slab + ones, 0xff, zeros - 4 * star_mark_at(V) - ones, 0);
  const unsigned epoch = 1;
  if (e == cudaSuccess) e = cudaMemcpy(&m->st->epoch, &epoch, sizeof(epoch), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    free_mesh(m);
    return cuda_fail(e, "mesh init");
  }
  int nsm = 0, per_sm = 0;
  e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  int per_sm2 = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_step, kThreads, 0);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm2, k_build, kThreads, 0);
  if (e != cudaSuccess || per_sm < 1 || per_sm2 < 1) {
    free_mesh(m);
    return cuda_fail(e == cudaSuccess ? cudaErrorInvalidConfiguration : e, "occupancy(k_step, k_build)");
  }
  m->coop_threads = kThreads;
  m->nsm = nsm;
  m->max_blocks_per_sm = per_sm;
  m->tail_items = kTailItems;
  m->substeps = kSubsteps;
  m->ncomp = 1;
  m->coop_blocks = nsm * per_sm;
  m->repair_blocks = nsm * per_sm2;
  *out = m;
  return MCL_OK;
}

// Convert and validate the reference AoS arrays; returns false on malformed input.
static bool aos_to_soa(const mcl_aos_view* a, std::vector<int4>& ev, std::vector<int4>& en, std::vector<int>& vhe,
                       std::string& why) {
  const int64_t V = a->V, HE = a->HE, E = HE / 2;
  if (HE % 2 || V < 4 || E < 5) { why = "bad sizes"; return false; }
  const int32_t* he = a->he;
  ev.assign(E, make_int4(0, 0, 0, 0));
  en.assign(E, make_int4(0, 0, 0, 0));
  std::vector<int> prev(HE, -1);
  for (int64_t h = 0; h < HE; ++h) {
    const int nx = he[4 * h], v = he[4 * h + 1], t = he[4 * h + 2], op = he[4 * h + 3];
    if (nx < 0 || nx >= HE || v < 0 || v >= V) { why = "half-edge index out of range"; return false; }
    if (t >= 0 && (op < 0 || op >= V)) { why = "opposite vertex out of range"; return false; }
    if (prev[nx] != -1) { why = "two half-edges share a next"; return false; }
    prev[nx] = (int)h;
  }
  for (int64_t h = 0; h < HE; ++h) {
    const int nx = he[4 * h];
    // the twin's origin must be this half-edge's destination
    if (he[4 * (h ^ 1) + 1] != he[4 * nx + 1]) { why = "twin/next inconsistent"; return false; }
    if (he[4 * h + 2] >= 0) {
      const int n2 = he[4 * nx], n3 = he[4 * n2];
      if (n3 != h) { why = "inner face is not a triangle"; return false; }
      if (he[4 * h + 3] != he[4 * n2 + 1]) { why = "opposite vertex inconsistent"; return false; }
    }
  }
  for (int64_t e = 0; e < E; ++e) {
    const int32_t* h0 = he + 8 * e;
    const int32_t* h1 = h0 + 4;
    ev[e] = make_int4(h0[1], h1[1], h0[2] >= 0 ? h0[3] : -1, h1[2] >= 0 ? h1[3] : -1);
    en[e] = make_int4(h0[0], prev[2 * e], h1[0], prev[2 * e + 1]);
  }
  vhe.assign(V, -1);
  for (int64_t v = 0; v < V; ++v) {
    const int h = a->v[2 * v + 1];
    if (h < 0 || h >= HE || he[4 * h + 1] != v) { why = "vertex he is not outgoing"; return false; }
    vhe[v] = h;
  }
  return true;
}

// mcl_mesh::square of a mesh that aos_to_soa has accepted.
static bool has_square(const mcl_aos_view* a) {
  int64_t border = 0;
  for (int64_t h = 0; h < a->HE; ++h) {
    if (a->he[4 * h + 2] >= 0) continue;
    const int from = a->he[4 * h + 1], to = a->he[4 * (h ^ 1) + 1];
    if (from > 3 || to != ((from + 3) & 3)) return false;
    ++border;
  }
  const mcl_float2* p = a->pos;
  return border == 4 && p[0].x < p[1].x && p[1].y < p[2].y && p[0].y == p[1].y && p[1].x == p[2].x &&
         p[2].y == p[3].y && p[3].x == p[0].x;
}

static int upload_soa(mcl_mesh* m, const mcl_float2* pos, const std::vector<int4>& ev, const std::vector<int4>& en,
                      const std::vector<int>& vhe) {
  std::vector<unsigned char> fix(m->V, 0);
  for (int i = 0; i < 4 && i < m->V; ++i) fix[i] = 1;
  m->cur = 0;
  m->valid_cur = true;
  CK(cudaMemcpy(m->pos[0], pos, 8 * m->V, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(m->pos[1], pos, 8 * m->V, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(m->ev, ev.data(), 16 * m->E, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(m->en, en.data(), 16 * m->E, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(m->vhe, vhe.data(), 4 * m->V, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(m->vfix, fix.data(), m->V, cudaMemcpyHostToDevice));
  return MCL_OK;
}

// transferToHost for the vertices [vb, vb + nv) and edges [eb, eb + ne) of one
// component (the whole mesh, or one mesh of a batch), renumbered from 0.
int download_range(mcl_mesh* m, int64_t vb, int64_t nv, int64_t eb, int64_t ne, int64_t T, mcl_float2* pos,
                   int32_t* v, int32_t* he, int32_t* t) {
  CK(cudaDeviceSynchronize());
  const int64_t V = nv, E = ne, HE = 2 * E;
  if (pos) CK(cudaMemcpy(pos, m->pos[m->cur] + vb, 8 * V, cudaMemcpyDeviceToHost));
  if (!v && !he && !t) return MCL_OK;
  std::vector<int4> ev(E), en(E);
  std::vector<int> vhe(V);
  CK(cudaMemcpy(ev.data(), m->ev + eb, 16 * E, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(en.data(), m->en + eb, 16 * E, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(vhe.data(), m->vhe + vb, 4 * V, cudaMemcpyDeviceToHost));
  const int hb = (int)(2 * eb), vbi = (int)vb;
  bool bad = false;
  auto lv = [&](int x) {
    if (x < 0) return -1;
    x -= vbi;
    if (x >= V || x < 0) bad = true;
    return x;
  };
  auto lh = [&](int x) {
    if (x < 0) return -1;
    x -= hb;
    if (x >= HE || x < 0) bad = true;
    return x;
  };
  for (int64_t e = 0; e < E; ++e) {
    ev[e] = make_int4(lv(ev[e].x), lv(ev[e].y), lv(ev[e].z), lv(ev[e].w));
    en[e] = make_int4(lh(en[e].x), lh(en[e].y), lh(en[e].z), lh(en[e].w));
  }
  for (int64_t i = 0; i < V; ++i) vhe[i] = lh(vhe[i]);
  if (bad) return fail(MCL_ERR_DEGENERATE_INPUT, "download: index outside the component");
  auto org = [&](int64_t h) { const int4& q = ev[h >> 1]; return (h & 1) ? q.y : q.x; };
  auto apex = [&](int64_t h) { const int4& q = ev[h >> 1]; return (h & 1) ? q.w : q.z; };
  auto nxt = [&](int64_t h) { const int4& q = en[h >> 1]; return (h & 1) ? q.z : q.x; };
  auto prv = [&](int64_t h) { const int4& q = en[h >> 1]; return (h & 1) ? q.w : q.y; };
  std::vector<int> face(HE, -1);
  int64_t nf = 0;
  std::vector<int> owner;
  owner.reserve(T);
  for (int64_t h = 0; h < HE; ++h) {
    if (apex(h) < 0 || org(h) < 0) continue;
    const int64_t n = nxt(h), p = prv(h);
    if (h < n && h < p) {
      face[h] = (int)nf++;
      owner.push_back((int)h);
    }
  }
  for (int64_t h = 0; h < HE; ++h) {
    if (apex(h) < 0 || org(h) < 0) continue;
    const int64_t n = nxt(h), p = prv(h);
    face[h] = face[std::min(h, std::min(n, p))];
  }
  if (he) {
    for (int64_t h = 0; h < HE; ++h) {
      he[4 * h] = nxt(h);
      he[4 * h + 1] = org(h);
      he[4 * h + 2] = face[h];
      he[4 * h + 3] = apex(h) >= 0 ? apex(h) : -1;
    }
  }
  if (v) {
    for (int64_t i = 0; i < V; ++i) {
      v[2 * i] = (int)i;
      v[2 * i + 1] = vhe[i];
    }
  }
  if (t) {
    for (int64_t i = 0; i < (int64_t)owner.size() && i < T; ++i) t[i] = owner[i];
  }
  if (nf != T) return fail(MCL_ERR_DEGENERATE_INPUT, "face count mismatch on download");
  return MCL_OK;
}

static KParams make_params(mcl_mesh* m, int mode) {
  KParams P;
  std::memset(&P, 0, sizeof(P));
  P.V = (int)m->V;
  P.E = (int)m->E;
  P.ev = m->ev;
  P.en = m->en;
  P.vhe = m->vhe;
  P.vfix = m->vfix;
  P.cand = m->cand;
  P.win = m->win;
  P.qmark = m->qmark;
  P.efa = m->efa;
  P.hard = m->hard;
  P.wl0 = m->wl[0];
  P.wl1 = m->wl[1];
  P.vl0 = m->vl[0];
  P.vl1 = m->vl[1];
  P.vmark = m->vmark;
  P.claim = m->claim;
  P.vfree = m->vfree;
  P.vhint = m->vhint;
  P.vaux = m->vaux;
  P.vloc = m->vloc;
  P.vlocf = m->vlocf;
  P.target = m->target;
  P.vprev = m->vprev;
  P.vl2 = m->vl2;
  P.srow = m->star;
  P.sext = m->star + (int64_t)kRow * m->V;
  P.smark = reinterpret_cast<unsigned*>(m->star + star_mark_at(m->V));
  P.sblk = m->star + star_sums_at(m->V);
  P.sinbox = reinterpret_cast<int*>(m->efa);
  P.srank = reinterpret_cast<unsigned long long*>(m->target);
  P.sbase = m->vloc;
  P.skey = reinterpret_cast<unsigned long long*>(m->vfree);
  P.vcomp = m->vcomp;
  P.cbase = m->cbase;
  P.cebase = m->cebase;
  P.st = m->st;
  P.mode = mode;
  P.max_rounds = 1 << 16;
  P.walk_cap = 1 << 18;
  P.tail_items = m->tail_items;
  P.rm_tile = m->rm_tile;
  P.substeps = m->vl2 ? m->substeps : 0;  // no scratch, no sub-steps
  P.vroot = m->vroot;
  P.nact = m->nact;
  P.E_it = m->nact ? m->act_E : (int)m->E;
  P.V_it = m->nact ? m->act_V : (int)m->V;
  if (m->nact) {
    const int64_t nc = m->ncomp;
    P.act_epre = m->act_dev;
    P.act_e0 = m->act_dev + nc + 1;
    P.act_vpre = m->act_dev + 2 * nc + 1;
    P.act_v0 = m->act_dev + 3 * nc + 2;
  }
  return P;
}

static int launch_engine(mcl_mesh* m, KParams& P, cudaStream_t s) {
  void* args[] = {&P};
  CK(cudaLaunchCooperativeKernel((void*)k_step, dim3(m->coop_blocks), dim3(m->coop_threads), args, 0, s));
  return MCL_OK;
}

static void fill_stats_from(const unsigned long long* c, int status, int site, mcl_step_stats* o);

static void fill_stats(const DevState& s, mcl_step_stats* o) {
  fill_stats_from(s.last, s.last_status, s.last_site, o);
  o->failed_launches = s.last_status != MCL_OK ? 1 : 0;
}

static void fill_stats_from(const unsigned long long* c, int status, int site, mcl_step_stats* o) {
  struct { const unsigned long long* c; } s{c};
  o->inverted_faces = (int64_t)s.c[C_INVERTED];
  o->reverted_vertices = (int64_t)s.c[C_REVERTED];
  o->removed_vertices = (int64_t)s.c[C_REMOVED];
  o->lawson_flips = (int64_t)s.c[C_LAWSON_FLIPS];
  o->lawson_rounds = (int64_t)s.c[C_LAWSON_ROUNDS];
  o->removal_flips = (int64_t)s.c[C_REMOVAL_FLIPS];
  o->insert_rounds = (int64_t)s.c[C_INSERT_ROUNDS];
  o->incircle_tests = (int64_t)s.c[C_INCIRCLE];
  o->incircle_fp64 = (int64_t)s.c[C_INCIRCLE_FP64];
  o->incircle_exact = (int64_t)s.c[C_INCIRCLE_EXACT];
  o->orient_fp64 = (int64_t)s.c[C_ORIENT_FP64];
  o->orient_exact = (int64_t)s.c[C_ORIENT_EXACT];
  o->sos_decisions = (int64_t)s.c[C_SOS];
  o->substep_vertices = (int64_t)s.c[C_SUBSTEP_DONE];
  o->status = status;
  o->error_site = site;
  o->failed_launches = 0;
}

static int checked(mcl_mesh* m, int status) {
  m->last_status = status;
  return status == MCL_OK ? MCL_OK : fail(status, std::string("device status: ") + mcl_status_string(status));
}
static int finish(mcl_mesh* m, cudaStream_t s, mcl_step_stats* stats) {
  if (!stats) return MCL_OK;
  CK(cudaMemcpyAsync(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  fill_stats(*m->st_host, stats);
  return checked(m, m->st_host->last_status);
}

// Run the engine.  Position buffers: pos[cur] holds the positions the mesh
// must be repaired to; when valid_cur is false (points were moved since the
// last validated state) pos[cur^1] holds the validated positions.  A fused move
// (valid_cur true) reads pos[cur] and writes pos[cur^1].
// stats_mapped (may be NULL): device-visible pinned host record the launch
// itself fills at its end.
static int run_step(mcl_mesh* m, int move_mode, const float2* d, cudaStream_t s, mcl_step_stats* stats,
                    mcl_step_stats* stats_mapped = nullptr) {
  KParams P = make_params(m, ENGINE_STEP);
  P.stats_out = stats ? m->stats_map : stats_mapped;  // no caller gives both
  if (move_mode != MOVE_NONE) {
    if (m->dirty) {
      // the launch writes the other position buffer for the active meshes
      // only: the inactive meshes whose buffers differ are brought in step first
      if (m->nact) {
        std::vector<unsigned char> on((size_t)m->ncomp, 0);
        for (int i = 0; i < m->nact; ++i) on[(size_t)m->act_list[i]] = 1;
        int64_t stale = 0;
        for (int64_t c = 0; c < m->ncomp; ++c) stale += (!on[(size_t)c] && m->dirty[c]) ? 1 : 0;
        if (stale > 16) {
          // many small copies cost more than one copy of every position (the
          // launch rewrites the active meshes' part anyway)
          CK(cudaMemcpyAsync(m->pos[m->cur ^ 1], m->pos[m->cur], 8 * m->V, cudaMemcpyDeviceToDevice, s));
          std::memset(m->dirty, 0, (size_t)m->ncomp);
        } else {
          for (int64_t c = 0; c < m->ncomp; ++c) {
            if (on[(size_t)c] || !m->dirty[c]) continue;
            const int64_t v0 = m->comp_host[4 * c], nv = m->comp_host[4 * c + 1];
            CK(cudaMemcpyAsync(m->pos[m->cur ^ 1] + v0, m->pos[m->cur] + v0, 8 * nv, cudaMemcpyDeviceToDevice, s));
            m->dirty[c] = 0;
          }
        }
        for (int i = 0; i < m->nact; ++i) m->dirty[m->act_list[i]] = 1;
      } else {
        std::memset(m->dirty, 1, (size_t)m->ncomp);
      }
    }
    P.pos_old = m->pos[m->cur];
    P.pos = m->pos[m->cur ^ 1];
    P.move_mode = move_mode;
    P.disp = d;
    m->cur ^= 1;
  } else {
    P.pos = m->pos[m->cur];
    P.pos_old = m->valid_cur ? m->pos[m->cur] : m->pos[m->cur ^ 1];
  }
  P.sparse_ok = m->delaunay ? 1 : 0;
  P.square = m->square ? 1 : 0;
  int rc = launch_engine(m, P, s);
  if (rc != MCL_OK) return rc;
  m->valid_cur = true;
  m->delaunay = true;  // a step ends Delaunay (or with an error status)
  if (!stats) return MCL_OK;
  CK(cudaStreamSynchronize(s));
  *stats = *m->stats_host;
  return checked(m, stats->status);
}

// Structural invariants of the device mesh (counted per kind):
//  0 next/prev not inverse   1 inner face not a 3-cycle   2 apex != origin(prev)
//  3 origin(next) != origin(twin)   4 vhe not outgoing   5 face not positive
//  6 dead edge   7 index out of range
__global__ void k_validate(KParams P, unsigned long long* bad) {
  LocalCounters lc = {0, 0, 0, 0, 0, 0, 0};
  const int HE = 2 * P.E;
  for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < HE + P.V; h += gridDim.x * blockDim.x) {
    if (h >= HE) {
      const int v = h - HE;
      const int o = ld_i(P.vhe + v);
      if (o < 0) continue;
      if (bad_h(P, o)) { atomicAdd(bad + 7, 1ull); continue; }
      if (he_origin(P, o) != v) atomicAdd(bad + 4, 1ull);
      continue;
    }
    if (he_origin(P, h) < 0) { atomicAdd(bad + 6, 1ull); continue; }
    const int n = he_next(P, h), p = he_prev(P, h);
    if (bad_h(P, n) || bad_h(P, p)) { atomicAdd(bad + 7, 1ull); continue; }
    if (he_prev(P, n) != h || he_next(P, p) != h) atomicAdd(bad + 0, 1ull);
    if (he_origin(P, n) != he_origin(P, h ^ 1)) atomicAdd(bad + 3, 1ull);
    const int ap = he_apex(P, h);
    if (ap >= 0) {
      if (he_next(P, n) != p) atomicAdd(bad + 1, 1ull);
      if (ap != he_origin(P, p)) atomicAdd(bad + 2, 1ull);
      if (h < n && h < p) {
        const int a = he_origin(P, h), b = he_origin(P, n), c = he_origin(P, p);
        if (bad_v(P, a) || bad_v(P, b) || bad_v(P, c)) { atomicAdd(bad + 7, 1ull); continue; }
        if (orient_v(P, ldpos(P, a), ldpos(P, b), ldpos(P, c), lc) <= 0) atomicAdd(bad + 5, 1ull);
      }
    }
  }
}

}  // namespace mcl

using namespace mcl;

// ---------------------------------------------------------------------------
// Plain move kernels for the API calls that only move (movePoints without a step).
__global__ void k_move_only(int V, const unsigned char* fix, const float2* src, float2* dst, const float2* d,
                            const float* dt, const float2* vel, int mode) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  float2 p = src[v];
  if (!fix[v]) {
    if (mode == MOVE_DISPLACE) {
      p.x = fadd(p.x, d[v].x);
      p.y = fadd(p.y, d[v].y);
    } else {
      p.x = fadd(p.x, fmul(vel[v].x, dt[v]));
      p.y = fadd(p.y, fmul(vel[v].y, dt[v]));
    }
  }
  dst[v] = p;
}

extern "C" {

const char* mcl_status_string(int status) {
  switch (status) {
    case MCL_OK: return "ok";
    case MCL_ERR_INVALID_ARGUMENT: return "invalid argument";
    case MCL_ERR_CUDA: return "CUDA error";
    case MCL_ERR_OUT_OF_MEMORY: return "out of device memory";
    case MCL_ERR_NO_CONVERGENCE: return "iteration cap reached";
    case MCL_ERR_CAPACITY: return "buffer capacity exceeded";
    case MCL_ERR_DEGENERATE_INPUT: return "degenerate input (duplicate point, point outside the bounding square, or invalid mesh)";
    case MCL_ERR_PREDICATE: return "exact predicate capacity exceeded";
    case MCL_ERR_NO_DEVICE: return "no CUDA device";
    default: return "unknown status";
  }
}

const char* mcl_last_error(void) { return mcl::g_last_error.c_str(); }
int mcl_version(void) { return 1; }

int mcl_mesh_totals(mcl_mesh* m, mcl_step_stats* totals, int64_t* calls) {
  if (!m || !totals) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost));
  const DevState& t = *m->st_host;
  fill_stats_from(t.tot, t.last_status, t.last_site, totals);
  totals->failed_launches = (int64_t)t.failed;
  if (calls) *calls = (int64_t)t.calls;
  return MCL_OK;
}

int mcl_debug_timeline(mcl_mesh* m, int64_t* out48) {
  if (!m || !out48) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost));
  for (int i = 0; i < kTimeline; ++i) out48[i] = (int64_t)m->st_host->ts[i];
  return MCL_OK;
}

int mcl_debug_insert_timeline(mcl_mesh* m, int64_t* out64) {
  if (!m || !out64) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost));
  for (int i = 0; i < 64; ++i) out64[i] = (int64_t)m->st_host->ts_insert[i];
  return MCL_OK;
}

int mcl_debug_remove_timeline(mcl_mesh* m, int64_t* out64) {
  if (!m || !out64) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost));
  for (int i = 0; i < 64; ++i) out64[i] = (int64_t)m->st_host->ts_remove[i];
  for (int i = 0; i < 16; ++i) {
    out64[64 + i] = (int64_t)m->st_host->rm_slow[i];
    out64[80 + i] = (int64_t)m->st_host->rm_uncached[i];
  }
  // the next launches accumulate from zero
  static_assert(offsetof(DevState, rm_uncached) == offsetof(DevState, rm_slow) + 16 * 8, "layout");
  unsigned long long zero[32] = {};
  CK(cudaMemcpy(reinterpret_cast<char*>(m->st) + offsetof(DevState, rm_slow), zero, sizeof(zero),
                cudaMemcpyHostToDevice));
  return MCL_OK;
}

int mcl_debug_counters(mcl_mesh* m, int64_t* out, int n) {
  if (!m || !out || n < 1) return fail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost));
  for (int i = 0; i < n && i < C_COUNT; ++i) out[i] = (int64_t)m->st_host->last[i];
  return C_COUNT;
}

int mcl_debug_state(mcl_mesh* m, int32_t* out68) {
  if (!m || !out68) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  CK(cudaMemcpy(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost));
  for (int i = 0; i < 68; ++i) out68[i] = m->st_host->dbg[i];
  return MCL_OK;
}

int mcl_mesh_validate(mcl_mesh* m, int64_t* counts8) {
  if (!m || !counts8) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  KParams P = make_params(m, ENGINE_STEP);
  P.pos = m->pos[m->cur];
  P.pos_old = P.pos;
  CK(cudaMemset(m->scratch, 0, 64));
  k_validate<<<1024, 256>>>(P, m->scratch);
  CK(cudaGetLastError());
  unsigned long long h[8];
  CK(cudaMemcpy(h, m->scratch, 64, cudaMemcpyDeviceToHost));
  for (int i = 0; i < 8; ++i) counts8[i] = (int64_t)h[i];
  return MCL_OK;
}

int mcl_mesh_create_from_aos(const mcl_aos_view* a, mcl_mesh** out) {
  if (!a || !out || !a->pos || !a->v || !a->he) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  std::vector<int4> ev, en;
  std::vector<int> vhe;
  std::string why;
  if (!aos_to_soa(a, ev, en, vhe, why)) return fail(MCL_ERR_INVALID_ARGUMENT, "malformed mesh: " + why);
  mcl_mesh* m = nullptr;
  int rc = alloc_mesh(a->V, a->HE / 2, &m);
  if (rc != MCL_OK) return rc;
  rc = upload_soa(m, a->pos, ev, en, vhe);
  if (rc != MCL_OK) { free_mesh(m); return rc; }
  m->delaunay = false;  // a caller's mesh: the first step classifies every edge
  m->square = has_square(a);
  *out = m;
  return MCL_OK;
}

int mcl_mesh_upload_aos(mcl_mesh* m, const mcl_aos_view* a) {
  if (!m || !a) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  if (a->V != m->V || a->HE != 2 * m->E) return fail(MCL_ERR_INVALID_ARGUMENT, "size mismatch");
  std::vector<int4> ev, en;
  std::vector<int> vhe;
  std::string why;
  if (!aos_to_soa(a, ev, en, vhe, why)) return fail(MCL_ERR_INVALID_ARGUMENT, "malformed mesh: " + why);
  m->delaunay = false;
  m->square = has_square(a);
  return upload_soa(m, a->pos, ev, en, vhe);
}

int mcl_mesh_destroy(mcl_mesh* m) {
  if (!m) return MCL_OK;
  cudaDeviceSynchronize();
  free_mesh(m);
  return MCL_OK;
}

int mcl_mesh_sizes(const mcl_mesh* m, int64_t* V, int64_t* HE, int64_t* T) {
  if (!m) return fail(MCL_ERR_INVALID_ARGUMENT, "null mesh");
  if (V) *V = m->V;
  if (HE) *HE = 2 * m->E;
  if (T) *T = m->T;
  return MCL_OK;
}

int mcl_mesh_positions(mcl_mesh* m, mcl_float2** pos_dev) {
  if (!m || !pos_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  *pos_dev = reinterpret_cast<mcl_float2*>(m->pos[m->cur]);
  return MCL_OK;
}

int mcl_mesh_copy_positions(mcl_mesh* m, mcl_float2* dst, int to_host, void* stream) {
  if (!m || !dst) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  CK(cudaMemcpyAsync(dst, m->pos[m->cur], 8 * m->V, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice,
                     (cudaStream_t)stream));
  if (to_host) CK(cudaStreamSynchronize((cudaStream_t)stream));
  return MCL_OK;
}

int mcl_mesh_download_aos(mcl_mesh* m, mcl_float2* pos, int32_t* v, int32_t* he, int32_t* t) {
  if (!m) return fail(MCL_ERR_INVALID_ARGUMENT, "null mesh");
  return download_range(m, 0, m->V, 0, m->E, m->T, pos, v, he, t);
}

int mcl_move(mcl_mesh* m, const mcl_float2* d_dev, void* stream) {
  if (!m || !d_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  if (m->nact) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_move: a subset of the batch is active (use mcl_step)");
  if (m->dirty) std::memset(m->dirty, 1, (size_t)m->ncomp);
  cudaStream_t s = (cudaStream_t)stream;
  const int src = m->cur, dst = m->valid_cur ? m->cur ^ 1 : m->cur;
  k_move_only<<<(unsigned)((m->V + 255) / 256), 256, 0, s>>>((int)m->V, m->vfix, m->pos[src], m->pos[dst],
                                                              (const float2*)d_dev, nullptr, nullptr, MOVE_DISPLACE);
  CK(cudaGetLastError());
  m->cur = dst;
  m->valid_cur = false;
  return MCL_OK;
}

int mcl_integrate(mcl_mesh* m, const float* dt_dev, const mcl_float2* v_dev, void* stream) {
  if (!m || !dt_dev || !v_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  if (m->nact) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_integrate: a subset of the batch is active (use mcl_step)");
  if (m->dirty) std::memset(m->dirty, 1, (size_t)m->ncomp);
  cudaStream_t s = (cudaStream_t)stream;
  const int src = m->cur, dst = m->valid_cur ? m->cur ^ 1 : m->cur;
  k_move_only<<<(unsigned)((m->V + 255) / 256), 256, 0, s>>>((int)m->V, m->vfix, m->pos[src], m->pos[dst], nullptr,
                                                              dt_dev, (const float2*)v_dev, MOVE_INTEGRATE);
  CK(cudaGetLastError());
  m->cur = dst;
  m->valid_cur = false;
  return MCL_OK;
}

int mcl_untangle(mcl_mesh* m, void* stream, mcl_step_stats* stats) {
  if (!m) return fail(MCL_ERR_INVALID_ARGUMENT, "null mesh");
  return run_step(m, MOVE_NONE, nullptr, (cudaStream_t)stream, stats);
}

int mcl_delaunay_restore(mcl_mesh* m, void* stream, mcl_step_stats* stats) {
  if (!m) return fail(MCL_ERR_INVALID_ARGUMENT, "null mesh");
  return run_step(m, MOVE_NONE, nullptr, (cudaStream_t)stream, stats);
}

int mcl_step(mcl_mesh* m, const mcl_float2* d_dev, void* stream, mcl_step_stats* stats) {
  if (!m || !d_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  if (!m->valid_cur) {
    int rc = mcl_move(m, d_dev, stream);
    if (rc != MCL_OK) return rc;
    return run_step(m, MOVE_NONE, nullptr, (cudaStream_t)stream, stats);
  }
  return run_step(m, MOVE_DISPLACE, (const float2*)d_dev, (cudaStream_t)stream, stats);
}

int mcl_step_host(mcl_mesh* m, const mcl_float2* d_host, void* stream, mcl_step_stats* stats) {
  if (!m || !d_host) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  cudaStream_t s = (cudaStream_t)stream;
  CK(cudaMemcpyAsync(m->dstage, d_host, 8 * m->V, cudaMemcpyHostToDevice, s));
  return mcl_step(m, reinterpret_cast<const mcl_float2*>(m->dstage), stream, stats);
}

}  // extern "C"

namespace mcl {
// the counters of the last launch as an mcl_step_stats, in device memory
__global__ void k_publish_stats(const DevState* st, mcl_step_stats* out) {
  if (threadIdx.x != 0) return;
  unsigned long long c[C_COUNT];
  for (int i = 0; i < C_COUNT; ++i) c[i] = st->last[i];
  publish_counts(c, st->last_status, st->last_site, out);
}
}  // namespace mcl

extern "C" {

int mcl_step_host_async(mcl_mesh* m, const mcl_float2* d_host, void* stream, mcl_step_stats* stats_pinned) {
  if (!m || !d_host) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  if (!m->valid_cur || m->nact) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_step_host_async: needs a validated mesh "
                                                                      "and every mesh of a batch active");
  cudaStream_t s = (cudaStream_t)stream;
  if (!m->copy_stream) {
    CK(cudaMalloc((void**)&m->dstage2, 8 * m->V));
    CK(cudaMalloc((void**)&m->stats_dev, 2 * sizeof(mcl_step_stats)));
    CK(cudaStreamCreateWithFlags(&m->copy_stream, cudaStreamNonBlocking));
    for (int i = 0; i < 2; ++i) {
      CK(cudaEventCreateWithFlags(&m->ev_copied[i], cudaEventDisableTiming));
      CK(cudaEventCreateWithFlags(&m->ev_used[i], cudaEventDisableTiming));
      CK(cudaEventRecord(m->ev_used[i], m->copy_stream));
    }
  }
  const int k = m->stage_idx;
  m->stage_idx ^= 1;
  float2* buf = k ? m->dstage2 : m->dstage;
  // the copy into buffer k waits for the step that last read it, then runs on
  // the copy stream, overlapping the step in flight on `stream`
  CK(cudaStreamWaitEvent(m->copy_stream, m->ev_used[k], 0));
  CK(cudaMemcpyAsync(buf, d_host, 8 * m->V, cudaMemcpyHostToDevice, m->copy_stream));
  CK(cudaEventRecord(m->ev_copied[k], m->copy_stream));
  CK(cudaStreamWaitEvent(s, m->ev_copied[k], 0));
  // a pinned record the device can address is filled by the step itself
  // (no publishing kernel and copy between steps); otherwise it is copied
  mcl_step_stats* mapped = nullptr;
  if (stats_pinned && cudaHostGetDevicePointer((void**)&mapped, stats_pinned, 0) != cudaSuccess) {
    (void)cudaGetLastError();
    mapped = nullptr;
  }
  const int rc = run_step(m, MOVE_DISPLACE, buf, s, nullptr, mapped);
  if (rc != MCL_OK) return rc;
  CK(cudaEventRecord(m->ev_used[k], s));
  if (stats_pinned && !mapped) {
    k_publish_stats<<<1, 32, 0, s>>>(m->st, m->stats_dev + k);
    CK(cudaMemcpyAsync(stats_pinned, m->stats_dev + k, sizeof(mcl_step_stats), cudaMemcpyDeviceToHost, s));
  }
  return MCL_OK;
}

int mcl_mesh_last_status(mcl_mesh* m, void* stream, mcl_step_stats* stats) {
  if (!m) return fail(MCL_ERR_INVALID_ARGUMENT, "null mesh");
  mcl_step_stats tmp;
  return finish(m, (cudaStream_t)stream, stats ? stats : &tmp);
}

// HostTriangulation::addDelaunayPoints on the GPU: Morton sort with the reference's
// comparator (include/Host_Triangulation.h:287-300), then the triangulation.  Distinct
// keys are sorted on the device; where keys are equal std::sort decides, as in the
// reference: on records with their keys (the same comparisons, so the same order; three
// times as fast as working out both keys in each comparison).
int mcl_mesh_build(mcl_float2* pts, int64_t n, mcl_mesh** out) {
  if (!pts || !out || n < 0) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  const float lo = -kSquare, hi = kSquare;
  bool inside = true;
  for (int64_t i = 0; i < n; ++i) inside &= pts[i].x > lo && pts[i].x < hi && pts[i].y > lo && pts[i].y < hi;
  if (!inside) return fail(MCL_ERR_DEGENERATE_INPUT, "point outside the bounding square");
  const int64_t V = n + 4, E = 5 + 3 * n;
  mcl_mesh* m = nullptr;
  int rc = alloc_mesh(V, E, &m);
  if (rc != MCL_OK) return rc;
  m->square = true;
  KParams P = make_params(m, ENGINE_BUILD);
  P.pos = m->pos[0];
  P.pos_old = m->pos[0];
  // the mesh's arrays are not in use yet: the records fit the edges', the digit counts
  // the stars'
  SortArgs A;
  A.in = m->dstage;
  A.rec[0] = reinterpret_cast<ulonglong2*>(m->ev);
  A.rec[1] = reinterpret_cast<ulonglong2*>(m->en);
  A.hist = m->star;
  A.out[0] = m->pos[0];
  A.out[1] = m->pos[1];
  A.key = P.skey;
  A.st = m->st;
  A.n = (int)n;
  const int blocks = (int)std::min<int64_t>(3 * m->nsm, std::max<int64_t>(1, (n + kThreads - 1) / kThreads));
  int sorted = 0;
  void* sort_args[] = {&A};
  void* args[] = {&P, &sorted};
  cudaError_t e = cudaMemsetAsync(m->vfix, 0, V, 0);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->vfix, 1, 4, 0);
  if (e == cudaSuccess && n) e = cudaMemcpyAsync(m->dstage, pts, 8 * n, cudaMemcpyHostToDevice, 0);
  if (e == cudaSuccess) e = cudaLaunchCooperativeKernel((void*)k_sort_points, dim3(blocks), dim3(kThreads), sort_args, 0, 0);
  auto launch = [&] {
    if (e == cudaSuccess)
      e = cudaLaunchCooperativeKernel((void*)k_build, dim3(m->repair_blocks), dim3(m->coop_threads), args, 0, 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(m->st_host, m->st, sizeof(DevState), cudaMemcpyDeviceToHost, 0);
  };
  launch();
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  if (e == cudaSuccess && m->st_host->sort_ties) {
    struct Keyed {
      unsigned long long key;
      mcl_float2 p;
    };
    std::vector<Keyed> v((size_t)n);
    for (int64_t i = 0; i < n; ++i) v[(size_t)i] = {morton_key(pts[i].x, pts[i].y), pts[i]};
    std::sort(v.begin(), v.end(), [](const Keyed& a, const Keyed& b) { return a.key < b.key; });
    for (int64_t i = 0; i < n; ++i) pts[i] = v[(size_t)i].p;
    for (int k = 0; k < 2 && e == cudaSuccess; ++k)
      e = cudaMemcpyAsync(m->pos[k] + 4, pts, 8 * n, cudaMemcpyHostToDevice, 0);
    sorted = 1;
    launch();
  } else if (e == cudaSuccess && n) {
    e = cudaMemcpyAsync(pts, m->pos[0] + 4, 8 * n, cudaMemcpyDeviceToHost, 0);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  if (e != cudaSuccess) { free_mesh(m); return cuda_fail(e, "build"); }
  if (m->st_host->last_status != MCL_OK) {
    const int st = m->st_host->last_status;
    free_mesh(m);
    return fail(st, std::string("build failed: ") + mcl_status_string(st));
  }
  *out = m;
  return MCL_OK;
}

}  // extern "C"
