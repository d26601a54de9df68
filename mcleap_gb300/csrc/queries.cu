// Neighbourhood queries on the device mesh and the uniform grid, plus the
// predicate diagnostics entry points.
//
//   one-ring      DeviceTriangulation::oneRing / oneRing2   (include/kernels.cuh:54-121)
//   closest       DeviceTriangulation::closestNeighbors[2]  (include/kernels.cuh:129-165)
//   mesh FRNN     DeviceTriangulation::getFRNN / getFRNN2   (include/kernels.cuh:169-272)
//   grid          GridCount2d (include/gridCount2d.h): counting sort of points
//                 into row-major cells, stable inside a cell,
//                 then fixed-radius queries over the (2w+1)^2 cell stencil.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "engine.cuh"

using namespace mcl;

namespace {

int qfail(int code, const std::string& msg) {
  mcl_set_last_error(msg);
  return code;
}

#define QCK(call)                                                                       \
  do {                                                                                  \
    cudaError_t _e = (call);                                                            \
    if (_e != cudaSuccess) return qfail(MCL_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
  } while (0)

// Reference squared distance, include/kernels.cuh:125-127: no FMA contraction.
__device__ __forceinline__ float sqdist(float2 a, float2 b) {
  const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y);
  return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
}

struct MeshView {
  const int4* ev;
  const int4* en;
  const int* vhe;
  const float2* pos;
  int V, E;
};

__device__ __forceinline__ int mv_origin(const MeshView& M, int h) {
  return __ldg(reinterpret_cast<const int*>(M.ev) + 4 * (h >> 1) + (h & 1));
}
__device__ __forceinline__ int mv_next(const MeshView& M, int h) {
  return __ldg(reinterpret_cast<const int*>(M.en) + 4 * (h >> 1) + 2 * (h & 1));
}
__device__ __forceinline__ int mv_prev(const MeshView& M, int h) {
  return __ldg(reinterpret_cast<const int*>(M.en) + 4 * (h >> 1) + 2 * (h & 1) + 1);
}
// The reference's PREV_OUTGOING(h) = next(twin(h)): the next outgoing half-edge
// clockwise around the origin (include/kernels.cuh:52).
__device__ __forceinline__ int mv_rot(const MeshView& M, int h) { return mv_next(M, h ^ 1); }

constexpr int kMaxDeg = 4096;

// ---------------------------------------------------------------------------
// A count that the host waits for (truncated rings, overflowing lists): the
// kernel adds to cell[0], and its last block writes the sum to pinned host memory
// and leaves the cell at zero for the next call, so that a query is one launch and
// one wait (a memset before and a copy after it cost a small query as much as the
// kernel).  cell[1] counts the blocks that have finished; the cell is the call's own
// while it is in flight (CountSlot).  Each thread says whether its own query counts, a
// block adds once (500,000 rows all cut off and added one by one: 350 us).  A call that
// asks for no count passes no cell.
// count_add: of a kernel that another one of the same call follows.
__device__ __forceinline__ void count_add(bool mine, unsigned long long* cell) {
  const int all = __syncthreads_count(mine);
  if (threadIdx.x == 0 && all) atomicAdd(cell, (unsigned long long)all);
}
__device__ __forceinline__ void count_done(bool mine, unsigned long long* cell, unsigned long long* host) {
  count_add(mine, cell);
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(cell + 1, 1ull) == gridDim.x - 1) {
      __threadfence();
      *host = atomicExch(cell, 0ull);
      cell[1] = 0;
    }
  }
}

// One-ring, one thread per vertex.  What bounds it is the chain of dependent
// record reads, so the ring is walked both ways at once: the record of a spoke links
// to both its neighbours, and a ring of six closes after three links.  The record
// of spoke k holds its own end and, as the apexes of its two faces, the ends of
// spokes k - 1 and k + 1, so the ends are read at every other spoke.  Rings of up to
// 15 spokes are kept in shared memory, then written starting at the smallest
// neighbour; a row layout is written by four lanes per row, four words each (a thread
// per row wrote seven words of 32 rows apart).  Longer rings and the rings
// of the corners (next to the outside, which has no apex) are walked spoke by spoke.
//
// A corner's ring can have hundreds of spokes when points sit on the sides of their
// box.  Its smallest neighbour is one of the two corners beside it (corners have
// the smallest ids of their mesh, and in a Delaunay mesh with a point no corner
// meets the one across), next to each other around the outside: its ring is written
// from there at once, and no further than the row.
//
// GB300, before (both records of every spoke in turn, corners walked whole) -> now:
// 1M points advected, column layout 50.9 -> 45 us (107 MB read); 500,000 points, row
// layout 49.2 -> 36.0 us; the precision-stress set of 500,000 after random walks
// (corners with long rings) 50.8 -> 24.0 us; 96 meshes of 1.4M points 83 -> 57 us.
constexpr int kRegRing = 16;
constexpr int kRingThreads = 128;

// Writes the row; returns whether it was cut off.
__device__ __noinline__ bool ring_walk(const MeshView M, int h0, int cap, size_t stride, int* row, bool corner_first) {
  int start = h0, best = mv_origin(M, h0 ^ 1), deg = 1, h = h0;
  if (corner_first) {
    const int h1 = mv_rot(M, h0);
    start = h = best < mv_origin(M, h1 ^ 1) ? h0 : h1;
    deg = 0;
    do {
      row[(size_t)(deg + 1) * stride] = mv_origin(M, h ^ 1);
      h = mv_rot(M, h);
      ++deg;
    } while (h != start && deg < cap);
    if (deg > 3 || h != start) {  // (a square with no point has its diagonal)
      row[0] = deg;
      return h != start;
    }
    start = h0;
    deg = 1;
  }
  // the smallest neighbour, both ways at once (a hub of 1,000 spokes:
  // 265 us one way, 195)
  int back = h = h0;
  bool closed = false;
  auto look = [&](int s) {
    const int w = mv_origin(M, s ^ 1);
    if (w < best) { best = w; start = s; }
    ++deg;
  };
  while (deg < kMaxDeg) {
    const int f = mv_rot(M, h), r = mv_prev(M, back) ^ 1;
    closed = f == back;
    if (closed) break;
    look(f);
    closed = f == r;
    if (closed) break;
    look(r);
    h = f;
    back = r;
  }
  if (!closed) {  // the first kMaxDeg of the walk stand for a ring that is longer
    start = h = h0;
    best = mv_origin(M, h0 ^ 1);
    for (deg = 1; deg < kMaxDeg && (h = mv_rot(M, h)) != h0;) look(h);
  }
  const int cnt = deg < cap ? deg : cap;
  h = start;
  for (int k = 0; k < cnt; ++k) {
    row[(size_t)(k + 1) * stride] = mv_origin(M, h ^ 1);
    h = mv_rot(M, h);
  }
  row[0] = cnt;
  return deg > cap;
}

// Rows for the vertices verts[0 .. n) (NULL: all of them).  delaunay: the mesh is the
// Delaunay triangulation of its square; vfix marks the corners.
template <bool kRow>
__global__ void __launch_bounds__(kRingThreads) k_one_ring(MeshView M, const int* __restrict__ verts, int n,
                                                           int max_ring, int* ring,
                                                           const unsigned char* __restrict__ vfix, int delaunay,
                                                           unsigned long long* cell, unsigned long long* host) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int i = q < n ? (verts ? __ldg(verts + q) : q) : -1;
  const int h0 = i >= 0 && i < M.V ? __ldg(M.vhe + i) : -1;
  const int cap = max_ring - 1;
  const size_t stride = kRow ? 1 : (size_t)n;
  int* row = kRow ? ring + (size_t)q * max_ring : ring + q;
  if (verts && q < n && h0 < 0) row[0] = 0;
  // neighbour k of the walk (negative: the other way) in slot k mod kRegRing, one
  // column per thread (conflict-free)
  __shared__ int sring[kRegRing][kRingThreads];
  int deg = 0, at = 0;
  bool done = h0 < 0, cut = false;
  if (!done) {
    int* col = &sring[0][threadIdx.x];
    int best = 0x7fffffff;
    bool plain = true;
    auto keep = [&](int k, int w) {
      plain = plain && w >= 0;
      col[(k & (kRegRing - 1)) * kRingThreads] = w;
      if (w < best) { best = w; at = k; }
    };
    const int4 n0 = __ldg(M.en + (h0 >> 1)), e0 = __ldg(M.ev + (h0 >> 1));
    int a = (h0 & 1) ? n0.x : n0.z, b = ((h0 & 1) ? n0.w : n0.y) ^ 1;  // spokes 1 and -1
    keep(0, (h0 & 1) ? e0.x : e0.y);
    keep(1, (h0 & 1) ? e0.z : e0.w);
    keep(-1, (h0 & 1) ? e0.w : e0.z);
    for (int k = 1; plain && k < kRegRing / 2; ++k) {
      // spokes k and -k; the records of the even ones hold the ends around them
      if (k & 1) {
        if (a == b) { deg = 2 * k; break; }
      }
      const int4 na = __ldg(M.en + (a >> 1)), nb = __ldg(M.en + (b >> 1));
      if (!(k & 1)) {
        const int4 ea = __ldg(M.ev + (a >> 1)), eb = __ldg(M.ev + (b >> 1));
        keep(k, (a & 1) ? ea.x : ea.y);
        if (a == b) { deg = 2 * k; break; }
        keep(-k, (b & 1) ? eb.x : eb.y);
        if (k + 1 < kRegRing / 2) {
          keep(k + 1, (a & 1) ? ea.z : ea.w);
          keep(-k - 1, (b & 1) ? eb.w : eb.z);
        }
      }
      const int a1 = (a & 1) ? na.x : na.z;
      if (a1 == b) { deg = 2 * k + 1; break; }
      a = a1;
      b = ((b & 1) ? nb.w : nb.y) ^ 1;
      plain = plain && a >= 0 && b >= 0;
    }
    if (!plain || !deg) {
      bool corners = false;
      if (delaunay && vfix[i]) {
        const int c = mv_origin(M, h0 ^ 1), d = mv_origin(M, mv_rot(M, h0) ^ 1);
        corners = vfix[c] && vfix[d];
      }
      cut = ring_walk(M, h0, cap, stride, row, corners);
      done = true;
    } else {
      cut = deg > cap;
    }
  }
  if (kRow) {
    __syncwarp();
    // eight rows a turn, four lanes each, four words a lane (one store where the row
    // lies on 16 bytes and all four are written: slots past the ring stay as they are)
    const int j = 4 * (lane & 3), first = q - lane;
    const bool vec = ((max_ring & 3) | (int)((size_t)ring & 15)) == 0;
    for (int r = 0; r < 32; r += 8) {
      const int src = r + (lane >> 2);
      const int d = __shfl_sync(0xffffffffu, deg, src), a = __shfl_sync(0xffffffffu, at, src);
      const bool skip = __shfl_sync(0xffffffffu, (int)done, src) != 0;
      const int c = min(d, cap);
      if (skip || j > c) continue;
      int x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // entry j + k - 1 from the smallest: the ring index in -(d - 1) / 2 .. d / 2
        int o = a + j + k - 1;
        if (o > d / 2) o -= d;
        x[k] = j + k == 0 ? c : sring[o & (kRegRing - 1)][(threadIdx.x & ~31) + src];
      }
      int* to = ring + (size_t)(first + src) * max_ring + j;
      if (vec && j + 3 <= c) {
        *reinterpret_cast<int4*>(to) = make_int4(x[0], x[1], x[2], x[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (j + k <= c) to[k] = x[k];
      }
    }
  } else if (!done) {
    const int c = min(deg, cap);
    int o = at;
    for (int k = 0; k < c; ++k) {
      row[(size_t)(k + 1) * stride] = sring[o & (kRegRing - 1)][threadIdx.x];
      if (++o > deg / 2) o -= deg;
    }
    row[0] = c;
  }
  if (host) count_done(cut, cell, host);
}

// Nearest entry of each ring row.  kVec: rows are read four words at a time (row
// layout, rows on 16 bytes: two loads for the usual ring instead of eight, each a
// tag lookup per lane; 500,000 rows 22.1 -> 14.4 us).
template <bool kVec>
__global__ void k_closest(const float2* pos, int V, int layout, int max_ring, const int* ring, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V) return;
  const float2 p = pos[i];
  int best = -1;
  float bd = 0.f;
  auto look = [&](int j) {
    const float d = sqdist(p, pos[j]);
    if (best < 0 || d < bd || (d == bd && j < best)) { best = j; bd = d; }
  };
  if (kVec) {
    const int4* row = reinterpret_cast<const int4*>(ring + (size_t)i * max_ring);
    const int4 a = row[0];
    const int cnt = a.x;
    if (cnt > 0) look(a.y);
    if (cnt > 1) look(a.z);
    if (cnt > 2) look(a.w);
    for (int k = 3; k < cnt; k += 4) {
      const int4 b = row[(k + 1) >> 2];
      look(b.x);
      if (cnt > k + 1) look(b.y);
      if (cnt > k + 2) look(b.z);
      if (cnt > k + 3) look(b.w);
    }
  } else {
    const int cnt = layout == MCL_LAYOUT_COLUMN ? ring[i] : ring[(size_t)i * max_ring];
    for (int k = 0; k < cnt; ++k)
      look(layout == MCL_LAYOUT_COLUMN ? ring[(size_t)(k + 1) * V + i] : ring[(size_t)i * max_ring + k + 1]);
  }
  out[i] = best;
}

// Mesh FRNN: search over the mesh from i through vertices within r (the
// reference's getFRNN, include/Host_Triangulation.h:525-560 and
// include/kernels.cuh:169-219); the found set is written sorted ascending.
constexpr int kFrnnLocal = 256;

// One thread's search, in the order found, for sets that a part's lists do not hold:
// up to kFrnnLocal vertices, in a thread-local list.  Writes the row; returns whether it
// or the list was too short.
__device__ __noinline__ bool frnn_serial(const MeshView M, int i, float r2, int cap, size_t stride, int* row) {
  int found[kFrnnLocal];
  int nf = 0;
  int top = 0;  // found[top..nf): vertices whose rings are still to scan
  bool over = false;
  const float2 pi = M.pos[i];
  int cur = i;
  for (int guard = 0; guard < (1 << 20); ++guard) {
    const int h0 = __ldg(M.vhe + cur);
    if (h0 >= 0) {
      int h = h0, deg = 0;
      do {
        const int w = mv_origin(M, h ^ 1);
        if (w != i) {
          bool seen = sqdist(pi, M.pos[w]) > r2;
          for (int k = 0; k < nf && !seen; ++k) seen = found[k] == w;
          if (!seen) {
            if (nf < kFrnnLocal) found[nf++] = w;
            else over = true;
          }
        }
        h = mv_rot(M, h);
        ++deg;
      } while (h != h0 && deg < kMaxDeg);
    }
    if (top >= nf) break;
    cur = found[top++];
  }
  for (int a = 1; a < nf; ++a) {
    const int x = found[a];
    int b = a - 1;
    while (b >= 0 && found[b] > x) { found[b + 1] = found[b]; --b; }
    found[b + 1] = x;
  }
  const int cnt = nf < cap ? nf : cap;
  for (int k = 0; k < cnt; ++k) row[(size_t)(k + 1) * stride] = found[k];
  row[0] = cnt;
  return over || nf > cap;
}

// The search of kLanes lanes (half a warp), breadth first: two lanes walk the ring of one
// vertex of the frontier from its first spoke, one each way, until they meet; a lane's
// neighbour within r joins through a hash set in shared memory.  The search is a chain of
// dependent loads, so the time is the number of steps one after another: about
// four a level for a ring of six, three or four levels for r = 2 x spacing, where a
// thread alone takes a step for each of some eighty spokes and looks each up in its
// own list in local memory.  With a warp to a query 13 of its lanes had work and it was
// bound by instruction issue (2600 a query); a frontier is seldom wider than the eight
// vertices that half a warp takes at once.  60,000 queries, r = 2 x spacing, GB300:
// 567 us by threads, 168 us by warps; the served list 163 us by warps, 120 by half warps
// (127 by quarters).
constexpr int kFrnnWarps = 4;
constexpr int kFrnnFound = 64;
constexpr int kFrnnHash = 128;

// All parts of a warp call it together; a part with no query has i = -1.  Returns
// false in a part that found more than its list holds.
template <int kLanes>
__device__ __forceinline__ bool part_search(const MeshView& M, int i, float r2, int* found, int* hash, int* count) {
  const int lane = threadIdx.x & 31, sub = lane & (kLanes - 1), way = lane & 1;
  const unsigned part = ((1u << kLanes) - 1u) << (lane - sub), lt = part & ((1u << lane) - 1u);
#pragma unroll
  for (int k = 0; k < kFrnnHash / kLanes; ++k) hash[kLanes * k + sub] = -1;
  __syncwarp();
  bool live = i >= 0, fits = true;
  const float2 pi = live ? M.pos[i] : make_float2(0.f, 0.f);
  int nf = 0, lo = -1;  // the frontier: i, then found[lo .. hi)
  while (__any_sync(0xffffffffu, live && lo < nf)) {
    const int hi = lo < 0 ? 0 : nf;
    for (int c = lo; __any_sync(0xffffffffu, live && c < hi); c += kLanes / 2) {
      const int j = c + (sub >> 1);
      const int u = !live || c >= hi ? -1 : (lo < 0 ? (j == lo ? i : -1) : (j < hi ? found[j] : -1));
      const int h0 = u >= 0 ? __ldg(M.vhe + u) : -1;
      bool on = h0 >= 0;
      int cur = h0;
      if (on && way) {
        cur = mv_prev(M, h0) ^ 1;
        on = cur != h0;  // a ring of one spoke is the other lane's
      }
      bool last = !__shfl_xor_sync(0xffffffffu, (int)on, 1);
      for (int step = 0; step < kMaxDeg && __any_sync(0xffffffffu, on); ++step) {
        int w = -1, nxt = -1;
        if (on) {
          w = mv_origin(M, cur ^ 1);
          nxt = way ? mv_prev(M, cur) ^ 1 : mv_rot(M, cur);
        }
        bool fresh = false;
        if (on && w != i && w >= 0 && sqdist(pi, M.pos[w]) <= r2) {
          unsigned k = ((unsigned)w * 2654435761u) >> 25;
          for (;;) {
            const int old = atomicCAS(hash + k, -1, w);
            fresh = old == -1;
            if (fresh || old == w) break;
            k = (k + 1) & (kFrnnHash - 1);
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, fresh) & part;
        if (fresh) {
          const int at = nf + __popc(m & lt);
          if (at < kFrnnFound) found[at] = w;
        }
        nf += __popc(m);
        const int ocur = __shfl_xor_sync(0xffffffffu, cur, 1), onxt = __shfl_xor_sync(0xffffffffu, nxt, 1);
        if (on) {
          if (last || nxt == ocur || nxt < 0) on = false;  // met, or the one between has been taken
          else if (nxt == onxt) {                          // one between: this way takes it
            last = true;
            if (way) on = false;
          }
          cur = nxt;
        }
        if (nf > kFrnnFound) on = live = fits = false;
      }
      __syncwarp();
    }
    lo = hi;
  }
  *count = nf;
  return fits;
}

// Rows for the vertices verts[0 .. n) (NULL: all of them), kLanes lanes each.  With
// rcomp the radius of vertex i is rcomp[vcomp[i]] (one radius per mesh of a batch; a
// plain mesh has vcomp == nullptr and one radius).
//
// Sets that the lists do not hold are one thread's work.  Up to kFrnnFew queries the
// part's first lane does it; of more they are left, marked by a count of kFrnnLeft, to
// k_mesh_frnn_left, a thread each: one lane in sixteen at work is bound by instruction
// issue (78 neighbours each: 200,000 queries 66 ms by first lanes, 9.9 by threads; 20,000:
// 8.4 and 2.5; 1,000: 1.1 and 2.8).
struct FrnnQuery {
  const int* verts;
  int n;
  float r2;
  int layout, max_frnn;
  int* out;
  const float* rcomp;
  const int* vcomp;

  __device__ __forceinline__ int vertex(const MeshView& M, int q) const {
    const int i = q < n ? (verts ? __ldg(verts + q) : q) : -1;
    return i >= M.V || (i >= 0 && __ldg(M.vhe + i) < 0) ? -1 : i;
  }
  __device__ __forceinline__ float radius2(int i) const {
    if (!rcomp || i < 0) return r2;
    const float rc = rcomp[vcomp ? vcomp[i] : 0];
    return __fmul_rn(rc, rc);
  }
  __device__ __forceinline__ int* row(int q) const {
    return layout == MCL_LAYOUT_COLUMN ? out + q : out + (size_t)q * max_frnn;
  }
  __device__ __forceinline__ size_t stride() const { return layout == MCL_LAYOUT_COLUMN ? (size_t)n : 1; }
};
constexpr int kFrnnFew = 2048;
constexpr int kFrnnLeft = -1;

template <int kLanes>
__global__ void __launch_bounds__(32 * kFrnnWarps) k_mesh_frnn(MeshView M, FrnnQuery Q, unsigned long long* cell,
                                                               unsigned long long* host) {
  constexpr int kPer = 32 / kLanes * kFrnnWarps;  // queries per block
  __shared__ int found_s[kPer][kFrnnFound];
  __shared__ int hash_s[kPer][kFrnnHash];
  const int sub = threadIdx.x & (kLanes - 1), slot = threadIdx.x / kLanes;
  const int q = blockIdx.x * kPer + slot, i = Q.vertex(M, q), cap = Q.max_frnn - 1;
  int* row = Q.row(q);
  const size_t stride = Q.stride();
  if (q < Q.n && i < 0 && sub == 0) row[0] = 0;
  const float r2 = Q.radius2(i);
  const int* found = found_s[slot];
  int nf = 0;
  const bool fits = part_search<kLanes>(M, i, r2, found_s[slot], hash_s[slot], &nf);
  bool cut = false;
  __syncwarp();
  if (i >= 0 && fits) {
    for (int k = sub; k < nf; k += kLanes) {
      const int x = found[k];
      int rank = 0;
      for (int j = 0; j < nf; ++j) rank += found[j] < x ? 1 : 0;
      if (rank < cap) row[(size_t)(rank + 1) * stride] = x;
    }
    if (sub == 0) {
      row[0] = nf < cap ? nf : cap;
      cut = nf > cap;
    }
  } else if (i >= 0 && sub == 0) {
    if (Q.n > kFrnnFew) row[0] = kFrnnLeft;
    else cut = frnn_serial(M, i, r2, cap, stride, row);
  }
  if (Q.n > kFrnnFew) {
    if (host) count_add(cut, cell);
  } else if (host) {
    count_done(cut, cell, host);
  }
}

// The same for more than kFrnnMany queries, whose time is the work: small sets are a
// thread's own (up to kFrnnThread found, in its column of shared memory, and no more than
// kFrnnRing of them beside i: more promise many), the others of the warp's 32 queries are
// taken by its parts of kLanes lanes, as many at a time as there are.  us by threads
// alone, by half warps alone, and by the form that the number of queries selects:
//   queries    r / spacing  threads  halves     now
//      60,000     0.3            42      44      44
//                 2             343      95      94
//     100,000     0.3            41      63      47
//                 2             442     135     125
//     200,000     0.3            43      98      43
//                 2             610     247     348
//                 5          10,770  66,300   9,860
//   1,000,000     0.3           104     475     119
//                 1             353     743     353
//                 2           1,755   1,173   1,394
//                 5          45,700     (*)  41,100
// (*) a lone lane in sixteen for sets of more than 64.
constexpr int kFrnnQuarters = 65536;  // quarter warps from here on, ...
constexpr int kFrnnMany = 100000;     // ... and threads first
constexpr int kFrnnThread = 12;
constexpr int kFrnnRing = 4;
template <int kLanes>
__global__ void __launch_bounds__(32 * kFrnnWarps) k_mesh_frnn_many(MeshView M, FrnnQuery Q, unsigned long long* cell,
                                                                    unsigned long long* host) {
  constexpr int kParts = 32 / kLanes;
  __shared__ int pool[kFrnnWarps][kParts * (kFrnnFound + kFrnnHash)];
  static_assert(kParts * (kFrnnFound + kFrnnHash) >= 32 * kFrnnThread, "the threads' columns fit the parts' lists");
  const int lane = threadIdx.x & 31, sub = lane & (kLanes - 1), part = lane / kLanes, cap = Q.max_frnn - 1;
  const int q = blockIdx.x * blockDim.x + threadIdx.x, q0 = q - lane;
  const int i = Q.vertex(M, q);
  const size_t stride = Q.stride();
  const float r2 = Q.radius2(i);
  int* mine = pool[threadIdx.x >> 5];
  int* col = mine + lane;
  int nf = 0, cut = 0;
  bool many = false;
  if (i >= 0) {
    const float2 pi = M.pos[i];
    int top = 0, cur = i;
    while (!many) {
      const int h0 = __ldg(M.vhe + cur);
      int h = h0, deg = 0;
      if (h0 >= 0) {
        do {
          const int w = mv_origin(M, h ^ 1);
          if (w != i && sqdist(pi, M.pos[w]) <= r2) {
            bool seen = false;
            for (int k = 0; k < nf && !seen; ++k) seen = col[32 * k] == w;
            if (!seen) {
              many = nf == (cur == i ? kFrnnRing : kFrnnThread);
              if (many) break;
              col[32 * nf++] = w;
            }
          }
          h = mv_rot(M, h);
          ++deg;
        } while (h != h0 && deg < kMaxDeg);
      }
      if (top >= nf) break;
      cur = col[32 * top++];
    }
  }
  if (q < Q.n && !many) {
    for (int a = 1; a < nf; ++a) {
      const int x = col[32 * a];
      int b = a - 1;
      while (b >= 0 && col[32 * b] > x) { col[32 * (b + 1)] = col[32 * b]; --b; }
      col[32 * (b + 1)] = x;
    }
    int* row = Q.row(q);
    const int cnt = nf < cap ? nf : cap;
    for (int k = 0; k < cnt; ++k) row[(size_t)(k + 1) * stride] = col[32 * k];
    row[0] = cnt;
    cut = nf > cap;
  }
  __syncwarp();
  int* found = mine + part * (kFrnnFound + kFrnnHash);
  for (unsigned todo = __ballot_sync(0xffffffffu, many); todo;) {
    unsigned rest = todo;
    for (int p = 0; p < part; ++p) rest &= rest - 1u;
    const int src = rest ? __ffs((int)rest) - 1 : lane;
    const int u = __shfl_sync(0xffffffffu, i, src);
    const float ru = __shfl_sync(0xffffffffu, r2, src);
    int got = 0;
    const bool fits = part_search<kLanes>(M, rest ? u : -1, ru, found, found + kFrnnFound, &got);
    __syncwarp();
    if (rest) {
      int* row = Q.row(q0 + src);
      if (fits) {
        for (int k = sub; k < got; k += kLanes) {
          const int x = found[k];
          int rank = 0;
          for (int j = 0; j < got; ++j) rank += found[j] < x ? 1 : 0;
          if (rank < cap) row[(size_t)(rank + 1) * stride] = x;
        }
      }
      if (sub == 0) {
        row[0] = !fits ? kFrnnLeft : (got < cap ? got : cap);
        cut += fits && got > cap ? 1 : 0;
      }
    }
    for (int p = 0; p < kParts; ++p) todo &= todo - 1u;
    __syncwarp();
  }
  if (!host) return;
  cut = __reduce_add_sync(0xffffffffu, cut);
  if (lane == 0 && cut) atomicAdd(cell, (unsigned long long)cut);
}

__global__ void __launch_bounds__(128) k_mesh_frnn_left(MeshView M, FrnnQuery Q, unsigned long long* cell,
                                                        unsigned long long* host) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  bool cut = false;
  if (q < Q.n) {
    int* row = Q.row(q);
    if (row[0] == kFrnnLeft) {
      const int i = Q.vertex(M, q);
      cut = frnn_serial(M, i, Q.radius2(i), Q.max_frnn - 1, Q.stride(), row);
    }
  }
  if (host) count_done(cut, cell, host);
}

// Diffusion-limited aggregation contact (the reference's check_if_close_diffusion,
// experiments/diffusion_limited_aggregation.cu:51-60, over mesh FRNN
// neighbours): a free walker freezes when a vertex frozen before this call
// lies within its mesh's radius.  Decisions read frozen_in only, so the result
// does not depend on thread order.
__global__ void k_dla_freeze(MeshView M, ActV A, const unsigned char* vfix, const float* rcomp, const int* vcomp,
                             const unsigned char* frozen_in, unsigned char* frozen_out,
                             unsigned long long* newly) {
  const int ii = blockIdx.x * blockDim.x + threadIdx.x;
  if (ii >= A.V_it) return;
  const int i = A.at(ii);
  unsigned char f = frozen_in[i];
  if (!f && !vfix[i] && __ldg(M.vhe + i) >= 0) {
    const float rc = rcomp[vcomp ? vcomp[i] : 0];
    const float r2 = __fmul_rn(rc, rc);
    int found[kFrnnLocal];
    int nf = 0, top = 0;
    const float2 pi = M.pos[i];
    int cur = i;
    for (int guard = 0; guard < (1 << 20) && !f; ++guard) {
      const int h0 = __ldg(M.vhe + cur);
      if (h0 >= 0) {
        int h = h0, deg = 0;
        do {
          const int w = mv_origin(M, h ^ 1);
          if (w != i) {
            bool seen = false;
            for (int k = 0; k < nf; ++k)
              if (found[k] == w) { seen = true; break; }
            if (!seen && sqdist(pi, M.pos[w]) <= r2) {
              if (frozen_in[w]) { f = 1; break; }
              if (nf < kFrnnLocal) found[nf++] = w;
            }
          }
          h = mv_rot(M, h);
          ++deg;
        } while (h != h0 && deg < kMaxDeg);
      }
      if (f || top >= nf) break;
      cur = found[top++];
    }
    if (f) atomicAdd(newly, 1ull);
  }
  frozen_out[i] = f;
}

// frozen[i] |= fnew[i] over the same vertices (second half of an in-place call)
__global__ void k_dla_commit(ActV A, unsigned char* frozen, const unsigned char* fnew) {
  const int ii = blockIdx.x * blockDim.x + threadIdx.x;
  if (ii >= A.V_it) return;
  const int i = A.at(ii);
  frozen[i] = fnew[i];
}

}  // namespace

// ---------------------------------------------------------------------------
// Grid.
struct mcl_grid {
  int64_t n;
  float minx, miny, cx, cy;
  int nx, ny;
  int flags;
  int morton;           // cells numbered along a Morton curve (else row-major)
  int mbits;            // Morton side = 1 << mbits
  int64_t ncells;       // size of the cell tables
  int* cell;            // per point: cell id (input order)
  int* count;           // per cell, then the out-of-domain flag and the scan's ticket
  int* start;           // per cell, then n
  int* local;           // per cell: start within its scan block
  int* bucket;          // per slot: input index, in arrival order
  int* perm;            // d_ind: sorted slot of input point i
  int* src;             // per sorted slot: input index
  float2* tmp;          // sorted positions / velocities scratch
  float2* tmp2;
  void* scan_tmp;
  size_t scan_tmp_bytes;
  int built;            // mcl_grid_build ran: tmp holds the sorted copy
};

namespace {

struct GridView {
  float minx, miny, cx, cy;
  int nx, ny, morton, periodic;
};

__device__ __forceinline__ int cell_coord(float p, float mn, float c, int n, int periodic, int* outside = nullptr) {
  float kf = floorf(__fdiv_rn(__fsub_rn(p, mn), c));
  kf = fminf(fmaxf(kf, -1.0e9f), 1.0e9f);  // also maps NaN to a border cell
  int k = (int)kf;
  if (outside && (k < 0 || k >= n)) *outside = 1;
  if (periodic) {
    k %= n;
    if (k < 0) k += n;
  } else {
    k = k < 0 ? 0 : (k >= n ? n - 1 : k);
  }
  return k;
}

__device__ __forceinline__ int cell_id(const GridView& G, int x, int y) {
  return y * G.nx + x;
}

// Points into cells, in the input's order within each cell.  Five launches: the counts
// cleared; every point's cell and its place in it by arrival; the scan of the counts;
// the points of each cell together in order of arrival; and a thread per point that
// counts the smaller indices of its cell, which gives its slot.  Nothing is sorted in
// place, so no lone thread orders a crowded cell.  Bound by launches below 100,000
// points and by scattered atomics and stores above (1,000,000 points, 2.4 per cell:
// 57 -> 48 us; a pass over 10,000 points takes 30 us
// less; the ten launches before had a scan in three, a copy of the starts as
// cursors with a second round of atomics, an insertion sort per cell and a gather).
constexpr int kScanThreads = 1024;
constexpr int kScanCells = 4 * kScanThreads;  // cells per block of the scan

// outside (may be NULL): set when a point's cell coordinate lies outside the
// grid before wrapping or clamping (the point is outside the domain).
__global__ void k_grid_hash(GridView G, int n, const float2* pos, int* cell, int* count, int* rank, int* outside) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float2 p = pos[i];
  int out = 0;
  const int c = cell_id(G, cell_coord(p.x, G.minx, G.cx, G.nx, G.periodic, &out),
                        cell_coord(p.y, G.miny, G.cy, G.ny, G.periodic, &out));
  cell[i] = c;
  rank[i] = atomicAdd(count + c, 1);
  if (out && outside) atomicOr(outside, 1);
}

// Exclusive scan of a value per thread of the block; the block's total in every thread.
__device__ __forceinline__ int scan_block(int x, int* total) {
  __shared__ int w[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += y;
  }
  __syncthreads();
  if (lane == 31) w[warp] = s;
  __syncthreads();
  int v = w[lane];  // kScanThreads / 32 of them
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  *total = __shfl_sync(0xffffffffu, v, 31);
  const int before = __shfl_sync(0xffffffffu, v, warp ? warp - 1 : 0);
  return s - x + (warp ? before : 0);
}

// local[c]: points in the block's cells before c.  The block that finishes last turns
// the blocks' totals into pre[b], the points in the blocks before b.
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(int64_t ncells, const int* count, int* local, int* pre,
                                                            int* ticket) {
  const int64_t c0 = (int64_t)blockIdx.x * kScanCells + 4 * threadIdx.x;
  int x[4], sum = 0, total;
  const bool whole = c0 + 4 <= ncells;  // the tables start on 16 bytes
  if (whole) {
    const int4 q = *reinterpret_cast<const int4*>(count + c0);
    x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
  } else {
    for (int k = 0; k < 4; ++k) x[k] = c0 + k < ncells ? count[c0 + k] : 0;
  }
  for (int k = 0; k < 4; ++k) sum += x[k];
  int at = scan_block(sum, &total);
  int y[4];
  for (int k = 0; k < 4; ++k) {
    y[k] = at;
    at += x[k];
  }
  if (whole) {
    *reinterpret_cast<int4*>(local + c0) = make_int4(y[0], y[1], y[2], y[3]);
  } else {
    for (int k = 0; k < 4; ++k)
      if (c0 + k < ncells) local[c0 + k] = y[k];
  }
  __shared__ bool last;
  if (threadIdx.x == 0) {
    pre[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  int carry = 0;
  for (int b = 0; b < (int)gridDim.x; b += kScanThreads) {
    const int i = b + threadIdx.x, v = i < (int)gridDim.x ? __ldcg(pre + i) : 0;
    const int before = scan_block(v, &total);
    if (i < (int)gridDim.x) pre[i] = carry + before;
    carry += total;
  }
}

__global__ void k_grid_bucket(int n, const int* cell, const int* rank, const int* local, const int* pre, int* bucket) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cell[i];
  if (c >= 0) bucket[pre[(unsigned)c / kScanCells] + local[c] + rank[i]] = i;
}

// One thread per slot of the buckets (m of them), and the cells' starts by the same
// threads.  perm and second (with out2) may be NULL.
__global__ void k_grid_place(int m, int64_t ncells, const int* cell, const int* count, const int* local, const int* pre,
                             const int* bucket, const float2* pos, const float2* second, int* start, int* perm,
                             int* src, float2* out, float2* out2) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t c = a; c <= ncells; c += (int64_t)gridDim.x * blockDim.x)
    start[c] = c < ncells ? pre[c / kScanCells] + local[c] : m;
  if (a >= m) return;
  const int i = bucket[a], c = cell[i];
  const int b = pre[(unsigned)c / kScanCells] + local[c], k = count[c];
  int at = b;
  for (int j = b; j < b + k; ++j) at += bucket[j] < i ? 1 : 0;
  src[at] = i;
  if (perm) perm[i] = at;
  out[at] = pos[i];
  if (second) out2[at] = second[i];
}

// The tables from `count` (with the ticket, zero), `cell` and `rank` on: m of the n
// points have a cell.  rank and perm may share an array.
void launch_cells(int n, int m, int64_t ncells, const int* cell, int* count, int* ticket, int* rank, int* local, int* pre,
                  int* bucket, const float2* pos, const float2* second, int* start, int* perm, int* src, float2* out,
                  float2* out2, cudaStream_t s) {
  k_cell_scan<<<(unsigned)((ncells + kScanCells - 1) / kScanCells), kScanThreads, 0, s>>>(ncells, count, local, pre,
                                                                                         ticket);
  k_grid_bucket<<<(n + 255) / 256, 256, 0, s>>>(n, cell, rank, local, pre, bucket);
  k_grid_place<<<(std::max(m, 1) + 255) / 256, 256, 0, s>>>(m, ncells, cell, count, local, pre, bucket, pos, second,
                                                            start, perm, src, out, out2);
}

// Exclusive scan, single-pass per block + block offsets.
__global__ void k_scan_blocks(const int* in, int* out, int* block_sums, int64_t n) {
  __shared__ int s[1024];
  const int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x;
  const int x = i < n ? in[i] : 0;
  s[threadIdx.x] = x;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int y = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
    __syncthreads();
    s[threadIdx.x] += y;
    __syncthreads();
  }
  if (i < n) out[i] = s[threadIdx.x] - x;
  if (threadIdx.x == 1023) block_sums[blockIdx.x] = s[1023];
}

__global__ void k_scan_add(int* out, const int* block_prefix, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x;
  if (i < n) out[i] += block_prefix[blockIdx.x];
}

// Fixed-radius query, one thread per sorted slot i (threads of a warp are
// neighbouring points of one cell row, so their candidates overlap in L1).
// Cells are row-major, so each stencil row is one contiguous range of sorted
// points (up to three with periodic wrap).  The stencil is the disk: for each
// cell row the x extent comes from the query's own position and the row's
// vertical distance, widened by a margin far above float rounding; cells it
// skips hold no point within r, so the result and its order equal the full
// (2w+1)^2 stencil's: rows bottom to top, cells left to right in stencil
// order, points of a cell in sorted order (the reference's SaveNeighborsFunctor
// order, gridCount2d.h:263-296).  Distances use the reference formula
// fl(fl(dx*dx) + fl(dy*dy)) <= fl(r*r) without FMA; periodic grids take the
// minimum image (|d| > L/2 -> d -= copysign(L, d)).  A candidate is tested
// without branches: its distance from i in the order is written to the thread's
// shared row at slot nf and nf advances on a hit (a range takes this path only when
// the row has room for all of it and 16 bits for the distance).  Rows hold up to
// kStageCap neighbours and are flushed by their own warp one after the other
// (coalesced), ids and rows mapped through src when given; what does not fit goes
// straight to global memory.
// Bound by the latency of the candidates' loads (some 50 per point at r = 1.92 cells of
// 2.4 points): rows of 16 bits leave the L1 twice the room and let 48 warps reside
// instead of 32 (41 are active on average), and both coordinates of a candidate share an instruction.  r = 3 x
// spacing, 1,000,000 points, periodic: 176 -> 131 us (rows of 32 bits: 174).
constexpr int kStageCap = 48;
constexpr int kFrnnThreads = 128;
constexpr int kFrnnBlocks = 12;  // per SM: 40 registers (14 blocks spill: 152 us for 131; 10: 139)

// To 2 ulp, where a margin of 1e-4 follows.
__device__ __forceinline__ float near_sqrt(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Two floats in one register pair: both lanes rounded to nearest, as one at a time.
__device__ __forceinline__ unsigned long long pair_of(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ unsigned long long pair_add(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// fl(fl(x x) + fl(y y))
__device__ __forceinline__ float pair_norm2(unsigned long long d) {
  float x, y;
  asm("{\n\t.reg .b64 q;\n\tmul.rn.f32x2 q, %2, %2;\n\tmov.b64 {%0, %1}, q;\n\t}" : "=f"(x), "=f"(y) : "l"(d));
  return __fadd_rn(x, y);
}

// The candidates b .. e - 1 within r of a point, from slot nf of its row on.  The
// differences have the opposite sign of the reference's (candidate - point, minus the
// shift): rounding is symmetric and they are squared.
template <bool kShift>
__device__ __forceinline__ int near_range(const float2* __restrict__ pos, int b, int e, unsigned long long minus_p,
                                          unsigned long long minus_shift, float r2, int i, short* mine, int nf) {
  const unsigned long long* at = reinterpret_cast<const unsigned long long*>(pos);
#pragma unroll 4
  for (int j = b; j < e; ++j) {
    unsigned long long d = pair_add(at[j], minus_p);
    if (kShift) d = pair_add(d, minus_shift);
    const bool hit = (pair_norm2(d) <= r2) & (j != i);
    mine[nf] = (short)(j - i);
    nf += hit ? 1 : 0;
  }
  return nf;
}

// How a grid's rows end: points beyond the domain clamped into the border cells; the
// minimum image by row segment (see k_grid_frnn); the minimum image per candidate.
enum : int { kNearClamp = 0, kNearSegment = 1, kNearWrap = 2 };

struct NearQuery {
  float r, ix, iy, Lx, Ly;  // radius, 1 / cell, domain
  int max_nb, scap;         // neighbours wanted, and how many of them are staged
};

// The neighbours of point i into its stage row (past scap into direct); how many.
template <int kMode>
__device__ __forceinline__ int near_rows(const GridView& G, const NearQuery& Q, const float2* __restrict__ pos,
                                         const int* __restrict__ start, float2 p, int i, short* mine, int* direct,
                                         const int* __restrict__ src) {
  int nf = 0;
  const float r = Q.r, r2 = __fmul_rn(r, r);
  const float hx = 0.5f * Q.Lx, hy = 0.5f * Q.Ly;
  const float mx = 1e-3f * G.cx + 1e-5f * (fabsf(p.x) + fabsf(G.minx) + r);
  const float my = 1e-3f * G.cy + 1e-5f * (fabsf(p.y) + fabsf(G.miny) + r);
  const float px = p.x - G.minx, py = p.y - G.miny;
  const unsigned long long minus_p = pair_of(-p.x, -p.y);
  int ylo = (int)floorf(fmaxf(fminf((py - r - my) * Q.iy, 1e9f), -1e9f));
  int yhi = (int)floorf(fmaxf(fminf((py + r + my) * Q.iy, 1e9f), -1e9f));
  if (kMode == kNearClamp) {
    ylo = ylo < 0 ? 0 : (ylo >= G.ny ? G.ny - 1 : ylo);
    yhi = yhi < 0 ? 0 : (yhi >= G.ny ? G.ny - 1 : yhi);
  } else if (kMode == kNearWrap && yhi - ylo + 1 > G.ny) {
    ylo = 0; yhi = G.ny - 1;  // the disk covers every row: visit each once
  }
  for (int yy = ylo; yy <= yhi; ++yy) {
    // vertical distance from p to the row's slab (0 inside), minus the margin;
    // without wrap the border rows also hold the points clamped into them,
    // so their slabs extend to infinity
    float slo = yy * G.cy, shi = slo + G.cy;
    if (kMode == kNearClamp) {
      if (yy == 0) slo = -INFINITY;
      if (yy == G.ny - 1) shi = INFINITY;
    }
    const float dym = fmaxf(fmaxf(slo - py, py - shi) - my, 0.f);
    const float hw = (kMode == kNearWrap && yhi - ylo + 1 >= G.ny) ? r + mx
                                                                   : near_sqrt(fmaxf(r2 - dym * dym, 0.f)) * 1.0001f + mx;
    int xlo = (int)floorf(fmaxf(fminf((px - hw) * Q.ix, 1e9f), -1e9f));
    int xhi = (int)floorf(fmaxf(fminf((px + hw) * Q.ix, 1e9f), -1e9f));
    int y = yy;
    float xs = 0.f, ys = 0.f;
    if (kMode == kNearSegment) {
      if (y < 0) { y += G.ny; ys = Q.Ly; }
      else if (y >= G.ny) { y -= G.ny; ys = -Q.Ly; }
    } else if (kMode == kNearWrap) {
      y %= G.ny;
      if (y < 0) y += G.ny;
      if (xhi - xlo + 1 > G.nx) { xlo = 0; xhi = G.nx - 1; }
    } else {
      xlo = xlo < 0 ? 0 : (xlo >= G.nx ? G.nx - 1 : xlo);
      xhi = xhi < 0 ? 0 : (xhi >= G.nx ? G.nx - 1 : xhi);
    }
    const int* row = start + y * G.nx;
    // [xlo, xhi] in stencil order: from its wrapped start to the end of the row, then
    // on from cell 0.  By segment, cells left of 0 are the row's end (+Lx), right of
    // nx - 1 its start (-Lx).
    int sa = xlo, more = -1;
    if (kMode == kNearSegment) {
      if (xlo < 0) { sa += G.nx; xs = Q.Lx; }
    } else if (kMode == kNearWrap) {
      sa = (xlo % G.nx + G.nx) % G.nx;
    }
    int sb = sa + (xhi - xlo);
    if (kMode != kNearClamp && sb >= G.nx) {
      more = sb - G.nx;
      sb = G.nx - 1;
    }
    for (;;) {
      const int b = __ldg(row + sa), e = __ldg(row + sb + 1);
      const bool fits = nf + (e - b) <= Q.scap && b - i >= -32768 && e - i <= 32768;
      if (fits && kMode == kNearWrap) {
#pragma unroll 4
        for (int j = b; j < e; ++j) {
          const float2 o = pos[j];
          float dx = __fsub_rn(p.x, o.x), dy = __fsub_rn(p.y, o.y);
          dx = fabsf(dx) > hx ? __fsub_rn(dx, copysignf(Q.Lx, dx)) : dx;
          dy = fabsf(dy) > hy ? __fsub_rn(dy, copysignf(Q.Ly, dy)) : dy;
          const bool hit = (__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) <= r2) & (j != i);
          mine[nf] = (short)(j - i);
          nf += hit ? 1 : 0;
        }
      } else if (fits) {
        if (kMode == kNearSegment && (xs != 0.f || ys != 0.f))
          nf = near_range<true>(pos, b, e, minus_p, pair_of(-xs, -ys), r2, i, mine, nf);
        else
          nf = near_range<false>(pos, b, e, minus_p, 0, r2, i, mine, nf);
      } else {
        for (int j = b; j < e; ++j) {
          const float2 o = pos[j];
          float dx = __fsub_rn(p.x, o.x), dy = __fsub_rn(p.y, o.y);
          if (kMode != kNearClamp) {
            dx = fabsf(dx) > hx ? __fsub_rn(dx, copysignf(Q.Lx, dx)) : dx;
            dy = fabsf(dy) > hy ? __fsub_rn(dy, copysignf(Q.Ly, dy)) : dy;
          }
          if ((__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) <= r2) & (j != i)) {
            const bool near = j - i >= -32768 && j - i < 32768;
            if (nf < Q.scap) mine[nf] = near ? (short)(j - i) : (short)0;  // 0: written already
            if (nf < Q.max_nb && (nf >= Q.scap || !near)) direct[nf] = src ? __ldg(src + j) : j;
            ++nf;
          }
        }
      }
      if (kMode == kNearClamp || more < 0) break;
      sa = 0;
      sb = more;
      more = -1;
      xs = kMode == kNearSegment && xs == 0.f ? -Q.Lx : 0.f;
    }
  }
  return nf;
}

template <bool kPeriodic>
__global__ void __launch_bounds__(kFrnnThreads, kFrnnBlocks) k_grid_frnn(GridView G, NearQuery Q, int n,
                                                           const float2* __restrict__ pos,
                                                           const int* __restrict__ start, int* __restrict__ counts,
                                                           int* __restrict__ ids, unsigned long long* overflow,
                                                           const int* __restrict__ src,
                                                           const int* __restrict__ outside, int wrap_by_segment) {
  __shared__ short stage[kFrnnThreads * (kStageCap + 1)];
  const int t = threadIdx.x, lane = t & 31, i = blockIdx.x * kFrnnThreads + t;
  short* mine = stage + t * (kStageCap + 1);
  int nf = 0, row = -1;
  // Minimum image by segment: with every point inside the domain and the
  // stencil well under half the domain (checked by the caller), a candidate's
  // |dx| exceeds half the domain exactly when its cell was reached across the
  // wrap, so the per-candidate test "|dx| > Lx/2: dx -= copysign(Lx, dx)" is
  // the constant shift of its row segment: dx + xs, with the same rounding.
  const bool seg = kPeriodic && wrap_by_segment && outside && __ldg(outside) == 0;
  if (i < n) {
    const float2 p = pos[i];
    row = src ? __ldg(src + i) : i;
    int* direct = ids + (size_t)row * Q.max_nb;
    if (!kPeriodic) nf = near_rows<kNearClamp>(G, Q, pos, start, p, i, mine, direct, src);
    else if (seg) nf = near_rows<kNearSegment>(G, Q, pos, start, p, i, mine, direct, src);
    else nf = near_rows<kNearWrap>(G, Q, pos, start, p, i, mine, direct, src);
    counts[row] = nf < Q.max_nb ? nf : Q.max_nb;
    if (nf > Q.max_nb) atomicAdd(overflow, 1ull);
  }
  const int staged = min(nf, Q.scap);
  __syncwarp();
  const short* theirs = stage + (t & ~31) * (kStageCap + 1);
#pragma unroll 4
  for (int rr = 0; rr < 32; ++rr) {
    const int cr = __shfl_sync(0xffffffffu, staged, rr), to = __shfl_sync(0xffffffffu, row, rr);
    int* dst = ids + (size_t)to * Q.max_nb;
    const short* from = theirs + rr * (kStageCap + 1);
    for (int k = lane; k < cr; k += 32) {
      const int d = from[k], j = i - lane + rr + d;
      if (d) dst[k] = src ? __ldg(src + j) : j;
    }
  }
}

// outside: the out-of-domain flag of the hashing of `pos` (NULL: unknown).
int launch_grid_frnn(const GridView& G, int n, const float2* pos, const int* start, float r, float Lx, float Ly,
                     int max_nb, int* counts, int* ids, unsigned long long* ovf, const int* src, cudaStream_t s,
                     const int* outside) {
  const unsigned blocks = (unsigned)((n + kFrnnThreads - 1) / kFrnnThreads);
  // the minimum image by row segment is exact when every candidate cell lies
  // within 0.45 of the domain of the query point (stencil half-width + a
  // cell + the kernel's margins, with slack) and a row spans under nx cells
  auto fits = [&](float c, float L, int cells, float mn) {
    const double margin = 1e-3 * c + 1e-5 * (2.0 * std::fabs((double)mn) + L + r);
    return cells >= 20 && (1.0001 * r + margin + c) * 1.01 <= 0.45 * L;
  };
  const int by_segment = G.periodic && outside && fits(G.cx, Lx, G.nx, G.minx) && fits(G.cy, Ly, G.ny, G.miny);
  const NearQuery Q = {r, 1.0f / G.cx, 1.0f / G.cy, Lx, Ly, max_nb, std::min(max_nb, kStageCap)};
  auto kernel = G.periodic ? k_grid_frnn<true> : k_grid_frnn<false>;
  kernel<<<blocks, kFrnnThreads, 0, s>>>(G, Q, n, pos, start, counts, ids, ovf, src, outside, by_segment);
  QCK(cudaGetLastError());
  return MCL_OK;
}

__global__ void k_mean_occupancy(int64_t ncells, const int* count, unsigned long long* acc) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const int k = count[c];
  if (k > 0) {
    atomicAdd(acc, 1ull);
    atomicAdd(acc + 1, (unsigned long long)k);
  }
}

// Exclusive scan of up to a few hundred thousand ints in one block, entirely on
// the device (each thread scans a contiguous chunk, then the chunk totals).
__global__ void k_scan_one_block(const int* in, int* out, int64_t n) {
  __shared__ int tot[1024];
  const int64_t per = (n + blockDim.x - 1) / blockDim.x;
  const int64_t lo = threadIdx.x * per, hi = min(n, lo + per);
  int run = 0;
  for (int64_t i = lo; i < hi; ++i) run += in[i];
  tot[threadIdx.x] = run;
  __syncthreads();
  for (int o = 1; o < (int)blockDim.x; o <<= 1) {
    const int y = threadIdx.x >= (unsigned)o ? tot[threadIdx.x - o] : 0;
    __syncthreads();
    tot[threadIdx.x] += y;
    __syncthreads();
  }
  int acc = threadIdx.x ? tot[threadIdx.x - 1] : 0;
  for (int64_t i = lo; i < hi; ++i) {
    const int x = in[i];
    out[i] = acc;
    acc += x;
  }
}

// Exclusive scan of n ints, entirely on the device (no host round trip, so the
// grid build can sit inside a captured CUDA graph): per-block scans, one block
// scanning the block totals, then the block offsets added.  tmp holds nb ints
// and tmp2 nb ints, nb = ceil(n / 1024).
int scan_exclusive(const int* in, int* out, int64_t n, int* tmp, int* tmp2, cudaStream_t s) {
  const int64_t nb = (n + 1023) / 1024;
  k_scan_blocks<<<(unsigned)nb, 1024, 0, s>>>(in, out, tmp, n);
  if (nb > 1) {
    k_scan_one_block<<<1, 1024, 0, s>>>(tmp, tmp2, nb);
    k_scan_add<<<(unsigned)nb, 1024, 0, s>>>(out, tmp2, n);
  }
  QCK(cudaGetLastError());
  return MCL_OK;
}

GridView view_of(const mcl_grid* g) {
  GridView G;
  G.minx = g->minx; G.miny = g->miny; G.cx = g->cx; G.cy = g->cy;
  G.nx = g->nx; G.ny = g->ny; G.morton = g->morton; G.periodic = (g->flags & MCL_GRID_PERIODIC) ? 1 : 0;
  return G;
}

}  // namespace

// ---------------------------------------------------------------------------
// Predicate diagnostics.
namespace {

struct StageCounters {
  unsigned long long orient_fp64, orient_exact, incircle_fp64, incircle_exact, sos;
};

__host__ __device__ inline int eval_pred(int kind, const float* q, const int* ids, int* stage) {
  StageCounters c = {0, 0, 0, 0, 0};
  int ovf = 0, s;
  if (kind == 0) {
    s = orient2d(q[0], q[1], q[2], q[3], q[4], q[5], &c, &ovf);
    *stage = c.orient_exact ? 2 : (c.orient_fp64 ? 1 : 0);
  } else if (kind == 1) {
    s = incircle(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], &c, &ovf);
    *stage = c.incircle_exact ? 2 : (c.incircle_fp64 ? 1 : 0);
  } else {
    s = incircle_sos(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], ids[0], ids[1], ids[2], ids[3], &c, &ovf);
    *stage = c.sos ? 3 : (c.incircle_exact ? 2 : (c.incircle_fp64 ? 1 : 0));
  }
  if (ovf) *stage = -1;
  return s;
}

__global__ void k_debug_pred(int kind, const float* pts, const int* ids, int64_t n, int* sign, int* stage) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int w = kind == 0 ? 6 : 8;
  int st = 0;
  const int s = eval_pred(kind, pts + w * i, ids ? ids + 4 * i : nullptr, &st);
  sign[i] = s;
  if (stage) stage[i] = st;
}

}  // namespace

namespace {

// Counted queries: a cell pair per slot in the mesh's device scratch, a word per slot in
// its pinned host memory (count_done).
constexpr int kCells = 8;
static_assert((kCells + 2 * kCountSlots) * 8 <= kScratchBytes, "the cells fit the scratch");

MeshView mesh_view(const mcl_mesh* m) {
  return MeshView{m->ev, m->en, m->vhe, m->pos[m->cur], (int)m->V, (int)m->E};
}

// launch(cell, host): the query's kernel with the cell pair and the host word of its count.
template <typename Launch>
int counted(mcl_mesh* m, cudaStream_t s, int64_t* out, Launch launch) {
  if (!out) {
    launch(nullptr, nullptr);
    QCK(cudaGetLastError());
    return MCL_OK;
  }
  const CountSlot slot(&m->count_slots);
  launch(m->scratch + kCells + 2 * slot.at, m->counts_dev + slot.at);
  QCK(cudaGetLastError());
  QCK(cudaStreamSynchronize(s));
  *out = (int64_t) * (volatile unsigned long long*)(m->counts_host + slot.at);
  return MCL_OK;
}

int launch_one_ring(mcl_mesh* m, const int* verts, int64_t n, int layout, int max_ring, int* out, cudaStream_t s,
                    int64_t* truncated) {
  if (n == 0) {
    if (truncated) QCK(cudaStreamSynchronize(s));
    if (truncated) *truncated = 0;
    return MCL_OK;
  }
  const unsigned blocks = (unsigned)((n + kRingThreads - 1) / kRingThreads);
  const int delaunay = m->delaunay && m->valid_cur && m->square ? 1 : 0;
  auto kernel = layout == MCL_LAYOUT_COLUMN ? k_one_ring<false> : k_one_ring<true>;
  return counted(m, s, truncated, [&](unsigned long long* cell, unsigned long long* host) {
    kernel<<<blocks, kRingThreads, 0, s>>>(mesh_view(m), verts, (int)n, max_ring, out, m->vfix, delaunay, cell, host);
  });
}

int launch_mesh_frnn(mcl_mesh* m, const int* verts, int64_t n, float r2, const float* rcomp, int layout, int max_frnn,
                     int* out, cudaStream_t s, int64_t* overflow) {
  if (n == 0) {
    if (overflow) QCK(cudaStreamSynchronize(s));
    if (overflow) *overflow = 0;
    return MCL_OK;
  }
  const FrnnQuery Q = {verts, (int)n, r2, layout, max_frnn, out, rcomp, rcomp ? m->vcomp : nullptr};
  constexpr int kThreads = 32 * kFrnnWarps;
  const int per = n <= kFrnnQuarters ? kThreads / 16 : n <= kFrnnMany ? kThreads / 8 : kThreads;  // queries per block
  auto kernel = n <= kFrnnQuarters ? k_mesh_frnn<16> : n <= kFrnnMany ? k_mesh_frnn<8> : k_mesh_frnn_many<16>;
  return counted(m, s, overflow, [&](unsigned long long* cell, unsigned long long* host) {
    kernel<<<(unsigned)((n + per - 1) / per), kThreads, 0, s>>>(mesh_view(m), Q, cell, host);
    if (n > kFrnnFew)
      k_mesh_frnn_left<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mesh_view(m), Q, cell, host);
  });
}

}  // namespace

extern "C" {

int mcl_debug_predicates_host(int kind, const float* pts, const int32_t* ids, int64_t n, int32_t* sign,
                              int32_t* stage) {
  if (!pts || !sign || kind < 0 || kind > 2 || (kind == 2 && !ids)) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  const int w = kind == 0 ? 6 : 8;
  for (int64_t i = 0; i < n; ++i) {
    int st = 0;
    sign[i] = eval_pred(kind, pts + w * i, ids ? ids + 4 * i : nullptr, &st);
    if (stage) stage[i] = st;
  }
  return MCL_OK;
}

int mcl_debug_predicates_device(int kind, const float* pts, const int32_t* ids, int64_t n, int32_t* sign,
                                int32_t* stage, void* stream) {
  if (!pts || !sign || kind < 0 || kind > 2 || (kind == 2 && !ids)) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  if (n == 0) return MCL_OK;
  k_debug_pred<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(kind, pts, ids, n, sign, stage);
  QCK(cudaGetLastError());
  return MCL_OK;
}

int mcl_one_ring(mcl_mesh* m, int layout, int max_ring, int32_t* ring, void* stream, int64_t* truncated) {
  if (!m || !ring || max_ring < 2 || (layout != MCL_LAYOUT_COLUMN && layout != MCL_LAYOUT_ROW))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  return launch_one_ring(m, nullptr, m->V, layout, max_ring, ring, (cudaStream_t)stream, truncated);
}

int mcl_closest_neighbors(mcl_mesh* m, int layout, int max_ring, const int32_t* ring, int32_t* out, void* stream) {
  if (!m || !ring || !out || max_ring < 2) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  const bool vec = layout != MCL_LAYOUT_COLUMN && max_ring % 4 == 0 && ((uintptr_t)ring & 15) == 0;
  auto kernel = vec ? k_closest<true> : k_closest<false>;
  kernel<<<(unsigned)((m->V + 255) / 256), 256, 0, (cudaStream_t)stream>>>(m->pos[m->cur], (int)m->V, layout, max_ring,
                                                                          ring, out);
  QCK(cudaGetLastError());
  return MCL_OK;
}

int mcl_mesh_frnn(mcl_mesh* m, float r, int layout, int max_frnn, int32_t* out, void* stream, int64_t* overflow) {
  if (!m || !out || max_frnn < 2 || !(r >= 0.f)) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  return launch_mesh_frnn(m, nullptr, m->V, r * r, nullptr, layout, max_frnn, out, (cudaStream_t)stream, overflow);
}

int mcl_batch_frnn(mcl_mesh* m, const float* r_dev, int layout, int max_frnn, int32_t* out, void* stream,
                   int64_t* overflow) {
  if (!m || !r_dev || !out || max_frnn < 2 || (layout != MCL_LAYOUT_COLUMN && layout != MCL_LAYOUT_ROW))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  return launch_mesh_frnn(m, nullptr, m->V, 0.f, r_dev, layout, max_frnn, out, (cudaStream_t)stream, overflow);
}

int mcl_batch_frnn_list(mcl_mesh* m, const float* r_dev, const int32_t* verts_dev, int64_t n, int layout,
                        int max_frnn, int32_t* out_dev, void* stream, int64_t* overflow) {
  if (!m || !r_dev || (n > 0 && (!verts_dev || !out_dev)) || n < 0 || max_frnn < 2 ||
      (layout != MCL_LAYOUT_COLUMN && layout != MCL_LAYOUT_ROW))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  return launch_mesh_frnn(m, verts_dev, n, 0.f, r_dev, layout, max_frnn, out_dev, (cudaStream_t)stream, overflow);
}

int mcl_one_ring_list(mcl_mesh* m, const int32_t* verts_dev, int64_t n, int layout, int max_ring, int32_t* out_dev,
                      void* stream, int64_t* truncated) {
  if (!m || (n > 0 && (!verts_dev || !out_dev)) || n < 0 || max_ring < 2 ||
      (layout != MCL_LAYOUT_COLUMN && layout != MCL_LAYOUT_ROW))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  return launch_one_ring(m, verts_dev, n, layout, max_ring, out_dev, (cudaStream_t)stream, truncated);
}

int mcl_dla_freeze(mcl_mesh* m, const float* r_dev, uint8_t* frozen, void* stream, int64_t* newly_frozen) {
  if (!m || !r_dev || !frozen) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  cudaStream_t s = (cudaStream_t)stream;
  if (!m->fnew && cudaMalloc((void**)&m->fnew, m->V) != cudaSuccess)
    return qfail(MCL_ERR_OUT_OF_MEMORY, "mcl_dla_freeze: scratch");
  unsigned long long* cnt = m->scratch + 1;
  MeshView M{m->ev, m->en, m->vhe, m->pos[m->cur], (int)m->V, (int)m->E};
  const ActV A = act_of(m);
  QCK(cudaMemsetAsync(cnt, 0, 8, s));
  if (A.V_it > 0) {
    k_dla_freeze<<<(unsigned)((A.V_it + 127) / 128), 128, 0, s>>>(M, A, m->vfix, r_dev, m->vcomp, frozen, m->fnew, cnt);
    k_dla_commit<<<(unsigned)((A.V_it + 255) / 256), 256, 0, s>>>(A, frozen, m->fnew);
  }
  QCK(cudaGetLastError());
  if (newly_frozen) {
    unsigned long long t = 0;
    QCK(cudaMemcpyAsync(&t, cnt, 8, cudaMemcpyDeviceToHost, s));
    QCK(cudaStreamSynchronize(s));
    *newly_frozen = (int64_t)t;
  }
  return MCL_OK;
}

int mcl_grid_create(int64_t n, float minx, float miny, float cx, float cy, int32_t nx, int32_t ny, int flags,
                    mcl_grid** out) {
  if (!out || n < 0 || nx < 1 || ny < 1 || !(cx > 0.f) || !(cy > 0.f) || (int64_t)nx * ny > (1ll << 30))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad grid");
  mcl_grid* g = new mcl_grid();
  std::memset(g, 0, sizeof(*g));
  g->n = n; g->minx = minx; g->miny = miny; g->cx = cx; g->cy = cy; g->nx = nx; g->ny = ny; g->flags = flags;
  int side = 1, bits = 0;
  while (side < std::max(nx, ny)) { side <<= 1; ++bits; }
  const int64_t mcells = (int64_t)side * side;
  g->morton = 0;  // row-major: a stencil row of cells is one contiguous range of sorted points
  g->mbits = bits;
  g->ncells = g->morton ? mcells : (int64_t)nx * ny;
  const int64_t nn = std::max<int64_t>(n, 1);
  const int64_t nb = (g->ncells + kScanCells - 1) / kScanCells + 4;
  cudaError_t e = cudaSuccess;
  auto A = [&](void** p, size_t b) { if (e == cudaSuccess) e = cudaMalloc(p, b); };
  A((void**)&g->cell, 4 * nn);
  A((void**)&g->count, 4 * (g->ncells + 2));
  A((void**)&g->start, 4 * (g->ncells + 1));
  A((void**)&g->local, 4 * g->ncells);
  A((void**)&g->bucket, 4 * nn);
  A((void**)&g->perm, 4 * nn);
  A((void**)&g->src, 4 * nn);
  A((void**)&g->tmp, 8 * nn);
  A((void**)&g->tmp2, 8 * nn);
  A(&g->scan_tmp, 4 * nb);  // also the query's overflow count and the occupancy sums
  if (e == cudaSuccess) e = cudaMemset(g->count, 0, 4 * (g->ncells + 2));
  if (e == cudaSuccess) e = cudaMemset(g->start, 0, 4 * (g->ncells + 1));
  if (e != cudaSuccess) {
    mcl_grid_destroy(g);
    return qfail(MCL_ERR_OUT_OF_MEMORY, "grid allocation");
  }
  *out = g;
  return MCL_OK;
}

int mcl_grid_destroy(mcl_grid* g) {
  if (!g) return MCL_OK;
  void* ptrs[] = {g->cell, g->count, g->start, g->local, g->bucket, g->perm, g->src, g->tmp, g->tmp2, g->scan_tmp};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  delete g;
  return MCL_OK;
}

}  // extern "C"

namespace {
// Cell tables for the positions pos (input order) and their sorted copy in g->tmp, that
// of vel (may be NULL) in g->tmp2; pos and vel themselves are not written.
int grid_build_tables(mcl_grid* g, const float2* pos, const float2* vel, cudaStream_t s) {
  const int n = (int)g->n;
  int* flag = g->count + g->ncells;
  QCK(cudaMemsetAsync(g->count, 0, 4 * (g->ncells + 2), s));
  k_grid_hash<<<(n + 255) / 256, 256, 0, s>>>(view_of(g), n, pos, g->cell, g->count, g->perm, flag);
  launch_cells(n, n, g->ncells, g->cell, g->count, flag + 1, g->perm, g->local, (int*)g->scan_tmp, g->bucket, pos, vel,
               g->start, g->perm, g->src, g->tmp, g->tmp2, s);
  QCK(cudaGetLastError());
  return MCL_OK;
}
}  // namespace

extern "C" {

int mcl_grid_update(mcl_grid* g, mcl_float2* pos, mcl_float2* vel, void* stream) {
  if (!g || !pos) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  cudaStream_t s = (cudaStream_t)stream;
  const int n = (int)g->n;
  if (n == 0) return MCL_OK;
  const int rc = grid_build_tables(g, (const float2*)pos, (const float2*)vel, s);
  if (rc != MCL_OK) return rc;
  QCK(cudaMemcpyAsync(pos, g->tmp, 8 * (size_t)n, cudaMemcpyDeviceToDevice, s));
  if (vel) QCK(cudaMemcpyAsync(vel, g->tmp2, 8 * (size_t)n, cudaMemcpyDeviceToDevice, s));
  QCK(cudaGetLastError());
  g->built = 1;
  return MCL_OK;
}

int mcl_grid_build(mcl_grid* g, const mcl_float2* pos, void* stream) {
  if (!g || !pos) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  if (g->n == 0) return MCL_OK;
  const int rc = grid_build_tables(g, (const float2*)pos, nullptr, (cudaStream_t)stream);
  if (rc == MCL_OK) g->built = 1;
  return rc;
}

int mcl_grid_frnn_ids(mcl_grid* g, float r, int max_nb, int32_t* counts, int32_t* ids, void* stream,
                      int64_t* overflow) {
  if (!g || !counts || !ids || max_nb < 1 || !(r >= 0.f)) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  if (!g->built) return qfail(MCL_ERR_INVALID_ARGUMENT, "mcl_grid_frnn_ids: call mcl_grid_build first");
  cudaStream_t s = (cudaStream_t)stream;
  const int n = (int)g->n;
  if (n == 0) return MCL_OK;
  const GridView G = view_of(g);
  unsigned long long* ovf = (unsigned long long*)g->scan_tmp;
  QCK(cudaMemsetAsync(ovf, 0, 8, s));
  const int rc = launch_grid_frnn(G, n, g->tmp, g->start, r, g->cx * g->nx, g->cy * g->ny, max_nb, counts,
                                  ids, ovf, g->src, s, g->count + g->ncells);
  if (rc != MCL_OK) return rc;
  if (overflow) {
    unsigned long long t = 0;
    QCK(cudaMemcpyAsync(&t, ovf, 8, cudaMemcpyDeviceToHost, s));
    QCK(cudaStreamSynchronize(s));
    *overflow = (int64_t)t;
  }
  return MCL_OK;
}

int mcl_grid_tables(mcl_grid* g, const int32_t** perm, const int32_t** start, const int32_t** count, int32_t* cx,
                    int32_t* cy) {
  if (!g) return qfail(MCL_ERR_INVALID_ARGUMENT, "null grid");
  if (perm) *perm = g->perm;
  if (start) *start = g->start;
  if (count) *count = g->count;
  if (cx) *cx = g->nx;
  if (cy) *cy = g->ny;
  return MCL_OK;
}

int mcl_grid_describe(mcl_grid* g, mcl_grid_desc* d) {
  if (!g || !d) return qfail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  d->min_x = g->minx; d->min_y = g->miny; d->cell_x = g->cx; d->cell_y = g->cy;
  d->cells_x = g->nx; d->cells_y = g->ny; d->morton = g->morton;
  d->periodic = (g->flags & MCL_GRID_PERIODIC) ? 1 : 0;
  d->table_size = g->ncells; d->num_points = g->n;
  d->perm_dev = g->perm; d->cell_start_dev = g->start; d->cell_count_dev = g->count;
  return MCL_OK;
}

int mcl_grid_frnn(mcl_grid* g, const mcl_float2* pos, float r, int max_nb, int32_t* counts, int32_t* ids, void* stream,
                  int64_t* overflow) {
  if (!g || !pos || !counts || !ids || max_nb < 1 || !(r >= 0.f)) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  cudaStream_t s = (cudaStream_t)stream;
  const int n = (int)g->n;
  if (n == 0) return MCL_OK;
  const GridView G = view_of(g);
  unsigned long long* ovf = (unsigned long long*)g->scan_tmp;
  QCK(cudaMemsetAsync(ovf, 0, 8, s));
  const int rc = launch_grid_frnn(G, n, (const float2*)pos, g->start, r, g->cx * g->nx, g->cy * g->ny,
                                  max_nb, counts, ids, ovf, nullptr, s, nullptr);
  if (rc != MCL_OK) return rc;
  if (overflow) {
    unsigned long long t = 0;
    QCK(cudaMemcpyAsync(&t, ovf, 8, cudaMemcpyDeviceToHost, s));
    QCK(cudaStreamSynchronize(s));
    *overflow = (int64_t)t;
  }
  return MCL_OK;
}

int mcl_grid_mean_occupancy(mcl_grid* g, float* mean) {
  if (!g || !mean) return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  unsigned long long* acc = (unsigned long long*)g->scan_tmp;
  QCK(cudaMemset(acc, 0, 16));
  k_mean_occupancy<<<(unsigned)((g->ncells + 255) / 256), 256>>>(g->ncells, g->count, acc);
  unsigned long long h[2];
  QCK(cudaMemcpy(h, acc, 16, cudaMemcpyDeviceToHost));
  *mean = h[0] ? (float)h[1] / (float)h[0] : 0.f;
  return MCL_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Batch FRNN over per-mesh grids (mcl_batch_frnn_grid): mesh c gets a uniform
// grid over [lo, hi)^2 with cells of its own radius (so the disk touches at
// most 3 x 3 cells), its cells numbered after those of the meshes before it;
// one counting sort orders every point of every mesh, then one query kernel
// answers every point with its own mesh's grid.  Same results as
// mcl_batch_frnn (rows ascending), without walking the mesh.
namespace {

__device__ __forceinline__ int bg_coord(float p, float lo, float c, int n) {
  float kf = floorf(__fdiv_rn(__fsub_rn(p, lo), c));
  kf = fminf(fmaxf(kf, -1.0e9f), 1.0e9f);
  const int k = (int)kf;
  return k < 0 ? 0 : (k >= n ? n - 1 : k);
}

__global__ void k_bgrid_hash(int V, const float2* pos, const unsigned char* vfix, const int* vcomp, const int4* par,
                             float lo, int* cell, int* count, int* rank, int* out, int F) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  if (vfix[v]) {  // bounding corners hold no neighbour within any radius
    cell[v] = -1;
    out[(size_t)v * F] = 0;
    return;
  }
  const int4 q = par[vcomp ? vcomp[v] : 0];
  const float c = __int_as_float(q.x);
  const float2 p = pos[v];
  const int x = bg_coord(p.x, lo, c, q.y), y = bg_coord(p.y, lo, c, q.y);
  const int id = q.z + y * q.y + x;
  cell[v] = id;
  rank[v] = atomicAdd(count + id, 1);
}

// One thread per sorted slot (neighbouring points of one cell row of one
// mesh); disk-culled rows of the mesh's grid, branch-free candidate test,
// ids staged per thread in shared memory, sorted there and written out one row
// per warp step.  Rows: out[v*F] = count, out[v*F + 1 + k] ascending.
// The stage rows are as long as the caller's.  Bound by the candidates' loads and the
// sort (r = 2 x spacing, 1,400,000 points, 12.6 neighbours: 201 -> 154 us).
constexpr int kBStage = 48;

__global__ void __launch_bounds__(kFrnnThreads, kFrnnBlocks) k_bgrid_frnn(int n, const float2* __restrict__ spos,
                                                            const int* __restrict__ src, const int* __restrict__ vcomp,
                                                            const int4* __restrict__ par, const float* __restrict__ rc,
                                                            float lo, const int* __restrict__ start, int F,
                                                            int* __restrict__ out, unsigned long long* overflow) {
  extern __shared__ int bstage[];
  const int t = threadIdx.x, lane = t & 31, i = blockIdx.x * kFrnnThreads + t;
  const int cap = F - 1;        // <= kBStage (checked by the host)
  const int len = F | 1;        // one more than cap, and odd
  int* mine = bstage + t * len;
  int nf = 0, v = 0;
  if (i < n) {
    v = __ldg(src + i);
    const int mesh = vcomp ? __ldg(vcomp + v) : 0;
    const int4 q = __ldg(par + mesh);
    const float c = __int_as_float(q.x), inv = 1.0f / c;
    const float r = __ldg(rc + mesh);
    const float r2 = __fmul_rn(r, r);
    const float2 p = spos[i];
    const unsigned long long minus_p = pair_of(-p.x, -p.y);
    const int nx = q.y;
    const float mg = 1e-3f * c + 1e-5f * (fabsf(p.x) + fabsf(p.y) + fabsf(lo) + r);
    const float px = p.x - lo, py = p.y - lo;
    int ylo = (int)floorf(fmaxf(fminf((py - r - mg) * inv, 1e9f), -1e9f));
    int yhi = (int)floorf(fmaxf(fminf((py + r + mg) * inv, 1e9f), -1e9f));
    ylo = ylo < 0 ? 0 : (ylo >= nx ? nx - 1 : ylo);
    yhi = yhi < 0 ? 0 : (yhi >= nx ? nx - 1 : yhi);
    for (int yy = ylo; yy <= yhi; ++yy) {
      float slo = yy * c, shi = slo + c;
      if (yy == 0) slo = -INFINITY;
      if (yy == nx - 1) shi = INFINITY;
      const float dym = fmaxf(fmaxf(slo - py, py - shi) - mg, 0.f);
      const float hw = near_sqrt(fmaxf(r2 - dym * dym, 0.f)) * 1.0001f + mg;
      int xlo = (int)floorf(fmaxf(fminf((px - hw) * inv, 1e9f), -1e9f));
      int xhi = (int)floorf(fmaxf(fminf((px + hw) * inv, 1e9f), -1e9f));
      xlo = xlo < 0 ? 0 : (xlo >= nx ? nx - 1 : xlo);
      xhi = xhi < 0 ? 0 : (xhi >= nx ? nx - 1 : xhi);
      const int* row = start + q.z + yy * nx;
      const int b = __ldg(row + xlo), e = __ldg(row + xhi + 1);
      const unsigned long long* at = reinterpret_cast<const unsigned long long*>(spos);
      if (nf + (e - b) <= cap) {
#pragma unroll 4
        for (int j = b; j < e; ++j) {
          const bool hit = (pair_norm2(pair_add(at[j], minus_p)) <= r2) & (j != i);
          mine[nf] = j;
          nf += hit ? 1 : 0;
        }
      } else {
        for (int j = b; j < e; ++j) {
          if ((pair_norm2(pair_add(at[j], minus_p)) <= r2) & (j != i)) {
            if (nf < cap) mine[nf] = j;
            ++nf;
          }
        }
      }
    }
    if (nf > cap) atomicAdd(overflow, 1ull);
    const int m = nf < cap ? nf : cap;
    // vertex ids, ascending
    for (int a = 0; a < m; ++a) mine[a] = __ldg(src + mine[a]);
    for (int a = 1; a < m; ++a) {
      const int x = mine[a];
      int bb = a - 1;
      while (bb >= 0 && mine[bb] > x) { mine[bb + 1] = mine[bb]; --bb; }
      mine[bb + 1] = x;
    }
    nf = m;
  } else {
    nf = -1;
  }
  __syncwarp();
  const int* theirs = bstage + (t & ~31) * len;
#pragma unroll 4
  for (int rr = 0; rr < 32; ++rr) {
    const int cr = __shfl_sync(0xffffffffu, nf, rr), to = __shfl_sync(0xffffffffu, v, rr);
    int* dst = out + (size_t)to * F;
    const int* from = theirs + rr * len;
    if (lane == 0 && cr >= 0) dst[0] = cr;
    for (int k = lane; k < cr; k += 32) dst[k + 1] = from[k];
  }
}

}  // namespace

extern "C" int mcl_batch_frnn_grid(mcl_mesh* m, const float* r_host, const float* r_dev, float lo, float hi,
                                   int max_frnn, int32_t* out_dev, void* stream, int64_t* overflow) {
  if (!m || !r_host || !r_dev || !out_dev || !(hi > lo) || max_frnn < 2)
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  if (max_frnn - 1 > kBStage) return qfail(MCL_ERR_CAPACITY, "mcl_batch_frnn_grid: max_frnn above 49");
  if (m->nact) return qfail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_frnn_grid: runs over every mesh of the batch");
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nc = m->ncomp, V = m->V;
  // per-mesh grids: cells of the mesh's radius, at most 4096 per side
  std::vector<int4> par((size_t)nc);
  int64_t cells = 0;
  for (int64_t c = 0; c < nc; ++c) {
    const float r = r_host[c];
    if (!(r > 0.f)) return qfail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_frnn_grid: radius must be positive");
    int side = (int)std::min<double>(4096.0, std::ceil((double)(hi - lo) / r));
    side = std::max(side, 1);
    float cell = (hi - lo) / (float)side;
    if (cell < r) cell = r;  // a cell never narrower than the radius
    int v;
    std::memcpy(&v, &cell, 4);
    par[(size_t)c] = make_int4(v, side, (int)cells, 0);
    cells += (int64_t)side * side;
    if (cells > (1ll << 30)) return qfail(MCL_ERR_CAPACITY, "mcl_batch_frnn_grid: more than 2^30 cells");
  }
  if (!m->bg_cell) {
    auto A = [&](void** p, size_t b) { return cudaMalloc(p, b) == cudaSuccess; };
    if (!A((void**)&m->bg_cell, 4 * V) || !A((void**)&m->bg_src, 4 * V) || !A((void**)&m->bg_rank, 4 * V) || !A((void**)&m->bg_bucket, 4 * V) ||
        !A((void**)&m->bg_pos, 8 * V) || !A((void**)&m->bg_par, sizeof(int4) * nc) ||
        cudaMallocHost((void**)&m->bg_par_host, sizeof(int4) * nc) != cudaSuccess)
      return qfail(MCL_ERR_OUT_OF_MEMORY, "mcl_batch_frnn_grid: point tables");
  }
  if (m->bg_cap < cells) {
    if (m->bg_count) { cudaFree(m->bg_count); cudaFree(m->bg_start); cudaFree(m->bg_local); cudaFree(m->bg_pre); }
    m->bg_count = m->bg_start = m->bg_local = m->bg_pre = nullptr;
    const int64_t nb = (cells + kScanCells - 1) / kScanCells;
    if (cudaMalloc((void**)&m->bg_count, 4 * (cells + 1)) != cudaSuccess ||
        cudaMalloc((void**)&m->bg_start, 4 * (cells + 1)) != cudaSuccess ||
        cudaMalloc((void**)&m->bg_local, 4 * cells) != cudaSuccess ||
        cudaMalloc((void**)&m->bg_pre, 4 * nb) != cudaSuccess) {
      m->bg_cap = 0;
      return qfail(MCL_ERR_OUT_OF_MEMORY, "mcl_batch_frnn_grid: cell tables");
    }
    m->bg_cap = cells;
  }
  // the parameters are uploaded only when they change, from a pinned buffer the
  // mesh keeps (a call captured in a CUDA graph then holds no host copy, or
  // reads memory that outlives the call)
  if (m->bg_cells != cells || std::memcmp(m->bg_par_host, par.data(), sizeof(int4) * nc) != 0) {
    QCK(cudaStreamSynchronize(s));  // the previous upload has been read
    std::memcpy(m->bg_par_host, par.data(), sizeof(int4) * nc);
    QCK(cudaMemcpyAsync(m->bg_par, m->bg_par_host, sizeof(int4) * nc, cudaMemcpyHostToDevice, s));
    m->bg_cells = cells;
  }
  const float2* pos = m->pos[m->cur];
  const int Vi = (int)V;
  QCK(cudaMemsetAsync(m->bg_count, 0, 4 * (cells + 1), s));
  k_bgrid_hash<<<(Vi + 255) / 256, 256, 0, s>>>(Vi, pos, m->vfix, m->vcomp, m->bg_par, lo, m->bg_cell, m->bg_count,
                                                m->bg_rank, out_dev, max_frnn);
  const int npts = (int)(V - 4 * nc);
  launch_cells(Vi, npts, cells, m->bg_cell, m->bg_count, m->bg_count + cells, m->bg_rank, m->bg_local, m->bg_pre,
               m->bg_bucket, pos, nullptr, m->bg_start, nullptr, m->bg_src, m->bg_pos, nullptr, s);
  unsigned long long* ovf = m->scratch + 4;
  QCK(cudaMemsetAsync(ovf, 0, 8, s));
  k_bgrid_frnn<<<(unsigned)((npts + kFrnnThreads - 1) / kFrnnThreads), kFrnnThreads,
                 sizeof(int) * kFrnnThreads * (max_frnn | 1), s>>>(npts, m->bg_pos, m->bg_src, m->vcomp, m->bg_par,
                                                                   r_dev, lo, m->bg_start, max_frnn, out_dev, ovf);
  QCK(cudaGetLastError());
  if (overflow) {
    unsigned long long t = 0;
    QCK(cudaMemcpyAsync(&t, ovf, 8, cudaMemcpyDeviceToHost, s));
    QCK(cudaStreamSynchronize(s));
    *overflow = (int64_t)t;
  }
  return MCL_OK;
}

// ---------------------------------------------------------------------------
// Grid neighbours without allocation.
//
// Some callers cannot allocate device memory at all: host frameworks that
// reserve the whole GPU up front and hand memory out only through their own
// pool, and real-time loops that must never block in an allocator.  For them
// this variant of GridCount2d::update + apply_f_frnn keeps its scratch (cell
// tables and per-point work arrays) in one fixed array that lives in the
// library's device image, so the call itself allocates nothing.  Limits:
// at most kNoAllocMaxPoints points and kNoAllocMaxCells cell-table entries
// (cells_x * cells_y, row-major cells as mcl_grid_create).  Every GPU that loads the
// library holds these 6.3 MB until the process exits.
constexpr int64_t kNoAllocMaxPoints = 262144;
constexpr int64_t kNoAllocMaxCells = 262144;
constexpr int64_t kNoAllocWords = 3 * kNoAllocMaxPoints + 3 * kNoAllocMaxCells + kNoAllocMaxCells / kScanCells + 64;
static __device__ __align__(256) int g_noalloc_scratch[kNoAllocWords];

namespace {
int* g_noalloc_ptr[64];  // device address of the scratch array, per device id
std::mutex g_noalloc_mutex;

int noalloc_scratch(int** out) {
  int dev = 0;
  QCK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return qfail(MCL_ERR_NO_DEVICE, "device id out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return qfail(MCL_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_noalloc_ptr[dev] = static_cast<int*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return MCL_OK;
}
}  // namespace

extern "C" int mcl_grid_frnn_noalloc(const mcl_float2* pos, int64_t n, float min_x, float min_y, float cell_x,
                                     float cell_y, int32_t cells_x, int32_t cells_y, int flags, float r, int max_nb,
                                     mcl_float2* sorted_pos, int32_t* perm, int32_t* counts, int32_t* ids,
                                     void* stream, int64_t* overflow) {
  if (!pos || !sorted_pos || !perm || !counts || !ids || n < 0 || cells_x < 1 || cells_y < 1 || max_nb < 1 ||
      !(cell_x > 0.f) || !(cell_y > 0.f) || !(r >= 0.f))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  const int morton = 0;  // row-major cells, as mcl_grid_create
  const int64_t ncells = (int64_t)cells_x * cells_y;
  if (n > kNoAllocMaxPoints)
    return qfail(MCL_ERR_CAPACITY, "mcl_grid_frnn_noalloc: more than 262144 points");
  if (ncells > kNoAllocMaxCells)
    return qfail(MCL_ERR_CAPACITY, "mcl_grid_frnn_noalloc: cell table larger than 262144 entries");
  if (n == 0) return MCL_OK;
  int* base = nullptr;
  const int rc = noalloc_scratch(&base);
  if (rc != MCL_OK) return rc;
  int* cell = base;
  int* src = cell + kNoAllocMaxPoints;
  int* count = src + kNoAllocMaxPoints;
  int* local = count + kNoAllocMaxCells + 4;  // the scan's ticket behind the counts
  int* bucket = local + kNoAllocMaxCells;
  int* pre = bucket + kNoAllocMaxPoints;
  int* start = pre + kNoAllocMaxCells / kScanCells;
  unsigned long long* ovf = reinterpret_cast<unsigned long long*>(start + kNoAllocMaxCells + 4);
  cudaStream_t s = (cudaStream_t)stream;
  GridView G;
  G.minx = min_x; G.miny = min_y; G.cx = cell_x; G.cy = cell_y;
  G.nx = cells_x; G.ny = cells_y; G.morton = morton; G.periodic = (flags & MCL_GRID_PERIODIC) ? 1 : 0;
  const int nn = (int)n;
  // the array keeps the previous call's contents: clear what must start at zero
  int* ticket = count + ncells;
  QCK(cudaMemsetAsync(count, 0, 4 * (ncells + 1), s));
  QCK(cudaMemsetAsync(ovf, 0, 8, s));
  k_grid_hash<<<(nn + 255) / 256, 256, 0, s>>>(G, nn, (const float2*)pos, cell, count, perm, nullptr);
  launch_cells(nn, nn, ncells, cell, count, ticket, perm, local, pre, bucket, (const float2*)pos, nullptr, start, perm,
               src, (float2*)sorted_pos, nullptr, s);
  const int rc2 = launch_grid_frnn(G, nn, (const float2*)sorted_pos, start, r, cell_x * cells_x,
                                   cell_y * cells_y, max_nb, counts, ids, ovf, nullptr, s, nullptr);
  if (rc2 != MCL_OK) return rc2;
  if (overflow) {
    unsigned long long t = 0;
    QCK(cudaMemcpyAsync(&t, ovf, 8, cudaMemcpyDeviceToHost, s));
    QCK(cudaStreamSynchronize(s));
    *overflow = (int64_t)t;
  }
  return MCL_OK;
}

// ---------------------------------------------------------------------------
// The reference's AoS mesh arrays written on the device (DeviceTriangulation's
// public m_v / m_he / m_t, include/Device_Triangulation.h:139-142), in the
// layout and face numbering of mcl_mesh_download_aos: faces numbered in the
// order of their smallest half-edge.
namespace {

__device__ __forceinline__ bool aos_owner(const int4* ev, const int4* en, int64_t h, int* nxt, int* prv) {
  const int4 q = ev[h >> 1], w = en[h >> 1];
  const bool odd = h & 1;
  const int org = odd ? q.y : q.x, apex = odd ? q.w : q.z;
  *nxt = odd ? w.z : w.x;
  *prv = odd ? w.w : w.y;
  return apex >= 0 && org >= 0;
}

__global__ void k_aos_flags(const int4* ev, const int4* en, int64_t HE, int* flag) {
  const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= HE) return;
  int n, p;
  const bool inner = aos_owner(ev, en, h, &n, &p);
  flag[h] = inner && h < n && h < p ? 1 : 0;
}

__global__ void k_aos_write(const int4* ev, const int4* en, const int* vhe, int64_t V, int64_t HE, const int* fid,
                            int* v, int* he, int* t) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < HE) {
    int n, p;
    const bool inner = aos_owner(ev, en, i, &n, &p);
    const int4 q = ev[i >> 1];
    const bool odd = i & 1;
    const int org = odd ? q.y : q.x, apex = odd ? q.w : q.z;
    int face = -1;
    if (inner) {
      const int64_t f = min(i, (int64_t)min(n, p));
      if (f >= 0 && f < HE) face = fid[f];
      if (t && i < n && i < p) t[fid[i]] = (int)i;
    }
    if (he) *reinterpret_cast<int4*>(he + 4 * i) = make_int4(n, org, face, apex >= 0 ? apex : -1);
  }
  if (v && i < V) *reinterpret_cast<int2*>(v + 2 * i) = make_int2((int)i, vhe[i]);
}

}  // namespace

extern "C" int mcl_mesh_export_aos(mcl_mesh* m, int32_t* v_dev, int32_t* he_dev, int32_t* t_dev, void* stream) {
  if (!m) return qfail(MCL_ERR_INVALID_ARGUMENT, "mcl_mesh_export_aos: null mesh");
  if (((uintptr_t)v_dev & 7) || ((uintptr_t)he_dev & 15))
    return qfail(MCL_ERR_INVALID_ARGUMENT, "mcl_mesh_export_aos: m_v must be 8-byte and m_he 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t HE = 2 * m->E, nb = (HE + 1023) / 1024;
  const int64_t need = 2 * HE + 2 * (nb + 2);
  if (m->aos_cap < need) {
    if (m->aos_tmp) QCK(cudaFree(m->aos_tmp));
    m->aos_tmp = nullptr;
    m->aos_cap = 0;
    if (cudaMalloc((void**)&m->aos_tmp, 4 * need) != cudaSuccess) {
      (void)cudaGetLastError();
      return qfail(MCL_ERR_OUT_OF_MEMORY, "mcl_mesh_export_aos: scratch");
    }
    m->aos_cap = need;
  }
  int* flag = m->aos_tmp;
  int* fid = flag + HE;
  int* tmp = fid + HE;
  const unsigned gb = (unsigned)((std::max(HE, m->V) + 255) / 256);
  k_aos_flags<<<(unsigned)((HE + 255) / 256), 256, 0, s>>>(m->ev, m->en, HE, flag);
  const int rc = scan_exclusive(flag, fid, HE, tmp, tmp + nb + 1, s);
  if (rc != MCL_OK) return rc;
  k_aos_write<<<gb, 256, 0, s>>>(m->ev, m->en, m->vhe, m->V, HE, fid, v_dev, he_dev, t_dev);
  QCK(cudaGetLastError());
  return MCL_OK;
}
