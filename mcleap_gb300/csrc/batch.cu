// Batches of independent meshes, motion models and settling of coincident moves.
//
// A batch is one mcl_mesh whose connected components are the meshes: their
// vertex and edge records are concatenated (ids offset), each keeps its own
// bounding square, and nothing links two components.  Every kernel of the
// engine walks the topology, so it never leaves a component; the one place
// that needs a starting half-edge by id (point location after a removal) falls
// back to the component's own half-edge 0 (vroot).  One cooperative launch of
// the kinetic step therefore steps every mesh of the batch.
//
// Motion:
//   mcl_walk           Gaussian random walk with a per-mesh sigma, clamped to
//                      a box, optionally only for unfrozen walkers (the
//                      diffusion-limited-aggregation motion of
//                      experiments/diffusion_limited_aggregation.cu:51-60,
//                      263-268 in the reference).
//   mcl_settle_moves   refuses moves that would make two vertices of one mesh
//                      coincide (the triangulation of coincident points is
//                      undefined); see the rule below.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "engine.cuh"

namespace cg = cooperative_groups;
using namespace mcl;

namespace {

#define BCK(call)                                    \
  do {                                               \
    cudaError_t _e = (call);                         \
    if (_e != cudaSuccess) return cuda_fail(_e, #call); \
  } while (0)

// ---------------------------------------------------------------------------
// Batch assembly: copy one mesh's records into the batch with offset ids.
__global__ void k_append(int V, int E, const float2* pos, const int4* ev, const int4* en, const int* vhe,
                         const unsigned char* vfix, int vb, int eb, int comp, float2* pos0, float2* pos1, int4* ev_o,
                         int4* en_o, int* vhe_o, unsigned char* vfix_o, int* vcomp, int* vroot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int hb = 2 * eb;
  if (i < E) {
    const int4 q = ev[i];
    ev_o[eb + i] = make_int4(q.x < 0 ? -1 : q.x + vb, q.y < 0 ? -1 : q.y + vb, q.z < 0 ? -1 : q.z + vb,
                             q.w < 0 ? -1 : q.w + vb);
    const int4 n = en[i];
    en_o[eb + i] = make_int4(n.x < 0 ? -1 : n.x + hb, n.y < 0 ? -1 : n.y + hb, n.z < 0 ? -1 : n.z + hb,
                             n.w < 0 ? -1 : n.w + hb);
  }
  if (i < V) {
    const float2 p = pos[i];
    pos0[vb + i] = p;
    pos1[vb + i] = p;
    const int h = vhe[i];
    vhe_o[vb + i] = h < 0 ? -1 : h + hb;
    vfix_o[vb + i] = vfix[i];
    vcomp[vb + i] = comp;
    vroot[vb + i] = hb;
  }
}

// ---------------------------------------------------------------------------
// Counter-based random numbers: SplitMix64's finaliser (Steele, Lea and Flood,
// "Fast splittable pseudorandom number generators", 2014) over
// (seed, step, vertex, draw); uniforms in (0, 1] from the top 24 bits; normal
// pairs by the Box-Muller transform.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ float2 normal2(unsigned long long seed, unsigned long long step, int v) {
  const unsigned long long a = mix64(seed ^ mix64(step * 0x100000001B3ull + (unsigned long long)v));
  const float u1 = ((unsigned)(a >> 40) + 1u) * (1.0f / 16777216.0f);  // (0, 1]
  const float u2 = ((unsigned)(a >> 16) & 0xFFFFFFu) * (1.0f / 16777216.0f);
  const float rad = sqrtf(-2.0f * logf(u1));
  float s, c;
  sincospif(2.0f * u2, &s, &c);
  return make_float2(rad * c, rad * s);
}

// d[v] = clamp(pos + sigma * N(0, I), lo, hi) - pos for free, unfrozen vertices;
// a displacement whose rounded sum would leave [lo, hi] is dropped.
// The draws of vertex v of mesh c are keyed by (seed + c, local id of v), so a
// mesh draws the same numbers alone (with seed + c) and inside a batch.
__global__ void k_walk(ActV A, const float2* __restrict__ pos, const unsigned char* __restrict__ vfix,
                       const int* __restrict__ vcomp, const int* __restrict__ cbase, const float* __restrict__ sigma,
                       const unsigned char* __restrict__ frozen, unsigned long long seed,
                       const unsigned long long* __restrict__ seeds,
                       const unsigned long long* __restrict__ counter, float lo, float hi, float2* __restrict__ d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.V_it) return;
  const int v = A.at(i);
  float2 out = make_float2(0.f, 0.f);
  if (!vfix[v] && !(frozen && frozen[v])) {
    const int c = vcomp ? vcomp[v] : 0;
    const float sg = sigma[c];
    const float2 z = normal2(seeds ? seeds[c] : seed + (unsigned long long)c, counter[c], cbase ? v - cbase[c] : v);
    const float2 p = pos[v];
    const float tx = fminf(fmaxf(__fadd_rn(p.x, __fmul_rn(sg, z.x)), lo), hi);
    const float ty = fminf(fmaxf(__fadd_rn(p.y, __fmul_rn(sg, z.y)), lo), hi);
    out = make_float2(__fsub_rn(tx, p.x), __fsub_rn(ty, p.y));
    const float nx = __fadd_rn(p.x, out.x), ny = __fadd_rn(p.y, out.y);
    if (!(nx >= lo && nx <= hi)) out.x = 0.f;
    if (!(ny >= lo && ny <= hi)) out.y = 0.f;
  }
  d[v] = out;
}

// counter[c] += 1 for every active mesh c (every mesh when n == 0)
__global__ void k_advance(unsigned long long* counter, int n, const int* act, int ncomp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (n ? i < n : i < ncomp) counter[n ? act[i] : i] += 1;
}

// ---------------------------------------------------------------------------
// Settling coincident moves.
//
// Rule (a least fixed point, independent of thread order): start with every
// vertex at pos + d; while two vertices of one mesh sit at the same point,
// every MOVING vertex among them (d != 0) is sent back to pos (its d zeroed).
// Old positions are distinct, so the loop ends with distinct positions; a
// vertex that did not move never yields.
//
// Only a pair with a mover can coincide.  Each pass inserts the movers' candidate
// positions into an open-addressing table keyed by (mesh, x, y); a mover whose
// position is already there marks itself and the holder.  After a grid barrier every
// other vertex of a mesh that has a mover looks its position up (one read of an empty
// slot, as a rule) and marks the holder.  The marked movers, listed, are sent back.
// What can coincide after that is a mover with a vertex just sent back, so each
// further pass looks up the old positions of the last list alone, until none is
// marked.  (Slots are not freed: a holder is compared at the position it has now.)
//
// What bounds it is one scattered atomic per mover and one scattered read per other
// vertex: four vertices a thread keep four of them in flight.  The table holds ids
// alone (4 bytes, four slots per vertex, emptied before the call), so an insertion
// is one compare-and-swap; with stamped entries that are never cleared it was a read
// and a swap, after a pass that looked for meshes with movers, with the static
// vertices inserted too (with the clearing: 1M vertices, all moving 125 -> 58 us, 2 % of
// them 94 -> 40; 200,000 in one mesh 61 -> 31, in 64 meshes 97 -> 42).
__device__ __forceinline__ unsigned fbits(float x) { return x == 0.f ? 0u : __float_as_uint(x); }

__device__ __forceinline__ float2 cand_pos(const float2* pos, const float2* d, const unsigned char* vfix, int v) {
  const float2 p = pos[v];
  if (vfix[v]) return p;
  const float2 q = d[v];
  return make_float2(__fadd_rn(p.x, q.x), __fadd_rn(p.y, q.y));
}

struct SettleArgs {
  ActV A;
  const float2* pos;
  float2* d;
  const unsigned char* vfix;
  const int* vcomp;
  int* table;              // kNoVertex: empty
  unsigned mask;
  int* smark;
  int* list0;              // the movers to send back, per pass (two in turn)
  int* list1;
  unsigned* smove;         // per mesh: stamp of the call if it has a mover
  DevState* st;
  int max_passes;
};
constexpr int kNoVertex = -1;
constexpr int kSettleUnroll = 4;

__device__ __forceinline__ unsigned settle_slot(float2 p, int comp, unsigned mask) {
  const unsigned long long key = ((unsigned long long)fbits(p.x) << 32) | fbits(p.y);
  return (unsigned)mix64(key ^ ((unsigned long long)comp * 0x9E3779B97F4A7C15ull)) & mask;
}
__device__ __forceinline__ bool settle_same(const SettleArgs& A, int u, float2 p, int comp) {
  const float2 q = cand_pos(A.pos, A.d, A.vfix, u);
  return (A.vcomp ? A.vcomp[u] : 0) == comp && fbits(q.x) == fbits(p.x) && fbits(q.y) == fbits(p.y);
}

// A mover that coincides joins the pass's list once.
__device__ __forceinline__ void settle_mark(const SettleArgs& A, int v, unsigned stamp, int pass) {
  if ((unsigned)atomicExch(A.smark + v, (int)stamp) == stamp) return;
  const unsigned at = atomicAdd(A.st->settle + 1 + pass % 3, 1u);
  __stcg((pass & 1 ? A.list1 : A.list0) + at, v);  // at most one entry per vertex and pass
}

// words: [0] last stamp used, [1..3] listed per pass (triple-buffered), [4] sent back,
// [5] status
__global__ void __launch_bounds__(256) k_settle(SettleArgs A) {
  cg::grid_group g = cg::this_grid();
  const int stride = gridDim.x * blockDim.x;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned* words = A.st->settle;
  const unsigned base = (unsigned)ld_i(reinterpret_cast<const int*>(words));
  constexpr int U = kSettleUnroll;
  unsigned stamp = base + 1;
  bool lost = false;
  // the mesh that this block has last stamped for the j-th vertices of its threads: without
  // it the first wave's warps all stamp the few meshes there are (29,000 stores to one
  // address, 60 us)
  __shared__ int s_stamped[U];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < U) s_stamped[threadIdx.x] = -1;
  if (gtid == 0) words[2] = 0;
  __syncthreads();
  for (int first0 = gtid - lane; first0 < A.A.V_it; first0 += stride * U) {
    const int first = first0 + lane;
    int v[U], comp[U], holder[U];
    unsigned h[U];
    float2 p[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int vi = first + j * stride;
      v[j] = vi < A.A.V_it ? A.A.at(vi) : -1;
      holder[j] = kNoVertex;
      if (v[j] < 0) continue;
      const float2 q = A.d[v[j]], o = A.pos[v[j]];
      if (A.vfix[v[j]] || (q.x == 0.f && q.y == 0.f)) { v[j] = -1; continue; }
      p[j] = make_float2(__fadd_rn(o.x, q.x), __fadd_rn(o.y, q.y));
      comp[j] = A.vcomp ? A.vcomp[v[j]] : 0;
      h[j] = settle_slot(p[j], comp[j], A.mask);
    }
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (v[j] >= 0) holder[j] = atomicCAS(A.table + h[j], kNoVertex, v[j]);
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int c = v[j] >= 0 ? comp[j] : -1;
      const unsigned same = __match_any_sync(0xffffffffu, c);
      if (c >= 0 && __ffs((int)same) - 1 == lane && atomicExch(s_stamped + j, c) != c &&
          (unsigned)ld_i(reinterpret_cast<const int*>(A.smove) + c) != stamp)
        __stcg(A.smove + c, stamp);
      if (c < 0) continue;
      unsigned it = 0;
      while (holder[j] != kNoVertex) {
        if (settle_same(A, holder[j], p[j], comp[j])) {
          settle_mark(A, v[j], stamp, 0);
          settle_mark(A, holder[j], stamp, 0);
          break;
        }
        if (++it > A.mask) { lost = true; break; }
        h[j] = (h[j] + 1) & A.mask;
        holder[j] = atomicCAS(A.table + h[j], kNoVertex, v[j]);
      }
    }
  }
  g.sync();
  for (int first = gtid; first < A.A.V_it; first += stride * U) {
    int v[U], comp[U], holder[U];
    unsigned h[U];
    float2 p[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int vi = first + j * stride;
      v[j] = vi < A.A.V_it ? A.A.at(vi) : -1;
      holder[j] = kNoVertex;
      if (v[j] < 0) continue;
      const float2 q = A.d[v[j]];
      const bool fixed = A.vfix[v[j]] != 0;
      if (!fixed && (q.x != 0.f || q.y != 0.f)) continue;
      comp[j] = A.vcomp ? A.vcomp[v[j]] : 0;
      if (A.smove[comp[j]] != stamp) continue;  // through L1: nothing is stamped any more
      p[j] = A.pos[v[j]];
      h[j] = settle_slot(p[j], comp[j], A.mask);
      holder[j] = ld_i(A.table + h[j]);
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      unsigned it = 0;
      while (holder[j] != kNoVertex) {
        if (settle_same(A, holder[j], p[j], comp[j])) {
          settle_mark(A, holder[j], stamp, 0);
          break;
        }
        if (++it > A.mask) { lost = true; break; }
        h[j] = (h[j] + 1) & A.mask;
        holder[j] = ld_i(A.table + h[j]);
      }
    }
  }
  if (lost) atomicOr(words + 5, 2u);
  g.sync();
  int pass = 0;
  for (; pass < A.max_passes; ++pass) {
    const int n = ld_i(reinterpret_cast<const int*>(words) + 1 + pass % 3);
    if (n == 0 || ld_i(reinterpret_cast<const int*>(words + 5))) break;
    const int* list = pass & 1 ? A.list1 : A.list0;
    if (gtid == 0) words[1 + (pass + 2) % 3] = 0;
    int sent = 0;
    for (int i = gtid; i < n; i += stride) {
      __stcg(A.d + ld_i(list + i), make_float2(0.f, 0.f));
      ++sent;
    }
    if (sent) atomicAdd(words + 4, (unsigned)sent);
    g.sync();
    ++stamp;
    for (int i = gtid; i < n; i += stride) {
      const int v = ld_i(list + i), comp = A.vcomp ? A.vcomp[v] : 0;
      const float2 p = A.pos[v];
      unsigned h = settle_slot(p, comp, A.mask);
      int u;
      for (unsigned it = 0; it <= A.mask && (u = ld_i(A.table + h)) != kNoVertex; ++it) {
        const float2 q = __ldcg(A.d + u);
        if ((q.x != 0.f || q.y != 0.f) && settle_same(A, u, p, comp)) {
          settle_mark(A, u, stamp, pass + 1);
          break;
        }
        h = (h + 1) & A.mask;
      }
    }
    g.sync();
  }
  if (gtid == 0) {
    words[0] = base + 1 + (unsigned)A.max_passes;  // the next call's stamps are fresh
    if (pass >= A.max_passes) words[5] |= 1u;
  }
}

int ensure_settle_scratch(mcl_mesh* m) {
  if (m->table) return MCL_OK;
  int64_t size = 1;
  while (size < 4 * m->V && size < (1ll << 31)) size <<= 1;
  BCK(cudaMalloc((void**)&m->table, 4 * size));
  BCK(cudaMalloc((void**)&m->smark, 4 * m->V));
  BCK(cudaMalloc((void**)&m->smove, 4 * std::max<int64_t>(1, m->ncomp)));
  BCK(cudaMemset(m->smark, 0, 4 * m->V));
  BCK(cudaMemset(m->smove, 0xFF, 4 * std::max<int64_t>(1, m->ncomp)));
  m->table_size = size;
  int per_sm = 0;
  BCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_settle, 256, 0));
  if (per_sm < 1) return fail(MCL_ERR_CUDA, "k_settle cannot be resident");
  m->settle_blocks = m->nsm * std::min(per_sm, 6);
  return MCL_OK;
}

}  // namespace

extern "C" {

int mcl_batch_create(mcl_mesh* const* meshes, int64_t count, mcl_mesh** out) {
  if (!meshes || !out || count < 1) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_create: no meshes");
  int64_t V = 0, E = 0;
  for (int64_t i = 0; i < count; ++i) {
    if (!meshes[i]) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_create: null mesh");
    if (meshes[i]->ncomp != 1) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_create: nested batch");
    V += meshes[i]->V;
    E += meshes[i]->E;
  }
  if (V > (1ll << 30) || E > (1ll << 29))
    return fail(MCL_ERR_CAPACITY, "mcl_batch_create: more than 2^30 vertices or 2^29 edges in one batch");
  mcl_mesh* b = nullptr;
  int rc = alloc_mesh(V, E, &b);
  if (rc != MCL_OK) return rc;
  auto bail = [&](int code) {
    free_mesh(b);
    return code;
  };
  if (cudaMalloc((void**)&b->vcomp, 4 * V) != cudaSuccess || cudaMalloc((void**)&b->vroot, 4 * V) != cudaSuccess ||
      cudaMalloc((void**)&b->cbase, 4 * (count + 1)) != cudaSuccess ||
      cudaMalloc((void**)&b->cebase, 4 * count) != cudaSuccess)
    return bail(fail(MCL_ERR_OUT_OF_MEMORY, "mcl_batch_create: component tables"));
  b->ncomp = count;
  b->square = true;
  b->comp_host = new int64_t[4 * count];
  std::vector<int> base((size_t)count + 1), ebase((size_t)count);
  b->T = 0;
  int64_t vb = 0, eb = 0;
  for (int64_t i = 0; i < count; ++i) {
    mcl_mesh* m = meshes[i];
    b->comp_host[4 * i] = vb;
    base[(size_t)i] = (int)vb;
    ebase[(size_t)i] = (int)eb;
    b->comp_host[4 * i + 1] = m->V;
    b->comp_host[4 * i + 2] = eb;
    b->comp_host[4 * i + 3] = m->E;
    const int n = (int)std::max(m->V, m->E);
    k_append<<<(n + 255) / 256, 256>>>((int)m->V, (int)m->E, valid_positions(m), m->ev, m->en, m->vhe, m->vfix,
                                       (int)vb, (int)eb, (int)i, b->pos[0], b->pos[1], b->ev, b->en, b->vhe, b->vfix,
                                       b->vcomp, b->vroot);
    if (cudaGetLastError() != cudaSuccess) return bail(fail(MCL_ERR_CUDA, "mcl_batch_create: append"));
    b->T += m->T;
    b->square = b->square && m->square;
    vb += m->V;
    eb += m->E;
  }
  base[(size_t)count] = (int)vb;
  if (cudaMemcpy(b->cbase, base.data(), 4 * (count + 1), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(b->cebase, ebase.data(), 4 * count, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaDeviceSynchronize() != cudaSuccess)
    return bail(fail(MCL_ERR_CUDA, "mcl_batch_create: sync"));
  b->dirty = new unsigned char[(size_t)count]();
  b->act_list = new int[(size_t)count];
  if (cudaMalloc((void**)&b->act_dev, 4 * (5 * count + 2)) != cudaSuccess ||
      cudaMallocHost((void**)&b->act_host, 4 * (5 * count + 2)) != cudaSuccess)
    return bail(fail(MCL_ERR_OUT_OF_MEMORY, "mcl_batch_create: active tables"));
  b->cur = 0;
  b->valid_cur = true;
  *out = b;
  return MCL_OK;
}

int mcl_batch_count(const mcl_mesh* m, int64_t* count) {
  if (!m || !count) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  *count = m->ncomp;
  return MCL_OK;
}

int mcl_batch_range(const mcl_mesh* m, int64_t i, int64_t* v0, int64_t* nv, int64_t* e0, int64_t* ne) {
  if (!m || i < 0 || i >= m->ncomp) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_range: bad mesh index");
  const int64_t* c = m->comp_host ? m->comp_host + 4 * i : nullptr;
  if (v0) *v0 = c ? c[0] : 0;
  if (nv) *nv = c ? c[1] : m->V;
  if (e0) *e0 = c ? c[2] : 0;
  if (ne) *ne = c ? c[3] : m->E;
  return MCL_OK;
}

int mcl_batch_vertex_mesh(const mcl_mesh* m, const int32_t** vcomp_dev) {
  if (!m || !vcomp_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  *vcomp_dev = m->vcomp;
  return MCL_OK;
}

int mcl_batch_download_aos(mcl_mesh* m, int64_t i, mcl_float2* pos, int32_t* v, int32_t* he, int32_t* t) {
  int64_t v0 = 0, nv = 0, e0 = 0, ne = 0;
  const int rc = mcl_batch_range(m, i, &v0, &nv, &e0, &ne);
  if (rc != MCL_OK) return rc;
  return download_range(m, v0, nv, e0, ne, 2 * (nv - 4) + 2, pos, v, he, t);
}

int mcl_mesh_clone(const mcl_mesh* src, mcl_mesh** out) {
  if (!src || !out) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  mcl_mesh* m = nullptr;
  int rc = alloc_mesh(src->V, src->E, &m);
  if (rc != MCL_OK) return rc;
  const int64_t V = src->V, E = src->E;
  cudaError_t e = cudaMemcpy(m->pos[0], valid_positions(src), 8 * V, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(m->pos[1], valid_positions(src), 8 * V, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(m->ev, src->ev, 16 * E, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(m->en, src->en, 16 * E, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(m->vhe, src->vhe, 4 * V, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(m->vfix, src->vfix, V, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess && src->vcomp) {
    e = cudaMalloc((void**)&m->vcomp, 4 * V);
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->vroot, 4 * V);
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->cbase, 4 * (src->ncomp + 1));
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->cebase, 4 * src->ncomp);
    if (e == cudaSuccess) e = cudaMemcpy(m->vcomp, src->vcomp, 4 * V, cudaMemcpyDeviceToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->vroot, src->vroot, 4 * V, cudaMemcpyDeviceToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->cbase, src->cbase, 4 * (src->ncomp + 1), cudaMemcpyDeviceToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->cebase, src->cebase, 4 * src->ncomp, cudaMemcpyDeviceToDevice);
  }
  if (e != cudaSuccess) {
    free_mesh(m);
    return cuda_fail(e, "mcl_mesh_clone");
  }
  m->T = src->T;
  m->square = src->square;
  m->ncomp = src->ncomp;
  if (src->comp_host) {
    m->comp_host = new int64_t[4 * src->ncomp];
    std::memcpy(m->comp_host, src->comp_host, sizeof(int64_t) * 4 * src->ncomp);
  }
  m->tail_items = src->tail_items;
  m->rm_tile = src->rm_tile;
  m->coop_blocks = src->coop_blocks;
  if (src->substeps > 0 && (rc = mcl_mesh_set_substeps(m, src->substeps)) != MCL_OK) {
    free_mesh(m);
    return rc;
  }
  if (src->dirty) {
    const int64_t nc = src->ncomp;
    m->dirty = new unsigned char[(size_t)nc]();
    m->act_list = new int[(size_t)nc];
    if (cudaMalloc((void**)&m->act_dev, 4 * (5 * nc + 2)) != cudaSuccess ||
        cudaMallocHost((void**)&m->act_host, 4 * (5 * nc + 2)) != cudaSuccess) {
      free_mesh(m);
      return fail(MCL_ERR_OUT_OF_MEMORY, "mcl_mesh_clone: active tables");
    }
  }
  *out = m;
  return MCL_OK;
}

int mcl_batch_set_active(mcl_mesh* m, const int32_t* meshes_host, int64_t n, void* stream) {
  if (!m || n < 0 || (n > 0 && !meshes_host)) return fail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  if (n == 0) {
    m->nact = 0;
    return MCL_OK;
  }
  if (!m->dirty) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_set_active: not a batch");
  if (n > m->ncomp) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_set_active: more meshes than the batch has");
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<unsigned char> seen((size_t)m->ncomp, 0);
  // the staging buffer may still feed the previous call's copy
  BCK(cudaStreamSynchronize(s));
  const int64_t nc = m->ncomp;
  int* epre = m->act_host;
  int* e0 = epre + nc + 1;
  int* vpre = e0 + nc;
  int* v0 = vpre + nc + 1;
  int* ids = v0 + nc;
  int64_t E = 0, V = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int c = meshes_host[i];
    if (c < 0 || c >= nc || seen[(size_t)c])
      return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_batch_set_active: mesh index out of range or repeated");
    seen[(size_t)c] = 1;
    m->act_list[i] = c;
    ids[i] = c;
    epre[i] = (int)E;
    e0[i] = (int)m->comp_host[4 * c + 2];
    vpre[i] = (int)V;
    v0[i] = (int)m->comp_host[4 * c];
    E += m->comp_host[4 * c + 3];
    V += m->comp_host[4 * c + 1];
  }
  epre[n] = (int)E;
  vpre[n] = (int)V;
  BCK(cudaMemcpyAsync(m->act_dev, m->act_host, 4 * (5 * nc + 2), cudaMemcpyHostToDevice, s));
  m->nact = (int)n;
  m->act_E = (int)E;
  m->act_V = (int)V;
  return MCL_OK;
}

int mcl_mesh_set_tuning(mcl_mesh* m, int blocks_per_sm, int tail_items) {
  if (!m || blocks_per_sm < 0 || tail_items < 0) return fail(MCL_ERR_INVALID_ARGUMENT, "bad tuning");
  const int bps = blocks_per_sm == 0 ? m->max_blocks_per_sm : blocks_per_sm;
  if (bps > m->max_blocks_per_sm)
    return fail(MCL_ERR_INVALID_ARGUMENT, "blocks per SM above the kernel's co-resident limit");
  m->coop_blocks = m->nsm * bps;
  m->tail_items = tail_items == 0 ? kTailItems : tail_items;
  return MCL_OK;
}

int mcl_mesh_set_removal_tile(mcl_mesh* m, int tile) {
  if (!m || tile < 0 || tile > 32) return fail(MCL_ERR_INVALID_ARGUMENT, "removal tile must be in [0, 32]");
  m->rm_tile = tile;
  return MCL_OK;
}

int mcl_mesh_get_removal_tile(const mcl_mesh* m, int* tile) {
  if (!m || !tile) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  *tile = m->rm_tile;
  return MCL_OK;
}

int mcl_mesh_set_substeps(mcl_mesh* m, int substeps) {
  if (!m || substeps < 0 || substeps > 64) return fail(MCL_ERR_INVALID_ARGUMENT, "substeps must be in [0, 64]");
  if (substeps > 0 && !m->vl2) {
    // the sub-step scratch (24 B per vertex) exists only for meshes that use it
    BCK(cudaMalloc((void**)&m->vprev, 8 * m->V));
    const cudaError_t e = cudaMalloc((void**)&m->vl2, 16 * m->V);
    if (e != cudaSuccess) {
      cudaFree(m->vprev);
      m->vprev = nullptr;
      return cuda_fail(e, "cudaMalloc(sub-step scratch)");
    }
  }
  m->substeps = substeps;
  return MCL_OK;
}

int mcl_mesh_get_tuning(const mcl_mesh* m, int* blocks_per_sm, int* tail_items, int* max_blocks_per_sm) {
  if (!m) return fail(MCL_ERR_INVALID_ARGUMENT, "null mesh");
  if (blocks_per_sm) *blocks_per_sm = m->coop_blocks / std::max(1, m->nsm);
  if (tail_items) *tail_items = m->tail_items;
  if (max_blocks_per_sm) *max_blocks_per_sm = m->max_blocks_per_sm;
  return MCL_OK;
}

static int walk(mcl_mesh* m, const float* sigma_dev, const uint8_t* frozen_dev, uint64_t seed,
                const uint64_t* seeds_dev, uint64_t* counter_dev, float lo, float hi, mcl_float2* d_dev,
                void* stream) {
  if (!m || !sigma_dev || !counter_dev || !d_dev || !(lo <= hi)) return fail(MCL_ERR_INVALID_ARGUMENT, "bad args");
  cudaStream_t s = (cudaStream_t)stream;
  const int V = (int)m->V;
  const ActV A = act_of(m);
  (void)V;
  if (A.V_it > 0)
    k_walk<<<(A.V_it + 255) / 256, 256, 0, s>>>(A, m->pos[m->cur], m->vfix, m->vcomp, m->cbase, sigma_dev, frozen_dev,
                                                seed, reinterpret_cast<const unsigned long long*>(seeds_dev),
                                                reinterpret_cast<const unsigned long long*>(counter_dev), lo, hi,
                                                reinterpret_cast<float2*>(d_dev));
  const int na = m->nact ? m->nact : (int)m->ncomp;
  k_advance<<<(na + 255) / 256, 256, 0, s>>>(reinterpret_cast<unsigned long long*>(counter_dev), m->nact,
                                             m->nact ? m->act_dev + 4 * m->ncomp + 2 : nullptr,
                                             (int)m->ncomp);
  BCK(cudaGetLastError());
  return MCL_OK;
}

int mcl_walk(mcl_mesh* m, const float* sigma_dev, const uint8_t* frozen_dev, uint64_t seed,
             uint64_t* counter_dev, float lo, float hi, mcl_float2* d_dev, void* stream) {
  return walk(m, sigma_dev, frozen_dev, seed, nullptr, counter_dev, lo, hi, d_dev, stream);
}

int mcl_walk_seeded(mcl_mesh* m, const float* sigma_dev, const uint8_t* frozen_dev, const uint64_t* seeds_dev,
                    uint64_t* counter_dev, float lo, float hi, mcl_float2* d_dev, void* stream) {
  if (!seeds_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_walk_seeded: null seed table");
  return walk(m, sigma_dev, frozen_dev, 0, seeds_dev, counter_dev, lo, hi, d_dev, stream);
}

int mcl_settle_moves(mcl_mesh* m, mcl_float2* d_dev, void* stream, int64_t* sent_back_host) {
  if (!m || !d_dev) return fail(MCL_ERR_INVALID_ARGUMENT, "null argument");
  if (!m->valid_cur) return fail(MCL_ERR_INVALID_ARGUMENT, "mcl_settle_moves: points were moved without a step");
  int rc = ensure_settle_scratch(m);
  if (rc != MCL_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  SettleArgs A;
  A.A = act_of(m);
  A.pos = m->pos[m->cur];
  A.d = reinterpret_cast<float2*>(d_dev);
  A.vfix = m->vfix;
  A.vcomp = m->vcomp;
  // as much of the table as the active vertices need: clearing all of it took 42 us a
  // call for one mesh of a batch of 20M vertices
  int64_t slots = 1;
  while (slots < 4 * (int64_t)A.A.V_it && slots < m->table_size) slots <<= 1;
  A.table = m->table;
  A.mask = (unsigned)(slots - 1);
  A.smark = m->smark;
  A.list0 = m->vl[0];  // the step's own lists, idle between steps
  A.list1 = m->vl[1];
  A.smove = m->smove;
  A.st = m->st;
  A.max_passes = 64;
  void* args[] = {&A};
  // words 1..5 (pass counters, total, status) start at zero; the stamp (word 0) persists
  BCK(cudaMemsetAsync(m->st->settle + 1, 0, 5 * sizeof(unsigned), s));
  BCK(cudaMemsetAsync(m->table, 0xff, 4 * (size_t)slots, s));
  BCK(cudaLaunchCooperativeKernel((void*)k_settle, dim3(m->settle_blocks), dim3(256), args, 0, s));
  if (sent_back_host) {
    unsigned h[6];
    BCK(cudaMemcpyAsync(h, m->st->settle, sizeof(h), cudaMemcpyDeviceToHost, s));
    BCK(cudaStreamSynchronize(s));
    if (h[5] & 2u) return fail(MCL_ERR_CAPACITY, "mcl_settle_moves: position table full");
    if (h[5]) return fail(MCL_ERR_NO_CONVERGENCE, "mcl_settle_moves: pass limit reached");
    *sent_back_host = h[4];
  }
  return MCL_OK;
}

}  // extern "C"
