// Untangling by rebuilding stars.
//
// A step that turns faces over leaves a topology that no longer fits the
// positions.  Instead of moving vertices back, removing and reinserting them,
// every vertex works out its own star (its Delaunay neighbours in angular
// order) from the vertices that were around it, all at once and without
// touching the mesh:
//
//   star     the old neighbours and the vertices across its link edges (a
//            vertex no bad edge's quad holds keeps its old ring), sorted by
//            angle, then a circular Graham scan with incircle: the Delaunay
//            neighbours of v among a candidate set are the convex hull of the
//            candidates under inversion about v, and angular order is hull order;
//   check    every edge must be seen by both ends, between the same two faces;
//            the vertices of an edge that is not compute their star again from
//            the stars of their neighbours (star splaying: J. R. Shewchuk,
//            "Star splaying: an algorithm for repairing Delaunay triangulations
//            and convex hulls", SoCG 2005), until all agree;
//   number   edges get consecutive ids in the order of their smaller end (an
//            exclusive scan), the four sides of the square the first four;
//   write    every vertex writes its own fields of its edges' records.
//
// Stars that agree everywhere are positive closed fans that glue to a
// triangulation of the square, once over it when the edges number 3 n + 1 +
// the sides, and each edge is locally Delaunay in the star that holds it: the
// unique (perturbed) Delaunay triangulation.  All tests are the exact ladder.
// The mesh is only written after every star agrees, so whatever cannot be
// decided here (a vertex outside the square, coincident vertices, a row pool
// that is full) is left to the removal path as if nothing had run.
//
// What bounds it: below some ten thousand vertices the latency of one vertex's
// dependent loads and tests and five to ten grid barriers; above, instruction issue
// (456 warp instructions per vertex of a 1M-point step, with 12.6 of 32 lanes at work:
// rings and candidate lists differ in length), barriers and L2 latency.  A step at sigma =
// 0.1 x spacing, from the call to its record, by removal -> by stars, GB300: 1,000 points
// 460 -> 110 us, 10,000 points 610 -> 185 us, 500,000 points 1290 -> 780 us, 1,000,000
// points 1640 -> 1230 us; a pass of the precision-stress set of 500,000 (a third of it in
// clusters that move 1.4 of their spacings) 2860 -> 1860 us.
//
// The bodies are host/device code: tests/cpp/star_rounds.cu runs them vertex by vertex
// on the CPU.
#pragma once

#include "engine.cuh"

namespace mcl {

constexpr int kRow = 16;          // ints per star row: header, up to 15 neighbours
constexpr int kRowInline = 15;
constexpr int kExtRow = 128;      // ints of an overflow row (wider stars)
constexpr int kStarCand = 128;    // candidates a star can be made of
// A row's header: the number of neighbours, which of the first 15 edges are v's
// own (from bit 8), and two flags.
constexpr int kRowOpen = 1 << 30;  // the fan did not close
constexpr int kRowExt = 1 << 29;   // the neighbours are in overflow row id[0]
constexpr int kRowCount = 255;
constexpr int kRowOwn = 8;
constexpr int kInbox = 8;         // ints per vertex: how many, then up to 7 vertices to consider
constexpr int kStarRounds = 64;   // rounds of disagreeing stars before the removal path takes over

// Overflow rows of a mesh of V vertices.
MCL_HD int star_ext_rows(int64_t V) { return (int)(V / 64 + 64); }
constexpr int kStarBlocks = 1024;  // most blocks of a launch (four sums each)
// The scratch of such a mesh, in ints (all but the last part on 16 bytes): rows,
// overflow rows, the block sums, a mark per vertex.  The inboxes share the flip rounds'
// claims (`efa`): a launch that makes stars flips nothing unless they fail, and then
// after the last of them has been read.
MCL_HD int64_t star_sums_at(int64_t V) { return kRow * V + (int64_t)kExtRow * star_ext_rows(V); }
MCL_HD int64_t star_mark_at(int64_t V) { return star_sums_at(V) + 4 * kStarBlocks; }
MCL_HD int64_t star_ints(int64_t V) { return star_mark_at(V) + V; }

// What a phase reads it does not write, and a grid barrier lies between a phase
// and the one before (its acquire drops stale lines), so reads go through L1:
// neighbouring vertices share most of each other's records and rows.
MCL_HD int sld(const int* p) { return *p; }
MCL_HD int4 sld4(const int4* p) { return *p; }
MCL_HD float2 spos(const KParams& P, int v) { return P.pos[v]; }
#if defined(__CUDA_ARCH__)
MCL_HD void sst(int* p, int x) { __stcg(p, x); }
MCL_HD void sst4(int4* p, int4 x) { __stcg(p, x); }
MCL_HD int sadd(int* p, int x) { return atomicAdd(p, x); }
#else
MCL_HD void sst(int* p, int x) { *p = x; }
MCL_HD void sst4(int4* p, int4 x) { *p = x; }
MCL_HD int sadd(int* p, int x) { const int r = *p; *p += x; return r; }
#endif

MCL_HD void star_count(LocalCounters& lc, const LocalCounters& m) {
  lc.orient_fp64 += m.orient_fp64;
  lc.orient_exact += m.orient_exact;
  lc.incircle_fp64 += m.incircle_fp64;
  lc.incircle_exact += m.incircle_exact;
  lc.sos += m.sos;
  lc.incircle += m.incircle;
  lc.overflow |= m.overflow;
}

// First vertex and first edge of the mesh of v: the corners are v0 .. v0 + 3.
struct MeshBase {
  int v0, v1, e0;  // vertices v0 .. v1 - 1
};
MCL_HD MeshBase star_base(const KParams& P, int v) {
  MeshBase m = {0, P.V, 0};
  if (P.vcomp) {
    const int c = P.vcomp[v];
    m.v0 = P.cbase[c];
    m.v1 = P.cbase[c + 1];
    m.e0 = P.cebase[c];
  }
  return m;
}
// Edge (v, w) belongs to its smaller end; an edge to a corner to the other end.
MCL_HD bool star_owned(int v, int w, int c4) { return w > v || w < c4; }

// ---------------------------------------------------------------------------
// Candidate lists: ids with their positions relative to v (rounded once: the
// differences that the FP32 filters of orient2d and incircle start from with v
// as the last point), in angular order.
struct Cand {
  float x, y;
  int id;
};
struct LocalCand {
  Cand c_[kStarCand];
  MCL_HD int cap() const { return kStarCand; }
  MCL_HD Cand get(int i) const { return c_[i]; }
  MCL_HD void set(int i, Cand c) { c_[i] = c; }
};

enum : int { kStarOk = 0, kStarDegenerate = 1, kStarFull = 2 };

// Candidate w at x, seen from pv.
MCL_HD Cand star_cand(float2 pv, int w, float2 x) { return Cand{fsub(x.x, pv.x), fsub(x.y, pv.y), w}; }

// Its pseudo-angle in [0, 4], monotone in the angle up to 2e-6 (differences,
// quotient and sums rounded once each, the quotient to 2 ulp); NaN when it lies on v.
// Angles are counted from `from`, the pseudo-angle of the first candidate, so that a
// ring comes in order.
MCL_HD float star_key(const Cand& c, float from) {
  const float s = fabsf(c.x) + fabsf(c.y);
#if defined(__CUDA_ARCH__)
  const float t = __fdividef(c.y, s);  // s is at most 4e7, far below its limit
#else
  const float t = c.y / s;
#endif
  const float k = (c.x >= 0.f ? (c.y >= 0.f ? t : 4.f + t) : 2.f - t) - from;
  return k < 0.f ? k + 4.f : k;
}
constexpr float kStarSameKey = 8e-6f;

// Sign of the cross product a x c (orient2d(a, c, v)); 2: not decided.
MCL_HD int star_cross(const Cand& a, const Cand& c) {
  const float l = fmul(a.x, c.y), r = fmul(a.y, c.x);
  const float det = fsub(l, r), sum = fadd(fabsf(l), fabsf(r)), err = fmul(kCcwErrF, sum);
  const int s = det > err ? 1 : (-det > err ? -1 : 2);
  return (sum > kTinyF) & (sum < 1e37f) ? s : 2;
}

// Sign of incircle(a, c, b, v): positive when b lies outside the circle of a
// wedge v, a, c below 180 degrees (moving v to the front turns the sign); 2: not
// decided.
MCL_HD int star_outside(const Cand& a, const Cand& c, const Cand& b) {
  const float cxby = fmul(c.x, b.y), bxcy = fmul(b.x, c.y);
  const float al = fadd(fmul(a.x, a.x), fmul(a.y, a.y));
  const float bxay = fmul(b.x, a.y), axby = fmul(a.x, b.y);
  const float cl = fadd(fmul(c.x, c.x), fmul(c.y, c.y));
  const float axcy = fmul(a.x, c.y), cxay = fmul(c.x, a.y);
  const float bl = fadd(fmul(b.x, b.x), fmul(b.y, b.y));
  const float det = fadd(fadd(fmul(al, fsub(cxby, bxcy)), fmul(cl, fsub(bxay, axby))), fmul(bl, fsub(axcy, cxay)));
  const float perm = fadd(fadd(fmul(fadd(fabsf(cxby), fabsf(bxcy)), al), fmul(fadd(fabsf(bxay), fabsf(axby)), cl)),
                          fmul(fadd(fabsf(axcy), fabsf(cxay)), bl));
  const float err = fmul(kIccErrF, perm);
  const int s = det > err ? 1 : (-det > err ? -1 : 2);
  return (perm > kTinyF) & (perm < 1e37f) ? s : 2;
}

// What the filters leave open, from the positions by the full ladder.
MCL_HD_NOINLINE int star_cross_exact(const float2* pos, int v, int a, int c, LocalCounters* lc) {
  const float2 pv = pos[v], pa = pos[a], pc = pos[c];
  return orient2d(pa.x, pa.y, pc.x, pc.y, pv.x, pv.y, lc, &lc->overflow);
}
MCL_HD_NOINLINE int star_outside_exact(const float2* pos, int v, int a, int c, int b, LocalCounters* lc) {
  const float2 pv = pos[v], pa = pos[a], pb = pos[b], pc = pos[c];
  return incircle_sos(pa.x, pa.y, pc.x, pc.y, pb.x, pb.y, pv.x, pv.y, a, c, b, v, lc, &lc->overflow);
}

// Of two candidates on one ray: is w nearer than u?  The coordinates decide
// (-1: they coincide).
MCL_HD_NOINLINE int star_nearer(const float2* pos, int v, int u, int w) {
  const float2 pv = pos[v], pu = pos[u], pw = pos[w];
  const bool byx = pu.x != pv.x;
  const float a = byx ? (pu.x > pv.x ? pu.x : -pu.x) : (pu.y > pv.y ? pu.y : -pu.y);
  const float b = byx ? (pu.x > pv.x ? pw.x : -pw.x) : (pu.y > pv.y ? pw.y : -pw.y);
  return a == b ? -1 : (b < a ? 1 : 0);
}

// Insert candidate c in angular order; of two on one ray only the nearer stays.
// far: leave c out when it lies outside the circle of the entries beside it
// (every wedge of the list is below 180 degrees).
template <typename List>
MCL_HD int star_insert(const KParams& P, int v, float from, List& L, int& n, Cand c, bool far, LocalCounters& lc) {
  const float key = star_key(c, from);
  if (!(key >= 0.f)) return kStarDegenerate;
  int j = n;
#pragma unroll 1
  while (j > 0) {
    const Cand u = L.get(j - 1);
    if (u.id == c.id) return kStarOk;
    const float ku = star_key(u, from);
    bool before = ku < key;
    if (fabsf(ku - key) < kStarSameKey) {
      int s = star_cross(u, c);
      if (s == 2) {
        LocalCounters m = {0, 0, 0, 0, 0, 0, 0};
        s = star_cross_exact(P.pos, v, u.id, c.id, &m);
        star_count(lc, m);
        if (s == 0) {
          const int near = star_nearer(P.pos, v, u.id, c.id);
          if (near < 0) return kStarDegenerate;
          if (near) L.set(j - 1, c);
          return kStarOk;
        }
      }
      before = s > 0;
    }
    if (before) break;
    --j;
  }
  if (far && star_outside(L.get(j == 0 ? n - 1 : j - 1), L.get(j == n ? 0 : j), c) == 1) return kStarOk;
  if (n >= L.cap()) return kStarFull;
#pragma unroll 1
  for (int i = n; i > j; --i) L.set(i, L.get(i - 1));
  L.set(j, c);
  ++n;
  return kStarOk;
}

// Circular Graham scan over the n sorted candidates: b, between a and c, is no
// neighbour when it lies outside the circle of (v, a, c); where a -> c spans 180
// degrees or more it is needed.  One test per turn of one loop, so that the
// threads of a warp stay together: first along the list (the stack is its front,
// c the next candidate), then around its end until nothing drops.  The star is
// left in entries f .. t; returns whether the fan is closed.
template <typename List>
MCL_HD bool star_scan(const KParams& P, int v, List& L, int n, int* first, int* last, LocalCounters& lc) {
  if (n < 3) return false;
  int f = 0, t = 1, i = 2, ia = 0, ib = 1;
  Cand c = L.get(2);
#pragma unroll 1
  for (;;) {
    const Cand a = L.get(ia), b = L.get(ib);
    int s = star_cross(a, c);
    if (s == 1) {
      lc.incircle++;
      s = star_outside(a, c, b);
    }
    if (s == 2) {
      LocalCounters m = {0, 0, 0, 0, 0, 0, 0};
      s = star_cross_exact(P.pos, v, a.id, c.id, &m);
      if (s > 0) s = star_outside_exact(P.pos, v, a.id, c.id, b.id, &m);
      star_count(lc, m);
    }
    const bool drop = s > 0;
    if (i < n) {  // along the list
      if (drop) --t;
      if (!drop || t < 1) {
        L.set(++t, c);
        ++i;
      }
      if (i < n) {
        c = L.get(i);
        ia = t - 1;
        ib = t;
        continue;
      }
    } else if (ib == t) {  // the last entry against the first
      if (drop) {
        --t;
      } else {
        if (t - f < 2) break;
        ia = t;
        ib = f;
        c = L.get(f + 1);
        continue;
      }
    } else {  // the first entry against the last
      if (!drop) break;
      ++f;
    }
    if (t - f < 2) break;
    ia = t - 1;
    ib = t;
    c = L.get(f);
  }
  *first = f;
  *last = t;
  if (t - f < 2) return false;
  Cand a = L.get(t);
#pragma unroll 1
  for (int k = f; k <= t; ++k) {
    const Cand b = L.get(k);
    int s = star_cross(a, b);
    if (s == 2) {
      LocalCounters m = {0, 0, 0, 0, 0, 0, 0};
      s = star_cross_exact(P.pos, v, a.id, b.id, &m);
      star_count(lc, m);
    }
    if (s <= 0) return false;
    a = b;
  }
  return true;
}

// ---------------------------------------------------------------------------
// Rows.
MCL_HD const int* star_ext(const KParams& P, int row) { return P.sext + (size_t)row * kExtRow; }

// The neighbours f .. t of the list as the row of v; false when no overflow row
// is left.  again: this launch has written the row before; an overflow row it
// has stays its own.
template <typename List>
MCL_HD bool star_write(const KParams& P, int v, int c4, const List& L, int f, int t, bool closed, bool again) {
  int4* row = reinterpret_cast<int4*>(P.srow + (size_t)v * kRow);
  const int n = t - f + 1, flags = closed ? 0 : kRowOpen;
  if (n <= kRowInline) {
    int x[kRow];
    int own = 0;
#pragma unroll
    for (int i = 0; i < kRowInline; ++i) {
      x[i + 1] = i < n ? L.get(f + i).id : -1;
      if (i < n && star_owned(v, x[i + 1], c4)) own |= 1 << i;
    }
    x[0] = n | flags | own << kRowOwn;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < 2 || n > 7) sst4(row + i, make_int4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]));
    return true;
  }
  if (n > kExtRow) return false;
  const int4 old = sld4(row);
  const int e = again && (old.x & kRowExt) ? old.y : sadd(&P.st->star_ext, 1);
  if (e < 0 || e >= star_ext_rows(P.V)) return false;
  int* x = P.sext + (size_t)e * kExtRow;
  for (int i = 0; i < n; ++i) sst(x + i, L.get(f + i).id);
  sst4(row, make_int4(n | flags | kRowExt, e, -1, -1));
  return true;
}

// Where a row stands: the entries are read one by one from rows wider than 15.
struct RowRef {
  int n;          // neighbours
  bool open;
  const int* at;  // first entry
};
MCL_HD RowRef star_row(const KParams& P, int v) {
  RowRef r;
  const int* row = P.srow + (size_t)v * kRow;
  const int4 q = sld4(reinterpret_cast<const int4*>(row));  // the header and its overflow row together
  const int h = q.x, e = q.y;
  r.n = h & kRowCount;
  r.open = (h & kRowOpen) != 0;
  r.at = row + 1;
  if (h & kRowExt) {
    if (e >= 0 && e < star_ext_rows(P.V)) r.at = star_ext(P, e);
    else r.n = 0;
    if (r.n > kExtRow) r.n = 0;
  } else if (r.n > kRowInline) {
    r.n = 0;
  }
  return r;
}

// Position of v in the row of w (-1: not there), the entries before and after
// it, and how many of the row's own edges come before it.  Out of line: one copy
// of its code serves the checks and the writing.
struct RowFind {
  int pos, before, after, rank;
};
MCL_HD_NOINLINE RowFind star_find(const int* srow, const int* sext, int ext_rows, int w, int v, int c4, int4 q0,
                                  int4 q1) {
  const int4* row = reinterpret_cast<const int4*>(srow + (size_t)w * kRow);
  int x[kRow];
  x[0] = q0.x; x[1] = q0.y; x[2] = q0.z; x[3] = q0.w;
  x[4] = q1.x; x[5] = q1.y; x[6] = q1.z; x[7] = q1.w;
  const bool longer = !(x[0] & kRowExt) && (x[0] & kRowCount) > 7;
  const int4 none = {-1, -1, -1, -1};
  const int4 q2 = longer ? sld4(row + 2) : none, q3 = longer ? sld4(row + 3) : none;
  x[8] = q2.x; x[9] = q2.y; x[10] = q2.z; x[11] = q2.w;
  x[12] = q3.x; x[13] = q3.y; x[14] = q3.z; x[15] = q3.w;
  RowFind r = {-1, -1, -1, 0};
  const int n = x[0] & kRowCount;
  if (x[0] & kRowExt) {
    if (n > kExtRow || x[1] < 0 || x[1] >= ext_rows) return r;
    const int* e = sext + (size_t)x[1] * kExtRow;
    int own = 0;
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const int u = sld(e + i);
      if (u == v) {
        r.pos = i;
        r.rank = own;
        r.before = sld(e + (i ? i - 1 : n - 1));
        r.after = sld(e + (i + 1 < n ? i + 1 : 0));
        break;
      }
      own += star_owned(w, u, c4) ? 1 : 0;
    }
    return r;
  }
  int lastid = -1;
  auto look = [&](int i) {
    if (i < n) {
      lastid = x[i + 1];
      if (lastid == v) {
        r.pos = i;
        r.before = x[i];
        r.after = x[i + 2 < kRow ? i + 2 : 0];
      }
    }
  };
#pragma unroll
  for (int i = 0; i < 7; ++i) look(i);
  if (longer) {
#pragma unroll
    for (int i = 7; i < kRowInline; ++i) look(i);
  }
  if (r.pos >= 0) {
    const unsigned mine = (unsigned)x[0] >> kRowOwn & ((1u << r.pos) - 1u);
#if defined(__CUDA_ARCH__)
    r.rank = __popc(mine);
#else
    r.rank = __builtin_popcount(mine);
#endif
  }
  if (r.pos == 0) r.before = lastid;
  if (r.pos == n - 1) r.after = x[1];
  return r;
}
MCL_HD RowFind star_find(const KParams& P, int w, int v, int c4) {
  const int4* row = reinterpret_cast<const int4*>(P.srow + (size_t)w * kRow);
  return star_find(P.srow, P.sext, star_ext_rows(P.V), w, v, c4, sld4(row), sld4(row + 1));
}

// ---------------------------------------------------------------------------
// The four corners added to entries f .. t (moved to the front); returns how many
// entries there are, or -1.
template <typename List>
MCL_HD int star_corners(const KParams& P, int v, int v0, float from, List& L, int f, int t, LocalCounters& lc) {
  const float2 pv = spos(P, v);
  int n = 0;
#pragma unroll 1
  for (int i = f; i <= t; ++i, ++n) L.set(n, L.get(i));
#pragma unroll 1
  for (int c = 0; c < 4; ++c)
    if (star_insert(P, v, from, L, n, star_cand(pv, v0 + c, spos(P, v0 + c)), false, lc) != kStarOk) return -1;
  return n;
}

// The star from the sorted candidates, written as v's row.  Where the fan does
// not close (v moved out of its candidates' hull) the corners join them: what has
// dropped stays redundant.
template <typename List>
MCL_HD int star_finish(const KParams& P, int v, int v0, float from, List& L, int n, bool again, LocalCounters& lc) {
  int f = 0, t = n - 1;
  bool closed = false;
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    closed = star_scan(P, v, L, n, &f, &t, lc);
    if (closed || pass) break;
    n = star_corners(P, v, v0, from, L, f, n < 3 ? n - 1 : t, lc);
    if (n < 0) return L.cap() < kStarCand ? kStarFull : kStarDegenerate;
    f = 0;
    t = n - 1;
  }
  return star_write(P, v, v0 + 4, L, f, t, closed, again) ? kStarOk : kStarDegenerate;
}

// The star of v from the old mesh: kept as it is, or made from the old ring and
// the vertices across those of its sides that the classification (stamp bad in
// `cand`) found not Delaunay or at a turned face.  Returns kStarOk, or what went
// wrong (kStarFull: try again with a longer list).
template <typename List>
MCL_HD int star_from_mesh(const KParams& P, int v, bool keep, unsigned bad, List& L, LocalCounters& lc) {
  const MeshBase mb = star_base(P, v);
  const int HE = 2 * P.E;
  const int s0 = sld(P.vhe + v);
  if (s0 < 0 || s0 >= HE) return kStarDegenerate;
  const float2 pv = spos(P, v);
  sst(P.sinbox + (size_t)kInbox * v, 0);
  // the next spoke's record and end are asked for before this one's are used
  int n = 0, h = s0, o = -1;
  bool across = false, round = false, first = true;
  float from = 0.f;
  int4 r = sld4(P.en + (h >> 1));
  float2 px = pv, po = pv, pu = pv;
#pragma unroll 1
  for (int turn = 0; turn < 2 * kStarCand; ++turn) {
    int x;
    if (across) {
      x = o;
      px = po;
      across = false;
    } else {
      if (round) break;
      const int nx = (h & 1) ? r.z : r.x, pr = (h & 1) ? r.w : r.y;
      if (nx < 0 || nx >= HE || pr < 0 || pr >= HE) return kStarDegenerate;
      h = pr ^ 1;
      round = h == s0;
      r = sld4(P.en + (h >> 1));
      const int4 e = sld4(P.ev + (nx >> 1));
      const bool open = !keep && (unsigned)sld(reinterpret_cast<const int*>(P.cand) + (nx >> 1)) == bad;
      const int u = (nx & 1) ? e.x : e.y;
      x = (nx & 1) ? e.y : e.x;
      o = (nx & 1) ? e.z : e.w;
      if (x < mb.v0 || x >= mb.v1 || u < mb.v0 || u >= mb.v1 || o >= mb.v1 || x == v) return kStarDegenerate;
      across = open && o >= mb.v0 && o != v;
      px = pu;
      if (!keep) {
        if (first) px = spos(P, x);
        pu = spos(P, u);  // the next spoke's end
        if (across) po = spos(P, o);
      }
      first = false;
    }
    if (keep) {
      if (n >= L.cap()) return kStarFull;
      L.set(n++, Cand{0.f, 0.f, x});
      continue;
    }
    const Cand c = star_cand(pv, x, px);
    if (n == 0) from = star_key(c, 0.f);
    const int rc = star_insert(P, v, from, L, n, c, false, lc);
    if (rc != kStarOk) return rc;
  }
  if (!round) return kStarDegenerate;
  if (keep) return star_write(P, v, mb.v0 + 4, L, 0, n - 1, true, false) ? kStarOk : kStarDegenerate;
  return star_finish(P, v, mb.v0, from, L, n, false, lc);
}

// The star of v again: its present star and the vertices the last check left in
// its inbox.
template <typename List>
MCL_HD int star_from_stars(const KParams& P, int v, List& L, LocalCounters& lc) {
  const MeshBase mb = star_base(P, v);
  const float2 pv = spos(P, v);
  const RowRef me = star_row(P, v);
  int* box = P.sinbox + (size_t)kInbox * v;
  const int got = sld(box), m = got < kInbox - 1 ? got : kInbox - 1;
  int n = 0;
  bool far = false;
  float from = 0.f;
  auto entry = [&](int i) { return i < me.n + m ? sld(i < me.n ? me.at + i : box + 1 + (i - me.n)) : v; };
  int x1 = entry(0);
  float2 p1 = x1 >= mb.v0 && x1 < mb.v1 ? spos(P, x1) : pv;  // the next entry's place, a turn ahead
#pragma unroll 1
  for (int i = 0; i < me.n + m; ++i) {
    const int x = x1;
    const float2 px = p1;
    if (x < mb.v0 || x >= mb.v1 || x == v) return kStarDegenerate;
    x1 = entry(i + 1);
    if (x1 >= mb.v0 && x1 < mb.v1) p1 = spos(P, x1);
    if (i == me.n) far = !me.open && n >= 3;  // every wedge of the list is below 180 degrees
    const Cand c = star_cand(pv, x, px);
    if (i == 0) from = star_key(c, 0.f);
    const int rc = star_insert(P, v, from, L, n, c, far, lc);
    if (rc != kStarOk) return rc;
  }
  const int rc = star_finish(P, v, mb.v0, from, L, n, true, lc);
  if (rc == kStarOk) sst(box, 0);
  return rc;
}

// ---------------------------------------------------------------------------
// libmorton's m2D_e_LUT<uint_fast32_t,uint_fast32_t>(x, y) as the reference calls it:
// each float truncated to an integer (two's complement for negative values), the low
// 32 bits of x in the even bit positions, y in the odd ones.
MCL_HD unsigned long long morton_spread(unsigned long long w) {
  w &= 0xFFFFFFFFull;
  w = (w | (w << 16)) & 0x0000FFFF0000FFFFull;
  w = (w | (w << 8)) & 0x00FF00FF00FF00FFull;
  w = (w | (w << 4)) & 0x0F0F0F0F0F0F0F0Full;
  w = (w | (w << 2)) & 0x3333333333333333ull;
  w = (w | (w << 1)) & 0x5555555555555555ull;
  return w;
}
MCL_HD unsigned long long morton_cell(unsigned x, unsigned y) {
  return morton_spread(x) | morton_spread(y) << 1;
}
MCL_HD unsigned long long morton_key(float x, float y) {
  return morton_cell((unsigned)(long long)x, (unsigned)(long long)y);
}

// The points of an aligned square cell are consecutive in the Morton order, so a cell
// is found by bisection.  The cell around v is the smallest that holds kOrderNear
// consecutive points with v among them: its size follows the density of the points.

MCL_HD unsigned long long order_key(const KParams& P, int v) { return P.skey[v]; }
// First vertex in [lo, hi] whose key is at least k (hi + 1: none).
MCL_HD int order_bisect(const KParams& P, unsigned long long k, int lo, int hi) {
  int n = hi - lo + 1;
  while (n > 0) {
    const int h = n >> 1;
    if (order_key(P, lo + h) < k) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return lo;
}
constexpr int kOrderNear = 3;
constexpr int kOrderCell = 3;  // candidates from each of the nine cells
// Side of that cell as a power of two, for window k of kOrderNear consecutive points.
MCL_HD int order_cell(const KParams& P, int v, int k, int lo, int hi) {
  const int a = v - k, b = a + kOrderNear - 1;
  if (a < lo || b > hi) return 32;
  const unsigned long long d = order_key(P, a) ^ order_key(P, b);
  int bits = 0;
  while (bits < 32 && d >> (2 * bits)) ++bits;
  return bits;
}

// ---------------------------------------------------------------------------
// x is left for v to consider when it makes its star again.
MCL_HD void star_tell(const KParams& P, int v, int x, int c4) {
  if (v < c4 || x == v) return;
  int* box = P.sinbox + (size_t)kInbox * v;
  const int at = sadd(box, 1);
  if (at < kInbox - 1) sst(box + 1 + at, x);
}

// The two entries of w's row whose wedge holds the direction of v.
MCL_HD_NOINLINE int2 star_wedge(const int* srow, const int* sext, int ext_rows, const float2* pos, int w, int v) {
  const int4 q = sld4(reinterpret_cast<const int4*>(srow + (size_t)w * kRow));
  const int n = q.x & kRowCount;
  const int* at = srow + (size_t)w * kRow + 1;
  if (q.x & kRowExt) at = sext + (size_t)(q.y >= 0 && q.y < ext_rows ? q.y : 0) * kExtRow;
  if (n < 2 || n > ((q.x & kRowExt) ? kExtRow : kRowInline)) return make_int2(-1, -1);
  const float2 pw = pos[w];
  const float k = star_key(star_cand(pw, v, pos[v]), 0.f);
  int lo = -1, hi = -1, least = -1, most = -1;  // nearest keys below and above k, the extremes
  float klo = -1.f, khi = 9.f, kleast = 9.f, kmost = -1.f;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const int u = sld(at + i);
    if (u < 0) return make_int2(-1, -1);
    const float ku = star_key(star_cand(pw, u, pos[u]), 0.f);
    if (ku <= k && ku > klo) { klo = ku; lo = u; }
    if (ku > k && ku < khi) { khi = ku; hi = u; }
    if (ku < kleast) { kleast = ku; least = u; }
    if (ku > kmost) { kmost = ku; most = u; }
  }
  return make_int2(lo >= 0 ? lo : most, hi >= 0 ? hi : least);
}

// Do v and its neighbours agree?  For every neighbour w (all: both ends look;
// else only the end that does not own the edge, the count of edges covers the
// other way) v must be in w's row between the same two vertices.  mark(u) is
// called for the ends of an edge that disagrees, and each is told of the vertices
// the other sees there: v of the two beside it in w's row (or, where w does not
// hold v, of those whose wedge holds v), w of v and the two beside it in v's row.
// Returns the number of own edges; *inner: own edges to other points minus edges
// owned by other points; *ranks: four bits per entry, the rank of v among w's own
// edges.
// One entry w of v's row, between bf and af (q0, q1: the first half of w's row):
// returns the rank (0 where there is
// none to give), or -1 where the edge disagrees.
template <typename Mark>
MCL_HD int star_check_entry(const KParams& P, int v, int w, int bf, int af, int c4, bool all, int4 q0, int4 q1,
                            Mark mark) {
  // of two corners in a row the second follows the first around the square
  if (w < c4) return af < c4 && ((w - c4 + 5) & 3) != ((af - c4 + 4) & 3) ? -1 : 0;
  const bool mine = star_owned(v, w, c4);
  if (mine && !all) return 0;
  const RowFind r = star_find(P.srow, P.sext, star_ext_rows(P.V), w, v, c4, q0, q1);
  if (r.pos >= 0 && r.before == af && r.after == bf) return mine ? 0 : r.rank;
  mark(w);
  const bool gone = r.pos < 0;
  int ga = r.before, gb = r.after;
  if (gone) {
    star_tell(P, w, v, c4);
    const int2 g = star_wedge(P.srow, P.sext, star_ext_rows(P.V), P.pos, w, v);
    ga = g.x;
    gb = g.y;
  }
  if (gone || ga != af) {
    star_tell(P, w, af, c4);
    if (ga >= 0) star_tell(P, v, ga, c4);
  }
  if (gone || gb != bf) {
    star_tell(P, w, bf, c4);
    if (gb >= 0) star_tell(P, v, gb, c4);
  }
  return -1;
}
template <typename Mark>
MCL_HD int star_check(const KParams& P, int v, int c4, bool all, Mark mark, int* inner, unsigned long long* ranks) {
  const RowRef me = star_row(P, v);
  int own = 0, in = 0;
  unsigned long long rk = 0;
  bool bad = me.open || me.n < 3;
  if (me.n >= 3) {
    int bf = sld(me.at + me.n - 1), w = sld(me.at);
    const int first = w;
    int4 n0 = {0, 0, 0, 0}, n1 = n0;  // the next neighbour's row, asked for a turn ahead
    auto ask = [&](int u) {
      if (u < c4 || (!all && u > v)) return;
      const int4* row = reinterpret_cast<const int4*>(P.srow + (size_t)u * kRow);
      n0 = sld4(row);
      n1 = sld4(row + 1);
    };
    ask(w);
#pragma unroll 1
    for (int i = 0; i < me.n; ++i) {
      const int af = i + 1 < me.n ? sld(me.at + i + 1) : first;
      const int4 q0 = n0, q1 = n1;
      if (i + 1 < me.n) ask(af);
      const bool mine = star_owned(v, w, c4);
      own += mine ? 1 : 0;
      if (w >= c4) in += mine ? 1 : -1;
      const int r = star_check_entry(P, v, w, bf, af, c4, all, q0, q1, mark);
      if (r < 0) bad = true;
      else if (i < kRowInline) rk |= (unsigned long long)(r < 15 ? r : 15) << (4 * i);
      bf = w;
      w = af;
    }
  }
  if (bad) mark(v);
  *inner = in;
  *ranks = rk;
  return own;
}

// First edge of v's own edges once every base is known: the sides of the square
// are the mesh's first four edges.
MCL_HD int star_edge0(const KParams& P, MeshBase mb, int v) {
  return mb.e0 + 4 + sld(P.sbase + v) - sld(P.sbase + mb.v0 + 4);
}

// Half-edge v -> w_i for entry i of v's row; mine: own edges before entry i.
MCL_HD int star_spoke(const KParams& P, MeshBase mb, int v, int w, int i, int base, int mine, bool wide,
                      unsigned long long ranks) {
  if (star_owned(v, w, mb.v0 + 4)) return 2 * (base + mine);
  int r = (int)((ranks >> (4 * (i & 15))) & 15u);
  if (wide || r == 15) {  // the ranks hold 15 entries, and ranks below 15
    const RowFind g = star_find(P, w, v, mb.v0 + 4);
    if (g.pos < 0) return -1;
    r = g.rank;
  }
  return 2 * (star_edge0(P, mb, w) + r) + 1;
}

// v's fields of the records of its edge to w, between bf and af: h, hb and ha are
// the half-edges from v to the three.  In the face (v, w, af) v knows the
// half-edges v -> w and af -> v, so it sets prev of the one and next of the other;
// every face is covered by its three vertices.  An edge to a corner has no other
// end that writes: its owner finds the corner's two half-edges through the vertices
// beside it.  Two corners in a row: v also writes that side of the square.
MCL_HD bool star_put(const KParams& P, MeshBase mb, int v, int w, int bf, int af, int h, int hb, int ha) {
  const int c4 = mb.v0 + 4, e = h >> 1;
  int* en = reinterpret_cast<int*>(P.en);
  if (h & 1) {
    sst(en + 4 * e + 3, ha ^ 1);  // prev(v -> w)
    sst(en + 4 * e, hb);          // next(w -> v)
    return true;
  }
  sst4(P.ev + e, make_int4(v, w, af, bf));
  if (w >= c4) {
    sst(en + 4 * e + 1, ha ^ 1);
    sst(en + 4 * e + 2, hb);
    return true;
  }
  const int c = w - mb.v0;
  int nx, pv;
  if (af < c4) {
    nx = 2 * (mb.e0 + c);
  } else {
    const RowFind g = star_find(P, af, w, c4);
    if (g.pos < 0) return false;
    nx = 2 * (star_edge0(P, mb, af) + g.rank) + 1;
  }
  if (bf < c4) {
    pv = 2 * (mb.e0 + ((c + 3) & 3));
  } else {
    const RowFind g = star_find(P, bf, w, c4);
    if (g.pos < 0) return false;
    pv = 2 * (star_edge0(P, mb, bf) + g.rank);
  }
  sst4(P.en + e, make_int4(nx, ha ^ 1, hb, pv));
  if (af < c4) {
    const int s = mb.e0 + c;  // side w -> af, its inner face holds v
    sst4(P.ev + s, make_int4(w, af, v, -1));
    sst4(P.en + s, make_int4(ha ^ 1, h, 2 * (mb.e0 + ((c + 3) & 3)) + 1, 2 * (mb.e0 + ((c + 1) & 3)) + 1));
    sst(P.vhe + w, 2 * s);
  }
  return true;
}

// All of v's edges, in turn.
MCL_HD bool star_commit(const KParams& P, int v) {
  const MeshBase mb = star_base(P, v);
  const int c4 = mb.v0 + 4;
  const RowRef me = star_row(P, v);
  const bool wide = me.n > kRowInline;
  const unsigned long long ranks = P.srank[v];
  const int base = star_edge0(P, mb, v);
  // own edges before the last entry, to know its half-edge first
  int mine = 0;
#pragma unroll 1
  for (int i = 0; i + 1 < me.n; ++i) mine += star_owned(v, sld(me.at + i), c4) ? 1 : 0;
  int bf = sld(me.at + me.n - 1);
  int hb = star_spoke(P, mb, v, bf, me.n - 1, base, mine, wide, ranks);
  const int hlast = hb;
  int w = sld(me.at);
  const int first = w;
  int h = star_spoke(P, mb, v, w, 0, base, 0, wide, ranks);
  const int hfirst = h;
  if ((unsigned)h >= (unsigned)(2 * P.E) || (unsigned)hb >= (unsigned)(2 * P.E)) return false;
  sst(P.vhe + v, h);
  mine = star_owned(v, w, c4) ? 1 : 0;
#pragma unroll 1
  for (int i = 0; i < me.n; ++i) {
    int af = first, ha = hfirst;
    if (i + 1 < me.n) {
      af = sld(me.at + i + 1);
      ha = i + 2 == me.n ? hlast : star_spoke(P, mb, v, af, i + 1, base, mine, wide, ranks);
      mine += star_owned(v, af, c4) ? 1 : 0;
    }
    if ((unsigned)ha >= (unsigned)(2 * P.E) || !star_put(P, mb, v, w, bf, af, h, hb, ha)) return false;
    bf = w;
    hb = h;
    w = af;
    h = ha;
  }
  return true;
}

}  // namespace mcl
