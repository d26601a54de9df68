// Serial run, on the CPU, of the bodies that untangle by stars (mcleap_gb300/csrc/star.cuh),
// vertex by vertex in the order of the step's phases: classification, first stars,
// checks and stars again until all agree, numbering, writing.  Within a phase no vertex
// reads what another writes but for the inboxes, whose order of arrival does not matter
// to the result, so this checks the thread forms' logic and indexing without a GPU.
//
// int star_untangle(V, E, pos, ev, en, vhe, comps, cbase, cebase, info): a mesh or a batch
// (comps meshes, first vertices and edges with the end after the last vertex) whose points
// have moved to pos; ev, en and vhe are rewritten.  info: {rounds, stars made anew,
// overflow rows taken, non-positive faces seen, rows wider than 15}.  Returns 0, or what
// went wrong: 1 a first star, 2 a later star, 3 rounds, 4 the count of edges, 5 writing.
#include <cstdint>
#include <vector>

#include "engine.cuh"
#include "star.cuh"

using namespace mcl;

extern "C" int star_untangle(int V, int E, const float* pos, int* ev, int* en, int* vhe, int comps, const int* cbase,
                             const int* cebase, int* info) {
  std::vector<int> star((size_t)star_ints(V), 0x7abcdef1), inbox((size_t)kInbox * V), base(V), own(V), vcomp(V);
  std::vector<unsigned> cand(E, 0), touched(V, 0), listed(V, 0);
  std::vector<unsigned long long> ranks(V);
  std::vector<char> fixed(V, 0);
  for (int c = 0; c < comps; ++c) {
    for (int v = cbase[c]; v < cbase[c + 1]; ++v) vcomp[v] = c;
    for (int v = cbase[c]; v < cbase[c] + 4; ++v) fixed[v] = 1;
  }
  DevState* st = new DevState();
  KParams P = {};
  P.V = V;
  P.E = E;
  P.pos = reinterpret_cast<float2*>(const_cast<float*>(pos));
  P.ev = reinterpret_cast<int4*>(ev);
  P.en = reinterpret_cast<int4*>(en);
  P.vhe = vhe;
  P.srow = star.data();
  P.sext = star.data() + (size_t)kRow * V;
  P.sinbox = inbox.data();
  P.srank = ranks.data();
  P.sbase = base.data();
  P.cand = cand.data();
  P.vcomp = comps > 1 ? vcomp.data() : nullptr;
  P.cbase = cbase;
  P.cebase = cebase;
  P.st = st;
  LocalCounters lc = {0, 0, 0, 0, 0, 0, 0};
  auto sign = [&](int a, int b, int c) {
    return orient2d(P.pos[a].x, P.pos[a].y, P.pos[b].x, P.pos[b].y, P.pos[c].x, P.pos[c].y, &lc, &lc.overflow);
  };
  for (int e = 0; e < E; ++e) {
    const int4 q = P.ev[e];
    const int sa = q.z >= 0 ? sign(q.x, q.y, q.z) : 1, sb = q.w >= 0 ? sign(q.y, q.x, q.w) : 1;
    bool bad = sa <= 0 || sb <= 0;
    info[3] += (sa <= 0) + (sb <= 0);
    if (!bad && q.z >= 0 && q.w >= 0) {
      const float2 a = P.pos[q.x], b = P.pos[q.y], c = P.pos[q.z], d = P.pos[q.w];
      bad = incircle_sos(a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, q.x, q.y, q.z, q.w, &lc, &lc.overflow) > 0;
    }
    if (!bad) continue;
    cand[e] = 1;
    for (int v : {q.x, q.y, q.z, q.w})
      if (v >= 0) touched[v] = 1;
  }
  int rc = 0;
  auto done = [&](int code) {
    info[2] = st->star_ext;
    for (int v = 0; v < V && code == 0; ++v) info[4] += !fixed[v] && (star[(size_t)kRow * v] & kRowExt) ? 1 : 0;
    delete st;
    return code;
  };
  for (int v = 0; v < V; ++v) {
    if (fixed[v]) continue;
    LocalCand L;
    info[1] += (int)touched[v];
    if (star_from_mesh(P, v, !touched[v], 1, L, lc) != kStarOk) return done(1);
  }
  unsigned stamp = 0;
  for (bool both = false;;) {
    std::vector<int> list;
    auto mark = [&](int u) {
      if (listed[u] < stamp) {
        listed[u] = stamp;
        list.push_back(u);
      }
    };
    ++stamp;
    long long balance = 0, inner = 0;
    for (int v = 0; v < V; ++v) {
      own[v] = 0;
      if (fixed[v]) continue;
      const int c4 = star_base(P, v).v0 + 4;
      int in;
      own[v] = star_check(P, v, c4, both, mark, &in, &ranks[v]);
      balance += own[v] - 3 - (v == c4 ? 1 : 0);
      inner += in;
    }
    if (list.empty()) {
      if (balance == 0 && inner == 0) break;
      if (both) return done(4);
      both = true;
      continue;
    }
    while (!list.empty()) {
      if (++info[0] > kStarRounds) return done(3);
      for (int v : list) {
        LocalCand L;
        if (star_from_stars(P, v, L, lc) != kStarOk) return done(2);
      }
      std::vector<int> made;
      made.swap(list);
      ++stamp;
      int in;
      for (int v : made) star_check(P, v, star_base(P, v).v0 + 4, true, mark, &in, &ranks[v]);
    }
  }
  for (int v = 0, at = 0; v < V; ++v) {
    base[v] = at;
    at += own[v];
  }
  for (int v = 0; v < V; ++v)
    if (!fixed[v] && !star_commit(P, v)) rc = 5;
  return done(rc);
}
