// sbc_clean.cuh -- rows A9-A18 of one pair in general position: every hit a
// proper crossing inside both edges, labelled a crossing.  That is nearly
// every pair of real-valued polygons, with any number of components.
//
// In general position the reference's linked lists (copyToLinkedList,
// src/clip.cpp:606-695; labelIntersections2 and createResult2,
// foster/polyclip.h:337-759; Foster's component loops, lib/
// optimizedFostersAlgorithm/polyclip.cpp:335-780) hold nothing that the order
// of the crossings along each polygon does not say: a list is the vertices
// with each edge's crossings after them, entry and exit alternate along a
// component, and a ring is an alternating cycle of two pairings of the
// crossings (each with its neighbour along the base, and along the overlay,
// in the direction of its status).  So nothing of the merged arrays, labels,
// lists or pools is built: a counting sort by edge, a sort of each edge's few
// crossings, pointer doubling over the crossings, and each leg of a ring is
// written to its place.  Every test that decides whether a pair is in general
// position repeats the reference's own arithmetic; a pair that fails one is
// left untouched for the engine that follows the lists.
#pragma once

#include "sbc_group.cuh"
#include "sbc_pairops.cuh"
#include "sbc_serial.cuh"

namespace sbc {
namespace {

// The hits of a pair: base and overlay edge, type, first emission, alpha and
// beta.  kSparse: sorted by base edge, of a base so large that nothing is
// kept per base edge.
struct SoaHits {
  static constexpr bool kSparse = false;
  const int *hb, *hc, *ht;  // 2 * base edge, 2 * overlay edge, type
  const unsigned long long* hkey;
  const double *hal, *hbt;
  __device__ int b(int h) const { return hb[h] >> 1; }
  __device__ int c(int h) const { return hc[h] >> 1; }
  __device__ int type(int h) const { return ht[h]; }
  __device__ unsigned long long key(int h) const { return hkey[h]; }
  __device__ double al(int h) const { return hal[h]; }
  __device__ double bt(int h) const { return hbt[h]; }
};

// one past the last k < n that in_run(k) accepts, from x (accepted) on; the
// run is contiguous
template <class InRun>
__device__ __forceinline__ int run_end(int n, int x, InRun in_run) {
  int in = x, out = x + 1;
  for (int d = 1; out < n && in_run(out); d *= 2) {
    in = out;
    out += d;
  }
  if (out > n) out = n;
  while (out - in > 1) {
    const int k = (in + out) >> 1;
    if (in_run(k)) in = k;
    else out = k;
  }
  return out;
}

__device__ __forceinline__ void swap_arrays(int*& a, int*& b) {
  int* t = a;
  a = b;
  b = t;
}

template <class Hits>
struct CleanIn {
  const double* b;
  int nb;
  const double* c;
  int nc;
  const int* bnx;  // successor of each vertex within its component (null: one ring)
  const int* cnx;
  int K;
  Hits hits;
  int base_steps;  // sparse: the base edges' winding steps about the overlay's first vertex
  int unite;
  int rcap, vcap;      // room for rings and their vertices
  int *rootB, *rootC;  // scratch: first vertices of the components (n + 1)
  int *inB, *inC;      // scratch: per component, first vertex inside the other polygon
  int *nxt, *prv;      // scratch: vcap each
  int* roff;           // out: rings, their vertices, and where each vertex comes from
  double* rxy;
  unsigned long long* sort;  // shared memory: room for sort_room keys per warp
  int sort_room;
  int4* tape;  // {0, base vertex} {1, overlay vertex} {2, base edge, overlay edge}, ring in .w
};

// Working arrays, in shared memory or the pair's arena.  A hit h has rank
// rP[h] along the base and rQ[h] along the overlay; hP and hQ are the
// inverses, and ends[e] is one past edge e's last rank.
struct CleanMem {
  int *endB, *endC;
  int *hP, *hQ, *rP, *rQ, *eP, *eQ, *aB, *aC;
  double *x, *y;
  int4 *A, *B;
};

// nb: base edges to keep an end for (0: a sparse base)
__host__ __device__ __forceinline__ CleanMem clean_carve(Carver& cv, int nb, int nc, int K) {
  CleanMem m;
  m.endB = cv.take<int>(nb > 0 ? nb + 1 : 0);
  m.endC = cv.take<int>(nc + 1);
  m.hP = cv.take<int>(K);
  m.hQ = cv.take<int>(K);
  m.rP = cv.take<int>(K);
  m.rQ = cv.take<int>(K);
  m.eP = cv.take<int>(K);
  m.eQ = cv.take<int>(K);
  m.aB = cv.take<int>(K);
  m.aC = cv.take<int>(K);
  m.x = cv.take<double>(K);
  m.y = cv.take<double>(K);
  m.A = cv.take<int4>(K + 4);
  m.B = cv.take<int4>(K + 4);
  return m;
}

__host__ __device__ __forceinline__ size_t clean_bytes(int nb, int nc, int K) {
  Carver cv{nullptr, 0};
  clean_carve(cv, nb, nc, K);
  return (cv.off + 15) & ~(size_t)15;
}

// the components of an n-vertex polygon: their first vertices, then n
template <class G>
__device__ int clean_components(G& g, int n, const int* nx, int* root) {
  int count = 0;
  for (int i0 = 0; i0 < n; i0 += G::N) {
    const int v = i0 + g.rank();
    const bool first = v < n && (v == 0 || nx[v - 1] != v);
    int tot;
    const int k = count + g.before(first, &tot);
    if (first) root[k] = v;
    count += tot;
  }
  if (g.rank() == 0) root[count] = n;
  g.sync();
  return count;
}

// Done (rings, their count and vertices, and the area), not in general
// position, or out of room for ring vertices; the same on every thread, and
// where not done the outputs' contents are unspecified.  s_sum: a shared
// double per warp of a block.
enum { CLEAN_DONE = 0, CLEAN_NOT = 1, CLEAN_ROOM = 2 };
template <int n>
using Left = std::integral_constant<int, n>;
template <class G, class Hits>
__device__ int clean_clip(G& g, const CleanIn<Hits>& in, CleanMem m, double* s_sum,
                          int* nrings_out, int* nverts_out, double* area_out) {
  constexpr bool kSparse = Hits::kSparse;
  const Hits hits = in.hits;
  const int lane = g.rank();
  constexpr int N = G::N;
  const int K = in.K, nb = in.nb, nc = in.nc;
  const double *b = in.b, *c = in.c;
  auto bsucc = [&](int i) { return in.bnx ? in.bnx[i] : (i + 1 == nb ? 0 : i + 1); };
  auto csucc = [&](int i) { return in.cnx ? in.cnx[i] : (i + 1 == nc ? 0 : i + 1); };
  // ---- A10-A12: ranks along both polygons
  if (!kSparse)
    for (int i = lane; i <= nb; i += N) m.endB[i] = 0;
  for (int i = lane; i <= nc; i += N) m.endC[i] = 0;
  g.sync();
  bool bad = false;
  for (int h = lane; h < K; h += N) {
    const int e = hits.b(h), f = hits.c(h);
    if (hits.type(h) != 1) bad = true;
    if (kSparse) m.hP[h] = h;
    else atomicAdd(&m.endB[e], 1);
    atomicAdd(&m.endC[f], 1);
    // the crossing (saveIntersectionsParallel, oacc_segment_tree.cpp:7257-7341)
    const double al = hits.al(h), oma = dsub(1.0, al);
    const int e2 = bsucc(e), f2 = csucc(f);
    const double p1x = b[2 * e], p1y = b[2 * e + 1], p2x = b[2 * e2], p2y = b[2 * e2 + 1];
    const double x = dadd(dmul(oma, p1x), dmul(al, p2x)), y = dadd(dmul(oma, p1y), dmul(al, p2y));
    m.x[h] = x;
    m.y[h] = y;
    const int a = alpha_to_int(al), t = alpha_to_int(hits.bt(h));
    if (a < 0 || t < 0) bad = true;
    m.aB[h] = a % 1000000000;
    m.aC[h] = t % 1000000000;
    // apart from the four ends (an equal slot stops the list walk early, and
    // provenance goes by coordinates)
    auto meets = [&](double px, double py) { return same_value(px, x) && same_value(py, y); };
    if (meets(p1x, p1y) || meets(p2x, p2y) || meets(c[2 * f], c[2 * f + 1]) ||
        meets(c[2 * f2], c[2 * f2 + 1]))
      bad = true;
  }
  auto out = [&](auto left, int r) {  // with `left` phases not entered
    g.template leave<decltype(left)::value>();
    return r;
  };
  if (g.any(bad)) return out(Left<5>{}, CLEAN_NOT);
  if (K > 0) {
    if (!kSparse) group_scan(g, m.endB, nb + 1);
    group_scan(g, m.endC, nc + 1);
    g.sync();
    for (int h = lane; h < K; h += N) {  // a start moves up to its end
      if (!kSparse) m.hP[atomicAdd(&m.endB[hits.b(h)], 1)] = h;
      m.hQ[atomicAdd(&m.endC[hits.c(h)], 1)] = h;
    }
    g.sync();
  }
  auto startC = [&](int e) { return e == 0 ? 0 : m.endC[e - 1]; };
  auto startB = [&](int e) { return e == 0 ? 0 : m.endB[e - 1]; };  // (not sparse)
  auto countB = [&](int e) { return m.endB[e] - startB(e); };
  auto countC = [&](int f) { return m.endC[f] - startC(f); };
  // per edge: alpha order, ties in record order (base edge, then emission).
  // A hit of a short run counts the run's hits before it: its loads do not
  // wait for one another, and no thread sorts alone.  (An insertion sort per
  // edge, each step a trip to the arena, took a third of the pairwise block
  // kernel.)  A long run is sorted by alpha and index as one key, in the
  // group's shared memory where it fits.  From v to out: src(k) is entry k of
  // v, start(k) and end(k) the run's.
  constexpr int kRankMost = 64;
  auto order = [&](auto src, auto start, auto end, int* out, const int* alpha, auto less) {
    group_items(
        g, K, m.eP,
        [&](int k) {
          const int s = start(k), t = end(k);
          if (t - s > kRankMost) return k == s ? t - s : 0;
          const int h = src(k), a = alpha[h];
          int r = s;
#pragma unroll 4
          for (int i = s; i < t; ++i) {
            const int o = src(i), ao = alpha[o];
            r += ao < a || (ao == a && o != h && less(o, h));
          }
          out[r] = h;
          return 0;
        },
        [](int, int) {},
        [&](auto& gg, int s, int k) {
          const int np = npow2_dev(k);
          constexpr bool whole = G::kBlock && std::remove_reference_t<decltype(gg)>::kBlock;
          const int room = whole ? in.sort_room * G::N / 32 : in.sort_room;
          unsigned long long* o = (unsigned long long*)m.A + 2 * s;
          if (np <= room) o = in.sort + (whole ? 0 : in.sort_room * (int)(threadIdx.x >> 5));
          for (int i = gg.rank(); i < np; i += gg.N) {
            unsigned long long x = ~0ull;
            if (i < k) {
              const int h = src(s + i);
              x = ((unsigned long long)(unsigned)alpha[h] << 32) | (unsigned)h;
            }
            o[i] = x;
          }
          gg.sync();
          group_bitonic(gg, np, [&](int i, int j, bool up) {
            const unsigned long long x = o[i], y = o[j];
            if ((x > y) == up) {
              o[i] = y;
              o[j] = x;
            }
          });
          int* v = out + s;
          bool tie = false;
          for (int i = gg.rank(); i < k; i += gg.N) {
            tie |= i > 0 && (o[i] >> 32) == (o[i - 1] >> 32);
            v[i] = (int)(unsigned)o[i];
          }
          if (gg.any(tie)) {
            unsigned* scr = (unsigned*)o;
            for (int i = gg.rank(); i < np; i += gg.N) scr[i] = i < k ? (unsigned)v[i] : ~0u;
            gg.sync();
            group_bitonic(gg, np, [&](int i, int j, bool up) {
              const unsigned x = scr[i], y = scr[j];
              const bool lt = x != ~0u && (y == ~0u || (x != y && less((int)x, (int)y)));
              const bool gt = y != ~0u && (x == ~0u || (x != y && less((int)y, (int)x)));
              if (up ? gt : lt) {
                scr[i] = y;
                scr[j] = x;
              }
            });
            for (int i = gg.rank(); i < k; i += gg.N) v[i] = (int)scr[i];
          }
          gg.sync();
        });
    g.sync();
  };
  if (K > 0) {
    // (out is the inverses' arrays, which come after)
    order([&](int k) { return kSparse ? k : m.hP[k]; },
          [&](int k) {
            if (!kSparse) return startB(hits.b(m.hP[k]));
            const int e = hits.b(k);  // the run's first: its mirror image's end
            return K - run_end(K, K - 1 - k, [&](int i) { return hits.b(K - 1 - i) == e; });
          },
          [&](int k) {
            if (!kSparse) return m.endB[hits.b(m.hP[k])];
            const int e = hits.b(k);
            return run_end(K, k, [&](int i) { return hits.b(i) == e; });
          },
          m.rP, m.aB, [&](int u, int v) {
            return m.aB[u] != m.aB[v] ? m.aB[u] < m.aB[v] : hits.key(u) < hits.key(v);
          });
    order([&](int k) { return m.hQ[k]; }, [&](int k) { return startC(hits.c(m.hQ[k])); },
          [&](int k) { return m.endC[hits.c(m.hQ[k])]; }, m.rQ, m.aC, [&](int u, int v) {
            if (m.aC[u] != m.aC[v]) return m.aC[u] < m.aC[v];
            return hits.b(u) != hits.b(v) ? hits.b(u) < hits.b(v) : hits.key(u) < hits.key(v);
          });
    swap_arrays(m.hP, m.rP);
    swap_arrays(m.hQ, m.rQ);
    for (int k = lane; k < K; k += N) {
      const int h = m.hP[k], q = m.hQ[k];
      m.rP[h] = k;
      m.eP[k] = hits.b(h);
      m.rQ[q] = k;
      m.eQ[k] = hits.c(q);
    }
    g.sync();
  }
  g.phase();
  if (K > 0) {
    // ---- A14: every initial label a crossing (calculateInitLabelParallel,
    // oacc_segment_tree.cpp:7925-7988): the overlay's neighbours of the
    // crossing lie on different sides of the base there
    for (int k = lane; k < K && !bad; k += N) {
      const int h = m.hP[k], e = m.eP[k], q = m.rQ[h], f = m.eQ[q];
      const double cx = m.x[h], cy = m.y[h];
      const int hm = k > 0 && m.eP[k - 1] == e ? m.hP[k - 1] : -1;
      const int hp = k + 1 < K && m.eP[k + 1] == e ? m.hP[k + 1] : -1;
      const int gm = q > startC(f) ? m.hQ[q - 1] : -1, gp = q + 1 < m.endC[f] ? m.hQ[q + 1] : -1;
      // a crossing next to this one on both polygons: another label
      if ((hm >= 0 && (hm == gm || hm == gp)) || (hp >= 0 && (hp == gm || hp == gp))) {
        bad = true;
        break;
      }
      // nor two crossings of an edge at one point (provenance by coordinates)
      auto at = [&](int o) { return o >= 0 && same_value(m.x[o], cx) && same_value(m.y[o], cy); };
      if (at(hm) || at(hp) || at(gm) || at(gp)) {
        bad = true;
        break;
      }
      const int e2 = bsucc(e), f2 = csucc(f);
      const double pmx = hm >= 0 ? m.x[hm] : b[2 * e], pmy = hm >= 0 ? m.y[hm] : b[2 * e + 1];
      const double ppx = hp >= 0 ? m.x[hp] : b[2 * e2], ppy = hp >= 0 ? m.y[hp] : b[2 * e2 + 1];
      const double s3 = area3(pmx, pmy, cx, cy, ppx, ppy);
      auto right = [&](double qx, double qy) {
        const double s1 = area3(qx, qy, pmx, pmy, cx, cy), s2 = area3(qx, qy, cx, cy, ppx, ppy);
        if (is_pos(s3)) return !(is_pos(s1) && is_pos(s2));
        return is_neg(s1) && is_neg(s2);
      };
      const bool rm = gm >= 0 ? right(m.x[gm], m.y[gm]) : right(c[2 * f], c[2 * f + 1]);
      const bool rp = gp >= 0 ? right(m.x[gp], m.y[gp]) : right(c[2 * f2], c[2 * f2 + 1]);
      if (rm == rp) bad = true;
    }
    if (g.any(bad)) return out(Left<4>{}, CLEAN_NOT);
  }
  g.phase();
  // ---- components, and whether each one's first vertex lies in the other
  // polygon (pointInPoly over the list's edges): a thread per polygon edge
  // without crossings and per piece between two list nodes, not per edge (an
  // edge near the ray can hold most of a pair's crossings)
  const int ncb = in.bnx ? clean_components(g, nb, in.bnx, in.rootB) : 1;
  const int ncc = in.cnx ? clean_components(g, nc, in.cnx, in.rootC) : 1;
  // The few pieces whose orientation decides go on a list (over A and B), so
  // that their FP64 runs once, in full warps.
  auto inside = [&](bool overlay, double rx, double ry) {
    const double* p = overlay ? c : b;
    const bool sparse = kSparse && !overlay;
    const int* list = overlay ? m.hQ : m.hP;
    const int* edge = overlay ? m.eQ : m.eP;
    double2 *from = (double2*)m.A, *to = (double2*)m.B;
    int part = 0, listed = 0;  // (listed: a warp's; a block's is shared)
    if constexpr (G::kBlock) {
      if (lane == 0) g.s->count = 0;
      g.sync();
    }
    auto piece = [&](bool act, double x0, double y0, double x1, double y1) {
      bool area = false;
      const int d = act ? pip_quick(x0, y0, x1, y1, rx, ry, &area) : 0;
      if (!area) part += d;
      const unsigned w = __ballot_sync(0xffffffffu, area);
      if (w == 0u) return;
      int at = listed;
      if constexpr (G::kBlock) {
        if ((lane & 31) == 0) at = atomicAdd(&g.s->count, __popc(w));
        at = __shfl_sync(0xffffffffu, at, 0);
      } else {
        listed += __popc(w);
      }
      at += __popc(w & ((1u << (lane & 31)) - 1u));
      if (area && at < K + 4) {
        from[at] = make_double2(x0, y0);
        to[at] = make_double2(x1, y1);
      } else if (area) {
        part += pip_decide(x0, y0, x1, y1, rx, ry);
      }
    };
    const int n = sparse ? 0 : overlay ? nc : nb;
    for (int e0 = 0; e0 < n; e0 += N) {
      const int e = e0 + lane;
      double x0 = 0.0, y0 = 0.0, x1 = 0.0, y1 = 0.0;
      bool act = e < n;
      if (act) {
        x0 = p[2 * e];
        y0 = p[2 * e + 1];
        if (abs_bits(x0) > kInfBits || abs_bits(y0) > kInfBits) bad = true;
        act = (overlay ? countC(e) : countB(e)) == 0;
      }
      if (act) {
        const int e2 = overlay ? csucc(e) : bsucc(e);
        x1 = p[2 * e2];
        y1 = p[2 * e2 + 1];
      }
      piece(act, x0, y0, x1, y1);
    }
    for (int k0 = 0; k0 < K; k0 += N) {  // the piece that ends at crossing k, and the last
      const int k = k0 + lane;
      const bool act = k < K;
      int e = 0;
      bool last = false;
      double x0 = 0.0, y0 = 0.0, x1 = 0.0, y1 = 0.0, x2 = 0.0, y2 = 0.0;
      if (act) {
        const int h = list[k];
        e = edge[k];
        if (k == 0 || edge[k - 1] != e) {
          x0 = p[2 * e];
          y0 = p[2 * e + 1];
        } else {
          x0 = m.x[list[k - 1]];
          y0 = m.y[list[k - 1]];
        }
        x1 = m.x[h];
        y1 = m.y[h];
        last = k + 1 == K || edge[k + 1] != e;
        if (last) {
          const int e2 = overlay ? csucc(e) : bsucc(e);
          x2 = p[2 * e2];
          y2 = p[2 * e2 + 1];
        }
      }
      piece(act, x0, y0, x1, y1);
      piece(last, x1, y1, x2, y2);
      if (sparse && last) part -= pip_step(p[2 * e], p[2 * e + 1], x2, y2, rx, ry);
    }
    g.sync();
    if constexpr (G::kBlock) listed = g.s->count;
    if (listed > K + 4) listed = K + 4;
    for (int i = lane; i < listed; i += N) {
      const double2 u = from[i], v = to[i];
      part += pip_decide(u.x, u.y, v.x, v.y, rx, ry);
    }
    return (g.sum(part) + (sparse ? in.base_steps : 0)) & 1;
  };
  int inP = 0, inQ = 0;  // of a single component
  if (ncb == 1) inP = inside(true, b[0], b[1]);
  if (ncc == 1) inQ = inside(false, c[0], c[1]);
  for (int side = 0; side < 2; ++side) {
    const int n = side ? ncc : ncb;
    if (n == 1) continue;
    for (int k = 0; k < n; ++k) {
      const int v = side ? in.rootC[k] : in.rootB[k];
      const int x = side ? inside(false, c[2 * v], c[2 * v + 1]) : inside(true, b[2 * v], b[2 * v + 1]);
      if (lane == 0) (side ? in.inC : in.inB)[k] = x;
    }
  }
  // a component: its vertices [v0, v1), its crossings [lo, hi), and whether
  // its first vertex is inside
  struct Comp {
    int v0, v1, lo, hi, in;
  };
  auto comp = [&](int side, int k) {
    Comp r;
    if (side) {
      r.v0 = ncc == 1 ? 0 : in.rootC[k];
      r.v1 = ncc == 1 ? nc : in.rootC[k + 1];
      r.lo = startC(r.v0);
      r.hi = m.endC[r.v1 - 1];
      r.in = ncc == 1 ? inQ : in.inC[k];
    } else {
      r.v0 = ncb == 1 ? 0 : in.rootB[k];
      r.v1 = ncb == 1 ? nb : in.rootB[k + 1];
      r.lo = kSparse ? 0 : startB(r.v0);
      r.hi = kSparse ? K : m.endB[r.v1 - 1];
      r.in = ncb == 1 ? inP : in.inB[k];
    }
    return r;
  };
  auto comp_of = [&](int side, int e) {  // of the edge (or vertex) e
    int lo = 0, hi = (side ? ncc : ncb) - 1;
    const int* root = side ? in.rootC : in.rootB;
    while (lo < hi) {
      const int x = (lo + hi + 1) >> 1;
      if (root[x] <= e) lo = x;
      else hi = x - 1;
    }
    return comp(side, lo);
  };
  if (g.any(bad)) return out(Left<3>{}, CLEAN_NOT);  // also: the flags are visible
  for (int side = 0; side < 2; ++side)
    for (int k = lane; k < (side ? ncc : ncb); k += N) {
      const Comp r = comp(side, k);
      if ((r.hi - r.lo) & 1) bad = true;
    }
  if (g.any(bad)) return out(Left<3>{}, CLEAN_NOT);
  g.phase();
  // ---- rings: first the components without crossings that lie inside (or
  // outside, for the union), whole and in order
  int rings = 0, verts = 0;
  for (int side = 0; side < 2; ++side)
    for (int k = 0; k < (side ? ncc : ncb); ++k) {
      const Comp r = comp(side, k);
      if (r.hi != r.lo || !(r.in ^ in.unite)) continue;
      if (rings >= in.rcap) return out(Left<2>{}, CLEAN_NOT);
      if (verts + r.v1 - r.v0 > in.vcap) return out(Left<2>{}, CLEAN_ROOM);
      const double* p = side ? c : b;
      for (int v = r.v0 + lane; v < r.v1; v += N) {
        const int at = verts + v - r.v0;
        in.rxy[2 * at] = p[2 * v];
        in.rxy[2 * at + 1] = p[2 * v + 1];
        in.tape[at] = make_int4(side, v, 0, rings);
      }
      if (lane == 0) in.roff[rings] = verts;
      ++rings;
      verts += r.v1 - r.v0;
    }
  // ---- then the traced ones.  The legs from crossing k (rank along the
  // base): along the base to crossing kp, then along the overlay, from its
  // rank m1 to m2, which is crossing kn
  struct Leg {
    int e, cnt, v0, v1, to;  // cnt vertices from edge e on, to the crossing of rank `to`
    bool fwd;
  };
  auto leg = [&](int side, int k) {
    const int* ek = side ? m.eQ : m.eP;
    Leg l;
    l.e = ek[k];
    const Comp r = (side ? ncc : ncb) == 1 ? comp(side, 0) : comp_of(side, l.e);
    const int entry = (r.in ^ 1) ^ ((k - r.lo) & 1);
    l.fwd = entry != in.unite;
    l.to = l.fwd ? (k + 1 == r.hi ? r.lo : k + 1) : (k == r.lo ? r.hi - 1 : k - 1);
    l.v0 = r.v0;
    l.v1 = r.v1;
    l.cnt = l.fwd ? ek[l.to] - l.e : l.e - ek[l.to];
    if (l.cnt < 0 || (l.cnt == 0 && (l.fwd ? l.to < k : l.to > k))) l.cnt += r.v1 - r.v0;
    return l;
  };
  int4* A = m.A;
  int4* B = m.B;
  for (int k = lane; k < K; k += N) {
    const Leg p = leg(0, k), q = leg(1, m.rQ[m.hP[p.to]]);
    A[k] = make_int4(m.rP[m.hQ[q.to]], k, 0, p.cnt + q.cnt + 2);
  }
  g.sync();
  // orbits of k -> kn (see pw_label_trace_block): the least crossing, and the
  // vertices to it
  while (K > 0) {
    bool changed = false;
    for (int k = lane; k < K; k += N) {
      int4 x = A[k];
      const int4 y = A[x.x];
      if (y.y < x.y) {
        x.y = y.y;
        x.z = (int)((unsigned)x.w + (unsigned)y.z);
        changed = true;
      }
      x.x = y.x;
      x.w = (int)((unsigned)x.w + (unsigned)y.w);
      B[k] = x;
    }
    int4* t = A;
    A = B;
    B = t;
    if (!g.any(changed)) break;
  }
  // B: {offset, length, number} of the ring, at its first crossing
  for (int i0 = 0; i0 < K; i0 += N) {
    const int k = i0 + lane;
    int len = 0;
    if (k < K && A[k].y == k) {
      const Leg p = leg(0, k);
      if (k < A[p.to].y) {
        const Leg q = leg(1, m.rQ[m.hP[p.to]]);
        len = p.cnt + q.cnt + 2 + A[m.rP[m.hQ[q.to]]].z;
      }
    }
    int tr, tv;
    const int r = rings + g.before(len > 0, &tr);
    const int o = verts + g.excl(len, &tv);
    if (len > 0) {
      B[k] = make_int4(o, len, r, 0);
      if (r < in.rcap) in.roff[r] = o;
    }
    rings += tr;
    verts += tv;
  }
  if (rings > in.rcap) return out(Left<2>{}, CLEAN_NOT);
  if (verts > in.vcap) return out(Left<2>{}, CLEAN_ROOM);
  if (lane == 0) in.roff[rings] = verts;
  g.sync();
  g.phase();
  // the legs to their places: a lane writes a short one, the warp a long one
  constexpr int kShort = 8;
  for (int i0 = 0; i0 < K; i0 += N) {
    const int k = i0 + lane;
    bool act = false;
    Leg p{}, q{};
    int at = 0, ring = 0;
    if (k < K) {
      p = leg(0, k);
      const int s = A[k].y;
      act = s < A[p.to].y;  // this sense of the cycle
      if (act) {
        q = leg(1, m.rQ[m.hP[p.to]]);
        const int4 o = B[s];
        at = o.x + (s == k ? 0 : o.y - A[k].z);
        ring = o.z;
      }
    }
    for (int side = 0; side < 2; ++side) {
      const Leg& l = side ? q : p;
      const double* poly = side ? c : b;
      auto put = [&](int e, int fwd, int v0, int v1, int to, int r, int t) {
        int u = fwd ? e + 1 + t : e - t;
        if (u >= v1) u -= v1 - v0;
        if (u < v0) u += v1 - v0;
        in.rxy[2 * to] = poly[2 * u];
        in.rxy[2 * to + 1] = poly[2 * u + 1];
        in.tape[to] = make_int4(side, u, 0, r);
      };
      if (act) {
        if (l.cnt <= kShort)
          for (int t = 0; t < l.cnt; ++t) put(l.e, l.fwd, l.v0, l.v1, at + t, ring, t);
        const int h = side ? m.hQ[l.to] : m.hP[l.to], to = at + l.cnt;
        in.rxy[2 * to] = m.x[h];
        in.rxy[2 * to + 1] = m.y[h];
        in.tape[to] = make_int4(2, hits.b(h), hits.c(h), ring);
      }
      __syncwarp();
      for (unsigned w = __ballot_sync(0xffffffffu, act && l.cnt > kShort); w; w &= w - 1) {
        const int src = __ffs(w) - 1;
        const int e = __shfl_sync(0xffffffffu, l.e, src), cnt = __shfl_sync(0xffffffffu, l.cnt, src);
        const int fwd = __shfl_sync(0xffffffffu, (int)l.fwd, src);
        const int v0 = __shfl_sync(0xffffffffu, l.v0, src), v1 = __shfl_sync(0xffffffffu, l.v1, src);
        const int to = __shfl_sync(0xffffffffu, at, src), r = __shfl_sync(0xffffffffu, ring, src);
        for (int t = threadIdx.x & 31; t < cnt; t += 32) put(e, fwd, v0, v1, to + t, r, t);
      }
      at += l.cnt + 1;
    }
  }
  g.sync();
  g.phase();
  // ---- cleanUpResult2 (foster/polyclip.h:767-787): a vertex with |area3| <
  // eps goes.  And the area: the shoelace terms in an order that the rings and
  // the group size fix.
  auto area_at = [&](int u, int v, int x) {
    return area3(in.rxy[2 * u], in.rxy[2 * u + 1], in.rxy[2 * v], in.rxy[2 * v + 1],
                 in.rxy[2 * x], in.rxy[2 * x + 1]);
  };
  auto term = [&](double s, int v, int vp) {
    return dadd(s, dsub(dmul(in.rxy[2 * v], in.rxy[2 * vp + 1]),
                        dmul(in.rxy[2 * vp], in.rxy[2 * v + 1])));
  };
  double s2 = 0.0;
  bool flat = false;
  for (int v = lane; v < verts; v += N) {
    const int r = in.tape[v].w, s = in.roff[r], e = in.roff[r + 1];
    const int vp = v + 1 == e ? s : v + 1;
    if (abs_lt(area_at(v == s ? e - 1 : v - 1, v, vp), kEps)) {
      flat = true;
      in.tape[v].w = ~r;
    }
    s2 = term(s2, v, vp);
  }
  if (g.any(flat)) {  // (rare: one pair in thousands of random ones)
    // The reference's walk, a thread per ring, over links that start as the
    // ring's order; a vertex with its first neighbours that was not flat then
    // is passed over.  tape[].w < 0 ends as "removed".
    for (int v = lane; v < verts; v += N) {
      const int w = in.tape[v].w, r = w < 0 ? ~w : w, s = in.roff[r], e = in.roff[r + 1];
      in.nxt[v] = v + 1 == e ? s : v + 1;
      in.prv[v] = v == s ? e - 1 : v - 1;
    }
    g.sync();
    for (int r = lane; r < rings; r += N) {
      const int s = in.roff[r], e = in.roff[r + 1];
      int root = s;
      auto is_flat = [&](int v) { return abs_lt(area_at(in.prv[v], v, in.nxt[v]), kEps); };
      auto remove = [&](int v) {
        if (root == v) {
          root = in.nxt[v];
          if (in.nxt[root] == root) root = -1;
        }
        in.nxt[in.prv[v]] = in.nxt[v];
        in.prv[in.nxt[v]] = in.prv[v];
        in.tape[v].w = ~r;
      };
      while (root >= 0 && is_flat(root)) remove(root);
      if (root < 0) {
        for (int v = s; v < e; ++v) in.tape[v].w = ~r;
      } else {
        for (int v = root; v < e; ++v) {
          if (in.tape[v].w >= 0 && in.prv[v] == v - 1 && in.nxt[v] == v + 1) continue;
          if (is_flat(v)) remove(v);
          else in.tape[v].w = r;
        }
      }
      in.nxt[s] = root;  // (the ring's links are done with)
    }
    g.sync();
    // the rings left get new numbers; each vertex: its ring's, and whether it
    // is the first
    int left = 0;
    for (int r0 = 0; r0 < rings; r0 += N) {
      const int r = r0 + lane;
      const bool keep = r < rings && in.nxt[in.roff[r]] >= 0;
      int n;
      const int id = left + g.before(keep, &n);
      if (r < rings) in.prv[in.roff[r]] = id;
      left += n;
    }
    g.sync();
    for (int v = lane; v < verts; v += N) {
      const int r = in.tape[v].w;
      if (r < 0) continue;
      const int s = in.roff[r];
      in.tape[v].w = 2 * in.prv[s] + (in.nxt[s] == v);
    }
    g.sync();
    int kept = 0;
    for (int v0 = 0; v0 < verts; v0 += N) {  // to lower places, chunk by chunk
      const int v = v0 + lane;
      int4 t = make_int4(0, 0, 0, -1);
      double x = 0.0, y = 0.0;
      if (v < verts) {
        t = in.tape[v];
        x = in.rxy[2 * v];
        y = in.rxy[2 * v + 1];
      }
      g.sync();
      const bool first = t.w & 1;
      int n;
      const int to = kept + g.before(t.w >= 0, &n);
      kept += n;
      if (t.w >= 0) {
        t.w >>= 1;
        in.tape[to] = t;
        in.rxy[2 * to] = x;
        in.rxy[2 * to + 1] = y;
        if (first) in.roff[t.w] = to;
      }
      g.sync();
    }
    verts = kept;
    rings = left;
    if (lane == 0) in.roff[rings] = verts;
    g.sync();
    s2 = 0.0;
    for (int v = lane; v < verts; v += N) {
      const int r = in.tape[v].w, e = in.roff[r + 1];
      s2 = term(s2, v, v + 1 == e ? in.roff[r] : v + 1);
    }
  }
  for (int o = 16; o > 0; o >>= 1) s2 = dadd(s2, __shfl_xor_sync(0xffffffffu, s2, o));
  if constexpr (G::kBlock) {
    if ((lane & 31) == 0) s_sum[g.warp()] = s2;
    g.sync();
    s2 = s_sum[0];
    for (int k = 1; k < G::kWarps; ++k) s2 = dadd(s2, s_sum[k]);
  }
  *nrings_out = rings;
  *nverts_out = verts;
  *area_out = dmul(0.5, s2);
  return CLEAN_DONE;
}

}  // namespace
}  // namespace sbc
