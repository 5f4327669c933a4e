// sbc_general.cu -- rows A9-A18 of a pair in general position, data-parallel
// over the whole GPU, straight from the exact stage's hits to rings.
//
// The same observation as sbc_clean.cuh, for the pair pipeline: where every
// hit is a proper crossing labelled a crossing, the merged arrays, labels and linked lists
// (src/clip.cpp:368-695, foster/polyclip.h:337-787) say no more than the order
// of the crossings along each polygon.  Crossings are ranked along both
// polygons (counting sort by edge, alpha order per edge); entry and exit
// alternate from each polygon's first vertex; the rings are the alternating
// cycles of the two neighbour pairings; pointer doubling over the crossings
// gives each leg of each ring its place.  About 16 launches and one host
// read, where the stages that build the arrays take 65 launches, 25 memsets
// and four host reads.  A pair that fails a test takes those stages, from the
// same hits; so does a request for their arrays (Pipeline::build_records).
// Where a result vertex may lie in line with its neighbours the clean-up
// kernels of the list-ranking back end follow (clean_up_rings).
//
// Bound by dependent gathers over the crossings (a few hundred bytes each,
// L2-resident) and, below some 10,000 vertices, by the launches.  A clip
// through host arrays, before and after: 24 x 18 vertices 650 and 335 us,
// 10,000 x 8,000 1.48 and 0.85 ms, 1M x 1M 2.71 and 1.95 ms; five overlays in
// one tree 3.50 and 1.52 ms.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "sbc_group.cuh"
#include "sbc_pairops.cuh"
#include "sbc_pipeline.cuh"
#include "sbc_serial.cuh"

namespace sbc {

namespace {

// A hit h has rank rP[h] along the base and rQ[h] along the overlay (hP and
// hQ are the inverses, eP and eQ the edges by rank); endB[e] is one past base
// edge e's last rank.
struct Gp {
  int K, nb, nc, cStart, unite;
  const int *rb, *rc, *rt;
  const unsigned long long* rkey;
  const double2* rab;
  const double *b, *c;  // each with its closing vertex
  int *endB, *endC;
  int *hP, *hQ, *rP, *rQ, *eP, *eQ, *aB, *aC;
  double2* xy;
  int4 *A, *B;
  int* wind;      // winding number of the base's first vertex in the overlay, and the reverse
  unsigned* bad;  // 1: not in general position, 2: a vertex in line with its neighbours
  int* longs;     // edges with many crossings (base edges, then nb + overlay edges)
  unsigned* nlong;
  __device__ int cedge(int h) const { return (rc[h] >> 1) - cStart; }
  __device__ int startB(int e) const { return e == 0 ? 0 : endB[e - 1]; }
  __device__ int startC(int e) const { return e == 0 ? 0 : endC[e - 1]; }
  // record order (base edge, then first emission) breaks ties in alpha
  __device__ bool lessB(int u, int v) const {
    return aB[u] != aB[v] ? aB[u] < aB[v] : rkey[u] < rkey[v];
  }
  __device__ bool lessC(int u, int v) const {
    if (aC[u] != aC[v]) return aC[u] < aC[v];
    return rb[u] != rb[v] ? rb[u] < rb[v] : rkey[u] < rkey[v];
  }
};

__global__ void k_gp_hits(Gp g) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= g.K) return;
  const int e = g.rb[h] >> 1, f = g.cedge(h);
  atomicAdd(&g.endB[e], 1);
  atomicAdd(&g.endC[f], 1);
  const double2 ab = g.rab[h];
  // the crossing (saveIntersectionsParallel, oacc_segment_tree.cpp:7257-7341)
  const double2 p1 = ((const double2*)g.b)[e], p2 = ((const double2*)g.b)[e + 1];
  const double2 q1 = ((const double2*)g.c)[f], q2 = ((const double2*)g.c)[f + 1];
  const double oma = dsub(1.0, ab.x);
  const double x = dadd(dmul(oma, p1.x), dmul(ab.x, p2.x));
  const double y = dadd(dmul(oma, p1.y), dmul(ab.x, p2.y));
  g.xy[h] = make_double2(x, y);
  const int a = alpha_to_int(ab.x), t = alpha_to_int(ab.y);
  g.aB[h] = a % 1000000000;
  g.aC[h] = t % 1000000000;
  // a slot equal to the next vertex stops the list walk early
  auto meets = [&](double2 p) { return p.x == x && p.y == y; };
  if (g.rt[h] != 1 || a < 0 || t < 0 || meets(p1) || meets(p2) || meets(q1) || meets(q2)) *g.bad = 1u;
}

__global__ void k_gp_scatter(Gp g) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= g.K) return;
  g.hP[atomicAdd(&g.endB[g.rb[h] >> 1], 1)] = h;  // a start moves up to its end
  g.hQ[atomicAdd(&g.endC[g.cedge(h)], 1)] = h;
}

// The crossings of each edge in alpha order: a lane per edge up to 4 of them,
// the warp up to 128 (each lane ranks up to four against all), a block above
// (k_gp_order_long).  With the warp's line at 32, 10,000 x 8,000 stars (19 to
// 24 crossings an edge, up to a hundred) left 0.17 ms to the blocks.
constexpr int kGpLane = 4, kGpWarp = 128, kGpLongMost = 4096;
// A warp looks after `per` edges: 32, or 4 where edges have many crossings (a
// warp's edges take turns).
__global__ void __launch_bounds__(256) k_gp_order(Gp g, int per) {
  const int lane = threadIdx.x & 31;
  const int x = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per + lane;
  const int n = g.nb + g.nc;
  const bool base = x < g.nb;
  int s = 0, m = 0;
  if (lane < per && x < n) {
    const int e = base ? x : x - g.nb;
    s = base ? g.startB(e) : g.startC(e);
    m = (base ? g.endB[e] : g.endC[e]) - s;
  }
  if (m > 1 && m <= kGpLane) {
    int* v = (base ? g.hP : g.hQ) + s;
    for (int i = 1; i < m; ++i) {
      const int h = v[i];
      int j = i;
      while (j > 0 && (base ? g.lessB(h, v[j - 1]) : g.lessC(h, v[j - 1]))) {
        v[j] = v[j - 1];
        --j;
      }
      v[j] = h;
    }
  } else if (m > kGpWarp) {
    if (m > kGpLongMost) *g.bad = 1u;
    else g.longs[atomicAdd(g.nlong, 1u)] = x;
  }
  for (unsigned w = __ballot_sync(0xffffffffu, m > kGpLane && m <= kGpWarp); w; w &= w - 1) {
    const int src = __ffs(w) - 1;
    const int ss = __shfl_sync(0xffffffffu, s, src), mm = __shfl_sync(0xffffffffu, m, src);
    const bool bb = __shfl_sync(0xffffffffu, (int)base, src);
    int* v = (bb ? g.hP : g.hQ) + ss;
    if (mm <= 32) {
      const int h = lane < mm ? v[lane] : -1;
      const int a = lane < mm ? (bb ? g.aB[h] : g.aC[h]) : INT_MAX;
      int rank = 0;
      bool tie = false;
      for (int j = 0; j < mm; ++j) {
        const int aj = __shfl_sync(0xffffffffu, a, j);
        rank += aj < a;
        tie |= aj == a && j != lane;
      }
      if (__any_sync(0xffffffffu, tie && lane < mm)) {
        rank = 0;
        if (lane < mm)
          for (int j = 0; j < mm; ++j) rank += bb ? g.lessB(v[j], h) : g.lessC(v[j], h);
      }
      __syncwarp();
      if (lane < mm) v[rank] = h;
      __syncwarp();
      continue;
    }
    constexpr int kPer = kGpWarp / 32;
    int h[kPer], a[kPer], rank[kPer];
    bool tie = false;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * 32 + lane;
      h[u] = i < mm ? v[i] : -1;
      a[u] = i < mm ? (bb ? g.aB[h[u]] : g.aC[h[u]]) : INT_MAX;
      rank[u] = 0;
    }
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int left = min(32, mm - t * 32);
      for (int j = 0; j < left; ++j) {
        const int aj = __shfl_sync(0xffffffffu, a[t], j);
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          rank[u] += aj < a[u];
          tie |= aj == a[u] && h[u] >= 0 && (u != t || j != lane);
        }
      }
    }
    if (__any_sync(0xffffffffu, tie)) {
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        if (h[u] < 0) continue;
        rank[u] = 0;
        for (int j = 0; j < mm; ++j) rank[u] += bb ? g.lessB(v[j], h[u]) : g.lessC(v[j], h[u]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (h[u] >= 0) v[rank[u]] = h[u];
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256) k_gp_order_long(Gp g) {
  using G = BlockGroup<256>;
  __shared__ G::Shared sh;
  G grp(&sh);
  const unsigned cnt = *g.nlong;
  for (unsigned i = blockIdx.x; i < cnt; i += gridDim.x) {
    const int x = g.longs[i];
    const bool base = x < g.nb;
    const int e = base ? x : x - g.nb;
    const int s = base ? g.startB(e) : g.startC(e), m = (base ? g.endB[e] : g.endC[e]) - s;
    int* v = (base ? g.hP : g.hQ) + s;
    unsigned* scr = (unsigned*)(base ? g.A : g.B) + 4 * (size_t)s;  // the edge's own part
    const int np = npow2_dev(m);
    for (int k = grp.rank(); k < np; k += 256) scr[k] = k < m ? (unsigned)v[k] : ~0u;
    grp.sync();
    group_bitonic(grp, np, [&](int p, int q, bool up) {
      const unsigned u = scr[p], w = scr[q];
      auto less = [&](unsigned a, unsigned b) {
        if (a == ~0u || a == b) return false;
        return b == ~0u || (base ? g.lessB((int)a, (int)b) : g.lessC((int)a, (int)b));
      };
      if (up ? less(w, u) : less(u, w)) {
        scr[p] = w;
        scr[q] = u;
      }
    });
    for (int k = grp.rank(); k < m; k += 256) v[k] = (int)scr[k];
    grp.sync();
  }
}

__global__ void k_gp_rank(Gp g) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g.K) return;
  const int h = g.hP[k], q = g.hQ[k];
  g.rP[h] = k;
  g.eP[k] = g.rb[h] >> 1;
  g.rQ[q] = k;
  g.eQ[k] = g.cedge(q);
}

// pointInPoly (foster/polygon.h:427-448) of each polygon's first vertex in the
// other, over the list's edges: blockIdx.y 0 the overlay's edges, 1 the base's.
// Few polygon edges reach the ray's height; a warp takes each of those with
// its crossings together (an edge may have hundreds).
__global__ void __launch_bounds__(256) k_gp_pip(Gp g) {
  const bool base = blockIdx.y == 1;
  const int n = base ? g.nb : g.nc;
  const double2* p = (const double2*)(base ? g.b : g.c);
  const double2 r = ((const double2*)(base ? g.c : g.b))[0];
  int part = 0;
  const int lane = threadIdx.x & 31;
  for (int e0 = blockIdx.x * blockDim.x + threadIdx.x - lane; e0 < n; e0 += gridDim.x * blockDim.x) {
    const int e = e0 + lane;
    double2 u = make_double2(0.0, 0.0), v = u;
    int s = 0, t = 0;
    bool near = false;
    if (e < n) {
      u = p[e];
      v = p[e + 1];
      if (!(u.x == u.x && u.y == u.y)) *g.bad = 1u;
      near = ray_near(u.y, v.y, r.y);
      if (near && g.K > 0) {
        s = base ? g.startB(e) : g.startC(e);
        t = base ? g.endB[e] : g.endC[e];
      }
      if (near && t == s) part += pip_step(u.x, u.y, v.x, v.y, r.x, r.y);
    }
    for (unsigned w = __ballot_sync(0xffffffffu, near && t > s); w; w &= w - 1) {
      const int src = __ffs(w) - 1, ee = e0 + src;
      const int ss = __shfl_sync(0xffffffffu, s, src), m = __shfl_sync(0xffffffffu, t, src) - ss;
      // pieces 0 .. m: from point i - 1 (the vertex before all) to point i
      for (int i = lane; i <= m; i += 32) {
        const int* hs = base ? g.hP : g.hQ;
        const double2 a = i == 0 ? p[ee] : g.xy[hs[ss + i - 1]];
        const double2 b = i == m ? p[ee + 1] : g.xy[hs[ss + i]];
        part += pip_step(a.x, a.y, b.x, b.y, r.x, r.y);
      }
    }
  }
  part = __reduce_add_sync(0xffffffffu, part);
  if ((threadIdx.x & 31) == 0 && part) atomicAdd(&g.wind[base ? 1 : 0], part);
}

// The leg from the crossing of rank k along one polygon: cnt vertices from
// edge e on, to the crossing of rank `to`.
struct GpLeg {
  int e, cnt, to;
  bool fwd;
};
__device__ __forceinline__ GpLeg gp_leg(const Gp& g, int side, int inside, int k) {
  const int* ek = side ? g.eQ : g.eP;
  GpLeg l;
  l.e = ek[k];
  const int entry = (inside ^ 1) ^ (k & 1);
  l.fwd = entry != g.unite;
  l.to = l.fwd ? (k + 1 == g.K ? 0 : k + 1) : (k == 0 ? g.K - 1 : k - 1);
  l.cnt = l.fwd ? ek[l.to] - l.e : l.e - ek[l.to];
  if (l.cnt < 0 || (l.cnt == 0 && (l.fwd ? l.to < k : l.to > k))) l.cnt += side ? g.nc : g.nb;
  return l;
}

// In line with its neighbours as cleanUpResult2 (foster/polyclip.h:767-787)
// sees it, in either order of the ring: each order's area3 rounds the products
// about its own first point.  With m the largest difference from p, either
// area is within 1.3e-15 m^2 of the exact one (2^-53 times 16.4 m^2 about q,
// whose differences reach 2 m, and 8.2 m^2 about p), so the two differ by less
// than 4e-15 m^2 < 2^(2 e - 45) for m < 2^(e + 1), and one area above twice the
// larger of that and kEps settles both, as nearly all do.  By the words that
// hold the exponents: k_gp_legs is bound by FP64, and with this threshold as
// two FP64 operations it takes 98 us for a 1M x 1M clip, so 72.
__device__ __forceinline__ bool gp_flat(double2 p, double2 v, double2 q) {
  auto high = [](double x) { return __double2hiint(x) & 0x7fffffff; };
  const double a = area3(p.x, p.y, v.x, v.y, q.x, q.y);
  const int m = max(max(high(dsub(v.x, p.x)), high(dsub(v.y, p.y))),
                    max(high(dsub(q.x, p.x)), high(dsub(q.y, p.y))));
  const int t = max(min(2 * (m >> 20) - 1067, 0x7ff) * (1 << 20), __double2hiint(2.0 * kEps));
  if (high(a) > t && high(a) < 0x7ff00000) return false;
  return abs_lt(a, kEps) || abs_lt(area3(q.x, q.y, v.x, v.y, p.x, p.y), kEps);
}

// Per crossing: its label (calculateInitLabelParallel, oacc_segment_tree.cpp:
// 7925-7988), whether it stays in the result, and its first step of the
// pointer doubling.  Per vertex: whether it stays in the result.
__global__ void __launch_bounds__(256) k_gp_legs(Gp g) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int inP = g.wind[0] & 1, inQ = g.wind[1] & 1;
  const double2* b = (const double2*)g.b;
  const double2* c = (const double2*)g.c;
  if (x < g.K) {
    const int k = x, h = g.hP[k], e = g.eP[k], m = g.rQ[h], f = g.eQ[m];
    const double2 v = g.xy[h];
    const int hm = k > g.startB(e) ? g.hP[k - 1] : -1, hp = k + 1 < g.endB[e] ? g.hP[k + 1] : -1;
    const int gm = m > g.startC(f) ? g.hQ[m - 1] : -1, gp = m + 1 < g.endC[f] ? g.hQ[m + 1] : -1;
    const double2 pm = hm >= 0 ? g.xy[hm] : b[e], pp = hp >= 0 ? g.xy[hp] : b[e + 1];
    const double2 qm = gm >= 0 ? g.xy[gm] : c[f], qp = gp >= 0 ? g.xy[gp] : c[f + 1];
    bool bad = (hm >= 0 && (hm == gm || hm == gp || g.rc[hm] == g.rc[h])) ||
               (hp >= 0 && (hp == gm || hp == gp));
    // nor two crossings of an edge at one point: the provenance of such a ring
    // vertex is its first record's, and the hits here are in no order
    auto at = [&](double2 q) { return same_value(q.x, v.x) && same_value(q.y, v.y); };
    if (at(pm) || at(pp) || at(qm) || at(qp)) bad = true;
    const double s3 = area3(pm.x, pm.y, v.x, v.y, pp.x, pp.y);
    auto right = [&](double2 q) {
      const double s1 = area3(q.x, q.y, pm.x, pm.y, v.x, v.y);
      const double s2 = area3(q.x, q.y, v.x, v.y, pp.x, pp.y);
      if (s3 > 0) return !(s1 > 0 && s2 > 0);
      return s1 < 0 && s2 < 0;
    };
    if (right(qm) == right(qp)) bad = true;
    const GpLeg p = gp_leg(g, 0, inP, k), own = gp_leg(g, 1, inQ, m);
    // its neighbours in the result: along each polygon in the leg's direction
    if (gp_flat(p.fwd ? pp : pm, v, own.fwd ? qp : qm)) atomicOr(g.bad, 2u);
    if (bad) *g.bad = 1u;
    const GpLeg q = gp_leg(g, 1, inQ, g.rQ[g.hP[p.to]]);
    g.A[k] = make_int4(g.rP[g.hQ[q.to]], k, 0, p.cnt + q.cnt + 2);
    return;
  }
  const int y = x - g.K;
  if (y >= g.nb + g.nc) return;
  const bool base = y < g.nb;
  const int u = base ? y : y - g.nb, n = base ? g.nb : g.nc;
  const int* end = base ? g.endB : g.endC;
  const int* hs = base ? g.hP : g.hQ;
  const double2* p = base ? b : c;
  const int s = u == 0 ? 0 : end[u - 1];  // crossings before vertex u
  const int in = (base ? inP : inQ) ^ (s & 1);
  if (!(in ^ g.unite)) return;  // not in the result
  const int pe = u == 0 ? n - 1 : u - 1, ps = pe == 0 ? 0 : end[pe - 1], pt = end[pe];
  const double2 prev = pt > ps ? g.xy[hs[pt - 1]] : p[pe];
  const double2 next = end[u] > s ? g.xy[hs[s]] : p[u + 1];
  if (gp_flat(prev, p[u], next)) atomicOr(g.bad, 2u);
}

// One doubling round over this thread's crossings: x = (next, least crossing
// of the window, vertices to it, vertices of the window).
__device__ __forceinline__ bool gp_round(int K, const int4* __restrict__ in, int4* __restrict__ out,
                                         int first, int step) {
  bool changed = false;
  constexpr int kBatch = 4;  // loads in flight
  for (int k0 = first; k0 < K; k0 += kBatch * step) {
    int4 x[kBatch], y[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int k = k0 + u * step;
      x[u] = k < K ? __ldcg(&in[k]) : make_int4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) y[u] = __ldcg(&in[x[u].x]);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int k = k0 + u * step;
      if (k >= K) continue;
      if (y[u].y < x[u].y) {
        x[u].y = y[u].y;
        x[u].z = (int)((unsigned)x[u].w + (unsigned)y[u].z);
        changed = true;
      }
      x[u].x = y[u].x;
      x[u].w = (int)((unsigned)x[u].w + (unsigned)y[u].w);
      __stcg(&out[k], x[u]);
    }
  }
  return changed;
}

// Doubling until a round changes no minimum (every orbit is covered then:
// its least crossing reaches a new one in every round until it has reached
// all); at most 32 rounds, as a window doubles in each.  Results in A.
__global__ void __launch_bounds__(1024) k_gp_jump_block(int K, int4* A, int4* B) {
  int4* in = A;
  int4* out = B;
  for (int r = 0; r < 32; ++r) {
    const bool ch = gp_round(K, in, out, threadIdx.x, 1024);
    int4* t = in;
    in = out;
    out = t;
    if (!__syncthreads_or(ch)) break;
  }
  if (in != A)
    for (int k = threadIdx.x; k < K; k += 1024) A[k] = in[k];
}

// flags: three words, zero; a round's word is cleared two rounds later
__global__ void __launch_bounds__(256) k_gp_jump_coop(int K, int4* A, int4* B, unsigned* flags) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  int4* in = A;
  int4* out = B;
  for (int r = 0; r < 32; ++r) {
    if (tid == 0) flags[(r + 1) % 3] = 0u;
    const bool ch = gp_round(K, in, out, tid, nth);
    if (__any_sync(0xffffffffu, ch) && (threadIdx.x & 31) == 0) atomicOr(&flags[r % 3], 1u);
    grid.sync();
    int4* t = in;
    in = out;
    out = t;
    if (*(volatile unsigned*)&flags[r % 3] == 0u) break;
  }
  if (in != A)
    for (int k = tid; k < K; k += nth) A[k] = __ldcg(&in[k]);
}

// a ring and its vertices at its first crossing, zero elsewhere (K + 1 entries)
__global__ void __launch_bounds__(256) k_gp_starts(Gp g, int* __restrict__ ring, int* __restrict__ len) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > g.K) return;
  int n = 0;
  if (k < g.K && g.A[k].y == k) {
    const int inP = g.wind[0] & 1, inQ = g.wind[1] & 1;
    const GpLeg p = gp_leg(g, 0, inP, k);
    if (k < g.A[p.to].y) {
      const GpLeg q = gp_leg(g, 1, inQ, g.rQ[g.hP[p.to]]);
      n = p.cnt + q.cnt + 2 + g.A[g.rP[g.hQ[q.to]]].z;
    }
  }
  ring[k] = n > 0 ? 1 : 0;
  len[k] = n;
}

// long runs of vertices, copied by a warp each: {side | 2 * forwards, edge,
// vertices, place}
constexpr int kGpInline = 16, kGpPiece = 1024;

__device__ __forceinline__ double2 gp_vertex(const Gp& g, int side, bool fwd, int e, int t) {
  const int n = side ? g.nc : g.nb;
  int u = fwd ? e + 1 + t : e - t;
  if (u >= n) u -= n;
  if (u < 0) u += n;
  return ((const double2*)(side ? g.c : g.b))[u];
}

// every leg of a ring's sense to its place; ring offsets; the counts
__global__ void __launch_bounds__(256) k_gp_emit(Gp g, const int* __restrict__ ring,
                                                 const int* __restrict__ at0, int* __restrict__ off,
                                                 double2* __restrict__ out, int4* __restrict__ pieces,
                                                 unsigned* __restrict__ npieces, unsigned cap) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) off[ring[g.K]] = at0[g.K];
  if (k >= g.K) return;
  const int inP = g.wind[0] & 1, inQ = g.wind[1] & 1;
  const GpLeg p = gp_leg(g, 0, inP, k);
  const int4 a = g.A[k];
  const int s = a.y;
  if (s > g.A[p.to].y) return;  // the other sense
  const GpLeg q = gp_leg(g, 1, inQ, g.rQ[g.hP[p.to]]);
  int at = s == k ? at0[s] : at0[s + 1] - a.z;
  if (s == k) off[ring[s]] = at;
  for (int side = 0; side < 2; ++side) {
    const GpLeg l = side ? q : p;
    bool listed = false;
    if (l.cnt > kGpInline) {
      const unsigned need = (l.cnt + kGpPiece - 1) / kGpPiece;
      const unsigned i = atomicAdd(npieces, need);
      if (i + need <= cap) {
        for (unsigned j = 0; j < need; ++j)
          pieces[i + j] = make_int4(side | (l.fwd ? 2 : 0), l.fwd ? l.e + (int)j * kGpPiece : l.e - (int)j * kGpPiece,
                                    min(kGpPiece, l.cnt - (int)j * kGpPiece), at + (int)j * kGpPiece);
        listed = true;
      } else {
        // no room: the reserved entries stay empty
        for (unsigned j = i; j < i + need && j < cap; ++j) pieces[j] = make_int4(0, 0, 0, 0);
      }
    }
    if (!listed)
      for (int t = 0; t < l.cnt; ++t) out[at + t] = gp_vertex(g, side, l.fwd, l.e, t);
    out[at + l.cnt] = g.xy[side ? g.hQ[l.to] : g.hP[l.to]];
    at += l.cnt + 1;
  }
}

__global__ void __launch_bounds__(256) k_gp_pieces(Gp g, const int4* __restrict__ pieces,
                                                   const unsigned* __restrict__ npieces, unsigned cap,
                                                   double2* __restrict__ out) {
  const unsigned n = min(*npieces, cap), nw = gridDim.x * 8;
  for (unsigned i = blockIdx.x * 8 + (threadIdx.x >> 5); i < n; i += nw) {
    const int4 s = pieces[i];
    // an edge number past the ends wraps once (gp_vertex)
    const int n1 = (s.x & 1) ? g.nc : g.nb;
    int e = s.y;
    if (e >= n1) e -= n1;
    if (e < 0) e += n1;
    for (int t = threadIdx.x & 31; t < s.z; t += 32)
      out[s.w + t] = gp_vertex(g, s.x & 1, (s.x & 2) != 0, e, t);
  }
}

// no crossings: each polygon inside the other (outside it, for the union) is
// a ring, the base first (cnt: rings, vertices)
__global__ void __launch_bounds__(256) k_gp_whole(Gp g, int* __restrict__ cnt, int* __restrict__ off,
                                                  double2* __restrict__ out) {
  const bool keep[2] = {((g.wind[0] & 1) ^ g.unite) != 0, ((g.wind[1] & 1) ^ g.unite) != 0};
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int n0 = keep[0] ? g.nb : 0, n1 = keep[1] ? g.nc : 0;
  if (x == 0) {
    int r = 0;
    off[0] = 0;
    if (keep[0]) off[++r] = n0;
    if (keep[1]) off[++r] = n0 + n1;
    cnt[0] = r;
    cnt[1] = n0 + n1;
  }
  if (x < n0 + n1) {
    const bool base = x < n0;
    const int u = base ? x : x - n0, n = base ? g.nb : g.nc;
    const double2* p = (const double2*)(base ? g.b : g.c);
    out[x] = p[u];
    if (gp_flat(p[u == 0 ? n - 1 : u - 1], p[u], p[u + 1])) atomicOr(g.bad, 2u);
  }
}

// cooperative doubling on as many blocks as can be resident; false where the
// launch is refused
bool gp_jump(int K, int4* A, int4* B, unsigned* flags, cudaStream_t st) {
  if (K <= 4096) {  // one block: a barrier a round instead of a grid's
    ::sbc::KProbe kp_("k_gp_jump_block", st);
    k_gp_jump_block<<<1, 1024, 0, st>>>(K, A, B);
    return true;
  }
  static std::mutex mu;
  static int cap[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  int most = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!cap[dev]) {
      int per = 0, sms = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_gp_jump_coop, 256, 0) != cudaSuccess ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || per < 1)
        return false;
      cap[dev] = per * sms;
    }
    most = cap[dev];
  }
  const int blocks = std::min((K + 255) / 256, most);
  void* args[] = {&K, &A, &B, &flags};
  ::sbc::KProbe kp_("k_gp_jump_coop", st);
  if (cudaLaunchCooperativeKernel((const void*)k_gp_jump_coop, dim3(blocks), dim3(256), args, 0, st) ==
      cudaSuccess)
    return true;
  cudaGetLastError();  // this refused launch's own error
  return false;
}

}  // namespace

int Pipeline::stage_general(int cType, const int* rb, const int* rc, const int* rt,
                            const unsigned long long* rkey, long long nhits, OverlayOut& out,
                            bool* done) {
  *done = false;
  const int cStart = hcS[cType - 1], nc = hcS[cType] - hcS[cType - 1] - 1;
  // crossings come in pairs along a closed curve
  if (force_serial_backend || !raw_ab_ || (nhits & 1) || !overlay_ids_fit()) return kOk;
  if (nhits + nb + (long long)nc >= (1LL << 30)) return kOk;
  const int K = (int)nhits;
  cudaStream_t st = st_;
  const std::string tg = std::to_string((int)(&out - &outs_[0]));
  Gp g;
  g.K = K;
  g.nb = nb;
  g.nc = nc;
  g.cStart = cStart;
  g.unite = unite ? 1 : 0;
  g.rb = rb;
  g.rc = rc;
  g.rt = rt;
  g.rkey = rkey;
  g.rab = raw_ab_;
  g.b = bP;
  g.c = cP + 2 * (long long)cStart;
  // cleared together: the edge ends and 16 words (bad, long edges, pieces,
  // winding numbers, rounds, counts)
  const size_t cleared = sizeof(int) * ((size_t)nb + nc + 4 + 16);
  int* zero = (int*)pool_.get("gp_zero", cleared);
  int* ranks = (int*)pool_.get("gp_ranks", sizeof(int) * 8 * ((size_t)K + 1));
  g.xy = (double2*)pool_.get("gp_xy", sizeof(double2) * ((size_t)K + 1));
  g.A = (int4*)pool_.get("gp_A", sizeof(int4) * ((size_t)K + 4));
  g.B = (int4*)pool_.get("gp_B", sizeof(int4) * ((size_t)K + 4));
  const unsigned cap = (unsigned)((nb + (long long)nc) / kGpInline + 2);
  int4* pieces = (int4*)pool_.get("gp_pieces", sizeof(int4) * cap);
  int* ring = (int*)pool_.get("gp_ring", sizeof(int) * 2 * ((size_t)K + 2));
  void* sscr = pool_.get_zeroed(
      "gp_scan", scan_set_scratch_bytes(std::max((long long)std::max(nb, nc), (long long)K) + 2, 2), st);
  int* ooff = (int*)pool_.get("ring_off_" + tg, sizeof(int) * ((size_t)K / 2 + 4));
  auto* oxy = (double2*)pool_.get("ring_xy_" + tg, sizeof(double2) * ((size_t)K + nb + nc + 1));
  if (pool_.failed) return fail(kENoMem, "device allocation failed (general position)");
  int* words = zero;
  g.bad = (unsigned*)words;
  g.nlong = (unsigned*)words + 1;
  unsigned* npieces = (unsigned*)words + 2;
  g.wind = words + 3;
  unsigned* flags = (unsigned*)words + 5;
  int* cnt = words + 8;
  g.endB = words + 16;
  g.endC = g.endB + nb + 2;
  int* at = ranks;
  for (int** p : {&g.hP, &g.hQ, &g.rP, &g.rQ, &g.eP, &g.eQ, &g.aB, &g.aC}) {
    *p = at;
    at += K + 1;
  }
  g.longs = g.rP;  // until the ranks are known: at most 2 K / 129 long edges
  cudaMemsetAsync(zero, 0, cleared, st);
  const unsigned kg = grid_for(K > 0 ? K : 1, 256);
  if (K > 0) {
    {
      ::sbc::KProbe kp_("k_gp_hits", st, 108.0 * K);
      k_gp_hits<<<kg, 256, 0, st>>>(g);
    }
    {
      int* const arrs[2] = {g.endB, g.endC};
      const long long ns[2] = {nb + 1LL, nc + 1LL};
      exclusive_scan_i32_set(arrs, ns, 2, sscr, st, true);
    }
    {
      ::sbc::KProbe kp_("k_gp_scatter", st, 16.0 * K);
      k_gp_scatter<<<kg, 256, 0, st>>>(g);
    }
    {
      ::sbc::KProbe kp_("k_gp_order", st, 4.0 * (nb + nc) + 16.0 * K);
      const int per = K > 2LL * (nb + nc) ? 4 : 32;
      k_gp_order<<<grid_for((nb + (long long)nc) * (32 / per), 256), 256, 0, st>>>(g, per);
    }
    {
      ::sbc::KProbe kp_("k_gp_order_long", st);
      k_gp_order_long<<<std::min(304u, (unsigned)(2 * (K / kGpWarp) + 1)), 256, 0, st>>>(g);
    }
    {
      ::sbc::KProbe kp_("k_gp_rank", st, 40.0 * K);
      k_gp_rank<<<kg, 256, 0, st>>>(g);
    }
  }
  {
    ::sbc::KProbe kp_("k_gp_pip", st, 20.0 * (nb + nc) + 40.0 * K);
    k_gp_pip<<<dim3(std::min(grid_for(std::max(nb, nc), 256), 1216u), 2), 256, 0, st>>>(g);
  }
  const int* r_cnt = nullptr;
  if (K == 0) {
    ::sbc::KProbe kp_("k_gp_whole", st, 32.0 * (nb + nc));
    k_gp_whole<<<grid_for(nb + (long long)nc, 256), 256, 0, st>>>(g, cnt, ooff, oxy);
    r_cnt = rd_.get(cnt, HostReads::kBack + 8, st, 2);
  } else {
    {
      ::sbc::KProbe kp_("k_gp_legs", st, 24.0 * (nb + nc) + 180.0 * K);
      k_gp_legs<<<grid_for((long long)K + nb + nc, 256), 256, 0, st>>>(g);
    }
    if (!gp_jump(K, g.A, g.B, flags, st)) return kOk;
    int* len = ring + K + 2;
    {
      ::sbc::KProbe kp_("k_gp_starts", st, 24.0 * K);
      k_gp_starts<<<grid_for(K + 1LL, 256), 256, 0, st>>>(g, ring, len);
    }
    {
      int* const arrs[2] = {ring, len};
      const long long ns[2] = {K + 1LL, K + 1LL};
      exclusive_scan_i32_set(arrs, ns, 2, sscr, st, true);
    }
    {
      ::sbc::KProbe kp_("k_gp_emit", st, 100.0 * K);
      k_gp_emit<<<kg, 256, 0, st>>>(g, ring, len, ooff, oxy, pieces, npieces, cap);
    }
    {
      ::sbc::KProbe kp_("k_gp_pieces", st);
      k_gp_pieces<<<std::min(grid_for(cap, 8), 608u), 256, 0, st>>>(g, pieces, npieces, cap, oxy);
    }
    int* two = (int*)rd_.get(ring + K, HostReads::kBack + 8, st);
    cudaMemcpyAsync(two + 1, len + K, sizeof(int), cudaMemcpyDeviceToHost, st);
    r_cnt = two;
  }
  const unsigned* r_bad = rd_.get(g.bad, HostReads::kBack, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return fail(kECuda, "general position");
  if (*r_bad & 1u) return kOk;
  out.unique = K;
  out.slots_b = nb + (long long)K;
  out.slots_c = nc + (long long)K;
  out.slow_path = 0;
  out.d_off = ooff;
  out.d_xy = (double*)oxy;
  out.nrings = r_cnt[0];
  out.nverts = r_cnt[1];
  out.counts = nullptr;
  // the records, in no particular order (the arrays built from them: on
  // demand, build_records)
  dbg_ub = const_cast<int*>(rb);
  dbg_uc = const_cast<int*>(rc);
  dbg_ut = const_cast<int*>(rt);
  dbg_K = K;
  dbg_isxy = (double*)g.xy;
  lazy_ = {cType, rb, rc, rt, rkey, nhits};
  *done = true;
  if (*r_bad == 0u || out.nverts == 0) return kOk;
  // some ring may lose vertices: from a copy into the same buffers
  int* roff = (int*)pool_.get("gp_roff", sizeof(int) * ((size_t)out.nrings + 1));
  auto* rxy = (double2*)pool_.get("gp_rxy", sizeof(double2) * (size_t)out.nverts);
  if (pool_.failed) return fail(kENoMem, "device allocation failed (general position)");
  cudaMemcpyAsync(roff, ooff, sizeof(int) * ((size_t)out.nrings + 1), cudaMemcpyDeviceToDevice, st);
  cudaMemcpyAsync(rxy, oxy, sizeof(double2) * (size_t)out.nverts, cudaMemcpyDeviceToDevice, st);
  out.d_off = roff;
  out.d_xy = (double*)rxy;
  return clean_up_rings(*this, out);
}

}  // namespace sbc
