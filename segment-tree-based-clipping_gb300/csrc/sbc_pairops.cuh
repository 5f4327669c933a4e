// sbc_pairops.cuh -- per-pair device helpers shared by the batched pair engine
// (sbc_batch.cu), the one-base-many-overlays engine (sbc_pairwise.cu) and the
// pair pipeline's general-position stage (sbc_general.cu).
#pragma once

#include "sbc_internal.cuh"

namespace sbc {
namespace {

// Arrays of one pair, carved in a fixed order from a base pointer (a null
// base gives the byte count).
struct Carver {
  unsigned char* base;
  size_t off;
  template <class T>
  __host__ __device__ T* take(long long n) {
    off = (off + 15) & ~(size_t)15;
    T* r = (T*)(base + off);
    off += sizeof(T) * (size_t)(n > 0 ? n : 0);
    return r;
  }
};

__host__ __device__ __forceinline__ int npow2_dev(int n) {
  int p = 1;
  while (p < n) p <<= 1;
  return p;
}

// ------------------------------------------------------------------ small helpers
__device__ __forceinline__ double bvx(const double* p, int n, int i) { return p[2 * (i % n)]; }
__device__ __forceinline__ double bvy(const double* p, int n, int i) { return p[2 * (i % n) + 1]; }

__device__ __forceinline__ bool lsmf_d(double p1x, double p1y, double p2x, double p2y, double q1x,
                                       double q1y, double q2x, double q2y) {
  // on order keys: integer compares instead of FP64 ones, same decisions
  return lsmf_keys(okey(p1x), okey(p1y), okey(p2x), okey(p2y), okey(q1x), okey(q1y), okey(q2x),
                   okey(q2y));
}

// stable bottom-up merge sort of idx[0..n) by less(a, b)
template <class Less>
__device__ void merge_sort(int* idx, int* tmp, int n, Less less) {
  for (int w = 1; w < n; w <<= 1) {
    for (int lo = 0; lo < n; lo += 2 * w) {
      const int mid = min(lo + w, n), hi = min(lo + 2 * w, n);
      int i = lo, j = mid, o = lo;
      while (i < mid && j < hi) tmp[o++] = less(idx[j], idx[i]) ? idx[j++] : idx[i++];
      while (i < mid) tmp[o++] = idx[i++];
      while (j < hi) tmp[o++] = idx[j++];
    }
    for (int i = 0; i < n; ++i) idx[i] = tmp[i];
  }
}

__device__ __forceinline__ bool canonical_s(int v, int logL, int l, int r1) {
  const int L = 1 << logL;
  const int d = 31 - __clz(v), h = logL - d;
  const int lo = (v << h) - L, hi = ((v + 1) << h) - L;
  if (lo < l || hi > r1) return false;
  if (v == 1) return true;
  const int p = v >> 1;
  const int plo = (p << (h + 1)) - L, phi = ((p + 1) << (h + 1)) - L;
  return !(plo >= l && phi <= r1);
}

__device__ __forceinline__ bool below_s(int x, int v, int logL) {
  if (x < 0) return false;
  const int h = logL - (31 - __clz(v));
  return (x >> h) == v;
}

// Emission count and first-emission key of base edge b with overlay edge c
// (the candidate loops of saveIntersectionsIdsMulticore,
// oacc_segment_tree.cpp:6010-6244, as a rule over the two edges): rb, rc are
// the edges' covered leaf ranges [l, r1), eb0/eb1 and ec0/ec1 their end-list
// leaves (aft, bef; -1 when dropped); c is the overlay edge's index in the
// pair's edge numbering and cId its id.  Kind 0 (v in both cover lists) and
// kind 1 (v covers b, c ends below v) carry cId; kind 2 (v covers c, b ends
// below v) carries c.
__device__ unsigned emission_q(int2 rb, int2 rc, int eb0, int eb1, int ec0, int ec1, int c,
                               int cId, int logL, unsigned long long* key) {
  const int L = 1 << logL;
  unsigned n = 0;
  unsigned long long best = ~0ull;
  for (int a = rb.x + L, z = rb.y + L; a < z; a >>= 1, z >>= 1) {
    for (int side = 0; side < 2; ++side) {
      int v = -1;
      if (side == 0 && (a & 1)) v = a++;
      if (side == 1 && (z & 1)) v = --z;
      if (v < 0) continue;
      if (canonical_s(v, logL, rc.x, rc.y)) {
        n += 2;
        best = min(best, ((unsigned long long)v << 33) | (unsigned)cId);
      }
      if (below_s(ec0, v, logL) || below_s(ec1, v, logL)) {
        n += 1;
        best = min(best, ((unsigned long long)v << 33) | (1ull << 31) | (unsigned)cId);
      }
    }
  }
  for (int a = rc.x + L, z = rc.y + L; a < z; a >>= 1, z >>= 1) {
    for (int side = 0; side < 2; ++side) {
      int v = -1;
      if (side == 0 && (a & 1)) v = a++;
      if (side == 1 && (z & 1)) v = --z;
      if (v < 0) continue;
      if (below_s(eb0, v, logL) || below_s(eb1, v, logL)) {
        n += 1;
        best = min(best, ((unsigned long long)v << 33) | (1ull << 32) | (unsigned)c);
      }
    }
  }
  *key = best;
  return n;
}

__device__ __forceinline__ bool nd_b(int t) { return t == 1 || t == 3 || t == 5 || t == 7; }
__device__ __forceinline__ bool nd_c(int t) { return t == 1 || t == 2 || t == 6; }

// status codes of one pair
enum { PS_OK = 0, PS_UNDEF = 2, PS_CAP = 3 };


// The gradient (gx, gy) of a crossing's coordinates chained to the ends of its
// edges b1b2 and c1c2: I = (1 - alpha) b1 + alpha b2, alpha = A1 / (A1 - A2),
// A1 = A(b1, c1, c2), A2 = A(b2, c1, c2); A(P, Q, R) partials: dP = (Qy - Ry,
// Rx - Qx), dQ = (Ry - Py, Px - Rx), dR = (Py - Qy, Qx - Px)
// One reciprocal and explicit fused multiply-adds: the FP64 rate bounds the
// backward pass, and three divisions without fma took about twice as many
// operations.
struct CrossGrad {
  double gx, gy, al, k1, k2;
  double2 b1c1, b1c2, b2c1, b2c2, c12;  // c1 - b1, c2 - b1, c1 - b2, c2 - b2, c1 - c2
  __device__ __forceinline__ CrossGrad(const double* b, int i1, int i2, const double* c, int j1,
                                       int j2, double gx_, double gy_)
      : gx(gx_), gy(gy_) {
    const double b1x = b[2 * i1], b1y = b[2 * i1 + 1], b2x = b[2 * i2], b2y = b[2 * i2 + 1];
    const double c1x = c[2 * j1], c1y = c[2 * j1 + 1], c2x = c[2 * j2], c2y = c[2 * j2 + 1];
    b1c1 = make_double2(c1x - b1x, c1y - b1y);
    b1c2 = make_double2(c2x - b1x, c2y - b1y);
    b2c1 = make_double2(c1x - b2x, c1y - b2y);
    b2c2 = make_double2(c2x - b2x, c2y - b2y);
    c12 = make_double2(c1x - c2x, c1y - c2y);
    const double A1 = fma(b1c1.x, b1c2.y, -(b1c1.y * b1c2.x));
    const double A2 = fma(b2c1.x, b2c2.y, -(b2c1.y * b2c2.x));
    const double d = A1 - A2, r = 1.0 / d, q = A1 * r;
    al = fma(fma(-q, d, A1), r, q);  // A1 / d, corrected once
    const double ga = fma(gx, b2x - b1x, gy * (b2y - b1y)) * r * r;  // dA/dalpha / d^2
    k1 = -A2 * ga;  // dalpha/dA1
    k2 = A1 * ga;   // dalpha/dA2
  }
  __device__ __forceinline__ double2 b1() const {
    const double u = 1.0 - al;
    return make_double2(fma(k1, c12.y, u * gx), fma(-k1, c12.x, u * gy));
  }
  __device__ __forceinline__ double2 b2() const {
    return make_double2(fma(k2, c12.y, al * gx), fma(-k2, c12.x, al * gy));
  }
  __device__ __forceinline__ double2 c1() const {
    return make_double2(fma(k1, b1c2.y, k2 * b2c2.y), -fma(k1, b1c2.x, k2 * b2c2.x));
  }
  __device__ __forceinline__ double2 c2() const {
    return make_double2(-fma(k1, b1c1.y, k2 * b2c1.y), fma(k1, b1c1.x, k2 * b2c1.x));
  }
};

}  // namespace
}  // namespace sbc
