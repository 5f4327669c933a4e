// sbc_group.cuh -- the threads that work on one pair together: a warp, or a
// whole block for a pair too large for one warp.  The steps of the pair
// engines (sbc_pwpair.cuh, sbc_batch.cu, sbc_pairwise.cu) are written once
// against this interface.  Every collective below is called by all threads of
// the group; a group-wide result is the same on every thread, and memory
// written before a collective that synchronises (all but first() on a warp)
// is visible to the group after it.
#pragma once

#include <climits>

#include "sbc_internal.cuh"

namespace sbc {
namespace {

struct WarpGroup {
  // where the warps of a kernel may wait for one another (PhasedWarp)
  __device__ __forceinline__ void phase() const {}
  template <int n>
  __device__ __forceinline__ void leave() const {}
  static constexpr int N = 32;
  static constexpr int kWarps = 1;
  static constexpr bool kBlock = false;
  __device__ __forceinline__ int rank() const { return threadIdx.x & 31; }
  __device__ __forceinline__ int warp() const { return 0; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ bool any(bool b) const {
    __syncwarp();
    return __any_sync(0xffffffffu, b);
  }
  __device__ __forceinline__ int sum(int x) const { return __reduce_add_sync(0xffffffffu, x); }
  __device__ __forceinline__ int min_of(int x) const { return __reduce_min_sync(0xffffffffu, x); }
  // threads of lower rank with f set; *total: all of them
  __device__ __forceinline__ int before(bool f, int* total) const {
    const unsigned m = __ballot_sync(0xffffffffu, f);
    *total = __popc(m);
    return __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
  }
  // exclusive sum of x over the ranks; *total: the sum over all
  __device__ __forceinline__ int excl(int x, int* total) const {
    const int lane = threadIdx.x & 31;
    int s = x;
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= d) s += t;
    }
    *total = __shfl_sync(0xffffffffu, s, 31);
    return s - x;
  }
  // first i in [0, n) with pred(i), or -1
  template <class Pred>
  __device__ int first(int n, Pred pred) const {
    const int lane = threadIdx.x & 31;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      const unsigned m = __ballot_sync(0xffffffffu, i < n && pred(i));
      if (m) return i0 + __ffs(m) - 1;
    }
    return -1;
  }
  // a value every thread has computed by itself from the same data
  __device__ __forceinline__ int same(int x) const { return x; }
};

// A warp whose block's other warps do the same steps on other data: they enter
// each of kPhases steps together, so that its instructions are fetched once
// (nothing else depends on it).  Each warp of the block of T threads, with a
// pair or without, passes exactly kPhases times through one named barrier,
// wherever in the code (which PTX allows; __syncthreads would have to be the
// same call for all): a warp that is done after step k leaves the kernel by
// leave<kPhases - k>(), which passes what is left.  It holds nothing meanwhile
// that its block would not.  (k_batch_clean, 65,536 pairs of 4 to 64 vertices:
// 0.86 ms, 1.02 without the steps; 0.94 where the warps that are done go on to
// the kernel's end, 1.95 with an mbarrier from which they drop.)
template <int T>
struct PhasedWarp : WarpGroup {
  static constexpr int kPhases = 5;  // clean_clip's
  __device__ __forceinline__ void phase() const {
    asm volatile("barrier.cta.sync.aligned 1, %0;" ::"n"(T) : "memory");
  }
  template <int n>
  __device__ __forceinline__ void leave() const {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < n; ++i) phase();
    asm volatile("exit;");
    __builtin_unreachable();
  }
};

// A block of T threads (a multiple of 32, at most 1,024).  The collectives
// alternate between two halves of the scratch words, so one barrier each is
// enough: a half is written again only after the next collective's barrier,
// which every reader of it has passed.
template <int T>
struct BlockGroup {
  __device__ __forceinline__ void phase() const {}
  template <int n>
  __device__ __forceinline__ void leave() const {}
  static constexpr int N = T;
  static constexpr int kWarps = T / 32;
  static constexpr bool kBlock = true;
  struct Shared {
    int w[2][kWarps];
    int count;  // entries of a work list
  };
  Shared* s;
  int half = 0;
  __device__ explicit BlockGroup(Shared* sh) : s(sh) {}
  __device__ __forceinline__ int rank() const { return threadIdx.x; }
  __device__ __forceinline__ int warp() const { return threadIdx.x >> 5; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ __forceinline__ bool any(bool b) const { return __syncthreads_or(b); }
  __device__ int sum(int x) {
    x = __reduce_add_sync(0xffffffffu, x);
    int* w = flip();
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = x;
    __syncthreads();
    int t = 0;
    for (int i = 0; i < kWarps; ++i) t += w[i];
    return t;
  }
  __device__ int min_of(int x) {
    x = __reduce_min_sync(0xffffffffu, x);
    int* w = flip();
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = x;
    __syncthreads();
    int t = INT_MAX;
    for (int i = 0; i < kWarps; ++i) t = min(t, w[i]);
    return t;
  }
  __device__ int before(bool f, int* total) {
    const unsigned m = __ballot_sync(0xffffffffu, f);
    int* w = flip();
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = __popc(m);
    __syncthreads();
    return prefix(w, total) + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
  }
  __device__ int excl(int x, int* total) {
    const int lane = threadIdx.x & 31;
    int v = x;
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, d);
      if (lane >= d) v += t;
    }
    int* w = flip();
    if (lane == 31) w[threadIdx.x >> 5] = v;
    __syncthreads();
    return prefix(w, total) + v - x;
  }
  template <class Pred>
  __device__ int first(int n, Pred pred) {
    int at = INT_MAX;
    for (int i = threadIdx.x; i < n; i += T)
      if (pred(i)) {
        at = i;
        break;
      }
    __syncwarp();
    at = min_of(at);
    return at == INT_MAX ? -1 : at;
  }
  // thread 0's value
  __device__ int same(int x) {
    int* w = flip();
    if (threadIdx.x == 0) w[0] = x;
    __syncthreads();
    return w[0];
  }

 private:
  __device__ __forceinline__ int* flip() {
    half ^= 1;
    return s->w[half];
  }
  __device__ __forceinline__ int prefix(const int* w, int* total) const {
    const int me = threadIdx.x >> 5;
    int b = 0, t = 0;
    for (int i = 0; i < kWarps; ++i) {
      if (i < me) b += w[i];
      t += w[i];
    }
    *total = t;
    return b;
  }
};

// exclusive prefix sums of a[0..n) in place by the group; returns the total.
// Element i is read and written by the thread of rank i % N.
template <class G>
__device__ int group_scan(G& g, int* a, int n) {
  int carry = 0;
  for (int i0 = 0; i0 < n; i0 += G::N) {
    const int i = i0 + g.rank();
    int tot;
    const int e = g.excl(i < n ? a[i] : 0, &tot);
    if (i < n) a[i] = carry + e;
    carry += tot;
  }
  return carry;
}

// one round trip of a bitonic network over np (a power of two) slots: each
// thread takes compare-exchange pairs (m, m + j), so none idles in a round.
// swap_if(m, l, up): orders slots m < l ascending when up, else descending.
template <class G, class SwapIf>
__device__ void group_bitonic(G& g, int np, SwapIf swap_if) {
  for (int k = 2; k <= np; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int q = g.rank(); q < (np >> 1); q += G::N) {
        const int m = ((q & ~(j - 1)) << 1) | (q & (j - 1));
        swap_if(m, m | j, (m & k) == 0);
      }
      g.sync();
    }
}

}  // namespace
}  // namespace sbc
