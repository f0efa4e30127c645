// sort.cuh -- segmented stable LSD radix sort of (uint64 key, int payload).
#pragma once
#include "common.cuh"

namespace prsb {

typedef unsigned long long u64;
typedef unsigned int u32;

// 62-bit fixed point of the double behind an ordered key, the unit 2^(em - 1084)
// (truncated towards zero: non-decreasing in the value)
__device__ __forceinline__ int key_exp(u64 k) {
  const u64 b = (k >> 63) ? (k ^ 0x8000000000000000ull) : ~k;
  return (int)((b >> 52) & 0x7FF);
}
__device__ __forceinline__ ll key_fixed(u64 k, int em) {
  const bool neg = (k >> 63) == 0;
  const u64 b = neg ? ~k : k ^ 0x8000000000000000ull;
  const int e = (int)((b >> 52) & 0x7FF);
  u64 m = b & 0xFFFFFFFFFFFFFull;
  if (e) m |= 1ull << 52;
  const int sh = em - (e ? e : 1);  // >= 0
  m = sh < 63 ? (m << 9) >> sh : 0ull;
  return neg ? -(ll)m : (ll)m;
}

// Exclusive scan of a[0..m) in place and its largest entry, by the CTA of
// THREADS threads (a: room for W counts, 16-byte aligned).
template <int W, int THREADS>
__device__ __forceinline__ u32 cta_scan(u32 *a, int m) {
  constexpr int PER = W / THREADS, NW = THREADS / 32;
  static_assert(PER % 4 == 0 && NW <= 32, "whole vectors per thread");
  __shared__ u32 ws[32], wm[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k0 = threadIdx.x * PER;
  uint4 *a4 = reinterpret_cast<uint4 *>(a + k0);
  u32 v[PER], sum = 0, big = 0;
#pragma unroll
  for (int r = 0; r < PER; r += 4) {
    const uint4 c = k0 + r < m ? a4[r / 4] : make_uint4(0, 0, 0, 0);
    v[r] = c.x, v[r + 1] = c.y, v[r + 2] = c.z, v[r + 3] = c.w;
  }
#pragma unroll
  for (int r = 0; r < PER; r++) {
    if (k0 + r >= m) v[r] = 0u;
    sum += v[r], big = max(big, v[r]);
  }
  u32 x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  big = __reduce_max_sync(0xffffffffu, big);
  if (lane == 31) ws[warp] = x, wm[warp] = big;
  __syncthreads();
  u32 run = __reduce_add_sync(0xffffffffu, lane < warp ? ws[lane] : 0u) + x - sum;
  big = __reduce_max_sync(0xffffffffu, lane < NW ? wm[lane] : 0u);
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const u32 c = v[r];
    v[r] = run;
    run += c;
  }
#pragma unroll
  for (int r = 0; r < PER; r += 4)
    if (k0 + r < m) a4[r / 4] = make_uint4(v[r], v[r + 1], v[r + 2], v[r + 3]);
  __syncthreads();
  return big;
}

// Workspace reused across calls (grown on demand).
struct SortWs {
  DBuf<u64> ktmp;
  DBuf<int> vtmp;
  DBuf<u32> counts;     // [256][ntiles]
  DBuf<u32> totals;     // [256]
  DBuf<u32> hist_all;   // [npass][256]
  // sort_by_value
  DBuf<u32> q;          // 32-bit keys (their other buffer: ktmp)
  DBuf<u32> mark;       // a bit per item
  DBuf<int> pos;        // positions, where the full keys are sorted
  DBuf<u64> range;      // smallest and largest key, runs that cannot be listed, runs listed,
                        // the longest of these
  DBuf<int2> runs;      // long runs out of order: start, length
  // gives the buffers of more than `keep` items back to the pool
  void trim(ll keep) {
    auto drop = [keep](auto &b) {
      if ((ll)b.n > keep) b.release();
    };
    drop(ktmp), drop(vtmp), drop(q), drop(pos);
  }
};

// Sort pairs (keys[i], vals[i]), i < n, stably by (seg_of_val[vals[i]], key).
// seg_of_val may be null (one segment); nseg is the number of segments
// (segment ids must lie in [0, nseg)).  On return *keys / *vals point at the
// sorted arrays, which are either the inputs or the workspace buffers (the
// pointers are swapped with ws buffers as needed; the caller's DBufs are
// swapped correspondingly).
void seg_sort_pairs(DBuf<u64> &keys, DBuf<int> &vals, ll n,
                    const int *seg_of_val, ll nseg, SortWs &ws);

// Sort (keys[i], vals[i]), i < n, stably by key inside each segment, for keys
// that order doubles (ordered_key).  seg_of_pos[i] (may be null: one segment)
// is the segment of position i, non-decreasing in [0, nseg); no segment is
// longer than max_len; iota: vals[i] is i.  Same result as seg_sort_pairs with the segment of
// every value; keys / vals point at the sorted arrays on return.
void sort_by_value(DBuf<u64> &keys, DBuf<int> &vals, ll n, const int *seg_of_pos, ll nseg,
                   ll max_len, SortWs &ws, bool iota = false);

}  // namespace prsb
