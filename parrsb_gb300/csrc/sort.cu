// sort.cu -- segmented stable LSD radix sort for sm_103a.
//
// Replaces the reference's distributed stable sorts (parallel_sort_,
// src/sort.c:182-213, bin sort src/sort-bin.c:36-50, local gslib sorts
// src/sort.c:72-104).  A segmented sort by (segment, key) is an LSD sort on
// the key bytes followed by the segment-id bytes; every pass is stable, so
// ties keep their current order (the canonical tie-break).
//
// Per pass: a tile histogram kernel (4096 items per 512-thread CTA), a
// per-digit exclusive scan over tiles, and a scatter kernel that loads its
// 8 items per thread up front, ranks them stably inside the CTA (warp w owns
// items [w*256, w*256+256) of the tile, processed 32 at a time in order; the
// lanes with the same digit by a ballot per bit), stages the tile in shared
// memory in digit order and writes each digit's run with consecutive addresses.  One
// up-front kernel builds the global digit histograms of every pass; passes
// whose digit is constant over all items are skipped.
#include <algorithm>

#include "sort.cuh"

namespace prsb {

namespace {

constexpr int SORT_THREADS = 512;
constexpr int ITEMS_PER_THREAD = 8;
constexpr int NWARP = SORT_THREADS / 32;
constexpr int TILE = SORT_THREADS * ITEMS_PER_THREAD;  // 4096
constexpr int MAX_PASSES = 12;                           // 8 key + 4 seg bytes
constexpr size_t SCATTER_SMEM = (size_t)TILE * (8 + 4 + 1);  // staged keys, values, digits

struct PassDesc {
  int is_seg;
  int shift;
};

__device__ __forceinline__ u32 digit_of(u64 key, int val, const int *seg_of_val,
                                         int is_seg, int shift) {
  if (is_seg) return ((u32)seg_of_val[val] >> shift) & 255u;
  return (u32)(key >> shift) & 255u;
}

__global__ void k_hist_all(const u64 *__restrict__ keys, const int *__restrict__ vals,
                           ll n, const int *__restrict__ seg_of_val, int nkey,
                           int nseg_pass, u32 *__restrict__ hist_all) {
  __shared__ u32 h[MAX_PASSES][256];
  int np = nkey + nseg_pass;
  for (int i = threadIdx.x; i < np * 256; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  ll stride = (ll)gridDim.x * blockDim.x;
  for (ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    u64 k = keys[i];
    for (int b = 0; b < nkey; b++) atomicAdd(&h[b][(u32)(k >> (8 * b)) & 255u], 1u);
    if (nseg_pass) {
      u32 s = (u32)seg_of_val[vals[i]];
      for (int b = 0; b < nseg_pass; b++)
        atomicAdd(&h[nkey + b][(s >> (8 * b)) & 255u], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < np * 256; i += blockDim.x) {
    u32 c = (&h[0][0])[i];
    if (c) atomicAdd(&hist_all[i], c);
  }
}

__global__ void __launch_bounds__(SORT_THREADS)
k_tile_hist(const u64 *__restrict__ keys, const int *__restrict__ vals, ll n,
            const int *__restrict__ seg_of_val, int is_seg, int shift,
            u32 *__restrict__ counts, int ntiles) {
  __shared__ u32 h[NWARP][256];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < NWARP * 256; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  ll base = (ll)blockIdx.x * TILE + warp * (32 * ITEMS_PER_THREAD);
  u32 d[ITEMS_PER_THREAD];
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    ll i = base + r * 32 + lane;
    d[r] = i < n ? digit_of(keys[i], is_seg ? vals[i] : 0, seg_of_val, is_seg, shift) : 256u;
  }
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++)
    if (d[r] < 256) atomicAdd(&h[warp][d[r]], 1u);
  __syncthreads();
  for (int dd = threadIdx.x; dd < 256; dd += blockDim.x) {
    u32 s = 0;
#pragma unroll
    for (int w = 0; w < NWARP; w++) s += h[w][dd];
    counts[(ll)dd * ntiles + blockIdx.x] = s;
  }
}

// One CTA per digit: exclusive prefix of counts[d][0..ntiles) in place.
__global__ void k_tile_scan(u32 *__restrict__ counts, int ntiles,
                            u32 *__restrict__ totals) {
  __shared__ u32 wsum[32];
  __shared__ u32 carry_s;
  u32 *row = counts + (ll)blockIdx.x * ntiles;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int nw = blockDim.x >> 5;
  for (int base = 0; base < ntiles; base += blockDim.x) {
    int i = base + threadIdx.x;
    u32 v = i < ntiles ? row[i] : 0u;
    u32 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      u32 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      u32 s = lane < nw ? wsum[lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        u32 y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      if (lane < nw) wsum[lane] = s;
    }
    __syncthreads();
    u32 carry = carry_s;
    u32 excl = carry + (warp ? wsum[warp - 1] : 0u) + x - v;
    if (i < ntiles) row[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry_s = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry_s;
}

// lanes with the same 8-bit digit (of the lanes in `valid`), by a ballot per
// bit: __match_any_sync takes longer the more digits a warp holds
__device__ __forceinline__ u32 digit_peers(u32 d, u32 valid) {
  u32 peers = valid;
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool bit = (d >> b) & 1u;
    const u32 bal = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? bal : ~bal;
  }
  return peers;
}

__global__ void __launch_bounds__(SORT_THREADS)
k_scatter(const u64 *__restrict__ kin, const int *__restrict__ vin,
          u64 *__restrict__ kout, int *__restrict__ vout, ll n,
          const int *__restrict__ seg_of_val, int is_seg, int shift,
          const u32 *__restrict__ counts, const u32 *__restrict__ totals,
          int ntiles) {
  __shared__ u32 wcnt[NWARP][256];
  __shared__ u32 dbase[256];
  __shared__ u32 tl[256];  // tile-local start of each digit
  __shared__ u32 ws[8], ws2[8];
  extern __shared__ __align__(16) unsigned char sc_smem[];
  u64 *skey = reinterpret_cast<u64 *>(sc_smem);             // TILE
  int *sval = reinterpret_cast<int *>(skey + TILE);          // TILE
  unsigned char *sdig = reinterpret_cast<unsigned char *>(sval + TILE);  // TILE
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < NWARP * 256; i += blockDim.x) (&wcnt[0][0])[i] = 0;
  // global start of every digit in this tile: exclusive scan of the 256
  // digit totals (threads 0..255, one digit each) plus the tile's offset
  {
    const u32 v = threadIdx.x < 256 ? totals[threadIdx.x] : 0u;
    u32 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      u32 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (threadIdx.x < 256 && lane == 31) ws[warp] = x;
    __syncthreads();
    if (threadIdx.x < 256) {
      u32 off = 0;
      for (int w = 0; w < warp; w++) off += ws[w];
      dbase[threadIdx.x] = off + x - v + counts[(ll)threadIdx.x * ntiles + blockIdx.x];
    }
  }
  // every load of the tile is issued before the ranking loop
  u64 key[ITEMS_PER_THREAD];
  int val[ITEMS_PER_THREAD];
  u32 rank[ITEMS_PER_THREAD];
  u32 dig[ITEMS_PER_THREAD];
  const unsigned lt_mask = (1u << lane) - 1u;
  const ll base = (ll)blockIdx.x * TILE + warp * (32 * ITEMS_PER_THREAD);
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    const ll i = base + r * 32 + lane;
    if (i < n) {
      key[r] = kin[i];
      val[r] = vin[i];
    }
  }
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    const ll i = base + r * 32 + lane;
    dig[r] = i < n ? digit_of(key[r], val[r], seg_of_val, is_seg, shift) : 256u;
  }
  // stable rank within the warp's items (32 at a time, in order)
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    const u32 d = dig[r];
    const bool valid = d < 256;
    const unsigned peers = digit_peers(d, __ballot_sync(0xffffffffu, valid));
    u32 before = 0;
    if (valid) before = wcnt[warp][d];
    __syncwarp();
    if (valid) {
      rank[r] = before + __popc(peers & lt_mask);
      if (lane == __ffs(peers) - 1) wcnt[warp][d] = before + __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  // exclusive scan over warps per digit, then over the digits of the tile
  {
    u32 run = 0;
    if (threadIdx.x < 256) {
      const int d = threadIdx.x;
#pragma unroll
      for (int w = 0; w < NWARP; w++) {
        u32 t = wcnt[w][d];
        wcnt[w][d] = run;
        run += t;
      }
    }
    u32 x = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      u32 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (threadIdx.x < 256 && lane == 31) ws2[warp] = x;
    __syncthreads();
    if (threadIdx.x < 256) {
      u32 off = 0;
      for (int w = 0; w < warp; w++) off += ws2[w];
      tl[threadIdx.x] = off + x - run;
    }
  }
  __syncthreads();
  // stage the tile in digit order, then write every digit run with
  // consecutive addresses (coalesced stores instead of 256 scattered streams)
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    if (dig[r] < 256) {
      const u32 lp = tl[dig[r]] + wcnt[warp][dig[r]] + rank[r];
      skey[lp] = key[r];
      sval[lp] = val[r];
      sdig[lp] = (unsigned char)dig[r];
    }
  }
  __syncthreads();
  const ll t0 = (ll)blockIdx.x * TILE;
  const int tn = (int)(n - t0 < TILE ? n - t0 : TILE);
  for (int t = threadIdx.x; t < tn; t += blockDim.x) {
    const u32 d = sdig[t];
    const u32 pos = dbase[d] + ((u32)t - tl[d]);
    kout[pos] = skey[t];
    vout[pos] = sval[t];
  }
}

// ---------------------------------------------------------------------------
// Sort of doubles inside contiguous segments (sort_by_value).  The segments
// tile the positions, so they never move and need no digit passes of their
// own; what remains depends on the longest one:
//   up to RANK_MAX      every item counts the items of its segment before it
//   up to LOCAL_MAX     a CTA sorts whole segments in shared memory: a bucket
//                       per item of the segment, by value over the segment's
//                       range, and inside a bucket every item counts the ones
//                       before it (ties by position: stable); a bitonic
//                       network where too many items share a bucket
//   longer              four radix passes over 32-bit keys (segment, then the
//                       value in fixed point over the range of all values),
//                       half the bytes and half the passes of the 64-bit keys;
//                       the few items that share a 32-bit key are then put
//                       right by their full keys (k_fix_runs), long runs (a
//                       value that many items share, and one beside it) by a
//                       CTA each.  Runs too long for that (many values that
//                       differ in their last bits only, or one far outside the
//                       range of the others) or too many take the full radix
//                       sort, after the passes: RCB of 1M hexes 1.50 ms, with
//                       one far element 2.22, by the full sort alone 2.05 (8M:
//                       5.0, 7.6 and 8.2).  Asking a sample of 1024 keys first
//                       took 0.1 ms off the second and put 7 us on every sort
//                       of the first.
// ---------------------------------------------------------------------------
constexpr int RANK_MAX = 32;
constexpr int RANK_THREADS = 512;
constexpr int LOCAL_MAX = 4096;
constexpr int BUCKET_MAX = 128;  // items of a bucket that are ranked by counting
constexpr int FIX_MAX = 32;  // items of a run that one thread puts right
// Longer runs that CTAs put right.  A pipe of 96 x 72 x 106 without jitter has
// 3500 of 212 (two last-bit forms of a value, 106 times each): RCB of it takes
// 2.02 ms with them sorted by CTAs of 128 threads, 2.48 with the full sort, 2.37
// by the full sort alone.
constexpr int RUN_LIST = 1 << 16;
constexpr int RUN_SHORT = 512;  // items of a run that 128 threads sort

// keys[i], vals[i] of the segments of at most RANK_MAX items, out of place.
// The CTA sees its positions and RANK_MAX more on both sides.
__global__ void __launch_bounds__(RANK_THREADS)
k_seg_rank(const u64 *__restrict__ keys, const int *__restrict__ vals,
           const int *__restrict__ seg, ll n, u64 *__restrict__ kout, int *__restrict__ vout) {
  constexpr int W = RANK_THREADS + 2 * RANK_MAX;
  __shared__ u64 sk[W];
  __shared__ int ss[W];
  const ll base = (ll)blockIdx.x * RANK_THREADS - RANK_MAX;
  for (int k = threadIdx.x; k < W; k += RANK_THREADS) {
    const ll i = base + k;
    const bool in = i >= 0 && i < n;
    sk[k] = in ? keys[i] : 0ull;
    ss[k] = in ? seg[i] : -1 - (i < 0 ? 0 : 1);
  }
  __syncthreads();
  const int me = threadIdx.x + RANK_MAX;
  const ll i = base + me;
  if (i >= n) return;
  const u64 key = sk[me];
  const int s = ss[me];
  int before = 0, j = me - 1;
  for (; j >= 0 && ss[j] == s; j--) before += sk[j] <= key;
  const int first = j + 1;
  for (j = me + 1; j < W && ss[j] == s; j++) before += sk[j] < key;
  const ll to = base + first + before;
  kout[to] = key;
  vout[to] = vals[i];
}

// (one item of padding per eight, against bank conflicts)
__host__ __device__ constexpr int lo_at(int i) { return i + (i >> 3); }
constexpr size_t local_smem(int w) { return (size_t)lo_at(w) * 12; }
struct LoItem {
  u64 k;
  u32 p;  // segment above bit 16, place below (ties by place)
};
__device__ __forceinline__ void lo_exchange(LoItem &a, LoItem &b, bool up) {
  const u32 ga = a.p >> 16, gb = b.p >> 16;
  const bool gt = ga != gb ? ga > gb : (a.k != b.k ? a.k > b.k : a.p > b.p);
  if (gt == up) {
    const LoItem t = a;
    a = b;
    b = t;
  }
}
// K strides of the network, st, st / 2, ..., at once: a thread keeps the 2^K
// items they connect in registers, so a pass over shared memory does three
// steps instead of one (32 segments of 8192 items: 116 -> 96 us)
template <int THREADS, int K>
__device__ __forceinline__ void lo_steps(u64 *sk, u32 *sp, int p2, int size, int st) {
  const int lo = st >> (K - 1);
  for (int u = threadIdx.x; u < p2 >> K; u += THREADS) {
    const int low = u & (lo - 1), base = ((u - low) << K) + low;
    const bool up = (base & size) == 0;
    LoItem v[1 << K];
#pragma unroll
    for (int j = 0; j < 1 << K; j++) {
      const int i = lo_at(base + j * lo);
      v[j].k = sk[i], v[j].p = sp[i];
    }
#pragma unroll
    for (int b = K - 1; b >= 0; b--)
#pragma unroll
      for (int j = 0; j < 1 << K; j++)
        if (!(j & (1 << b))) lo_exchange(v[j], v[j | (1 << b)], up);
#pragma unroll
    for (int j = 0; j < 1 << K; j++) {
      const int i = lo_at(base + j * lo);
      sk[i] = v[j].k, sp[i] = v[j].p;
    }
  }
  __syncthreads();
}
// p2 (a power of two) items in shared memory, by the whole CTA
template <int THREADS>
__device__ __forceinline__ void bitonic_sort(u64 *sk, u32 *sp, int p2) {
  for (int size = 2; size <= p2; size <<= 1) {
    int st = size >> 1;
    for (; st >= 4; st >>= 3) lo_steps<THREADS, 3>(sk, sp, p2, size, st);
    if (st == 2)
      lo_steps<THREADS, 2>(sk, sp, p2, size, st);
    else if (st == 1)
      lo_steps<THREADS, 1>(sk, sp, p2, size, st);
  }
}
// the sorted items out: keys from sk, values moved from their old places
template <int W, int THREADS>
__device__ __forceinline__ void local_store(const u64 *sk, const u32 *sp, int m,
                                            u64 *__restrict__ keys, int *__restrict__ vals) {
  int v[W / THREADS];
#pragma unroll
  for (int r = 0; r < W / THREADS; r++) {
    const int k = threadIdx.x + r * THREADS;
    v[r] = k < m ? vals[sp[lo_at(k)] & 0xFFFFu] : 0;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < W / THREADS; r++) {
    const int k = threadIdx.x + r * THREADS;
    if (k < m) keys[k] = sk[lo_at(k)], vals[k] = v[r];
  }
}
// Segments of at most W / 2 items: CTA b sorts those that start in
// [b W / 2, (b + 1) W / 2), in place.  Bound by its shared-memory accesses
// (about 40 per item; the bitonic network took 1000 instructions): 8M points
// in lines of 512, 428 -> 273 us.
template <int W>
constexpr size_t seg_local_smem() {
  return (size_t)lo_at(W) * 8 + (size_t)W * 12;
}
template <int W, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
k_seg_local(u64 *__restrict__ keys, int *__restrict__ vals, const int *__restrict__ seg, ll n) {
  constexpr int H = W / 2, PER = W / THREADS;
  extern __shared__ __align__(16) unsigned char lo_smem[];
  u64 *sk = reinterpret_cast<u64 *>(lo_smem);
  u32 *A = reinterpret_cast<u32 *>(sk + lo_at(W)), *B = A + W, *C = B + W;
  unsigned short *list = reinterpret_cast<unsigned short *>(C);
  __shared__ int s_lo, s_hi;
  __shared__ u64 s_min, s_max;
  const ll b0 = (ll)blockIdx.x * H;
  if (threadIdx.x == 0) s_lo = 1 << 30, s_hi = 1 << 30, s_min = ~0ull, s_max = 0ull;
  __syncthreads();
  // the first start at or after b0, and at or after b0 + H (else the end)
  for (int k = threadIdx.x; k <= W; k += THREADS) {
    const ll i = b0 + k;
    if (i > n) break;
    if (i == n || i == 0 || (seg ? seg[i] != seg[i - 1] : false)) {
      if (k < H) atomicMin(&s_lo, k);
      if (k >= H || i == n) atomicMin(&s_hi, k);
    }
  }
  __syncthreads();
  const int lo = s_lo, hi = s_hi;
  const int m = hi - lo;
  if (lo >= H || m <= 1 || m > W) return;
  const ll i0 = b0 + lo;
  const int seg0 = seg ? seg[i0] : 0;
  u64 mn = ~0ull, mx = 0ull;
  for (int k = threadIdx.x; k < m; k += THREADS) {
    const u64 key = keys[i0 + k];
    sk[lo_at(k)] = key;
    A[k] = (u32)(seg ? seg[i0 + k] - seg0 : 0);
    B[k] = 0xFFFFFFFFu;
    C[k] = 0u;
    mn = key < mn ? key : mn;
    mx = key > mx ? key : mx;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const u64 a = __shfl_xor_sync(0xffffffffu, mn, o), b = __shfl_xor_sync(0xffffffffu, mx, o);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
  if ((threadIdx.x & 31) == 0) atomicMin(&s_min, mn), atomicMax(&s_max, mx);
  __syncthreads();
  // every item's segment (first place, length) and its value in 32-bit fixed
  // point over the CTA's range
  const u64 k0 = s_min, k1 = s_max;
  const int em = max(1, max(key_exp(k0), key_exp(k1)));
  const ll f0 = key_fixed(k0, em);
  const int sh = max(0, 32 - __clzll((ll)(u64)(key_fixed(k1, em) - f0)));
  int first[PER], len[PER];
  u32 q[PER];
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int k = threadIdx.x + r * THREADS;
    first[r] = 0, len[r] = m, q[r] = 0;
    if ((k & ~31) >= m) continue;  // (warp-uniform)
    const bool in = k < m;
    if (in && seg) {
      const u32 s = A[k];
      int a = 0, b = k;  // first place of the segment
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (A[mid] < s)
          a = mid + 1;
        else
          b = mid;
      }
      first[r] = a;
      int c = k + 1, d = min(m, a + H);  // first place after it
      while (c < d) {
        const int mid = (c + d) >> 1;
        if (A[mid] == s)
          c = mid + 1;
        else
          d = mid;
      }
      len[r] = c - a;
    }
    if (in) q[r] = (u32)((u64)(key_fixed(sk[lo_at(k)], em) - f0) >> sh);
    // one atomic a warp where it lies in one segment
    const int a0 = __shfl_sync(0xffffffffu, first[r], 0);
    if (__all_sync(0xffffffffu, in && first[r] == a0)) {
      const u32 lo = __reduce_min_sync(0xffffffffu, q[r]);
      const u32 hi = __reduce_max_sync(0xffffffffu, q[r]);
      if ((threadIdx.x & 31) == 0) atomicMin(&B[a0], lo), atomicMax(&C[a0], hi);
    } else if (in) {
      atomicMin(&B[first[r]], q[r]);
      atomicMax(&C[first[r]], q[r]);
    }
  }
  __syncthreads();
  // bucket: a place of the segment, linear in the value (float conversion,
  // product and truncation never decrease)
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int k = threadIdx.x + r * THREADS;
    if (k >= m) continue;
    const u32 q0 = B[first[r]];
    const float scale = (float)len[r] / ((float)(C[first[r]] - q0) + 1.0f);
    const int off = min(len[r] - 1, (int)((float)(q[r] - q0) * scale));
    q[r] = (u32)(first[r] + off);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += THREADS) A[k] = 0u, B[k] = 0u;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < PER; r++)
    if (threadIdx.x + r * THREADS < m) atomicAdd(&A[q[r]], 1u);
  __syncthreads();
  const u32 big = cta_scan<W, THREADS>(A, m);
  if (big > BUCKET_MAX) {
    // (A and B become the places; an item's segment is known by its first place)
    u32 *sp = A;
    int p2 = 2;
    while (p2 < m) p2 <<= 1;
#pragma unroll
    for (int r = 0; r < PER; r++) {
      const int k = threadIdx.x + r * THREADS;
      if (k >= p2) continue;
      if (k >= m) sk[lo_at(k)] = ~0ull;
      sp[lo_at(k)] = k < m ? (u32)first[r] << 16 | (u32)k : 0xFFFF0000u | (u32)k;
    }
    __syncthreads();
    bitonic_sort<THREADS>(sk, sp, p2);
    local_store<W, THREADS>(sk, sp, m, keys + i0, vals + i0);
    return;
  }
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int k = threadIdx.x + r * THREADS;
    if (k < m) list[A[q[r]] + atomicAdd(&B[q[r]], 1u)] = (unsigned short)k;
  }
  __syncthreads();
  int v[PER];
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int k = threadIdx.x + r * THREADS;
    if (k >= m) continue;
    const u64 key = sk[lo_at(k)];
    const int a = (int)A[q[r]], c = (int)B[q[r]];
    int before = 0;
    for (int j = a; j < a + c; j++) {
      const int o = list[j];
      const u64 ko = sk[lo_at(o)];
      before += ko < key || (ko == key && o < k);
    }
    q[r] = (u32)(a + before);
    v[r] = vals[i0 + k];
  }
  __syncthreads();  // every value is read before the first is written
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int k = threadIdx.x + r * THREADS;
    if (k < m) keys[i0 + q[r]] = sk[lo_at(k)], vals[i0 + q[r]] = v[r];
  }
}

__global__ void k_range_init(u64 *__restrict__ range) {
  range[0] = ~0ull, range[1] = 0ull, range[2] = 0ull, range[3] = 0ull, range[4] = 0ull;
}
__global__ void k_key_range(const u64 *__restrict__ keys, ll n, u64 *__restrict__ range) {
  u64 mn = ~0ull, mx = 0ull;
  const ll stride = (ll)gridDim.x * blockDim.x;
  for (ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const u64 k = keys[i];
    mn = k < mn ? k : mn;
    mx = k > mx ? k : mx;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const u64 a = __shfl_xor_sync(0xffffffffu, mn, o), b = __shfl_xor_sync(0xffffffffu, mx, o);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
  __shared__ u64 smn[32], smx[32];
  if ((threadIdx.x & 31) == 0) smn[threadIdx.x >> 5] = mn, smx[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      mn = smn[w] < mn ? smn[w] : mn;
      mx = smx[w] > mx ? smx[w] : mx;
    }
    atomicMin(&range[0], mn);
    atomicMax(&range[1], mx);
  }
}

// q[i] = segment (top sb bits), value over the range (32 - sb bits)
constexpr int QU_THREADS = 256, QU_ITEMS = 4;  // (the range's shifts once per thread)
__global__ void __launch_bounds__(QU_THREADS)
k_quant(const u64 *__restrict__ keys, const int *__restrict__ seg, ll n, int sb,
        const u64 *__restrict__ range, u32 *__restrict__ q) {
  const ll i0 = (ll)blockIdx.x * (QU_THREADS * QU_ITEMS) + threadIdx.x;
  const u64 k0 = range[0], k1 = range[1];
  const int em = max(1, max(key_exp(k0), key_exp(k1)));
  const ll f0 = key_fixed(k0, em);
  const u64 r = (u64)(key_fixed(k1, em) - f0);
  const int s = max(0, 64 - __clzll((ll)r) - (32 - sb));
  u64 k[QU_ITEMS];
  u32 g[QU_ITEMS];
#pragma unroll
  for (int u = 0; u < QU_ITEMS; u++) {
    const ll i = i0 + u * QU_THREADS;
    k[u] = i < n ? keys[i] : 0ull;
    g[u] = seg && sb && i < n ? (u32)seg[i] << (32 - sb) : 0u;
  }
#pragma unroll
  for (int u = 0; u < QU_ITEMS; u++) {
    const ll i = i0 + u * QU_THREADS;
    if (i < n) q[i] = (u32)((u64)(key_fixed(k[u], em) - f0) >> s) | g[u];
  }
}

__global__ void __launch_bounds__(SORT_THREADS)
k_tile_hist32(const u32 *__restrict__ q, ll n, int shift, u32 *__restrict__ counts, int ntiles) {
  __shared__ u32 h[NWARP][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < NWARP * 256; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  const ll base = (ll)blockIdx.x * TILE + warp * (32 * ITEMS_PER_THREAD);
  u32 d[ITEMS_PER_THREAD];
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    const ll i = base + r * 32 + lane;
    d[r] = i < n ? (q[i] >> shift) & 255u : 256u;
  }
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++)
    if (d[r] < 256) atomicAdd(&h[warp][d[r]], 1u);
  __syncthreads();
  for (int dd = threadIdx.x; dd < 256; dd += blockDim.x) {
    u32 s = 0;
#pragma unroll
    for (int w = 0; w < NWARP; w++) s += h[w][dd];
    counts[(ll)dd * ntiles + blockIdx.x] = s;
  }
}

// k_scatter for 32-bit keys: a pair is one 8-byte word in shared memory; vin
// null: the positions.  The peers of all rounds are found before the counts,
// which are a serial chain (8M random digits: 91 -> 56 us).
__global__ void __launch_bounds__(SORT_THREADS)
k_scatter32(const u32 *__restrict__ kin, const int *__restrict__ vin, u32 *__restrict__ kout,
            int *__restrict__ vout, ll n, int shift, const u32 *__restrict__ counts,
            const u32 *__restrict__ totals, int ntiles) {
  __shared__ u32 wcnt[NWARP][256];
  __shared__ u32 gbase[256];  // global place of a digit's first item of this tile, minus its local one
  __shared__ u32 tl[256];
  __shared__ u32 ws[8], ws2[8];
  extern __shared__ __align__(16) unsigned char sc_smem[];
  uint2 *st = reinterpret_cast<uint2 *>(sc_smem);  // TILE
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < NWARP * 256; i += blockDim.x) (&wcnt[0][0])[i] = 0;
  u32 dbase = 0;
  {
    const u32 v = threadIdx.x < 256 ? totals[threadIdx.x] : 0u;
    u32 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (threadIdx.x < 256 && lane == 31) ws[warp] = x;
    __syncthreads();
    if (threadIdx.x < 256) {
      u32 off = 0;
      for (int w = 0; w < warp; w++) off += ws[w];
      dbase = off + x - v + counts[(ll)threadIdx.x * ntiles + blockIdx.x];
    }
  }
  u32 key[ITEMS_PER_THREAD], rank[ITEMS_PER_THREAD];
  int val[ITEMS_PER_THREAD];
  const unsigned lt_mask = (1u << lane) - 1u;
  const ll base = (ll)blockIdx.x * TILE + warp * (32 * ITEMS_PER_THREAD);
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    const ll i = base + r * 32 + lane;
    key[r] = i < n ? kin[i] : 0u;
    val[r] = i < n ? (vin ? vin[i] : (int)i) : 0;
  }
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++)
    rank[r] = digit_peers(key[r] >> shift,
                          __ballot_sync(0xffffffffu, base + r * 32 + lane < n));
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++) {
    const bool valid = base + r * 32 + lane < n;
    const u32 d = valid ? (key[r] >> shift) & 255u : 256u;
    const unsigned peers = rank[r];
    u32 before = 0;
    if (valid) before = wcnt[warp][d];
    __syncwarp();
    rank[r] = before + __popc(peers & lt_mask);
    if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    u32 run = 0;
    if (threadIdx.x < 256) {
      const int d = threadIdx.x;
#pragma unroll
      for (int w = 0; w < NWARP; w++) {
        const u32 t = wcnt[w][d];
        wcnt[w][d] = run;
        run += t;
      }
    }
    u32 x = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (threadIdx.x < 256 && lane == 31) ws2[warp] = x;
    __syncthreads();
    if (threadIdx.x < 256) {
      u32 off = 0;
      for (int w = 0; w < warp; w++) off += ws2[w];
      const u32 t0 = off + x - run;
      tl[threadIdx.x] = t0;
      gbase[threadIdx.x] = dbase - t0;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS_PER_THREAD; r++)
    if (base + r * 32 + lane < n) {
      const u32 d = (key[r] >> shift) & 255u;
      st[tl[d] + wcnt[warp][d] + rank[r]] = make_uint2(key[r], (u32)val[r]);
    }
  __syncthreads();
  const ll t0 = (ll)blockIdx.x * TILE;
  const int tn = (int)(n - t0 < TILE ? n - t0 : TILE);
  for (int t = threadIdx.x; t < tn; t += blockDim.x) {
    const uint2 kv = st[t];
    const u32 pos = gbase[(kv.x >> shift) & 255u] + (u32)t;
    kout[pos] = kv.x;
    vout[pos] = (int)kv.y;
  }
}

// idx: positions in, values out (null vals: the positions)
__global__ void k_gather_kv(int *__restrict__ idx, const u64 *__restrict__ keys,
                            const int *__restrict__ vals, ll n, u64 *__restrict__ kout) {
  const ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int j = idx[i];
  kout[i] = keys[j];
  if (vals) idx[i] = vals[j];
}

__global__ void k_gather_val(const int *__restrict__ idx, const int *__restrict__ in, ll n,
                             int *__restrict__ out) {
  const ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[idx[i]];
}
__global__ void k_iota_pos(int *__restrict__ a, ll n) {
  const ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = (int)i;
}

// Runs of equal 32-bit keys into the order of their full keys: the thread of a
// run's first item sorts a run of at most FIX_MAX by insertion (stable); of a
// longer one every pair of neighbours is checked, and a run that is not in
// order is listed once (mark, a bit per item, zero before the launch) for
// k_sort_run.
// range[2]: a run cannot be listed; range[3]: runs listed.
__device__ __forceinline__ ll run_bound(const u32 *__restrict__ q, ll n, u64 v) {
  ll lo = 0, hi = n;  // first position with q >= v
  while (lo < hi) {
    const ll mid = (lo + hi) >> 1;
    if ((u64)q[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}
__device__ __forceinline__ void list_run(const u32 *__restrict__ q, ll n, u32 qi,
                                         u64 *__restrict__ range, u32 *__restrict__ mark,
                                         int2 *__restrict__ runs) {
  if (*(volatile u64 *)&range[2]) return;
  const ll b = run_bound(q, n, qi);
  const u32 bit = 1u << (b & 31);
  if (atomicOr(&mark[b >> 5], bit) & bit) return;
  const ll e = run_bound(q, n, (u64)qi + 1);
  const u64 at = e - b <= LOCAL_MAX ? atomicAdd(&range[3], 1ull) : (u64)RUN_LIST;
  if (at < RUN_LIST) {
    runs[at] = make_int2((int)b, (int)(e - b));
    if (range[4] < (u64)(e - b)) atomicMax(&range[4], (u64)(e - b));
  } else
    range[2] = 1ull;
}
__global__ void k_fix_runs(const u32 *__restrict__ q, ll n, u64 *__restrict__ keys,
                           int *__restrict__ vals, u64 *__restrict__ range,
                           u32 *__restrict__ mark, int2 *__restrict__ runs) {
  const ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = i < n;
  const u32 qi = in ? q[i] : 0u;
  const bool first = in && !(i > 0 && q[i - 1] == qi);
  const bool list = in && !first && i >= FIX_MAX && q[i - FIX_MAX] == qi && keys[i] < keys[i - 1];
  const unsigned lists = __ballot_sync(0xffffffffu, list);
  if (lists) {  // (the first of a run's lanes: the run is looked up once a warp)
    const int lane = threadIdx.x & 31;
    const unsigned before = lists & ((1u << lane) - 1u);
    const u32 qb = __shfl_sync(0xffffffffu, qi, before ? 31 - __clz((int)before) : lane);
    if (list && (!before || qb != qi)) list_run(q, n, qi, range, mark, runs);
  }
  if (!first) return;
  int len = 1;
  bool sorted = true;
  u64 prev = keys[i];
  while (len <= FIX_MAX && i + len < n && q[i + len] == qi) {
    const u64 k = keys[i + len];
    sorted = sorted && prev <= k;
    prev = k;
    len++;
  }
  if (sorted) return;
  if (len > FIX_MAX) {
    list_run(q, n, qi, range, mark, runs);
    return;
  }
  for (int a = 1; a < len; a++) {
    const u64 k = keys[i + a];
    const int v = vals[i + a];
    int b = a;
    while (b > 0 && keys[i + b - 1] > k) {
      keys[i + b] = keys[i + b - 1];
      vals[i + b] = vals[i + b - 1];
      b--;
    }
    keys[i + b] = k;
    vals[i + b] = v;
  }
}
// one CTA per listed run of more than MIN and at most MAX items
template <int MIN, int MAX, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_sort_run(const int2 *__restrict__ runs, u64 *__restrict__ keys, int *__restrict__ vals) {
  extern __shared__ __align__(16) unsigned char lo_smem[];
  u64 *sk = reinterpret_cast<u64 *>(lo_smem);
  u32 *sp = reinterpret_cast<u32 *>(sk + lo_at(MAX));
  const int2 r = runs[blockIdx.x];
  if (r.y <= MIN || r.y > MAX) return;
  int p2 = 2;
  while (p2 < r.y) p2 <<= 1;
  for (int k = threadIdx.x; k < p2; k += THREADS) {
    sk[lo_at(k)] = k < r.y ? keys[r.x + k] : ~0ull;
    sp[lo_at(k)] = k < r.y ? (u32)k : 0xFFFF0000u | (u32)k;
  }
  __syncthreads();
  bitonic_sort<THREADS>(sk, sp, p2);
  local_store<MAX, THREADS>(sk, sp, r.y, keys + r.x, vals + r.x);
}

int bits_for(ll nseg) {
  int b = 0;
  while (nseg > 1 && ((ll)1 << b) < nseg) b++;
  return b;
}

}  // namespace

void seg_sort_pairs(DBuf<u64> &keys, DBuf<int> &vals, ll n,
                    const int *seg_of_val, ll nseg, SortWs &ws) {
  if (n <= 1) return;
  cudaStream_t st = ctx().stream;
  int seg_bits = seg_of_val ? bits_for(nseg) : 0;
  int nseg_pass = (seg_bits + 7) / 8;
  int nkey = 8;
  int np = nkey + nseg_pass;
  int ntiles = (int)((n + TILE - 1) / TILE);
  ws.ktmp.ensure((size_t)n);
  ws.vtmp.ensure((size_t)n);
  ws.counts.ensure((size_t)256 * ntiles);
  ws.totals.ensure(256);
  ws.hist_all.ensure((size_t)MAX_PASSES * 256);
  CK(cudaMemsetAsync(ws.hist_all.p, 0, (size_t)np * 256 * sizeof(u32), st));
  int gblocks = (int)((n + 255) / 256);
  if (gblocks > 152 * 8) gblocks = 152 * 8;
  k_hist_all<<<gblocks, 256, 0, st>>>(keys.p, vals.p, n, seg_of_val, nkey,
                                       nseg_pass, ws.hist_all.p);
  CK_LAUNCH();
  std::vector<u32> h((size_t)np * 256);
  d2h(h.data(), ws.hist_all.p, h.size());
  sync();
  PassDesc passes[MAX_PASSES];
  int npasses = 0;
  for (int b = 0; b < np; b++) {
    bool trivial = false;
    for (int d = 0; d < 256; d++)
      if (h[(size_t)b * 256 + d] == (u32)n) trivial = true;
    if (trivial) continue;
    passes[npasses].is_seg = b >= nkey;
    passes[npasses].shift = b >= nkey ? 8 * (b - nkey) : 8 * b;
    npasses++;
  }
  ensure_smem_limit(k_scatter, (int)SCATTER_SMEM);  // staging exceeds the 48 KB default
  for (int q = 0; q < npasses; q++) {
    const PassDesc &pd = passes[q];
    k_tile_hist<<<ntiles, SORT_THREADS, 0, st>>>(keys.p, vals.p, n, seg_of_val,
                                                 pd.is_seg, pd.shift,
                                                 ws.counts.p, ntiles);
    CK_LAUNCH();
    k_tile_scan<<<256, 1024, 0, st>>>(ws.counts.p, ntiles, ws.totals.p);
    CK_LAUNCH();
    k_scatter<<<ntiles, SORT_THREADS, SCATTER_SMEM, st>>>(keys.p, vals.p, ws.ktmp.p,
                                               ws.vtmp.p, n, seg_of_val,
                                               pd.is_seg, pd.shift, ws.counts.p,
                                               ws.totals.p, ntiles);
    CK_LAUNCH();
    std::swap(keys.p, ws.ktmp.p);
    std::swap(keys.n, ws.ktmp.n);
    std::swap(vals.p, ws.vtmp.p);
    std::swap(vals.n, ws.vtmp.n);
  }
}

void sort_by_value(DBuf<u64> &keys, DBuf<int> &vals, ll n, const int *seg_of_pos, ll nseg,
                   ll max_len, SortWs &ws, bool iota) {
  if (n <= 1 || max_len <= 1) return;
  cudaStream_t st = ctx().stream;
  if (!seg_of_pos) nseg = 1;
  if (seg_of_pos && max_len <= RANK_MAX) {
    ws.ktmp.ensure((size_t)n);
    ws.vtmp.ensure((size_t)n);
    k_seg_rank<<<grid_for(n, RANK_THREADS), RANK_THREADS, 0, st>>>(keys.p, vals.p, seg_of_pos, n,
                                                                   ws.ktmp.p, ws.vtmp.p);
    CK_LAUNCH();
    std::swap(keys, ws.ktmp);
    std::swap(vals, ws.vtmp);
    return;
  }
  if (max_len <= 1024) {
    k_seg_local<2048, 512><<<grid_for(n, 1024), 512, seg_local_smem<2048>(), st>>>(
        keys.p, vals.p, seg_of_pos, n);
    CK_LAUNCH();
    return;
  }
  if (max_len <= LOCAL_MAX) {
    auto kern = k_seg_local<2 * LOCAL_MAX, 1024>;
    ensure_smem_limit(kern, (int)seg_local_smem<2 * LOCAL_MAX>());
    kern<<<grid_for(n, LOCAL_MAX), 1024, seg_local_smem<2 * LOCAL_MAX>(), st>>>(keys.p, vals.p,
                                                                                seg_of_pos, n);
    CK_LAUNCH();
    return;
  }
  const int sb = bits_for(nseg);
  bool full = sb > 16;  // too few bits left for the values
  if (!full) {
    ws.range.ensure(5);
    ws.runs.ensure((size_t)std::min<ll>(RUN_LIST, n / FIX_MAX + 1));
    ws.q.ensure((size_t)n), ws.mark.ensure((size_t)(n + 31) / 32);
    ws.ktmp.ensure((size_t)n), ws.vtmp.ensure((size_t)n);
    // the passes go from (qa, ia) to (qb, ib) and back; ktmp holds the second
    // pair until it takes the sorted keys
    u32 *qa = ws.q.p, *qb = reinterpret_cast<u32 *>(ws.ktmp.p);
    int *ia = ws.vtmp.p, *ib = reinterpret_cast<int *>(qb + n);
    const int ntiles = (int)((n + TILE - 1) / TILE);
    ws.counts.ensure((size_t)256 * ntiles);
    ws.totals.ensure(256);
    k_range_init<<<1, 1, 0, st>>>(ws.range.p);
    CK_LAUNCH();
    k_key_range<<<(unsigned)std::min<ll>((n + 1023) / 1024, 152 * 4), 256, 0, st>>>(keys.p, n,
                                                                                  ws.range.p);
    CK_LAUNCH();
    k_quant<<<grid_for(n, QU_THREADS * QU_ITEMS), QU_THREADS, 0, st>>>(keys.p, seg_of_pos, n, sb,
                                                                       ws.range.p, ws.q.p);
    CK_LAUNCH();
    ensure_smem_limit(k_scatter32, (int)(TILE * sizeof(uint2)));  // with the tables over 48 KB
    for (int shift = 0; shift < 32; shift += 8) {  // (an even number: back in qa, ia)
      k_tile_hist32<<<ntiles, SORT_THREADS, 0, st>>>(qa, n, shift, ws.counts.p, ntiles);
      CK_LAUNCH();
      k_tile_scan<<<256, 1024, 0, st>>>(ws.counts.p, ntiles, ws.totals.p);
      CK_LAUNCH();
      k_scatter32<<<ntiles, SORT_THREADS, TILE * sizeof(uint2), st>>>(
          qa, shift ? ia : nullptr, qb, ib, n, shift, ws.counts.p, ws.totals.p, ntiles);
      CK_LAUNCH();
      std::swap(qa, qb);
      std::swap(ia, ib);
    }
    k_gather_kv<<<grid_for(n, 256), 256, 0, st>>>(ws.vtmp.p, keys.p, iota ? nullptr : vals.p, n,
                                                  ws.ktmp.p);
    CK_LAUNCH();
    CK(cudaMemsetAsync(ws.mark.p, 0, (size_t)(n + 31) / 32 * sizeof(u32), st));
    k_fix_runs<<<grid_for(n, 256), 256, 0, st>>>(ws.q.p, n, ws.ktmp.p, ws.vtmp.p, ws.range.p,
                                                 ws.mark.p, ws.runs.p);
    CK_LAUNCH();
    u64 said[3] = {0, 0, 0};
    d2h(said, ws.range.p + 2, 3);
    sync();
    full = said[0] != 0;
    if (!full && said[1] > 0) {
      k_sort_run<0, RUN_SHORT, 128><<<(unsigned)said[1], 128, local_smem(RUN_SHORT), st>>>(
          ws.runs.p, ws.ktmp.p, ws.vtmp.p);
      CK_LAUNCH();
    }
    if (!full && said[2] > RUN_SHORT) {
      auto kern = k_sort_run<RUN_SHORT, LOCAL_MAX, 1024>;
      ensure_smem_limit(kern, (int)local_smem(LOCAL_MAX));
      kern<<<(unsigned)said[1], 1024, local_smem(LOCAL_MAX), st>>>(ws.runs.p, ws.ktmp.p,
                                                                   ws.vtmp.p);
      CK_LAUNCH();
    }
  }
  if (!full) {
    std::swap(keys, ws.ktmp);
    std::swap(vals, ws.vtmp);
    return;
  }
  // the full radix sort; of (key, position) where the segments go by position
  if (nseg == 1) {
    seg_sort_pairs(keys, vals, n, nullptr, 1, ws);
    return;
  }
  ws.q.release();
  ws.pos.ensure((size_t)n);
  k_iota_pos<<<grid_for(n, 256), 256, 0, st>>>(ws.pos.p, n);
  CK_LAUNCH();
  seg_sort_pairs(keys, ws.pos, n, seg_of_pos, nseg, ws);
  ws.vtmp.ensure((size_t)n);
  k_gather_val<<<grid_for(n, 256), 256, 0, st>>>(ws.pos.p, vals.p, n, ws.vtmp.p);
  CK_LAUNCH();
  std::swap(vals, ws.vtmp);
}

}  // namespace prsb
