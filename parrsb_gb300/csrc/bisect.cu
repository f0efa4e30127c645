// bisect.cu -- element centroids and the segmented RCB / RIB engine.
//
// Restates, for all groups of a recursion level at once:
//   rcb / rcb_level / rcb_local / get_axis_len   src/rcb.c:7-137
//   rib / rib_level / rib_local / get_rib_axis   src/rib.c:6-111
//   power_serial                                  src/fiedler.c:38-73
//   load_balance centroids                        src/parrsb.c:139-145
// A group of p virtual ranks is a segment [start, start+n) of the element
// order; each recursion step sorts every active segment stably along its
// axis (one segmented radix sort for the whole level) and splits it at the
// element count of its lower ceil(p/2) ranks.  Arithmetic that decides the
// order (centroid sums, RIB means, inertia sums, power iteration, projection
// keys) uses round-to-nearest intrinsics with no FMA, so keys are bit-equal
// to the CPU restatement's.  Group sums use the canonical 32-wide tile tree.
#include <float.h>

#include <algorithm>

#include "bisect.cuh"

#include <type_traits>

namespace prsb {

namespace {

// Bound by the FP64 pipe (64 cycles a warp instruction) and then by memory:
// corners come through shared memory, the first one needs no addition, and a
// division by 4 or 8 is an exact product.  8M hexes: 0.84 -> 0.44 ms.
constexpr int CE_ELEMS = 128;
__device__ __forceinline__ double no_minus_zero(double x) {  // 0.0 + x
  return (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) == 0u ? 0.0 : x;
}
template <int NV>
__global__ void __launch_bounds__(CE_ELEMS)
k_centroids(const double *__restrict__ xyz, int nel, double *__restrict__ cent) {
  constexpr int ND = NV == 8 ? 3 : 2, ROW = NV * ND, PAD = ROW + 1;
  extern __shared__ double ce_smem[];
  const int e0 = blockIdx.x * CE_ELEMS, ne = min(CE_ELEMS, nel - e0);
  const double *x = xyz + (ll)e0 * ROW;
#pragma unroll 8
  for (int k = threadIdx.x; k < ne * ROW; k += CE_ELEMS) ce_smem[k / ROW * PAD + k % ROW] = x[k];
  __syncthreads();
  if ((int)threadIdx.x >= ne) return;
  const double *c = ce_smem + threadIdx.x * PAD;
  const ll e = e0 + threadIdx.x;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double s = 0.0;
    if (d < ND) {
      s = no_minus_zero(c[d]);
#pragma unroll
      for (int v = 1; v < NV; v++) s = __dadd_rn(s, c[v * ND + d]);
      s = __dmul_rn(s, 1.0 / NV);
    }
    cent[d * (ll)nel + e] = s;
  }
}
// without coordinates, or with another number of corners
__global__ void k_centroids_any(const double *__restrict__ xyz, int nel, int nv, int ndim,
                                double *__restrict__ cent) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nel) return;
  double c[3] = {0.0, 0.0, 0.0};
  if (xyz) {
    const double *x = xyz + (ll)e * nv * ndim;
    for (int v = 0; v < nv; v++)
      for (int d = 0; d < ndim; d++) c[d] = __dadd_rn(c[d], x[v * ndim + d]);
    for (int d = 0; d < ndim; d++) c[d] = __ddiv_rn(c[d], (double)nv);
  }
  cent[e] = c[0];
  cent[(ll)nel + e] = c[1];
  cent[2 * (ll)nel + e] = c[2];
}

enum Gen { GEN_MEAN = 1, GEN_INERTIA = 2, GEN_ARRAY = 3 };

// Segment "active" rule shared by all kernels.
__device__ __forceinline__ bool seg_active(int p, ll n, int do_local) {
  return p > 1 || (do_local && p == 1 && n >= 2);
}

// Two canonical shuffle trees (offsets 16 .. 1) in one: after the first step
// the lanes of bit 4 carry the second value (a + b gives the same bits in
// either order), so two sums take five additions of the warp instead of ten;
// the FP64 pipe takes 16 cycles per warp instruction whatever its lanes do.
// a's sum ends on lane 0, b's on lane 16.
__device__ __forceinline__ double tree_pair(double a, double b) {
  const bool up = (threadIdx.x & 16) != 0;
  const double keep = up ? b : a, send = up ? a : b;
  double v = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, 16));
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, off));
  return v;
}

// the V values whose sums a segment takes, of element e (avg: the segment's means)
template <int V, int GEN>
__device__ __forceinline__ void seg_values(const double *__restrict__ cent, ll N, int e,
                                           const double *__restrict__ avg, double *v) {
  const double c0 = cent[e], c1 = cent[N + e], c2 = cent[2 * N + e];
  if (GEN == GEN_MEAN) {
    v[0] = c0, v[1] = c1, v[2] = c2;
  } else {  // inertia products (00, 01, 02, 11, 12, 22)
    const double x = __dsub_rn(c0, avg[0]), y = __dsub_rn(c1, avg[1]), z = __dsub_rn(c2, avg[2]);
    v[0] = __dmul_rn(x, x);
    v[1] = __dmul_rn(x, y);
    v[2] = __dmul_rn(x, z);
    v[3] = __dmul_rn(y, y);
    v[V - 2] = __dmul_rn(y, z);
    v[V - 1] = __dmul_rn(z, z);
  }
}

// V sums per segment (even V): one block per 1024 consecutive items of a
// segment takes two levels of the canonical 32-wide tree at once (a warp per
// 32-item tile, then the first warp over the tiles); a segment's count shrinks
// by 1024 per launch.  GEN_ARRAY reduces the previous launch's values.  Only
// segments with cnt[s] > 0 take part; a segment that already has one value is
// copied, not reduced again (the canonical tree stops at one value).
template <int V, int GEN>
__global__ void __launch_bounds__(1024)
k_seg_tree(const int *__restrict__ perm, const double *__restrict__ cent, ll N,
           const ll *__restrict__ seg_start, const int *__restrict__ cnt, ll nseg,
           const int *__restrict__ off, const double *__restrict__ in,
           const int *__restrict__ in_off, const double *__restrict__ avg,
           double *__restrict__ out) {
  static_assert(V % 2 == 0, "sums are folded in pairs");
  __shared__ double sv[V][32];
  __shared__ int s_seg;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int)blockIdx.x >= off[nseg]) return;
  if (threadIdx.x == 0) {
    ll lo = 0, hi = nseg - 1;  // last s with off[s] <= blockIdx.x
    while (lo < hi) {
      const ll mid = (lo + hi + 1) >> 1;
      if (off[mid] <= (int)blockIdx.x)
        lo = mid;
      else
        hi = mid - 1;
    }
    s_seg = (int)lo;
  }
  __syncthreads();
  const int s = s_seg;
  const int m = cnt[s], i = ((int)blockIdx.x - off[s]) * 1024 + (int)threadIdx.x;
  double v[V];
#pragma unroll
  for (int q = 0; q < V; q++) v[q] = 0.0;
  if (i < m) {
    if (GEN == GEN_ARRAY) {
      const ll src = ((ll)in_off[s] + i) * V;
#pragma unroll
      for (int q = 0; q < V; q++) v[q] = in[src + q];
    } else {
      seg_values<V, GEN>(cent, N, perm[seg_start[s] + i], avg + 3 * s, v);
    }
  }
  const int tiles = (m + 31) / 32;
  if (GEN == GEN_ARRAY && m == 1) {  // copied
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < V; q++) out[(ll)blockIdx.x * V + q] = v[q];
    return;
  }
#pragma unroll
  for (int q = 0; q < V; q += 2) {
    const double t = tree_pair(v[q], v[q + 1]);
    if (lane == 0) sv[q][warp] = t;
    if (lane == 16) sv[q + 1][warp] = t;
  }
  __syncthreads();
  if (warp > 0) return;
  const int mine = min(32, tiles - ((int)blockIdx.x - off[s]) * 32);  // tiles of this block
#pragma unroll
  for (int q = 0; q < V; q += 2) {
    const double a = lane < mine ? sv[q][lane] : 0.0, b = lane < mine ? sv[q + 1][lane] : 0.0;
    if (tiles == 1) {  // one value after the first level
      if (lane == 0) out[(ll)blockIdx.x * V + q] = a, out[(ll)blockIdx.x * V + q + 1] = b;
    } else {
      const double t = tree_pair(a, b);
      if (lane == 0) out[(ll)blockIdx.x * V + q] = t;
      if (lane == 16) out[(ll)blockIdx.x * V + q + 1] = t;
    }
  }
}

// The same sums where no segment has more than 1024 items: the whole tree of a
// segment in one block of as many threads as the largest asks for, or in a warp
// up to 32 items; sums of segment s at s V.  With a block of 1024 threads for
// every segment a level of 262144 segments of four elements took 14.0 ms for its
// two sums and their tables; these take 0.56.
template <int V, int GEN>
__global__ void __launch_bounds__(1024)
k_seg_block(const int *__restrict__ perm, const double *__restrict__ cent, ll N,
            const ll *__restrict__ seg_start, const ll *__restrict__ seg_n,
            const int *__restrict__ p, const double *__restrict__ avg, double *__restrict__ out) {
  __shared__ double sv[V][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ll s = blockIdx.x;
  if (p[s] <= 1) return;
  const int m = (int)seg_n[s], tiles = (m + 31) / 32;
  double v[V];
#pragma unroll
  for (int q = 0; q < V; q++) v[q] = 0.0;
  if ((int)threadIdx.x < m)
    seg_values<V, GEN>(cent, N, perm[seg_start[s] + threadIdx.x], avg + 3 * s, v);
#pragma unroll
  for (int q = 0; q < V; q += 2) {
    const double t = tree_pair(v[q], v[q + 1]);
    if (lane == 0) sv[q][warp] = t;
    if (lane == 16) sv[q + 1][warp] = t;
  }
  __syncthreads();
  if (warp > 0) return;
#pragma unroll
  for (int q = 0; q < V; q += 2) {
    double a = lane < tiles ? sv[q][lane] : 0.0, b = lane < tiles ? sv[q + 1][lane] : 0.0;
    if (tiles > 1) {  // (one value after the first level is the sum)
      const double t = tree_pair(a, b);
      a = t, b = __shfl_sync(0xffffffffu, t, 16);
    }
    if (lane == 0) out[s * V + q] = a, out[s * V + q + 1] = b;
  }
}
template <int V, int GEN>
__global__ void __launch_bounds__(256)
k_seg_warp(const int *__restrict__ perm, const double *__restrict__ cent, ll N,
           const ll *__restrict__ seg_start, const ll *__restrict__ seg_n,
           const int *__restrict__ p, ll nseg, const double *__restrict__ avg,
           double *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const ll s = ((ll)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= nseg || p[s] <= 1) return;  // (whole warps)
  double v[V];
#pragma unroll
  for (int q = 0; q < V; q++) v[q] = 0.0;
  if (lane < (int)seg_n[s])
    seg_values<V, GEN>(cent, N, perm[seg_start[s] + lane], avg + 3 * s, v);
#pragma unroll
  for (int q = 0; q < V; q += 2) {
    const double t = tree_pair(v[q], v[q + 1]);
    if (lane == 0) out[s * V + q] = t;
    if (lane == 16) out[s * V + q + 1] = t;
  }
}

// Tree launch l of a level reduces cnt_l[s] items of segment s (cnt_0: its
// elements, 0 without ranks to split; then a value per block of the launch
// before); off_l = exclusive scan of its blocks of 1024 items, off_l[nseg] all
// of them.  All launches' tables at once, at tab + 2 l (nseg + 1).
__global__ void __launch_bounds__(1024)
k_tree_offsets(const ll *__restrict__ n, const int *__restrict__ p, ll nseg, int launches,
               int *__restrict__ tab) {
  __shared__ int ws[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int *cnt = tab + 2 * (ll)blockIdx.x * (nseg + 1), *off = cnt + nseg + 1;
  int run = 0;
  for (ll b = 0; b < nseg; b += 1024) {
    const ll s = b + threadIdx.x;
    int c = s < nseg && p[s] > 1 ? (int)n[s] : 0;
    for (int l = 0; l < (int)blockIdx.x; l++) c = (c + 1023) / 1024;
    if (s < nseg) cnt[s] = c;
    const int v = (c + 1023) / 1024;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < 32; w++) {
      if (w < warp) before += ws[w];
      all += ws[w];
    }
    if (s < nseg) off[s] = run + before + x - v;
    run += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) off[nseg] = run;
}

// RCB boxes on the dense coordinate ranks: per segment and axis the minimum
// rank (slots 0..2) and the minimum complemented rank (slots 3..5, i.e. the
// maximum).  Integer atomics are order-independent, so the box does not
// depend on the grid; uniq[rank] turns a rank back into the exact coordinate.
// A thread reduces RBOX_ITEMS consecutive positions, a warp and then the
// block combine when they cover one segment (the common case), and only the
// threads that straddle a segment boundary issue their own atomics.
constexpr int RBOX_THREADS = 256, RBOX_ITEMS = 16;

__device__ __forceinline__ void rbox_flush(u32 *rbox, int s, int ndim, const u32 *v) {
  for (int a = 0; a < ndim; a++) {
    atomicMin(&rbox[6 * (ll)s + a], v[a]);
    atomicMin(&rbox[6 * (ll)s + 3 + a], v[3 + a]);
  }
}

__global__ void __launch_bounds__(RBOX_THREADS)
k_rank_box(const int *__restrict__ perm, const u32 *__restrict__ rank, ll N, int ndim,
           const int *__restrict__ seg_of_pos, u32 *__restrict__ rbox) {
  constexpr int NWB = RBOX_THREADS / 32;
  __shared__ int wseg[NWB];
  __shared__ u32 wval[NWB][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ll i0 = ((ll)blockIdx.x * RBOX_THREADS + threadIdx.x) * RBOX_ITEMS;
  int sg[RBOX_ITEMS], el[RBOX_ITEMS];
#pragma unroll
  for (int r = 0; r < RBOX_ITEMS; r++) {
    const bool ok = i0 + r < N;
    sg[r] = ok ? seg_of_pos[i0 + r] : -1;
    el[r] = ok ? perm[i0 + r] : 0;
  }
  u32 rk[3][RBOX_ITEMS];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int r = 0; r < RBOX_ITEMS; r++)
      rk[a][r] = (a < ndim && sg[r] >= 0) ? rank[(ll)a * N + el[r]] : 0u;
  int s = -1;
  u32 v[6];
#pragma unroll
  for (int q = 0; q < 6; q++) v[q] = ~0u;
#pragma unroll
  for (int r = 0; r < RBOX_ITEMS; r++) {
    if (sg[r] < 0) continue;
    if (sg[r] != s) {  // a segment boundary inside this thread's run
      if (s >= 0) rbox_flush(rbox, s, ndim, v);
#pragma unroll
      for (int q = 0; q < 6; q++) v[q] = ~0u;
      s = sg[r];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      v[a] = min(v[a], rk[a][r]);
      v[3 + a] = min(v[3 + a], ~rk[a][r]);
    }
  }
  // warp: one segment among the lanes that hold one -> shuffle-free reduce
  const int smin = (int)__reduce_min_sync(0xffffffffu, (unsigned)(s >= 0 ? s : 0x7fffffff));
  const int smax = (int)__reduce_max_sync(0xffffffffu, (unsigned)(s + 1)) - 1;
  if (smax >= 0 && smin == smax) {
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = __reduce_min_sync(0xffffffffu, v[q]);
    if (lane == 0) {
      wseg[warp] = smax;
#pragma unroll
      for (int q = 0; q < 6; q++) wval[warp][q] = v[q];
    }
  } else {
    if (s >= 0) rbox_flush(rbox, s, ndim, v);
    if (lane == 0) wseg[warp] = -1;
  }
  __syncthreads();
  if (warp == 0) {
    const int ws = lane < NWB ? wseg[lane] : -1;
    const int bmin = (int)__reduce_min_sync(0xffffffffu, (unsigned)(ws >= 0 ? ws : 0x7fffffff));
    const int bmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)(ws + 1)) - 1;
    u32 bv[6];
#pragma unroll
    for (int q = 0; q < 6; q++) bv[q] = ws >= 0 ? wval[lane < NWB ? lane : 0][q] : ~0u;
    if (bmax >= 0 && bmin == bmax) {
#pragma unroll
      for (int q = 0; q < 6; q++) bv[q] = __reduce_min_sync(0xffffffffu, bv[q]);
      if (lane == 0) rbox_flush(rbox, bmax, ndim, bv);
    } else if (ws >= 0) {
      rbox_flush(rbox, ws, ndim, bv);
    }
  }
}

// Longest box edge per segment from the rank boxes (strictly longer wins, so
// ties keep the lower axis, as with coordinate boxes).
__global__ void k_rcb_axis_rank(const u32 *__restrict__ rbox, const double *__restrict__ uniq,
                                ll N, const int *__restrict__ p, const ll *__restrict__ n,
                                ll nseg, int ndim, int do_local, int *__restrict__ axis) {
  ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  double len[3] = {0.0, 0.0, 0.0};
  if (n[s] > 0)
    for (int d = 0; d < ndim; d++) {
      const u32 lo = rbox[6 * s + d], hi = ~rbox[6 * s + 3 + d];
      len[d] = __dsub_rn(uniq[(ll)d * N + hi], uniq[(ll)d * N + lo]);
    }
  int ax = 0;
  for (int d = 1; d < ndim; d++)
    if (len[d] > len[ax]) ax = d;
  axis[s] = seg_active(p[s], n[s], do_local) ? ax : -1;
}

// Power iteration (fixed start vector (31, 17, 43)/50) on the first N*N
// entries of the row-major 3x3 tensor, as power_serial reads it, by the four
// lanes of a quad: lane j < N holds row j and y_j.  A dependent FP64
// instruction takes 64 cycles and a division about 570, so the rows' products
// run side by side and the two divisions of an iteration are one instruction
// sequence: lanes 0..2 scale by 1 / |Ay| while lane 3 takes the relative
// change of the eigenvalue.  Same operations in the same order per value as
// the serial loop: 68 -> 45 us per level.  Every lane of the warp calls it;
// quads that are done idle.
__device__ double power_quad(bool active, int N, const double *A) {
  const int j = threadIdx.x & 3, q0 = threadIdx.x & 28;
  const double start[3] = {31.0 / 50.0, 17.0 / 50.0, 43.0 / 50.0};
  double norm = 0.0;
  for (int i = 0; i < N; i++) norm = __dadd_rn(norm, __dmul_rn(start[i], start[i]));
  double y = __dmul_rn(j < N ? start[j < 3 ? j : 0] : 0.0, __ddiv_rn(1.0, __dsqrt_rn(norm)));
  double lambda = 0.0;
  bool run = active;
  for (int i = 0; i < 100; i++) {
    if (!__any_sync(0xffffffffu, run)) break;
    double ay = 0.0;
    for (int k = 0; k < N; k++) {
      const double yk = __shfl_sync(0xffffffffu, y, q0 + k);
      ay = __dadd_rn(ay, __dmul_rn(j < N ? A[j * N + k] : 0.0, yk));
    }
    const double sq = __dmul_rn(ay, ay);
    norm = 0.0;
    for (int k = 0; k < N; k++) norm = __dadd_rn(norm, __shfl_sync(0xffffffffu, sq, q0 + k));
    const double sn = __dsqrt_rn(norm);
    const double d = __ddiv_rn(j == 3 ? __dsub_rn(sn, lambda) : 1.0, j == 3 ? lambda : sn);
    const double err = i > 0 ? __shfl_sync(0xffffffffu, d, q0 + 3) : 1.0;
    if (run) {
      lambda = sn;
      y = __dmul_rn(ay, d);
      if (fabs(err) < 1e-12) run = false;
    }
  }
  return y;
}

// The same iteration by one thread, for more than RIB_QUADS segments: a quad
// costs the pipe twice as much per segment, which counts once the quads' warps
// fill it (quads against threads at 4096 segments 125 and 222 us, 8192: 188 and
// 222, 16384: 347 and 224, 262144: 5086 and 2521).
constexpr ll RIB_QUADS = 8192;
__device__ void power_serial(double *y, int N, const double *A) {
  const double start[3] = {31.0 / 50.0, 17.0 / 50.0, 43.0 / 50.0};
  double norm = 0.0;
  for (int i = 0; i < N; i++) norm = __dadd_rn(norm, __dmul_rn(start[i], start[i]));
  const double scale = __ddiv_rn(1.0, __dsqrt_rn(norm));
  for (int i = 0; i < N; i++) y[i] = __dmul_rn(start[i], scale);
  double ay[3], lambda = 0.0;
  for (int i = 0; i < 100; i++) {
    norm = 0.0;
    for (int j = 0; j < N; j++) {
      ay[j] = 0.0;
      for (int k = 0; k < N; k++) ay[j] = __dadd_rn(ay[j], __dmul_rn(A[j * N + k], y[k]));
      norm = __dadd_rn(norm, __dmul_rn(ay[j], ay[j]));
    }
    const double sn = __dsqrt_rn(norm);
    const double err = i > 0 ? __ddiv_rn(__dsub_rn(sn, lambda), lambda) : 1.0;
    lambda = sn;
    const double inv = __ddiv_rn(1.0, sn);
    for (int j = 0; j < N; j++) y[j] = __dmul_rn(ay[j], inv);
    if (fabs(err) < 1e-12) break;
  }
}

// RIB axis per segment.  Group segments (p > 1) use the tree sums in
// sums/isums; rank-local segments (p == 1) sum sequentially over their
// elements in order, as get_rib_axis does with c == NULL.
__global__ void k_rib_mean_local(const int *__restrict__ perm,
                                 const double *__restrict__ cent, ll N,
                                 const ll *__restrict__ seg_start,
                                 const ll *__restrict__ seg_n,
                                 const int *__restrict__ p, ll nseg,
                                 int do_local, double *__restrict__ avg) {
  ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  if (!(do_local && p[s] == 1 && seg_n[s] >= 2)) return;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  ll st = seg_start[s], n = seg_n[s];
  for (ll i = 0; i < n; i++) {
    int e = perm[st + i];
    a0 = __dadd_rn(a0, cent[e]);
    a1 = __dadd_rn(a1, cent[N + e]);
    a2 = __dadd_rn(a2, cent[2 * N + e]);
  }
  double dn = (double)n;
  avg[3 * s + 0] = __ddiv_rn(a0, dn);
  avg[3 * s + 1] = __ddiv_rn(a1, dn);
  avg[3 * s + 2] = __ddiv_rn(a2, dn);
}

__global__ void k_rib_mean_group(const double *__restrict__ sums, const int *__restrict__ off,
                                 const ll *__restrict__ seg_n,
                                 const int *__restrict__ p, ll nseg,
                                 double *__restrict__ avg) {
  ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg || p[s] <= 1) return;
  double dn = (double)seg_n[s];
  for (int d = 0; d < 3; d++)  // (the sums of 4, the last one unused)
    avg[3 * s + d] = __ddiv_rn(sums[4 * (off ? (ll)off[s] : s) + d], dn);
}

template <bool QUAD>
__global__ void __launch_bounds__(128)
k_rib_axis(const int *__restrict__ perm, const double *__restrict__ cent, ll N,
           const ll *__restrict__ seg_start, const ll *__restrict__ seg_n,
           const int *__restrict__ p, ll nseg, int ndim, int do_local,
           const double *__restrict__ avg, const double *__restrict__ isums,
           const int *__restrict__ off, double *__restrict__ ev, int *__restrict__ act) {
  const ll s = ((ll)blockIdx.x * blockDim.x + threadIdx.x) >> (QUAD ? 2 : 0);
  const int j = QUAD ? threadIdx.x & 3 : 0;
  const bool in = s < nseg;
  const bool active = in && seg_active(p[in ? s : 0], seg_n[in ? s : 0], do_local);
  if (in && j == 0) act[s] = active;
  double I6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (active) {
    if (p[s] > 1) {
      for (int q = 0; q < 6; q++) I6[q] = isums[6 * (off ? (ll)off[s] : s) + q];
    } else {
      const double *a = avg + 3 * s;
      ll st = seg_start[s], n = seg_n[s];
      for (ll i = 0; i < n; i++) {
        int e = perm[st + i];
        double x = __dsub_rn(cent[e], a[0]), y = __dsub_rn(cent[N + e], a[1]),
               z = __dsub_rn(cent[2 * N + e], a[2]);
        I6[0] = __dadd_rn(I6[0], __dmul_rn(x, x));
        I6[1] = __dadd_rn(I6[1], __dmul_rn(x, y));
        I6[2] = __dadd_rn(I6[2], __dmul_rn(x, z));
        I6[3] = __dadd_rn(I6[3], __dmul_rn(y, y));
        I6[4] = __dadd_rn(I6[4], __dmul_rn(y, z));
        I6[5] = __dadd_rn(I6[5], __dmul_rn(z, z));
      }
    }
  }
  const double I[9] = {I6[0], I6[1], I6[2], I6[1], I6[3], I6[4], I6[2], I6[4], I6[5]};
  if (QUAD) {
    const double y = power_quad(active, ndim, I);
    if (active && j < 3) ev[3 * s + j] = j < ndim ? y : 0.0;
  } else if (active) {
    double y[3] = {0.0, 0.0, 0.0};
    power_serial(y, ndim, I);
    ev[3 * s] = y[0], ev[3 * s + 1] = y[1], ev[3 * s + 2] = ndim == 3 ? y[2] : 0.0;
  }
}

template <int KIND>
__global__ void k_keys(const int *__restrict__ perm, const double *__restrict__ cent,
                       const u32 *__restrict__ rank, ll N, const int *__restrict__ seg_of_pos,
                       const int *__restrict__ axis_or_act,
                       const double *__restrict__ avg,
                       const double *__restrict__ ev, u64 *__restrict__ keys,
                       int *__restrict__ vals) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int s = seg_of_pos[i];
  int e = perm[i];
  u64 k = 0x8000000000000000ull;  // (the key of 0.0: a segment that keeps its order)
  if (KIND == BISECT_RCB) {  // segment id above the dense rank of the coordinate
    int ax = axis_or_act[s];
    k = (u64)(unsigned)s << 32;
    if (ax >= 0) k |= rank[(ll)ax * N + e];
  } else {
    if (axis_or_act[s]) {
      const double *a = avg + 3 * s, *v = ev + 3 * s;
      double x = __dsub_rn(cent[e], a[0]), y = __dsub_rn(cent[N + e], a[1]),
             z = __dsub_rn(cent[2 * N + e], a[2]);
      double key = __dadd_rn(__dadd_rn(__dmul_rn(x, v[0]), __dmul_rn(y, v[1])),
                             __dmul_rn(z, v[2]));
      k = ordered_key(key);
    }
  }
  keys[i] = k;
  vals[i] = e;
}

__global__ void k_child_counts(const int *__restrict__ p, const ll *__restrict__ n,
                               ll nseg, int do_local, int *__restrict__ cnt,
                               int *__restrict__ nactive) {
  ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  int a = seg_active(p[s], n[s], do_local);
  cnt[s] = a ? 2 : 1;
  if (a) atomicAdd(nactive, 1);
}

__global__ void k_children(const ll *__restrict__ st, const ll *__restrict__ n,
                           const int *__restrict__ p, const int *__restrict__ r0,
                           ll nseg, int do_local, const ll *__restrict__ off,
                           ll *__restrict__ st2, ll *__restrict__ n2,
                           int *__restrict__ p2, int *__restrict__ r02) {
  ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  ll o = off[s];
  if (!seg_active(p[s], n[s], do_local)) {
    st2[o] = st[s], n2[o] = n[s], p2[o] = p[s], r02[o] = r0[s];
    return;
  }
  ll L;
  int h, pl, pr;
  if (p[s] > 1) {
    L = lower_count(n[s], p[s]);
    h = (p[s] + 1) / 2;
    pl = h, pr = p[s] - h;
  } else {
    L = n[s] / 2;
    h = 0;
    pl = 1, pr = 1;
  }
  st2[o] = st[s], n2[o] = L, p2[o] = pl, r02[o] = r0[s];
  st2[o + 1] = st[s] + L, n2[o + 1] = n[s] - L, p2[o + 1] = pr, r02[o + 1] = r0[s] + h;
}

__global__ void k_part_from_segs(const int *__restrict__ perm,
                                 const int *__restrict__ seg_of_pos,
                                 const int *__restrict__ r0, ll N,
                                 int *__restrict__ part) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) part[perm[i]] = r0[seg_of_pos[i]];
}

// ---------------------------------------------------------------------------
// Dense coordinate ranks.  RCB only ever compares centroid coordinates along
// one axis and takes min / max for the bounding boxes, so every coordinate
// can be replaced by its dense rank among all centroids on that axis (equal
// values -> equal rank): stable sorts by rank give the same order as stable
// sorts by value, and a box edge is uniq[max rank] - uniq[min rank], the same
// difference of the same two doubles.  Ranks are 32-bit keys (fewer radix
// passes than 64-bit ordered doubles) and are computed once per call.
// ---------------------------------------------------------------------------
__global__ void k_axis_keys(const double *__restrict__ cent, ll N, int a,
                            u64 *__restrict__ keys, int *__restrict__ vals) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  keys[i] = ordered_key(cent[(ll)a * N + i]);
  vals[i] = (int)i;
}

__global__ void k_rank_flags(const u64 *__restrict__ keys, ll N, int *__restrict__ flag) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) flag[i] = (i > 0 && keys[i] != keys[i - 1]) ? 1 : 0;
}

// cnt += positions whose key differs from the one before
__global__ void __launch_bounds__(256)
k_count_changes(const u64 *__restrict__ keys, ll N, unsigned long long *__restrict__ cnt) {
  unsigned c = 0;
  for (ll i = (ll)blockIdx.x * 256 + threadIdx.x; i < N; i += (ll)gridDim.x * 256)
    c += i > 0 && keys[i] != keys[i - 1];
  c = __reduce_add_sync(0xffffffffu, c);
  __shared__ unsigned sh[8];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; w++) t += sh[w];
    atomicAdd(cnt, t);
  }
}

// flag null: every key differs from the one before
__global__ void k_rank_write(const u64 *__restrict__ keys, const int *__restrict__ vals,
                             const int *__restrict__ flag, const ll *__restrict__ excl, ll N,
                             u32 *__restrict__ rank, double *__restrict__ uniq) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  ll r = flag ? excl[i] + flag[i] : i;
  rank[vals[i]] = (u32)r;
  if (i == 0 || !flag || flag[i]) {
    u64 k = keys[i];
    u64 bits = (k >> 63) ? (k ^ 0x8000000000000000ull) : ~k;
    uniq[r] = __longlong_as_double((long long)bits);
  }
}

// ---------------------------------------------------------------------------
// Whole-recursion RCB of one small segment per CTA (n <= SMALL_MAX).
// Every recursion level of the segment runs inside the CTA: the sub-range of
// position x at depth d follows from (n, p) alone (rank split at
// lower_count(len, p) while p > 1, then, with LOCAL, halving at len / 2 as
// rcb_local does, src/rcb.c:39-72).  The dense ranks of the segment's
// elements sit in shared memory for the whole recursion; a thread keeps the
// sub-range of each of its positions in registers and advances it by one
// split per level.  Per level:
//   starts  - the active sub-ranges, appended to a list by the threads that
//             hold their first positions;
//   boxes   - those longer than SMALL_SHORT by warp reductions and shared-
//             memory atomics (table slot start / SMALL_SHORT: long sub-ranges
//             are disjoint and longer than SMALL_SHORT, so their slots
//             differ), the others by their thread of the list;
//   axis    - longest edge, uniq[max] - uniq[min] per axis, by the threads of
//             the list: a warp instruction in FP64 takes 64 cycles for one
//             lane as for 32, so the lanes are filled;
//   order   - stable sort of each sub-range by its axis rank: a bucket per
//             position, by rank and then by position, and an element's new
//             place is the number of elements before it in (rank, position)
//             order inside its bucket.  Where a bucket holds too many, an LSD
//             radix in shared memory over the varying bytes of the rank, then
//             of the sub-range start (__match_any_sync).
// The positions are dealt to the warps in rounds of 32, as many rounds each
// as n asks for.  Bound by the barriers (about ten a level) and the shared-
// memory accesses between them.  3315 elements into 6 parts (three levels):
// 96 -> 43 us; radix passes and 64-bit divisions took most of it before.
// Gives exactly the order of the level-by-level global path.
// ---------------------------------------------------------------------------
constexpr int SMALL_MAX = 8192;
constexpr int SMALL_THREADS = 1024;
constexpr int SMALL_WARPS = SMALL_THREADS / 32;
constexpr int SMALL_ITEMS = SMALL_MAX / SMALL_THREADS;  // positions per thread
constexpr int SMALL_SHORT = 32;   // sequential boxes up to this sub-range length
constexpr int SMALL_NLONG = SMALL_MAX / SMALL_SHORT;  // box table slots
// items of a bucket ranked by counting: 8192 items in buckets of 40 cost what
// the four radix passes do, and the largest bucket is seldom the usual one
constexpr int SMALL_BUCKET = 64;

// lower_count for the small segments (n <= SMALL_MAX).  The quotient comes from
// a single-precision one, which is off by one at most; every position takes
// one per level, and the integer division is three times as long.
__device__ __forceinline__ int lower_count_small(int n, int p) {
  const int h = (int)((unsigned)(p + 1) / 2u);
  int nelt = 0, nrem = n;
  if (p <= n) {
    nelt = (int)__fdividef((float)n, (float)p);
    nrem = n - p * nelt;
    if (nrem < 0) nelt--, nrem += p;
    if (nrem >= p) nelt++, nrem -= p;
  }
  if (nrem == 0) return h * nelt;
  const int s = p - nrem;
  return h * nelt + (h > s ? h - s : 0);
}

// Longest box edge from rank boxes: uniq[max] - uniq[min] per axis, the
// first strictly longest wins.
__device__ __forceinline__ int small_axis(const double *uniq, ll N, int ndim, const u32 *mn,
                                          const u32 *mx) {
  double l[3];
#pragma unroll
  for (int q = 0; q < 3; q++)
    l[q] = q < ndim ? __dsub_rn(uniq[(ll)q * N + mx[q]], uniq[(ll)q * N + mn[q]]) : 0.0;
  int ax = 0;
#pragma unroll
  for (int q = 1; q < 3; q++)
    if (q < ndim && l[q] > l[ax]) ax = q;
  return ax;
}

// Sub-ranges of a thread's positions in the CTA-resident recursions: start |
// length << 16, virtual ranks and the first of them (not tracked for a
// segment with one virtual rank).
template <bool PONE>
struct SmallPos {
  u32 sl[SMALL_ITEMS];
  int p[PONE ? 1 : SMALL_ITEMS], rk[PONE ? 1 : SMALL_ITEMS];
};

// Appends the active sub-ranges that start at one of the warp's positions to
// list (start | length << 16).  Returns bit r for a position of round r in one
// of them; alive: some sub-range is cut again (with more ranks than elements
// it may be a single one, which has nothing to order).
template <bool LOCAL, bool PONE>
__device__ __forceinline__ u32 small_starts(const SmallPos<PONE> &pos, int x0, int R, int n,
                                            u32 *list, int *count, bool *alive) {
  const int lane = threadIdx.x & 31;
  u32 act = 0, first = 0;
  int total = 0;
  *alive = false;
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    if (r >= R) break;
    const int x = x0 + r * 32, ln = (int)(pos.sl[r] >> 16);
    const bool cut = x < n && ((!PONE && pos.p[r] > 1) || (LOCAL && ln >= 2));
    const bool a = cut && ln >= 2;
    *alive = *alive || cut;
    const bool f = a && (int)(pos.sl[r] & 0xFFFFu) == x;
    if (a) act |= 1u << r;
    if (f) first |= 1u << r;
    total += __popc(__ballot_sync(0xffffffffu, f));
  }
  if (!total) return act;
  int at = 0;
  if (lane == 0) at = atomicAdd(count, total);
  at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    if (r >= R) break;
    const bool f = (first >> r) & 1u;
    const u32 b = __ballot_sync(0xffffffffu, f);
    if (f) list[at + __popc(b & ((1u << lane) - 1u))] = pos.sl[r];
    at += __popc(b);
  }
  return act;
}

// Items of the radix passes: local id in bits 0-15, sub-range start in bits
// 16-30, bit 31 set while the sub-range is active.
constexpr u32 ITEM_ACTIVE = 0x80000000u;
__device__ __forceinline__ u32 item_st(u32 it) { return (it >> 16) & 0x7FFFu; }
// axis rank of an item; 0 for inactive sub-ranges (their axis slot is unset)
__device__ __forceinline__ u32 kx_key(const u32 *rk, const unsigned char *sax, u32 it) {
  return (it & ITEM_ACTIVE) ? rk[sax[item_st(it)] * SMALL_MAX + (it & 0xFFFFu)] : 0u;
}

// shared memory of k_rcb_small
struct SmallSmem {
  u32 *rk;               // [3][SMALL_MAX] dense ranks by local id
  u32 *item, *item2;     // local id by position; item2 also: bucket line by start / 2
  u32 *cnt;              // buckets; also wcnt of the radix passes
  u32 *box;              // [SMALL_NLONG][6] min0..2, max0..2
  unsigned short *list;  // positions by bucket; also the start list
  unsigned char *sax;    // axis by sub-range start
};
constexpr size_t small_smem_bytes() {
  return (size_t)SMALL_MAX * (3 * 4 + 4 + 4 + 4 + 2 + 1) + (size_t)SMALL_NLONG * 6 * 4;
}
__device__ __forceinline__ SmallSmem small_carve(u32 *s) {
  SmallSmem m;
  m.rk = s;
  m.item = m.rk + 3 * SMALL_MAX;
  m.item2 = m.item + SMALL_MAX;
  m.cnt = m.item2 + SMALL_MAX;
  m.box = m.cnt + SMALL_MAX;
  m.list = reinterpret_cast<unsigned short *>(m.box + SMALL_NLONG * 6);
  m.sax = reinterpret_cast<unsigned char *>(m.list + SMALL_MAX);
  return m;
}

// Boxes of the long sub-ranges (slot start / SMALL_SHORT of the table).  A
// lane folds its rounds while the warp stays in one sub-range; the warp
// reduces when that changes.
__device__ __forceinline__ void small_boxes(const SmallSmem &m, const u32 *item, const u32 *sl,
                                            u32 act, int x0, int R, int ndim) {
  const int lane = threadIdx.x & 31;
  u32 mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
  int cur = -1;  // start of the sub-range that the lanes fold
  auto flush = [&]() {
    if (cur < 0) return;
    u32 *o = m.box + 6 * (cur / SMALL_SHORT);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      if (q >= ndim) break;
      const u32 a = __reduce_min_sync(0xffffffffu, mn[q]), b = __reduce_max_sync(0xffffffffu, mx[q]);
      if (lane == q) atomicMin(o + q, a), atomicMax(o + 3 + q, b);
      mn[q] = 0xFFFFFFFFu, mx[q] = 0u;
    }
  };
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    if (r >= R) break;
    const bool lng = ((act >> r) & 1u) && (int)(sl[r] >> 16) > SMALL_SHORT;
    const int st = (int)(sl[r] & 0xFFFFu);
    u32 left = __ballot_sync(0xffffffffu, lng);
    if (!left) continue;
    const u32 id = item[x0 + r * 32] & 0xFFFFu;  // (of a long one: below n)
    while (left) {  // usually one sub-range; a boundary makes it two
      const int s = __shfl_sync(0xffffffffu, st, __ffs(left) - 1);
      if (s != cur) flush(), cur = s;
      const bool mine = lng && st == s;
      if (mine)
#pragma unroll
        for (int q = 0; q < 3; q++)
          if (q < ndim) {
            const u32 k = m.rk[q * SMALL_MAX + id];
            mn[q] = min(mn[q], k), mx[q] = max(mx[q], k);
          }
      left &= ~__ballot_sync(0xffffffffu, mine);
    }
  }
  flush();
}

// One level's order by LSD radix passes over the varying bytes of the rank,
// then of the sub-range start; the result ends in item (swapped with item2).
__device__ __forceinline__ void small_radix(const SmallSmem &m, u32 *&item, u32 *&item2,
                                            const u32 *sl, u32 act, int x0, int R, int n) {
  __shared__ unsigned dbase[256];
  __shared__ u32 s_and, s_or, s_stand, s_stor;
  unsigned short *wcnt = reinterpret_cast<unsigned short *>(m.cnt);  // [SMALL_WARPS][256]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  if (threadIdx.x == 0) s_and = 0xFFFFFFFFu, s_or = 0u, s_stand = 0xFFFFFFFFu, s_stor = 0u;
  u32 kand = 0xFFFFFFFFu, kor = 0u, stand = 0xFFFFFFFFu, stor = 0u;
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    const int x = x0 + r * 32;
    if (r >= R || x >= n) break;
    const u32 st = sl[r] & 0xFFFFu;
    const u32 it = (st << 16) | (item[x] & 0xFFFFu) | (((act >> r) & 1u) ? ITEM_ACTIVE : 0u);
    const u32 k = kx_key(m.rk, m.sax, it);
    item[x] = it;
    kand &= k, kor |= k, stand &= st, stor |= st;
  }
  __syncthreads();
  atomicAnd(&s_and, kand);
  atomicOr(&s_or, kor);
  atomicAnd(&s_stand, stand);
  atomicOr(&s_stor, stor);
  __syncthreads();
  const u32 kdiff = s_and ^ s_or, sdiff = s_stand ^ s_stor;
  for (int b = 0; b < 6; b++) {
    const bool is_st = b >= 4;
    const int shift = is_st ? 8 * (b - 4) : 8 * b;
    if ((((is_st ? sdiff : kdiff) >> shift) & 255u) == 0) continue;
    for (int i = threadIdx.x; i < SMALL_WARPS * 256; i += blockDim.x) wcnt[i] = 0;
    __syncthreads();
    unsigned rd[SMALL_ITEMS];  // digit << 16 | rank among the warp's equal digits
    u32 itv[SMALL_ITEMS];
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      rd[r] = 256u << 16, itv[r] = 0;
      if (r >= R) continue;
      const int x = x0 + r * 32;
      unsigned dgt = 256;
      if (x < n) {
        const u32 it = item[x];
        itv[r] = it;
        // inactive positions carry key 0 (their sub-range keeps its order)
        const u32 k = is_st ? item_st(it) : kx_key(m.rk, m.sax, it);
        dgt = (k >> shift) & 255u;
      }
      const unsigned peers = __match_any_sync(0xffffffffu, dgt);
      unsigned before = 0;
      if (dgt < 256) before = wcnt[warp * 256 + dgt];
      __syncwarp();
      if (dgt < 256) {
        rd[r] = (dgt << 16) | (before + __popc(peers & lt_mask));
        if (lane == __ffs(peers) - 1)
          wcnt[warp * 256 + dgt] = (unsigned short)(before + __popc(peers));
      }
      __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < 256) {
      unsigned run = 0;
      for (int w = 0; w < SMALL_WARPS; w++) {
        const unsigned t = wcnt[w * 256 + threadIdx.x];
        wcnt[w * 256 + threadIdx.x] = (unsigned short)run;
        run += t;
      }
      dbase[threadIdx.x] = run;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan of the 256 digit totals
      unsigned v[8], s2 = 0;
      for (int j = 0; j < 8; j++) v[j] = dbase[threadIdx.x * 8 + j], s2 += v[j];
      unsigned incl = s2;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += y;
      }
      unsigned run = incl - s2;
      for (int j = 0; j < 8; j++) dbase[threadIdx.x * 8 + j] = run, run += v[j];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      const unsigned dgr = rd[r] >> 16;
      if (dgr < 256) item2[dbase[dgr] + wcnt[warp * 256 + dgr] + (rd[r] & 0xFFFFu)] = itv[r];
    }
    __syncthreads();
    u32 *t = item;
    item = item2;
    item2 = t;
  }
}

// The level loop; PONE: the segment has one virtual rank (only the local
// halving: no rank counts to track, every part is r0).
template <bool LOCAL, bool PONE>
__device__ __forceinline__ void small_levels(const SmallSmem &m, int *__restrict__ perm,
                                             const double *uniq, ll N, int ndim, ll start, int n,
                                             int p0, int r0, int *__restrict__ part,
                                             int *s_nst) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int R = (n + SMALL_THREADS - 1) / SMALL_THREADS;  // rounds per warp
  const int x0 = warp * R * 32 + lane;                    // first position
  u32 *item = m.item, *item2 = m.item2;
  u32 *starts = reinterpret_cast<u32 *>(m.list);
  SmallPos<PONE> pos;
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    pos.sl[r] = (u32)n << 16;
    if (!PONE) pos.p[r] = p0, pos.rk[r] = 0;
  }
  for (int d = 0; d < 64; d++) {
    if (d > 0) {  // advance every position's sub-range by the previous cut
#pragma unroll
      for (int r = 0; r < SMALL_ITEMS; r++) {
        if (r >= R) break;
        const int x = x0 + r * 32;
        int st = (int)(pos.sl[r] & 0xFFFFu), ln = (int)(pos.sl[r] >> 16);
        const int p = PONE ? 1 : pos.p[r];
        int L, h;
        if (p > 1) {
          L = lower_count_small(ln, p);
          h = (p + 1) / 2;
        } else if (LOCAL && ln >= 2) {
          L = ln / 2;
          h = 0;
        } else {
          continue;  // finished sub-range keeps its place
        }
        const bool up = x >= st + L;
        st += up ? L : 0;
        ln = up ? ln - L : L;
        pos.sl[r] = (u32)st | ((u32)ln << 16);
        if (!PONE && p > 1) pos.p[r] = up ? p - h : h, pos.rk[r] += up ? h : 0;
      }
    }
    bool alive;
    const u32 act = small_starts<LOCAL, PONE>(pos, x0, R, n, starts, &s_nst[d & 1], &alive);
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      if (r >= R) break;
      const int st = (int)(pos.sl[r] & 0xFFFFu);
      if (st == x0 + r * 32 && (int)(pos.sl[r] >> 16) > SMALL_SHORT) {
        u32 *o = m.box + 6 * (st / SMALL_SHORT);
        o[0] = o[1] = o[2] = 0xFFFFFFFFu, o[3] = o[4] = o[5] = 0u;
      }
    }
    if (!__syncthreads_or(alive)) break;
    const int nst = s_nst[d & 1];
    if (threadIdx.x == 0) s_nst[(d + 1) & 1] = 0;
    small_boxes(m, item, pos.sl, act, x0, R, ndim);
    for (int k = threadIdx.x; k < n; k += SMALL_THREADS) m.cnt[k] = 0u;
    __syncthreads();
    // axis, and the line that maps ranks to buckets: first rank and buckets
    // per rank, in item2 (active sub-ranges have two positions or more)
    for (int i = threadIdx.x; i < nst; i += SMALL_THREADS) {
      const int st = (int)(starts[i] & 0xFFFFu), ln = (int)(starts[i] >> 16);
      u32 mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
      if (ln > SMALL_SHORT) {
        const u32 *o = m.box + 6 * (st / SMALL_SHORT);
#pragma unroll
        for (int q = 0; q < 3; q++) mn[q] = o[q], mx[q] = o[3 + q];
      } else {
        for (int y = st; y < st + ln; y++) {
          const u32 id = item[y] & 0xFFFFu;
#pragma unroll
          for (int q = 0; q < 3; q++)
            if (q < ndim) {
              const u32 k = m.rk[q * SMALL_MAX + id];
              mn[q] = min(mn[q], k), mx[q] = max(mx[q], k);
            }
        }
      }
      const int ax = small_axis(uniq, N, ndim, mn, mx);
      m.sax[st] = (unsigned char)ax;
      const u32 lo = ax == 0 ? mn[0] : ax == 1 ? mn[1] : mn[2];
      const u32 hi = ax == 0 ? mx[0] : ax == 1 ? mx[1] : mx[2];
      reinterpret_cast<uint2 *>(item2)[st >> 1] =
          make_uint2(lo, __float_as_uint((float)ln / ((float)(hi - lo) + 1.0f)));
    }
    __syncthreads();
    // bucket of every position: (rank - first + (x - st) / len) x line.  The
    // fraction spreads equal ranks over their buckets; every operation is
    // monotonic and the fraction below one, so (rank, position) order is
    // bucket order
    u32 bk[SMALL_ITEMS];
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      const int x = x0 + r * 32;
      if (r >= R || x >= n) break;
      const int st = (int)(pos.sl[r] & 0xFFFFu), ln = (int)(pos.sl[r] >> 16);
      bk[r] = (u32)x;
      if ((act >> r) & 1u) {
        const u32 k = m.rk[m.sax[st] * SMALL_MAX + (item[x] & 0xFFFFu)];
        const uint2 line = reinterpret_cast<const uint2 *>(item2)[st >> 1];
        const float f = (float)(k - line.x) + __fdividef((float)(x - st), (float)ln);
        bk[r] = (u32)(st + min(ln - 1, (int)(f * __uint_as_float(line.y))));
      }
      atomicAdd(&m.cnt[bk[r]], 1u);
    }
    __syncthreads();
    const u32 big = cta_scan<SMALL_MAX, SMALL_THREADS>(m.cnt, n);
    if (big > SMALL_BUCKET) {
      small_radix(m, item, item2, pos.sl, act, x0, R, n);
      continue;
    }
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      const int x = x0 + r * 32;
      if (r >= R || x >= n) break;
      m.list[atomicAdd(&m.cnt[bk[r]], 1u)] = (unsigned short)x;
    }
    __syncthreads();  // (cnt: now the end of every bucket)
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      const int x = x0 + r * 32;
      if (r >= R || x >= n) break;
      const int b0 = bk[r] ? (int)m.cnt[bk[r] - 1] : 0, b1 = (int)m.cnt[bk[r]];
      const u32 it = item[x] & 0xFFFFu;
      int to = b0;
      if (b1 - b0 > 1) {
        const u32 *rk = m.rk + m.sax[pos.sl[r] & 0xFFFFu] * SMALL_MAX;
        const u32 k = rk[it];
        for (int j = b0; j < b1; j++) {
          const int y = m.list[j];
          const u32 k2 = rk[item[y] & 0xFFFFu];
          to += (k2 < k) || (k2 == k && y < x);
        }
      }
      item2[to] = it;
    }
    __syncthreads();
    u32 *t = item;
    item = item2;
    item2 = t;
  }
  // ---- write the order (and ranks) back: read every old entry, then write
  int ev[SMALL_ITEMS];
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    const int x = x0 + r * 32;
    ev[r] = r < R && x < n ? perm[start + (item[x] & 0xFFFFu)] : 0;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    const int x = x0 + r * 32;
    if (r < R && x < n) {
      perm[start + x] = ev[r];
      if (part) part[ev[r]] = r0 + (PONE ? 0 : pos.rk[r]);
    }
  }
}

// sparse: null, or one segment of all N elements, whose ranks on axis q with
// sparse[q] set are the numbers of elements strictly below (equal coordinates
// leave numbers out); they are made dense first, in uniq too.
template <bool LOCAL>
__global__ void __launch_bounds__(SMALL_THREADS)
k_rcb_small(int *__restrict__ perm, const u32 *__restrict__ rank, double *uniq, ll N, int ndim,
            const ll *__restrict__ seg_start, const ll *__restrict__ seg_n,
            const int *__restrict__ seg_p, const int *__restrict__ seg_r0,
            int *__restrict__ part, const int *__restrict__ sparse) {
  extern __shared__ __align__(16) u32 smem_u32[];
  const SmallSmem m = small_carve(smem_u32);
  __shared__ int s_nst[2];
  const ll sg = blockIdx.x;
  const ll start = seg_start[sg];
  const int n = (int)seg_n[sg], p0 = seg_p[sg], r0 = seg_r0[sg];
  const bool seg_act = p0 > 1 || (LOCAL && p0 == 1 && n >= 2);
  if (n <= 0 || p0 <= 0) return;
  if (!seg_act || n > SMALL_MAX) {
    if (part && n <= SMALL_MAX && p0 == 1)
      for (int x = threadIdx.x; x < n; x += blockDim.x) part[perm[start + x]] = r0;
    return;
  }
  if (threadIdx.x == 0) s_nst[0] = s_nst[1] = 0;
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    const int e = perm[start + x];
    for (int q = 0; q < ndim; q++) m.rk[q * SMALL_MAX + x] = rank[(ll)q * N + e];
    m.item[x] = (u32)x;
  }
  if (sparse) {
    for (int q = 0; q < ndim; q++) {
      if (!sparse[q]) continue;
      __syncthreads();
      u32 *rk = m.rk + q * SMALL_MAX;
      for (int x = threadIdx.x; x < n; x += blockDim.x) m.cnt[x] = 0u;
      __syncthreads();
      double v[SMALL_ITEMS];
#pragma unroll
      for (int r = 0; r < SMALL_ITEMS; r++) {
        const int x = threadIdx.x + r * SMALL_THREADS;
        if (x < n) m.cnt[rk[x]] = 1u, v[r] = uniq[(ll)q * N + rk[x]];
      }
      __syncthreads();
      cta_scan<SMALL_MAX, SMALL_THREADS>(m.cnt, n);
#pragma unroll
      for (int r = 0; r < SMALL_ITEMS; r++) {
        const int x = threadIdx.x + r * SMALL_THREADS;
        if (x < n) rk[x] = m.cnt[rk[x]], uniq[(ll)q * N + rk[x]] = v[r];
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (p0 == 1)
    small_levels<LOCAL, true>(m, perm, uniq, N, ndim, start, n, p0, r0, part, s_nst);
  else
    small_levels<LOCAL, false>(m, perm, uniq, N, ndim, start, n, p0, r0, part, s_nst);
}

// children of every segment; lc: active segments, those with more than one
// rank, the largest active one, the largest of all
__global__ void k_level_counts(const int *__restrict__ p, const ll *__restrict__ n, ll nseg,
                               int do_local, int *__restrict__ cnt, unsigned *__restrict__ lc) {
  const ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned any = s < nseg ? (unsigned)n[s] : 0u;
  const bool a = s < nseg && seg_active(p[s], n[s], do_local);
  if (s < nseg) cnt[s] = a ? 2 : 1;
  const unsigned na = __popc(__ballot_sync(0xffffffffu, a)),
                 ng = __popc(__ballot_sync(0xffffffffu, s < nseg && p[s] > 1));
  const unsigned ma = __reduce_max_sync(0xffffffffu, a ? any : 0u),
                 mn = __reduce_max_sync(0xffffffffu, any);
  if ((threadIdx.x & 31) == 0) {  // one atomic per warp and number
    if (na) atomicAdd(&lc[0], na);
    if (ng) atomicAdd(&lc[1], ng);
    if (ma) atomicMax(&lc[2], ma);
    if (mn) atomicMax(&lc[3], mn);
  }
}

__global__ void k_max_active_n(const int *__restrict__ p, const ll *__restrict__ n, ll nseg,
                               int do_local, unsigned long long *__restrict__ mx) {
  ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s < nseg && seg_active(p[s], n[s], do_local)) atomicMax(mx, (unsigned long long)n[s]);
}

inline int tree_launches(ll maxn) {
  int l = 1;
  for (; maxn > 1024; maxn = (maxn + 1023) / 1024) l++;
  return l;
}

// Sums of V values over every segment with more than one rank, in the
// canonical tree; the sums of segment s are at off[s] V of the returned buffer
// (off null: s V; the tables of k_tree_offsets are for segments of more than
// 1024 items, maxn the largest).  No host wait: the launches cover the largest
// possible number of blocks.
template <int V, int GEN0>
const double *seg_tree_reduce(const int *perm, const double *cent, ll N, SegTable &t,
                              const double *avg, ll maxn, int launches, BisectWs &ws,
                              const int **off_out) {
  cudaStream_t st = ctx().stream;
  const ll nseg = t.count;
  if (maxn <= 1024) {
    *off_out = nullptr;
    ws.red_a.ensure((size_t)nseg * V);
    if (maxn <= 32)
      k_seg_warp<V, GEN0><<<grid_for(nseg * 32, 256), 256, 0, st>>>(
          perm, cent, N, t.start.p, t.n.p, t.p.p, nseg, avg, ws.red_a.p);
    else
      k_seg_block<V, GEN0><<<(unsigned)nseg, (unsigned)((maxn + 31) / 32 * 32), 0, st>>>(
          perm, cent, N, t.start.p, t.n.p, t.p.p, avg, ws.red_a.p);
    CK_LAUNCH();
    return ws.red_a.p;
  }
  DBuf<double> *bufs[2] = {&ws.red_a, &ws.red_b};
  ll items = N;
  for (int l = 0; l < launches; l++) {
    const int *cnt = ws.tree_tab.p + 2 * (ll)l * (nseg + 1), *off = cnt + nseg + 1;
    const ll blocks = std::max<ll>(1, std::min<ll>(items, items / 1024 + nseg));  // at most
    DBuf<double> &out = *bufs[l & 1];
    out.ensure((size_t)blocks * V);
    if (l == 0)
      k_seg_tree<V, GEN0><<<(unsigned)blocks, 1024, 0, st>>>(perm, cent, N, t.start.p, cnt, nseg,
                                                             off, nullptr, nullptr, avg, out.p);
    else
      k_seg_tree<V, GEN_ARRAY><<<(unsigned)blocks, 1024, 0, st>>>(
          perm, cent, N, t.start.p, cnt, nseg, off, bufs[(l - 1) & 1]->p, off - 2 * (nseg + 1),
          avg, out.p);
    CK_LAUNCH();
    items = blocks;
    *off_out = off;
  }
  return bufs[(launches - 1) & 1]->p;
}

}  // namespace

int rcb_small_max() { return SMALL_MAX; }

cudaError_t rcb_small_prepare() {
  cudaError_t e = cudaFuncSetAttribute(k_rcb_small<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)small_smem_bytes());
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_rcb_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)small_smem_bytes());
}

cudaError_t rcb_small_launch(int *perm, const u32 *rank, double *uniq, ll N, int ndim,
                             const ll *seg_start, const ll *seg_n, const int *seg_p,
                             const int *seg_r0, ll nseg, bool local, const int *sparse, int *part,
                             cudaStream_t stream) {
  if (local)
    k_rcb_small<true><<<(unsigned)nseg, SMALL_THREADS, small_smem_bytes(), stream>>>(
        perm, rank, uniq, N, ndim, seg_start, seg_n, seg_p, seg_r0, part, sparse);
  else
    k_rcb_small<false><<<(unsigned)nseg, SMALL_THREADS, small_smem_bytes(), stream>>>(
        perm, rank, uniq, N, ndim, seg_start, seg_n, seg_p, seg_r0, part, sparse);
  return cudaGetLastError();
}

void compute_centroids(const double *xyz, int nel, int nv, double *cent) {
  int ndim = (nv == 8) ? 3 : 2;
  const size_t smem = (size_t)CE_ELEMS * (nv * ndim + 1) * sizeof(double);
  if (xyz && nv == 8)
    k_centroids<8><<<grid_for(nel, CE_ELEMS), CE_ELEMS, smem, ctx().stream>>>(xyz, nel, cent);
  else if (xyz && nv == 4)
    k_centroids<4><<<grid_for(nel, CE_ELEMS), CE_ELEMS, smem, ctx().stream>>>(xyz, nel, cent);
  else
    k_centroids_any<<<grid_for(nel, 256), 256, 0, ctx().stream>>>(xyz, nel, nv, ndim, cent);
  CK_LAUNCH();
}

// ---------------------------------------------------------------------------
// RCB on presorted coordinate lists, used when every axis rank is unique (no
// two centroids share a coordinate on any axis).  Then a stable sort of a
// segment by its axis rank does not depend on the segment's current order,
// so each level needs no sort: every segment keeps, per axis a, the list of
// its elements in increasing rank a (lists[a], in the segment's positions).
// Its box is the ranks of the first and last entry of each list; its cut
// sends the first `split` entries of the cut axis' list to the lower child;
// the other lists are partitioned stably by that side (a segmented prefix
// count, no comparison).  The tree, the cuts and the final order are those
// of the sort-per-level path (the order of a segment that is not cut again
// is its list along the axis of the cut that made it).  A level moves about
// 130 B per element instead of four or five radix passes.
// ---------------------------------------------------------------------------
constexpr int PS_THREADS = 1024, PS_ITEMS = 4, PS_TILE = PS_THREADS * PS_ITEMS;

// per segment: cut axis (-1: not cut at this level) and the lower child's size
__global__ void k_ps_axis(const int *__restrict__ lists, const u32 *__restrict__ rank,
                          const double *__restrict__ uniq, ll N, int ndim,
                          const ll *__restrict__ st, const ll *__restrict__ n,
                          const int *__restrict__ p, ll nseg, int do_local,
                          int *__restrict__ axis, ll *__restrict__ split) {
  const ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  if (!seg_active(p[s], n[s], do_local)) {
    axis[s] = -1;
    split[s] = n[s];
    return;
  }
  double len[3] = {0.0, 0.0, 0.0};
  if (n[s] > 0)
    for (int d = 0; d < ndim; d++) {
      const u32 lo = rank[(ll)d * N + lists[(ll)d * N + st[s]]];
      const u32 hi = rank[(ll)d * N + lists[(ll)d * N + st[s] + n[s] - 1]];
      len[d] = __dsub_rn(uniq[(ll)d * N + hi], uniq[(ll)d * N + lo]);
    }
  int ax = 0;
  for (int d = 1; d < ndim; d++)
    if (len[d] > len[ax]) ax = d;  // strictly longer wins: ties keep the lower axis
  axis[s] = ax;
  split[s] = p[s] > 1 ? lower_count(n[s], p[s]) : n[s] / 2;
}

// The kernels over list positions below take PS_ITEMS rounds of 32 positions
// per warp, the loads of all rounds first: each position is a chain of three
// or four dependent loads, and their latency, not memory, bounded a thread per
// position (8M elements: side 71 -> 52 us, flags 79 -> 59, scatter
// 124 -> 58).

// side of every element of a cut segment: 1 for the upper child (side is zero
// before: half of the scattered stores)
__global__ void __launch_bounds__(256)
k_ps_side(const int *__restrict__ lists, ll N, const int *__restrict__ seg_of_pos,
          const ll *__restrict__ st, const int *__restrict__ axis, const ll *__restrict__ split,
          unsigned char *__restrict__ side) {
  const ll j0 = ((ll)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * PS_ITEMS + (threadIdx.x & 31);
  int s[PS_ITEMS], a[PS_ITEMS], e[PS_ITEMS];
  ll cut[PS_ITEMS];
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) s[r] = j0 + 32 * r < N ? seg_of_pos[j0 + 32 * r] : -1;
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) {
    a[r] = s[r] >= 0 ? axis[s[r]] : -1;
    cut[r] = s[r] >= 0 ? st[s[r]] + split[s[r]] : 0;
  }
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) e[r] = a[r] >= 0 ? lists[(ll)a[r] * N + j0 + 32 * r] : 0;
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++)
    if (a[r] >= 0 && j0 + 32 * r >= cut[r]) side[e[r]] = 1;
}

__device__ __forceinline__ int ps_block_excl(int v, int *total) {
  __shared__ int ws[PS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int t = lane < PS_THREADS / 32 ? ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < PS_THREADS / 32) ws[lane] = t;
  }
  __syncthreads();
  const int excl = (warp ? ws[warp - 1] : 0) + x - v;
  *total = ws[PS_THREADS / 32 - 1];
  __syncthreads();
  return excl;
}

// per tile of PS_TILE positions (PS_TILE / 32 words): the lower-child flags
// of every list as one bit per position (warp ballots; a position of a
// segment that is not cut gets 0), each word's count of lower flags before
// it inside the tile, and the tile's count
constexpr int PS_WORDS = PS_TILE / 32;
__global__ void __launch_bounds__(PS_THREADS)
k_ps_flags(const int *__restrict__ lists, ll N, int ndim, const int *__restrict__ seg_of_pos,
           const int *__restrict__ axis, int own, const unsigned char *__restrict__ side,
           u32 *__restrict__ bits, int *__restrict__ wpre, int *__restrict__ bsum, int nblk) {
  __shared__ int wtot[3][PS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ll nw = (N + 31) >> 5;
  const ll w0 = (ll)blockIdx.x * PS_WORDS + (ll)warp * PS_ITEMS;  // this warp's first word
  int e[3][PS_ITEMS], ax[PS_ITEMS];
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) {
    const ll j = (w0 + r) * 32 + lane;
    ax[r] = j < N ? seg_of_pos[j] : -1;
#pragma unroll
    for (int b = 0; b < 3; b++) e[b][r] = b < ndim && j < N ? lists[(ll)b * N + j] : -1;
  }
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) ax[r] = ax[r] >= 0 ? axis[ax[r]] : -1;
#pragma unroll
  for (int b = 0; b < 3; b++)
#pragma unroll
    for (int r = 0; r < PS_ITEMS; r++) {
      const bool look = e[b][r] >= 0 && ax[r] >= 0 && !(own && ax[r] == b);
      e[b][r] = look ? side[e[b][r]] : 1;  // 0: goes to the lower child
    }
  int pre[3][PS_ITEMS];
#pragma unroll
  for (int b = 0; b < 3; b++) {
    if (b >= ndim) break;
    int c = 0;
#pragma unroll
    for (int r = 0; r < PS_ITEMS; r++) {
      const u32 bal = __ballot_sync(0xffffffffu, e[b][r] == 0);
      if (lane == 0 && w0 + r < nw) bits[(ll)b * nw + w0 + r] = bal;
      pre[b][r] = c;
      c += __popc(bal);
    }
    if (lane == 0) wtot[b][warp] = c;
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < 3; b++) {
    if (b >= ndim) break;
    const int v = wtot[b][lane];  // PS_THREADS / 32 == 32
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const int base = __shfl_sync(0xffffffffu, inc - v, warp);
    if (lane < PS_ITEMS && w0 + lane < nw) {
      int pv = pre[b][0];
#pragma unroll
      for (int r = 1; r < PS_ITEMS; r++)
        if (lane == r) pv = pre[b][r];
      wpre[(ll)b * nw + w0 + lane] = base + pv;
    }
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    if (threadIdx.x == 0) bsum[(ll)b * nblk + blockIdx.x] = total;
  }
}

// per list (blockIdx.x): exclusive scan of its tiles' counts, in place
__global__ void __launch_bounds__(PS_THREADS) k_ps_bscan(int *__restrict__ bsum, int nblk) {
  int *v = bsum + (ll)blockIdx.x * nblk;
  const int per = (nblk + PS_THREADS - 1) / PS_THREADS;
  const int i0 = threadIdx.x * per;
  int c = 0;
  for (int k = 0; k < per; k++)
    if (i0 + k < nblk) c += v[i0 + k];
  int total;
  int run = ps_block_excl(c, &total);
  for (int k = 0; k < per; k++)
    if (i0 + k < nblk) {
      const int x = v[i0 + k];
      v[i0 + k] = run;
      run += x;
    }
}

// stable partition of every cut segment of each list by side, and the
// segment of every position in the children's table (child_off: the first
// child of each segment, the lower one of a cut)
__global__ void __launch_bounds__(256)
k_ps_scatter(const int *__restrict__ lists, ll N, int ndim, const int *__restrict__ seg_of_pos,
             const ll *__restrict__ st, const int *__restrict__ axis, int own,
             const ll *__restrict__ split, const u32 *__restrict__ bits,
             const int *__restrict__ wpre, const int *__restrict__ bsum, int nblk,
             const ll *__restrict__ child_off, int *__restrict__ lists2,
             int *__restrict__ seg_of_pos2) {
  const int lane = threadIdx.x & 31;
  const ll j0 = ((ll)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * PS_ITEMS + lane;
  const ll nw = (N + 31) >> 5;
  int s[PS_ITEMS], e[3][PS_ITEMS], ax[PS_ITEMS], s0[PS_ITEMS], up[PS_ITEMS], child[PS_ITEMS];
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) {
    const ll j = j0 + 32 * r;
    s[r] = j < N ? seg_of_pos[j] : -1;
#pragma unroll
    for (int b = 0; b < 3; b++) e[b][r] = b < ndim && j < N ? lists[(ll)b * N + j] : -1;
  }
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++) {
    const bool in = s[r] >= 0;
    ax[r] = in ? axis[s[r]] : -1;
    s0[r] = in ? (int)st[s[r]] : 0;
    up[r] = in ? s0[r] + (int)split[s[r]] : 0;  // first position of the upper child
    child[r] = in ? (int)child_off[s[r]] : 0;
  }
#pragma unroll
  for (int r = 0; r < PS_ITEMS; r++)
    if (s[r] >= 0)
      seg_of_pos2[j0 + 32 * r] = child[r] + (ax[r] >= 0 && j0 + 32 * r >= up[r] ? 1 : 0);
#pragma unroll
  for (int b = 0; b < 3; b++) {
    if (b >= ndim) break;
    const u32 *bb = bits + (ll)b * nw;
    const int *wp = wpre + (ll)b * nw, *bs = bsum + (ll)b * nblk;
    int dest[PS_ITEMS];
#pragma unroll
    for (int r = 0; r < PS_ITEMS; r++) {
      const int j = (int)(j0 + 32 * r);
      dest[r] = j;
      if (ax[r] >= 0 && !(own && ax[r] == b)) {
        const u32 word = bb[j >> 5];
        // lower entries of the segment before j
        const int c = bs[j / PS_TILE] + wp[j >> 5] + __popc(word & ((1u << lane) - 1u)) -
                      (bs[s0[r] / PS_TILE] + wp[s0[r] >> 5] +
                       __popc(bb[s0[r] >> 5] & ((1u << (s0[r] & 31)) - 1u)));
        dest[r] = (word >> lane & 1u) ? s0[r] + c : up[r] + (j - s0[r] - c);
      }
    }
#pragma unroll
    for (int r = 0; r < PS_ITEMS; r++)
      if (s[r] >= 0) lists2[(ll)b * N + dest[r]] = e[b][r];
  }
}

// the axis whose list orders each child: the cut's axis, or the parent's
__global__ void k_ps_oaxis(const int *__restrict__ axis, const int *__restrict__ oax, ll nseg,
                           const ll *__restrict__ off, int *__restrict__ oax2) {
  const ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  const ll o = off[s];
  if (axis[s] >= 0)
    oax2[o] = oax2[o + 1] = axis[s];
  else
    oax2[o] = oax[s];
}

__global__ void k_ps_seg_keys(const int *__restrict__ sorted, const int *__restrict__ seg_of_elem,
                              ll N, u64 *__restrict__ keys, int *__restrict__ vals) {
  const ll r = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  const int e = sorted[r];
  keys[r] = (u64)(unsigned)seg_of_elem[e];
  vals[r] = e;
}

__global__ void k_ps_seg_of_elem(const int *__restrict__ perm, const int *__restrict__ seg_of_pos,
                                 ll N, int *__restrict__ seg_of_elem) {
  const ll j = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < N) seg_of_elem[perm[j]] = seg_of_pos[j];
}

// The groups of RSB's next level are the halves of this level's (each old
// group becomes one or two consecutive new segments over its own positions),
// so the next call's lists are this call's group lists partitioned stably by
// half.  Per old group: its first child in the new table, whether it has two
// (axis 0, else -1) and the first child's size; `bad` is set when the new
// table does not refine the old one that way.
__global__ void k_inherit_tab(const ll *__restrict__ ost, const ll *__restrict__ on, ll ocount,
                              const ll *__restrict__ nst, const ll *__restrict__ nn,
                              const int *__restrict__ nseg_of_pos, int *__restrict__ axis,
                              ll *__restrict__ split, ll *__restrict__ child_off,
                              int *__restrict__ bad) {
  const ll s = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ocount) return;
  const ll s0 = ost[s], n = on[s];
  axis[s] = -1, split[s] = n, child_off[s] = 0;
  if (n <= 0) return;
  const int c0 = nseg_of_pos[s0], c1 = nseg_of_pos[s0 + n - 1];
  bool ok = nst[c0] == s0 && (c1 == c0 || c1 == c0 + 1) && nst[c1] + nn[c1] == s0 + n;
  if (c1 == c0 + 1) ok = ok && nst[c1] == s0 + nn[c0];
  if (!ok) atomicOr(bad, 1);
  axis[s] = c1 == c0 + 1 ? 0 : -1;
  split[s] = nn[c0];
  child_off[s] = c0;
}

// side of every element in its old group: 1 for the second child
__global__ void k_inherit_side(const int *__restrict__ perm, ll N,
                               const int *__restrict__ oseg_of_pos,
                               const int *__restrict__ nseg_of_pos,
                               const ll *__restrict__ child_off, unsigned char *__restrict__ side) {
  const ll j = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  side[perm[j]] = nseg_of_pos[j] != (int)child_off[oseg_of_pos[j]] ? 1 : 0;
}

__global__ void k_ps_final(const int *__restrict__ lists, ll N, const int *__restrict__ seg_of_pos,
                           const int *__restrict__ oax, int *__restrict__ perm) {
  const ll j = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const int a = oax[seg_of_pos[j]];
  if (a >= 0) perm[j] = lists[(ll)a * N + j];
}

// The remaining levels of every segment of at most SMALL_MAX elements in
// one CTA each, on presorted lists (every rank unique).  An element's local
// id is its place in the segment's axis-0 list at launch; the CTA holds the
// segment's three lists of local ids in shared memory and, per level, for
// every active sub-range (tracked per position in registers as k_rcb_small
// does): its cut axis from the first and last entry of each list, the side
// of each element from the cut axis' list, and a stable partition of every
// list by side.  The partition counts lower flags with one warp ballot per
// 32 positions: the count before a position is the totals of the warps
// before its warp (a shuffle scan), the totals of the rounds before its
// round inside its warp, and the ballot's bits below its lane.  All three
// lists move to three spare buffers in the same pass, so a level takes four
// CTA barriers.  Same tree, same order as the sort-per-level kernels;
// without LOCAL a sub-range that is no longer cut keeps the list of the axis
// that cut it last.
constexpr int SMALL_ROUNDS = SMALL_MAX / 32;  // ballots per list
constexpr size_t pss_smem_bytes() {
  // local id -> element (int); six list buffers and the lower child's size
  // by sub-range start (u16); side and cut axis (u8); the start list (u32 per
  // two positions); per list the ballots (u32) and the in-warp prefix of each
  // round (u16)
  return (size_t)SMALL_MAX * (sizeof(int) + 7 * sizeof(unsigned short) + 2 + 2) +
         (size_t)3 * SMALL_ROUNDS * (sizeof(u32) + sizeof(unsigned short));
}

struct PssSmem {
  int *gl;               // local id -> element
  u32 *bal;              // [3][SMALL_ROUNDS] lower flags, one word per 32 positions
  u32 *starts;           // active sub-ranges: start | length << 16
  unsigned short *buf;   // [6][SMALL_MAX]: three lists and three spares
  unsigned short *spl;   // lower child's size by sub-range start
  unsigned short *wpre;  // [3][SMALL_ROUNDS] lower flags before the round in its warp
  unsigned char *side;   // side by local id
  unsigned char *sax;    // cut axis by sub-range start
};

__device__ __forceinline__ PssSmem pss_carve(unsigned char *s) {
  PssSmem m;
  m.gl = reinterpret_cast<int *>(s);
  m.bal = reinterpret_cast<u32 *>(m.gl + SMALL_MAX);
  m.starts = m.bal + 3 * SMALL_ROUNDS;
  m.buf = reinterpret_cast<unsigned short *>(m.starts + SMALL_MAX / 2);
  m.spl = m.buf + 6 * SMALL_MAX;
  m.wpre = m.spl + SMALL_MAX;
  m.side = reinterpret_cast<unsigned char *>(m.wpre + 3 * SMALL_ROUNDS);
  m.sax = m.side + SMALL_MAX;
  return m;
}

// The level loop of k_rcb_small_ps; PONE: the segment has one virtual rank
// (only the local halving: no rank counts to track, every part is r0).
template <bool LOCAL, bool PONE>
__device__ __forceinline__ void pss_levels(int *__restrict__ perm, const double *__restrict__ cent,
                                           ll N, int ndim, ll start, int n, int p0, int r0,
                                           int *__restrict__ part, const PssSmem &m,
                                           int (*wsum)[SMALL_WARPS], int *s_nst) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const u32 lt = (1u << lane) - 1u;
  const int R = (n + SMALL_THREADS - 1) / SMALL_THREADS;  // rounds per warp
  const int inv_r = (65536 + R - 1) / R;                  // k / R for k < 256: k inv_r >> 16
  const int x0 = warp * R * 32 + lane;                    // first position
  // sub-range and virtual ranks of each own position, and the axis that cut
  // it last
  SmallPos<PONE> pos;
  signed char oax_r[SMALL_ITEMS];
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    pos.sl[r] = (u32)n << 16, oax_r[r] = -1;
    if (!PONE) pos.p[r] = p0, pos.rk[r] = 0;
  }
  int cur = 0;  // the lists are in buffers 3 cur .. 3 cur + 2, the spares in the others
  for (int d = 0; d < 64; d++) {
    if (d > 0) {  // advance every position's sub-range by the previous cut
#pragma unroll
      for (int r = 0; r < SMALL_ITEMS; r++) {
        if (r >= R) break;
        const int x = x0 + r * 32;
        int st = (int)(pos.sl[r] & 0xFFFFu), ln = (int)(pos.sl[r] >> 16);
        const int p = PONE ? 1 : pos.p[r];
        if (x >= n || !(p > 1 || (LOCAL && ln >= 2))) continue;  // no longer cut
        const int L = m.spl[st], h = p > 1 ? (p + 1) / 2 : 0;
        if (ln >= 2) oax_r[r] = (signed char)m.sax[st];
        const bool up = x >= st + L;
        st += up ? L : 0;
        ln = up ? ln - L : L;
        pos.sl[r] = (u32)st | ((u32)ln << 16);
        if (!PONE && p > 1) pos.p[r] = up ? p - h : h, pos.rk[r] += up ? h : 0;
      }
    }
    // the reads of sax and spl above and the previous level's partition are
    // done at the barrier, before the cut axes are written and the lists read
    bool alive;
    const u32 act = small_starts<LOCAL, PONE>(pos, x0, R, n, m.starts, &s_nst[d & 1], &alive);
    if (!__syncthreads_or(alive)) break;
    const int nst = s_nst[d & 1];
    if (threadIdx.x == 0) s_nst[(d + 1) & 1] = 0;
    const unsigned short *Lc = m.buf + 3 * cur * SMALL_MAX;   // current lists
    unsigned short *Ls = m.buf + 3 * (cur ^ 1) * SMALL_MAX;  // spares
    // lower child's size of each active sub-range
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      if (r >= R) break;
      const int st = (int)(pos.sl[r] & 0xFFFFu), ln = (int)(pos.sl[r] >> 16);
      const int p = PONE ? 1 : pos.p[r];
      if (x0 + r * 32 != st || st >= n || !(p > 1 || (LOCAL && ln >= 2))) continue;
      m.spl[st] = (unsigned short)(p > 1 ? lower_count_small(ln, p) : ln / 2);
    }
    // and its cut axis: the coordinates of the first and last entry of each
    // list.  By the threads of the start list: a warp instruction in FP64
    // takes 64 cycles for one lane as for 32 (4096 elements to single ones:
    // 190 -> 137 us, the rest is instruction issue of one SM)
    for (int i = threadIdx.x; i < nst; i += SMALL_THREADS) {
      const int st = (int)(m.starts[i] & 0xFFFFu), ln = (int)(m.starts[i] >> 16);
      double len[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 3; q++) {
        if (q >= ndim) break;
        const unsigned short *Lq = Lc + q * SMALL_MAX;
        const int lo = m.gl[Lq[st]], hi = m.gl[Lq[st + ln - 1]];
        len[q] = __dsub_rn(cent[(ll)q * N + hi], cent[(ll)q * N + lo]);
      }
      int ax = 0;
#pragma unroll
      for (int q = 1; q < 3; q++)
        if (q < ndim && len[q] > len[ax]) ax = q;
      m.sax[st] = (unsigned char)ax;
    }
    __syncthreads();
    // side of every element of a cut sub-range, from the cut axis' list
#pragma unroll
    for (int r = 0; r < SMALL_ITEMS; r++) {
      if (r >= R || !((act >> r) & 1u)) continue;
      const int x = x0 + r * 32;
      const int st = (int)(pos.sl[r] & 0xFFFFu);
      m.side[Lc[m.sax[st] * SMALL_MAX + x]] = (x - st) >= (int)m.spl[st] ? 1 : 0;
    }
    __syncthreads();
    // lower flags of every list: one ballot per round of 32 positions, the
    // in-warp prefix of each round and each warp's total
    for (int q = 0; q < ndim; q++) {
      const unsigned short *Lq = Lc + q * SMALL_MAX;
      int cnt = 0;
#pragma unroll
      for (int r = 0; r < SMALL_ITEMS; r++) {
        if (r >= R) break;
        const int x = x0 + r * 32;
        const bool f = ((act >> r) & 1u) && m.side[Lq[x]] == 0;  // act implies x < n
        const u32 b = __ballot_sync(0xffffffffu, f);
        if (lane == 0) {
          m.bal[q * SMALL_ROUNDS + warp * R + r] = b;
          m.wpre[q * SMALL_ROUNDS + warp * R + r] = (unsigned short)cnt;
        }
        cnt += __popc(b);
      }
      if (lane == 0) wsum[q][warp] = cnt;
    }
    __syncthreads();
    // stable partition of each list by side into its spare buffer; a
    // position outside a cut sub-range keeps its place
    for (int q = 0; q < ndim; q++) {
      const int wv = wsum[q][lane];  // SMALL_WARPS == 32
      int inc = wv;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      const int exc = inc - wv;  // lane w: lower flags of the warps before w
      const int base_x = __shfl_sync(0xffffffffu, exc, warp);
      const unsigned short *Lq = Lc + q * SMALL_MAX;
      unsigned short *Tq = Ls + q * SMALL_MAX;
      const u32 *bq = m.bal + q * SMALL_ROUNDS;
      const unsigned short *wq = m.wpre + q * SMALL_ROUNDS;
#pragma unroll
      for (int r = 0; r < SMALL_ITEMS; r++) {
        if (r >= R) break;
        const int x = x0 + r * 32;
        const bool a = (act >> r) & 1u;
        const int st = a ? (int)(pos.sl[r] & 0xFFFFu) : x;
        const int base_st = __shfl_sync(0xffffffffu, exc, ((st >> 5) * inv_r) >> 16);
        if (x >= n) continue;
        const unsigned short id = Lq[x];
        int dest = x;
        if (a) {
          const int k = warp * R + r, ks = st >> 5;
          const u32 bx = bq[k];
          const int before = (base_x + (int)wq[k] + __popc(bx & lt)) -
                             (base_st + (int)wq[ks] + __popc(bq[ks] & ((1u << (st & 31)) - 1u)));
          dest = ((bx >> lane) & 1u) ? st + before : st + (int)m.spl[st] + (x - st - before);
        }
        Tq[dest] = id;
      }
    }
    cur ^= 1;
  }
  // order: a LOCAL recursion ends in single elements (every list agrees);
  // otherwise each position takes the list of the axis that cut it last
  const unsigned short *Lc = m.buf + 3 * cur * SMALL_MAX;
#pragma unroll
  for (int r = 0; r < SMALL_ITEMS; r++) {
    const int x = x0 + r * 32;
    if (r < R && x < n) {
      const int a = oax_r[r] < 0 ? 0 : oax_r[r];
      const int e = m.gl[Lc[a * SMALL_MAX + x]];
      perm[start + x] = e;
      if (part) part[e] = r0 + (PONE ? 0 : pos.rk[r]);
    }
  }
}

template <bool LOCAL>
__global__ void __launch_bounds__(SMALL_THREADS)
k_rcb_small_ps(int *__restrict__ perm, const int *__restrict__ lists, int *__restrict__ loc,
               const double *__restrict__ cent, ll N, int ndim,
               const ll *__restrict__ seg_start, const ll *__restrict__ seg_n,
               const int *__restrict__ seg_p, const int *__restrict__ seg_r0,
               int *__restrict__ part) {
  extern __shared__ __align__(16) unsigned char pss_smem[];
  const PssSmem m = pss_carve(pss_smem);
  __shared__ int wsum[3][SMALL_WARPS];
  __shared__ int s_nst[2];
  if (threadIdx.x == 0) s_nst[0] = s_nst[1] = 0;
  const ll sg = blockIdx.x;
  const ll start = seg_start[sg];
  const int n = (int)seg_n[sg], p0 = seg_p[sg], r0 = seg_r0[sg];
  if (n <= 0 || p0 <= 0) return;
  const bool seg_act = p0 > 1 || (LOCAL && p0 == 1 && n >= 2);
  if (!seg_act || n > SMALL_MAX) {
    if (part && n <= SMALL_MAX && p0 == 1)
      for (int x = threadIdx.x; x < n; x += blockDim.x) part[perm[start + x]] = r0;
    return;
  }
  const int *gl0 = lists + start;  // local id k -> element gl0[k]
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    const int e = gl0[x];
    loc[e] = x;
    m.gl[x] = e;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    m.buf[x] = (unsigned short)x;
    for (int d = 1; d < ndim; d++)
      m.buf[d * SMALL_MAX + x] = (unsigned short)loc[lists[(ll)d * N + start + x]];
  }
  __syncthreads();
  if (p0 == 1)
    pss_levels<LOCAL, true>(perm, cent, N, ndim, start, n, p0, r0, part, m, wsum, s_nst);
  else
    pss_levels<LOCAL, false>(perm, cent, N, ndim, start, n, p0, r0, part, m, wsum, s_nst);
}

static void rcb_presorted(DBuf<int> &perm, SegTable &t, const double *cent, ll N, int ndim,
                          bool do_local, int *part_of_elem, BisectWs &ws) {
  cudaStream_t st = ctx().stream;
  const ll n3 = (ll)ndim * N;
  ws.lists.ensure((size_t)n3);
  ws.lists2.ensure((size_t)n3);
  ws.side.ensure((size_t)N);
  const int nblk = (int)((N + PS_TILE - 1) / PS_TILE);
  ws.bsum.ensure((size_t)ndim * nblk);
  ws.seg_of_pos2.ensure((size_t)N);
  ws.pbits.ensure((size_t)ndim * ((N + 31) >> 5));
  ws.pwpre.ensure((size_t)ndim * ((N + 31) >> 5));
  // lists of the initial segments: the global rank order of each axis,
  // grouped stably by segment; when the segments are the halves of the
  // previous call's (RSB's next level), that call's lists partitioned by half
  fill_seg_of_pos(t, ws.seg_of_pos.p, N);
  bool built = false;
  if (t.count == 1) {
    CK(cudaMemcpyAsync(ws.lists.p, ws.sorted.p, (size_t)n3 * sizeof(int),
                       cudaMemcpyDeviceToDevice, st));
    built = true;
  } else if (ws.g_ok && ws.g_N == N && ws.g_ndim == ndim && ws.gt.count > 0 &&
             t.count <= 2 * ws.gt.count) {
    const ll oc = ws.gt.count;
    ws.oseg.ensure((size_t)N);
    fill_seg_of_pos(ws.gt, ws.oseg.p, N);
    ws.axis.ensure((size_t)oc);
    ws.split.ensure((size_t)oc);
    ws.child_off.ensure((size_t)oc + 1);
    DBuf<int> bad(1);
    CK(cudaMemsetAsync(bad.p, 0, sizeof(int), st));
    k_inherit_tab<<<grid_for(oc, 256), 256, 0, st>>>(ws.gt.start.p, ws.gt.n.p, oc, t.start.p,
                                                     t.n.p, ws.seg_of_pos.p, ws.axis.p,
                                                     ws.split.p, ws.child_off.p, bad.p);
    CK_LAUNCH();
    int h_bad = 1;
    d2h(&h_bad, bad.p, 1);
    sync();
    if (!h_bad) {
      k_inherit_side<<<grid_for(N, 256), 256, 0, st>>>(perm.p, N, ws.oseg.p, ws.seg_of_pos.p,
                                                       ws.child_off.p, ws.side.p);
      CK_LAUNCH();
      k_ps_flags<<<(unsigned)nblk, PS_THREADS, 0, st>>>(ws.glists.p, N, ndim, ws.oseg.p,
                                                        ws.axis.p, 0, ws.side.p, ws.pbits.p,
                                                        ws.pwpre.p, ws.bsum.p, nblk);
      CK_LAUNCH();
      k_ps_bscan<<<(unsigned)ndim, PS_THREADS, 0, st>>>(ws.bsum.p, nblk);
      CK_LAUNCH();
      k_ps_scatter<<<grid_for(N, 256 * PS_ITEMS), 256, 0, st>>>(
          ws.glists.p, N, ndim, ws.oseg.p, ws.gt.start.p, ws.axis.p, 0, ws.split.p, ws.pbits.p,
          ws.pwpre.p, ws.bsum.p, nblk, ws.child_off.p, ws.lists.p, ws.seg_of_pos2.p);
      CK_LAUNCH();
      built = true;
    }
  }
  if (!built) {
    k_ps_seg_of_elem<<<grid_for(N, 256), 256, 0, st>>>(perm.p, ws.seg_of_pos.p, N,
                                                        ws.seg_of_elem.p);
    CK_LAUNCH();
    for (int a = 0; a < ndim; a++) {
      k_ps_seg_keys<<<grid_for(N, 256), 256, 0, st>>>(ws.sorted.p + (ll)a * N, ws.seg_of_elem.p,
                                                      N, ws.keys.p, ws.vals.p);
      CK_LAUNCH();
      seg_sort_pairs(ws.keys, ws.vals, N, nullptr, 1, ws.sort);
      CK(cudaMemcpyAsync(ws.lists.p + (ll)a * N, ws.vals.p, (size_t)N * sizeof(int),
                         cudaMemcpyDeviceToDevice, st));
    }
  }
  // this call's group lists and table, for the next call's lists
  ws.glists.ensure((size_t)n3);
  CK(cudaMemcpyAsync(ws.glists.p, ws.lists.p, (size_t)n3 * sizeof(int),
                     cudaMemcpyDeviceToDevice, st));
  ws.gt.reserve(t.count);
  CK(cudaMemcpyAsync(ws.gt.start.p, t.start.p, (size_t)t.count * sizeof(ll),
                     cudaMemcpyDeviceToDevice, st));
  CK(cudaMemcpyAsync(ws.gt.n.p, t.n.p, (size_t)t.count * sizeof(ll), cudaMemcpyDeviceToDevice,
                     st));
  ws.gt.count = t.count;
  ws.g_ok = true, ws.g_N = N, ws.g_ndim = ndim;
  ws.oax.ensure((size_t)t.count);
  CK(cudaMemsetAsync(ws.oax.p, 0xFF, (size_t)t.count * sizeof(int), st));  // -1: input order
  DBuf<int> nact_d(1);
  DBuf<unsigned long long> maxn_d(1);
  for (int level = 0; level < 200; level++) {
    const ll nseg = t.count;
    ws.child_cnt.ensure((size_t)nseg);
    CK(cudaMemsetAsync(nact_d.p, 0, sizeof(int), st));
    CK(cudaMemsetAsync(maxn_d.p, 0, sizeof(unsigned long long), st));
    k_child_counts<<<grid_for(nseg, 256), 256, 0, st>>>(t.p.p, t.n.p, nseg, do_local,
                                                        ws.child_cnt.p, nact_d.p);
    CK_LAUNCH();
    k_max_active_n<<<grid_for(nseg, 256), 256, 0, st>>>(t.p.p, t.n.p, nseg, do_local, maxn_d.p);
    CK_LAUNCH();
    int nact = 0;
    unsigned long long maxn = 0;
    d2h(&nact, nact_d.p, 1);
    d2h(&maxn, maxn_d.p, 1);
    sync();
    // (seg_of_pos follows the table: filled before the loop, then written
    // for the children by k_ps_scatter)
    if (nact == 0) break;
    if (maxn <= (unsigned long long)SMALL_MAX) {
      // every remaining level in one CTA per segment, on the segment's lists
      // (k_rcb_small_ps); a segment that is no longer cut takes its list here
      k_ps_final<<<grid_for(N, 256), 256, 0, st>>>(ws.lists.p, N, ws.seg_of_pos.p, ws.oax.p,
                                                    perm.p);
      CK_LAUNCH();
      ws.loc.ensure((size_t)N);
      const size_t smem = pss_smem_bytes();
      if (do_local) {
        ensure_smem_limit(k_rcb_small_ps<true>, (int)smem);
        k_rcb_small_ps<true><<<(unsigned)nseg, SMALL_THREADS, smem, st>>>(
            perm.p, ws.lists.p, ws.loc.p, cent, N, ndim, t.start.p, t.n.p, t.p.p, t.r0.p,
            part_of_elem);
      } else {
        ensure_smem_limit(k_rcb_small_ps<false>, (int)smem);
        k_rcb_small_ps<false><<<(unsigned)nseg, SMALL_THREADS, smem, st>>>(
            perm.p, ws.lists.p, ws.loc.p, cent, N, ndim, t.start.p, t.n.p, t.p.p, t.r0.p,
            part_of_elem);
      }
      CK_LAUNCH();
      return;
    }
    ws.axis.ensure((size_t)nseg);
    ws.split.ensure((size_t)nseg);
    k_ps_axis<<<grid_for(nseg, 256), 256, 0, st>>>(ws.lists.p, ws.rank.p, ws.uniq.p, N, ndim,
                                                   t.start.p, t.n.p, t.p.p, nseg, do_local,
                                                   ws.axis.p, ws.split.p);
    CK_LAUNCH();
    CK(cudaMemsetAsync(ws.side.p, 0, (size_t)N, st));
    k_ps_side<<<grid_for(N, 256 * PS_ITEMS), 256, 0, st>>>(ws.lists.p, N, ws.seg_of_pos.p, t.start.p,
                                                ws.axis.p, ws.split.p, ws.side.p);
    CK_LAUNCH();
    k_ps_flags<<<(unsigned)nblk, PS_THREADS, 0, st>>>(ws.lists.p, N, ndim, ws.seg_of_pos.p,
                                                      ws.axis.p, 1, ws.side.p, ws.pbits.p,
                                                      ws.pwpre.p, ws.bsum.p, nblk);
    CK_LAUNCH();
    k_ps_bscan<<<(unsigned)ndim, PS_THREADS, 0, st>>>(ws.bsum.p, nblk);
    CK_LAUNCH();
    // children (a cut segment has two, the others one)
    ws.child_off.ensure((size_t)nseg + 1);
    exclusive_scan_int_to_ll_async(ws.child_cnt.p, ws.child_off.p, nseg);
    const ll nchild = nseg + nact;
    k_ps_scatter<<<grid_for(N, 256 * PS_ITEMS), 256, 0, st>>>(
        ws.lists.p, N, ndim, ws.seg_of_pos.p, t.start.p, ws.axis.p, 1, ws.split.p, ws.pbits.p,
        ws.pwpre.p, ws.bsum.p, nblk, ws.child_off.p, ws.lists2.p, ws.seg_of_pos2.p);
    CK_LAUNCH();
    std::swap(ws.lists.p, ws.lists2.p);
    std::swap(ws.lists.n, ws.lists2.n);
    std::swap(ws.seg_of_pos.p, ws.seg_of_pos2.p);
    std::swap(ws.seg_of_pos.n, ws.seg_of_pos2.n);
    // the children's table, and the list that orders each of them
    ws.t2.reserve(nchild);
    k_children<<<grid_for(nseg, 256), 256, 0, st>>>(
        t.start.p, t.n.p, t.p.p, t.r0.p, nseg, do_local, ws.child_off.p, ws.t2.start.p,
        ws.t2.n.p, ws.t2.p.p, ws.t2.r0.p);
    CK_LAUNCH();
    ws.oax2.ensure((size_t)nchild);
    k_ps_oaxis<<<grid_for(nseg, 256), 256, 0, st>>>(ws.axis.p, ws.oax.p, nseg, ws.child_off.p,
                                                    ws.oax2.p);
    CK_LAUNCH();
    std::swap(ws.oax.p, ws.oax2.p);
    std::swap(ws.oax.n, ws.oax2.n);
    ws.t2.count = nchild;
    std::swap(t.start, ws.t2.start);
    std::swap(t.n, ws.t2.n);
    std::swap(t.p, ws.t2.p);
    std::swap(t.r0, ws.t2.r0);
    std::swap(t.count, ws.t2.count);
  }
  k_ps_final<<<grid_for(N, 256), 256, 0, st>>>(ws.lists.p, N, ws.seg_of_pos.p, ws.oax.p, perm.p);
  CK_LAUNCH();
  if (part_of_elem) {
    k_part_from_segs<<<grid_for(N, 256), 256, 0, st>>>(perm.p, ws.seg_of_pos.p, t.r0.p, N,
                                                        part_of_elem);
    CK_LAUNCH();
  }
}

void bisect_segments(BisectKind kind, DBuf<int> &perm, SegTable &t,
                     const double *cent, ll N, int ndim, bool do_local,
                     int *part_of_elem, BisectWs &ws) {
  cudaStream_t st = ctx().stream;
  if (N <= 0) return;
  ws.seg_of_pos.ensure((size_t)N);
  ws.seg_of_elem.ensure((size_t)N);
  ws.keys.ensure((size_t)N);
  ws.vals.ensure((size_t)N);
  DBuf<unsigned> lc_d(4);  // k_level_counts
  const size_t small_smem = small_smem_bytes();
  // PARRSB_GPU_LEVEL_LOG=1: per-level times on stderr (synchronises)
  const bool level_log = getenv("PARRSB_GPU_LEVEL_LOG") != nullptr;
  cudaEvent_t lg_e0 = nullptr, lg_e1 = nullptr, lg_part[4] = {};
  float lg_sum[4] = {};  // box + axis, keys, sort, children: summed over levels
  if (level_log) {
    CK(cudaEventCreate(&lg_e0));
    CK(cudaEventCreate(&lg_e1));
    for (auto &e : lg_part) CK(cudaEventCreate(&e));
    CK(cudaEventRecord(lg_e0, st));
  }
  auto lg_mark = [&](int i) {
    if (level_log && kind == BISECT_RCB) CK(cudaEventRecord(lg_part[i], st));
  };
  if (kind == BISECT_RCB && ws.rank_of != cent) {
    // dense ranks of the centroid coordinates, once per set of centroids
    ws.rank.ensure((size_t)3 * N);
    ws.uniq.ensure((size_t)3 * N);
    ws.sorted.ensure((size_t)ndim * N);
    DBuf<int> flag;
    DBuf<ll> excl;
    DBuf<unsigned long long> changes(1);
    ws.unique = true;
    for (int a = 0; a < ndim; a++) {
      k_axis_keys<<<grid_for(N, 256), 256, 0, st>>>(cent, N, a, ws.keys.p, ws.vals.p);
      CK_LAUNCH();
      sort_by_value(ws.keys, ws.vals, N, nullptr, 1, N, ws.sort, true);
      CK(cudaMemsetAsync(changes.p, 0, sizeof(unsigned long long), st));
      k_count_changes<<<std::min(grid_for(N, 256), 152u * 8u), 256, 0, st>>>(ws.keys.p, N,
                                                                            changes.p);
      CK_LAUNCH();
      unsigned long long h_changes = 0;
      d2h(&h_changes, changes.p, 1);
      sync();
      const bool ties = (ll)h_changes != N - 1;  // two centroids share a coordinate
      if (ties) {
        ws.unique = false;
        flag.ensure((size_t)N), excl.ensure((size_t)N);
        k_rank_flags<<<grid_for(N, 256), 256, 0, st>>>(ws.keys.p, N, flag.p);
        CK_LAUNCH();
        exclusive_scan_int_to_ll_async(flag.p, excl.p, N);
      }
      k_rank_write<<<grid_for(N, 256), 256, 0, st>>>(ws.keys.p, ws.vals.p,
                                                      ties ? flag.p : nullptr, excl.p, N,
                                                      ws.rank.p + (ll)a * N,
                                                      ws.uniq.p + (ll)a * N);
      CK_LAUNCH();
      CK(cudaMemcpyAsync(ws.sorted.p + (ll)a * N, ws.vals.p, (size_t)N * sizeof(int),
                         cudaMemcpyDeviceToDevice, st));
    }
    ws.rank_of = cent;
    ws.g_ok = false;  // lists of other centroids
    ws.sort.trim(1ll << 18);  // (with unique ranks nothing more is sorted)
  }
  // PARRSB_GPU_RCB_PRESORT=0: the sort-per-level path even for unique ranks
  if (kind == BISECT_RCB && ws.unique) {
    const char *e = getenv("PARRSB_GPU_RCB_PRESORT");
    if (!(e && atoi(e) == 0)) {
      rcb_presorted(perm, t, cent, N, ndim, do_local, part_of_elem, ws);
      return;
    }
  }
  ws.g_ok = false;  // the next presorted call builds its lists afresh
  for (int level = 0; level < 200; level++) {
    ll nseg = t.count;
    // active segments, their largest size, and children counts
    ws.child_cnt.ensure((size_t)nseg);
    CK(cudaMemsetAsync(lc_d.p, 0, 4 * sizeof(unsigned), st));
    k_level_counts<<<grid_for(nseg, 256), 256, 0, st>>>(t.p.p, t.n.p, nseg, do_local,
                                                        ws.child_cnt.p, lc_d.p);
    CK_LAUNCH();
    unsigned lc[4] = {0, 0, 0, 0};
    d2h(lc, lc_d.p, 4);
    sync();
    const int nact = (int)lc[0], ngroup = (int)lc[1];
    const unsigned long long maxn = lc[2], maxn_any = lc[3];
    if (level_log && kind == BISECT_RCB) {  // time of the global levels so far
      CK(cudaEventRecord(lg_e1, st));
      CK(cudaEventSynchronize(lg_e1));
      float ms = 0.f;
      CK(cudaEventElapsedTime(&ms, lg_e0, lg_e1));
      if (level > 0) {
        float d[4];
        CK(cudaEventElapsedTime(&d[0], lg_e0, lg_part[0]));
        for (int i = 1; i < 4; i++) CK(cudaEventElapsedTime(&d[i], lg_part[i - 1], lg_part[i]));
        for (int i = 0; i < 4; i++) lg_sum[i] += d[i];
      }
      fprintf(stderr, "parrsb_gb300: rcb level %d segments=%lld active=%d max_n=%llu: %.3f ms"
              " (sums box %.2f keys %.2f sort %.2f children %.2f)\n",
              level, (long long)nseg, nact, maxn, ms, lg_sum[0], lg_sum[1], lg_sum[2], lg_sum[3]);
      CK(cudaEventRecord(lg_e0, st));
    }
    if (kind == BISECT_RCB && nact > 0 && maxn <= (unsigned long long)SMALL_MAX) {
      // every remaining level of every segment in one launch
      if (do_local) {
        CK(cudaFuncSetAttribute(k_rcb_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)small_smem));
        k_rcb_small<true><<<(unsigned)nseg, SMALL_THREADS, small_smem, st>>>(
            perm.p, ws.rank.p, ws.uniq.p, N, ndim, t.start.p, t.n.p, t.p.p, t.r0.p,
            part_of_elem, nullptr);
      } else {
        CK(cudaFuncSetAttribute(k_rcb_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)small_smem));
        k_rcb_small<false><<<(unsigned)nseg, SMALL_THREADS, small_smem, st>>>(
            perm.p, ws.rank.p, ws.uniq.p, N, ndim, t.start.p, t.n.p, t.p.p, t.r0.p,
            part_of_elem, nullptr);
      }
      CK_LAUNCH();
      if (level_log) {
        CK(cudaEventRecord(lg_e1, st));
        CK(cudaEventSynchronize(lg_e1));
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, lg_e0, lg_e1));
        fprintf(stderr, "parrsb_gb300: rcb small-segment kernel segments=%lld: %.3f ms\n",
                (long long)nseg, ms);
        cudaEventDestroy(lg_e0);
        cudaEventDestroy(lg_e1);
        for (auto &e : lg_part) cudaEventDestroy(e);
      }
      return;
    }
    if (level_log && kind == BISECT_RCB) CK(cudaEventRecord(lg_e0, st));
    fill_seg_of_pos(t, ws.seg_of_pos.p, N);
    if (nact == 0) break;
    ws.axis.ensure((size_t)nseg);
    if (kind == BISECT_RCB) {
      ws.rbox.ensure((size_t)nseg * 6);
      CK(cudaMemsetAsync(ws.rbox.p, 0xFF, (size_t)nseg * 6 * sizeof(u32), st));
      k_rank_box<<<grid_for(N, RBOX_THREADS * RBOX_ITEMS), RBOX_THREADS, 0, st>>>(
          perm.p, ws.rank.p, N, ndim, ws.seg_of_pos.p, ws.rbox.p);
      CK_LAUNCH();
      k_rcb_axis_rank<<<grid_for(nseg, 256), 256, 0, st>>>(ws.rbox.p, ws.uniq.p, N, t.p.p,
                                                           t.n.p, nseg, ndim, do_local,
                                                           ws.axis.p);
      CK_LAUNCH();
      lg_mark(0);
      k_keys<BISECT_RCB><<<grid_for(N, 256), 256, 0, st>>>(
          perm.p, cent, ws.rank.p, N, ws.seg_of_pos.p, ws.axis.p, nullptr, nullptr, ws.keys.p,
          ws.vals.p);
      CK_LAUNCH();
      lg_mark(1);
    } else {
      DBuf<double> avg((size_t)nseg * 3);
      ws.ev.ensure((size_t)nseg * 3);
      const int *off = nullptr;
      const double *isums = nullptr;
      const int launches = tree_launches((ll)maxn);
      if (ngroup) {
        if (maxn > 1024) {
          ws.tree_tab.ensure((size_t)2 * launches * (nseg + 1));
          k_tree_offsets<<<launches, 1024, 0, st>>>(t.n.p, t.p.p, nseg, launches, ws.tree_tab.p);
          CK_LAUNCH();
        }
        const double *sums = seg_tree_reduce<4, GEN_MEAN>(perm.p, cent, N, t, nullptr, (ll)maxn,
                                                          launches, ws, &off);
        k_rib_mean_group<<<grid_for(nseg, 256), 256, 0, st>>>(sums, off, t.n.p, t.p.p, nseg,
                                                              avg.p);
        CK_LAUNCH();
      }
      if (do_local) {
        k_rib_mean_local<<<grid_for(nseg, 128), 128, 0, st>>>(
            perm.p, cent, N, t.start.p, t.n.p, t.p.p, nseg, 1, avg.p);
        CK_LAUNCH();
      }
      if (ngroup)
        isums = seg_tree_reduce<6, GEN_INERTIA>(perm.p, cent, N, t, avg.p, (ll)maxn, launches, ws,
                                                &off);
      if (nseg <= RIB_QUADS)
        k_rib_axis<true><<<grid_for(4 * nseg, 128), 128, 0, st>>>(
            perm.p, cent, N, t.start.p, t.n.p, t.p.p, nseg, ndim, do_local ? 1 : 0,
            avg.p, isums, off, ws.ev.p, ws.axis.p);
      else
        k_rib_axis<false><<<grid_for(nseg, 128), 128, 0, st>>>(
            perm.p, cent, N, t.start.p, t.n.p, t.p.p, nseg, ndim, do_local ? 1 : 0,
            avg.p, isums, off, ws.ev.p, ws.axis.p);
      CK_LAUNCH();
      k_keys<BISECT_RIB><<<grid_for(N, 256), 256, 0, st>>>(
          perm.p, cent, nullptr, N, ws.seg_of_pos.p, ws.axis.p, avg.p, ws.ev.p, ws.keys.p,
          ws.vals.p);
      CK_LAUNCH();
    }
    // RCB keys carry the segment id above the rank; RIB keys are full doubles
    if (kind == BISECT_RCB)
      seg_sort_pairs(ws.keys, ws.vals, N, nullptr, 1, ws.sort);
    else
      sort_by_value(ws.keys, ws.vals, N, ws.seg_of_pos.p, nseg, (ll)maxn_any, ws.sort);
    lg_mark(2);
    std::swap(perm.p, ws.vals.p);
    std::swap(perm.n, ws.vals.n);
    // children
    ws.child_off.ensure((size_t)nseg + 1);
    exclusive_scan_int_to_ll_async(ws.child_cnt.p, ws.child_off.p, nseg);
    const ll nchild = nseg + nact;
    ws.t2.reserve(nchild);
    k_children<<<grid_for(nseg, 256), 256, 0, st>>>(
        t.start.p, t.n.p, t.p.p, t.r0.p, nseg, do_local, ws.child_off.p, ws.t2.start.p,
        ws.t2.n.p, ws.t2.p.p, ws.t2.r0.p);
    CK_LAUNCH();
    lg_mark(3);
    ws.t2.count = nchild;
    std::swap(t.start, ws.t2.start);
    std::swap(t.n, ws.t2.n);
    std::swap(t.p, ws.t2.p);
    std::swap(t.r0, ws.t2.r0);
    std::swap(t.count, ws.t2.count);
  }
  if (part_of_elem) {
    k_part_from_segs<<<grid_for(N, 256), 256, 0, st>>>(perm.p, ws.seg_of_pos.p, t.r0.p,
                                                        N, part_of_elem);
    CK_LAUNCH();
  }
}

}  // namespace prsb
