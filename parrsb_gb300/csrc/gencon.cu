// gencon.cu -- tolerance-based unique-vertex numbering on the GPU.
//
// Restates parrsb_conn_mesh for one rank (src/con.c:189-295):
//   mesh_init (symmetric corner order, src/con.c:14-50)
//   find_min_neighbor_distance (src/con.c:68-103)
//   find_unique_vertices (src/con-unique-vertices.c:445-505): ndim*ndim
//     passes; each sorts every current segment of points by one coordinate
//     and starts a new segment where (dx_j)^2 > min(dx2_j, dx2_{j-1}) tol^2
//   set_global_id / send_back (src/con.c:108-148)
//   element_check / face_check (src/con-check.c:197-288)
//   compressPeriodicVertices (identity without periodic faces)
// Every segmented sort is stable (the reference's per-segment heapsort,
// src/con-unique-vertices.c:6-58, is replaced by the canonical stable order;
// both give the same ids unless a split decision sits on an exact tie).
#include <cmath>

#include "gencon.cuh"

namespace prsb {

namespace {

__constant__ int c_pre_to_sym[8] = {0, 1, 3, 2, 4, 5, 7, 6};
// faces in symmetric corner order (0-based), src/con-periodic.c:8-10
__constant__ int c_face_mask3[6] = {
    (1 << 0) | (1 << 4) | (1 << 6) | (1 << 2), (1 << 1) | (1 << 3) | (1 << 7) | (1 << 5),
    (1 << 0) | (1 << 1) | (1 << 5) | (1 << 4), (1 << 2) | (1 << 6) | (1 << 7) | (1 << 3),
    (1 << 0) | (1 << 2) | (1 << 3) | (1 << 1), (1 << 4) | (1 << 5) | (1 << 7) | (1 << 6)};

__device__ __forceinline__ double dsq(double a, double b) {
  double t = __dsub_rn(a, b);
  return __dmul_rn(t, t);
}

// not a number, by 32-bit halves (a test of the 64 bits compiles to an FP64
// comparison again)
__device__ __forceinline__ bool nan_bits(double x) {
  return ((unsigned)__double2hiint(x) & 0x7FFFFFFFu) + (__double2loint(x) != 0 ? 1u : 0u) >
         0x7FF00000u;
}
// m < d ? m : d for squares (never negative: their bits order as they do)
// without the FP64 pipe's comparison
__device__ __forceinline__ double min_sq(double m, double d) {
  const bool lt = __double_as_longlong(m) < __double_as_longlong(d);
  return lt && !nan_bits(m) && !nan_bits(d) ? m : d;
}

// Points in symmetric order: coordinates and min squared neighbour distance,
// one 32-byte sector a point (what a later pass gathers comes with one access,
// whichever fields it needs).  A CTA
// stages its elements' corners in shared memory (coalesced loads and stores:
// 0.46 -> 0.20 ms per million hexes) and a thread takes an element: each of
// the 12 edges (4 in 2D) is measured once for its two corners, since the FP64
// pipe bounds the kernel ((a - b)^2 and (b - a)^2 are the same bits).
constexpr int GP_ELEMS = 128;
template <int NDIM>
__global__ void __launch_bounds__(GP_ELEMS)
k_points(const double *__restrict__ coord, ll nel, double4_32a *__restrict__ pt) {
  constexpr int NV = NDIM == 2 ? 4 : 8, ROW = NV * NDIM;
  constexpr int PAD = ROW + 1;  // an element's row in shared memory
  extern __shared__ double gp[];
  const ll e0 = (ll)blockIdx.x * GP_ELEMS;
  const int ne = (int)(nel - e0 < GP_ELEMS ? nel - e0 : GP_ELEMS);
  for (int k = threadIdx.x; k < ne * ROW; k += GP_ELEMS)
    gp[(k / ROW) * PAD + k % ROW] = coord[e0 * ROW + k];
  __syncthreads();
  double m[NV];
  if ((int)threadIdx.x < ne) {
    const double *c = gp + threadIdx.x * PAD;
    double px[NV][NDIM];
#pragma unroll
    for (int k = 0; k < NV; k++) {
      constexpr int sym[8] = {0, 1, 3, 2, 4, 5, 7, 6};
#pragma unroll
      for (int q = 0; q < NDIM; q++) px[k][q] = c[sym[k] * NDIM + q];
      m[k] = 1.7976931348623157e308;
    }
    // edge by edge; a corner meets its neighbours in increasing order
    auto edge = [&](int a, int b) {
      double d = __dadd_rn(dsq(px[a][0], px[b][0]), dsq(px[a][1], px[b][1]));
      if (NDIM == 3) d = __dadd_rn(d, dsq(px[a][NDIM - 1], px[b][NDIM - 1]));
      m[a] = min_sq(m[a], d);
      m[b] = min_sq(m[b], d);
    };
    edge(0, 1), edge(0, 2);
    if (NDIM == 3) edge(0, NV - 4);
    edge(1, 3);
    if (NDIM == 3) edge(1, NV - 3);
    edge(2, 3);
    if (NDIM == 3)
      edge(2, NV - 2), edge(3, NV - 1), edge(NV - 4, NV - 3), edge(NV - 4, NV - 2),
          edge(NV - 3, NV - 1), edge(NV - 2, NV - 1);
  }
  __syncthreads();
  // the distances to shared memory, then whole points in order
  double *sm = gp + GP_ELEMS * PAD;
  if ((int)threadIdx.x < ne)
#pragma unroll
    for (int k = 0; k < NV; k++) sm[threadIdx.x * (NV + 1) + k] = m[k];
  __syncthreads();
  for (int k = threadIdx.x; k < ne * NV; k += GP_ELEMS) {
    const int e = k / NV, v = k % NV;
    const double *c = gp + e * PAD + c_pre_to_sym[v] * NDIM;
    pt[e0 * NV + k] = make_double4_32a(c[0], c[1], NDIM == 3 ? c[NDIM - 1] : 0.0, sm[e * (NV + 1) + v]);
  }
}

// x: coordinate d of the points
__global__ void k_gc_keys(const int *__restrict__ ord, const double *__restrict__ x, ll np,
                          u64 *__restrict__ keys) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < np) keys[i] = ordered_key(x[4 * (ll)ord[i]]);
}

__global__ void k_iota(int *__restrict__ a, ll n) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = (int)i;
}

// |x| to 23 bits, truncated, without the FP64 pipe (a conversion would use it);
// below the normal range 0, above it infinity, not a number as it is
__device__ __forceinline__ float rough(double x) {
  const u32 hi = (u32)__double2hiint(x) & 0x7FFFFFFFu;
  const int e = (int)(hi >> 20) - 896;
  const u32 f = __funnelshift_l((u32)__double2loint(x), hi, 3) - (896u << 23);
  if (nan_bits(x)) return __int_as_float(0x7FC00000);
  return e <= 0 ? 0.0f : e >= 255 ? __int_as_float(0x7F800000) : __int_as_float((int)f);
}
// bounds of a non-negative value from its rough one (an error of 2^-18
// covers the truncations and roundings on both sides)
__device__ __forceinline__ float rough_lo(float f) {
  return f < 1e-30f ? 0.0f : fminf(f, 3.0e38f) * (1.0f - 0x1p-18f);
}
__device__ __forceinline__ float rough_hi(float f) { return fmaxf(f, 1e-30f) * (1.0f + 0x1p-18f); }

struct Tol2 {
  double x;      // tol^2
  float lo, hi;  // around it
};
Tol2 tol2_of(double tol) {
  const double x = tol * tol;
  const float f = (float)x;
  return {x, std::nextafterf(f, -1.0f), std::nextafterf(f, INFINITY)};
}

// whether a gap separates sorted neighbours x, xl with the smallest neighbour
// distances da, db: (x - xl)^2 > min(da, db) tol^2.  In FP64 that is five
// instructions of 64 cycles on a sub-partition's pipe; only the difference is
// taken there, and single precision with error bounds decides unless the two
// sides agree to 2^-17 (settling 8M points: 321 -> 84 us)
__device__ __forceinline__ bool gap_between(double x, double xl, double da, double db,
                                            const Tol2 &tol) {
  const double d = __dsub_rn(x, xl), m = min_sq(da, db);
  const float df = rough(d), q = __fmul_rn(df, df), mf = rough(m);
  if (q == q && mf == mf) {
    if (rough_lo(q) > __fmul_ru(rough_hi(mf), tol.hi)) return true;
    if (rough_hi(q) <= __fmul_rd(rough_lo(mf), tol.lo)) return false;
  }
  return __dmul_rn(d, d) > __dmul_rn(m, tol.x);
}

// flag[j] |= gap between sorted neighbours j-1, j along axis d, which was
// sorted last.  A warp's lane takes its left neighbour's point from the lane
// beside it, so a point is gathered once; and its coordinate along axis next
// goes out as the next sort's key (next >= 0), which saves another gather of
// the same points (65 us per 8M).
__global__ void k_gaps(const int *__restrict__ ord, const double4_32a *__restrict__ pt, ll np,
                       Tol2 tol2, int first_pass, int d, int next, u64 *__restrict__ keys,
                       int *__restrict__ flag) {
  const ll j = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  auto along = [](const double4_32a &p, int q) { return q == 0 ? p.x : q == 1 ? p.y : p.z; };
  double x = 0.0, w = 0.0;
  if (j < np) {
    const double4_32a p = pt[ord[j]];
    x = along(p, d), w = p.w;
    if (next >= 0) keys[j] = ordered_key(along(p, next));
  }
  double xl = __shfl_up_sync(0xffffffffu, x, 1), wl = __shfl_up_sync(0xffffffffu, w, 1);
  if (j >= np) return;
  if (lane == 0 && j > 0) {
    const double4_32a p = pt[ord[j - 1]];
    xl = along(p, d), wl = p.w;
  }
  if (j == 0) {
    flag[0] = 1;
    return;
  }
  const int f = gap_between(x, xl, w, wl, tol2) ? 1 : 0;
  if (first_pass)
    flag[j] = f;
  else if (f)
    flag[j] = 1;
}

// After the first round of sorts: when every two neighbours inside a segment
// are in order along every axis, the later rounds move nothing, and what is
// left of them is the gaps along each axis between neighbours: they enter flag
// here and the rounds are skipped.  (The copies of a vertex usually carry the
// same bits, so its segment is in order along every axis.)  unsettled: some
// pair is out of order; flag2 is then ignored.
__global__ void k_gc_settle(const int *__restrict__ ord, const double4_32a *__restrict__ pt,
                            const int *__restrict__ flag, ll np, int ndim, Tol2 tol2,
                            int *__restrict__ flag2, int *__restrict__ unsettled) {
  const ll j = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  double v[4] = {0.0, 0.0, 0.0, 0.0}, l[4];
  auto load = [&](ll i, double *o) {
    const double4_32a p = pt[ord[i]];
    o[0] = p.x, o[1] = p.y, o[2] = p.z, o[3] = p.w;
  };
  if (j < np) load(j, v);
#pragma unroll
  for (int q = 0; q < 4; q++) l[q] = __shfl_up_sync(0xffffffffu, v[q], 1);
  bool bad = false;
  if (j < np) {
    if (lane == 0 && j > 0) load(j - 1, l);
    int f = flag[j];
    if (!f) {
#pragma unroll
      for (int q = 0; q < 3; q++) {
        if (q >= ndim) break;
        if (ordered_key(l[q]) > ordered_key(v[q])) bad = true;
        // (equal coordinates have no gap unless the distance is not a number)
        if (__double_as_longlong(l[q]) != __double_as_longlong(v[q]) || nan_bits(v[q]))
          if (gap_between(v[q], l[q], v[3], l[3], tol2)) f = 1;
      }
    }
    flag2[j] = f;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) *unsettled = 1;
}

// Segment of every position from the start flags (flag[0] is set): tile sums,
// their scan by one block, and the tiles again.  The segments' starts come
// out with it; the longest one needs them (k_max_len).
constexpr int GS_THREADS = 256, GS_ITEMS = 16, GS_TILE = GS_THREADS * GS_ITEMS;
__device__ __forceinline__ int gs_block_excl(int v, int *total) {
  __shared__ int ws[GS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < GS_THREADS / 32; w++) {
    if (w < warp) before += ws[w];
    all += ws[w];
  }
  __syncthreads();
  *total = all;
  return before + x - v;
}
// the flags of a warp's GS_ITEMS words of 32 positions, and their number
__device__ __forceinline__ int gs_words(const int *__restrict__ flag, ll i0, ll np, u32 *w) {
  int c = 0;
#pragma unroll
  for (int r = 0; r < GS_ITEMS; r++) {
    const ll i = i0 + r * 32 + (threadIdx.x & 31);
    w[r] = __ballot_sync(0xffffffffu, i < np && flag[i] != 0);
    c += __popc(w[r]);
  }
  return c;
}
__global__ void __launch_bounds__(GS_THREADS)
k_gs_sums(const int *__restrict__ flag, ll np, int *__restrict__ bsum) {
  u32 w[GS_ITEMS];
  const ll i0 = (ll)blockIdx.x * GS_TILE + (threadIdx.x >> 5) * (32 * GS_ITEMS);
  const int c = gs_words(flag, i0, np, w);
  int total;
  gs_block_excl((threadIdx.x & 31) == 0 ? c : 0, &total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}
__global__ void __launch_bounds__(GS_THREADS)
k_gs_scan(int *__restrict__ bsum, int nb, int *__restrict__ out) {
  int run = 0;
  for (int b = 0; b < nb; b += GS_THREADS) {
    const int i = b + threadIdx.x;
    const int v = i < nb ? bsum[i] : 0;
    int total;
    const int ex = gs_block_excl(v, &total);
    if (i < nb) bsum[i] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) out[0] = run, out[1] = 0;  // segments; longest one (k_max_len)
}
__global__ void __launch_bounds__(GS_THREADS)
k_gs_write(const int *__restrict__ flag, ll np, const int *__restrict__ bsum,
           int *__restrict__ seg, int *__restrict__ seg_start) {
  u32 w[GS_ITEMS];
  const int lane = threadIdx.x & 31;
  const ll i0 = (ll)blockIdx.x * GS_TILE + (threadIdx.x >> 5) * (32 * GS_ITEMS);
  const int c = gs_words(flag, i0, np, w);
  int total;
  const int before = gs_block_excl(lane == 0 ? c : 0, &total);
  int run = bsum[blockIdx.x] + __shfl_sync(0xffffffffu, before, 0);
#pragma unroll
  for (int r = 0; r < GS_ITEMS; r++) {
    const ll i = i0 + r * 32 + lane;
    const int s = run + __popc(w[r] & (0xFFFFFFFFu >> (31 - lane))) - 1;
    run += __popc(w[r]);
    if (i >= np) continue;
    seg[i] = s;
    if ((w[r] >> lane) & 1u) seg_start[s] = (int)i;
  }
}
__global__ void k_max_len(const int *__restrict__ seg_start, int *__restrict__ nseg_max, ll np) {
  const ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  const int n = nseg_max[0];
  int len = 0;
  if (i < n) len = (int)((i + 1 < n ? seg_start[i + 1] : np) - seg_start[i]);
  len = (int)__reduce_max_sync(0xffffffffu, (unsigned)len);
  if ((threadIdx.x & 31) == 0 && len > nseg_max[1]) atomicMax(&nseg_max[1], len);
}

__global__ void k_ids(const int *__restrict__ ord, const int *__restrict__ seg,
                      ll np, ll *__restrict__ ids, int *__restrict__ ids32) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const int p = ord[i], s = seg[i];
  ids[p] = s;
  ids32[p] = s;
}

__global__ void k_element_check(const int *__restrict__ ids, ll nel, int nv,
                                int *__restrict__ err) {
  ll e = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nel) return;
  int g[8];
  for (int k = 0; k < nv; k++) g[k] = ids[e * nv + k];
  for (int a = 0; a < nv; a++)
    for (int b = a + 1; b < nv; b++)
      if (g[a] == g[b]) {
        atomicOr(err, 1);
        return;
      }
}

// face_check: an element e that contains exactly 3 of the 4 corners of a
// face of element i is an error.  Candidates e are the elements sharing a
// vertex with i (the points of i's vertex segments).  A thread takes a corner
// of i and adds it to the corner sets of the elements around it, in a small
// table of the element's; then its eight threads look at the sets.  Nothing of
// the candidates is read but their numbers: 0.52 -> 0.31 ms per million hexes
// against comparing their ids.  Elements with more neighbours than the table
// has slots compare ids.  Nothing is done when the element check has failed
// (*err): points that ran together make vertices that any number of elements
// share, and the work grows with its square (a call on 8M graded points: 64 -> 7 ms).
constexpr int FC_SLOTS = 64;
__device__ __forceinline__ bool split_face(unsigned mask) {
  bool bad = false;
#pragma unroll
  for (int f = 0; f < 6; f++) bad = bad || __popc(mask & c_face_mask3[f]) == 3;
  return bad;
}
__global__ void __launch_bounds__(256)
k_face_check(const int *__restrict__ ids, const int *__restrict__ ord,
             const int *__restrict__ seg_start, int nseg, ll np, int *__restrict__ err) {
  __shared__ int s_key[32][FC_SLOTS + 1];
  __shared__ unsigned s_mask[32][FC_SLOTS + 1];
  __shared__ int s_failed;
  if (threadIdx.x == 0) s_failed = *(volatile int *)err;
  __syncthreads();
  const ll p = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = threadIdx.x & 7, row = threadIdx.x >> 3;
  const unsigned group = 0xFFu << (threadIdx.x & 24);
  if (p >= np || s_failed) return;  // (whole elements)
  int *key = s_key[row];
  unsigned *mask = s_mask[row];
  for (int u = k; u < FC_SLOTS; u += 8) key[u] = -1, mask[u] = 0u;
  __syncwarp(group);
  const int me = (int)(p >> 3), s = ids[p];
  const int q0 = seg_start[s], q1 = s + 1 < nseg ? seg_start[s + 1] : (int)np;
  bool fits = true;
  for (int q = q0; q < q1 && fits; q++) {
    const int el = ord[q] >> 3;
    if (el == me) continue;  // (holds all four corners of every face)
    int u = (int)(((u32)el * 2654435761u) >> 26), tries = 0;
    for (; tries < FC_SLOTS; tries++, u = (u + 1) & (FC_SLOTS - 1)) {
      const int was = atomicCAS(&key[u], -1, el);
      if (was == -1 || was == el) break;
    }
    fits = tries < FC_SLOTS;
    if (fits) atomicOr(&mask[u], 1u << k);
  }
  __syncwarp(group);
  if (__all_sync(group, fits)) {
    bool bad = false;
    for (int u = k; u < FC_SLOTS; u += 8) {
      const unsigned m = mask[u];
      if (__popc(m) >= 3) bad = bad || split_face(m);
    }
    if (bad) atomicOr(err, 1);
    return;
  }
  // e is examined once, at the lowest corner of i that it contains
  int gi[8];
  for (int u = 0; u < 8; u++) gi[u] = ids[(p & ~7ll) + u];
  for (int q = q0; q < q1; q++) {
    const int el = ord[q] >> 3;
    if (el == me) continue;
    unsigned m = 0;
    for (int v = 0; v < 8; v++) {
      const int g = ids[(ll)el * 8 + v];
      for (int u = 0; u < 8; u++) m |= g == gi[u] ? 1u << u : 0u;
    }
    if ((__ffs(m) - 1) != k) continue;  // seen at a lower corner
    if (split_face(m)) {
      atomicOr(err, 1);
      return;
    }
  }
}

__global__ void k_plus_one(const ll *__restrict__ ids, ll n, long long *__restrict__ out) {
  ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = ids[i] + 1;
}

// segments of the positions from the start flags: seg, seg_start, their
// number and the longest one
void segments_of(GenconWs &ws, const int *flag, ll np, ll *nseg, ll *longest) {
  cudaStream_t st = ctx().stream;
  const int nb = (int)((np + GS_TILE - 1) / GS_TILE);
  ws.bsum.ensure((size_t)nb);
  k_gs_sums<<<nb, GS_THREADS, 0, st>>>(flag, np, ws.bsum.p);
  CK_LAUNCH();
  k_gs_scan<<<1, GS_THREADS, 0, st>>>(ws.bsum.p, nb, ws.nseg_max.p);
  CK_LAUNCH();
  k_gs_write<<<nb, GS_THREADS, 0, st>>>(flag, np, ws.bsum.p, ws.seg.p, ws.seg_start.p);
  CK_LAUNCH();
  k_max_len<<<grid_for(np, 256), 256, 0, st>>>(ws.seg_start.p, ws.nseg_max.p, np);
  CK_LAUNCH();
  int h[2];
  d2h(h, ws.nseg_max.p, 2);
  sync();
  *nseg = h[0], *longest = h[1];
}

}  // namespace

int gencon_device(long long *d_vtx, const double *d_coord, ll nel, int ndim,
                  double tol, GenconWs &ws, ll *nseg_out, ll *d_ids_out) {
  cudaStream_t st = ctx().stream;
  int nv = ndim == 2 ? 4 : 8;
  ll np = nel * nv;
  if (np == 0) {
    if (nseg_out) *nseg_out = 0;
    return PARRSB_OK;
  }
  if (np > 0x7FFFFFFFll) throw ArgError{PARRSB_ERR_UNSUPPORTED, "more than 2^31 corners"};
  ws.pt.ensure((size_t)np);
  ws.keys.ensure((size_t)np);
  ws.ord.ensure((size_t)np);
  ws.flag.ensure((size_t)np);
  ws.seg.ensure((size_t)np);
  ws.seg_start.ensure((size_t)np);
  ws.nseg_max.ensure(2);
  {
    const size_t smem = (size_t)GP_ELEMS * (nv * ndim + 1 + nv + 1) * sizeof(double);
    const unsigned nb = grid_for(nel, GP_ELEMS);
    if (ndim == 2)
      k_points<2><<<nb, GP_ELEMS, smem, st>>>(d_coord, nel, ws.pt.p);
    else
      k_points<3><<<nb, GP_ELEMS, smem, st>>>(d_coord, nel, ws.pt.p);
    CK_LAUNCH();
  }
  k_iota<<<grid_for(np, 256), 256, 0, st>>>(ws.ord.p, np);
  CK_LAUNCH();
  const Tol2 tol2 = tol2_of(tol);
  ll nseg = 1, longest = np;
  DBuf<int> err(2);
  CK(cudaMemsetAsync(err.p, 0, 2 * sizeof(int), st));
  int keys_of = -1;  // axis whose coordinates ws.keys holds, in the current order
  for (int t = 0; t < ndim; t++) {
    if (t == 1) {
      // nothing left to sort: the later rounds' gaps at once
      k_gc_settle<<<grid_for(np, 256), 256, 0, st>>>(ws.ord.p, ws.pt.p, ws.flag.p, np, ndim, tol2,
                                                     ws.flag2(), err.p + 1);
      CK_LAUNCH();
      keys_of = -1;
      int unsettled = 0;
      d2h(&unsettled, err.p + 1, 1);
      sync();
      if (!unsettled) {
        segments_of(ws, ws.flag2(), np, &nseg, &longest);
        break;
      }
    }
    for (int d = 0; d < ndim; d++) {
      const bool first = t == 0 && d == 0;
      if (!first && longest <= 1) continue;  // no two points left to compare
      if (keys_of != d) {
        k_gc_keys<<<grid_for(np, 256), 256, 0, st>>>(
            ws.ord.p, reinterpret_cast<const double *>(ws.pt.p) + d, np, ws.keys.p);
        CK_LAUNCH();
      }
      sort_by_value(ws.keys, ws.ord, np, first ? nullptr : ws.seg.p, nseg, longest, ws.sort, first);
      // (after the first round the points are usually settled)
      keys_of = t == 0 && d == ndim - 1 ? -1 : (d + 1) % ndim;
      k_gaps<<<grid_for(np, 256), 256, 0, st>>>(ws.ord.p, ws.pt.p, np, tol2, first ? 1 : 0, d,
                                                keys_of, ws.keys.p, ws.flag.p);
      CK_LAUNCH();
      segments_of(ws, ws.flag.p, np, &nseg, &longest);
    }
  }
  if (nseg_out) *nseg_out = nseg;
  k_ids<<<grid_for(np, 256), 256, 0, st>>>(ws.ord.p, ws.seg.p, np, ws.ids(), ws.ids32());
  CK_LAUNCH();
  if (d_ids_out)
    CK(cudaMemcpyAsync(d_ids_out, ws.ids(), np * sizeof(ll), cudaMemcpyDeviceToDevice, st));
  {
    StageTimer tm(PARRSB_STAGE_CHECK);
    k_element_check<<<grid_for(nel, 256), 256, 0, st>>>(ws.ids32(), nel, nv, err.p);
    CK_LAUNCH();
    if (ndim == 3) {  // in 2D an edge has two corners: a count of 3 is impossible
      k_face_check<<<grid_for(np, 256), 256, 0, st>>>(ws.ids32(), ws.ord.p, ws.seg_start.p,
                                                      (int)nseg, np, err.p);
      CK_LAUNCH();
    }
    int h_err = 0;
    d2h(&h_err, err.p, 1);
    sync();
    if (h_err) return 1;
  }
  if (d_vtx) {
    k_plus_one<<<grid_for(np, 256), 256, 0, st>>>(ws.ids(), np, d_vtx);
    CK_LAUNCH();
  }
  return PARRSB_OK;
}

}  // namespace prsb
