// noalloc.cu -- RCB partition of a small mesh without any allocation.
//
// For callers that cannot allocate device memory at the time of the call: a
// caller whose device memory all comes from its own pool or arena, a
// long-running service or solver loop that must not grow or fragment the
// device heap between steps, or code that runs where the runtime may not
// allocate.  Inputs and outputs are the caller's device buffers; every
// intermediate lives in one file-scope __device__ array of fixed size, and
// the kernels run on the caller's stream.
//
// Same result as parrsb_part_mesh with partitioner = 1 (RCB, src/rcb.c:7-137)
// for meshes of at most NA_MAX elements: the same centroids (sequential
// corner sums, then a division by nv; src/parrsb.c:103-166), order-preserving
// coordinate ranks, and the same CTA-per-segment recursion kernel.
#include <mutex>

#include "../../include/parrsb.h"
#include "bisect.cuh"

namespace prsb {
namespace {

constexpr int NA_MAX = 8192;  // elements (the CTA-resident recursion limit)
constexpr int NA_MAXDEV = 64;
constexpr int NA_THREADS = 1024, NA_CROWD = 64;  // k_na_ranks
constexpr int NA_SHARE = NA_THREADS / 4;         // elements that a block ranks
constexpr int NA_RANKS_SMEM = NA_MAX * (8 + 4 + 2 + 4);         // keys, counts, list, values below

constexpr size_t na_round(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t NA_CENT = 0;                                           // double [3][NA_MAX]
constexpr size_t NA_UNIQ = NA_CENT + na_round(3 * NA_MAX * sizeof(double));  // double [3][NA_MAX]
constexpr size_t NA_RANK = NA_UNIQ + na_round(3 * NA_MAX * sizeof(double));  // u32 [3][NA_MAX]
constexpr size_t NA_PERM = NA_RANK + na_round(3 * NA_MAX * sizeof(u32));     // int [NA_MAX]
constexpr size_t NA_SEG = NA_PERM + na_round(NA_MAX * sizeof(int));          // 2 ll + 5 int
constexpr size_t NA_BYTES = NA_SEG + 256;                                    // 524,544 bytes

// Nothing in it needs to start at zero: every word a kernel reads is written
// earlier in the same call (ranks index only written `uniq` slots).
static __device__ __align__(256) unsigned char na_scratch[NA_BYTES];

struct NaDev {
  unsigned char *ptr = nullptr;
  bool ready = false;
};
NaDev na_dev[NA_MAXDEV];
std::mutex na_mu;

__global__ void k_na_ranks(const double *__restrict__ cent, int n, u32 *__restrict__ rank,
                           double *__restrict__ uniq, int *__restrict__ sparse);

// Once per device, with that device current: the scratch address and the
// shared-memory limits of the rank and recursion kernels.
cudaError_t na_setup(int dev, unsigned char **out) {
  std::lock_guard<std::mutex> lk(na_mu);
  if (!na_dev[dev].ready) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, na_scratch);
    if (e != cudaSuccess) return e;
    e = rcb_small_prepare();
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_na_ranks, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             NA_RANKS_SMEM);
    if (e != cudaSuccess) return e;
    na_dev[dev].ptr = static_cast<unsigned char *>(p);
    na_dev[dev].ready = true;
  }
  *out = na_dev[dev].ptr;
  return cudaSuccess;
}

// centroids with the arithmetic of the allocating path, identity order and
// the single segment [0, n) of nparts ranks
__global__ void k_na_init(const double *__restrict__ xyz, int n, int nv, int ndim, int nparts,
                          double *__restrict__ cent, int *__restrict__ perm,
                          ll *__restrict__ seg_ll, int *__restrict__ seg_int) {
  // a thread per element and axis: three times the chains in flight
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) seg_ll[0] = 0, seg_ll[1] = n, seg_int[0] = nparts, seg_int[1] = 0;
  const int e = t / ndim, d = t - e * ndim;
  if (e >= n) return;
  const double *x = xyz + (ll)e * nv * ndim + d;
  double c = 0.0;
  for (int v = 0; v < nv; v++) c = __dadd_rn(c, x[v * ndim]);
  cent[(ll)d * n + e] = __ddiv_rn(c, (double)nv);
  if (d == 0) perm[e] = e;
}

// rank = number of values below on the axis (ties share a rank, the order is
// that of the values); uniq[rank] = the value.  Every block of axis blockIdx.y
// puts all n centroids into buckets, one per element, linear in the value,
// marks one item of every value, and ranks its share of the elements: the
// values of the buckets below, and the smaller ones of its own bucket.  Where
// more than NA_CROWD items with different values share a bucket, marking would
// take too long: the rank is then the number of elements below (sparse[axis]).
// Bound by the latency of about eight barriers; counting against all n values
// took twice as long (31 -> 17 us at 3315 elements).  Four threads rank an
// element, so that values that crowd into few buckets (outliers, graded
// meshes) stay within the cost of that; where one bucket holds most of them,
// against all values in order, which takes a third of the list's instructions
// (8000 elements into 16 parts, one of them far: 0.54 -> 0.21 ms, 0.26 by counting alone).
__global__ void __launch_bounds__(NA_THREADS)
k_na_ranks(const double *__restrict__ cent, int n, u32 *__restrict__ rank,
           double *__restrict__ uniq, int *__restrict__ sparse) {
  extern __shared__ __align__(16) unsigned long long na_keys[];
  u32 *cnt = reinterpret_cast<u32 *>(na_keys + NA_MAX);
  unsigned short *list = reinterpret_cast<unsigned short *>(cnt + NA_MAX);
  u32 *below = reinterpret_cast<u32 *>(list + NA_MAX);  // values before a position of list
  __shared__ unsigned long long s_min, s_max;
  constexpr unsigned short FIRST = 0x8000;  // list: the marked item of a value
  constexpr int PER = NA_MAX / NA_THREADS;
  const int a = blockIdx.y;
  const double *c = cent + (ll)a * n;
  if (threadIdx.x == 0) s_min = ~0ull, s_max = 0ull;
  __syncthreads();
  unsigned long long mn = ~0ull, mx = 0ull;
  for (int j = threadIdx.x; j < n; j += NA_THREADS) {
    const unsigned long long k = ordered_key(c[j]);
    na_keys[j] = k;
    cnt[j] = 0u;
    mn = k < mn ? k : mn, mx = k > mx ? k : mx;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long p = __shfl_xor_sync(0xffffffffu, mn, o);
    const unsigned long long q = __shfl_xor_sync(0xffffffffu, mx, o);
    mn = p < mn ? p : mn, mx = q > mx ? q : mx;
  }
  if ((threadIdx.x & 31) == 0) atomicMin(&s_min, mn), atomicMax(&s_max, mx);
  __syncthreads();
  const int em = max(1, max(key_exp(s_min), key_exp(s_max)));
  const ll f0 = key_fixed(s_min, em);
  const unsigned long long range = (unsigned long long)(key_fixed(s_max, em) - f0);
  const int sh = max(0, 32 - __clzll((ll)range));
  const float line = (float)n / ((float)(u32)(range >> sh) + 1.0f);
  auto bucket = [&](unsigned long long k) {
    const u32 q = (u32)((unsigned long long)(key_fixed(k, em) - f0) >> sh);
    return min(n - 1, (int)((float)q * line));
  };
  int bk[PER];
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int j = threadIdx.x + r * NA_THREADS;
    if (j >= n) break;
    bk[r] = bucket(na_keys[j]);
    atomicAdd(&cnt[bk[r]], 1u);
  }
  __syncthreads();
  cta_scan<NA_MAX, NA_THREADS>(cnt, n);
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int j = threadIdx.x + r * NA_THREADS;
    if (j >= n) break;
    const u32 p = atomicAdd(&cnt[bk[r]], 1u);
    list[p] = (unsigned short)j;
    below[p] = 0u;
    bk[r] |= (int)p << 16;
  }
  __syncthreads();  // (cnt: now the end of every bucket)
  // a bucket is crowded when it is long and some item differs from its first
  bool crowd = false;
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int j = threadIdx.x + r * NA_THREADS;
    if (j >= n) break;
    const int b = bk[r] & 0xFFFF, j0 = b ? (int)cnt[b - 1] : 0, j1 = (int)cnt[b];
    crowd = crowd || (j1 - j0 > NA_CROWD && na_keys[list[j0]] != na_keys[j]);
  }
  const bool dense = !__syncthreads_or(crowd);
  if (blockIdx.x == 0 && threadIdx.x == 0) sparse[a] = !dense;
  if (dense) {
    // marked: no item before it in the list of its bucket holds the same value
    // (a long bucket holds a single value)
    u32 first = 0;
#pragma unroll
    for (int r = 0; r < PER; r++) {
      const int j = threadIdx.x + r * NA_THREADS;
      if (j >= n) break;
      const unsigned long long k = na_keys[j];
      const int b = bk[r] & 0xFFFF, p = bk[r] >> 16;
      bool f = true;
      for (int q = b ? (int)cnt[b - 1] : 0; q < p && f; q++) f = na_keys[list[q]] != k;
      first |= f ? 1u << r : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < PER; r++)
      if ((first >> r) & 1u) {
        const int p = bk[r] >> 16;
        list[p] |= FIRST;
        below[p] = 1u;
      }
    __syncthreads();
    cta_scan<NA_MAX, NA_THREADS>(below, n);
  }
  const int i = blockIdx.x * NA_SHARE + (threadIdx.x >> 2), sub = threadIdx.x & 3;
  const bool in = i < n;
  const unsigned long long k = na_keys[in ? i : 0];
  const int b = bucket(k), j0 = b ? (int)cnt[b - 1] : 0, j1 = (int)cnt[b];
  u32 r = 0;
  if (!in || (dense && j1 - j0 > NA_CROWD)) {
    // nothing to rank, or a single value
  } else if (!dense && 2 * (j1 - j0) > n) {
#pragma unroll 8
    for (int j = sub; j < n; j += 4) r += na_keys[j] < k;
  } else {
    for (int j = j0 + sub; j < j1; j += 4) {
      const unsigned l = list[j];
      r += (!dense || (l & FIRST)) && na_keys[l & ~(unsigned)FIRST] < k;
    }
  }
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  if (!in || sub) return;
  if (dense)
    r += below[j0];
  else if (2 * (j1 - j0) <= n)
    r += (u32)j0;
  rank[(ll)a * n + i] = r;
  const double v = c[i];
  uniq[(ll)a * n + r] = v == 0.0 ? 0.0 : v;  // -0 and +0 share a rank
}

}  // namespace
}  // namespace prsb

using namespace prsb;

extern "C" PARRSB_API int parrsb_part_mesh_rcb_noalloc(int *d_part, const double *d_xyz,
                                                       int nel, int nv, int nparts,
                                                       void *stream) {
  if (nel < 0 || (nel > 0 && (!d_part || !d_xyz)) || (nv != 4 && nv != 8) || nparts < 1)
    return PARRSB_ERR_ARGS;
  if (nel > NA_MAX) return PARRSB_ERR_UNSUPPORTED;  // more than 8192 elements
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NA_MAXDEV) return PARRSB_ERR_CUDA;
  unsigned char *base = nullptr;
  if (na_setup(dev, &base) != cudaSuccess) return PARRSB_ERR_CUDA;
  if (nel == 0) return PARRSB_OK;  // setup only
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int ndim = nv == 8 ? 3 : 2;
  const int P = nparts > nel ? nel : nparts;
  double *cent = reinterpret_cast<double *>(base + NA_CENT);
  double *uniq = reinterpret_cast<double *>(base + NA_UNIQ);
  u32 *rank = reinterpret_cast<u32 *>(base + NA_RANK);
  int *perm = reinterpret_cast<int *>(base + NA_PERM);
  ll *seg_ll = reinterpret_cast<ll *>(base + NA_SEG);
  int *seg_int = reinterpret_cast<int *>(base + NA_SEG + 2 * sizeof(ll));
  k_na_init<<<(nel * ndim + 127) / 128, 128, 0, st>>>(d_xyz, nel, nv, ndim, P, cent, perm, seg_ll,
                                                      seg_int);
  if (cudaGetLastError() != cudaSuccess) return PARRSB_ERR_CUDA;
  if (P == 1) {
    if (cudaMemsetAsync(d_part, 0, (size_t)nel * sizeof(int), st) != cudaSuccess)
      return PARRSB_ERR_CUDA;
    return PARRSB_OK;
  }
  k_na_ranks<<<dim3((nel + NA_SHARE - 1) / NA_SHARE, ndim), NA_THREADS, NA_RANKS_SMEM, st>>>(
      cent, nel, rank, uniq, seg_int + 2);
  if (cudaGetLastError() != cudaSuccess) return PARRSB_ERR_CUDA;
  if (rcb_small_launch(perm, rank, uniq, nel, ndim, seg_ll, seg_ll + 1, seg_int, seg_int + 1, 1,
                       false, seg_int + 2, d_part, st) != cudaSuccess)
    return PARRSB_ERR_CUDA;
  return PARRSB_OK;
}
