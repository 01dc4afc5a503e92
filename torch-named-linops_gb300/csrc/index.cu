// Sampling at integer locations (the Sampling linop, NUFFT mode "sampling"):
// a gather (index) and its adjoint, a scatter-add (index_adjoint).
//
// The reference (functional/_index/index.py:17-49,75-100) ravels the D index
// tensors with Python's non-negative modulo (ravel, :187-201), gathers with
// index_select, and scatters with index_add_ (multi_grid, :141-184): float
// atomics on a GPU, so its adjoint is not deterministic there. Here a plan,
// built once per index set, holds the raveled cell of every sample and the
// samples sorted by cell (a stable radix sort, so the samples of a cell stay
// in ascending order) with per-cell offsets. The adjoint is output-stationary:
// each cell sums its samples in ascending sample order starting from zero, the
// order of a sequential index_add_, so it is bit-identical to the reference's
// CPU path and to itself run to run. No atomics touch the values.

#include <algorithm>
#include <string>
#include <type_traits>

#include "common.cuh"

namespace tlgb {
namespace {

struct IdxGeo {
  int ndim;
  int64_t size[TLGB_INDEX_MAX_DIM];
  int64_t stride[TLGB_INDEX_MAX_DIM];  // row-major cell strides
  int64_t ncells, npts, nbatch;
};

// Plan layout: flat[npts] int32 | perm[npts] int32 | off[ncells + 1] uint32
struct IdxLayout {
  int64_t off_flat, off_perm, off_cells, bytes;
  int64_t t_keys, t_keys2, t_vals2, t_counts, t_cnt, t_scan, t_bad, t_bytes;
};

// cell of sample m (Python modulo per dim, as the reference's ravel); the
// lowest out-of-range dim (index >= size or < -size, the reference's
// IndexError) is recorded in *bad
__global__ void index_ravel_kernel(IdxGeo g, const int64_t* __restrict__ idx, int32_t* __restrict__ flat,
                                   uint32_t* __restrict__ keys, int32_t* __restrict__ vals, uint32_t* __restrict__ cnt,
                                   int* __restrict__ bad) {
  for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < g.npts; m += (int64_t)gridDim.x * blockDim.x) {
    int64_t c = 0;
    int worst = TLGB_INDEX_MAX_DIM;
    for (int d = 0; d < g.ndim; ++d) {
      const int64_t i = idx[(int64_t)d * g.npts + m];
      const int64_t s = g.size[d];
      if (i >= s || i < -s) worst = min(worst, d);
      int64_t r = i % s;
      if (r < 0) r += s;
      c += r * g.stride[d];
    }
    if (worst < TLGB_INDEX_MAX_DIM) {
      atomicMin(bad, worst);
      c = 0;  // keeps the plan in range; the build reports the error
    }
    flat[m] = (int32_t)c;
    keys[m] = (uint32_t)c;
    vals[m] = (int32_t)m;
    atomicAdd(cnt + c, 1u);  // integer counts: the same totals in any order
  }
}

// out[b][m] = vals[b][flat[m]]: a copy of E-sized elements. Bound by the
// scattered reads, of which each moves a 32-byte sector: the entries go one
// after the other over blockIdx.y, so that one entry's grid is read at a time
// and stays in L2 (33 MB of 160^3 complex64; all 8 entries at once are 262 MB),
// and a thread has S reads in flight. The output is stored to leave L2 early. 8 entries of 160^3 at 2^20 samples:
// 79 us with one read in flight and the entries in the inner loop, 48 us now.
template <typename E, int S>
__global__ void __launch_bounds__(256) index_fwd_kernel(const E* __restrict__ vals, const int32_t* __restrict__ flat,
                                                        E* __restrict__ out, int64_t npts, int64_t ncells, int64_t nbatch) {
  const int64_t m0 = (int64_t)blockIdx.x * (256 * S) + threadIdx.x;
  int32_t c[S];
#pragma unroll
  for (int i = 0; i < S; ++i) c[i] = m0 + i * 256 < npts ? flat[m0 + i * 256] : 0;  // cell 0 is always there
  for (int64_t b = blockIdx.y; b < nbatch; b += gridDim.y) {
    E v[S];
#pragma unroll
    for (int i = 0; i < S; ++i) v[i] = vals[b * ncells + c[i]];
#pragma unroll
    for (int i = 0; i < S; ++i)
      if (m0 + i * 256 < npts) __stcs(&out[b * npts + m0 + i * 256], v[i]);
  }
}

template <typename E>
void launch_index_fwd(const IdxGeo& g, const void* vals, const int32_t* flat, void* out, cudaStream_t s) {
  constexpr int S = 8;
  const unsigned gy = (unsigned)std::min<int64_t>(g.nbatch, 65535);
  // eight reads in flight where that leaves four CTAs per SM, one (and eight times the CTAs) below
  if (cdiv(g.npts, 256 * S) * g.nbatch >= 4ll * sm_count())
    index_fwd_kernel<E, S><<<dim3((unsigned)cdiv(g.npts, 256 * S), gy), 256, 0, s>>>((const E*)vals, flat, (E*)out, g.npts,
                                                                                   g.ncells, g.nbatch);
  else
    index_fwd_kernel<E, 1><<<dim3((unsigned)cdiv(g.npts, 256), gy), 256, 0, s>>>((const E*)vals, flat, (E*)out, g.npts,
                                                                                g.ncells, g.nbatch);
}

template <typename T>
struct Acc {
  T v;
  __device__ Acc() : v(T(0)) {}
  __device__ void add(const T& x) { v = v + x; }
};
template <>
struct Acc<float2> {
  float2 v;
  __device__ Acc() : v(make_float2(0.f, 0.f)) {}
  __device__ void add(const float2& x) {
    v.x = v.x + x.x;
    v.y = v.y + x.y;
  }
};
template <>
struct Acc<double2> {
  double2 v;
  __device__ Acc() : v(make_double2(0.0, 0.0)) {}
  __device__ void add(const double2& x) {
    v.x = v.x + x.x;
    v.y = v.y + x.y;
  }
};

// out[b][c] = sum over the samples of cell c, in ascending sample order,
// starting from zero; every cell is written. A thread that follows its cells'
// bounds, sample numbers and values itself is bound by that chain of three
// loads, most of them by lanes whose neighbours have nothing to do (a cell
// holds a quarter sample on average in the case below). The samples of a run of cells are a
// run of perm, though, so a CTA fetches the values of its 256 C cells in sorted
// order into shared memory with all lanes, U entries at a time, and each thread
// then adds its own cells' values from there, in the same order as before.
// Results are stored to leave L2 early: the values, which are read in random
// order, stay there. 8 entries of 160^3 at 2^20 samples: 156 us as a chain of
// single loads, 143 with eight entries per chain, 104 us now.
constexpr int kAdjChunk = 256;  // samples in shared memory
// Resident CTAs, by registers: 104 us with 4, 124 and 143 with 5 and 6, which spill
constexpr int adj_ctas(size_t bytes, int entries) { return entries == 1 ? (bytes > 8 ? 4 : 8) : (bytes > 8 ? 3 : 4); }

// One cell's samples, a run of perm, in order; K values are read ahead of adding
// them. Whole groups of K go without checks, which kept the loads from overlapping
// (2^22 samples in 512 cells of 160^3: 2.3 ms, 1.4 without).
template <typename T, int K>
__device__ __forceinline__ T cell_sum(const T* __restrict__ vb, const int32_t* __restrict__ perm, uint32_t k0, uint32_t k1) {
  Acc<T> a;
  T v[K];
  uint32_t k = k0;
  for (; k1 - k >= K; k += K) {  // whole groups: nothing to check between the loads
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = vb[perm[k + i]];
#pragma unroll
    for (int i = 0; i < K; ++i) a.add(v[i]);
  }
  if (k < k1) {
#pragma unroll
    for (int i = 0; i < K - 1; ++i)
      if (k + i < k1) v[i] = vb[perm[k + i]];
#pragma unroll
    for (int i = 0; i < K - 1; ++i)
      if (k + i < k1) a.add(v[i]);
  }
  return a.v;
}

// The cells [first, last) of a CTA where samples crowd into few of
// them, as around a trajectory's centre: light cells by their own threads, and the
// crowded ones, when they are at most kCrowdPerWarp for each warp, by a warp each.
// Its lanes fetch 64 samples' values of U entries ahead, and lane u adds entry u's
// from shared memory, 32 at a time, in order: 15 cycles a sample against 200 of a
// thread's chain, which is why more crowded cells than that are left to their
// threads. 2^21 samples in 512 cells of 160^3, 2 entries: 0.94 ms (12.3 ms when the
// staged chunks of such a run were added by one lane after the other, 3.1 ms as
// chains of single loads).
constexpr uint32_t kCrowded = 256;  // samples
constexpr int kCrowdPerWarp = 12;
template <typename T, int U>
struct CrowdShared {
  T v[8][U][33];
  int list[kCrowdPerWarp * 8];
  int n;
};

template <typename T, int U>
__device__ __noinline__ void crowded_cells(const T* __restrict__ vals, const int32_t* __restrict__ perm,
                                           const uint32_t* __restrict__ off, T* __restrict__ out, int64_t npts, int64_t ncells,
                                           int64_t nbatch, int64_t first, int64_t last, CrowdShared<T, U>& sm) {
  constexpr int NT = 256, W = 8;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) sm.n = 0;
  __syncthreads();
  for (int64_t c = first + tid; c < last; c += NT)
    if (off[c + 1] - off[c] > kCrowded) {  // in any order: a cell's sum is its own
      const int i = atomicAdd(&sm.n, 1);
      if (i < kCrowdPerWarp * W) sm.list[i] = (int)(c - first);
    }
  __syncthreads();
  const int n = sm.n <= kCrowdPerWarp * W ? sm.n : 0;
  const uint32_t light = n > 0 ? kCrowded : 0xffffffffu;
  for (int64_t b = (int64_t)blockIdx.y * U; b < nbatch; b += (int64_t)gridDim.y * U) {
    for (int64_t e = b; e < min(nbatch, b + U); ++e)
#pragma unroll 1
      for (int64_t c = first + tid; c < last; c += NT)
        if (off[c + 1] - off[c] <= light) __stcs(&out[e * ncells + c], cell_sum<T, 8>(vals + e * npts, perm, off[c], off[c + 1]));
    for (int i = warp; i < n; i += W) {
      const int64_t c = first + sm.list[i];
      const uint32_t k0 = off[c], k1 = off[c + 1];
      T v[2][U];
      auto fetch = [&](T (&d)[U], uint32_t k) {
        if (k + lane >= k1) return;
        const int64_t m = perm[k + lane];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (b + u < nbatch) d[u] = vals[(b + u) * npts + m];
      };
      Acc<T> a;  // of entry b + lane
      fetch(v[0], k0);
      fetch(v[1], k0 + 32);
      for (uint32_t k = k0; k < k1; k += 64)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (k + 32 * q >= k1) break;
          __syncwarp();  // the 32 before have been added
#pragma unroll
          for (int u = 0; u < U; ++u) sm.v[warp][u][lane] = v[q][u];
          __syncwarp();
          if (k1 - k > 64 + 32 * q) fetch(v[q], k + 64 + 32 * q);
          if (lane < U) {
            const T* r = sm.v[warp][lane];
            const uint32_t len = k1 - k - 32 * q;
            if (len >= 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j) a.add(r[j]);
            } else {
              for (uint32_t j = 0; j < len; ++j) a.add(r[j]);
            }
          }
        }
      if (lane < U && b + lane < nbatch) __stcs(&out[(b + lane) * ncells + c], a.v);
    }
  }
}

template <typename T, int U, int C>
__global__ void __launch_bounds__(256, adj_ctas(sizeof(T), U)) index_adj_kernel(const T* __restrict__ vals, const int32_t* __restrict__ perm,
                                                        const uint32_t* __restrict__ off, T* __restrict__ out, int64_t npts,
                                                        int64_t ncells, int64_t nbatch) {
  __shared__ union Shared {
    T chunk[U][kAdjChunk];
    CrowdShared<T, U> crowd;
    __device__ Shared() {}
  } shared;
  T(&sm)[U][kAdjChunk] = shared.chunk;
  const int64_t first = (int64_t)blockIdx.x * (256 * C), c0 = first + threadIdx.x;
  const uint32_t ka = off[first], kb = off[min(first + 256 * C, ncells)];
  if (kb - ka > 2 * 256 * C) {
    crowded_cells<T, U>(vals, perm, off, out, npts, ncells, nbatch, first, min(first + 256 * C, ncells), shared.crowd);
    return;
  }
  uint32_t k0[C], k1[C];
#pragma unroll
  for (int j = 0; j < C; ++j) {
    const int64_t c = min(c0 + j * 256, ncells - 1);
    k0[j] = off[c];
    k1[j] = off[c + 1];
  }
  for (int64_t b = (int64_t)blockIdx.y * U; b < nbatch; b += (int64_t)gridDim.y * U) {
    Acc<T> a[U][C];
    for (uint32_t s0 = ka; s0 < kb; s0 += kAdjChunk) {
      const uint32_t n = min(kb - s0, (uint32_t)kAdjChunk);
      __syncthreads();  // the chunk before has been added
      if (threadIdx.x < n) {
        const int64_t m = perm[s0 + threadIdx.x];
        T v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (b + u < nbatch) v[u] = vals[(b + u) * npts + m];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (b + u < nbatch) sm[u][threadIdx.x] = v[u];
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < C; ++j) {
        const uint32_t hi = min(k1[j], s0 + n);
        for (uint32_t k = max(k0[j], s0); k < hi; ++k)
#pragma unroll
          for (int u = 0; u < U; ++u) a[u][j].add(sm[u][k - s0]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < C; ++j)
        if (b + u < nbatch && c0 + j * 256 < ncells) __stcs(&out[(b + u) * ncells + c0 + j * 256], a[u][j].v);
  }
}

// The same on grids whose cells hold several samples, a cell per thread with K
// values read ahead. The line is at one sample per cell: 2^22 complex64 samples on
// 160^3 take 71 us for 2 entries and 262 for 8 (through shared memory 91 and 384).
// K is 4, and 8 from two samples per cell on (complex64: from four): 8 entries at
// 2^23 samples 308 us with 8 and 316 with 4 (float32), 369 and 399 (int64), 463 and
// 398 (complex64). 20 entries of 320^2 at 2^20 samples: 89 us.
// 16-byte values, which fill the shared memory and the registers, cross over at a
// quarter sample and prefer K = 2: 2 entries of 160^3 at 2^20, 2^21 and 2^22 samples
// 82, 110 and 165 us, 4 entries a CTA through shared memory 149, 233 and 432, one
// value at a time 97, 129 and 197.
template <typename T, int K>
__global__ void __launch_bounds__(256) index_adj_dense_kernel(const T* __restrict__ vals, const int32_t* __restrict__ perm,
                                                              const uint32_t* __restrict__ off, T* __restrict__ out,
                                                              int64_t npts, int64_t ncells, int64_t nbatch) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const uint32_t k0 = off[c], k1 = off[c + 1];
  for (int64_t b = blockIdx.y; b < nbatch; b += gridDim.y) {
    out[b * ncells + c] = cell_sum<T, K>(vals + b * npts, perm, k0, k1);
  }
}

template <typename T, int U, int C>
void launch_index_adj_at(const IdxGeo& g, const void* vals, const int32_t* perm, const uint32_t* off, void* out,
                         cudaStream_t s) {
  const dim3 grd((unsigned)cdiv(g.ncells, 256 * C), (unsigned)std::min<int64_t>(cdiv(g.nbatch, U), 65535));
  index_adj_kernel<T, U, C><<<grd, 256, 0, s>>>((const T*)vals, perm, off, (T*)out, g.npts, g.ncells, g.nbatch);
}
template <typename T, int K>
void launch_index_adj_dense(const IdxGeo& g, const void* vals, const int32_t* perm, const uint32_t* off, void* out,
                            cudaStream_t s) {
  const dim3 grd((unsigned)cdiv(g.ncells, 128), (unsigned)std::min<int64_t>(g.nbatch, 65535));
  index_adj_dense_kernel<T, K><<<grd, 128, 0, s>>>((const T*)vals, perm, off, (T*)out, g.npts, g.ncells, g.nbatch);
}
// Through shared memory, as many cells and entries per CTA as leave four CTAs
// per SM; small grids take one cell per thread, and one entry where that is still
// too few. 16-byte values take at most two entries (four need 119 registers).
template <typename T>
void launch_index_adj(const IdxGeo& g, const void* vals, const int32_t* perm, const uint32_t* off, void* out, cudaStream_t s) {
  if constexpr (sizeof(T) > 8) {
    if (g.npts >= 16 * g.ncells) launch_index_adj_dense<T, 4>(g, vals, perm, off, out, s);
    else if (4 * g.npts >= g.ncells) launch_index_adj_dense<T, 2>(g, vals, perm, off, out, s);
    else if (g.nbatch == 1) launch_index_adj_at<T, 1, 4>(g, vals, perm, off, out, s);
    else launch_index_adj_at<T, 2, 4>(g, vals, perm, off, out, s);
  } else {
    const int64_t want = 4ll * sm_count(), groups = cdiv(g.nbatch, 4);
    if (g.npts >= (std::is_same<T, float2>::value ? 4 : 2) * g.ncells) launch_index_adj_dense<T, 8>(g, vals, perm, off, out, s);
    else if (g.npts >= g.ncells) launch_index_adj_dense<T, 4>(g, vals, perm, off, out, s);
    else if (g.nbatch > 1 && cdiv(g.ncells, 1024) * groups >= want) launch_index_adj_at<T, 4, 4>(g, vals, perm, off, out, s);
    else if (g.nbatch == 1 && cdiv(g.ncells, 1024) >= want) launch_index_adj_at<T, 1, 4>(g, vals, perm, off, out, s);
    else if (g.nbatch > 1 && cdiv(g.ncells, 256) * groups >= want) launch_index_adj_at<T, 4, 1>(g, vals, perm, off, out, s);
    else launch_index_adj_at<T, 1, 1>(g, vals, perm, off, out, s);
  }
}

int make_idx_geo(const tlgb_index_desc* d, IdxGeo& g) {
  if (!d) TLGB_FAIL(TLGB_ERR_INVALID, "null index descriptor");
  if (d->ndim < 1 || d->ndim > TLGB_INDEX_MAX_DIM) TLGB_FAIL(TLGB_ERR_INVALID, "index: ndim must be in [1, 8]");
  if (d->npts < 0 || d->nbatch < 0) TLGB_FAIL(TLGB_ERR_INVALID, "index: negative size");
  g.ndim = d->ndim;
  int64_t n = 1;
  for (int e = d->ndim - 1; e >= 0; --e) {
    if (d->grid_size[e] < 1) TLGB_FAIL(TLGB_ERR_INVALID, "index: grid sizes must be positive");
    g.size[e] = d->grid_size[e];
    g.stride[e] = n;
    if (n > (int64_t)INT32_MAX / d->grid_size[e]) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "index: grid above 2^31 - 1 cells");
    n *= d->grid_size[e];
  }
  g.ncells = n;
  if (d->npts > (int64_t)INT32_MAX - 1) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "index: 2^31 - 1 samples or more");
  g.npts = d->npts;
  g.nbatch = d->nbatch;
  return TLGB_OK;
}

IdxLayout idx_layout(const IdxGeo& g) {
  IdxLayout L;
  const int64_t m = std::max<int64_t>(g.npts, 1);
  size_t o = 0;
  L.off_flat = o;
  o = align_up(o + (size_t)m * 4, 256);
  L.off_perm = o;
  o = align_up(o + (size_t)m * 4, 256);
  L.off_cells = o;
  o = align_up(o + (size_t)(g.ncells + 1) * 4, 256);
  L.bytes = o;
  size_t t = 0;
  L.t_keys = t;
  t = align_up(t + (size_t)m * 4, 256);
  L.t_keys2 = t;
  t = align_up(t + (size_t)m * 4, 256);
  L.t_vals2 = t;
  t = align_up(t + (size_t)m * 4, 256);
  L.t_counts = t;
  t = align_up(t + (size_t)radix_counts_len(m) * 4, 256);
  L.t_cnt = t;
  t = align_up(t + (size_t)g.ncells * 4, 256);
  L.t_scan = t;
  t = align_up(t + (size_t)scan_scratch_len(g.ncells) * 4, 256);
  L.t_bad = t;
  t = align_up(t + 16, 256);
  L.t_bytes = t;
  return L;
}

int elem_bytes(int dtype) {
  switch (dtype) {
    case TLGB_F32: case TLGB_I32: return 4;
    case TLGB_F64: case TLGB_C64: case TLGB_I64: return 8;
    case TLGB_C128: return 16;
    case TLGB_RAW8: return 1;
    case TLGB_RAW16: return 2;
    default: return 0;
  }
}

int check_index_plan(const IdxGeo& g, const tlgb_index_plan_info* info, const void* plan) {
  if (!info || !plan) TLGB_FAIL(TLGB_ERR_INVALID, "index: null plan");
  if (info->ncells != g.ncells || info->npts != g.npts)
    TLGB_FAIL(TLGB_ERR_INVALID, "index: plan was built for another grid or sample count");
  return TLGB_OK;
}

unsigned grid_for(int64_t n) {
  const int64_t cap = (int64_t)sm_count() * 8;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(cap, cdiv(n, 256)));
}

}  // namespace
}  // namespace tlgb

using namespace tlgb;

extern "C" int tlgb_index_plan_size(const tlgb_index_desc* d, size_t* plan_bytes, size_t* tmp_bytes) {
  IdxGeo g;
  TLGB_TRY(make_idx_geo(d, g));
  if (!plan_bytes || !tmp_bytes) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  const IdxLayout L = idx_layout(g);
  *plan_bytes = (size_t)L.bytes;
  *tmp_bytes = (size_t)L.t_bytes;
  return TLGB_OK;
}

extern "C" int tlgb_index_plan_build(const tlgb_index_desc* d, const int64_t* idx, void* plan, size_t plan_bytes,
                                     void* tmp, size_t tmp_bytes, tlgb_index_plan_info* info, tlgb_stream_t stream) {
  IdxGeo g;
  TLGB_TRY(make_idx_geo(d, g));
  if (!plan || !tmp || !info || (g.npts > 0 && !idx)) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  const IdxLayout L = idx_layout(g);
  if (plan_bytes < (size_t)L.bytes || tmp_bytes < (size_t)L.t_bytes)
    TLGB_FAIL(TLGB_ERR_WORKSPACE, "index plan or temporary buffer too small");
  cudaStream_t s = (cudaStream_t)stream;
  char* P = static_cast<char*>(plan);
  char* T = static_cast<char*>(tmp);
  int32_t* flat = reinterpret_cast<int32_t*>(P + L.off_flat);
  int32_t* perm = reinterpret_cast<int32_t*>(P + L.off_perm);
  uint32_t* off = reinterpret_cast<uint32_t*>(P + L.off_cells);
  uint32_t* keys = reinterpret_cast<uint32_t*>(T + L.t_keys);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(T + L.t_cnt);
  int* bad = reinterpret_cast<int*>(T + L.t_bad);
  TLGB_CUDA(cudaMemsetAsync(cnt, 0, (size_t)g.ncells * 4, s));
  const int none = 0x7f7f7f7f;  // every byte 0x7f: above any dimension index
  TLGB_CUDA(cudaMemsetAsync(bad, 0x7f, sizeof(int), s));
  if (g.npts > 0) {
    index_ravel_kernel<<<grid_for(g.npts), 256, 0, s>>>(g, idx, flat, keys, perm, cnt, bad);
    TLGB_CHECK_LAUNCH();
    int bits = 1;
    while (bits < 32 && ((int64_t)1 << bits) < g.ncells) ++bits;
    TLGB_TRY(radix_sort_pairs(keys, perm, reinterpret_cast<uint32_t*>(T + L.t_keys2),
                              reinterpret_cast<int32_t*>(T + L.t_vals2), reinterpret_cast<uint32_t*>(T + L.t_counts),
                              g.npts, bits, s));
  }
  TLGB_TRY(exclusive_scan_u32(cnt, off, g.ncells, off + g.ncells, reinterpret_cast<uint32_t*>(T + L.t_scan), s));
  int worst = none;
  TLGB_CUDA(cudaMemcpyAsync(&worst, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  TLGB_CUDA(cudaStreamSynchronize(s));
  if (worst < none) {
    std::string shape;
    for (int e = 0; e < g.ndim; ++e) shape += (e ? ", " : "") + std::to_string(g.size[e]);
    if (g.ndim == 1) shape += ",";  // as Python prints a 1-tuple
    TLGB_FAIL(TLGB_ERR_INVALID, "Out-of-bounds index for grid of shape (" + shape + "): idx[" +
                                    std::to_string(worst) + "]");
  }
  memset(info, 0, sizeof(*info));
  info->ncells = g.ncells;
  info->npts = g.npts;
  info->off_flat = L.off_flat;
  info->off_perm = L.off_perm;
  info->off_cells = L.off_cells;
  info->plan_bytes = L.bytes;
  return TLGB_OK;
}

extern "C" int tlgb_index_forward(const tlgb_index_desc* d, const tlgb_index_plan_info* info, const void* plan,
                                  const void* vals, void* out, tlgb_stream_t stream) {
  IdxGeo g;
  TLGB_TRY(make_idx_geo(d, g));
  TLGB_TRY(check_index_plan(g, info, plan));
  if (g.npts == 0 || g.nbatch == 0) return TLGB_OK;
  if (!vals || !out) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  const int32_t* flat = reinterpret_cast<const int32_t*>(static_cast<const char*>(plan) + info->off_flat);
  switch (elem_bytes(d->dtype)) {
    case 1: launch_index_fwd<uint8_t>(g, vals, flat, out, s); break;
    case 2: launch_index_fwd<uint16_t>(g, vals, flat, out, s); break;
    case 4: launch_index_fwd<uint32_t>(g, vals, flat, out, s); break;
    case 8: launch_index_fwd<uint2>(g, vals, flat, out, s); break;
    case 16: launch_index_fwd<uint4>(g, vals, flat, out, s); break;
    default: TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "index: unsupported element type");
  }
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

extern "C" int tlgb_index_adjoint(const tlgb_index_desc* d, const tlgb_index_plan_info* info, const void* plan,
                                  const void* vals, void* out, tlgb_stream_t stream) {
  IdxGeo g;
  TLGB_TRY(make_idx_geo(d, g));
  TLGB_TRY(check_index_plan(g, info, plan));
  if (g.nbatch == 0) return TLGB_OK;
  if (!out || (g.npts > 0 && !vals)) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  const char* P = static_cast<const char*>(plan);
  const int32_t* perm = reinterpret_cast<const int32_t*>(P + info->off_perm);
  const uint32_t* off = reinterpret_cast<const uint32_t*>(P + info->off_cells);
  switch (d->dtype) {
    case TLGB_F32: launch_index_adj<float>(g, vals, perm, off, out, s); break;
    case TLGB_F64: launch_index_adj<double>(g, vals, perm, off, out, s); break;
    case TLGB_C64: launch_index_adj<float2>(g, vals, perm, off, out, s); break;
    case TLGB_C128: launch_index_adj<double2>(g, vals, perm, off, out, s); break;
    case TLGB_I32: launch_index_adj<int32_t>(g, vals, perm, off, out, s); break;
    case TLGB_I64: launch_index_adj<long long>(g, vals, perm, off, out, s); break;
    default: TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "index adjoint: unsupported element type");
  }
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}
