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
constexpr int adj_ctas(size_t bytes, int entries) { return (entries == 1 ? 8 : 4) / (bytes > 8 ? 2 : 1); }

template <typename T, int U, int C>
__global__ void __launch_bounds__(256, adj_ctas(sizeof(T), U)) index_adj_kernel(const T* __restrict__ vals, const int32_t* __restrict__ perm,
                                                        const uint32_t* __restrict__ off, T* __restrict__ out, int64_t npts,
                                                        int64_t ncells, int64_t nbatch) {
  __shared__ T sm[U][kAdjChunk];
  const int64_t first = (int64_t)blockIdx.x * (256 * C), c0 = first + threadIdx.x;
  const uint32_t ka = off[first], kb = off[min(first + 256 * C, ncells)];
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

// The same on grids whose cells hold several samples: a cell's samples are
// contiguous in perm, and K of its values are read ahead of adding them. 8
// entries of 64^2 at 2^20 samples: 2150 us one value at a time, 292 and 254 us
// with K = 4 and 8, 807 us through shared memory, where a chunk holds one cell
// and its CTA waits for that one lane; 12 entries of 320^2 (10 samples per
// cell): 187, 79 and 78, 129 us; at a quarter sample per cell 160^3 prefers
// shared memory, 104 against 160 us. The line is at two samples per cell.
template <typename T, int K>
__global__ void __launch_bounds__(256) index_adj_dense_kernel(const T* __restrict__ vals, const int32_t* __restrict__ perm,
                                                              const uint32_t* __restrict__ off, T* __restrict__ out,
                                                              int64_t npts, int64_t ncells, int64_t nbatch) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const uint32_t k0 = off[c], k1 = off[c + 1];
  for (int64_t b = blockIdx.y; b < nbatch; b += gridDim.y) {
    const T* vb = vals + b * npts;
    Acc<T> a;
    for (uint32_t k = k0; k < k1; k += K) {
      T v[K];
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (k + i < k1) v[i] = vb[perm[k + i]];
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (k + i < k1) a.add(v[i]);
    }
    out[b * ncells + c] = a.v;
  }
}

template <typename T, int U, int C>
void launch_index_adj_at(const IdxGeo& g, const void* vals, const int32_t* perm, const uint32_t* off, void* out,
                         cudaStream_t s) {
  const dim3 grd((unsigned)cdiv(g.ncells, 256 * C), (unsigned)std::min<int64_t>(cdiv(g.nbatch, U), 65535));
  index_adj_kernel<T, U, C><<<grd, 256, 0, s>>>((const T*)vals, perm, off, (T*)out, g.npts, g.ncells, g.nbatch);
}
// As many cells and entries per CTA as leave four CTAs per SM; small grids
// take one cell per thread, and one entry where that is still too few.
template <typename T>
void launch_index_adj(const IdxGeo& g, const void* vals, const int32_t* perm, const uint32_t* off, void* out, cudaStream_t s) {
  if (g.npts >= 2 * g.ncells) {
    const dim3 grd((unsigned)cdiv(g.ncells, 128), (unsigned)std::min<int64_t>(g.nbatch, 65535));
    index_adj_dense_kernel<T, 8><<<grd, 128, 0, s>>>((const T*)vals, perm, off, (T*)out, g.npts, g.ncells, g.nbatch);
    return;
  }
  const int64_t want = 4ll * sm_count(), groups = cdiv(g.nbatch, 4);
  if (g.nbatch > 1 && cdiv(g.ncells, 1024) * groups >= want) launch_index_adj_at<T, 4, 4>(g, vals, perm, off, out, s);
  else if (g.nbatch == 1 && cdiv(g.ncells, 1024) >= want) launch_index_adj_at<T, 1, 4>(g, vals, perm, off, out, s);
  else if (g.nbatch > 1 && cdiv(g.ncells, 256) * groups >= want) launch_index_adj_at<T, 4, 1>(g, vals, perm, off, out, s);
  else launch_index_adj_at<T, 1, 1>(g, vals, perm, off, out, s);
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
