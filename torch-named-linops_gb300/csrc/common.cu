// Error reporting, version, and the plan-time scan / stable radix sort.

#include <algorithm>
#include <string>

#include "common.cuh"

namespace tlgb {

static thread_local std::string g_last_error;

void set_error(const std::string& msg) { g_last_error = msg; }

namespace {

constexpr int kScanThreads = 1024;

// Single-CTA exclusive scan: each thread scans a contiguous segment.
__global__ void __launch_bounds__(kScanThreads) scan_kernel(const uint32_t* in, uint32_t* out, int64_t n,
                                                             uint32_t* total) {
  __shared__ uint32_t part[kScanThreads];
  const int64_t per = (n + kScanThreads - 1) / kScanThreads;
  const int64_t b = threadIdx.x * per;
  const int64_t e = b + per < n ? b + per : n;
  uint32_t s = 0;
  for (int64_t i = b; i < e; ++i) s += in[i];
  part[threadIdx.x] = s;
  __syncthreads();
  // Hillis-Steele inclusive scan of the partials
  for (int off = 1; off < kScanThreads; off <<= 1) {
    uint32_t v = threadIdx.x >= off ? part[threadIdx.x - off] : 0u;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  uint32_t run = threadIdx.x ? part[threadIdx.x - 1] : 0u;
  for (int64_t i = b; i < e; ++i) {
    const uint32_t v = in[i];
    out[i] = run;
    run += v;
  }
  if (threadIdx.x == kScanThreads - 1 && total) *total = part[kScanThreads - 1];
}

// Multi-CTA exclusive scan for long inputs: per-block sums, a scan of the
// sums (scan_kernel, one CTA), then each block's scan plus its offset.
constexpr int kScanBlock = 4096;  // elements per CTA (256 threads x 16)

__device__ __forceinline__ uint32_t block_sum_256(uint32_t v) {
  __shared__ uint32_t ws[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  if (threadIdx.x < 8) t = ws[threadIdx.x];
  if (threadIdx.x < 32) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;  // valid in thread 0
}

__global__ void __launch_bounds__(256) scan_block_sums_kernel(const uint32_t* __restrict__ in, int64_t n,
                                                              uint32_t* __restrict__ sums) {
  const int64_t b0 = (int64_t)blockIdx.x * kScanBlock;
  uint32_t s = 0;
  for (int i = threadIdx.x; i < kScanBlock; i += 256) {
    const int64_t k = b0 + i;
    if (k < n) s += in[k];
  }
  s = block_sum_256(s);
  if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) scan_blocks_kernel(const uint32_t* in, uint32_t* out, int64_t n,
                                                          const uint32_t* __restrict__ offsets) {
  __shared__ uint32_t tile[kScanBlock];
  __shared__ uint32_t wsum[8];
  const int64_t b0 = (int64_t)blockIdx.x * kScanBlock;
  for (int i = threadIdx.x; i < kScanBlock; i += 256) {
    const int64_t k = b0 + i;
    tile[i] = k < n ? in[k] : 0u;
  }
  __syncthreads();
  // each thread scans its 16 consecutive elements
  uint32_t loc[16], run = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    loc[j] = run;
    run += tile[threadIdx.x * 16 + j];
  }
  // exclusive scan of the thread totals: warp shuffles, then warp totals
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  uint32_t wbase = 0;
  for (int w = 0; w < warp; ++w) wbase += wsum[w];
  const uint32_t base = offsets[blockIdx.x] + wbase + x - run;
  __syncthreads();  // every thread has read its inputs from the tile
#pragma unroll
  for (int j = 0; j < 16; ++j) tile[threadIdx.x * 16 + j] = base + loc[j];
  __syncthreads();
  for (int i = threadIdx.x; i < kScanBlock; i += 256) {
    const int64_t k = b0 + i;
    if (k < n) out[k] = tile[i];
  }
}

// ---- stable radix sort
//
// A pass is three launches: digit counts of each CTA's 4096 pairs, a scan of
// the counts (one CTA per digit), and the scatter. The scatter ranks its pairs
// in shared memory (8 warps x 16 rounds of 32 pairs, equal digits of a round
// ranked by ballots), puts them in digit order there and then writes runs
// of equal digits, so the stores of a run are contiguous. The passes are
// short chains: at the sizes of one trajectory (10^5 to 10^7 pairs) a sort is
// bound by the launches and by each CTA's latency, not by HBM, so a warp
// walks 512 pairs, not a longer share, and the digits are as wide as one
// pass more would cost (9 bits: two passes up to 2^18 keys).
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // pairs per CTA
constexpr int kSortBits = 9;                          // widest digit
constexpr int kSortDigits = 1 << kSortBits;

struct SortJobs {
  SortJob j[2];
  int shift[2], dbits[2];
};

__device__ __forceinline__ int64_t job_len(const SortJob& j) { return j.n ? (int64_t)*j.n : j.n_max; }

// counts[d * stride + cta], stride = CTAs for n_max pairs
__device__ __forceinline__ int64_t job_stride(const SortJob& j) { return (j.n_max + kSortTile - 1) / kSortTile; }

__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(SortJobs jobs, int src) {
  __shared__ uint32_t hist[kSortDigits];
  const SortJob& j = jobs.j[blockIdx.y];
  const int64_t n = job_len(j), b = (int64_t)blockIdx.x * kSortTile;
  if (b >= n) return;
  const int shift = jobs.shift[blockIdx.y], nd = 1 << jobs.dbits[blockIdx.y];
  for (int d = threadIdx.x; d < nd; d += kSortThreads) hist[d] = 0;
  __syncthreads();
  const uint32_t* keys = j.keys[src];
  uint32_t k[kSortItems];
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const int64_t p = b + i * kSortThreads + threadIdx.x;
    if (p < n) k[i] = keys[p];
  }
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const int64_t p = b + i * kSortThreads + threadIdx.x;
    if (p < n) atomicAdd(&hist[(k[i] >> shift) & (nd - 1)], 1u);
  }
  __syncthreads();
  const int64_t stride = job_stride(j);
  for (int d = threadIdx.x; d < nd; d += kSortThreads) j.counts[d * stride + blockIdx.x] = hist[d];
}

// inclusive scan of one value per thread over a CTA of 256 threads
__device__ __forceinline__ uint32_t cta_scan_incl(uint32_t v, uint32_t* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) wsum[warp] = v;
  __syncthreads();
  uint32_t base = 0;
  for (int w = 0; w < warp; ++w) base += wsum[w];
  return v + base;
}

// CTA = one digit's row of counts: exclusive scan in place, total to the
// digit's slot after the rows
__global__ void __launch_bounds__(kSortThreads) radix_rows_kernel(SortJobs jobs) {
  __shared__ uint32_t wsum[kSortWarps];
  const SortJob& j = jobs.j[blockIdx.y];
  if (blockIdx.x >= 1u << jobs.dbits[blockIdx.y]) return;
  const int64_t n = job_len(j), ncta = (n + kSortTile - 1) / kSortTile, stride = job_stride(j);
  uint32_t* row = j.counts + blockIdx.x * stride;
  uint32_t run = 0;
  for (int64_t b = 0; b < ncta; b += kSortThreads * 4) {
    uint32_t v[4], s = 0;
    const int64_t i0 = b + threadIdx.x * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = i0 + i < ncta ? row[i0 + i] : 0u;
      s += v[i];
    }
    __syncthreads();  // the previous round's warp sums have been read
    const uint32_t incl = cta_scan_incl(s, wsum);
    uint32_t o = run + incl - s;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i0 + i < ncta) row[i0 + i] = o;
      o += v[i];
    }
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) tot += wsum[w];
    run += tot;
  }
  if (threadIdx.x == 0) j.counts[kSortDigits * stride + blockIdx.x] = run;
}

__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(SortJobs jobs, int src) {
  __shared__ uint16_t whist[kSortWarps][kSortDigits];  // counts, then each warp's first rank per digit
  __shared__ uint32_t lstart[kSortDigits];             // first local position of a digit
  __shared__ uint32_t gbase[kSortDigits];              // its global position minus the local one
  __shared__ uint32_t wsum[kSortWarps];
  __shared__ uint32_t skey[kSortTile];
  __shared__ int32_t sval[kSortTile];
  const SortJob& j = jobs.j[blockIdx.y];
  const int64_t n = job_len(j), b = (int64_t)blockIdx.x * kSortTile;
  if (b >= n) return;
  const int cnt = (int)(n - b < kSortTile ? n - b : kSortTile);
  const int shift = jobs.shift[blockIdx.y], dbits = jobs.dbits[blockIdx.y], nd = 1 << dbits;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = lane; i < kSortDigits; i += 32) whist[warp][i] = 0;
  const uint32_t* kin = j.keys[src] + b;
  const int32_t* vin = j.vals[src] + b;
  uint32_t key[kSortItems];
  int32_t val[kSortItems];
  uint16_t rank[kSortItems];
  const int w0 = warp * 32 * kSortItems + lane;
#pragma unroll
  for (int i = 0; i < kSortItems; ++i)
    if (w0 + 32 * i < cnt) key[i] = kin[w0 + 32 * i], val[i] = vin[w0 + 32 * i];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const bool on = w0 + 32 * i < cnt;
    const uint32_t d = on ? (key[i] >> shift) & (nd - 1) : 0u;
    unsigned peers = __ballot_sync(0xffffffffu, on);
    for (int k = 0; k < dbits; ++k) {
      const unsigned bal = __ballot_sync(0xffffffffu, (d >> k) & 1u);
      peers &= (d >> k) & 1u ? bal : ~bal;
    }
    const int before = __popc(peers & ((1u << lane) - 1u));
    uint16_t base = 0;
    if (on) base = whist[warp][d];
    __syncwarp();
    if (on) {
      rank[i] = (uint16_t)(base + before);
      if (before == 0) whist[warp][d] = (uint16_t)(base + __popc(peers));
    }
    __syncwarp();
  }
  __syncthreads();
  // digits 2 tid and 2 tid + 1: totals over the warps, their local and global starts
  const int64_t stride = job_stride(j);
  uint32_t tot[2] = {0, 0}, gt[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int d = 2 * tid + h;
    if (d < nd) {
      for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = whist[w][d];
        whist[w][d] = (uint16_t)tot[h];
        tot[h] += c;
      }
      gt[h] = j.counts[kSortDigits * stride + d];
    }
  }
  const uint32_t li = cta_scan_incl(tot[0] + tot[1], wsum) - tot[0] - tot[1];
  __syncthreads();
  const uint32_t gi = cta_scan_incl(gt[0] + gt[1], wsum) - gt[0] - gt[1];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int d = 2 * tid + h;
    if (d < nd) {
      const uint32_t l = li + (h ? tot[0] : 0u);
      lstart[d] = l;
      gbase[d] = gi + (h ? gt[0] : 0u) + j.counts[d * stride + blockIdx.x] - l;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    if (w0 + 32 * i < cnt) {
      const uint32_t d = (key[i] >> shift) & (nd - 1);
      const uint32_t l = lstart[d] + whist[warp][d] + rank[i];
      skey[l] = key[i];
      sval[l] = val[i];
    }
  }
  __syncthreads();
  uint32_t* kout = j.keys[src ^ 1];
  int32_t* vout = j.vals[src ^ 1];
  for (int i = tid; i < cnt; i += kSortThreads) {
    const uint32_t k = skey[i], o = gbase[(k >> shift) & (nd - 1)] + (uint32_t)i;
    kout[o] = k;
    vout[o] = sval[i];
  }
}

}  // namespace

int64_t scan_scratch_len(int64_t n) { return (n + kScanBlock - 1) / kScanBlock + 1; }

int exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* total_dev, uint32_t* scratch,
                       cudaStream_t s) {
  if (n <= 0) {
    if (total_dev) TLGB_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s));
    return TLGB_OK;
  }
  if (!scratch || n <= 4 * kScanBlock) {
    scan_kernel<<<1, kScanThreads, 0, s>>>(in, out, n, total_dev);
    TLGB_CHECK_LAUNCH();
    return TLGB_OK;
  }
  const int64_t nb = (n + kScanBlock - 1) / kScanBlock;
  scan_block_sums_kernel<<<(unsigned)nb, 256, 0, s>>>(in, n, scratch);
  TLGB_CHECK_LAUNCH();
  scan_kernel<<<1, kScanThreads, 0, s>>>(scratch, scratch, nb, total_dev);
  TLGB_CHECK_LAUNCH();
  scan_blocks_kernel<<<(unsigned)nb, 256, 0, s>>>(in, out, n, scratch);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

int radix_passes(int bits) { return (int)cdiv(std::max(bits, 1), kSortBits); }

int64_t radix_counts_len(int64_t n) {
  return kSortDigits * (cdiv(std::max<int64_t>(n, 1), kSortTile) + 1);  // digit rows, then the digits' totals
}

int radix_sort_jobs(const SortJob* jobs, int njobs, cudaStream_t s) {
  SortJobs J;
  int passes = 1;
  int64_t nmax = 0;
  for (int i = 0; i < njobs; ++i) {
    J.j[i] = jobs[i];
    passes = std::max(passes, radix_passes(jobs[i].bits));
    nmax = std::max(nmax, jobs[i].n_max);
  }
  if (nmax <= 0) return TLGB_OK;
  const dim3 grid((unsigned)cdiv(nmax, kSortTile), (unsigned)njobs);
  for (int p = 0; p < passes; ++p) {
    int widest = 1;
    for (int i = 0; i < njobs; ++i) {
      J.dbits[i] = (int)cdiv(std::max(jobs[i].bits, 1), passes);
      J.shift[i] = std::min(p * J.dbits[i], 31);
      widest = std::max(widest, J.dbits[i]);
    }
    radix_hist_kernel<<<grid, kSortThreads, 0, s>>>(J, p & 1);
    TLGB_CHECK_LAUNCH();
    radix_rows_kernel<<<dim3(1u << widest, (unsigned)njobs), kSortThreads, 0, s>>>(J);
    TLGB_CHECK_LAUNCH();
    radix_scatter_kernel<<<grid, kSortThreads, 0, s>>>(J, p & 1);
    TLGB_CHECK_LAUNCH();
  }
  return TLGB_OK;
}

int radix_sort_pairs(uint32_t* keys, int32_t* vals, uint32_t* keys_tmp, int32_t* vals_tmp, uint32_t* counts_tmp,
                     int64_t n, int bits, cudaStream_t s) {
  if (n <= 1) return TLGB_OK;
  const SortJob j = {{keys, keys_tmp}, {vals, vals_tmp}, counts_tmp, nullptr, n, bits};
  TLGB_TRY(radix_sort_jobs(&j, 1, s));
  if (radix_passes(bits) & 1) {
    TLGB_CUDA(cudaMemcpyAsync(keys, keys_tmp, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    TLGB_CUDA(cudaMemcpyAsync(vals, vals_tmp, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
  }
  return TLGB_OK;
}

int sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  if (cache[dev] == 0) {
    int n = 0;
    cache[dev] = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 152;
  }
  return cache[dev];
}

}  // namespace tlgb

extern "C" const char* tlgb_last_error(void) { return tlgb::g_last_error.c_str(); }

extern "C" int tlgb_version(void) { return 100; }
