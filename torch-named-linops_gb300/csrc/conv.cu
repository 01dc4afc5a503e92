// 3^3 convolution, 16 -> 16 channels, BF16 operands with FP32 accumulation, on
// the tensor cores: the layers of the learned CG preconditioner (no
// counterpart in the reference; it replaces nothing there).
//
// Layout: activations channels-last [D][H][W][16] bf16, zero padding 1, same
// spatial size in and out. Weights [27][16 out][16 in] bf16, tap t = (kd*3 +
// kh)*3 + kw. Forward and data-gradient are one implicit-GEMM kernel (the
// data gradient is the forward with flipped, transposed weights); the weight
// gradient is a second kernel with a fixed-order cross-CTA reduction.

#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "sm100.cuh"

namespace tlgb {
namespace {

constexpr int kTileW = 64;               // output voxels along W per CTA (4 warps x 16)
constexpr int kHaloW = kTileW + 2;       // input voxels along W per staged row
constexpr int kVoxBytes = 32;            // 16 bf16 channels
constexpr int kTaps = 27;

// 16-byte chunk c of row j in a 32-byte-row tile, XOR-swizzled so that the 8
// row addresses of one ldmatrix phase fall in distinct banks
__device__ __forceinline__ uint32_t swz(int j, int c) { return (uint32_t)(j * 32 + ((c ^ ((j >> 2) & 1)) << 4)); }

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// D(16x8, f32) += A(16x16, bf16, row) * B(16x8, bf16, col)
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}

// ---- the tcgen05 path of the forward / data gradient
//
// Persistent CTAs, two per SM: 4 epilogue warps, 4 loader warps and one warp
// that issues the MMAs. A work unit is a column segment of some output rows
// (unit_rows) (fixed d, consecutive h) of 128 voxels along W (MMA M = 128). The input
// rows (d + kd - 1, h'), kd = 0..2, contribute through their taps to the output
// rows h' - 1, h', h' + 1: one MMA of N = 48 per (kd, kw), whose B operand holds
// the weights of kh = 2, 1, 0 side by side, into the 128 x 48 FP32 accumulator
// of h'. An output row is the sum of one 16-column block of three neighbouring
// accumulators, added in the epilogue. So an output row costs 9 MMAs that read
// their A operand from shared memory, not 27 of N = 16 (those read 4 KB for 8
// cycles of products). The loaders copy the 3 kd rows of an h' as one ring slot,
// 16 bytes at a time into the canonical no-swizzle K-major layout (16-byte
// rows, the two 8-channel halves of a row 2176 bytes apart; a TMA box of this
// layout is 16 bytes wide, 780 such rows per h'); tap kw is the A operand kw
// rows into the slot. Accumulators sit in a ring of 5, so the epilogue of one
// row overlaps the MMAs of the next. Weights stay in shared memory for the
// CTA's lifetime. 128^3: 72 us (99 with 27 MMAs per row fed by TMA; 110 with one
// CTA per SM, whose waits nothing covers; 54 without the copies, 33 with one
// MMA per row and no copies or stores; HBM floor 20 us).
// Every wait is bounded; a timeout sets the status word and a CTA flag, every
// role stops, and the MMAs and copies in flight are waited for before TMEM is
// freed.
constexpr int kTcM = 128;
constexpr int kTcHalo = kTcM + 2;
constexpr int kTcHalfBytes = 2176;                        // >= 130 * 16, a multiple of 128
constexpr int kTcRowBytes = 2 * kTcHalfBytes;
constexpr int kTcSlotBytes = 3 * kTcRowBytes;             // the 3 kd rows of one h'
constexpr int kTcSlots = 5;
constexpr int kTcAhead = 3;                               // slots being copied at once
constexpr uint32_t kTcBTap = 1536;                        // B of one (kd, kw): [k half][6 n groups][8][16 B]
constexpr uint32_t kTcBBytes = 9 * kTcBTap;
constexpr int kTcAcc = 5;                                 // accumulators of 48 columns
constexpr int kTcBars = 2 * kTcSlots + 2 * kTcAcc + 1;    // slots full, empty; accumulators done, free; drain
constexpr uint32_t kTcSmem = kTcSlots * kTcSlotBytes + kTcBBytes + 8 * kTcBars + 16;
constexpr uint32_t kTcCols = 256;                         // TMEM columns, 240 used
constexpr int kTcCtas = 2;                                // CTAs per SM
constexpr int kTcThreads = 288;
constexpr uint32_t kTcWait = 1u << 22;

__device__ int g_conv_status;

template <int MODE, bool OUTF32>
__global__ void __launch_bounds__(kTcThreads, kTcCtas) conv3d_tc_kernel(int D, int H, int W, int rows, const uint4* __restrict__ x,
                                                                  const uint4* __restrict__ wts,
                                                                  const __nv_bfloat16* __restrict__ aux,
                                                                  void* __restrict__ y) {
  using namespace sm100;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sb = smem + kTcSlots * kTcSlotBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(sb + kTcBBytes);
  uint64_t* empty = full + kTcSlots;
  uint64_t* done = empty + kTcSlots;
  uint64_t* freed = done + kTcAcc;
  uint64_t* drain = freed + kTcAcc;
  uint32_t* slot = reinterpret_cast<uint32_t*>(drain + 1);  // [0] TMEM address, [1] failure flag
  volatile uint32_t* failed = slot + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntw = (W + kTcM - 1) / kTcM, nseg = (H + rows - 1) / rows;
  const long long nunits = (long long)D * ntw * nseg;
  if (warp == 0) {
    tmem_alloc(slot, kTcCols);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < kTcSlots; ++i) {
      mbar_init(&full[i], 128);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < kTcAcc; ++i) {
      mbar_init(&done[i], 1);
      mbar_init(&freed[i], 128);
    }
    mbar_init(drain, 1);
    fence_mbar_init();
    slot[1] = 0;
  }
  for (int i = tid; i < kTaps * 16 * 2; i += kTcThreads) {
    const int half = i & 1, co = (i >> 1) & 15, t = i >> 5, kd = t / 9, kh = t / 3 % 3, kw = t % 3;
    const int n = (2 - kh) * 16 + co;
    *reinterpret_cast<uint4*>(sb + (kd * 3 + kw) * kTcBTap + half * 768 + (n >> 3) * 128 + (n & 7) * 16) = __ldg(wts + i);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = slot[0];
  auto give_up = [&]() {
    *failed = 1;
    atomicExch(&g_conv_status, 2);
  };
  auto unit = [&](long long u, int& d, int& w0, int& h0, int& R) {
    const int hs = (int)(u % nseg);
    const long long dw = u / nseg;
    w0 = (int)(dw % ntw) * kTcM, d = (int)(dw / ntw), h0 = hs * rows, R = min(rows, H - h0);
  };

  if (warp >= 4 && warp < 8) {
    // ---- loaders
    const int lt = tid - 128;
    const uint32_t s0 = smem_u32(smem);
    constexpr int NC = (3 * kTcHalo * 2 + 127) / 128;
    uint32_t k = 0, sent = 0;  // slots begun, slots handed over
    bool ok = true;
    auto hand_over = [&]() {   // this thread's copies of slot `sent` have landed
      fence_proxy_async_smem();
      mbar_arrive(&full[sent % kTcSlots]);
      ++sent;
    };
    for (long long u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
      int d, w0, h0, R;
      unit(u, d, w0, h0, R);
      long long xoff[NC];
      uint32_t soff[NC];
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const int q = lt + 128 * i, kd = q / (kTcHalo * 2), j = (q >> 1) % kTcHalo, c = q & 1;
        const int di = d + kd - 1, wi = w0 - 1 + j;
        soff[i] = (uint32_t)(kd * kTcRowBytes + c * kTcHalfBytes + j * 16);
        xoff[i] = di >= 0 && di < D && wi >= 0 && wi < W ? ((long long)di * H * W + wi) * 2 + c : -1;
      }
      for (int hr = h0 - 1; hr <= h0 + R; ++hr, ++k) {
        const uint32_t s = k % kTcSlots;
        ok = mbar_wait_bounded(&empty[s], ((k / kTcSlots) & 1) ^ 1, kTcWait) && !*failed;
        if (!ok) break;
        const bool hin = hr >= 0 && hr < H;
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (lt + 128 * i < 3 * kTcHalo * 2) {
            const bool in = hin && xoff[i] >= 0;
            cp_async16_zfill(s0 + s * kTcSlotBytes + soff[i], in ? x + xoff[i] + (long long)hr * W * 2 : x, in);
          }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group %0;" ::"n"(kTcAhead - 1) : "memory");
        if (k >= kTcAhead - 1) hand_over();
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (ok)
      while (sent < k) hand_over();
    else
      give_up();
  } else if (warp == 8) {
    // ---- MMA issue, one thread
    if (lane == 0) {
      const uint32_t a0 = smem_u32(smem), b0 = smem_u32(sb);
      constexpr uint32_t idesc = idesc_bf16_f32(kTcM, 48);
      uint32_t k = 0;
      bool ok = true;
      for (long long u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
        int d, w0, h0, R;
        unit(u, d, w0, h0, R);
        for (int i = 0; i < R + 2; ++i, ++k) {  // input row h0 - 1 + i
          const uint32_t s = k % kTcSlots, q = k % kTcAcc;
          ok = mbar_wait_bounded(&freed[q], ((k / kTcAcc) & 1) ^ 1, kTcWait) &&
               mbar_wait_bounded(&full[s], (k / kTcSlots) & 1, kTcWait) && !*failed;
          if (!ok) break;
          tc_fence_after();
          for (int t = 0; t < 9; ++t)
            umma_bf16(tmem + q * 48,
                      smem_desc(a0 + s * kTcSlotBytes + (t / 3) * kTcRowBytes + (t % 3) * 16, kTcHalfBytes, 128),
                      smem_desc(b0 + t * kTcBTap, 768, 128), idesc, t > 0 ? 1u : 0u);
          umma_commit(&empty[s]);
          umma_commit(&done[q]);
        }
      }
      if (!ok) give_up();
      umma_commit(drain);  // nothing in flight when TMEM is freed
      if (!mbar_wait_bounded(drain, 0, kTcWait)) atomicExch(&g_conv_status, 2);
    }
    __syncwarp();
  } else {
    // ---- epilogue: warp = TMEM lanes 32 warp .., thread = voxel
    uint32_t k = 0;  // input row of the unit's first
    bool ok = true;
    for (long long u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
      int d, w0, h0, R;
      unit(u, d, w0, h0, R);
      const int w = w0 + tid;
      const uint32_t lanes = (uint32_t)(warp * 32) << 16;
      for (int r = 0; r < R; ++r) {
        // output row r: kh 0 of input row r, kh 1 of r + 1, kh 2 of r + 2 (whose MMAs follow the others')
        const uint32_t k2 = k + r + 2;
        ok = mbar_wait_bounded(&done[k2 % kTcAcc], (k2 / kTcAcc) & 1, kTcWait);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        float v[16], v1[16], v2[16];
        tmem_ld16(tmem + (k + r) % kTcAcc * 48 + 32 + lanes, v);
        tmem_ld16(tmem + (k + r + 1) % kTcAcc * 48 + 16 + lanes, v1);
        tmem_ld16(tmem + k2 % kTcAcc * 48 + lanes, v2);
        tc_fence_before();
        mbar_arrive(&freed[(k + r) % kTcAcc]);
        if (r == R - 1) {  // the unit's last two input rows have no further output row
          mbar_arrive(&freed[(k + r + 1) % kTcAcc]);
          mbar_arrive(&freed[k2 % kTcAcc]);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = v[i] + v1[i] + v2[i];
        if (w < W) {
          const long long vox = ((long long)d * H + (h0 + r)) * W + w;
          if (MODE == 1) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.f);
          } else if (MODE == 2) {
            const uint4* m4 = reinterpret_cast<const uint4*>(aux + vox * 16);
            uint4 mm[2] = {__ldg(m4), __ldg(m4 + 1)};
            const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(mm);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __bfloat162float(mb[i]) > 0.f ? v[i] : 0.f;
          }
          if (OUTF32) {
            float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(y) + vox * 16);
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          } else {
            uint4 pk[2];
            __nv_bfloat162* pb = reinterpret_cast<__nv_bfloat162*>(pk);
#pragma unroll
            for (int i = 0; i < 8; ++i) pb[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(y) + vox * 16);
            o[0] = pk[0];
            o[1] = pk[1];
          }
        }
      }
      k += R + 2;
    }
    if (!ok && lane == 0) give_up();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTcCols);
}

// Weight gradient: dW[t][co][ci] = sum over output voxels v of gy[v][co] *
// x[v + offset(t)][ci]. A work unit is a column segment of some output rows
// (unit_rows) (fixed d, consecutive h) of 64 voxels along W; CTA b takes units b, b +
// grid, ... (fixed), warp w the taps w, w + 4, ...; partial sums per CTA are
// reduced in CTA order. The input rows (d + kd - 1, h') sit in a ring of 4
// slots per kd: a new output row needs 3 new input rows and its gy row, copied
// asynchronously while the row before is multiplied (loading all 9 rows for
// every output row, with nothing in flight meanwhile, took 290 us at 128^3). What
// bounds it now are the ldmatrix reads: 512 shared-memory wavefronts per row
// of 64 voxels against 448 cycles of mma.sync.
constexpr int kWgTapsPerWarp = 7;
constexpr int kWgCtas = 4 * 152;                           // 4 per SM
constexpr int kWgRowBytes = kHaloW * kVoxBytes;            // one staged input row
constexpr int kWgCopies = (3 * kHaloW * 2 + 127) / 128;    // 16-byte copies per thread for the 3 kd rows

__global__ void __launch_bounds__(128, 4) conv3d_wgrad_kernel(int D, int H, int W, int rows, const uint4* __restrict__ x,
                                                              const uint4* __restrict__ gy,
                                                              float* __restrict__ partial) {
  __shared__ __align__(128) unsigned char halo[3 * 4 * kWgRowBytes];  // [kd][slot][voxel][32 B]
  __shared__ __align__(128) unsigned char gsm[2 * kTileW * kVoxBytes];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ntw = (W + kTileW - 1) / kTileW, nseg = (H + rows - 1) / rows;
  const long long nunits = (long long)D * ntw * nseg;
  float acc[kWgTapsPerWarp][2][4];
#pragma unroll
  for (int i = 0; i < kWgTapsPerWarp; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;
  // ldmatrix.trans roles. A = gy^T (16 out x 16 voxels) from gsm [voxel][co]:
  // matrix q holds voxels 8*(q >> 1).., channels 8*(q & 1)..
  const int ga_row = (lane & 7) + 8 * (lane >> 4), ga_chunk = (lane >> 3) & 1;
  // B = x (16 voxels x 8 in) from the halo [voxel][ci]: matrix q holds
  // voxels 8*(q & 1).., channels 8*(q >> 1)..
  const int xb_row = (lane & 7) + 8 * ((lane >> 3) & 1), xb_chunk = lane >> 4;
  const uint32_t hbase = smem_addr(halo), gbase = smem_addr(gsm);
  for (long long u = blockIdx.x; u < nunits; u += gridDim.x) {
    const int hs = (int)(u % nseg);
    const long long dw = u / nseg;
    const int wt = (int)(dw % ntw), d = (int)(dw / ntw);
    const int w0 = wt * kTileW, h0 = hs * rows, h1 = min(H, h0 + rows);
    // this thread's copies of an input row set: source (without the row) and slot offset
    long long xoff[kWgCopies];
    int soff[kWgCopies];
#pragma unroll
    for (int i = 0; i < kWgCopies; ++i) {
      const int q = tid + 128 * i, kd = q / (kHaloW * 2), j = (q >> 1) % kHaloW, c = q & 1;
      const int di = d + kd - 1, wi = w0 - 1 + j;
      soff[i] = q < 3 * kHaloW * 2 ? kd * 4 * kWgRowBytes + (int)swz(j, c) : -1;
      xoff[i] = di >= 0 && di < D && wi >= 0 && wi < W ? ((long long)di * H * W + wi) * 2 + c : -1;
    }
    auto load_x = [&](int hr) {  // the 3 kd rows (d + kd - 1, hr) into slot hr mod 4, zero outside the volume
      const bool hin = hr >= 0 && hr < H;
#pragma unroll
      for (int i = 0; i < kWgCopies; ++i)
        if (soff[i] >= 0) {
          const bool in = hin && xoff[i] >= 0;
          cp_async16_zfill(hbase + (hr & 3) * kWgRowBytes + soff[i], in ? x + xoff[i] + (long long)hr * W * 2 : x, in);
        }
    };
    auto load_g = [&](int h) {
      const int c = tid & 1, j = tid >> 1, w = w0 + j;
      const bool in = w < W;
      cp_async16_zfill(gbase + (h & 1) * kTileW * kVoxBytes + swz(j, c), in ? gy + (((long long)d * H + h) * W + w) * 2 + c : gy, in);
    };
    load_x(h0 - 1);
    load_x(h0);
    load_x(h0 + 1);
    load_g(h0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int h = h0; h < h1; ++h) {
      if (h + 1 < h1) {
        load_x(h + 2);
        load_g(h + 1);
      }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      const uint32_t gb = gbase + (h & 1) * kTileW * kVoxBytes;
#pragma unroll
      for (int ks = 0; ks < kTileW / 16; ++ks) {
        uint32_t a0, a1, a2, a3;
        ldsm_x4_t(gb + swz(ks * 16 + ga_row, ga_chunk), a0, a1, a2, a3);
        // A fragment order: (co 0-7, v 0-7), (co 8-15, v 0-7), (co 0-7, v 8-15), (co 8-15, v 8-15)
        // = stored blocks (v lo, c lo), (v lo, c hi), (v hi, c lo), (v hi, c hi): a0, a1, a2, a3
#pragma unroll
        for (int i = 0; i < kWgTapsPerWarp; ++i) {
          const int t = warp + 4 * i;
          if (t < kTaps) {
            const int kd = t / 9, kh = t / 3 % 3, kw = t % 3;
            uint32_t b0, b1, b2, b3;
            ldsm_x4_t(hbase + (kd * 4 + ((h + kh - 1) & 3)) * kWgRowBytes + swz(ks * 16 + kw + xb_row, xb_chunk), b0, b1, b2,
                      b3);
            // b0: (v lo, ci lo), b1: (v hi, ci lo), b2: (v lo, ci hi), b3: (v hi, ci hi)
            mma_bf16(acc[i][0], a0, a1, a2, a3, b0, b1);
            mma_bf16(acc[i][1], a0, a1, a2, a3, b2, b3);
          }
        }
      }
      __syncthreads();  // the row's slots have been read before the copies of the next step
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  const int gid = lane >> 2, tig = lane & 3;
  float* dst = partial + (long long)blockIdx.x * kTaps * 256;
#pragma unroll
  for (int i = 0; i < kWgTapsPerWarp; ++i) {
    const int t = warp + 4 * i;
    if (t >= kTaps) continue;
#pragma unroll
    for (int ch = 0; ch < 2; ++ch)
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int co = gid + 8 * hr, ci = ch * 8 + 2 * tig;
        *reinterpret_cast<float2*>(dst + t * 256 + co * 16 + ci) = make_float2(acc[i][ch][2 * hr], acc[i][ch][2 * hr + 1]);
      }
  }
}

// Sum of the CTAs' parts in order: thread (range r of 8, value) sums its
// range's parts, then the ranges are added in order. One chain of all parts
// per value took 28 us for 608 parts.
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ partial, int nparts,
                                                           float* __restrict__ dw) {
  __shared__ float rs[8][32];
  const int v = threadIdx.x & 31, r = threadIdx.x >> 5, i = blockIdx.x * 32 + v;
  const int b0 = (int)((long long)nparts * r / 8), b1 = (int)((long long)nparts * (r + 1) / 8);
  float s = 0.f;
#pragma unroll 8
  for (int b = b0; b < b1; ++b) s += partial[(long long)b * kTaps * 256 + i];
  rs[r][v] = s;
  __syncthreads();
  if (r == 0) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += rs[k][v];
    dw[i] = s;
  }
}

// complex64 [V] * scale -> bf16 [V][16]: channels 0, 1 = re, im rounded to
// bf16; with hilo, channels 2, 3 = the rounding remainders (a two-term bf16
// split carrying 16 mantissa bits); the rest 0
__global__ void pack_c64_kernel(const float2* __restrict__ z, long long nvox, const float* __restrict__ scale,
                                int hilo, uint4* __restrict__ out) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nvox) return;
  const float s = scale ? *scale : 1.f;
  const float2 a = z[v];
  const float re = a.x * s, im = a.y * s;
  const __nv_bfloat162 p = __floats2bfloat162_rn(re, im);
  uint32_t q = 0u;
  if (hilo) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(re - __bfloat162float(p.x), im - __bfloat162float(p.y));
    q = *reinterpret_cast<const uint32_t*>(&r);
  }
  out[2 * v] = make_uint4(*reinterpret_cast<const uint32_t*>(&p), q, 0u, 0u);
  out[2 * v + 1] = make_uint4(0u, 0u, 0u, 0u);
}

// float32 [V][16] channels 0, 1 -> complex64 [V]: out = scale * y + skip * z
__global__ void unpack_c64_kernel(const float* __restrict__ y, const float2* __restrict__ z, long long nvox,
                                  const float* __restrict__ scale, float skip, float2* __restrict__ out) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nvox) return;
  const float s = scale ? *scale : 1.f;
  const float2 a = *reinterpret_cast<const float2*>(y + v * 16);
  float2 r = make_float2(a.x * s, a.y * s);
  if (z) {
    const float2 b = z[v];
    r.x = fmaf(skip, b.x, r.x);
    r.y = fmaf(skip, b.y, r.y);
  }
  out[v] = r;
}

int check_conv(const tlgb_conv3d_desc* d) {
  if (!d) TLGB_FAIL(TLGB_ERR_INVALID, "null conv descriptor");
  if (d->D < 1 || d->H < 1 || d->W < 1) TLGB_FAIL(TLGB_ERR_INVALID, "conv3d: spatial sizes must be >= 1");
  if (d->H > 65535 || d->D > 65535) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "conv3d: D and H must be <= 65535");
  if (d->cin != 16 || d->cout != 16) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "conv3d: 16 input and 16 output channels (pad)");
  if (d->mode < 0 || d->mode > 2) TLGB_FAIL(TLGB_ERR_INVALID, "conv3d: unknown epilogue mode");
  return TLGB_OK;
}

// Output rows per work unit. A unit of R rows reads R + 2, and a persistent
// grid takes cdiv(units, CTAs) units one after the other, so R is the one with
// the least product: fixed units of 16 rows of 128^3 are 3.4 per CTA, whose last
// round three CTAs in five sit out (72 row steps; 63 with 19 rows: 77 -> 72.5 us,
// weight gradient 94 -> 91), and leave most SMs idle on small volumes.
int unit_rows(long long planes, int H, long long ctas) {
  int best = H;
  long long least = cdiv(planes, ctas) * (H + 2);
  for (int seg = 2; seg <= std::min(H, 256); ++seg) {
    const int r = (int)cdiv(H, seg);
    const long long steps = cdiv(planes * cdiv(H, r), ctas) * (r + 2);
    if (steps < least) least = steps, best = r;
  }
  return best;
}

template <int MODE, bool OUTF32>
int launch_conv_tc(const tlgb_conv3d_desc* d, const void* x, const void* w, const void* aux, void* y, cudaStream_t s) {
  auto* k = conv3d_tc_kernel<MODE, OUTF32>;
  TLGB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
  const long long planes = (long long)d->D * ((d->W + kTcM - 1) / kTcM), ctas = (long long)kTcCtas * sm_count();
  const int rows = unit_rows(planes, d->H, ctas);
  const unsigned grid = (unsigned)std::min<long long>(planes * cdiv(d->H, rows), ctas);
  k<<<grid, kTcThreads, kTcSmem, s>>>(d->D, d->H, d->W, rows, (const uint4*)x, (const uint4*)w, (const __nv_bfloat16*)aux, y);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

int wgrad_parts(const tlgb_conv3d_desc* d, int* rows) {
  const long long planes = (long long)d->D * ((d->W + kTileW - 1) / kTileW);
  *rows = unit_rows(planes, d->H, kWgCtas);
  return (int)std::min<long long>(planes * cdiv(d->H, *rows), kWgCtas);
}

}  // namespace
}  // namespace tlgb

using namespace tlgb;

extern "C" int tlgb_conv3d_fwd(const tlgb_conv3d_desc* d, const void* x, const void* w, const void* aux, void* y,
                               tlgb_stream_t stream) {
  TLGB_TRY(check_conv(d));
  if (!x || !w || !y || (d->mode == 2 && !aux)) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)aux) & 15)
    TLGB_FAIL(TLGB_ERR_INVALID, "conv3d: buffers must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  if (d->out_f32) {
    if (d->mode == 0) return launch_conv_tc<0, true>(d, x, w, aux, y, s);
    if (d->mode == 1) return launch_conv_tc<1, true>(d, x, w, aux, y, s);
    return launch_conv_tc<2, true>(d, x, w, aux, y, s);
  }
  if (d->mode == 0) return launch_conv_tc<0, false>(d, x, w, aux, y, s);
  if (d->mode == 1) return launch_conv_tc<1, false>(d, x, w, aux, y, s);
  return launch_conv_tc<2, false>(d, x, w, aux, y, s);
}

extern "C" int tlgb_conv3d_wgrad_scratch_size(const tlgb_conv3d_desc* d, size_t* bytes) {
  TLGB_TRY(check_conv(d));
  if (!bytes) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  int rows = 0;
  *bytes = (size_t)wgrad_parts(d, &rows) * kTaps * 256 * sizeof(float);
  return TLGB_OK;
}

extern "C" int tlgb_conv3d_wgrad(const tlgb_conv3d_desc* d, const void* x, const void* gy, float* dw, void* scratch,
                                 size_t scratch_bytes, tlgb_stream_t stream) {
  TLGB_TRY(check_conv(d));
  if (!x || !gy || !dw || !scratch) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  if (((uintptr_t)x | (uintptr_t)gy | (uintptr_t)scratch) & 15)
    TLGB_FAIL(TLGB_ERR_INVALID, "conv3d: buffers must be 16-byte aligned");
  size_t need = 0;
  TLGB_TRY(tlgb_conv3d_wgrad_scratch_size(d, &need));
  if (scratch_bytes < need) TLGB_FAIL(TLGB_ERR_WORKSPACE, "conv3d wgrad scratch too small");
  cudaStream_t s = (cudaStream_t)stream;
  int rows = 0;
  const int parts = wgrad_parts(d, &rows);
  conv3d_wgrad_kernel<<<parts, 128, 0, s>>>(d->D, d->H, d->W, rows, (const uint4*)x, (const uint4*)gy, (float*)scratch);
  TLGB_CHECK_LAUNCH();
  static_assert(kTaps * 256 % 32 == 0, "32 values per CTA");
  wgrad_reduce_kernel<<<kTaps * 256 / 32, 256, 0, s>>>((const float*)scratch, parts, dw);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

extern "C" int tlgb_conv3d_pack(const void* z, int64_t nvox, const float* scale, int32_t hilo, void* out,
                                tlgb_stream_t stream) {
  if (nvox < 0 || (nvox > 0 && (!z || !out))) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer or negative size");
  if (nvox == 0) return TLGB_OK;
  if ((uintptr_t)out & 15) TLGB_FAIL(TLGB_ERR_INVALID, "pack: output must be 16-byte aligned");
  pack_c64_kernel<<<(unsigned)cdiv(nvox, 256), 256, 0, (cudaStream_t)stream>>>((const float2*)z, nvox, scale, hilo,
                                                                               (uint4*)out);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

extern "C" int tlgb_conv3d_unpack(const float* y, const void* z, int64_t nvox, const float* scale, float skip,
                                  void* out, tlgb_stream_t stream) {
  if (nvox < 0 || (nvox > 0 && (!y || !out))) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer or negative size");
  if (nvox == 0) return TLGB_OK;
  unpack_c64_kernel<<<(unsigned)cdiv(nvox, 256), 256, 0, (cudaStream_t)stream>>>(y, (const float2*)z, nvox, scale,
                                                                                 skip, (float2*)out);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

namespace tlgb {
int conv_device_status(int* v, int clear) {
  int x = 0;
  TLGB_CUDA(cudaMemcpyFromSymbol(&x, g_conv_status, sizeof(int)));
  if (clear) {
    const int z = 0;
    TLGB_CUDA(cudaMemcpyToSymbol(g_conv_status, &z, sizeof(int)));
  }
  *v = x;
  return TLGB_OK;
}
}  // namespace tlgb
