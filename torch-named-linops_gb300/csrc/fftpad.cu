// Centred-FFT shifts folded into the pad and crop of the NUFFT chain, with
// the apodization and (for SENSE) the coil sensitivities fused in.
//
// The reference's NUFFT is Apodize -> Pad -> cfftn -> Interpolate, with
// cfftn = fftshift . fftn . ifftshift (linops/nufft.py:170-184,
// utils/_fft.py:7-60). Each shift is a full-grid pass. Here:
//   ifftshift(Pad(a x))[j] = a[i] x[i], i = (j + floor(Np/2)) mod Np - off
// is one gather (tlgb_pad_shift), and the k-space fftshift is a modulation
// of the same gather's output:
//   fftshift(fftn(z)) = fftn(z . m),  m[j] = prod_e exp(2 pi i j_e h_e / Np_e),
//   h_e = floor(Np_e / 2),
// which for even Np_e is the sign (-1)^j_e (exact). So an uncentred fftn of
// the gather's output is the reference's centred k-space, read at the
// reference's own interpolation coordinates. On the way back,
//   Crop(fftshift(ifftn(ifftshift(G))))[i] = conj(m[j]) ifftn(G)[j],
//   j = (i + off - floor(Np/2)) mod Np,
// is one gather (tlgb_crop_shift), which can also apply the conjugate coil
// maps, the coil sum and an axpy.

#include <algorithm>

#include "common.cuh"

namespace tlgb {
namespace {

struct PadGeo {
  int n[3], np[3], off[3], sh[3];  // internal dims padded to 3 (leading 1s)
  long long nvol, npvol;
  int modulate;  // multiply by m[j] (pad) / conj(m[j]) (crop)
};

// m[j] of the uncentred index j: a sign for even extents, a phase otherwise
__device__ __forceinline__ float2 modulation(const PadGeo& G, int j0, int j1, int j2) {
  const int j[3] = {j0, j1, j2};
  int sign = 0;
  float ph = 0.f;  // in units of pi
  bool odd = false;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if ((G.np[e] & 1) == 0) {
      sign ^= j[e] & 1;
    } else {
      odd = true;
      // 2 j h / Np with h = floor(Np / 2), reduced mod 2 in integers first
      ph += (float)((2ll * j[e] * (G.np[e] / 2)) % (2ll * G.np[e])) / (float)G.np[e];
    }
  }
  float c = 1.f, s = 0.f;
  if (odd) sincospif(ph, &s, &c);
  return sign ? make_float2(-c, -s) : make_float2(c, s);
}

// Rounded as written, so that an entry's result does not depend on the kernel
// that its batch's size takes.
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}

// row and column indices of voxel v of a volume with last extents n1, n2
__device__ __forceinline__ void split_index(long long v, long long vol, int n1, int n2, int& i0, int& i1, int& i2) {
  if (vol <= 0xffffffffll) {  // 32-bit divisions wherever the volume allows them
    const unsigned u = (unsigned)v, r = u / (unsigned)n2;
    i2 = (int)(u - r * (unsigned)n2);
    i0 = (int)(r / (unsigned)n1);
    i1 = (int)(r - (unsigned)i0 * (unsigned)n1);
  } else {
    const long long r = v / n2;
    i2 = (int)(v - r * n2);
    i0 = (int)(r / n1);
    i1 = (int)(r - (long long)i0 * n1);
  }
}

// Both kernels move a voxel of many batch entries per thread and are bound by
// memory. One thread per voxel that walks the whole batch leaves one load in
// flight per thread and too few CTAs for a 2D grid (256 entries of 256^2 in
// 320^2: 400 CTAs, 165 us to pad and 137 us to crop, 2.1 and 2.5 TB/s), so the
// batch is cut into blockIdx.y runs (batch_runs) and kBatchAhead loads are
// issued before the first store: 56 and 42 us, 6.1 and 6.4 TB/s.
constexpr int kBatchAhead = 8;
// With coil maps a pad reads its map and writes 1.95 times as much for each
// entry, and more resident threads serve it better than more loads each: 8
// coils on 160^3 take 83, 86, 87 and 97 us (with the call) at 1, 2, 4 and 8
// ahead. The crop, whose coils are a sum, keeps 8: 32 coils on 320^2 take 22, 31,
// 19 and 16 us, 8 coils on 160^3 63-68.
constexpr int kMapsPadAhead = 1;
// Fewer entries (or coils of a crop) than 8 are not worth the registers of the
// loads that never come. 205^3 in 256^3: one entry 165 us to pad and 161 to crop
// with 8 ahead, 104 and 65 with one; three entries 180 and 184, 137 and 89 with 4.
// 3 coils of 128^3, two entries: 67, 48 and 45 us with 8, 4 and one.
int ahead(long long n, int four_from) { return n >= kBatchAhead ? kBatchAhead : (n >= four_from ? 4 : 1); }

// out[e][j] = maps[e % C][i] * apod[i] * x[e / C][i] for the source i of j, else 0
template <bool MAPS, int AH>
__global__ void __launch_bounds__(256) pad_shift_kernel(PadGeo G, const float2* __restrict__ x, long long nent, long long run,
                                                        const float* __restrict__ apod, const float2* __restrict__ maps,
                                                        int nmaps, float2* __restrict__ out) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= G.npvol) return;
  int j0, j1, j2;
  split_index(j, G.npvol, G.np[1], G.np[2], j0, j1, j2);
  int i0 = j0 + G.sh[0], i1 = j1 + G.sh[1], i2 = j2 + G.sh[2];  // shifts are below the extents
  i0 -= (i0 >= G.np[0] ? G.np[0] : 0) + G.off[0];
  i1 -= (i1 >= G.np[1] ? G.np[1] : 0) + G.off[1];
  i2 -= (i2 >= G.np[2] ? G.np[2] : 0) + G.off[2];
  const bool in = i0 >= 0 && i0 < G.n[0] && i1 >= 0 && i1 < G.n[1] && i2 >= 0 && i2 < G.n[2];
  const long long i = in ? ((long long)i0 * G.n[1] + i1) * G.n[2] + i2 : 0;
  const float a = (in && apod) ? apod[i] : 1.f;
  const float2 md = (in && G.modulate) ? modulation(G, j0, j1, j2) : make_float2(1.f, 0.f);
  const long long e0 = blockIdx.y * run, e1 = min(nent, e0 + run);
  long long b = MAPS ? e0 / nmaps : e0;
  int c = MAPS ? (int)(e0 - b * nmaps) : 0;
  for (long long e = e0; e < e1; e += AH) {
    float2 v[AH];
#pragma unroll
    for (int u = 0; u < AH; ++u) {
      v[u] = make_float2(0.f, 0.f);
      if (!in || e + u >= e1) continue;
      const float2 q = x[b * G.nvol + i];
      v[u] = make_float2(__fmul_rn(q.x, a), __fmul_rn(q.y, a));
      if (MAPS) v[u] = cmul(maps[c * G.nvol + i], v[u]);
      if (!MAPS || ++c == nmaps) {
        c = 0;
        ++b;
      }
    }
#pragma unroll
    for (int u = 0; u < AH; ++u) {
      if (e + u >= e1) break;
      out[(e + u) * G.npvol + j] = in && G.modulate ? cmul(v[u], md) : v[u];
    }
  }
}

// out[b][i] = alpha * apod[i] * sum_c conj(maps[c][i]) z[(b*C + c)][src(i)] + beta * add[b][i]
template <bool MAPS, int AH>
__global__ void __launch_bounds__(256) crop_shift_kernel(PadGeo G, const float2* __restrict__ z, long long nbatch,
                                                         long long run, const float* __restrict__ apod,
                                                         const float2* __restrict__ maps, int nmaps, float alpha,
                                                         const float2* __restrict__ add, float beta,
                                                         float2* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= G.nvol) return;
  int i0, i1, i2;
  split_index(i, G.nvol, G.n[1], G.n[2], i0, i1, i2);
  int j0 = i0 + G.off[0] - G.sh[0], j1 = i1 + G.off[1] - G.sh[1], j2 = i2 + G.off[2] - G.sh[2];
  j0 += j0 < 0 ? G.np[0] : 0;  // off + n fits in Np, so one extent is enough
  j1 += j1 < 0 ? G.np[1] : 0;
  j2 += j2 < 0 ? G.np[2] : 0;
  const long long j = ((long long)j0 * G.np[1] + j1) * G.np[2] + j2;
  const float a = (apod ? apod[i] : 1.f) * alpha;
  float2 md = make_float2(1.f, 0.f);
  if (G.modulate) {
    md = modulation(G, j0, j1, j2);
    md.y = -md.y;  // conj(m[j])
  }
  const long long b0 = blockIdx.y * run, b1 = min(nbatch, b0 + run);
  constexpr int UB = MAPS ? 1 : AH, UC = MAPS ? AH : 1;  // coils ahead, or entries ahead
  const int C = MAPS ? nmaps : 1;
  for (long long b = b0; b < b1; b += UB) {
    float2 s[UB];
#pragma unroll
    for (int u = 0; u < UB; ++u) s[u] = make_float2(0.f, 0.f);
    for (int c = 0; c < C; c += UC) {
      float2 v[UB * UC], m[UC];
#pragma unroll
      for (int u = 0; u < UB * UC; ++u) {
        const bool live = MAPS ? c + u < C : b + u < b1;
        v[u] = live ? z[(MAPS ? b * C + c + u : b + u) * G.npvol + j] : make_float2(0.f, 0.f);
        if (MAPS) m[u] = live ? maps[(long long)(c + u) * G.nvol + i] : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < UB * UC; ++u) {
        if (MAPS && c + u >= C) break;
        if (G.modulate) v[u] = cmul(v[u], md);
        if (MAPS) {  // conj(m) * v
          s[0].x = __fadd_rn(s[0].x, fmaf(m[u].x, v[u].x, __fmul_rn(m[u].y, v[u].y)));
          s[0].y = __fadd_rn(s[0].y, fmaf(m[u].x, v[u].y, -__fmul_rn(m[u].y, v[u].x)));
        } else {
          s[u] = v[u];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < UB; ++u) {
      if (b + u >= b1) break;
      float2 o = make_float2(__fmul_rn(a, s[u].x), __fmul_rn(a, s[u].y));
      if (add) {
        const float2 q = add[(b + u) * G.nvol + i];
        o.x = fmaf(beta, q.x, o.x);
        o.y = fmaf(beta, q.y, o.y);
      }
      out[(b + u) * G.nvol + i] = o;
    }
  }
}

// Entries per blockIdx.y: whole groups of `ahead`, in as many runs as it
// takes for 16 CTAs per SM (8 fit at a time) where the volume alone has fewer.
long long batch_runs(long long ctas, long long nent, int ahead, unsigned& gy) {
  const long long groups = cdiv(nent, ahead);
  const long long want = std::min<long long>(std::max<long long>(cdiv(16ll * sm_count(), ctas), 1), std::min<long long>(groups, 65535));
  const long long run = cdiv(groups, want) * ahead;
  gy = (unsigned)cdiv(nent, run);
  return run;
}

int make_pad_geo(int32_t ndim, const int64_t* n, const int64_t* np, const int64_t* off, const int64_t* shift,
                 int32_t modulate, PadGeo& G) {
  G.modulate = modulate ? 1 : 0;
  if (ndim < 1 || ndim > 3 || !n || !np || !off || !shift) TLGB_FAIL(TLGB_ERR_INVALID, "pad/crop: bad dims");
  G.nvol = G.npvol = 1;
  for (int e = 0; e < 3; ++e) {
    const int a = e - (3 - ndim);
    const int64_t ne = a >= 0 ? n[a] : 1, pe = a >= 0 ? np[a] : 1, oe = a >= 0 ? off[a] : 0, se = a >= 0 ? shift[a] : 0;
    if (ne < 1 || pe < ne || oe < 0 || oe + ne > pe || pe >= (1ll << 30) || se < 0 || se >= pe)
      TLGB_FAIL(TLGB_ERR_INVALID, "pad/crop: sizes, offsets or shifts out of range");
    G.n[e] = (int)ne;
    G.np[e] = (int)pe;
    G.off[e] = (int)oe;
    G.sh[e] = (int)se;
    // one thread per padded voxel: grid x below 2^31 CTAs of 256
    if (G.npvol > ((1ll << 38) - 1) / pe)
      TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "pad/crop: padded volume too large for one launch");
    G.nvol *= ne;
    G.npvol *= pe;
  }
  return TLGB_OK;
}

}  // namespace
}  // namespace tlgb

using namespace tlgb;

extern "C" int tlgb_pad_shift_c64(const void* x, int64_t nbatch, int32_t ndim, const int64_t* n, const int64_t* np,
                                  const int64_t* off, const int64_t* shift, int32_t modulate, const float* apod,
                                  const void* maps, int32_t nmaps, void* out, tlgb_stream_t stream) {
  PadGeo G;
  TLGB_TRY(make_pad_geo(ndim, n, np, off, shift, modulate, G));
  if (nbatch < 0 || (maps && nmaps < 1)) TLGB_FAIL(TLGB_ERR_INVALID, "pad_shift: bad batch or map count");
  if (nbatch == 0) return TLGB_OK;
  if (!x || !out) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  const long long nent = (long long)nbatch * (maps ? nmaps : 1), ctas = cdiv(G.npvol, 256);
  dim3 grid((unsigned)ctas);
  const int ah = maps ? kMapsPadAhead : ahead(nent, 3);
  const long long run = batch_runs(ctas, nent, ah, grid.y);
  auto* k = maps ? pad_shift_kernel<true, kMapsPadAhead>
                 : (ah == 1 ? pad_shift_kernel<false, 1> : (ah == 4 ? pad_shift_kernel<false, 4> : pad_shift_kernel<false, kBatchAhead>));
  k<<<grid, 256, 0, (cudaStream_t)stream>>>(
      G, (const float2*)x, nent, run, apod, (const float2*)maps, nmaps, (float2*)out);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

extern "C" int tlgb_crop_shift_c64(const void* z, int64_t nbatch, int32_t ndim, const int64_t* n, const int64_t* np,
                                   const int64_t* off, const int64_t* shift, int32_t modulate, const float* apod,
                                   const void* maps, int32_t nmaps, float alpha, const void* add, float beta,
                                   void* out, tlgb_stream_t stream) {
  PadGeo G;
  TLGB_TRY(make_pad_geo(ndim, n, np, off, shift, modulate, G));
  if (nbatch < 0 || (maps && nmaps < 1)) TLGB_FAIL(TLGB_ERR_INVALID, "crop_shift: bad batch or map count");
  if (nbatch == 0) return TLGB_OK;
  if (!z || !out) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  const long long ctas = cdiv(G.nvol, 256);
  dim3 grid((unsigned)ctas);
  const int ah = maps ? ahead(nmaps, 4) : ahead(nbatch, 3);
  const long long run = batch_runs(ctas, nbatch, maps ? 1 : ah, grid.y);
  auto* k = maps ? (ah == 1 ? crop_shift_kernel<true, 1> : (ah == 4 ? crop_shift_kernel<true, 4> : crop_shift_kernel<true, kBatchAhead>))
                 : (ah == 1 ? crop_shift_kernel<false, 1> : (ah == 4 ? crop_shift_kernel<false, 4> : crop_shift_kernel<false, kBatchAhead>));
  k<<<grid, 256, 0, (cudaStream_t)stream>>>(
      G, (const float2*)z, nbatch, run, apod, (const float2*)maps, nmaps, alpha, (const float2*)add, beta, (float2*)out);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}
