// Kaiser-Bessel / spline interpolation (ungrid), gridding (adjoint) and the
// trajectory gradient, 1D-3D, for sm_103a.
//
// Replaces the reference's Triton kernels _ungrid{1,2,3}d (functional/_interp/
// ungrid.py:162-503) and _grid{1,2,3}d (grid.py:169-513); the arithmetic of a
// tap follows the reference's pure-torch path (ungrid_torch ungrid.py:624-684,
// grid_torch grid.py:571-639, weights_torch kernels.py:108-147,
// kaiser_bessel_torch kernels.py:28-89) operation for operation in float32.
//
// Design (GB300 first, not a translation of the Triton programs):
//  * Plan (once per trajectory, built on the device): every point is paired with
//    each output tile that its valid taps touch, "home" pairs (the tile holding
//    the first of them) first, and, for separable complex 2D and 3D geometries,
//    with each output block; both lists are sorted by a stable radix sort and cut
//    into work items. Such a plan also holds the points' tap weights: records in
//    the gather's order and rows over the blocks.
//  * Ungridding of complex values (gather_kernel): persistent CTAs whose producer
//    warps fill a ring of tile regions, a group of batch entries each, while the
//    consumer warps interpolate the tile's home points from the records.
//  * Gridding of complex values (adj_b3_kernel, adj_bn_kernel): a warp owns an
//    output block in registers and adds the entries of the block's list in order
//    as rank-8 updates on the tensor cores. Deterministic, no global atomics: every
//    cell is summed by one warp in plan order and written once; dense blocks are
//    split, their parts added in order by a second kernel.
//  * Real values, the radial norm, 1D and the widest kernels run on one-tile CTAs
//    (interp_fwd_kernel, interp_adj_kernel) that evaluate the weights themselves,
//    by the reference's A&S formula; nothing reads the kernel from a lookup table,
//    which would add an interpolation error on top of the 1e-5 budget.

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "sm100.cuh"

namespace tlgb {
namespace {

constexpr int NTMAX = 16;  // taps per dimension supported (width < 15)
constexpr int NWARP = 8;   // warps per CTA
constexpr int NTHR = 32 * NWARP;
constexpr int CGMAX = 8;   // batch entries per coil group

struct Geo {
  int ndim;
  int N[3];   // internal dims (x, y, z); leading inactive dims have N = 1
  int T[3];   // tile edge
  int lgT[3]; // log2 of the tile edge, -1 when it is no power of two
  int nt[3];  // tiles per dim
  int NT[3];  // taps per dim (inactive: 1)
  float r[3]; // kernel radius W/2 per dim
  float rinv[3];  // 1/r, used when r is a power of two (the product is then exact)
  int rpow2[3];
  int act[3];
  int kernel, norm, pad, cplx;
  float beta, beta_lo;  // beta_lo: what rounding beta to float32 left (0 unless the caller gives it)
  long long npts, nbatch;
  int wrap_safe;  // every active N >= NT: a window never overlaps itself
  long long tv_off;  // gridding: byte offset in scratch of the point-major values, -1 = none
  // test hook of the gather and the 2D gradient (tlgb_test_skip_region_copy): 1 = nothing is copied and the
  // consumers' waits run out, 2 = they run out while copies are under way
  int skip_copy;
  uint32_t wait;     // polls of the consumers' bounded waits, kWaitLimit without the hook
  int nrow;          // block lists: blocks a window can meet per dim (2 or 3), 0 = no block lists
};

// ---------------------------------------------------------------- kernels math

// A&S 9.8.1 / 9.8.2 coefficients (the reference's kernels.py:65-88)
__device__ __forceinline__ float kb_value(float x, float beta) {
  const float z = beta * __fsqrt_rn(__fsub_rn(1.0f, __fmul_rn(x, x)));
  const float t = __fdiv_rn(z, 3.75f);
  const float t2 = t * t;
  if (z < 3.75f) {
    const float t4 = t2 * t2, t6 = t4 * t2, t8 = t4 * t4, t10 = t6 * t4, t12 = t6 * t6;
    return 1.0f + 3.5156229f * t2 + 3.0899424f * t4 + 1.2067492f * t6 + 0.2659732f * t8 + 0.0360768f * t10 +
           0.0045813f * t12;
  }
  const float t3 = t2 * t, t4 = t2 * t2, t5 = t3 * t2, t6 = t4 * t2, t7 = t5 * t2, t8 = t4 * t4;
  const float poly = 0.39894228f + __fdiv_rn(0.01328592f, t) + __fdiv_rn(0.00225319f, t2) -
                     __fdiv_rn(0.00157565f, t3) + __fdiv_rn(0.00916281f, t4) - __fdiv_rn(0.02057706f, t5) +
                     __fdiv_rn(0.02635537f, t6) - __fdiv_rn(0.01647633f, t7) + __fdiv_rn(0.00392377f, t8);
  return __fdiv_rn(expf(z), __fsqrt_rn(z)) * poly;
}

// d KB(x) / dx of the same A&S expressions (x signed, |x| <= 1)
__device__ __forceinline__ float kb_deriv(float x, float beta) {
  const float z = beta * __fsqrt_rn(__fsub_rn(1.0f, __fmul_rn(x, x)));
  const float b2 = beta * beta;
  if (z < 3.75f) {
    const float u = (z / 3.75f) * (z / 3.75f);
    // P(u) = 1 + a1 u + ... + a6 u^6 ; P'(u)
    const float dp = 3.5156229f + u * (2.f * 3.0899424f + u * (3.f * 1.2067492f + u * (4.f * 0.2659732f +
                     u * (5.f * 0.0360768f + u * (6.f * 0.0045813f)))));
    return -2.0f * b2 * x * dp / (3.75f * 3.75f);
  }
  const float v = 3.75f / z;
  const float q = 0.39894228f + v * (0.01328592f + v * (0.00225319f + v * (-0.00157565f + v * (0.00916281f +
                  v * (-0.02057706f + v * (0.02635537f + v * (-0.01647633f + v * 0.00392377f)))))));
  const float dq = 0.01328592f + v * (2.f * 0.00225319f + v * (3.f * -0.00157565f + v * (4.f * 0.00916281f +
                   v * (5.f * -0.02057706f + v * (6.f * 0.02635537f + v * (7.f * -0.01647633f +
                   v * (8.f * 0.00392377f)))))));
  const float e = expf(z) / sqrtf(z);
  const float dI = e * (q * (1.0f - 0.5f / z) - dq * 3.75f / (z * z));
  return dI * (-b2 * x / z);
}

__device__ __forceinline__ float kern_value(int kernel, float ax, float beta) {
  return kernel == TLGB_KERNEL_KAISER_BESSEL ? kb_value(ax, beta) : fmaxf(1.0f - ax, 0.0f);
}

__device__ __forceinline__ float kern_deriv(int kernel, float d, float beta) {
  if (kernel == TLGB_KERNEL_KAISER_BESSEL) return kb_deriv(d, beta);
  return (fabsf(d) < 1.0f) ? (d > 0.f ? -1.0f : (d < 0.f ? 1.0f : 0.0f)) : 0.0f;
}

__device__ __forceinline__ bool coord_ok(float x) { return isfinite(x) && fabsf(x) < 16777216.0f; }

// One tap of one dimension: the reference's dlocs = (locs - grid_locs) / radius
// and its validity (kernels.py:126-146).
struct Tap {
  float d;     // signed normalised offset
  bool valid;
};

__device__ __forceinline__ Tap tap_eval(const Geo& g, int e, float x, int lower, int k) {
  Tap t;
  const float gk = (float)(lower + k);
  const float diff = __fsub_rn(x, gk);
  t.d = g.rpow2[e] ? __fmul_rn(diff, g.rinv[e]) : __fdiv_rn(diff, g.r[e]);
  const float ad = fabsf(t.d);
  bool v = ad <= g.r[e];
  if (g.kernel == TLGB_KERNEL_KAISER_BESSEL) v = v && (ad <= 1.0f);
  if (g.pad == TLGB_PAD_ZERO) v = v && (lower + k >= 0) && (lower + k < g.N[e]);
  t.valid = v;
  return t;
}

__device__ __forceinline__ int lower_of(const Geo& g, int e, float x) {
  return (int)ceilf(__fsub_rn(x, g.r[e]));
}

__device__ __forceinline__ int wrapi(int v, int n) {
  if (v >= 0 && v < n) return v;
  int m = v % n;
  return m < 0 ? m + n : m;
}

__device__ __forceinline__ float load_coord(const Geo& g, const float* locs, long long p, int e) {
  return __ldg(locs + p * g.ndim + (e - (3 - g.ndim)));
}

// --------------------------------------------------------------------- plan

__device__ __forceinline__ int tile_of(const Geo& g, int e, int v) {
  return g.lgT[e] >= 0 ? v >> g.lgT[e] : v / g.T[e];
}

// Distinct tiles touched along one dim by taps start .. start+n-1 (wrapped);
// the first is the home tile. At most 3 (a window crossing a ragged last tile
// and the wrap), see max_tiles_per_dim on the host.
__device__ __forceinline__ int axis_tiles(const Geo& g, int e, int start, int n, int* tl) {
  int cnt = 0;
  for (int k = 0; k < n; ++k) {
    int v = start + k;
    if (g.pad == TLGB_PAD_CIRCULAR) v = wrapi(v, g.N[e]);
    const int t = tile_of(g, e, v);
    bool seen = false;
    for (int i = 0; i < cnt; ++i) seen = seen || (tl[i] == t);
    if (!seen && cnt < 3) tl[cnt++] = t;
  }
  return cnt;
}

// ------------------------------------------------------------- value types

template <typename V>
struct VT;
template <>
struct VT<float> {
  __device__ static float zero() { return 0.f; }
  __device__ static void fma(float& a, float w, float v) { a = fmaf(w, v, a); }
  __device__ static void add(float& a, float b) { a += b; }
  __device__ static float shfl_xor(float v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
  __device__ static float re_dot(float a, float b) { return a * b; }
};
template <>
struct VT<float2> {
  __device__ static float2 zero() { return make_float2(0.f, 0.f); }
  __device__ static void fma(float2& a, float w, float2 v) {
    a.x = fmaf(w, v.x, a.x);
    a.y = fmaf(w, v.y, a.y);
  }
  __device__ static void add(float2& a, float2 b) {
    a.x += b.x;
    a.y += b.y;
  }
  __device__ static float2 shfl_xor(float2 v, int m) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
  }
  // Re(conj(a) * b)
  __device__ static float re_dot(float2 a, float2 b) { return a.x * b.x + a.y * b.y; }
};

// Per point: start coordinate and valid-tap count per internal dim, and the
// per-tap value used by the inner loops: the 1D weight (norm 1) or |d|
// (norm 2). The DERIV variant adds d weight / d x (norm 1) or signed d (norm 2).
template <bool DERIV>
struct PTaps {
  int start[3];
  int n[3];
  float w[3][NTMAX];
  float dw[DERIV ? 3 : 1][DERIV ? NTMAX : 1];
};
using PointTaps = PTaps<false>;

// Warp-cooperative tap evaluation of point p into `pt` (shared memory).
// Returns false (warp-uniform) if the point has no valid tap.
template <int NORM, bool DERIV>
__device__ __forceinline__ bool warp_point_taps(const Geo& g, const float* locs, long long p, PTaps<DERIV>& pt,
                                                int lane) {
  bool ok = true;
  for (int e = 0; e < 3; ++e) {
    if (!g.act[e]) {
      if (lane == 0) {
        pt.start[e] = 0;
        pt.n[e] = 1;
        pt.w[e][0] = NORM == 1 ? 1.f : 0.f;  // weight 1, or |d| = 0 for the radial norm
        if (DERIV) pt.dw[e][0] = 0.f;
      }
      continue;
    }
    const float x = load_coord(g, locs, p, e);
    if (!coord_ok(x)) {
      ok = false;
      break;
    }
    const int lower = lower_of(g, e, x);
    const int k = lane;
    Tap t;
    t.valid = false;
    t.d = 0.f;
    if (k < g.NT[e]) t = tap_eval(g, e, x, lower, k);
    const unsigned m = __ballot_sync(0xffffffffu, t.valid);
    if (m == 0) {
      ok = false;
      break;
    }
    const int s = __ffs(m) - 1;
    const int n = __popc(m);
    if (t.valid) {
      const int j = k - s;
      const float ad = fabsf(t.d);
      if (NORM == 1) {
        pt.w[e][j] = kern_value(g.kernel, ad, g.beta);
        if (DERIV) pt.dw[e][j] = kern_deriv(g.kernel, t.d, g.beta) / g.r[e];
      } else {
        pt.w[e][j] = ad;
        if (DERIV) pt.dw[e][j] = t.d;
      }
    }
    if (lane == 0) {
      int st = lower + s;
      if (g.pad == TLGB_PAD_CIRCULAR) st = wrapi(st, g.N[e]);
      pt.start[e] = st;
      pt.n[e] = n;
    }
  }
  __syncwarp();
  return ok;
}

// norm-2 weight of one tap combination (radial), 0 outside the unit ball
__device__ __forceinline__ float radial_w(const Geo& g, float a0, float a1, float a2) {
  const float rho = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(a0, a0), __fmul_rn(a1, a1)), __fmul_rn(a2, a2)));
  if (rho > 1.0f) return 0.f;
  return kern_value(g.kernel, rho, g.beta);
}

__device__ __forceinline__ int lg2i(int v) { return 31 - __clz(v); }

// ------------------------------------------------- lane-per-point taps

// KB(x) by the same A&S expansions as kb_value, with one division (3.75 / z)
// and Horner evaluation instead of one division per term: equal to kb_value
// to a few float32 ulps, ~3x fewer instructions. Used on the hot paths.
__device__ __forceinline__ float kb_fast(float x, float beta) {
  const float z = beta * __fsqrt_rn(__fsub_rn(1.0f, __fmul_rn(x, x)));
  if (z < 3.75f) {
    const float u = (z * (1.0f / 3.75f)) * (z * (1.0f / 3.75f));
    return 1.0f + u * (3.5156229f + u * (3.0899424f + u * (1.2067492f + u * (0.2659732f +
           u * (0.0360768f + u * 0.0045813f)))));
  }
  const float v = __fdiv_rn(3.75f, z);
  const float q = 0.39894228f + v * (0.01328592f + v * (0.00225319f + v * (-0.00157565f + v * (0.00916281f +
                  v * (-0.02057706f + v * (0.02635537f + v * (-0.01647633f + v * 0.00392377f)))))));
  return expf(z) * rsqrtf(z) * q;
}

__device__ __forceinline__ float kern_fast(int kernel, float ax, float beta) {
  return kernel == TLGB_KERNEL_KAISER_BESSEL ? kb_fast(ax, beta) : fmaxf(1.0f - ax, 0.0f);
}

// Per point record staged in shared memory: for each internal dim the taps
// that land in the CTA's tile (gridding) or region (gather), as a local
// coordinate and the 1D weight (norm 1) or |d| (norm 2). Taps outside the
// tile are dropped here, so the inner loops carry no bounds checks.
template <int NTB>
struct Rec {
  short lc[3][NTB];
  float wv[3][NTB];
  int m[3];
  int fast;  // every dim has <= 4 kept taps at consecutive local coordinates
};

// One lane builds the record of point p (coordinates x3) for the tile with
// origin o and extent T. region: gather mode, local coordinates run
// contiguously from the wrapped start (the staged region holds the wrap).
template <int NTB>
__device__ __forceinline__ void lane_rec(const Geo& g, const float (&x3)[3], const int (&o)[3], bool region,
                                         Rec<NTB>& R) {
  bool ok = true;
  for (int e = 0; e < 3; ++e) {
    if (!g.act[e]) {
      R.lc[e][0] = 0;
      R.wv[e][0] = g.norm == 1 ? 1.f : 0.f;
      R.m[e] = 1;
      continue;
    }
    const float x = x3[e];
    int cnt = 0;
    if (ok && coord_ok(x)) {
      const int lower = lower_of(g, e, x);
      int s = -1;
      for (int k = 0; k < g.NT[e]; ++k) {
        const Tap t = tap_eval(g, e, x, lower, k);
        if (!t.valid) continue;
        if (s < 0) s = k;
        int l;
        if (region) {
          int st = lower + s;
          if (g.pad == TLGB_PAD_CIRCULAR) st = wrapi(st, g.N[e]);
          l = st - o[e] + (k - s);
        } else {
          int gg = lower + k;
          if (g.pad == TLGB_PAD_CIRCULAR) gg = wrapi(gg, g.N[e]);
          l = gg - o[e];
          if (l < 0 || l >= g.T[e]) continue;
        }
        if (cnt < NTB) {
          const float ad = fabsf(t.d);
          R.lc[e][cnt] = (short)l;
          R.wv[e][cnt] = g.norm == 1 ? kern_fast(g.kernel, ad, g.beta) : ad;
          ++cnt;
        }
      }
    }
    R.m[e] = cnt;
    if (cnt == 0) ok = false;
  }
  if (!ok) R.m[0] = 0;
  bool fast = ok;
  for (int e = 0; e < 3 && fast; ++e) {
    const int m = R.m[e];
    fast = m <= 4 && (m == 0 || (int)R.lc[e][m - 1] - (int)R.lc[e][0] == m - 1);
  }
  R.fast = fast ? 1 : 0;
}

// N floats moved as one vector (a "coil unit": 1 or 2 batch entries)
template <int N>
struct VecF {
  float v[N];
};
template <int N>
__device__ __forceinline__ VecF<N> ldv(const float* p) {
  VecF<N> r;
  if constexpr (N == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    r.v[0] = t.x; r.v[1] = t.y;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int N>
__device__ __forceinline__ void stv(float* p, const VecF<N>& r) {
  if constexpr (N == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  } else if constexpr (N == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(r.v[0], r.v[1]);
  } else {
    *p = r.v[0];
  }
}

// Lane roles: lane = (ux, uz, cu); cu indexes coil units (lowest bits), uz
// the tap along z (4 slots), ux the tap along the split dim (x in 3D, y in
// 2D, more z slots in 1D).
struct Lanes {
  int cu, uz, ux, NUP, UX, lgn;
};
__device__ __forceinline__ Lanes lane_roles(int lane, int nunits) {
  Lanes L;
  L.NUP = nunits <= 1 ? 1 : (nunits <= 2 ? 2 : (nunits <= 4 ? 4 : 8));
  L.lgn = lg2i(L.NUP);
  L.cu = lane & (L.NUP - 1);
  L.uz = (lane >> L.lgn) & 3;
  L.ux = lane >> (L.lgn + 2);
  L.UX = 8 >> L.lgn;
  return L;
}

// Visit the taps of record R assigned to this lane: f(lx, ly, lz, w).
// 3D: x split over ux, z over uz, y looped; 2D: y over ux, z over uz;
// 1D: z over (ux, uz).
template <int NDIM, int NTB, typename F>
__device__ __forceinline__ void for_lane_taps(const Geo& g, const Rec<NTB>& R, const Lanes& L, F&& f) {
  if constexpr (NDIM == 3) {
    for (int kz = L.uz; kz < R.m[2]; kz += 4) {
      const int lz = R.lc[2][kz];
      const float wz = R.wv[2][kz];
      for (int kx = L.ux; kx < R.m[0]; kx += L.UX) {
        const int lx = R.lc[0][kx];
        const float wxz = R.wv[0][kx] * wz;
        for (int ky = 0; ky < R.m[1]; ++ky) {
          const float w = g.norm == 1 ? wxz * R.wv[1][ky] : radial_w(g, R.wv[0][kx], R.wv[1][ky], wz);
          f(lx, (int)R.lc[1][ky], lz, w);
        }
      }
    }
  } else if constexpr (NDIM == 2) {
    for (int kz = L.uz; kz < R.m[2]; kz += 4) {
      const int lz = R.lc[2][kz];
      const float wz = R.wv[2][kz];
      for (int ky = L.ux; ky < R.m[1]; ky += L.UX) {
        const float w = g.norm == 1 ? R.wv[1][ky] * wz : radial_w(g, 0.f, R.wv[1][ky], wz);
        f(0, (int)R.lc[1][ky], lz, w);
      }
    }
  } else {
    for (int kz = L.uz + 4 * L.ux; kz < R.m[2]; kz += 4 * L.UX) {
      const float w = g.norm == 1 ? R.wv[2][kz] : radial_w(g, 0.f, 0.f, R.wv[2][kz]);
      f(0, 0, (int)R.lc[2][kz], w);
    }
  }
}

// ------------------------------------------------------------------ forward

// Resident CTAs of the 8-warp kernel: three (80 registers) where the region
// leaves room for them, for one entry of 320^2 at 524,288 points 122 against 155
// us; with eight entries in 3D two, 449 against 474 (128 x 120 x 96).
constexpr int fwd_ctas(int n, int ndim, int ntb, int nw) { return nw == 8 && ntb == 5 && (ndim == 2 || n == 1) ? 3 : 1; }

// CTA = NW warps sharing one staged region (tile + halo, [x][y][z][batch]);
// each warp interpolates 32 home points per batch. A CTA takes `per` items one
// after the other and stages a region once for those of one tile.
template <int N, int NDIM, int NTB, int NW>
__global__ void __launch_bounds__(NW * 32, fwd_ctas(N, NDIM, NTB, NW))
    interp_fwd_kernel(Geo g, const int4* __restrict__ items, int nitems, int per, const int32_t* __restrict__ entries,
                      const float* __restrict__ locs, const float* __restrict__ gridv, float* __restrict__ out, int CG) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int es = g.cplx ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.y * CG;
  const int ncoil = (int)min((long long)CG, g.nbatch - c0);
  int o[3] = {0, 0, 0}, S[3];
  for (int e = 0; e < 3; ++e) S[e] = g.T[e] + g.NT[e] - 1;
  const int vstride = CG * es;  // floats per staged voxel
  float* reg = reinterpret_cast<float*>(smem);
  const size_t reg_bytes = (((size_t)S[0] * S[1] * S[2] * vstride * sizeof(float)) + 15) & ~(size_t)15;
  Rec<NTB>* rbuf = reinterpret_cast<Rec<NTB>*>(smem + reg_bytes) + warp * 32;

  // stage: rows (x, y) per warp, lanes over (z, batch entry), batch fastest
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  const int cgp = CG <= 1 ? 1 : (CG <= 2 ? 2 : (CG <= 4 ? 4 : 8));
  const int lgc = lg2i(cgp);
  const int rowlen = S[2] * cgp;
  constexpr bool MANY = NW == 8;  // a loop over items costs the 16-warp kernel half its speed (registers)
  int staged = -1;
  int item = MANY ? blockIdx.x * per : blockIdx.x;
  const int last = min(nitems, item + per);
  do {
    const int4 it = items[item];
    if (!MANY || it.x != staged) {
      int t = it.x;
      o[2] = t % g.nt[2] * g.T[2];
      t /= g.nt[2];
      o[1] = t % g.nt[1] * g.T[1];
      o[0] = t / g.nt[1] * g.T[0];
      if (MANY && staged >= 0) __syncthreads();  // the tile before has been read
      for (int row = warp; row < S[0] * S[1]; row += NW) {
        const int x = row / S[1], y = row - x * S[1];
        int gx = o[0] + x, gy = o[1] + y;
        bool rin = true;
        if (g.pad == TLGB_PAD_CIRCULAR) {
          gx = wrapi(gx, g.N[0]);
          gy = wrapi(gy, g.N[1]);
        } else {
          rin = gx < g.N[0] && gy < g.N[1];
        }
        const long long rbase = ((long long)gx * g.N[1] + gy) * g.N[2];
        float* rdst = reg + (size_t)(x * S[1] + y) * S[2] * vstride;
        // all loads of the row first (independent), then the stores
        constexpr int MAXI = 8;
        float2 vv[MAXI];
#pragma unroll
        for (int i = 0; i < MAXI; ++i) {
          vv[i] = make_float2(0.f, 0.f);
          const int idx = lane + 32 * i;
          if (idx < rowlen) {
            const int c = idx & (cgp - 1), z = idx >> lgc;
            int gz = o[2] + z;
            bool in = rin && c < ncoil;
            if (g.pad == TLGB_PAD_CIRCULAR) gz = wrapi(gz, g.N[2]);
            else in = in && gz < g.N[2];
            if (in) {
              const long long gi = (long long)(c0 + c) * gvol + rbase + gz;
              if (es == 2) vv[i] = __ldg(reinterpret_cast<const float2*>(gridv) + gi);
              else vv[i].x = __ldg(gridv + gi);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < MAXI; ++i) {
          const int idx = lane + 32 * i;
          if (idx < rowlen) {
            const int c = idx & (cgp - 1), z = idx >> lgc;
            if (c < CG) {
              float* d = rdst + z * vstride + c * es;
              if (es == 2) *reinterpret_cast<float2*>(d) = vv[i];
              else d[0] = vv[i].x;
            }
          }
        }
        for (int idx = lane + 32 * MAXI; idx < rowlen; idx += 32) {  // long rows (1D tiles)
          const int c = idx & (cgp - 1), z = idx >> lgc;
          if (c >= CG) continue;
          int gz = o[2] + z;
          bool in = rin && c < ncoil;
          if (g.pad == TLGB_PAD_CIRCULAR) gz = wrapi(gz, g.N[2]);
          else in = in && gz < g.N[2];
          float* d = rdst + z * vstride + c * es;
          const long long gi = (long long)(c0 + c) * gvol + rbase + gz;
          if (es == 2) *reinterpret_cast<float2*>(d) = in ? __ldg(reinterpret_cast<const float2*>(gridv) + gi) : make_float2(0.f, 0.f);
          else d[0] = in ? __ldg(gridv + gi) : 0.f;
        }
      }
      __syncthreads();
      staged = it.x;
    }

    const int U = N / es;  // batch entries per unit
    const int nunits = (CG + U - 1) / U;
    const Lanes L = lane_roles(lane, nunits);
    for (int b = it.y + warp * 32; b < it.z; b += NW * 32) {
      const int j = b + lane;
      const int nb = min(32, it.z - b);
      long long p = -1;
      if (j < it.z) {
        p = entries[j];
        float x3[3];
        for (int e = 0; e < 3; ++e) x3[e] = g.act[e] ? load_coord(g, locs, p, e) : 0.f;
        lane_rec<NTB>(g, x3, o, true, rbuf[lane]);
      }
      __syncwarp();
      for (int jj = 0; jj < nb; ++jj) {
        const Rec<NTB>& R = rbuf[jj];
        const long long pj = __shfl_sync(0xffffffffu, p, jj);
        if (R.m[0] == 0) continue;  // warp-uniform
        VecF<N> acc;
#pragma unroll
        for (int i = 0; i < N; ++i) acc.v[i] = 0.f;
        if (L.cu < nunits) {
          const float* base = reg + L.cu * N;
          for_lane_taps<NDIM, NTB>(g, R, L, [&](int lx, int ly, int lz, float w) {
            const VecF<N> v = ldv<N>(base + ((size_t)(lx * S[1] + ly) * S[2] + lz) * vstride);
#pragma unroll
            for (int i = 0; i < N; ++i) acc.v[i] = fmaf(w, v.v[i], acc.v[i]);
          });
        }
        for (int m = L.NUP; m < 32; m <<= 1)
#pragma unroll
          for (int i = 0; i < N; ++i) acc.v[i] += __shfl_xor_sync(0xffffffffu, acc.v[i], m);
        if (lane < L.NUP && L.cu < nunits) {
#pragma unroll
          for (int u = 0; u < N; u += (N >= 2 && es == 2) ? 2 : 1) {
            const int c = L.cu * U + u / es;
            if (c < ncoil) {
              float* dst = out + ((long long)(c0 + c) * g.npts + pj) * es;
              if (es == 2)
                *reinterpret_cast<float2*>(dst) = make_float2(acc.v[u], acc.v[u + 1]);
              else
                dst[0] = acc.v[u];
            }
          }
        }
      }
      __syncwarp();
    }
  } while (MANY && ++item < last);
}

// ------------------------------------------------------------------ adjoint

// One warp per CTA owns one output tile in shared memory ([x][y][z][batch]),
// so every cell is updated by one warp in plan order: deterministic.
template <int N, int NDIM, int NTB>
__global__ void __launch_bounds__(32) interp_adj_kernel(Geo g, const int4* __restrict__ items,
                                                        const int32_t* __restrict__ entries,
                                                        const float* __restrict__ locs,
                                                        const float* __restrict__ vals, float* __restrict__ gridv,
                                                        float* __restrict__ partial, int CG) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int es = g.cplx ? 2 : 1;
  const int4 it = items[blockIdx.x];
  const int lane = threadIdx.x;
  const int cg = blockIdx.y;
  const int c0 = cg * CG;
  const int ncoil = (int)min((long long)CG, g.nbatch - c0);
  int tc[3];
  {
    int t = it.x;
    tc[2] = t % g.nt[2];
    t /= g.nt[2];
    tc[1] = t % g.nt[1];
    tc[0] = t / g.nt[1];
  }
  int o[3];
  for (int e = 0; e < 3; ++e) o[e] = tc[e] * g.T[e];
  const int T1 = g.T[1], T2 = g.T[2];
  const int tvol = g.T[0] * T1 * T2;
  const int vstride = CG * es;
  const int tfl = (tvol * vstride + 3) & ~3;  // tile floats, rounded to whole float4
  float* acc = reinterpret_cast<float*>(smem);
  Rec<NTB>* rbuf = reinterpret_cast<Rec<NTB>*>(smem + (size_t)tfl * sizeof(float));
  float* pv = reinterpret_cast<float*>(rbuf + 32);  // [32][vstride]
  for (int i = lane * 4; i < tfl; i += 128) *reinterpret_cast<float4*>(acc + i) = make_float4(0.f, 0.f, 0.f, 0.f);

  const int U = N / es;
  const int nunits = (CG + U - 1) / U;
  const Lanes L = lane_roles(lane, nunits);

  // registers of the next batch (prefetched while the current one is spread)
  long long np_ = -1;
  float nx3[3] = {0.f, 0.f, 0.f};
  float nv[2 * CGMAX];
  auto prefetch = [&](int b) {
    const int j = b + lane;
    np_ = -1;
    if (j < it.z) {
      np_ = entries[j];
      for (int e = 0; e < 3; ++e) nx3[e] = g.act[e] ? load_coord(g, locs, np_, e) : 0.f;
#pragma unroll
      for (int c = 0; c < CGMAX; ++c) {
        if (c < ncoil) {
          if (es == 2) {
            const float2 v = __ldg(reinterpret_cast<const float2*>(vals) + (long long)(c0 + c) * g.npts + np_);
            nv[2 * c] = v.x;
            nv[2 * c + 1] = v.y;
          } else {
            nv[c] = __ldg(vals + (long long)(c0 + c) * g.npts + np_);
          }
        }
      }
    }
  };
  if (it.y < it.z) prefetch(it.y);
  for (int b = it.y; b < it.z; b += 32) {
    const int nb = min(32, it.z - b);
    __syncwarp();
    if (np_ >= 0) {
      lane_rec<NTB>(g, nx3, o, false, rbuf[lane]);
#pragma unroll
      for (int c = 0; c < CGMAX; ++c)
        if (c < CG) {
          if (es == 2) {
            pv[lane * vstride + 2 * c] = c < ncoil ? nv[2 * c] : 0.f;
            pv[lane * vstride + 2 * c + 1] = c < ncoil ? nv[2 * c + 1] : 0.f;
          } else {
            pv[lane * vstride + c] = c < ncoil ? nv[c] : 0.f;
          }
        }
    }
    __syncwarp();
    if (b + 32 < it.z) prefetch(b + 32);
    for (int jj = 0; jj < nb; ++jj) {
      const Rec<NTB>& R = rbuf[jj];
      // lanes of one warp update cells of consecutive points: order them
      __syncwarp();
      if (R.m[0] == 0 || L.cu >= nunits) continue;
      const VecF<N> v = ldv<N>(pv + jj * vstride + L.cu * N);
      float* base = acc + L.cu * N;
      if (g.wrap_safe) {
        for_lane_taps<NDIM, NTB>(g, R, L, [&](int lx, int ly, int lz, float w) {
          float* a = base + ((size_t)(lx * T1 + ly) * T2 + lz) * vstride;
          VecF<N> r = ldv<N>(a);
#pragma unroll
          for (int i = 0; i < N; ++i) r.v[i] = fmaf(w, v.v[i], r.v[i]);
          stv<N>(a, r);
        });
      } else if (L.ux == 0 && L.uz == 0) {
        // a window longer than the grid reaches a cell twice: taps in order,
        // lanes split by coil unit only
        for (int kx = 0; kx < R.m[0]; ++kx)
          for (int ky = 0; ky < R.m[1]; ++ky)
            for (int kz = 0; kz < R.m[2]; ++kz) {
              const float w = g.norm == 1 ? R.wv[0][kx] * R.wv[1][ky] * R.wv[2][kz]
                                          : radial_w(g, R.wv[0][kx], R.wv[1][ky], R.wv[2][kz]);
              float* a = base + ((size_t)(R.lc[0][kx] * T1 + R.lc[1][ky]) * T2 + R.lc[2][kz]) * vstride;
              VecF<N> r = ldv<N>(a);
#pragma unroll
              for (int i = 0; i < N; ++i) r.v[i] = fmaf(w, v.v[i], r.v[i]);
              stv<N>(a, r);
            }
      }
    }
  }
  __syncwarp();
  if (it.w >= 0) {
    float* dst = partial + ((long long)it.w * gridDim.y + cg) * tfl;
    for (int i = lane * 4; i < tfl; i += 128)
      *reinterpret_cast<float4*>(dst + i) = *reinterpret_cast<const float4*>(acc + i);
    return;
  }
  // write the tile: per (x, y) row, lanes over (batch entry, z) with the
  // batch entry fastest, so shared-memory reads are contiguous
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  const int cgp = CG <= 1 ? 1 : (CG <= 2 ? 2 : (CG <= 4 ? 4 : 8));
  const int lgc = lg2i(cgp);
  for (int row = 0; row < g.T[0] * T1; ++row) {
    const int x = row / T1, y = row - x * T1;
    const int gx = o[0] + x, gy = o[1] + y;
    if (gx >= g.N[0] || gy >= g.N[1]) continue;
    const float* srow = acc + (size_t)(x * T1 + y) * T2 * vstride;
    float* drow = gridv + (((long long)gx * g.N[1] + gy) * g.N[2] + o[2]) * es;
    for (int idx = lane; idx < T2 * cgp; idx += 32) {
      const int cc = idx & (cgp - 1);
      const int z = idx >> lgc;
      if (cc >= ncoil || o[2] + z >= g.N[2]) continue;
      const float* sp = srow + z * vstride + cc * es;
      float* d = drow + ((long long)(c0 + cc) * gvol + z) * es;
      if (es == 2)
        *reinterpret_cast<float2*>(d) = *reinterpret_cast<const float2*>(sp);
      else
        d[0] = sp[0];
    }
  }
}

// ------------------------------------------------ weights held by the plan

// The weight of a tap at normalised offset d = diff / r for the plan's
// records and rows, close to the float32 rounding of the A&S value in 64
// bits: z = beta sqrt(1 - d^2) is carried with its rounding error and beta's
// (exp(z) multiplies them by z, about 7 for the NUFFT's beta, in each
// dimension), from the exact products that fma gives. Evaluated once per
// point and tap while the plan is built, where the time is the pairs' and
// rows' bytes.
__device__ __forceinline__ float kern_precise(int kernel, float diff, float r, float d, float beta,
                                              float beta_lo) {
  const float x = fabsf(d), xe = __fdividef(fmaf(-x, r, fabsf(diff)), r);  // d = x + xe
  if (kernel != TLGB_KERNEL_KAISER_BESSEL) return fmaxf(1.0f - x - xe, 0.0f);
  const float p = x * x, pe = fmaf(x, x, -p) + 2.0f * x * xe;
  const float s = 1.0f - p, se = (1.0f - s) - p - pe;
  if (!(s > 0.f)) return 1.0f;  // I0(0)
  const float q = __fsqrt_rn(s), qe = (fmaf(-q, q, s) + se) * 0.5f * rsqrtf(s);
  const float z = beta * q, ze = fmaf(beta, q, -z) + fmaf(beta_lo, q, beta * qe);
  if (z < 3.75f) {
    const float u = (z * (1.0f / 3.75f)) * (z * (1.0f / 3.75f));
    const float v = 1.0f + u * (3.5156229f + u * (3.0899424f + u * (1.2067492f + u * (0.2659732f +
                    u * (0.0360768f + u * 0.0045813f)))));
    const float dv = 3.5156229f + u * (2.f * 3.0899424f + u * (3.f * 1.2067492f + u * (4.f * 0.2659732f +
                     u * (5.f * 0.0360768f + u * (6.f * 0.0045813f)))));
    return fmaf(dv * (2.0f / (3.75f * 3.75f)) * z, ze, v);
  }
  const float v = __fdividef(3.75f, z);
  const float h = 0.39894228f + v * (0.01328592f + v * (0.00225319f + v * (-0.00157565f + v * (0.00916281f +
                  v * (-0.02057706f + v * (0.02635537f + v * (-0.01647633f + v * 0.00392377f)))))));
  const float f = expf(z) * rsqrtf(z) * h;
  return fmaf(f, ze, f);
}

// ------------------------------------------------ block lists (gridding)
//
// The gridding of complex values works on output blocks of 4 x 4 x 4 cells
// in 3D and 8 x 8 cells in 2D (64 cells either way). A window of 4 taps per
// dimension meets 1.75 blocks of 4 (1.375 of 8) per dimension on average, and
// one warp holds a whole block for 8 entries. The plan lists per block the
// points whose window meets it, in point order. A window meets at most
// g.nrow blocks per dim: 2, or 3 for windows of more than 5 taps over blocks
// of 4 and for circular grids whose last block is a partial one (a window
// can cover the end of the grid, that block and the start).
constexpr int kBlkPart = 256;  // entries per work item: denser blocks are split into parts
constexpr int kCube = 4;       // blocks per edge of the cubes the gridding items visit in turn

// block edge along internal dim e: 4 in 3D; 8 along the two dims of a 2D
// grid (1 along its inactive leading dim)
__host__ __device__ __forceinline__ int block_edge(int ndim, int e) { return ndim == 3 ? 4 : (e == 0 ? 1 : 8); }
__host__ __device__ __forceinline__ int blocks_along(int n, int edge) { return (n + edge - 1) / edge; }
__host__ __device__ __forceinline__ int blocks_along(const Geo& g, int e) {
  return blocks_along(g.N[e], block_edge(g.ndim, e));
}
// An entry is point | selector << shift; the selector names the block among
// the point's blocks per dim: 3 bits i | j << 1 | k << 2 for 2 rows, 9 i +
// 3 j + k (5 bits) for 3.
__host__ __device__ constexpr int sel_shift(int nrow) { return nrow == 3 ? 27 : 29; }
template <int NROW>
__device__ __forceinline__ void sel_rows(uint32_t en, int& i, int& j, int& k) {
  const int s = (int)(en >> sel_shift(NROW));
  if constexpr (NROW == 2) {
    i = s & 1, j = (s >> 1) & 1, k = s >> 2;
  } else {
    i = (s * 57) >> 9;  // s / 9 for s < 27
    const int r = s - 9 * i;
    j = (r * 11) >> 5;  // r / 3 for r < 9
    k = r - 3 * j;
  }
}
// floats of tap rows per point: nrow rows per active dim, one weight per cell
__host__ __device__ constexpr int row_floats(int ndim, int nrow) { return nrow * (ndim == 3 ? 12 : 16); }

// Distinct blocks met along one dim by the cells st .. st+c-1 of a window
// (st in [0, N); wrapped in circular mode). The cells are a run, so a new
// block starts where the block index changes.
__device__ __forceinline__ int axis_blocks(const Geo& g, int e, int st, int c, int* bl) {
  const int lg = g.ndim == 3 ? 2 : (e == 0 ? 0 : 3);
  int cnt = 0, prev = -1;
  for (int k = 0; k < c; ++k) {
    int v = st + k;
    if (v >= g.N[e]) v -= g.N[e];
    const int b = v >> lg;
    if (b != prev && cnt < 3) bl[cnt++] = b;
    prev = b;
  }
  return cnt;
}

// ------------------------------------------------------------- plan kernels
//
// The plan is built on the device from start to end: the host reads the
// lists' lengths back once, after the last launch. Pairs, items and splits
// are counted per CTA, the CTAs' sums scanned, and emitted at their places,
// so every list's order depends on the points alone. A build is 16 to 30
// short launches: bound by them up to about 10^5 points, by the pairs' bytes
// (sorts, rows, records) above. Measured with the Python call around it:
// 2^21 points of a dense-centre ball in 256^3 1.0 ms (about 5.5 ms with host-built
// item lists, read-backs between the stages and one-warp sort chunks of 2048
// pairs), 2^18 in 160^3 0.32 ms (1.5 ms), 205,824 in 320^2 0.24 ms.
constexpr int kPlanPts = 256;  // points (or work units) per CTA
constexpr int kWinBits = 5;    // bits per tap count of a window

// exclusive scan of a uint4 per thread over the CTA (NT threads); total to `tot`
template <int NT>
__device__ __forceinline__ uint4 cta_scan4(uint4 v, uint4& tot) {
  __shared__ uint4 ws[NT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4 x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, x.x, o), b = __shfl_up_sync(0xffffffffu, x.y, o),
                   c = __shfl_up_sync(0xffffffffu, x.z, o), d = __shfl_up_sync(0xffffffffu, x.w, o);
    if (lane >= o) x.x += a, x.y += b, x.z += c, x.w += d;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  uint4 base = make_uint4(0, 0, 0, 0);
  tot = base;
  for (int w = 0; w < NT / 32; ++w) {
    const uint4 t = ws[w];
    if (w < warp) base.x += t.x, base.y += t.y, base.z += t.z, base.w += t.w;
    tot.x += t.x, tot.y += t.y, tot.z += t.z, tot.w += t.w;
  }
  __syncthreads();  // ws may be written again
  return make_uint4(base.x + x.x - v.x, base.y + x.y - v.y, base.z + x.z - v.z, base.w + x.w - v.w);
}

// CTA j scans job j's n CTA sums in place (exclusive); totals to tot[0..3]. With
// `most_y` > 0, a total of y above it becomes 0 and tot[3] is set.
struct ScanJob {
  uint4* sums;
  long long n;
  uint32_t* tot;
  uint32_t most_y;
};
__global__ void __launch_bounds__(1024) plan_scan_kernel(ScanJob j0, ScanJob j1, ScanJob j2) {
  const ScanJob j = blockIdx.x == 2 ? j2 : (blockIdx.x ? j1 : j0);
  const long long per = (j.n + 1023) / 1024, b = threadIdx.x * per;
  const long long e = b + per < j.n ? b + per : j.n;
  uint4 s = make_uint4(0, 0, 0, 0);
  for (long long i = b; i < e; ++i) {
    const uint4 v = j.sums[i];
    s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
  }
  uint4 tot;
  uint4 run = cta_scan4<1024>(s, tot);
  for (long long i = b; i < e; ++i) {
    const uint4 v = j.sums[i];
    j.sums[i] = run;
    run.x += v.x, run.y += v.y, run.z += v.z, run.w += v.w;
  }
  if (j.most_y > 0 && tot.y > j.most_y) tot.y = 0, tot.w = 1;
  if (threadIdx.x == 0) j.tot[0] = tot.x, j.tot[1] = tot.y, j.tot[2] = tot.z, j.tot[3] = tot.w;
}

__device__ __forceinline__ int win_cnt(const int4& w, int e) { return (w.w >> (kWinBits * e)) & ((1 << kWinBits) - 1); }
__device__ __forceinline__ int win_st(const int4& w, int e) { return e == 0 ? w.x : (e == 1 ? w.y : w.z); }

// tile pairs, block pairs and whether the point has taps (a home pair)
__device__ __forceinline__ uint4 win_pairs(const Geo& g, const int4& w) {
  if (w.w == 0) return make_uint4(0, 0, 0, 0);
  uint32_t t = 1, b = 1;
  for (int e = 0; e < 3; ++e) {
    int l[3];
    t *= (uint32_t)axis_tiles(g, e, win_st(w, e), win_cnt(w, e), l);
    if (g.nrow) b *= (uint32_t)axis_blocks(g, e, win_st(w, e), win_cnt(w, e), l);
  }
  return make_uint4(t, g.nrow ? b : 0u, 1u, 0u);
}

// Per point: its window (first valid tap per dim, wrapped into [0, N) in
// circular mode, and the tap counts; none when a dim has no valid tap) and the
// tap rows over the blocks it meets (`rows`):
// per active dim, one weight per cell of each block in axis_blocks order; a
// cell outside the window holds -0.0 (valid weights are >= +0), so the sign
// bit tells the gridding which cells the window covers. Each weight is
// evaluated once and the rows are put together in shared memory, stored as
// one contiguous run per CTA (evaluating every cell of every row in place
// and storing them one by one took 47 us for 2^18 points in 3D).
// NTM: taps evaluated per dim, at least the geometry's. With `total` (and no
// windows or sums) the block pairs are only counted.
template <int NTM>
__global__ void __launch_bounds__(kPlanPts) plan_points_kernel(Geo g, const float* __restrict__ locs,
                                                               int4* __restrict__ win, float* __restrict__ rows,
                                                               uint4* __restrict__ sums,
                                                               unsigned long long* __restrict__ total) {
  extern __shared__ __align__(16) float prow[];  // [points][row_floats], when rows are wanted
  const long long p0 = (long long)blockIdx.x * kPlanPts, p = p0 + threadIdx.x;
  const bool on = p < g.npts;
  const int RF = row_floats(g.ndim, g.nrow);
  float* mine = prow + threadIdx.x * RF;
  if (rows) {
    const float4 none = make_float4(-0.f, -0.f, -0.f, -0.f);
    for (int i = 0; i < RF / 4; ++i) reinterpret_cast<float4*>(mine)[i] = none;
  }
  int4 w4 = make_int4(0, 0, 0, 0);
  int cnts = 0;
  bool ok = on;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    int c = 0, st = 0;
    if (!g.act[e]) {
      c = 1;  // a leading dimension of a 1D or 2D geometry: one tap at 0
    } else if (on) {
      const float x = load_coord(g, locs, p, e);
      if (coord_ok(x)) {
        const int lower = lower_of(g, e, x);
        const int lg = g.ndim == 3 ? 2 : 3;
        float* row = mine + (e - (3 - g.ndim)) * (RF / g.ndim) - (1 << lg);
        int prev = -1;
#pragma unroll
        for (int k = 0; k < NTM; ++k) {
          if (k >= g.NT[e]) continue;
          const Tap t = tap_eval(g, e, x, lower, k);
          if (!t.valid) continue;
          if (c == 0) st = g.pad == TLGB_PAD_CIRCULAR ? wrapi(lower + k, g.N[e]) : lower + k;
          if (rows) {
            const float v = kern_precise(g.kernel, __fsub_rn(x, (float)(lower + k)), g.r[e], t.d, g.beta, g.beta_lo);
            int cell = st + c;
            if (cell >= g.N[e]) cell -= g.N[e];
            if (cell >> lg != prev) row += 1 << lg, prev = cell >> lg;
            row[cell & ((1 << lg) - 1)] = v;
          }
          ++c;
        }
      }
    }
    if (c == 0) ok = false;
    cnts |= c << (kWinBits * e);
    if (e == 0) w4.x = st;
    if (e == 1) w4.y = st;
    if (e == 2) w4.z = st;
  }
  w4.w = ok ? cnts : 0;
  if (on && win) win[p] = w4;
  uint4 tot;
  cta_scan4<kPlanPts>(on ? win_pairs(g, w4) : make_uint4(0, 0, 0, 0), tot);  // its barriers also publish the rows
  if (threadIdx.x == 0 && sums) sums[blockIdx.x] = tot;
  if (threadIdx.x == 0 && total) atomicAdd(total, (unsigned long long)tot.y);
  if (rows) {
    const long long n4 = min((long long)kPlanPts, g.npts - p0) * RF / 4;
    float4* dst = reinterpret_cast<float4*>(rows + p0 * RF);
    for (int i = threadIdx.x; i < n4; i += kPlanPts) dst[i] = reinterpret_cast<const float4*>(prow)[i];
  }
}

// (key, point) pairs of both lists at their places (point order)
__global__ void __launch_bounds__(kPlanPts) plan_emit_kernel(Geo g, const int4* __restrict__ win,
                                                             const uint4* __restrict__ sums,
                                                             uint32_t* __restrict__ tkeys, int32_t* __restrict__ tvals,
                                                             uint32_t* __restrict__ bkeys,
                                                             int32_t* __restrict__ bvals, uint32_t most_blk) {
  const long long p = (long long)blockIdx.x * kPlanPts + threadIdx.x;
  const int4 w = p < g.npts ? win[p] : make_int4(0, 0, 0, 0);
  uint4 tot;
  const uint4 x = cta_scan4<kPlanPts>(win_pairs(g, w), tot);
  if (w.w == 0) return;
  const uint4 base = sums[blockIdx.x];
  int l[3][3], nc[3];
  for (int e = 0; e < 3; ++e) nc[e] = axis_tiles(g, e, win_st(w, e), win_cnt(w, e), l[e]);
  uint32_t o = base.x + x.x;
  for (int i = 0; i < nc[0]; ++i)
    for (int j = 0; j < nc[1]; ++j)
      for (int k = 0; k < nc[2]; ++k) {
        const uint32_t tile = ((uint32_t)l[0][i] * g.nt[1] + l[1][j]) * g.nt[2] + l[2][k];
        tkeys[o] = tile * 2u + (i == 0 && j == 0 && k == 0 ? 0u : 1u);
        tvals[o] = (int32_t)p;
        ++o;
      }
  if (!g.nrow) return;
  for (int e = 0; e < 3; ++e) nc[e] = axis_blocks(g, e, win_st(w, e), win_cnt(w, e), l[e]);
  const uint32_t nb1 = (uint32_t)blocks_along(g, 1), nb2 = (uint32_t)blocks_along(g, 2);
  o = base.y + x.y;
  if (o + nc[0] * nc[1] * nc[2] > most_blk) return;  // more pairs than the caller counted: refused, the list is left empty
  for (int i = 0; i < nc[0]; ++i)
    for (int j = 0; j < nc[1]; ++j)
      for (int k = 0; k < nc[2]; ++k) {
        const uint32_t sel = g.nrow == 3 ? (uint32_t)(9 * i + 3 * j + k) : (uint32_t)(i | j << 1 | k << 2);
        bkeys[o] = ((uint32_t)l[0][i] * nb1 + (uint32_t)l[1][j]) * nb2 + (uint32_t)l[2][k];
        bvals[o] = (int32_t)((uint32_t)p | sel << sel_shift(g.nrow));
        ++o;
      }
}

// start[k] = first position of key k in the sorted keys, start[nkeys] = the
// list's length: one binary search per key (a histogram of the keys by
// atomics is slow where a dense centre puts thousands of them on one key)
__global__ void __launch_bounds__(256) plan_starts_kernel(const uint32_t* __restrict__ tkeys,
                                                          const uint32_t* __restrict__ bkeys,
                                                          const uint32_t* __restrict__ cnt, long long ntk,
                                                          long long nbk, uint32_t* __restrict__ tstart,
                                                          uint32_t* __restrict__ bstart) {
  long long k = (long long)blockIdx.x * 256 + threadIdx.x;
  const bool blk = k > ntk;
  if (blk) k -= ntk + 1;
  if (k > (blk ? nbk : ntk)) return;
  const uint32_t* keys = blk ? bkeys : tkeys;
  uint32_t lo = 0, hi = blk ? cnt[1] : cnt[0];
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if ((long long)keys[mid] < k)
      lo = mid + 1;
    else
      hi = mid;
  }
  (blk ? bstart : tstart)[k] = lo;
}

// Work units the items are made from: tiles, in the order of cubes of
// kTileCube^3 tiles (squares in 2D), and rows of kCube blocks along z, in the
// order of the cubes of kCube^3 blocks (kCube^2 in 2D). Neighbouring regions
// are so gathered close together in time and find their shared halos in L2,
// and the blocks a point meets its rows and values. Gathering 8 x 256^3 at
// 2^21 points of a ball in random order: 735 us in plain tile order, 587 in
// cubes of 2, 592 of 4, 590 of 8; 8 x 160^3 at 2^18 even points: 176, 153, 186,
// 198 us.
constexpr int kTileCube = 2;
struct PlanUnits {
  long long ntiles, ntu, nrows;  // tiles; units: of tiles (some outside the grid), of block rows
  int ntx, nty, ntz;             // tiles per dim
  int nbx, nby, nbz;             // blocks per dim
  int ncy, ncz;                  // cubes along y and z
  int per;                       // rows per cube
  int tile_ctas;
};

// the tile of unit u, -1 outside the grid
__device__ __forceinline__ long long unit_tile(const PlanUnits& U, long long u) {
  constexpr int C = kTileCube;
  if (u >= U.ntu) return -1;
  const int cx = U.ntx == 1 ? 1 : C, in = (int)(u % (cx * C * C));
  long long q = u / (cx * C * C);
  const int cy = (U.nty + C - 1) / C, cz = (U.ntz + C - 1) / C;
  const int z = (int)(q % cz) * C + in % C;
  q /= cz;
  const int y = (int)(q % cy) * C + in / C % C, x = (int)(q / cy) * cx + in / (C * C);
  if (x >= U.ntx || y >= U.nty || z >= U.ntz) return -1;
  return ((long long)x * U.nty + y) * U.ntz + z;
}

// the blocks [b0, b0 + n) of row unit u (n = 0: outside the grid)
__device__ __forceinline__ int row_blocks(const PlanUnits& U, long long u, int& b0) {
  const int in = (int)(u % U.per);
  long long c = u / U.per;
  const int cz = (int)(c % U.ncz);
  c /= U.ncz;
  const int cy = (int)(c % U.ncy), cx = (int)(c / U.ncy);
  const int bx = cx * (U.per / kCube) + in / kCube, by = cy * kCube + in % kCube, bz = cz * kCube;
  if (bx >= U.nbx || by >= U.nby) return 0;
  b0 = (bx * U.nby + by) * U.nbz + bz;
  return min(kCube, U.nbz - bz);
}

__device__ __forceinline__ int parts_of(int n, int chunk) { return (n + chunk - 1) / chunk; }

// Item counts of a unit (`u`: a tile or a block row). Tile: gather items, gridding items, parts of split
// tiles, split tiles. Block row: items, parts of split blocks, split blocks.
// A run of empty blocks of the row is one item.
__device__ __forceinline__ uint4 unit_items(const PlanUnits& U, bool tile, long long u, const uint32_t* tstart,
                                            const uint32_t* bstart, int fwd_chunk, int adj_chunk) {
  uint4 c = make_uint4(0, 0, 0, 0);
  if (tile) {
    const uint32_t b = tstart[2 * u], h = tstart[2 * u + 1], e = tstart[2 * u + 2];
    const int na = (int)(e - b);
    c.x = parts_of((int)(h - b), fwd_chunk);
    c.y = na <= adj_chunk ? 1 : parts_of(na, adj_chunk);
    if (na > adj_chunk) c.z = c.y, c.w = 1;
    return c;
  }
  int b0 = 0;
  const int nb = row_blocks(U, u, b0);
  bool empty = false;
  for (int i = 0; i < nb; ++i) {
    const int n = (int)(bstart[b0 + i + 1] - bstart[b0 + i]);
    if (n == 0) {
      c.x += empty ? 0 : 1;
    } else if (n <= kBlkPart) {
      c.x += 1;
    } else {
      const int k = parts_of(n, kBlkPart);
      c.x += k, c.y += k, c.z += 1;
    }
    empty = n == 0;
  }
  return c;
}

__global__ void __launch_bounds__(kPlanPts) plan_count_items_kernel(PlanUnits U, const uint32_t* __restrict__ tstart,
                                                                    const uint32_t* __restrict__ bstart, int fwd_chunk,
                                                                    int adj_chunk, uint4* __restrict__ sums,
                                                                    uint4* __restrict__ homes) {
  const bool tile = (int)blockIdx.x < U.tile_ctas;
  const long long u = (long long)(blockIdx.x - (tile ? 0 : U.tile_ctas)) * kPlanPts + threadIdx.x;
  uint4 c = make_uint4(0, 0, 0, 0), tot;
  const long long t = tile ? unit_tile(U, u) : (u < U.nrows ? u : -1);
  if (t >= 0) c = unit_items(U, tile, t, tstart, bstart, fwd_chunk, adj_chunk);
  cta_scan4<kPlanPts>(c, tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
  if (!tile) return;
  c = make_uint4(0, 0, 0, 0);
  if (t >= 0) c.x = tstart[2 * t + 1] - tstart[2 * t];
  cta_scan4<kPlanPts>(c, tot);
  if (threadIdx.x == 0) homes[blockIdx.x] = tot;
}

// The items at their places. A gather item is (tile, its entries [begin,
// end), index of its first point among the home points in item order). The tile gridding's
// items and the split blocks go to `adj` / `bsplit` with sort keys: they are
// put in falling order of their length afterwards (a long item or a long sum
// that starts last is waited for alone).
__global__ void __launch_bounds__(kPlanPts) plan_emit_items_kernel(
    PlanUnits U, const uint32_t* __restrict__ tstart, const uint32_t* __restrict__ bstart, int fwd_chunk, int adj_chunk,
    const uint4* __restrict__ sums, const uint4* __restrict__ homes, int4* __restrict__ fwd, int4* __restrict__ adj, uint32_t* __restrict__ akey,
    int32_t* __restrict__ aidx, int4* __restrict__ split, int4* __restrict__ bitems, int4* __restrict__ bsplit,
    uint32_t* __restrict__ skey, int32_t* __restrict__ sidx) {
  const bool tile = (int)blockIdx.x < U.tile_ctas;
  const long long u = (long long)(blockIdx.x - (tile ? 0 : U.tile_ctas)) * kPlanPts + threadIdx.x;
  const long long ut = tile ? unit_tile(U, u) : (u < U.nrows ? u : -1);
  const bool on = ut >= 0;
  uint4 c = make_uint4(0, 0, 0, 0), tot;
  if (on) c = unit_items(U, tile, ut, tstart, bstart, fwd_chunk, adj_chunk);
  uint4 o = cta_scan4<kPlanPts>(c, tot), ho = make_uint4(0, 0, 0, 0);
  if (tile) {
    if (on) ho.x = tstart[2 * ut + 1] - tstart[2 * ut];
    ho = cta_scan4<kPlanPts>(ho, tot);
  }
  if (!on) return;
  const uint4 base = sums[blockIdx.x];
  o.x += base.x, o.y += base.y, o.z += base.z, o.w += base.w;
  if (tile) {
    const int b = (int)tstart[2 * ut], h = (int)tstart[2 * ut + 1], e = (int)tstart[2 * ut + 2], t = (int)ut;
    const int h0 = (int)(homes[blockIdx.x].x + ho.x);
    for (int k = 0; k < (int)c.x; ++k)
      fwd[o.x + k] = make_int4(t, b + k * fwd_chunk, min(h, b + (k + 1) * fwd_chunk), h0 + k * fwd_chunk);
    if (c.w) split[o.w] = make_int4(t, (int)o.z, (int)c.z, 0);
    for (int k = 0; k < (int)c.y; ++k) {
      const int q0 = b + k * adj_chunk, q1 = min(e, q0 + adj_chunk);
      adj[o.y + k] = make_int4(t, q0, q1, c.w ? (int)o.z + k : -1);
      akey[o.y + k] = (uint32_t)(adj_chunk - (q1 - q0));
      aidx[o.y + k] = (int)(o.y + k);
    }
    return;
  }
  int b0 = 0;
  const int nb = row_blocks(U, u, b0);
  uint32_t item = o.x, part = o.y, sp = o.z;
  int run = 0;  // empty blocks of the run that ends here
  for (int i = 0; i < nb; ++i) {
    const int q0 = (int)bstart[b0 + i], q1 = (int)bstart[b0 + i + 1], n = q1 - q0;
    if (n == 0) {
      ++run;
      if (run == 1) ++item;
      bitems[item - 1] = make_int4(b0 + i + 1 - run, q0, q0, -run);
      continue;
    }
    run = 0;
    if (n <= kBlkPart) {
      bitems[item++] = make_int4(b0 + i, q0, q1, -1);
      continue;
    }
    const int k = parts_of(n, kBlkPart);
    bsplit[sp] = make_int4(b0 + i, (int)part, k, 0);
    skey[sp] = 65535u - (uint32_t)min(k, 65535);
    sidx[sp] = (int)sp;
    ++sp;
    for (int j = 0; j < k; ++j) bitems[item++] = make_int4(b0 + i, q0 + j * kBlkPart, min(q1, q0 + (j + 1) * kBlkPart), (int)part++);
  }
}

__global__ void __launch_bounds__(256) plan_order_kernel(const uint32_t* __restrict__ cnt, const int4* __restrict__ adj,
                                                         const int32_t* __restrict__ aidx, int4* __restrict__ adj_out,
                                                         const int4* __restrict__ bsplit,
                                                         const int32_t* __restrict__ sidx,
                                                         int4* __restrict__ bsplit_out) {
  const uint32_t n = blockIdx.y ? cnt[10] : cnt[5];
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    if (blockIdx.y)
      bsplit_out[i] = bsplit[sidx[i]];
    else
      adj_out[i] = adj[aidx[i]];
  }
}

// The same order without the sort's six launches, for short lists: an item's
// place is the number of items before it. A plan of 100 points on 321 x 203 took
// 208 us with the call, 177 so.
constexpr int64_t kRankItems = 1024;
__global__ void __launch_bounds__(256) plan_rank_kernel(const uint32_t* __restrict__ cnt, const int4* __restrict__ adj,
                                                        const uint32_t* __restrict__ akey, int4* __restrict__ adj_out,
                                                        const int4* __restrict__ bsplit, const uint32_t* __restrict__ skey,
                                                        int4* __restrict__ bsplit_out) {
  const uint32_t n = blockIdx.y ? cnt[10] : cnt[5], i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const uint32_t* keys = blockIdx.y ? skey : akey;
  const uint32_t key = keys[i];
  uint32_t place = 0;
#pragma unroll 8
  for (uint32_t j = 0; j < n; ++j) place += keys[j] < key || (keys[j] == key && j < i) ? 1u : 0u;
  if (blockIdx.y)
    bsplit_out[place] = bsplit[i];
  else
    adj_out[place] = adj[i];
}

// Compensated summation (Neumaier's variant of Kahan's method): s + c
// carries the running sum; c collects the low-order bits each addition
// loses, whichever operand is larger.
__device__ __forceinline__ void comp_add(float& s, float& c, float x) {
  const float t = s + x;
  c += fabsf(s) >= fabsf(x) ? (s - t) + x : (x - t) + s;
  s = t;
}

using sm100::fence_mbar_init;
using sm100::mbar_arrive_expect_tx;
using sm100::mbar_init;
using sm100::mbar_wait_bounded;
using sm100::smem_u32;
using sm100::tma_load_4d;

// device status word: set when a bounded wait gave up (see tlgb_interp_forward)
__device__ int g_tlgb_status;

// Point values [batch][npts] (complex) -> point-major [group][npts][8]: the
// gridding reads 64 contiguous bytes per (point, tile) pair instead of 8
// scattered 8-byte values. CTA = 128 points x 8 entries of one group: warp c
// loads entry c two points per 16-byte load (when the rows are 16-byte
// aligned), each thread stores two 16-byte pairs of entries; 32 bytes in
// flight per thread each way. Block (0, group) also zeroes the group's work
// counter of the gridding launched after it (ctr, when given).
constexpr int kTrPts = 128;
__global__ void __launch_bounds__(256) transpose_vals_kernel(const float2* __restrict__ vals, long long npts,
                                                             long long nbatch, float2* __restrict__ tv,
                                                             int* __restrict__ ctr) {
  __shared__ __align__(16) float2 sm[kTrPts][10];  // rows of 80 bytes: entry pairs 16-byte aligned
  const int grp = blockIdx.y;
  const long long p0 = (long long)blockIdx.x * kTrPts;
  const int t = threadIdx.x;
  if (ctr && blockIdx.x == 0 && t == 0) ctr[grp] = 0;
  {
    const int c = t >> 5, lane = t & 31;
    const long long cc = (long long)grp * 8 + c;
    const float2* src = vals + cc * npts;
    const bool vec = ((reinterpret_cast<uintptr_t>(vals) | (uintptr_t)(npts * 8)) & 15) == 0;
    float2 a[2], b[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long p = p0 + h * 64 + 2 * lane;
      a[h] = b[h] = make_float2(0.f, 0.f);
      if (cc < nbatch) {
        if (vec && p + 1 < npts) {
          const float4 v = __ldg(reinterpret_cast<const float4*>(src + p));
          a[h] = make_float2(v.x, v.y), b[h] = make_float2(v.z, v.w);
        } else {
          if (p < npts) a[h] = __ldg(src + p);
          if (p + 1 < npts) b[h] = __ldg(src + p + 1);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      sm[h * 64 + 2 * lane][c] = a[h];
      sm[h * 64 + 2 * lane + 1][c] = b[h];
    }
  }
  __syncthreads();
  float4* dst = reinterpret_cast<float4*>(tv) + (long long)grp * npts * 4;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int j = h * 256 + t, i = j >> 2, q = j & 3;  // point i, entries 2q and 2q + 1
    const long long p = p0 + i;
    if (p < npts) dst[p * 4 + q] = *reinterpret_cast<const float4*>(&sm[i][2 * q]);
  }
}

// Packed single-precision arithmetic of sm_100+ (two independent IEEE fp32
// operations, round to nearest: the same results as two scalar ones).
__device__ __forceinline__ unsigned long long f2_bits(float2 v) { return *reinterpret_cast<unsigned long long*>(&v); }
__device__ __forceinline__ float2 bits_f2(unsigned long long b) { return *reinterpret_cast<float2*>(&b); }
// acc += (w, w) * v
__device__ __forceinline__ void fma2_bcast(float2& acc, float w, float2 v) {
  unsigned long long a = f2_bits(acc);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(f2_bits(make_float2(w, w))), "l"(f2_bits(v)));
  acc = bits_f2(a);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return bits_f2(r);
}
// (s, s) * v
__device__ __forceinline__ float2 mul2_bcast(float s, float2 v) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(make_float2(s, s))), "l"(f2_bits(v)));
  return bits_f2(r);
}

// ------------------------------------------------- block gridding (3D, 8 entries)
//
// Work items are blocks, parts of dense blocks and runs of empty blocks. A
// persistent grid's warps take them one at a time, in list order, from a
// counter in global memory, so a dense block costs one warp, not a CTA, no
// SM idles behind a CTA's last items, and which warp takes an item does not
// change its result. A warp holds its item's 4 x 4 x 4-cell output
// block x 8 complex entries as the accumulators of warp-level tensor-core
// products (mma.sync m16n8k8, tf32 inputs, fp32 accumulation): the block's
// 64 cells are the 4 row tiles (one per x, rows (y, z)), the 8 entries'
// real and imaginary parts the 2 column tiles. The warp walks the block's
// list in chunks of 16 entries: two lanes copy one entry's values and the
// point's three rows of tap weights over this block (from the plan) into a
// buffer of the warp (cp.async). Then each group of 8 entries is one rank-8
// update of the block: weights (x row * y row * z row, built in registers)
// times values. fp32 accuracy from tf32 inputs: each operand is split into a
// high and a low tf32 part and the update is hi*hi + hi*lo + lo*hi (the
// lo*lo term is below 2^-22 of the product). The result depends only on the
// plan's order: bit-identical run to run. An item whose sums are not all
// finite is summed again entry by entry on the CUDA cores, each entry over the
// cells of its window only (a zero weight would carry its NaN or Inf to the
// whole block); the rows mark the cells outside the window with -0.0.
//
// Bound by issue and by the latency of dependent instructions at four warps
// per scheduler: with the same points for every block (all reads from L2) and
// without the stores it still takes 535 of 610 us at 2^21 points in 256^3 x 8.
// With one buffer of 32 entries per warp a chunk's copies were waited for in
// full (684 us, 830 us for 256 entries of 320^2 at 205,824 points with its
// transposition and reduction, whose groups were rows of the launch grid with
// a warp per item); now the next chunk is copied during a chunk's products,
// across items and groups, the splits and sums are packed two to an
// instruction, whole blocks are stored without a check per cell, and values
// are checked once per item: 595 and 671 us. Not faster: four lanes per entry
// (fewer lines per copy, 755 against 726 us at that stage), three or four
// buffers, two or four row tiles' products interleaved.
constexpr int kBC = 16;       // entries per chunk, two lanes per entry while staging
constexpr int kBWarps = 4;    // per CTA
constexpr int kBStages = 2;   // chunks of a warp in shared memory: one worked on, the other in flight
// Resident CTAs per SM of the persistent grid: with 128 registers nothing
// spills (256^3 below: 706 us with 4 CTAs, 735 and 860 with 5 and 6)
constexpr int kB3Ctas = 4;
constexpr int kBS = 40;       // floats per staged entry: x row 0-3 | y row 4-7 | z row 8-11 | values 16-31
                              // (40: the tensor-core operand loads of a group of 8 entries are free of
                              // bank conflicts)

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all copies of this thread but those of the last N committed groups
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The chunks of the items that one warp takes, ahead of the warp's work on
// them. A unit is (group of 8 entries, item), group after group; a warp's first
// unit is its number in the grid, the others come from the counter. Lane
// k & 7 keeps the descriptor and the group of the warp's k-th unit, requested
// when the cursor reaches unit k - 1, and the counter is asked one request
// ahead, so nothing waits for an atomic or a descriptor just issued.
struct ChunkStream {
  int4 desc;   // of unit k in lane k & 7; y < 0: past the end
  int group;
  int ticket;  // lane 0
  int k, y, z, cg;  // cursor: unit, next chunk's first entry, end of the unit, its group

  __device__ __forceinline__ void ask(int* ctr, int lane) {
    if (lane == 0) ticket = atomicAdd(ctr, 1) + (int)gridDim.x * kBWarps;
  }
  __device__ __forceinline__ void read(int slot, int unit, int nunits, int nitems, const int4* __restrict__ items, int lane) {
    if (lane != slot) return;
    group = unit / nitems;
    desc = unit < nunits ? items[unit - group * nitems] : make_int4(0, -1, -1, 0);
  }
  __device__ __forceinline__ void request(int slot, int nunits, int nitems, const int4* __restrict__ items, int* ctr, int lane) {
    const int unit = __shfl_sync(0xffffffffu, ticket, 0);
    read(slot, unit, nunits, nitems, items, lane);
    if (unit < nunits) ask(ctr, lane);
  }
  __device__ __forceinline__ void move_to(int unit) {
    k = unit;
    y = __shfl_sync(0xffffffffu, desc.y, k & 7);
    z = __shfl_sync(0xffffffffu, desc.z, k & 7);
    cg = __shfl_sync(0xffffffffu, group, k & 7);
  }
  __device__ __forceinline__ void start(int nunits, int nitems, const int4* __restrict__ items, int* ctr, int lane, int warp) {
    desc = make_int4(0, -1, -1, 0);
    group = 0;
    ticket = 0;
    ask(ctr, lane);
    read(0, (int)blockIdx.x * kBWarps + warp, nunits, nitems, items, lane);
    if ((int)blockIdx.x * kBWarps + warp < nunits) request(1, nunits, nitems, items, ctr, lane);
    move_to(0);
  }
  // this lane's entry of the next chunk, its group and size: -1 past the end, 0 for a run of empty blocks
  __device__ __forceinline__ int next(uint32_t& entry, int& ecg, int nunits, int nitems, const int4* __restrict__ items,
                                      const uint32_t* __restrict__ bentries, int* ctr, int lane) {
    if (y < 0) return -1;
    const int n = min(kBC, z - y), j = lane & (kBC - 1);
    entry = j < n ? bentries[y + j] : 0u;
    ecg = cg;
    y += kBC;
    if (y >= z) {
      move_to(k + 1);
      if (y >= 0) request((k + 1) & 7, nunits, nitems, items, ctr, lane);
    }
    return n;
  }
};

// x = hi + lo: hi the nearest tf32 value, lo the rest (exact; the tensor
// cores cut it to its upper 11 bits: an operand is up to 2^-21 off, 2^-22 with a
// rounded lo). With cvt.rna (ties away) and a rounded lo the gridding issued 45 warp
// instructions per (point, block) entry, 32 so (before the chunk stream); hi
// cut instead of rounded would bias every sum by 1.5e-7 (lo would have the
// sign of x, and the bits dropped from it would add up).
__device__ __forceinline__ void split_tf32(float x, unsigned& hi, unsigned& lo) {
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  lo = __float_as_uint(x - __uint_as_float(hi));
}
// the same of the product x * y, lo from its exact value
__device__ __forceinline__ void split_tf32_mul(float x, float y, unsigned& hi, unsigned& lo) {
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x * y));
  lo = __float_as_uint(fmaf(x, y, -__uint_as_float(hi)));
}

// the same of two products x * y.x and x * y.y, two at a time
__device__ __forceinline__ void split_tf32_mul2(float x, float2 y, unsigned* hi, unsigned* lo) {
  const float2 p = mul2_bcast(x, y);
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(hi[0]) : "f"(p.x));
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(hi[1]) : "f"(p.y));
  float2 l = mul2_bcast(-1.f, make_float2(__uint_as_float(hi[0]), __uint_as_float(hi[1])));
  fma2_bcast(l, x, y);
  lo[0] = __float_as_uint(l.x), lo[1] = __float_as_uint(l.y);
}

// d = a * b + c, m16n8k8, tf32 inputs, fp32 accumulators
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1,
                                         const float (&c)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// d += (ah + al) * (bh + bl) without the lo * lo term. The three products of
// one group of 8 entries are summed on their own, smallest first, and added
// to d on the CUDA cores: the tensor cores truncate their sums, and a chain of
// them through d pulls it towards zero (2.2e-6 relative after a few hundred
// entries per block, against 7e-7 for a chain of rounded additions).
__device__ __forceinline__ void mma_split(float (&d)[4], const unsigned (&ah)[4], const unsigned (&al)[4],
                                          const unsigned (&bh)[2], const unsigned (&bl)[2]) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mma_tf32(t, ah, bl[0], bl[1], t);
  mma_tf32(t, al, bh[0], bh[1], t);
  mma_tf32(t, ah, bh[0], bh[1], t);
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const float2 r = add2(make_float2(d[i], d[i + 1]), make_float2(t[i], t[i + 1]));
    d[i] = r.x, d[i + 1] = r.y;
  }
}

__device__ __forceinline__ void block_origin(const Geo& g, int key, int& bx, int& by, int& bz) {
  const int nb1 = blocks_along(g, 1), nb2 = blocks_along(g, 2);
  bz = key % nb2;
  const int t = key / nb2;
  by = t % nb1;
  bx = t / nb1;
}

// The accumulator fragment of lane (g8, t4): D[m][nt][2h + c] holds entry
// 4 nt + t4 (real part c = 0, imaginary c = 1) of the block cell
// 3D: (x m, y (g8 >> 2) + 2h, z g8 & 3); 2D: (y 2m + h, z g8).
template <int NDIM>
__device__ __forceinline__ void frag_cell(int m, int h, int g8, int& x, int& y, int& z) {
  if constexpr (NDIM == 3) {
    x = m, y = (g8 >> 2) + 2 * h, z = g8 & 3;
  } else {
    x = 0, y = 2 * m + h, z = g8;
  }
}
// index of a block cell in [x][y][z] order (64 cells)
template <int NDIM>
__device__ __forceinline__ int cell_index(int x, int y, int z) {
  return NDIM == 3 ? (x * 4 + y) * 4 + z : y * 8 + z;
}

// Stores the lane's cells of block key `blk` for entries below ncoil.
template <int NDIM>
__device__ __forceinline__ void frag_store(const Geo& g, float* __restrict__ gridv, int c0, int ncoil, int blk, int g8,
                                           int t4, const float (&D)[4][2][4]) {
  int bx, by, bz;
  block_origin(g, blk, bx, by, bz);
  const int B0 = bx * block_edge(NDIM, 0), B1 = by * block_edge(NDIM, 1), B2 = bz * block_edge(NDIM, 2);
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  if (ncoil == 8 && B0 + block_edge(NDIM, 0) <= g.N[0] && B1 + block_edge(NDIM, 1) <= g.N[1] && B2 + block_edge(NDIM, 2) <= g.N[2]) {
    int lx, ly, lz;
    frag_cell<NDIM>(0, 0, g8, lx, ly, lz);
    const long long s1 = g.N[2], sm = NDIM == 3 ? (long long)g.N[1] * s1 : 2 * s1, sh = NDIM == 3 ? 2 * s1 : s1;
    float2* q = reinterpret_cast<float2*>(gridv) + (c0 + t4) * gvol + ((long long)(B0 + lx) * g.N[1] + B1 + ly) * s1 + B2 + lz;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt, q += 4 * gvol)
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          // a grid larger than L2 leaves it early, before the rows and values
          // that other blocks still need (256^3: 707 -> 688 us; 2D: no change)
          const float2 v = make_float2(D[m][nt][2 * h], D[m][nt][2 * h + 1]);
          if constexpr (NDIM == 3) __stcs(&q[m * sm + h * sh], v);
          else q[m * sm + h * sh] = v;
        }
    return;
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int lx, ly, lz;
      frag_cell<NDIM>(m, h, g8, lx, ly, lz);
      const int x = B0 + lx, y = B1 + ly, z = B2 + lz;
      if (x >= g.N[0] || y >= g.N[1] || z >= g.N[2]) continue;
      const long long cell = ((long long)x * g.N[1] + y) * g.N[2] + z;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int e = 4 * nt + t4;
        if (e < ncoil)
          *reinterpret_cast<float2*>(gridv + ((long long)(c0 + e) * gvol + cell) * 2) =
              make_float2(D[m][nt][2 * h], D[m][nt][2 * h + 1]);
      }
    }
  }
}

// Sums of one item again, entry by entry on the CUDA cores, where the tensor
// cores gave a non-finite one: a NaN or Inf among the values only reaches the
// cells of its point's window (the rows hold -0.0 outside it).
template <int NDIM, int NROW>
__device__ __noinline__ void block_by_entry(const Geo& g, const uint32_t* __restrict__ bentries, const float* __restrict__ rows,
                                            const float2* __restrict__ vals, const float4* __restrict__ tv, int cg, int ncoil,
                                            int from, int to, int g8, int t4, float (&D)[4][2][4]) {
  for (int m = 0; m < 4; ++m)
    for (int nt = 0; nt < 2; ++nt)
      for (int i = 0; i < 4; ++i) D[m][nt][i] = 0.f;
  for (int q = from; q < to; ++q) {
    const uint32_t en = bentries[q];
    long long p = en & ((1u << sel_shift(NROW)) - 1u);
    if (!TLGB_IN_RANGE(p, g.npts)) p = 0;
    int ri, rj, rk;
    sel_rows<NROW>(en, ri, rj, rk);
    const float* r = rows + p * row_floats(NDIM, NROW);
    const float* rx = r + 4 * ri;
    const float* ry = NDIM == 3 ? r + 4 * (NROW + rj) : r + 8 * rj;
    const float* rz = NDIM == 3 ? r + 4 * (2 * NROW + rk) : r + 8 * (NROW + rk);
    float2 v[2];
    for (int nt = 0; nt < 2; ++nt) {
      const int e = 4 * nt + t4;
      v[nt] = make_float2(0.f, 0.f);
      if (e < ncoil)
        v[nt] = tv ? reinterpret_cast<const float2*>(tv + ((long long)cg * g.npts + p) * 4)[e]
                   : vals[((long long)cg * 8 + e) * g.npts + p];
    }
    for (int m = 0; m < 4; ++m)
      for (int h = 0; h < 2; ++h) {
        int lx, ly, lz;
        frag_cell<NDIM>(m, h, g8, lx, ly, lz);
        const float wx = NDIM == 3 ? rx[lx] : 1.f, y = ry[ly], z = rz[lz], w = wx * (y * z);
        if (signbit(wx) || signbit(y) || signbit(z)) continue;
        for (int nt = 0; nt < 2; ++nt) {
          D[m][nt][2 * h] = fmaf(w, v[nt].x, D[m][nt][2 * h]);
          D[m][nt][2 * h + 1] = fmaf(w, v[nt].y, D[m][nt][2 * h + 1]);
        }
      }
  }
}

template <int NDIM, int NROW>
__global__ void __launch_bounds__(kBWarps * 32, kB3Ctas) adj_b3_kernel(Geo g, const int4* __restrict__ items, int nitems,
                                                        int nunits, int cg0, int ncg,
                                                        const uint32_t* __restrict__ bentries,
                                                        const float* __restrict__ rows,
                                                        const float2* __restrict__ vals,
                                                        const float4* __restrict__ tv, float* __restrict__ gridv,
                                                        float* __restrict__ partial, int* __restrict__ ctr) {
  extern __shared__ __align__(16) float bsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* S = bsm + warp * (kBStages * kBC * kBS);
  const int g8 = lane >> 2, t4 = lane & 3, half = lane / kBC;
  float* const mine = S + (lane & (kBC - 1)) * kBS;  // this lane's entry of a chunk; it copies half of it
  ChunkStream cs;
  cs.start(nunits, nitems, items, ctr, lane, warp);
  auto stage = [&](float* sl, int n, uint32_t en, int cg) {
    const int j = lane & (kBC - 1);
    if (j < n) {
      long long p = en & ((1u << sel_shift(NROW)) - 1u);
      if (!TLGB_IN_RANGE(p, g.npts)) p = 0;
      const float* rsrc = rows + p * row_floats(NDIM, NROW);
      int ri, rj, rk;
      sel_rows<NROW>(en, ri, rj, rk);
      if constexpr (NDIM == 3) {  // rows of 4 cells: x 0-3, y 4-7, z 8-11
        if (half == 0) {
          cp_async16(sl + 0, rsrc + 4 * ri);
          cp_async16(sl + 4, rsrc + 4 * (NROW + rj));
        } else {
          cp_async16(sl + 8, rsrc + 4 * (2 * NROW + rk));
        }
      } else {  // rows of 8 cells: y 0-7, z 8-15
        const float* r = rsrc + 8 * (half ? NROW + rk : rj);
        cp_async16(sl + 8 * half, r);
        cp_async16(sl + 8 * half + 4, r + 4);
      }
      if (tv) {
        const float4* vsrc = tv + ((long long)(cg0 + cg) * g.npts + p) * 4 + 2 * half;
        cp_async16(sl + 16 + 8 * half, vsrc);
        cp_async16(sl + 20 + 8 * half, vsrc + 1);
      } else {
        const long long c0 = (long long)(cg0 + cg) * 8 + 4 * half;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (c0 + q < g.nbatch)
            cp_async8(sl + 16 + 8 * half + 2 * q, vals + (c0 + q) * g.npts + p);
          else
            *reinterpret_cast<float2*>(sl + 16 + 8 * half + 2 * q) = make_float2(0.f, 0.f);
        }
      }
    } else if (j < ((n + 7) & ~7)) {  // padding entries of the last group: zero weights and values
      const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
      float4* q4 = reinterpret_cast<float4*>(sl) + 2 * half;
      q4[0] = q4[1] = q4[4] = q4[5] = z4;
    }
  };
  // the copies of kBStages - 1 chunks and the entry numbers of the one after
  // them are in flight during the work on a chunk, across items
  uint32_t en = 0;
  int ecg = 0;
  unsigned sizes = 0;  // byte i: 1 + size of the i-th chunk from here, 0 past the end
  int n = cs.next(en, ecg, nunits, nitems, items, bentries, ctr, lane);
  if (n < 0) return;
#pragma unroll
  for (int i = 0; i < kBStages - 1; ++i) {
    if (n >= 0) stage(mine + i * (kBC * kBS), n, en, ecg);
    cp_async_commit();
    sizes |= (unsigned)(n + 1) << (8 * i);
    n = cs.next(en, ecg, nunits, nitems, items, bentries, ctr, lane);
  }
  float D[4][2][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) D[m][nt][i] = 0.f;
  int unit = 0;  // of this warp
  int c = __shfl_sync(0xffffffffu, cs.desc.y, 0), cend = __shfl_sync(0xffffffffu, cs.desc.z, 0);
  for (int buf = 0;; buf = buf + 1 == kBStages ? 0 : buf + 1) {
    if (n >= 0) stage(mine + (buf == 0 ? kBStages - 1 : buf - 1) * (kBC * kBS), n, en, ecg);
    cp_async_commit();
    sizes |= (unsigned)(n + 1) << (8 * (kBStages - 1));
    n = cs.next(en, ecg, nunits, nitems, items, bentries, ctr, lane);
    cp_async_wait<kBStages - 1>();
    const int now = (int)(sizes & 255u) - 1;  // entries of this chunk
    sizes >>= 8;
    const float* B = S + buf * (kBC * kBS);
    const int n8 = (now + 7) & ~7;  // the tensor-core steps read whole groups of 8 entries
    __syncwarp();  // the lanes' copies are in
    for (int kk = 0; kk < n8; kk += 8) {  // entries kk + t4 and kk + t4 + 4 of this lane's fragments
      const float* e0 = B + (kk + t4) * kBS;
      const float* e1 = e0 + 4 * kBS;
      unsigned bh[2][2], bl[2][2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        split_tf32(e0[16 + 8 * nt + g8], bh[nt][0], bl[nt][0]);
        split_tf32(e1[16 + 8 * nt + g8], bh[nt][1], bl[nt][1]);
      }
      // A fragments of row tile m: the weights of rows g8 and g8 + 8 for entries e0 and e1
      float u0[4], u1[4], va, vb, vc, vd;
      if constexpr (NDIM == 3) {  // x m * (y (g8 >> 2) + 2h * z g8 & 3)
        const float z0 = e0[8 + (g8 & 3)], z1 = e1[8 + (g8 & 3)];
        const float4 x0 = *reinterpret_cast<const float4*>(e0), x1 = *reinterpret_cast<const float4*>(e1);
        u0[0] = x0.x, u0[1] = x0.y, u0[2] = x0.z, u0[3] = x0.w;
        u1[0] = x1.x, u1[1] = x1.y, u1[2] = x1.z, u1[3] = x1.w;
        va = e0[4 + (g8 >> 2)] * z0, vb = e0[6 + (g8 >> 2)] * z0;
        vc = e1[4 + (g8 >> 2)] * z1, vd = e1[6 + (g8 >> 2)] * z1;
      } else {  // y 2m + h * z g8
        va = vb = e0[8 + g8], vc = vd = e1[8 + g8];
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        unsigned ah[4], al[4];
        if constexpr (NDIM == 3) {
          split_tf32_mul2(u0[m], make_float2(va, vb), ah, al);
          split_tf32_mul2(u1[m], make_float2(vc, vd), ah + 2, al + 2);
        } else {
          split_tf32_mul2(va, *reinterpret_cast<const float2*>(e0 + 2 * m), ah, al);
          split_tf32_mul2(vc, *reinterpret_cast<const float2*>(e1 + 2 * m), ah + 2, al + 2);
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          mma_split(D[m][nt], ah, al, bh[nt], bl[nt]);
        }
      }
    }
    c += kBC;
    if (c >= cend) {  // the item's last chunk
      const int ix = __shfl_sync(0xffffffffu, cs.desc.x, unit & 7), iw = __shfl_sync(0xffffffffu, cs.desc.w, unit & 7);
      const int cg = cg0 + __shfl_sync(0xffffffffu, cs.group, unit & 7), c0 = cg * 8;
      const int ncoil = (int)min(8ll, g.nbatch - c0);
      float bad = 0.f;  // NaN if any sum is not finite
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) bad = fmaf(D[m][nt][i], 0.f, bad);
      if (__any_sync(0xffffffffu, !(bad == 0.f))) {
        float again[4][2][4];
        block_by_entry<NDIM, NROW>(g, bentries, rows, vals, tv, cg, ncoil, __shfl_sync(0xffffffffu, cs.desc.y, unit & 7), cend,
                                   g8, t4, again);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) D[m][nt][i] = again[m][nt][i];
      }
      if (iw >= 0) {  // a part of a split block: its slot of the partial blocks, [cell][entry] complex
        float* dst = partial + ((long long)iw * ncg + cg) * 64 * 16;
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            int lx, ly, lz;
            frag_cell<NDIM>(m, h, g8, lx, ly, lz);
            const int cell = cell_index<NDIM>(lx, ly, lz);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
              *reinterpret_cast<float2*>(dst + cell * 16 + 2 * (4 * nt + t4)) =
                  make_float2(D[m][nt][2 * h], D[m][nt][2 * h + 1]);
          }
      } else {  // one block, or a run of -iw empty ones
        for (int b = 0; b < -iw; ++b) frag_store<NDIM>(g, gridv, c0, ncoil, ix + b, g8, t4, D);
      }
      if ((sizes & 255u) == 0) return;
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) D[m][nt][i] = 0.f;
      ++unit;
      c = __shfl_sync(0xffffffffu, cs.desc.y, unit & 7), cend = __shfl_sync(0xffffffffu, cs.desc.z, unit & 7);
    }
    __syncwarp();  // the chunk has been read before its buffer is staged again
  }
}

// Sum the partial blocks of one split block in slot order, compensated (the
// dense k-space centre piles thousands of points onto a cell; each part holds
// at most kBlkPart of them). CTA = 256 threads, thread (cell, entry pair) sums
// one float4 of every part, eight in flight. Most split blocks have a few
// parts, so small CTAs keep many blocks in flight per SM; the plan lists the
// blocks with the most parts (a few hundred at the centre of a dense
// trajectory) first, so their longer chains overlap the rest.
template <int NDIM>
__global__ void __launch_bounds__(256) adj_reduce_b3_kernel(Geo g, const int4* __restrict__ split,
                                                            const float* __restrict__ partial,
                                                            float* __restrict__ gridv) {
  const int4 sp = split[blockIdx.x];
  const int cg = blockIdx.y, ncg = gridDim.y, c0 = cg * 8;
  const int ncoil = (int)min(8ll, g.nbatch - c0);
  const int r = threadIdx.x;
  const int cell = r >> 2, ep = r & 3;  // entries 2 ep, 2 ep + 1
  const long long step = (long long)ncg * 64 * 4;  // float4s between consecutive partials
  const float4* src = reinterpret_cast<const float4*>(partial + ((long long)sp.y * ncg + cg) * 64 * 16) + r;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), comp = sum;
  int k = 0;
  for (; k + 8 <= sp.z; k += 8) {
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __ldg(src + (k + i) * step);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      comp_add(sum.x, comp.x, v[i].x);
      comp_add(sum.y, comp.y, v[i].y);
      comp_add(sum.z, comp.z, v[i].z);
      comp_add(sum.w, comp.w, v[i].w);
    }
  }
  if (k < sp.z) {  // the last 1-7 parts, loaded together
    float4 v[7];
#pragma unroll
    for (int i = 0; i < 7; ++i)
      if (k + i < sp.z) v[i] = __ldg(src + (k + i) * step);
#pragma unroll
    for (int i = 0; i < 7; ++i)
      if (k + i < sp.z) {
        comp_add(sum.x, comp.x, v[i].x);
        comp_add(sum.y, comp.y, v[i].y);
        comp_add(sum.z, comp.z, v[i].z);
        comp_add(sum.w, comp.w, v[i].w);
      }
  }
  int bx, by, bz;
  block_origin(g, sp.x, bx, by, bz);
  const int x = bx * block_edge(NDIM, 0) + (NDIM == 3 ? cell >> 4 : 0);
  const int y = by * block_edge(NDIM, 1) + (NDIM == 3 ? (cell >> 2) & 3 : cell >> 3);
  const int z = bz * block_edge(NDIM, 2) + (NDIM == 3 ? cell & 3 : cell & 7);
  if (x >= g.N[0] || y >= g.N[1] || z >= g.N[2]) return;
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  float* dst = gridv + ((long long)(c0 + 2 * ep) * gvol + ((long long)x * g.N[1] + y) * g.N[2] + z) * 2;
  if (2 * ep < ncoil) *reinterpret_cast<float2*>(dst) = make_float2(sum.x + comp.x, sum.y + comp.y);
  if (2 * ep + 1 < ncoil) *reinterpret_cast<float2*>(dst + gvol * 2) = make_float2(sum.z + comp.z, sum.w + comp.w);
}


// ------------------------------------ block gridding (3D, 1, 2 or 4 entries)
//
// The same work items, counter and staging as adj_b3_kernel, with the block
// factored the other way: accumulator rows are the 16 (y, z) cells of a block
// and columns (x, real/imaginary) for each entry, so one 16 x 8 tile per
// entry holds the whole 4 x 4 x 4 block. A rank-8 update is then
// A[(y, z), e] = y row * z row (shared by the entries) times
// B[e, (x, c)] = x row * value: one m16n8k8 product (three with the tf32
// split) per batch entry and group of 8 (point, block) entries, and 8 bytes
// of values staged per batch entry instead of a 64-byte row of 8. D[j] of lane (g8, t4) holds entry j of the cells (x t4, y g8 >> 2,
// z g8 & 3) (d0, d1) and (x t4, y (g8 >> 2) + 2, z g8 & 3) (d2, d3).
constexpr int kBSn = 20;  // floats per staged entry: x row 0-3 | y row 4-7 | z row 8-11 | E values 12-19
                          // (20: the operand loads of a group of 8 entries are free of bank conflicts)
constexpr int kBnCtas = 6;  // resident CTAs per SM of the persistent grid

template <int E>
__device__ __forceinline__ void bn_store(const Geo& g, float* __restrict__ gridv, int ncoil, int blk, int g8, int t4,
                                         const float (&D)[E][4]) {
  int bx, by, bz;
  block_origin(g, blk, bx, by, bz);
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  const int x = bx * 4 + t4, z = bz * 4 + (g8 & 3);
  if (x >= g.N[0] || z >= g.N[2]) return;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int y = by * 4 + (g8 >> 2) + 2 * h;
    if (y >= g.N[1]) continue;
    const long long cell = ((long long)x * g.N[1] + y) * g.N[2] + z;
#pragma unroll
    for (int j = 0; j < E; ++j)
      if (j < ncoil)
        *reinterpret_cast<float2*>(gridv + ((long long)j * gvol + cell) * 2) = make_float2(D[j][2 * h], D[j][2 * h + 1]);
  }
}

// Sums of one item again where one is not finite (see block_by_entry).
template <int E, int NROW>
__device__ __noinline__ void block_by_entry_n(const Geo& g, const uint32_t* __restrict__ bentries, const float* __restrict__ rows,
                                              const float2* __restrict__ vals, int ncoil, int from, int to, int g8, int t4,
                                              float (&D)[E][4]) {
  for (int j = 0; j < E; ++j)
    for (int i = 0; i < 4; ++i) D[j][i] = 0.f;
  for (int q = from; q < to; ++q) {
    const uint32_t en = bentries[q];
    long long p = en & ((1u << sel_shift(NROW)) - 1u);
    if (!TLGB_IN_RANGE(p, g.npts)) p = 0;
    int ri, rj, rk;
    sel_rows<NROW>(en, ri, rj, rk);
    const float* r = rows + p * row_floats(3, NROW);
    const float wx = r[4 * ri + t4], z = r[4 * (2 * NROW + rk) + (g8 & 3)];
    for (int h = 0; h < 2; ++h) {
      const float y = r[4 * (NROW + rj) + (g8 >> 2) + 2 * h], w = wx * (y * z);
      if (signbit(wx) || signbit(y) || signbit(z)) continue;
      for (int j = 0; j < ncoil; ++j) {
        const float2 v = vals[(long long)j * g.npts + p];
        D[j][2 * h] = fmaf(w, v.x, D[j][2 * h]);
        D[j][2 * h + 1] = fmaf(w, v.y, D[j][2 * h + 1]);
      }
    }
  }
}

template <int E, int NROW>
__global__ void __launch_bounds__(kBWarps * 32, kBnCtas) adj_bn_kernel(Geo g, const int4* __restrict__ items, int nitems,
                                                             const uint32_t* __restrict__ bentries,
                                                             const float* __restrict__ rows,
                                                             const float2* __restrict__ vals,
                                                             float* __restrict__ gridv, float* __restrict__ partial,
                                                             int* __restrict__ ctr) {
  extern __shared__ __align__(16) float bsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* S = bsm + warp * (kBStages * kBC * kBSn);
  const int ncoil = (int)min((long long)E, g.nbatch);
  const int g8 = lane >> 2, t4 = lane & 3, half = lane / kBC;
  float* const mine = S + (lane & (kBC - 1)) * kBSn;
  ChunkStream cs;
  cs.start(nitems, nitems, items, ctr, lane, warp);
  auto stage = [&](float* sl, int n, uint32_t en) {
    const int q = lane & (kBC - 1);
    if (q < n) {
      long long p = en & ((1u << sel_shift(NROW)) - 1u);
      if (!TLGB_IN_RANGE(p, g.npts)) p = 0;
      const float* rsrc = rows + p * row_floats(3, NROW);
      int ri, rj, rk;
      sel_rows<NROW>(en, ri, rj, rk);
      if (half == 0) {
        cp_async16(sl + 0, rsrc + 4 * ri);
        cp_async16(sl + 4, rsrc + 4 * (NROW + rj));
      } else {
        cp_async16(sl + 8, rsrc + 4 * (2 * NROW + rk));
      }
#pragma unroll
      for (int j = 0; j < E; ++j) {
        if ((j & 1) == half) continue;  // the lane with one row takes entries 0 and 2
        if (j < ncoil)
          cp_async8(sl + 12 + 2 * j, vals + (long long)j * g.npts + p);
        else
          *reinterpret_cast<float2*>(sl + 12 + 2 * j) = make_float2(0.f, 0.f);
      }
    } else if (q < ((n + 7) & ~7) && half == 0) {  // padding entries of the last group: zero weights and values
      const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
      float4* q4 = reinterpret_cast<float4*>(sl);
      q4[0] = q4[1] = q4[2] = z4;
#pragma unroll
      for (int j = 0; j < E; ++j) *reinterpret_cast<float2*>(sl + 12 + 2 * j) = make_float2(0.f, 0.f);
    }
  };
  uint32_t en = 0;
  int ecg = 0;
  unsigned sizes = 0;  // byte i: 1 + size of the i-th chunk from here, 0 past the end
  int n = cs.next(en, ecg, nitems, nitems, items, bentries, ctr, lane);
  if (n < 0) return;
#pragma unroll
  for (int i = 0; i < kBStages - 1; ++i) {
    if (n >= 0) stage(mine + i * (kBC * kBSn), n, en);
    cp_async_commit();
    sizes |= (unsigned)(n + 1) << (8 * i);
    n = cs.next(en, ecg, nitems, nitems, items, bentries, ctr, lane);
  }
  float D[E][4];
#pragma unroll
  for (int j = 0; j < E; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) D[j][i] = 0.f;
  int unit = 0;
  int c = __shfl_sync(0xffffffffu, cs.desc.y, 0), cend = __shfl_sync(0xffffffffu, cs.desc.z, 0);
  for (int buf = 0;; buf = buf + 1 == kBStages ? 0 : buf + 1) {
    if (n >= 0) stage(mine + (buf == 0 ? kBStages - 1 : buf - 1) * (kBC * kBSn), n, en);
    cp_async_commit();
    sizes |= (unsigned)(n + 1) << (8 * (kBStages - 1));
    n = cs.next(en, ecg, nitems, nitems, items, bentries, ctr, lane);
    cp_async_wait<kBStages - 1>();
    const int now = (int)(sizes & 255u) - 1;  // entries of this chunk
    sizes >>= 8;
    const float* B = S + buf * (kBC * kBSn);
    const int n8 = (now + 7) & ~7;
    __syncwarp();  // the lanes' copies are in
    for (int kk = 0; kk < n8; kk += 8) {  // entries kk + t4 and kk + t4 + 4 of this lane's fragments
      const float* e0 = B + (kk + t4) * kBSn;
      const float* e1 = e0 + 4 * kBSn;
      // A: rows g8 and g8 + 8 = (y (g8 >> 2) + 2h, z g8 & 3)
      const float z0 = e0[8 + (g8 & 3)], z1 = e1[8 + (g8 & 3)];
      unsigned ah[4], al[4];
      split_tf32_mul2(z0, make_float2(e0[4 + (g8 >> 2)], e0[6 + (g8 >> 2)]), ah, al);
      split_tf32_mul2(z1, make_float2(e1[4 + (g8 >> 2)], e1[6 + (g8 >> 2)]), ah + 2, al + 2);
      // B: column g8 = (x g8 >> 1, c g8 & 1) of entry j
      const float x0 = e0[g8 >> 1], x1 = e1[g8 >> 1];
#pragma unroll
      for (int j = 0; j < E; ++j) {
        unsigned bh[2], bl[2];
        split_tf32_mul(e0[12 + 2 * j + (g8 & 1)], x0, bh[0], bl[0]);
        split_tf32_mul(e1[12 + 2 * j + (g8 & 1)], x1, bh[1], bl[1]);
        mma_split(D[j], ah, al, bh, bl);
      }
    }
    c += kBC;
    if (c >= cend) {  // the item's last chunk
      const int ix = __shfl_sync(0xffffffffu, cs.desc.x, unit & 7), iw = __shfl_sync(0xffffffffu, cs.desc.w, unit & 7);
      float bad = 0.f;  // NaN if any sum is not finite
#pragma unroll
      for (int j = 0; j < E; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) bad = fmaf(D[j][i], 0.f, bad);
      if (__any_sync(0xffffffffu, !(bad == 0.f))) {
        float again[E][4];
        block_by_entry_n<E, NROW>(g, bentries, rows, vals, ncoil, __shfl_sync(0xffffffffu, cs.desc.y, unit & 7), cend, g8, t4,
                                  again);
#pragma unroll
        for (int j = 0; j < E; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) D[j][i] = again[j][i];
      }
      if (iw >= 0) {  // a part of a split block: its slot of the partial blocks, [cell][entry] complex
        float* dst = partial + (long long)iw * 64 * 2 * E;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int cell = cell_index<3>(t4, (g8 >> 2) + 2 * h, g8 & 3);
#pragma unroll
          for (int j = 0; j < E; ++j)
            *reinterpret_cast<float2*>(dst + (cell * E + j) * 2) = make_float2(D[j][2 * h], D[j][2 * h + 1]);
        }
      } else {  // one block, or a run of -iw empty ones
        for (int b = 0; b < -iw; ++b) bn_store<E>(g, gridv, ncoil, ix + b, g8, t4, D);
      }
      if ((sizes & 255u) == 0) return;
#pragma unroll
      for (int j = 0; j < E; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) D[j][i] = 0.f;
      ++unit;
      c = __shfl_sync(0xffffffffu, cs.desc.y, unit & 7), cend = __shfl_sync(0xffffffffu, cs.desc.z, unit & 7);
    }
    __syncwarp();  // the chunk has been read before its buffer is staged again
  }
}

// Sum the partial blocks of one split block of adj_bn_kernel in slot order,
// compensated. CTA = 256 threads: thread (range r, cell, entry) sums one
// complex value of every part of the r-th of 256 / (64 E) consecutive part
// ranges, eight in flight; then the ranges are added in order. With one or
// two entries the ranges cut the longest chain (the densest block has a few
// hundred parts) by 4 or 2.
template <int E>
__global__ void __launch_bounds__(256) adj_reduce_bn_kernel(Geo g, const int4* __restrict__ split,
                                                           const float* __restrict__ partial,
                                                           float* __restrict__ gridv) {
  constexpr int U = 64 * E, R = 256 / U;  // values per part, part ranges
  __shared__ float2 rs[R > 1 ? R - 1 : 1][U], rc[R > 1 ? R - 1 : 1][U];
  const int4 sp = split[blockIdx.x];
  const int r = threadIdx.x / U, t = threadIdx.x % U, cell = t / E, j = t % E;
  const int ncoil = (int)min((long long)E, g.nbatch);
  const float2* src = reinterpret_cast<const float2*>(partial) + (long long)sp.y * U + t;
  const int k0 = (int)((long long)sp.z * r / R), k1 = (int)((long long)sp.z * (r + 1) / R);
  float2 sum = make_float2(0.f, 0.f), comp = sum;
  int k = k0;
  for (; k + 8 <= k1; k += 8) {
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __ldg(src + (long long)(k + i) * U);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      comp_add(sum.x, comp.x, v[i].x);
      comp_add(sum.y, comp.y, v[i].y);
    }
  }
  for (; k < k1; ++k) {
    const float2 v = __ldg(src + (long long)k * U);
    comp_add(sum.x, comp.x, v.x);
    comp_add(sum.y, comp.y, v.y);
  }
  if constexpr (R > 1) {
    if (r > 0) {
      rs[r - 1][t] = sum;
      rc[r - 1][t] = comp;
    }
    __syncthreads();
    if (r > 0) return;
#pragma unroll
    for (int i = 0; i < R - 1; ++i) {  // the later ranges in order, their compensations with them
      const float2 s2 = rs[i][t], c2 = rc[i][t];
      comp_add(sum.x, comp.x, s2.x);
      comp_add(sum.y, comp.y, s2.y);
      comp.x += c2.x, comp.y += c2.y;
    }
  }
  if (j >= ncoil) return;
  int bx, by, bz;
  block_origin(g, sp.x, bx, by, bz);
  const int x = bx * 4 + (cell >> 4), y = by * 4 + ((cell >> 2) & 3), z = bz * 4 + (cell & 3);
  if (x >= g.N[0] || y >= g.N[1] || z >= g.N[2]) return;
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  *reinterpret_cast<float2*>(gridv + ((long long)j * gvol + ((long long)x * g.N[1] + y) * g.N[2] + z) * 2) =
      make_float2(sum.x + comp.x, sum.y + comp.y);
}

// ------------------------------------------------------------------ gather
//
// Ungridding of complex values in 2D and 3D from the plan's gather records.
// A persistent CTA works through units: one item (at most kGatherPts home
// points of one tile) and a run of groups of CG batch entries. The tile's
// region (12^3 cells in 3D; 20^2, or 24^2 for kernels of more than 5 taps, in
// 2D) of a group is one stage of a ring of NST buffers in shared memory, the
// item's records one of two record buffers, each with a full and an empty
// mbarrier. Five producer warps fill them ahead of the NW consumer warps: the
// region by one TMA tensor copy when it needs no wrap and its rows are 16-byte
// multiples, else by 8-byte asynchronous copies; the records, which lie in
// the items' order, by one bulk copy. So a copy's latency is paid once per
// CTA, not once per item (with one CTA per item, a tile of 33 points cost
// 8.6 us of latency and its 110 KB of copies 1.3).
// A consumer warp takes PPW points per step: lane = (point h, entry c, z tap
// kz); a lane sums its entry's y (and x) taps for EPL entries, the 4 z-tap
// lanes add up. The regions of the entries are a multiple of 128 bytes
// apart (the same banks), so lane group l reads its y taps from row l & 3 on:
// one load of a half-warp then spans all banks.
// Every wait is bounded: on a timeout the warp sets the device status and a
// CTA flag and returns; the producers always end with their copies landed.
constexpr int kGatherPts = 256;
constexpr uint32_t kWaitLimit = 1u << 22;   // polls of a bounded wait, each of some microseconds at most
constexpr uint32_t kDrainLimit = 1u << 18;  // for copies in flight at a producer's end: about a second
constexpr int kGatherProd = 160;  // producer threads (a 12 x 12 plane of a 3D region takes 144)

template <int NDIM, int KT>
struct __align__(16) GatherRec {
  float w[NDIM][KT];  // weights of the first KT valid taps per dim, zero beyond
  unsigned view;      // region cell of the first tap | fast << 20 (at most KT taps per dim) | partial << 21 (fewer in some)
  int p;              // point index
  int pad[2];
};
static_assert(sizeof(GatherRec<3, 4>) == 64 && sizeof(GatherRec<2, 4>) == 48 && sizeof(GatherRec<2, 8>) == 80, "records");

// region edge along an active dim: the tile and one cell more than KT - 1,
// for windows of KT + 1 taps (exact-integer coordinates)
template <int NDIM, int KT>
constexpr int region_edge() { return (NDIM == 3 ? 8 : 16) + KT; }
template <int NDIM, int KT>
constexpr int region_cells() {
  return (NDIM == 3 ? region_edge<NDIM, KT>() : 1) * region_edge<NDIM, KT>() * region_edge<NDIM, KT>();
}

template <int NDIM, int KT>
struct SlowTaps {  // a window of more than KT taps, one per consumer warp
  float w[NDIM][KT + 1];
  int n[NDIM], f[NDIM];
};

template <int NDIM, int KT, int CG, int NW, int NST>
constexpr size_t gather_smem() {
  return (size_t)NST * region_cells<NDIM, KT>() * CG * 8 + 2 * kGatherPts * sizeof(GatherRec<NDIM, KT>) +
         NW * sizeof(SlowTaps<NDIM, KT>) + 8 * (2 * NST + 4) + 16;
}

__device__ __forceinline__ void item_origin(const Geo& g, int tile, int (&o)[3]) {
  int t = tile;
  o[2] = (t % g.nt[2]) * g.T[2];
  t /= g.nt[2];
  o[1] = (t % g.nt[1]) * g.T[1];
  o[0] = (t / g.nt[1]) * g.T[0];
}

// One record per home point, in the order of the gather items' points
// (item.w is the first one's index), so an item's records are one run. For 3D
// plans also each point's place in that order (`rank`). And of every 16th
// item's points (jumps[-1]) how many lie in another 32-byte sector of an output
// row than the point before (jumps[0]: nearly all for points in random order,
// a quarter in runs). jumps[-2]: whether some window has fewer than KT taps in a
// dim.
template <int NDIM, int KT, bool FROM_ROWS>
__global__ void __launch_bounds__(128) plan_records_kernel(Geo g, const uint32_t* __restrict__ cnt,
                                                           const int4* __restrict__ win,
                                                           const float* __restrict__ rows,
                                                           const int4* __restrict__ items,
                                                           const int32_t* __restrict__ entries,
                                                           const float* __restrict__ locs,
                                                           GatherRec<NDIM, KT>* __restrict__ recs,
                                                           int32_t* __restrict__ rank, uint32_t* __restrict__ jumps) {
  constexpr int S = region_edge<NDIM, KT>();
  if (blockIdx.x >= cnt[4]) return;
  const int4 it = items[blockIdx.x];
  int o[3];
  item_origin(g, it.x, o);
  for (int j = it.y + threadIdx.x; j < it.z; j += 128) {
    const int p = entries[j];
    GatherRec<NDIM, KT> R;
    unsigned base = 0;
    bool fast = true, partial = false;
    int4 w4;
    if constexpr (FROM_ROWS) w4 = win[p];
#pragma unroll
    for (int d = 0; d < NDIM; ++d) {
      const int e = d + 3 - NDIM;
      int c = 0, st = 0;
      float w[KT + 1];
#pragma unroll
      for (int k = 0; k <= KT; ++k) w[k] = 0.f;
      if constexpr (FROM_ROWS) {
        // the window's weights are the row's cells with a clear sign, in order
        st = win_st(w4, e), c = win_cnt(w4, e);
        constexpr int EDGE = NDIM == 3 ? 4 : 8;
        const float4* row = reinterpret_cast<const float4*>(rows + (long long)p * row_floats(NDIM, g.nrow) + d * g.nrow * EDGE);
        int i0 = 0;
        for (int q = 0; q < g.nrow * EDGE / 4; ++q) {
          const float4 v4 = __ldg(row + q);
          const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (signbit(v[k])) continue;
#pragma unroll
            for (int i = 0; i < KT; ++i) w[i] = i0 == i ? v[k] : w[i];
            ++i0;
          }
        }
      } else {
        const float x = load_coord(g, locs, p, e);
        const int lower = lower_of(g, e, x);
#pragma unroll
        for (int k = 0; k <= KT; ++k) {
          if (k >= g.NT[e]) continue;
          const Tap t = tap_eval(g, e, x, lower, k);
          if (!t.valid) continue;
          if (c == 0) st = g.pad == TLGB_PAD_CIRCULAR ? wrapi(lower + k, g.N[e]) : lower + k;
          const float v = kern_precise(g.kernel, __fsub_rn(x, (float)(lower + k)), g.r[e], t.d, g.beta, g.beta_lo);
#pragma unroll
          for (int i = 0; i < KT; ++i) w[i] = c == i ? v : w[i];
          ++c;
        }
      }
#pragma unroll
      for (int k = 0; k < KT; ++k) R.w[d][k] = w[k];
      // a home point's first tap lies in the tile
      base = base * S + (unsigned)(st - o[e]);
      fast = fast && c <= KT;
      partial = partial || c < KT;
    }
    R.view = (fast ? base : 0u) | ((fast ? 1u : 0u) << 20) | ((partial ? 1u : 0u) << 21);
    if (fast && partial) jumps[-2] = 1u;
    R.p = p;
    R.pad[0] = R.pad[1] = 0;
    const float4* src = reinterpret_cast<const float4*>(&R);
    float4* dst = reinterpret_cast<float4*>(recs + it.w + (j - it.y));
#pragma unroll
    for (int q = 0; q < (int)(sizeof(R) / 16); ++q) dst[q] = src[q];
    if (rank) rank[p] = it.w + (j - it.y);
    if (blockIdx.x % 16 == 0) {
      const unsigned on = __activemask();
      const unsigned m = __ballot_sync(on, j == it.y || entries[j - 1] >> 2 != p >> 2);
      if ((threadIdx.x & 31) == 0) {
        atomicAdd(jumps, (uint32_t)__popc(m));
        atomicAdd(jumps - 1, (uint32_t)__popc(on));
      }
    }
  }
}

// The end of a producer thread, whether it has issued every copy or given up:
// nothing that it started is in flight when the CTA ends. A consumer whose wait
// ran out returns at once, and the CTA's shared memory may be another's next. In
// a pass without a failure the copies have landed or are about to.
__device__ __forceinline__ void producer_drain(uint64_t* full, uint32_t stages, uint32_t nst, uint64_t* rfull,
                                               uint32_t recs_sent, int pt) {
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (pt != 0) return;
  for (uint32_t i = stages > nst ? stages - nst : 0; i < stages; ++i) mbar_wait_bounded(&full[i % nst], (i / nst) & 1, kDrainLimit);
  for (uint32_t i = recs_sent > 2 ? recs_sent - 2 : 0; i < recs_sent; ++i) mbar_wait_bounded(&rfull[i & 1], (i >> 1) & 1, kDrainLimit);
}

// A region by asynchronous 8-byte copies of the producer threads, wrapped or
// zero-filled: a thread copies its (y, z) cells of every (entry, x) plane.
template <int NDIM, int KT, int CG>
__device__ __forceinline__ void copy_region(const Geo& g, const float* __restrict__ gridv, float2* reg, const int (&o)[3],
                                            int cg, int pt) {
  constexpr int S = region_edge<NDIM, KT>(), PLANE = S * S;
  constexpr int Q = (PLANE + kGatherProd - 1) / kGatherProd;
  const long long gpl = (long long)g.N[1] * g.N[2], gvol = gpl * g.N[0];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int cell = pt + q * kGatherProd;
    if (cell >= PLANE) break;
    const int y = cell / S, z = cell - y * S;
    int gy = o[1] + y, gz = o[2] + z;
    bool in = gy < g.N[1] && gz < g.N[2];
    if (g.pad == TLGB_PAD_CIRCULAR) gy = wrapi(gy, g.N[1]), gz = wrapi(gz, g.N[2]), in = true;
    const float2* src = reinterpret_cast<const float2*>(gridv) + (long long)(cg * CG) * gvol +
                        (in ? (long long)gy * g.N[2] + gz : 0);
    float2* dst = reg + cell;
    for (int c = 0; c < CG; ++c, src += gvol) {
      const bool cin = in && cg * CG + c < g.nbatch;
      if constexpr (NDIM == 3) {
        int gx = o[0];
        const float2* sx = src + (long long)gx * gpl;
        for (int x = 0; x < S; ++x, dst += PLANE, sx += gpl) {
          bool xin = cin;
          if (gx >= g.N[0]) {  // past the upper edge
            if (g.pad == TLGB_PAD_CIRCULAR)
              gx -= g.N[0], sx -= gvol;
            else
              xin = false;
          }
          sm100::cp_async8_zfill(dst, xin ? sx : reinterpret_cast<const float2*>(gridv), xin);
          ++gx;
        }
      } else {
        sm100::cp_async8_zfill(dst, cin ? src : reinterpret_cast<const float2*>(gridv), cin);
        dst += PLANE;
      }
    }
  }
}

// PARTIAL: some window has fewer than KT taps in a dim. Its zero weights carry a
// NaN or Inf of the box's cells past the window into the sum, so such results
// are summed again over the valid taps. Plans without such windows (width 4 or 8
// off the edges) leave the check out: it makes each step wait for its sums (256^3
// x 8: 573 -> 580 us; 256 entries of 320^2: 50 us of a training step's 2.75 ms).
// With zero padding few windows are cut, and only their steps wait: 8 entries of
// 128 x 120 x 96 at 262,144 points 85 us, 92 with every step waiting, 83 without.
template <int NDIM, int KT, int CG, int NW, int NST, int CTAS, bool PARTIAL>
__global__ void __launch_bounds__(NW * 32 + kGatherProd, CTAS)
    gather_kernel(const __grid_constant__ CUtensorMap tmap, int use_tma, Geo g, const int4* __restrict__ items, int nruns,
                  int run, int nunits, const GatherRec<NDIM, KT>* __restrict__ recs, const float* __restrict__ locs,
                  const float* __restrict__ gridv, float* __restrict__ out, float* __restrict__ sorted) {
  constexpr int S = region_edge<NDIM, KT>(), VOL = region_cells<NDIM, KT>(), PLANE = S * S;
  constexpr int CL = CG < 4 ? CG : 4, EPL = CG / CL, PPW = 8 / CL;
  constexpr uint32_t RBYTES = VOL * CG * 8;
  using Rec = GatherRec<NDIM, KT>;
  extern __shared__ __align__(128) unsigned char smem[];
  Rec* recbuf = reinterpret_cast<Rec*>(smem + NST * RBYTES);
  SlowTaps<NDIM, KT>* slow = reinterpret_cast<SlowTaps<NDIM, KT>*>(recbuf + 2 * kGatherPts);
  uint64_t* full = reinterpret_cast<uint64_t*>((reinterpret_cast<uintptr_t>(slow + NW) + 7) & ~(uintptr_t)7);
  uint64_t* empty = full + NST;
  uint64_t* rfull = empty + NST;
  uint64_t* rempty = rfull + 2;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(&full[i], kGatherProd);
      mbar_init(&empty[i], NW);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&rfull[i], 1);
      mbar_init(&rempty[i], NW);
    }
    fence_mbar_init();
    failed = 0;
  }
  __syncthreads();
  const uint32_t limit = g.wait;
  const int ncg = (int)((g.nbatch + CG - 1) / CG);
  volatile int* vfailed = &failed;
  if (warp >= NW) {
    // ---- producers
    if (g.skip_copy == 1) return;
    const int pt = tid - NW * 32;
    uint32_t k = 0, u_done = 0, recs_sent = 0;  // stages, units, record copies begun (thread 0)
    bool ok = true;
    int4 next = blockIdx.x < nunits ? items[blockIdx.x / nruns] : make_int4(0, 0, 0, 0);
    for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x, ++u_done) {
      const int4 it = next;
      if (u + (int)gridDim.x < nunits) next = items[(u + gridDim.x) / nruns];
      const int g0 = (u % nruns) * run, g1 = min(ncg, g0 + run);
      int o[3];
      item_origin(g, it.x, o);
      bool wraps = false;
      for (int e = 3 - NDIM; e < 3; ++e) wraps = wraps || (g.pad == TLGB_PAD_CIRCULAR && o[e] + S > g.N[e]);
      const bool tma = use_tma && !wraps;
      if (pt == 0) {
        const uint32_t b = u_done & 1;
        ok = mbar_wait_bounded(&rempty[b], ((u_done >> 1) & 1) ^ 1, kWaitLimit);
        if (ok) {
          const uint32_t bytes = (uint32_t)(it.z - it.y) * (uint32_t)sizeof(Rec);
          mbar_arrive_expect_tx(&rfull[b], bytes);
          sm100::bulk_load(recbuf + b * kGatherPts, recs + it.w, bytes, &rfull[b]);
          ++recs_sent;
        }
      }
      for (int cg = g0; cg < g1 && ok; ++cg, ++k) {
        const uint32_t s = k % NST;
        ok = mbar_wait_bounded(&empty[s], ((k / NST) & 1) ^ 1, kWaitLimit) && !*vfailed;
        if (!ok) break;
        float2* reg = reinterpret_cast<float2*>(smem + s * RBYTES);
        if (tma) {
          if (pt == 0) {
            sm100::fence_proxy_async_smem();  // the buffer may last have been filled by plain copies
            mbar_arrive_expect_tx(&full[s], RBYTES);
            tma_load_4d(reg, &tmap, &full[s], o[2], o[1], o[0], cg * CG);
          } else {
            sm100::mbar_arrive(&full[s]);
          }
          continue;
        }
        copy_region<NDIM, KT, CG>(g, gridv, reg, o, cg, pt);
        sm100::cp_async_mbar_arrive(&full[s]);
      }
      ok = ok && !*vfailed;
    }
    if (!ok && pt == 0) {
      *vfailed = 1;
      atomicExch(&g_tlgb_status, 1);
    }
    producer_drain(full, k, NST, rfull, recs_sent, pt);
    return;
  }
  // ---- consumers
  const int kz = lane & 3, c = (lane >> 2) % CL, h = lane / (4 * CL);
  int kyo[4], rowoff[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    kyo[t] = (t + (lane >> 2)) & 3;
    rowoff[t] = kyo[t] * S;
  }
  auto give_up = [&]() {
    if (lane == 0) {
      *vfailed = 1;
      atomicExch(&g_tlgb_status, 1);
    }
  };
  uint32_t k = 0, ui = 0;
  int4 next = blockIdx.x < nunits ? items[blockIdx.x / nruns] : make_int4(0, 0, 0, 0);
  for (int u = blockIdx.x; u < nunits; u += gridDim.x, ++ui) {
    const int4 it = next;
    if (u + (int)gridDim.x < nunits) next = items[(u + gridDim.x) / nruns];
    const int g0 = (u % nruns) * run, g1 = min(ncg, g0 + run), npt = it.z - it.y;
    const Rec* rec = recbuf + (ui & 1) * kGatherPts;
    if (!mbar_wait_bounded(&rfull[ui & 1], (ui >> 1) & 1, limit)) return give_up();
    for (int cg = g0; cg < g1; ++cg, ++k) {
      const uint32_t s = k % NST;
      if (!mbar_wait_bounded(&full[s], (k / NST) & 1, limit)) return give_up();
      const float2* reg = reinterpret_cast<const float2*>(smem + s * RBYTES);
      const int c0 = cg * CG;
      for (int base = warp * PPW; base < npt; base += NW * PPW) {
        const bool on = base + h < npt;
        const Rec& R = rec[on ? base + h : base];
        const unsigned view = R.view;
        const int p = R.p;
        const float2* a = reg + c * VOL + (view & 0xfffff) + kz;
        float2 acc[EPL];
#pragma unroll
        for (int q = 0; q < EPL; ++q) acc[q] = make_float2(0.f, 0.f);
        // the box's farthest cell from its first one, for the last entry
        if (TLGB_IN_RANGE((view & 0xfffff) + ((NDIM == 3 ? 3 * PLANE : 0) + (KT - 1) * S + KT - 1), VOL)) {
          if constexpr (NDIM == 3) {
            const float4 wx = *reinterpret_cast<const float4*>(R.w[0]);
            const float wz = R.w[2][kz];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const float wyz = R.w[1][kyo[t]] * wz;
#pragma unroll
              for (int q = 0; q < EPL; ++q) {
                const float2* ar = a + q * CL * VOL + rowoff[t];
                float2 sx = mul2_bcast(wx.x, ar[0]);
                fma2_bcast(sx, wx.y, ar[PLANE]);
                fma2_bcast(sx, wx.z, ar[2 * PLANE]);
                fma2_bcast(sx, wx.w, ar[3 * PLANE]);
                acc[q].x = fmaf(wyz, sx.x, acc[q].x);
                acc[q].y = fmaf(wyz, sx.y, acc[q].y);
              }
            }
          } else {
#pragma unroll
            for (int zb = 0; zb < KT; zb += 4) {
              const float wz = R.w[1][zb + kz];
#pragma unroll
              for (int yb = 0; yb < KT; yb += 4) {
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  const float w = R.w[0][yb + kyo[t]] * wz;
#pragma unroll
                  for (int q = 0; q < EPL; ++q) {
                    const float2 v = a[q * CL * VOL + yb * S + rowoff[t] + zb];
                    acc[q].x = fmaf(w, v.x, acc[q].x);
                    acc[q].y = fmaf(w, v.y, acc[q].y);
                  }
                }
              }
            }
          }
        }
        // the 4 z-tap lanes add up, each ending with one component
        float sum;
        int ent, comp;
        if constexpr (EPL == 2) {
          const bool hi = kz & 2;
          float2 keep = hi ? acc[1] : acc[0];
          const float2 send = hi ? acc[0] : acc[1];
          keep.x += __shfl_xor_sync(0xffffffffu, send.x, 2);
          keep.y += __shfl_xor_sync(0xffffffffu, send.y, 2);
          sum = kz & 1 ? keep.y : keep.x;
          sum += __shfl_xor_sync(0xffffffffu, kz & 1 ? keep.x : keep.y, 1);
          ent = c + (hi ? CL : 0), comp = kz & 1;
        } else {
          sum = kz & 1 ? acc[0].y : acc[0].x;
          sum += __shfl_xor_sync(0xffffffffu, kz & 1 ? acc[0].x : acc[0].y, 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          ent = c, comp = kz & 1;
        }
        const bool fast = (view >> 20) & 1;
        if (on && fast && (EPL == 2 || kz < 2) && c0 + ent < g.nbatch && TLGB_IN_RANGE(p, g.npts)) {
          if (sorted)
            sorted[(((long long)cg * g.npts + it.w + base + h) * CG + ent) * 2 + comp] = sum;
          else
            out[((long long)(c0 + ent) * g.npts + p) * 2 + comp] = sum;
        }
        // the step's points with more than KT taps in a dim (and those to sum
        // again), one at a time by the whole warp
        unsigned again;
        if constexpr (PARTIAL) {  // the first vote, which the other points' steps end with, does not wait for the sums
          const bool part = (view >> 21) & 1;
          again = __ballot_sync(0xffffffffu, on && (!fast || part));
          if (again) again = __ballot_sync(0xffffffffu, on && (!fast || (part && !(fabsf(sum) <= FLT_MAX))));
        } else {
          again = __ballot_sync(0xffffffffu, on && !fast);
        }
        unsigned rest = again;
        while (rest) {
          const int hh = (__ffs(rest) - 1) / (4 * CL);
          rest &= ~(((1u << (4 * CL)) - 1u) << (4 * CL * hh));
          const Rec& Q = rec[base + hh];
          SlowTaps<NDIM, KT>& T = slow[warp];
          {
            constexpr int NTM = KT + 1;
            const int d = lane / NTM, kk = lane % NTM, e = d + 3 - NDIM;
            Tap t;
            t.valid = false;
            float x = 0.f;
            int lower = 0;
            if (d < NDIM) {
              x = load_coord(g, locs, Q.p, e);
              lower = lower_of(g, e, x);
              if (kk < g.NT[e]) t = tap_eval(g, e, x, lower, kk);
            }
            const unsigned m = (__ballot_sync(0xffffffffu, t.valid) >> (d < NDIM ? d * NTM : 0)) & ((1u << NTM) - 1);
            if (t.valid)
              T.w[d][kk - (__ffs(m) - 1)] = kern_precise(g.kernel, __fsub_rn(x, (float)(lower + kk)), g.r[e], t.d, g.beta, g.beta_lo);
            if (d < NDIM && kk == 0) {
              int st = lower + __ffs(m) - 1;
              if (g.pad == TLGB_PAD_CIRCULAR) st = wrapi(st, g.N[e]);
              T.n[d] = __popc(m);
              int o[3];
              item_origin(g, it.x, o);
              T.f[d] = st - (e == 2 ? o[2] : (e == 1 ? o[1] : o[0]));
            }
          }
          __syncwarp();
          const int e8 = lane % CG, n2 = T.n[NDIM - 1], n1 = T.n[NDIM - 2], n0 = NDIM == 3 ? T.n[0] : 1;
          float2 v2 = make_float2(0.f, 0.f);
          // all KT + 1 taps per dim, for divisions by a constant: with the window's own counts 8 x 262,144 spline
          // points on 128 x 120 x 96 (5 taps each) took 1057 us, 934 so
          for (int t = lane / CG; t < (NDIM == 3 ? (KT + 1) * (KT + 1) : KT + 1) * (KT + 1); t += 32 / CG) {
            const int z = t % (KT + 1), yx = t / (KT + 1), y = yx % (KT + 1), x = yx / (KT + 1);
            if (z >= n2 || y >= n1 || x >= n0) continue;
            float w = T.w[NDIM - 2][y] * T.w[NDIM - 1][z];
            int cell = (T.f[NDIM - 2] + y) * S + T.f[NDIM - 1] + z;
            if (NDIM == 3) {
              w *= T.w[0][x];
              cell += (T.f[0] + x) * PLANE;
            }
            if (TLGB_IN_RANGE(cell, VOL)) fma2_bcast(v2, w, reg[e8 * VOL + cell]);
          }
          for (int m = CG; m < 32; m <<= 1) {
            v2.x += __shfl_xor_sync(0xffffffffu, v2.x, m);
            v2.y += __shfl_xor_sync(0xffffffffu, v2.y, m);
          }
          // only entries with a flagged component: in lanes 4 (e % CL) + 2 (e / CL) and one on from the point's first
          const bool mine = !PARTIAL || ((again >> ((4 * CL * hh + 4 * (lane % CL) + 2 * (lane / CL)) & 31)) & 3);
          if (lane < CG && mine && c0 + lane < g.nbatch && TLGB_IN_RANGE(Q.p, g.npts))
            *reinterpret_cast<float2*>(sorted ? sorted + (((long long)cg * g.npts + it.w + base + hh) * CG + lane) * 2
                                              : out + ((long long)(c0 + lane) * g.npts + Q.p) * 2) = v2;
          __syncwarp();
        }
      }
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&empty[s]);
    }
    if (lane == 0) sm100::mbar_arrive(&rempty[ui & 1]);
  }
}

// [group][place][4] -> [entry][point]: the gather's results out of the items'
// order (zero for points without taps). CTA = 128 points of one group; a
// thread reads 16 of a point's 32 bytes, a warp writes 32 points of an entry.
// HBM-bound: 64 MB out of 64 MB take 23 us.
__global__ void __launch_bounds__(256) unsort_kernel(const float4* __restrict__ sorted, const int32_t* __restrict__ rank,
                                                     long long npts, long long nbatch, float2* __restrict__ out) {
  __shared__ float2 sm[4][128 + 4];
  const int t = threadIdx.x, grp = blockIdx.y;
  const long long p0 = (long long)blockIdx.x * 128;
  {
    const int i = t >> 1, q = t & 1;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p0 + i < npts) {
      const int r = rank[p0 + i];
      if (r >= 0) v = __ldg(sorted + ((long long)grp * npts + r) * 2 + q);
    }
    sm[2 * q][i] = make_float2(v.x, v.y);
    sm[2 * q + 1][i] = make_float2(v.z, v.w);
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = (t >> 7) + 2 * h, i = t & 127;
    const long long cc = (long long)grp * 4 + c;
    if (p0 + i < npts && cc < nbatch) out[cc * npts + p0 + i] = sm[c][i];
  }
}

// Sum the partial tiles of one split tile in slot order, compensated, and
// write it out.
__global__ void __launch_bounds__(NTHR) adj_reduce_kernel(Geo g, const int4* __restrict__ split,
                                                          const float* __restrict__ partial,
                                                          float* __restrict__ gridv, int CG, int ncg) {
  const int4 sp = split[blockIdx.x];
  const int cg = blockIdx.y;
  const int c0 = cg * CG;
  const int es = g.cplx ? 2 : 1;
  const int ncoil = (int)min((long long)CG, g.nbatch - c0);
  int tc[3];
  {
    int t = sp.x;
    tc[2] = t % g.nt[2];
    t /= g.nt[2];
    tc[1] = t % g.nt[1];
    tc[0] = t / g.nt[1];
  }
  const int tvol = g.T[0] * g.T[1] * g.T[2];
  const int vstride = CG * es;
  const int tfl = (tvol * vstride + 3) & ~3;
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  for (int i = threadIdx.x; i < tvol * ncoil * es; i += NTHR) {
    const int f = i % es;
    int r = i / es;
    const int z = r % g.T[2];
    r /= g.T[2];
    const int y = r % g.T[1];
    r /= g.T[1];
    const int x = r % g.T[0];
    const int cc = r / g.T[0];
    const int gx = tc[0] * g.T[0] + x, gy = tc[1] * g.T[1] + y, gz = tc[2] * g.T[2] + z;
    if (gx >= g.N[0] || gy >= g.N[1] || gz >= g.N[2]) continue;
    const int li = ((x * g.T[1] + y) * g.T[2] + z) * vstride + cc * es + f;
    float s = partial[((long long)sp.y * ncg + cg) * tfl + li], c = 0.f;
    for (int k = 1; k < sp.z; ++k) comp_add(s, c, partial[((long long)(sp.y + k) * ncg + cg) * tfl + li]);
    gridv[((long long)(c0 + cc) * gvol + ((long long)gx * g.N[1] + gy) * g.N[2] + gz) * es + f] = s + c;
  }
}

// ------------------------------------------------------------ trajectory grad

template <typename V, int NORM>
__global__ void __launch_bounds__(NTHR) interp_grad_kernel(Geo g, const int4* __restrict__ items,
                                                              const int32_t* __restrict__ entries,
                                                              const float* __restrict__ locs,
                                                              const V* __restrict__ gridv, const V* __restrict__ a,
                                                              float* __restrict__ grad, int CG, int chunk,
                                                              float* __restrict__ partial) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int4 it = items[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tc[3];
  {
    int t = it.x;
    tc[2] = t % g.nt[2];
    t /= g.nt[2];
    tc[1] = t % g.nt[1];
    tc[0] = t / g.nt[1];
  }
  int o[3], S[3];
  for (int e = 0; e < 3; ++e) {
    o[e] = tc[e] * g.T[e];
    S[e] = g.T[e] + g.NT[e] - 1;
  }
  const int vol = S[0] * S[1] * S[2];
  V* reg = reinterpret_cast<V*>(smem);
  PTaps<true>* ptb = reinterpret_cast<PTaps<true>*>(smem + (size_t)vol * CG * sizeof(V));
  float* gacc = reinterpret_cast<float*>(ptb + NWARP);  // [chunk][3]
  PTaps<true>& pt = ptb[warp];
  const int npt = it.z - it.y;
  for (int i = threadIdx.x; i < npt * 3; i += NTHR) gacc[i] = 0.f;
  const long long gvol = (long long)g.N[0] * g.N[1] * g.N[2];
  const int CGP = CG <= 1 ? 1 : (CG <= 2 ? 2 : (CG <= 4 ? 4 : 8));
  const int lgc = lg2i(CGP);
  const int c = lane & (CGP - 1);
  const int q = lane >> lgc;
  const int QN = 32 >> lgc;
  const int ncg = (int)((g.nbatch + CG - 1) / CG);
  // blockIdx.y takes a contiguous share of the coil groups (all of them when
  // gridDim.y == 1); its sums go to its partial slot
  const int gps = (ncg + (int)gridDim.y - 1) / (int)gridDim.y;
  const int cg_end = min(ncg, ((int)blockIdx.y + 1) * gps);
  for (int cg = (int)blockIdx.y * gps; cg < cg_end; ++cg) {
    const int c0 = cg * CG;
    const int ncoil = (int)min((long long)CG, g.nbatch - c0);
    __syncthreads();
    for (int i = threadIdx.x; i < vol * ncoil; i += NTHR) {
      int z = i % S[2];
      int r = i / S[2];
      const int y = r % S[1];
      r /= S[1];
      const int x = r % S[0];
      const int cc = r / S[0];
      int gx = o[0] + x, gy = o[1] + y, gz = o[2] + z;
      V v = VT<V>::zero();
      bool in = true;
      if (g.pad == TLGB_PAD_CIRCULAR) {
        gx = wrapi(gx, g.N[0]);
        gy = wrapi(gy, g.N[1]);
        gz = wrapi(gz, g.N[2]);
      } else {
        in = gx < g.N[0] && gy < g.N[1] && gz < g.N[2];
      }
      if (in) v = __ldg(gridv + (long long)(c0 + cc) * gvol + ((long long)gx * g.N[1] + gy) * g.N[2] + gz);
      reg[((x * S[1] + y) * S[2] + z) * CG + cc] = v;
    }
    __syncthreads();
    for (int ei = it.y + warp; ei < it.z; ei += NWARP) {
      const long long p = entries[ei];
      if (!warp_point_taps<NORM, true>(g, locs, p, pt, lane)) continue;
      int l[3];
      for (int e = 0; e < 3; ++e) l[e] = pt.start[e] - o[e];
      V d0 = VT<V>::zero(), d1 = VT<V>::zero(), d2 = VT<V>::zero();
      for (int ka = 0; ka < pt.n[0]; ++ka) {
        for (int kb = 0; kb < pt.n[1]; ++kb) {
          const V* row = reg + (((l[0] + ka) * S[1] + (l[1] + kb)) * S[2] + l[2]) * CG + c;
          for (int kc = q; kc < pt.n[2]; kc += QN) {
            if (c >= ncoil) continue;
            const V gv = row[kc * CG];
            float w0, w1, w2;
            if (NORM == 1) {
              const float wa = pt.w[0][ka], wb = pt.w[1][kb], wc = pt.w[2][kc];
              w0 = pt.dw[0][ka] * wb * wc;
              w1 = wa * pt.dw[1][kb] * wc;
              w2 = wa * wb * pt.dw[2][kc];
            } else {
              const float a0 = pt.w[0][ka], a1 = pt.w[1][kb], a2 = pt.w[2][kc];
              const float rho = sqrtf(a0 * a0 + a1 * a1 + a2 * a2);
              float kd = 0.f;
              if (rho <= 1.0f && rho > 0.f) kd = kern_deriv(g.kernel, rho, g.beta) / rho;
              w0 = g.act[0] ? kd * pt.dw[0][ka] / g.r[0] : 0.f;
              w1 = g.act[1] ? kd * pt.dw[1][kb] / g.r[1] : 0.f;
              w2 = g.act[2] ? kd * pt.dw[2][kc] / g.r[2] : 0.f;
            }
            VT<V>::fma(d0, w0, gv);
            VT<V>::fma(d1, w1, gv);
            VT<V>::fma(d2, w2, gv);
          }
        }
      }
      float r0 = 0.f, r1 = 0.f, r2 = 0.f;
      if (c < ncoil) {
        const V av = __ldg(a + (long long)(c0 + c) * g.npts + p);
        r0 = VT<V>::re_dot(av, d0);
        r1 = VT<V>::re_dot(av, d1);
        r2 = VT<V>::re_dot(av, d2);
      }
      for (int m = 1; m < 32; m <<= 1) {
        r0 += __shfl_xor_sync(0xffffffffu, r0, m);
        r1 += __shfl_xor_sync(0xffffffffu, r1, m);
        r2 += __shfl_xor_sync(0xffffffffu, r2, m);
      }
      if (lane == 0) {
        float* ga = gacc + (ei - it.y) * 3;
        ga[0] += r0;
        ga[1] += r1;
        ga[2] += r2;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  float* dst = gridDim.y == 1 ? grad : partial + (long long)blockIdx.y * g.npts * g.ndim;
  for (int i = threadIdx.x; i < npt; i += NTHR) {
    const long long p = entries[it.y + i];
    for (int e = 3 - g.ndim; e < 3; ++e) dst[p * g.ndim + (e - (3 - g.ndim))] = gacc[i * 3 + e];
  }
}

// grad[i] = sum over slots s of partial[s][i], in slot order
__global__ void __launch_bounds__(256) grad_reduce_kernel(const float* __restrict__ partial, int nsplit, long long n,
                                                          float* __restrict__ grad) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = partial[i];
  for (int k = 1; k < nsplit; ++k) s += partial[(long long)k * n + i];
  grad[i] = s;
}

// ------------------------------------------------ 2D trajectory gradient
//
// d/d(y, z) of sum_b Re(conj(a[b, p]) ungrid(grid)[b, p]) for 2D geometries of at
// most 5 taps per dim, on the gather's ring (gather_kernel): a stage is the
// region of a group of 8 entries and the item's 8 x 256 values of a, gathered by
// the producers in the records' order, so runs of points are read in whole
// lines. The sum over the entries comes first: a tap's weight and derivative are
// the same for every entry, so a lane adds Re(conj(a) v) per tap over all groups
// of the unit in registers (4 y taps x 8 steps of 2 points) and the weights are
// applied once per point at the end, the derivatives evaluated there by 16
// lanes. (Weighting every product, adding the 32 lanes up for each group and the
// groups' partial results in a further pass took 1243 us for 205,824 points x
// 256 entries on 320^2; this takes 607 us.)
constexpr int kGradWarps = 16;
constexpr int kGradStages = 4;
constexpr int kGradSteps = kGatherPts / (2 * kGradWarps);
constexpr uint32_t kGradRegion = 20 * 20 * 8 * 8;
constexpr uint32_t kGradStage = kGradRegion + 8 * kGatherPts * 8;

struct GradTaps {  // a window of 5 taps, one per consumer warp
  float w[2][5], dw[2][5];
  int n[2], f[2];
};

constexpr size_t grad2_smem() {
  return (size_t)kGradStages * kGradStage + 2 * kGatherPts * sizeof(GatherRec<2, 4>) + kGatherPts * sizeof(float2) +
         kGradWarps * (sizeof(GradTaps) + 16 * sizeof(float)) + 8 * (2 * kGradStages + 4) + 16;
}

// AT: a is point-major ([group][point][8], transpose_vals_kernel's layout), for
// points in random order: gathered entry by entry there, every 8-byte value is a
// sector of its own (205,824 random points x 256 entries on 320^2: 1952 us, 765
// with the transposition; 8 entries 287 and 265 at 524,288 points on 512^2).
template <bool AT>
__global__ void __launch_bounds__(kGradWarps * 32 + kGatherProd, 1)
    grad2_kernel(const __grid_constant__ CUtensorMap tmap, int use_tma, Geo g, const int4* __restrict__ items, int nruns,
                 int run, int nunits, const GatherRec<2, 4>* __restrict__ recs, const float* __restrict__ locs,
                 const float* __restrict__ gridv, const float2* __restrict__ a, float* __restrict__ grad,
                 float* __restrict__ partial) {
  constexpr int S = 20, VOL = S * S, NW = kGradWarps, NST = kGradStages;
  using Rec = GatherRec<2, 4>;
  extern __shared__ __align__(128) unsigned char smem[];
  Rec* recbuf = reinterpret_cast<Rec*>(smem + NST * kGradStage);
  float2* far = reinterpret_cast<float2*>(recbuf + 2 * kGatherPts);  // sums of the unit's 5-tap windows
  GradTaps* slow = reinterpret_cast<GradTaps*>(far + kGatherPts);
  float* dwb = reinterpret_cast<float*>(slow + NW);                  // [warp][point][dim][4]
  uint64_t* full = reinterpret_cast<uint64_t*>((reinterpret_cast<uintptr_t>(dwb + NW * 16) + 7) & ~(uintptr_t)7);
  uint64_t* empty = full + NST;
  uint64_t* rfull = empty + NST;
  uint64_t* rempty = rfull + 2;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(&full[i], kGatherProd);
      mbar_init(&empty[i], NW);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&rfull[i], 1);
      mbar_init(&rempty[i], NW);
    }
    fence_mbar_init();
    failed = 0;
  }
  __syncthreads();
  const uint32_t limit = g.wait;
  const int ncg = (int)((g.nbatch + 7) / 8);
  volatile int* vfailed = &failed;
  if (warp >= NW) {
    // ---- producers
    if (g.skip_copy == 1) return;
    const int pt = tid - NW * 32;
    uint32_t k = 0, ui = 0, recs_sent = 0;  // stages, units, record copies begun (thread 0)
    bool ok = true;
    int4 next = items[blockIdx.x / nruns];
    for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x, ++ui) {
      const int4 it = next;
      if (u + (int)gridDim.x < nunits) next = items[(u + gridDim.x) / nruns];
      const int g0 = (u % nruns) * run, g1 = min(ncg, g0 + run), npt = it.z - it.y;
      int o[3];
      item_origin(g, it.x, o);
      const bool wraps = g.pad == TLGB_PAD_CIRCULAR && (o[1] + S > g.N[1] || o[2] + S > g.N[2]);
      const bool tma = use_tma && !wraps;
      const Rec* rec = recbuf + (ui & 1) * kGatherPts;
      if (pt == 0) {
        ok = mbar_wait_bounded(&rempty[ui & 1], ((ui >> 1) & 1) ^ 1, kWaitLimit);
        if (ok) {
          const uint32_t bytes = (uint32_t)npt * (uint32_t)sizeof(Rec);
          mbar_arrive_expect_tx(&rfull[ui & 1], bytes);
          sm100::bulk_load(recbuf + (ui & 1) * kGatherPts, recs + it.w, bytes, &rfull[ui & 1]);
          ++recs_sent;
        }
      }
      ok = ok && mbar_wait_bounded(&rfull[ui & 1], (ui >> 1) & 1, kWaitLimit);
      for (int cg = g0; cg < g1 && ok; ++cg, ++k) {
        const uint32_t s = k % NST;
        ok = mbar_wait_bounded(&empty[s], ((k / NST) & 1) ^ 1, kWaitLimit) && !*vfailed;
        if (!ok) break;
        float2* reg = reinterpret_cast<float2*>(smem + s * kGradStage);
        float2* av = reinterpret_cast<float2*>(smem + s * kGradStage + kGradRegion);
        if (tma) {
          if (pt == 0) {
            sm100::fence_proxy_async_smem();  // the buffer may last have been filled by plain copies
            sm100::mbar_expect_tx(&full[s], kGradRegion);
            tma_load_4d(reg, &tmap, &full[s], o[2], o[1], 0, cg * 8);
          }
        } else {
          copy_region<2, 4, 8>(g, gridv, reg, o, cg, pt);
        }
        if constexpr (AT) {  // 4 threads a point; the values of missing entries are zeros already
          for (int i = pt; i < npt * 4; i += kGatherProd) {
            const int p = rec[i >> 2].p;
            if (TLGB_IN_RANGE(p, g.npts)) cp_async16(av + 2 * i, a + ((long long)cg * g.npts + p) * 8 + 2 * (i & 3));
          }
        } else {
          for (int i = pt; i < npt; i += kGatherProd) {
            const int p = rec[i].p;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const bool in = cg * 8 + c < g.nbatch && TLGB_IN_RANGE(p, g.npts);
              sm100::cp_async8_zfill(av + c * kGatherPts + i, in ? a + (long long)(cg * 8 + c) * g.npts + p : a, in);
            }
          }
        }
        sm100::cp_async_mbar_arrive(&full[s]);
      }
      ok = ok && !*vfailed;
    }
    if (!ok && pt == 0) {
      *vfailed = 1;
      atomicExch(&g_tlgb_status, 1);
    }
    producer_drain(full, k, NST, rfull, recs_sent, pt);
    return;
  }
  // ---- consumers: lane = (point h of a step, entry c and c + 4, z tap kz)
  const int kz = lane & 3, c = (lane >> 2) & 3, h = lane >> 4;
  int kyo[4], rowoff[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    kyo[t] = (t + c) & 3;
    rowoff[t] = kyo[t] * S;
  }
  auto give_up = [&]() {
    if (lane == 0) {
      *vfailed = 1;
      atomicExch(&g_tlgb_status, 1);
    }
  };
  uint32_t k = 0, ui = 0;
  int4 next = items[blockIdx.x / nruns];
  for (int u = blockIdx.x; u < nunits; u += gridDim.x, ++ui) {
    const int4 it = next;
    if (u + (int)gridDim.x < nunits) next = items[(u + gridDim.x) / nruns];
    const int g0 = (u % nruns) * run, g1 = min(ncg, g0 + run), npt = it.z - it.y;
    const Rec* rec = recbuf + (ui & 1) * kGatherPts;
    if (!mbar_wait_bounded(&rfull[ui & 1], (ui >> 1) & 1, limit)) return give_up();
    float sum[kGradSteps][4];
#pragma unroll
    for (int st = 0; st < kGradSteps; ++st) {
#pragma unroll
      for (int t = 0; t < 4; ++t) sum[st][t] = 0.f;
      const int i = (st * NW + warp) * 2 + h;
      if ((lane & 15) == 0 && i < npt) far[i] = make_float2(0.f, 0.f);
    }
    __syncwarp();
    for (int cg = g0; cg < g1; ++cg, ++k) {
      const uint32_t s = k % NST;
      if (!mbar_wait_bounded(&full[s], (k / NST) & 1, limit)) return give_up();
      const float2* reg = reinterpret_cast<const float2*>(smem + s * kGradStage);
      const float2* av = reinterpret_cast<const float2*>(smem + s * kGradStage + kGradRegion);
#pragma unroll
      for (int st = 0; st < kGradSteps; ++st) {
        const int base = (st * NW + warp) * 2;
        if (base >= npt) break;
        const bool on = base + h < npt;
        const int i = on ? base + h : base;
        const unsigned view = rec[i].view;
        const float2* v = reg + c * VOL + (view & 0xfffff) + kz;
        const float2 a0 = av[AT ? i * 8 + c : c * kGatherPts + i], a1 = av[AT ? i * 8 + c + 4 : (c + 4) * kGatherPts + i];
        if (TLGB_IN_RANGE((view & 0xfffff) + 3 * S + 3, VOL)) {
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 v0 = v[rowoff[t]], v1 = v[4 * VOL + rowoff[t]];
            sum[st][t] = fmaf(a0.x, v0.x, sum[st][t]);
            sum[st][t] = fmaf(a0.y, v0.y, sum[st][t]);
            sum[st][t] = fmaf(a1.x, v1.x, sum[st][t]);
            sum[st][t] = fmaf(a1.y, v1.y, sum[st][t]);
          }
        }
        // windows of 5 taps, one at a time by the whole warp
        unsigned rest = __ballot_sync(0xffffffffu, on && !((view >> 20) & 1));
        while (rest) {
          const int hh = (__ffs(rest) - 1) >> 4;
          rest &= ~(0xffffu << (16 * hh));
          const int p = rec[base + hh].p;
          GradTaps& T = slow[warp];
          {
            const int d = lane / 5, kk = lane % 5, e = 1 + d;
            Tap t;
            t.valid = false;
            t.d = 0.f;
            float x = 0.f;
            int lower = 0;
            if (d < 2) {
              x = load_coord(g, locs, p, e);
              lower = lower_of(g, e, x);
              if (kk < g.NT[e]) t = tap_eval(g, e, x, lower, kk);
            }
            const unsigned m = (__ballot_sync(0xffffffffu, t.valid) >> (d < 2 ? 5 * d : 0)) & 31u;
            if (t.valid) {
              const int q = kk - (__ffs(m) - 1);
              T.w[d][q] = kern_value(g.kernel, fabsf(t.d), g.beta);
              T.dw[d][q] = kern_deriv(g.kernel, t.d, g.beta) / g.r[e];
            }
            if (d < 2 && kk == 0) {
              int stt = lower + __ffs(m) - 1, o[3];
              if (g.pad == TLGB_PAD_CIRCULAR) stt = wrapi(stt, g.N[e]);
              item_origin(g, it.x, o);
              T.n[d] = __popc(m);
              T.f[d] = stt - (e == 1 ? o[1] : o[2]);
            }
          }
          __syncwarp();
          const int c8 = lane & 7, n2 = T.n[1], tot = T.n[0] * n2;
          const float2 ac = av[AT ? (base + hh) * 8 + c8 : c8 * kGatherPts + base + hh];
          float ry = 0.f, rz = 0.f;
          auto tap = [&](int y, int z) {
            const int cell = (T.f[0] + y) * S + T.f[1] + z;
            if (!TLGB_IN_RANGE(cell, VOL)) return;
            const float2 vv = reg[c8 * VOL + cell];
            const float dot = fmaf(ac.x, vv.x, ac.y * vv.y);
            ry = fmaf(T.dw[0][y] * T.w[1][z], dot, ry);
            rz = fmaf(T.w[0][y] * T.dw[1][z], dot, rz);
          };
          // the loop that lets ptxas keep more of `sum` in registers, by variant: 810 against 860 us on radial
          // points, 755 against 850 on random ones (256 entries of 320^2)
          if constexpr (AT)
            for (int y = 0; y < T.n[0]; ++y)
              for (int z = lane >> 3; z < n2; z += 4) tap(y, z);
          else
            for (int t = lane >> 3; t < tot; t += 4) tap(t / n2, t % n2);
#pragma unroll
          for (int m = 1; m < 32; m <<= 1) {
            ry += __shfl_xor_sync(0xffffffffu, ry, m);
            rz += __shfl_xor_sync(0xffffffffu, rz, m);
          }
          if (lane == 0) {
            far[base + hh].x += ry;
            far[base + hh].y += rz;
          }
          __syncwarp();
        }
      }
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&empty[s]);
    }
    // the weights, once per point
    float* dst = nruns == 1 ? grad : partial + (long long)(u % nruns) * g.npts * 2;
    float* dw = dwb + warp * 16 + h * 8;
#pragma unroll
    for (int st = 0; st < kGradSteps; ++st) {
      const int base = (st * NW + warp) * 2;
      if (base >= npt) break;
      const bool on = base + h < npt;
      const int i = on ? base + h : base;
      const Rec& R = rec[i];
      const int d = (lane >> 3) & 1, kk = lane & 7, e = 1 + d;
      if (kk < 4) dw[4 * d + kk] = 0.f;
      __syncwarp();
      int ny, nz;  // the window's taps per dim: sums of cells past it may be NaN or Inf and are left out
      {
        Tap t;
        t.valid = false;
        t.d = 0.f;
        const float x = load_coord(g, locs, R.p, e);
        const int lower = lower_of(g, e, x);
        if (kk < 5 && kk < g.NT[e]) t = tap_eval(g, e, x, lower, kk);
        const unsigned m = (__ballot_sync(0xffffffffu, t.valid) >> (lane & 24)) & 255u;
        const int q = kk - (__ffs(m) - 1);
        if (t.valid && q < 4) dw[4 * d + q] = kern_deriv(g.kernel, t.d, g.beta) / g.r[e];
        ny = __shfl_sync(0xffffffffu, __popc(m), lane & 16), nz = __shfl_sync(0xffffffffu, __popc(m), (lane & 16) | 8);
      }
      __syncwarp();
      float ry = 0.f, rz = 0.f;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float v = kyo[t] < ny && kz < nz ? sum[st][t] : 0.f;
        ry = fmaf(dw[kyo[t]], v, ry);
        rz = fmaf(R.w[0][kyo[t]], v, rz);
      }
      ry *= R.w[1][kz];
      rz *= dw[4 + kz];
#pragma unroll
      for (int m = 1; m < 16; m <<= 1) {
        ry += __shfl_xor_sync(0xffffffffu, ry, m);
        rz += __shfl_xor_sync(0xffffffffu, rz, m);
      }
      if (on && (lane & 15) == 0 && TLGB_IN_RANGE(R.p, g.npts))
        *reinterpret_cast<float2*>(dst + (long long)R.p * 2) = (R.view >> 20) & 1 ? make_float2(ry, rz) : far[i];
      __syncwarp();
    }
    if (lane == 0) sm100::mbar_arrive(&rempty[ui & 1]);
  }
}

// ------------------------------------------------------------- host helpers

struct PlanLayout {
  int64_t e_max, max_fwd, max_adj, ntiles;
  int64_t off_entries, off_fwd, off_adj, off_split, off_recs, bytes;
  // block lists of the gridding of complex values (off_blk_entries == 0: none)
  int64_t nblocks, eb_max, max_blk_items, max_blk_split, off_blk_entries, off_blk_items, off_blk_split, off_blk_rows;
  // tmp: windows, CTA sums, counters, key starts; per list the sort's two key
  // buffers, second value buffer and counts, and the unordered items, splits
  // and their order
  int64_t t_win, t_sums, t_homes, t_cnt, t_tstart, t_bstart;
  int64_t t_keys[2][2], t_vals[2], t_counts[2], t_items[2], t_order[2];
  int64_t t_bytes;
};

constexpr int64_t kFwdChunk = 512;
constexpr int64_t kAdjChunk = 1024;

std::atomic<int> g_test_skip_copy{0};  // tlgb_test_skip_region_copy

// Taps per dim of the gather records, 0 for geometries without them: 3D grids
// of at least 8 cells per dim with at most 5 taps per dim (4 in a record; the
// fifth only at exact-integer coordinates), 2D grids of at least 16 with at
// most 9 (4 or 8 in a record), separable weights.
int rec_taps(const Geo& g) {
  if (g.norm != 1) return 0;
  const int nt = std::max(g.NT[0], std::max(g.NT[1], g.NT[2]));
  if (g.ndim == 3) return g.T[0] == 8 && g.T[1] == 8 && g.T[2] == 8 && nt <= 5 ? 4 : 0;
  return g.ndim == 2 && g.T[1] == 16 && g.T[2] == 16 && nt <= 9 ? (nt <= 5 ? 4 : 8) : 0;
}
bool records_ok(const Geo& g) { return rec_taps(g) > 0; }
size_t rec_bytes(const Geo& g) { return g.ndim == 3 ? 64 : (rec_taps(g) == 4 ? 48 : 80); }
// 3D plans: the points' places among the records follow the records
size_t rank_offset(const Geo& g, size_t off_records) { return align_up(off_records + (size_t)g.npts * rec_bytes(g), 256); }
// points of a gather item: what the record buffers of gather_kernel hold
int fwd_chunk(const Geo& g) { return records_ok(g) ? kGatherPts : (int)kFwdChunk; }

// The most blocks a window of NT cells meets along a dim (4 = too many for
// the block lists): the windows inside the grid at every offset in a block,
// and in circular mode those that cross the upper edge.
int max_blocks_per_dim(const Geo& g, int e) {
  if (!g.act[e]) return 1;
  const int edge = block_edge(g.ndim, e), N = g.N[e], NT = g.NT[e];
  int most = 1;
  for (int st = 0; st < N; st = (st >= edge && st < N - NT - edge) ? N - NT - edge : st + 1) {
    int n = 0, prev = -1;
    for (int k = 0; k < NT; ++k) {
      int v = st + k;
      if (v >= N) {
        if (g.pad != TLGB_PAD_CIRCULAR) break;
        v -= N;  // at most once: N >= NT there
      }
      const int b = edge == 4 ? v >> 2 : v >> 3;
      if (b != prev) ++n, prev = b;
    }
    most = std::max(most, n);
  }
  return std::min(most, 4);
}

// Rows of tap weights per dim in the block lists (the most blocks a window
// meets along a dim, 2 or 3), 0 for geometries without block lists. They
// need 2D or 3D, separable weights, at most 9 taps per dim (width up to 8)
// meeting at most 3 blocks, a grid on which a wrapped window meets no block
// twice, and counts that fit the entries' bits. The block lists beat tiles
// wherever both run: gridding 20 complex images of 320^2 from 131,072 points,
// width 6, zero padding, takes 125 us (855 us on interp_adj_kernel's one-warp
// tiles); 12 of 125 x 150 x 135 from 400,000 points, width 4, circular, 320 us
// (520 us on 8^3-cell register tiles, which the block lists replaced).
int block_rows(const Geo& g) {
  if (g.ndim < 2 || g.norm != 1) return 0;
  int rows = 2;
  for (int e = 3 - g.ndim; e < 3; ++e) {
    if (g.NT[e] > 9) return 0;
    if (g.pad == TLGB_PAD_CIRCULAR && g.N[e] < g.NT[e] + block_edge(g.ndim, e) - 1) return 0;
    const int m = max_blocks_per_dim(g, e);
    if (m > 3) return 0;
    rows = std::max(rows, m);
  }
  const int64_t nb = (int64_t)blocks_along(g, 0) * blocks_along(g, 1) * blocks_along(g, 2);
  if (nb >= (1ll << 31) || g.npts >= (1ll << sel_shift(rows))) return 0;
  return rows;
}

int make_geo(const tlgb_interp_desc* d, Geo& g) {
  if (!d) TLGB_FAIL(TLGB_ERR_INVALID, "null interp descriptor");
  if (d->ndim < 1 || d->ndim > 3) TLGB_FAIL(TLGB_ERR_INVALID, "ndim must be 1, 2 or 3");
  if (d->kernel != TLGB_KERNEL_KAISER_BESSEL && d->kernel != TLGB_KERNEL_SPLINE)
    TLGB_FAIL(TLGB_ERR_INVALID, "unknown kernel");
  if (d->norm != 1 && d->norm != 2) TLGB_FAIL(TLGB_ERR_INVALID, "norm must be 1 or 2");
  if (d->pad_mode != TLGB_PAD_CIRCULAR && d->pad_mode != TLGB_PAD_ZERO) TLGB_FAIL(TLGB_ERR_INVALID, "unknown pad mode");
  if (d->npts < 0 || d->nbatch < 0) TLGB_FAIL(TLGB_ERR_INVALID, "negative size");
  // the value transpose and the sums of parts launch one grid row per 8 batch entries (at most 65535)
  if (d->nbatch > TLGB_INTERP_MAX_BATCH)
    TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "batch above 524280 entries in one call: split the batch");
  memset(&g, 0, sizeof(g));
  g.skip_copy = g_test_skip_copy.load();
  g.wait = g.skip_copy ? 2u - g.skip_copy : kWaitLimit;
  g.ndim = d->ndim;
  const int off = 3 - d->ndim;
  int maxnt = 1;
  for (int e = 0; e < 3; ++e) {
    if (e < off) {
      g.N[e] = 1;
      g.NT[e] = 1;
      g.r[e] = 1.f;
      g.act[e] = 0;
      continue;
    }
    const int64_t n = d->grid_size[e - off];
    const float w = d->width[e - off];
    if (n < 1 || n > (1 << 24)) TLGB_FAIL(TLGB_ERR_INVALID, "grid size must be in [1, 2^24]");
    if (!(w > 0.f)) TLGB_FAIL(TLGB_ERR_INVALID, "kernel width must be positive");
    // len(torch.arange(w + 1)) taps, as the reference's diff grid
    const int nt = (int)ceil((double)w + 1.0);
    if (nt > NTMAX) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "kernel width must be below 15 grid units");
    g.N[e] = (int)n;
    g.NT[e] = nt;
    g.r[e] = w / 2.0f;
    {
      int ex = 0;
      const float mant = frexpf(g.r[e], &ex);
      g.rpow2[e] = (mant == 0.5f) ? 1 : 0;
      g.rinv[e] = 1.0f / g.r[e];
    }
    g.act[e] = 1;
    maxnt = std::max(maxnt, nt);
  }
  if (d->ndim == 3 && maxnt > 9) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "3D kernel width must be below 8 grid units");
  const int T3[3] = {8, 8, 8}, T2[3] = {1, 16, 16}, T1[3] = {1, 1, 512};
  const int* T = d->ndim == 3 ? T3 : (d->ndim == 2 ? T2 : T1);
  g.wrap_safe = 1;
  g.tv_off = -1;
  for (int e = 0; e < 3; ++e) {
    g.T[e] = std::min(T[e], g.N[e]);
    g.lgT[e] = -1;
    for (int k = 0; k < 10; ++k)
      if (g.T[e] == 1 << k) g.lgT[e] = k;
    g.nt[e] = (int)cdiv(g.N[e], g.T[e]);
    if (g.act[e] && g.N[e] < g.NT[e]) g.wrap_safe = 0;
  }
  g.kernel = d->kernel;
  g.norm = d->norm;
  g.pad = d->pad_mode;
  g.cplx = d->is_complex ? 1 : 0;
  g.beta = d->beta;
  // a remainder of beta is at most half an ulp: anything else in the
  // reserved field is no remainder
  memcpy(&g.beta_lo, &d->reserved, sizeof(float));
  if (!(std::fabs(g.beta_lo) <= std::fabs(g.beta) * 6e-8f)) g.beta_lo = 0.f;
  g.npts = d->npts;
  g.nbatch = d->nbatch;
  if ((int64_t)g.nt[0] * g.nt[1] * g.nt[2] >= (1ll << 30)) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "too many tiles");
  g.nrow = block_rows(g);
  return TLGB_OK;
}

// Tiles one point can touch along a dim: 2 for T >= taps - 1, 3 where a
// circular window can cross both a ragged last tile and the wrap.
int64_t max_tiles_per_dim(const Geo& g, int e) {
  if (g.nt[e] == 1) return 1;
  const int m = g.N[e] % g.T[e];
  if (g.pad == TLGB_PAD_CIRCULAR && m != 0 && m < g.NT[e] - 1) return std::min(3, g.nt[e]);
  return 2;
}

// in kernel_key: most points' outputs lie in another sector than the point's before
constexpr int64_t kScattered = (int64_t)1 << 52;
// in kernel_key: some window has fewer taps in a dim than its gather record holds
constexpr int64_t kPartial = (int64_t)1 << 53;

// The kernel, norm and beta a plan's records hold weights for
int64_t kernel_key(const Geo& g) {
  uint32_t bits;
  memcpy(&bits, &g.beta, 4);
  return (int64_t)bits | ((int64_t)g.kernel << 32) | ((int64_t)g.norm << 40) | ((int64_t)1 << 48);
}

PlanUnits plan_units(const Geo& g, int64_t ntiles, bool blocks) {
  PlanUnits U;
  U.ntiles = ntiles;
  U.nbx = blocks_along(g, 0), U.nby = blocks_along(g, 1), U.nbz = blocks_along(g, 2);
  const int cx = g.ndim == 3 ? kCube : 1;
  U.ncy = blocks_along(U.nby, kCube), U.ncz = blocks_along(U.nbz, kCube);
  U.per = cx * kCube;
  U.nrows = blocks ? (long long)blocks_along(U.nbx, cx) * U.ncy * U.ncz * U.per : 0;
  U.ntx = g.nt[0], U.nty = g.nt[1], U.ntz = g.nt[2];
  const int tx = g.nt[0] == 1 ? 1 : kTileCube;
  U.ntu = (long long)blocks_along(g.nt[0], tx) * blocks_along(g.nt[1], kTileCube) * blocks_along(g.nt[2], kTileCube) * tx *
          kTileCube * kTileCube;
  U.tile_ctas = (int)cdiv(U.ntu, kPlanPts);
  return U;
}

// `pairs`: the (point, block) pairs of the plan's points, -1 = not counted (room
// for as many as points can have). Without block lists when there are too many.
PlanLayout layout(const Geo& g, int64_t pairs) {
  PlanLayout L;
  L.e_max = g.npts * max_tiles_per_dim(g, 0) * max_tiles_per_dim(g, 1) * max_tiles_per_dim(g, 2);
  L.ntiles = (int64_t)g.nt[0] * g.nt[1] * g.nt[2];
  L.max_fwd = L.ntiles + cdiv(g.npts, fwd_chunk(g)) + 1;
  L.max_adj = L.ntiles + cdiv(L.e_max, kAdjChunk) + 1;
  size_t o = 0;
  L.off_entries = o;
  o = align_up(o + (size_t)std::max<int64_t>(L.e_max, 1) * 4, 256);
  L.off_fwd = o;
  o = align_up(o + (size_t)L.max_fwd * 16, 256);
  L.off_adj = o;
  o = align_up(o + (size_t)L.max_adj * 16, 256);
  L.off_split = o;
  o = align_up(o + (size_t)(L.ntiles + 1) * 16, 256);
  L.off_recs = 0;
  if (records_ok(g) && g.npts > 0) {
    L.off_recs = o;
    o = rank_offset(g, o);
    if (g.ndim == 3) o = align_up(o + (size_t)g.npts * 4, 256);
  }
  L.nblocks = L.eb_max = L.max_blk_items = L.max_blk_split = 0;
  L.off_blk_entries = L.off_blk_items = L.off_blk_split = L.off_blk_rows = 0;
  const int64_t most = g.npts * max_blocks_per_dim(g, 0) * max_blocks_per_dim(g, 1) * max_blocks_per_dim(g, 2);
  if (g.nrow && g.npts > 0 && (pairs >= 0 ? pairs : most) < (1ll << 31)) {
    L.nblocks = (int64_t)blocks_along(g, 0) * blocks_along(g, 1) * blocks_along(g, 2);
    L.eb_max = std::max<int64_t>(pairs >= 0 ? std::min(pairs, most) : most, 1);
    L.max_blk_items = L.nblocks + cdiv(L.eb_max, kBlkPart) + 1;
    L.max_blk_split = std::min(L.nblocks, L.eb_max / (kBlkPart + 1)) + 1;
    L.off_blk_entries = o;
    o = align_up(o + (size_t)L.eb_max * 4, 256);
    L.off_blk_items = o;
    o = align_up(o + (size_t)L.max_blk_items * 16, 256);
    L.off_blk_split = o;
    o = align_up(o + (size_t)L.max_blk_split * 16, 256);
    L.off_blk_rows = o;
    o = align_up(o + (size_t)g.npts * row_floats(g.ndim, g.nrow) * 4, 256);
  }
  L.bytes = o;
  size_t t = 0;
  auto tmp = [&](int64_t bytes) {
    const int64_t at = (int64_t)t;
    t = align_up(t + (size_t)std::max<int64_t>(bytes, 16), 256);
    return at;
  };
  const PlanUnits U = plan_units(g, L.ntiles, L.nblocks > 0);
  L.t_win = tmp(g.npts * 16);
  L.t_sums = tmp(std::max(cdiv(g.npts, kPlanPts), (int64_t)U.tile_ctas + cdiv(U.nrows, kPlanPts)) * 16);
  L.t_homes = tmp((int64_t)U.tile_ctas * 16);
  L.t_cnt = tmp(16 * 4);
  L.t_tstart = tmp((2 * L.ntiles + 1) * 4);
  L.t_bstart = tmp((L.nblocks + 1) * 4);
  for (int i = 0; i < 2; ++i) {  // the tile list and its gridding items; the block list and its splits
    const int64_t pairs = i ? L.eb_max : L.e_max, items = i ? L.max_blk_split : L.max_adj;
    if (i && !L.nblocks) break;
    const int64_t n = std::max<int64_t>(std::max(pairs, items), 1);
    L.t_keys[i][0] = tmp(n * 4);
    L.t_keys[i][1] = tmp(n * 4);
    L.t_vals[i] = tmp(n * 4);
    L.t_counts[i] = tmp(radix_counts_len(n) * 4);
    L.t_items[i] = tmp(items * 16);
    L.t_order[i] = tmp(items * 4);
  }
  L.t_bytes = (int64_t)t;
  return L;
}

int value_size(const Geo& g) { return g.cplx ? 8 : 4; }

constexpr int NWF = 16;  // warps of a forward CTA (one CTA per SM shares one staged region)

// taps stored per dim by the kernels: 5 covers widths < 4 (the NUFFT default)
int ntb_for(const Geo& g) {
  const int m = std::max(g.NT[0], std::max(g.NT[1], g.NT[2]));
  if (m <= 5) return 5;
  return g.ndim == 3 ? 9 : 16;
}
size_t pt_bytes(int ntb) {
  return ntb == 5 ? sizeof(Rec<5>) : (ntb == 9 ? sizeof(Rec<9>) : sizeof(Rec<16>));
}

int64_t region_vol(const Geo& g) {
  return (int64_t)(g.T[0] + g.NT[0] - 1) * (g.T[1] + g.NT[1] - 1) * (g.T[2] + g.NT[2] - 1);
}

// batch entries staged per forward CTA
int fwd_cg(const Geo& g) {
  int cg = (int)std::min<long long>(std::max<long long>(g.nbatch, 1), CGMAX);
  const int64_t cap = 220 * 1024 - NWF * 32 * (int64_t)pt_bytes(ntb_for(g));
  while (cg > 1 && region_vol(g) * cg * value_size(g) > cap) --cg;
  return cg;
}

size_t fwd_smem(const Geo& g, int cg, int warps) {
  return align_up((size_t)region_vol(g) * cg * value_size(g), 16) + warps * 32 * pt_bytes(ntb_for(g));
}

int adj_cg(const Geo& g) { return (int)std::min<long long>(std::max<long long>(g.nbatch, 1), CGMAX); }

// Gridding of complex values on the plan's block lists (adj_b3_kernel,
// adj_bn_kernel); the other calls (real values, the radial norm, 1D, widths
// above 8, grids too small for a window to meet a block once) run on
// interp_adj_kernel.
bool on_blocks(const Geo& g, const tlgb_interp_plan_info* info) {
  return g.cplx && g.nrow > 0 && info->n_blk_items > 0;
}

int64_t tile_floats(const Geo& g, int cg) {
  return ((int64_t)g.T[0] * g.T[1] * g.T[2] * cg * (g.cplx ? 2 : 1) + 3) & ~3ll;
}

size_t adj_smem(const Geo& g, int cg) {
  return (size_t)tile_floats(g, cg) * 4 + 32 * pt_bytes(ntb_for(g)) + 32 * (size_t)cg * (g.cplx ? 2 : 1) * 4;
}

// the grad kernel keeps the warp-cooperative tap buffers
int grad_cg(const Geo& g, size_t taps_bytes) {
  int cg = (int)std::min<long long>(std::max<long long>(g.nbatch, 1), CGMAX);
  const int64_t cap = 112 * 1024 - NWARP * (int64_t)taps_bytes - 1024;
  while (cg > 1 && region_vol(g) * cg * value_size(g) > cap) --cg;
  return cg;
}

size_t grad_smem(const Geo& g, int cg, size_t taps_bytes) {
  return (size_t)region_vol(g) * cg * value_size(g) + NWARP * taps_bytes;
}

// Parts the coil groups of the trajectory gradient are split into: enough
// CTAs to fill the device when a plan has few tiles and the batch many
// groups (each part restages the region and re-evaluates the taps).
int grad_splits(const Geo& g, const tlgb_interp_plan_info* info) {
  const int cg = grad_cg(g, sizeof(PTaps<true>));
  const long long ncg = cdiv(std::max<long long>(g.nbatch, 1), cg);
  const long long items = std::max<long long>(info->n_fwd_items, 1);
  const long long want = cdiv(8ll * sm_count(), items);  // ~8 CTAs per SM
  return (int)std::max(1ll, std::min(ncg, want));
}

size_t grad_scratch_bytes(const Geo& g, int nsplit) {
  return nsplit > 1 ? (size_t)nsplit * g.npts * g.ndim * sizeof(float) : 0;
}

// The 2D gradient on the gather's ring (grad2_kernel). A unit is an item and a
// run of groups of 8 entries; with several runs each adds its own partial slot.
// One run (no partial results) unless that leaves fewer units than SMs: each
// unit ends with some microseconds for its points' weights, so more are slower
// (20 entries of 256 x 240 at 65,536 points: 109 us with 4 units per SM, 77 so).
// Windows of the spline with width 4 always have 5 taps, which the ring takes one
// point at a time: the generic kernel is faster (512^2 at 524,288 points: one entry
// 383 us against 921, 8 entries 496 against 1119).
bool grad_on_ring(const Geo& g, const tlgb_interp_plan_info* info) {
  if (g.kernel != TLGB_KERNEL_KAISER_BESSEL && std::max(g.NT[1], g.NT[2]) > 4) return false;
  return g.cplx && g.ndim == 2 && rec_taps(g) == 4 && info->off_records > 0;
}
int64_t grad2_runs(const Geo& g, const tlgb_interp_plan_info* info) {
  const int64_t ncg = cdiv(std::max<long long>(g.nbatch, 1), 8), items = std::max<int64_t>(info->n_fwd_items, 1);
  int64_t run = ncg;
  while (run > 1 && items * cdiv(ncg, run) < sm_count()) run = cdiv(run, 2);
  return cdiv(ncg, run);
}
// the runs' partial results, then (points in random order) the point-major values
size_t grad2_partial_bytes(const Geo& g, const tlgb_interp_plan_info* info) {
  const int64_t n = grad2_runs(g, info);
  return n > 1 ? align_up((size_t)n * g.npts * 2 * sizeof(float), 256) : 0;
}
size_t grad2_scratch_bytes(const Geo& g, const tlgb_interp_plan_info* info) {
  const size_t at = (info->kernel_key & kScattered) && g.nbatch >= 4 ? (size_t)cdiv(g.nbatch, 8) * g.npts * 64 : 0;
  return grad2_partial_bytes(g, info) + at;
}

int check_plan(const Geo& g, const tlgb_interp_plan_info* info, const void* plan) {
  if (!info || !plan) TLGB_FAIL(TLGB_ERR_INVALID, "missing plan");
  for (int e = 0; e < 3; ++e)
    if (info->tile[e] != g.T[e] || info->n_tile[e] != g.nt[e])
      TLGB_FAIL(TLGB_ERR_INVALID, "plan was built for another grid");
  if (((info->off_records > 0 && records_ok(g)) || info->n_blk_items > 0) && (info->kernel_key & ~(kScattered | kPartial)) != kernel_key(g))
    TLGB_FAIL(TLGB_ERR_INVALID, "plan was built for another kernel, norm or beta (its tap weights are stored)");
  return TLGB_OK;
}

using CtxGetCurrentFn = CUresult (*)(CUcontext*);

CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<CtxGetCurrentFn>(p);
  });
  return fn;
}

// The current context's id, unique for the life of the process (its handle is
// not: contexts made one after the other get the same one); 0 = not known.
unsigned long long context_id() {
  using Fn = CUresult (*)(CUcontext, unsigned long long*);
  static Fn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<Fn>(p);
  });
  CtxGetCurrentFn get = ctx_get_current();
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!fn || !get || get(&ctx) != CUDA_SUCCESS || !ctx || fn(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// A kernel's shared-memory limit and carveout, set once per context (they belong
// to its module) and again when a launch needs more: set on every launch they
// add 3 us to a call of a small problem (64^2 ungrid and grid 45 -> 51 us).
int set_smem(const void* kernel, size_t bytes) {
  struct Entry {
    unsigned long long ctx;
    const void* kernel;
    size_t bytes;
  };
  static std::mutex mu;
  static std::vector<Entry> known;
  const unsigned long long ctx = context_id();
  std::lock_guard<std::mutex> lock(mu);
  Entry* mine = nullptr;
  for (Entry& e : known)
    if (ctx != 0 && e.kernel == kernel && e.ctx == ctx) {
      if (e.bytes >= bytes) return TLGB_OK;
      mine = &e;
    }
  TLGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  TLGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  if (mine) {
    mine->bytes = bytes;
  } else if (ctx != 0) {
    if (known.size() >= 1024) known.clear();  // contexts come and go in a long-lived host
    known.push_back({ctx, kernel, bytes});
  }
  return TLGB_OK;
}
template <typename F>
int set_smem(F* kernel, size_t bytes) {
  return set_smem(reinterpret_cast<const void*>(kernel), bytes);
}

}  // namespace
}  // namespace tlgb

using namespace tlgb;

extern "C" int tlgb_interp_plan_count(const tlgb_interp_desc* d, const float* locs, void* counter, int64_t* blk_entries,
                                      tlgb_stream_t stream) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  if (!blk_entries || !counter || (g.npts > 0 && !locs)) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  if ((uintptr_t)counter & 7) TLGB_FAIL(TLGB_ERR_INVALID, "plan count: the counter must be 8-byte aligned");
  *blk_entries = -1;
  if (g.nrow != 3 || g.npts == 0) return TLGB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  auto* total = static_cast<unsigned long long*>(counter);
  TLGB_CUDA(cudaMemsetAsync(total, 0, 8, s));
  const unsigned nb = (unsigned)cdiv(g.npts, kPlanPts);
  (std::max(g.NT[0], std::max(g.NT[1], g.NT[2])) <= 5 ? plan_points_kernel<5> : plan_points_kernel<9>)<<<nb, kPlanPts, 0, s>>>(
      g, locs, nullptr, nullptr, nullptr, total);
  TLGB_CHECK_LAUNCH();
  unsigned long long n = 0;
  TLGB_CUDA(cudaMemcpyAsync(&n, total, 8, cudaMemcpyDeviceToHost, s));
  TLGB_CUDA(cudaStreamSynchronize(s));
  *blk_entries = (int64_t)n;
  return TLGB_OK;
}

extern "C" int tlgb_interp_plan_size_counted(const tlgb_interp_desc* d, int64_t blk_entries, size_t* plan_bytes,
                                             size_t* tmp_bytes) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  const PlanLayout L = layout(g, blk_entries);
  if (L.e_max >= (1ll << 31)) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "too many points for one plan");
  if (plan_bytes) *plan_bytes = (size_t)L.bytes;
  if (tmp_bytes) *tmp_bytes = (size_t)L.t_bytes;
  return TLGB_OK;
}

extern "C" int tlgb_interp_plan_size(const tlgb_interp_desc* d, size_t* plan_bytes, size_t* tmp_bytes) {
  return tlgb_interp_plan_size_counted(d, -1, plan_bytes, tmp_bytes);
}

extern "C" int tlgb_interp_plan_build(const tlgb_interp_desc* d, const float* locs, void* plan, size_t plan_bytes,
                                      void* tmp, size_t tmp_bytes, tlgb_interp_plan_info* info,
                                      tlgb_stream_t stream) {
  return tlgb_interp_plan_build_counted(d, -1, locs, plan, plan_bytes, tmp, tmp_bytes, info, stream);
}

extern "C" int tlgb_interp_plan_build_counted(const tlgb_interp_desc* d, int64_t blk_entries, const float* locs, void* plan,
                                              size_t plan_bytes, void* tmp, size_t tmp_bytes, tlgb_interp_plan_info* info,
                                              tlgb_stream_t stream) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  const PlanLayout L = layout(g, blk_entries);
  if (L.e_max >= (1ll << 31)) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "too many points for one plan");
  if (L.nblocks == 0) g.nrow = 0;
  if (!info || !plan || !tmp || (g.npts > 0 && !locs)) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  if (plan_bytes < (size_t)L.bytes || tmp_bytes < (size_t)L.t_bytes) TLGB_FAIL(TLGB_ERR_WORKSPACE, "plan workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  char* P = (char*)plan;
  char* Tm = (char*)tmp;
  const bool blocks = L.nblocks > 0;
  const PlanUnits U = plan_units(g, L.ntiles, blocks);
  int4* win = (int4*)(Tm + L.t_win);
  uint4* sums = (uint4*)(Tm + L.t_sums);
  uint4* homes = (uint4*)(Tm + L.t_homes);
  uint32_t* cnt = (uint32_t*)(Tm + L.t_cnt);
  uint32_t* tstart = (uint32_t*)(Tm + L.t_tstart);
  uint32_t* bstart = (uint32_t*)(Tm + L.t_bstart);
  if (g.npts == 0) TLGB_CUDA(cudaMemsetAsync(cnt, 0, 16 * 4, s));  // the scans write every count
  // the sort of both lists: the pairs are emitted where an even or odd number
  // of passes leaves them in the plan
  SortJob jobs[2];
  const int njobs = blocks ? 2 : 1;
  auto bits_for = [](int64_t n) {
    int b = 1;
    while ((1ll << b) < n) ++b;
    return b;
  };
  const int tbits = bits_for(2 * L.ntiles), bbits = blocks ? bits_for(L.nblocks) : 1;
  const int odd = std::max(radix_passes(tbits), radix_passes(bbits)) & 1;
  for (int i = 0; i < njobs; ++i) {
    int32_t* fin = (int32_t*)(P + (i ? L.off_blk_entries : L.off_entries));
    int32_t* alt = (int32_t*)(Tm + L.t_vals[i]);
    jobs[i] = {{(uint32_t*)(Tm + L.t_keys[i][0]), (uint32_t*)(Tm + L.t_keys[i][1])},
               {odd ? alt : fin, odd ? fin : alt},
               (uint32_t*)(Tm + L.t_counts[i]), cnt + i, i ? L.eb_max : L.e_max, i ? bbits : tbits};
  }
  if (g.npts > 0) {
    const unsigned nb = (unsigned)cdiv(g.npts, kPlanPts);
    float* rows = blocks ? (float*)(P + L.off_blk_rows) : nullptr;
    const size_t sm = blocks ? (size_t)kPlanPts * row_floats(g.ndim, g.nrow) * 4 : 0;
    const int maxnt = std::max(g.NT[0], std::max(g.NT[1], g.NT[2]));
    auto points = [&](auto* k) -> int {
      TLGB_TRY(set_smem(k, sm));
      k<<<nb, kPlanPts, sm, s>>>(g, locs, win, rows, sums, nullptr);
      TLGB_CHECK_LAUNCH();
      return TLGB_OK;
    };
    TLGB_TRY(maxnt <= 5 ? points(plan_points_kernel<5>) : (maxnt <= 9 ? points(plan_points_kernel<9>) : points(plan_points_kernel<NTMAX>)));
    plan_scan_kernel<<<1, 1024, 0, s>>>({sums, (long long)nb, cnt, blocks ? (uint32_t)L.eb_max : 0u}, {}, {});
    TLGB_CHECK_LAUNCH();
    plan_emit_kernel<<<nb, kPlanPts, 0, s>>>(g, win, sums, jobs[0].keys[0], jobs[0].vals[0],
                                             blocks ? jobs[1].keys[0] : nullptr, blocks ? jobs[1].vals[0] : nullptr,
                                             (uint32_t)L.eb_max);
    TLGB_CHECK_LAUNCH();
    TLGB_TRY(radix_sort_jobs(jobs, njobs, s));
  }
  const int64_t nstart = 2 * L.ntiles + 1 + (blocks ? L.nblocks + 1 : 0);
  plan_starts_kernel<<<(unsigned)cdiv(nstart, 256), 256, 0, s>>>(jobs[0].keys[odd], blocks ? jobs[1].keys[odd] : nullptr,
                                                                 cnt, 2 * L.ntiles, blocks ? L.nblocks : -1, tstart,
                                                                 bstart);
  TLGB_CHECK_LAUNCH();

  // Work items. Results do not depend on their order, because every item
  // writes its own tile, block, slot or points.
  const unsigned row_ctas = (unsigned)cdiv(U.nrows, kPlanPts), unit_ctas = (unsigned)U.tile_ctas + row_ctas;
  plan_count_items_kernel<<<unit_ctas, kPlanPts, 0, s>>>(U, tstart, bstart, fwd_chunk(g), (int)kAdjChunk, sums, homes);
  TLGB_CHECK_LAUNCH();
  plan_scan_kernel<<<3, 1024, 0, s>>>({sums, U.tile_ctas, cnt + 4}, {sums + U.tile_ctas, (long long)row_ctas, cnt + 8},
                                      {homes, U.tile_ctas, cnt + 12});
  TLGB_CHECK_LAUNCH();
  int4* adj_any = (int4*)(Tm + L.t_items[0]);
  int4* bsplit_any = blocks ? (int4*)(Tm + L.t_items[1]) : nullptr;
  // the keys' buffers are free again: they order the items
  SortJob order[2];
  for (int i = 0; i < njobs; ++i)
    order[i] = {{jobs[i].keys[0], jobs[i].keys[1]},
                {(int32_t*)(Tm + L.t_order[i]), (int32_t*)(Tm + L.t_vals[i])},
                jobs[i].counts, cnt + (i ? 10 : 5), i ? L.max_blk_split : L.max_adj, i ? 16 : 11};
  plan_emit_items_kernel<<<unit_ctas, kPlanPts, 0, s>>>(
      U, tstart, bstart, fwd_chunk(g), (int)kAdjChunk, sums, homes, (int4*)(P + L.off_fwd), adj_any, order[0].keys[0],
      order[0].vals[0], (int4*)(P + L.off_split), blocks ? (int4*)(P + L.off_blk_items) : nullptr, bsplit_any,
      blocks ? order[1].keys[0] : nullptr, blocks ? order[1].vals[0] : nullptr);
  TLGB_CHECK_LAUNCH();
  if (L.off_recs > 0) {
    const int4* fwd = (const int4*)(P + L.off_fwd);
    const int32_t* entries = (const int32_t*)(P + L.off_entries);
    char* R = P + L.off_recs;
    const unsigned n = (unsigned)L.max_fwd;
    int32_t* rank = g.ndim == 3 ? (int32_t*)(P + rank_offset(g, L.off_recs)) : nullptr;
    if (rank) TLGB_CUDA(cudaMemsetAsync(rank, 0xff, (size_t)g.npts * 4, s));  // -1: no taps
    const float* rows = blocks ? (const float*)(P + L.off_blk_rows) : nullptr;
    auto records = [&](auto* from_rows, auto* from_locs, auto* out) {
      (blocks ? from_rows : from_locs)<<<n, 128, 0, s>>>(g, cnt, win, rows, fwd, entries, locs, out, rank, cnt + 15);
    };
    if (g.ndim == 3)
      records(plan_records_kernel<3, 4, true>, plan_records_kernel<3, 4, false>, (GatherRec<3, 4>*)R);
    else if (rec_taps(g) == 4)
      records(plan_records_kernel<2, 4, true>, plan_records_kernel<2, 4, false>, (GatherRec<2, 4>*)R);
    else
      records(plan_records_kernel<2, 8, true>, plan_records_kernel<2, 8, false>, (GatherRec<2, 8>*)R);
    TLGB_CHECK_LAUNCH();
  }
  const int64_t onmax = std::max(L.max_adj, L.max_blk_split);
  if (onmax <= kRankItems) {
    plan_rank_kernel<<<dim3((unsigned)cdiv(onmax, 256), (unsigned)njobs), 256, 0, s>>>(
        cnt, adj_any, order[0].keys[0], (int4*)(P + L.off_adj), bsplit_any, blocks ? order[1].keys[0] : nullptr,
        blocks ? (int4*)(P + L.off_blk_split) : nullptr);
    TLGB_CHECK_LAUNCH();
  } else {
    TLGB_TRY(radix_sort_jobs(order, njobs, s));
    const int ofin = std::max(radix_passes(order[0].bits), blocks ? radix_passes(order[1].bits) : 1) & 1;
    plan_order_kernel<<<dim3((unsigned)std::min<int64_t>(cdiv(onmax, 256), 8 * sm_count()), (unsigned)njobs), 256, 0, s>>>(
        cnt, adj_any, order[0].vals[ofin], (int4*)(P + L.off_adj), bsplit_any, blocks ? order[1].vals[ofin] : nullptr,
        blocks ? (int4*)(P + L.off_blk_split) : nullptr);
    TLGB_CHECK_LAUNCH();
  }
  uint32_t c[16];
  TLGB_CUDA(cudaMemcpyAsync(c, cnt, sizeof(c), cudaMemcpyDeviceToHost, s));
  TLGB_CUDA(cudaStreamSynchronize(s));
  if (c[3]) TLGB_FAIL(TLGB_ERR_INVALID, "interp plan: the points have more (point, block) pairs than were counted");
  if ((int64_t)c[4] > L.max_fwd || (int64_t)c[5] > L.max_adj || (blocks && ((int64_t)c[8] > L.max_blk_items || (int64_t)c[10] > L.max_blk_split)))
    TLGB_FAIL(TLGB_ERR_DEVICE, "work list larger than its bound");

  memset(info, 0, sizeof(*info));
  info->n_entries = c[0];
  info->n_tiles = L.ntiles;
  for (int e = 0; e < 3; ++e) {
    info->tile[e] = g.T[e];
    info->n_tile[e] = g.nt[e];
  }
  info->n_fwd_items = c[4];
  info->n_adj_items = c[5];
  info->n_partials = c[6];
  info->n_split_tiles = c[7];
  info->chunk = kAdjChunk;
  info->off_entries = L.off_entries;
  info->off_fwd_items = L.off_fwd;
  info->off_adj_items = L.off_adj;
  info->off_split = L.off_split;
  info->plan_bytes = L.bytes;
  info->off_records = L.off_recs;
  info->kernel_key = L.off_recs > 0 || blocks ? kernel_key(g) : 0;
  if (2ll * c[15] > (int64_t)c[14]) info->kernel_key |= kScattered;
  if (c[13]) info->kernel_key |= kPartial;
  info->n_home = c[2];
  if (blocks) {
    info->n_blk_entries = c[1];
    info->n_blk_items = c[8];
    info->n_blk_partials = c[9];
    info->n_blk_split = c[10];
    info->off_blk_entries = L.off_blk_entries;
    info->off_blk_items = L.off_blk_items;
    info->off_blk_split = L.off_blk_split;
    info->off_blk_rows = L.off_blk_rows;
  }
  return TLGB_OK;
}

namespace tlgb {
namespace {

// Batch entries per group of the block gridding: 1, 2 or 4 for 3D batches of
// at most 4 entries (adj_bn_kernel), else 8 (adj_b3_kernel).
int blk_entries(const Geo& g) {
  if (g.ndim != 3 || g.nbatch > 4) return 8;
  return g.nbatch <= 1 ? 1 : (g.nbatch <= 2 ? 2 : 4);
}

// bytes of the block path's partial blocks: 64 cells x E complex entries per
// part and group
size_t blk_partial_bytes(const tlgb_interp_plan_info* info, int64_t ncg, int E) {
  return align_up((size_t)info->n_blk_partials * ncg * 64 * 2 * E * sizeof(float), 256);
}

// Gridding scratch: the partial tiles of split tiles (block path: the partial
// blocks and the work counters), then (8-entry paths) the point values
// transposed to point-major order.
void adj_scratch_parts(const Geo& g, const tlgb_interp_plan_info* info, size_t& partial_bytes, size_t& tv_bytes) {
  if (on_blocks(g, info)) {
    const int E = blk_entries(g);
    const int64_t ncg = E < 8 ? 1 : cdiv(std::max<long long>(g.nbatch, 1), 8);
    partial_bytes = blk_partial_bytes(info, ncg, E) + align_up((size_t)ncg * sizeof(int), 256);
    tv_bytes = E < 8 ? 0 : (size_t)ncg * g.npts * 8 * 8;  // adj_bn_kernel reads the values in place
    return;
  }
  const int cg = adj_cg(g);
  const int64_t ncg = cdiv(std::max<long long>(g.nbatch, 1), cg);
  partial_bytes = align_up((size_t)info->n_partials * ncg * tile_floats(g, cg) * sizeof(float), 256);
  tv_bytes = 0;
}
}  // namespace
}  // namespace tlgb

extern "C" int tlgb_interp_adjoint_scratch_size(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info,
                                                size_t* bytes) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  if (!info || !bytes) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  size_t pb = 0, tb = 0;
  adj_scratch_parts(g, info, pb, tb);
  *bytes = pb + tb;
  return TLGB_OK;
}

namespace tlgb {
namespace {

template <int N, int NDIM, int NTB>
int launch_fwd_t2(const Geo& g, int cg, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                  const void* grid, void* out, cudaStream_t s) {
  const int64_t ncg = cdiv(g.nbatch, cg);
  // Real values on a plan with gather records: its items hold at most 256 points, a
  // batch of 32 for 8 warps. 16 would leave half of them idle and one CTA per SM
  // (2D, 131,072 points on 321 x 203: 82 -> 48 us for one entry, 99 -> 63 for 8).
  int nw = NWF;
  auto* k = interp_fwd_kernel<N, NDIM, NTB, NWF>;
  if constexpr (N <= 2 && NDIM >= 2)
    if (records_ok(g)) nw = 8, k = interp_fwd_kernel<N, NDIM, NTB, 8>;
  const size_t sm = fwd_smem(g, cg, nw);
  TLGB_TRY(set_smem(k, sm));
  // Tiles of many points are several such items: up to 4 in a CTA, unless that
  // leaves fewer than 8 CTAs per SM (2D) or 2 (3D, whose regions cost more to
  // stage). 8 entries of 64^3 at 524,288 points: 578 us staged for each item, 346
  // so, 397 with 8 CTAs per SM; of 320^2 at 524,288: 159, 212 with 2.
  int64_t per = nw == 8 ? std::min<int64_t>(4, info->n_fwd_items / std::max<int64_t>(info->n_tiles, 1)) : 1;
  per = std::max<int64_t>(1, std::min<int64_t>(per, info->n_fwd_items * ncg / ((g.ndim == 3 ? 2 : 8) * sm_count())));
  dim3 grd((unsigned)cdiv(info->n_fwd_items, per), (unsigned)ncg);
  k<<<grd, nw * 32, sm, s>>>(g, (const int4*)(P + info->off_fwd_items), (int)info->n_fwd_items, (int)per,
                             (const int32_t*)(P + info->off_entries), locs, (const float*)grid, (float*)out, cg);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

template <int N, int NDIM, int NTB>
int launch_adj_t2(const Geo& g, int cg, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                  const void* vals, void* grid, void* scratch, cudaStream_t s) {
  const int64_t ncg = cdiv(g.nbatch, cg);
  const size_t sm = adj_smem(g, cg);
  auto* k = interp_adj_kernel<N, NDIM, NTB>;
  TLGB_TRY(set_smem(k, sm));
  dim3 grd((unsigned)info->n_adj_items, (unsigned)ncg);
  k<<<grd, 32, sm, s>>>(g, (const int4*)(P + info->off_adj_items), (const int32_t*)(P + info->off_entries), locs,
                       (const float*)vals, (float*)grid, (float*)scratch, cg);
  TLGB_CHECK_LAUNCH();
  if (info->n_split_tiles > 0) {
    dim3 g2((unsigned)info->n_split_tiles, (unsigned)ncg);
    adj_reduce_kernel<<<g2, NTHR, 0, s>>>(g, (const int4*)(P + info->off_split), (const float*)scratch, (float*)grid,
                                          cg, (int)ncg);
    TLGB_CHECK_LAUNCH();
  }
  return TLGB_OK;
}

using sm100::tensor_map_encoder;

// [batch][X][Y][Z] complex64 as a 4D map of 8-byte elements, box edge^2
// (edge^3 in 3D) x cg entries; 0 when TMA cannot be used
int region_map(const Geo& g, const void* grid, int edge, int cg, CUtensorMap& tmap) {
  memset(&tmap, 0, sizeof(tmap));
  auto enc = tensor_map_encoder();
  const uint64_t zb = (uint64_t)g.N[2] * 8;
  if (!enc || (zb % 16) != 0 || ((uintptr_t)grid % 16) != 0) return 0;
  const cuuint64_t dims[4] = {(cuuint64_t)g.N[2], (cuuint64_t)g.N[1], (cuuint64_t)g.N[0], (cuuint64_t)g.nbatch};
  const cuuint64_t strides[3] = {zb, zb * g.N[1], zb * g.N[1] * g.N[0]};
  const cuuint32_t e = (cuuint32_t)edge, box[4] = {e, e, g.ndim == 3 ? e : 1, (cuuint32_t)cg};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void*>(grid), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 1 : 0;
}

// A unit is an item and `run` groups: all of them (an item's records are
// fetched once) unless that leaves fewer than 24 units per CTA.
template <int NDIM, int KT, int CG, int NW, int NST, int CTAS>
int launch_gather(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs, const void* grid,
                  void* out, cudaStream_t s, float* sorted = nullptr) {
  if ((uintptr_t)P & 15) TLGB_FAIL(TLGB_ERR_INVALID, "interp forward: the plan must be 16-byte aligned");
  CUtensorMap tmap;
  const int use_tma = region_map(g, grid, region_edge<NDIM, KT>(), CG, tmap);
  constexpr size_t sm = gather_smem<NDIM, KT, CG, NW, NST>();
  auto* k = gather_kernel<NDIM, KT, CG, NW, NST, CTAS, true>;
  if constexpr (KT == 4)  // the check costs nothing at KT = 8
    if (!(info->kernel_key & kPartial)) k = gather_kernel<NDIM, KT, CG, NW, NST, CTAS, false>;
  TLGB_TRY(set_smem(k, sm));
  const int64_t ncg = cdiv(g.nbatch, CG), items = info->n_fwd_items, ctas = (int64_t)CTAS * sm_count();
  int64_t run = ncg;
  // (item, run of groups) units go round the CTAs in turn, and items differ in
  // points: 24 units per CTA even out what 6 do not (320^2 x 20 at width 6: 178
  // -> 127 us; 320^2 x 256: 562 -> 526 us), at 48 the records' reloads show
  // (ragged 3D x 12: 247 -> 326 us)
  while (run > 1 && items * cdiv(ncg, run) < 24 * ctas) run = cdiv(run, 2);
  const int64_t nruns = cdiv(ncg, run), nunits = items * nruns;
  if (nunits >= (1ll << 31) - ctas) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "interp forward: too many points and batch entries in one call");
  k<<<(unsigned)std::min(nunits, ctas), NW * 32 + kGatherProd, sm, s>>>(
      tmap, use_tma, g, (const int4*)(P + info->off_fwd_items), (int)nruns, (int)run, (int)nunits,
      (const GatherRec<NDIM, KT>*)(P + info->off_records), locs, (const float*)grid, (float*)out, sorted);
  TLGB_CHECK_LAUNCH();
  return TLGB_OK;
}

// Points in random order: their 8-byte results are scattered over an output
// that L2 cannot hold, and every 32-byte sector is written back in pieces. With
// scratch the results go in the items' order (32 contiguous bytes per point
// and group) and a second pass brings them to the points' order. It pays where
// the output is a large part of L2: 8 x 2^21 points (134 MB) 720 -> 590 us.
size_t forward_scratch_bytes(const Geo& g, const tlgb_interp_plan_info* info) {
  if (g.ndim != 3 || !g.cplx || g.nbatch < 3 || !records_ok(g) || info->off_records == 0 || !(info->kernel_key & kScattered))
    return 0;
  if (g.nbatch * g.npts * 8 < (48ll << 20) || cdiv(g.nbatch, 4) > 65535) return 0;
  return (size_t)cdiv(g.nbatch, 4) * g.npts * 32;
}

// Ring shapes: what fits 227 KB with two record buffers beside it, for the
// fewest groups. 3D stages are 13.8 KB per entry: 4 entries per group in a ring
// of 3 feed 16 consumer warps; small batches run two CTAs per SM.
int launch_gather_any(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                      const void* grid, void* out, cudaStream_t s, void* scratch = nullptr, size_t scratch_bytes = 0) {
  const long long n = g.nbatch;
  if (g.ndim == 3) {
    const size_t need = forward_scratch_bytes(g, info);
    if (need > 0 && scratch && scratch_bytes >= need && ((uintptr_t)scratch & 15) == 0) {
      TLGB_TRY((launch_gather<3, 4, 4, 16, 3, 1>(g, info, P, locs, grid, out, s, (float*)scratch)));
      const dim3 grd((unsigned)cdiv(g.npts, 128), (unsigned)cdiv(n, 4));
      unsort_kernel<<<grd, 256, 0, s>>>((const float4*)scratch, (const int32_t*)(P + rank_offset(g, info->off_records)),
                                        g.npts, n, (float2*)out);
      TLGB_CHECK_LAUNCH();
      return TLGB_OK;
    }
    if (n == 1) return launch_gather<3, 4, 1, 8, 5, 2>(g, info, P, locs, grid, out, s);
    if (n == 2) return launch_gather<3, 4, 2, 16, 5, 1>(g, info, P, locs, grid, out, s);
    return launch_gather<3, 4, 4, 16, 3, 1>(g, info, P, locs, grid, out, s);
  }
  if (rec_taps(g) == 4) {
    if (n == 1) return launch_gather<2, 4, 1, 8, 6, 2>(g, info, P, locs, grid, out, s);
    if (n == 2) return launch_gather<2, 4, 2, 8, 6, 2>(g, info, P, locs, grid, out, s);
    if (n <= 4) return launch_gather<2, 4, 4, 8, 5, 2>(g, info, P, locs, grid, out, s);
    return launch_gather<2, 4, 8, 8, 3, 2>(g, info, P, locs, grid, out, s);
  }
  if (n <= 2) return launch_gather<2, 8, 2, 8, 4, 2>(g, info, P, locs, grid, out, s);
  if (n <= 4) return launch_gather<2, 8, 4, 8, 3, 2>(g, info, P, locs, grid, out, s);
  return launch_gather<2, 8, 8, 16, 4, 1>(g, info, P, locs, grid, out, s);
}

template <int E, int NROW>
int launch_adj_bn(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const void* vals, void* grid,
                  void* scratch, cudaStream_t s) {
  const size_t sm = kBWarps * kBStages * kBC * kBSn * sizeof(float);
  TLGB_TRY(set_smem(adj_bn_kernel<E, NROW>, sm));
  if (((uintptr_t)P & 15) || ((uintptr_t)scratch & 15))
    TLGB_FAIL(TLGB_ERR_INVALID, "interp adjoint: plan and scratch must be 16-byte aligned");
  if ((uintptr_t)vals & 7) TLGB_FAIL(TLGB_ERR_INVALID, "interp adjoint: values must be 8-byte aligned");
  // the work counter follows the partial blocks
  int* ctr = reinterpret_cast<int*>(static_cast<char*>(scratch) + blk_partial_bytes(info, 1, E));
  TLGB_CUDA(cudaMemsetAsync(ctr, 0, sizeof(int), s));
  const int64_t nctas = std::min<int64_t>(cdiv(info->n_blk_items, kBWarps), (int64_t)kBnCtas * sm_count());
  adj_bn_kernel<E, NROW><<<(unsigned)std::max<int64_t>(nctas, 1), kBWarps * 32, sm, s>>>(
      g, (const int4*)(P + info->off_blk_items), (int)info->n_blk_items, (const uint32_t*)(P + info->off_blk_entries),
      (const float*)(P + info->off_blk_rows), (const float2*)vals, (float*)grid, (float*)scratch, ctr);
  TLGB_CHECK_LAUNCH();
  if (info->n_blk_split > 0) {
    adj_reduce_bn_kernel<E><<<(unsigned)info->n_blk_split, 256, 0, s>>>(g, (const int4*)(P + info->off_blk_split),
                                                                       (const float*)scratch, (float*)grid);
    TLGB_CHECK_LAUNCH();
  }
  return TLGB_OK;
}

template <int NDIM, int NROW>
int launch_adj_b3(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                  const void* vals, void* grid, void* scratch, cudaStream_t s) {
  if constexpr (NDIM == 3) {
    switch (blk_entries(g)) {
      case 1: return launch_adj_bn<1, NROW>(g, info, P, vals, grid, scratch, s);
      case 2: return launch_adj_bn<2, NROW>(g, info, P, vals, grid, scratch, s);
      case 4: return launch_adj_bn<4, NROW>(g, info, P, vals, grid, scratch, s);
      default: break;
    }
  }
  const int64_t ncg = cdiv(g.nbatch, 8);
  const size_t sm = kBWarps * kBStages * kBC * kBS * sizeof(float);
  TLGB_TRY(set_smem(adj_b3_kernel<NDIM, NROW>, sm));
  // 16-byte asynchronous copies of the weight rows and transposed values
  if (((uintptr_t)P & 15) || ((uintptr_t)scratch & 15))
    TLGB_FAIL(TLGB_ERR_INVALID, "interp adjoint: plan and scratch must be 16-byte aligned");
  if ((uintptr_t)vals & 7) TLGB_FAIL(TLGB_ERR_INVALID, "interp adjoint: values must be 8-byte aligned");
  // the work counters (one per group of 8 entries) follow the partial blocks
  int* ctr = reinterpret_cast<int*>(static_cast<char*>(scratch) + blk_partial_bytes(info, ncg, 8));
  const float4* tv = nullptr;
  if (g.tv_off >= 0 && g.npts > 0) {
    float2* t = reinterpret_cast<float2*>(static_cast<char*>(scratch) + g.tv_off);
    dim3 gt((unsigned)cdiv(g.npts, kTrPts), (unsigned)ncg);
    transpose_vals_kernel<<<gt, 256, 0, s>>>((const float2*)vals, g.npts, g.nbatch, t, ctr);
    TLGB_CHECK_LAUNCH();
    tv = reinterpret_cast<const float4*>(t);
  } else {
    TLGB_CUDA(cudaMemsetAsync(ctr, 0, (size_t)ncg * sizeof(int), s));
  }
  // persistent: kB3Ctas CTAs per SM (fewer when there are few units), any
  // number of which may be resident at once; (group, item) units are counted
  // in 32 bits, the tickets of all warps above their number included
  const int64_t nitems = info->n_blk_items, max_ctas = (int64_t)kB3Ctas * sm_count();
  const int64_t per = std::max<int64_t>(1, (((int64_t)1 << 31) - 1 - 16 * max_ctas) / std::max<int64_t>(nitems, 1));
  for (int64_t cg0 = 0; cg0 < ncg; cg0 += per) {
    const int64_t nunits = nitems * std::min(per, ncg - cg0);
    const int64_t nctas = std::max<int64_t>(1, std::min(cdiv(nunits, kBWarps), max_ctas));
    adj_b3_kernel<NDIM, NROW><<<(unsigned)nctas, kBWarps * 32, sm, s>>>(
        g, (const int4*)(P + info->off_blk_items), (int)nitems, (int)nunits, (int)cg0, (int)ncg,
        (const uint32_t*)(P + info->off_blk_entries), (const float*)(P + info->off_blk_rows), (const float2*)vals, tv,
        (float*)grid, (float*)scratch, ctr + cg0);
    TLGB_CHECK_LAUNCH();
  }
  if (info->n_blk_split > 0) {
    dim3 g2((unsigned)info->n_blk_split, (unsigned)ncg);
    adj_reduce_b3_kernel<NDIM><<<g2, 256, 0, s>>>(g, (const int4*)(P + info->off_blk_split),
                                                 (const float*)scratch, (float*)grid);
    TLGB_CHECK_LAUNCH();
  }
  return TLGB_OK;
}

// floats per coil unit: 2 batch entries per unit when the group size is even
inline int unit_floats(const Geo& g, int cg) { return (g.cplx ? 2 : 1) * ((cg % 2 == 0) ? 2 : 1); }

template <int NDIM, int NTB>
int dispatch_fwd_n(const Geo& g, int cg, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                   const void* grid, void* out, cudaStream_t s) {
  switch (unit_floats(g, cg)) {
    case 4: return launch_fwd_t2<4, NDIM, NTB>(g, cg, info, P, locs, grid, out, s);
    case 2: return launch_fwd_t2<2, NDIM, NTB>(g, cg, info, P, locs, grid, out, s);
    default: return launch_fwd_t2<1, NDIM, NTB>(g, cg, info, P, locs, grid, out, s);
  }
}

template <int NDIM, int NTB>
int dispatch_adj_n(const Geo& g, int cg, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                   const void* vals, void* grid, void* scratch, cudaStream_t s) {
  switch (unit_floats(g, cg)) {
    case 4: return launch_adj_t2<4, NDIM, NTB>(g, cg, info, P, locs, vals, grid, scratch, s);
    case 2: return launch_adj_t2<2, NDIM, NTB>(g, cg, info, P, locs, vals, grid, scratch, s);
    default: return launch_adj_t2<1, NDIM, NTB>(g, cg, info, P, locs, vals, grid, scratch, s);
  }
}

int launch_fwd_rows(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs,
                    const void* grid, void* out, cudaStream_t s) {
  const int cg = fwd_cg(g);
  const bool small = ntb_for(g) == 5;
  if (g.ndim == 3) return small ? dispatch_fwd_n<3, 5>(g, cg, info, P, locs, grid, out, s) : dispatch_fwd_n<3, 9>(g, cg, info, P, locs, grid, out, s);
  if (g.ndim == 2) return small ? dispatch_fwd_n<2, 5>(g, cg, info, P, locs, grid, out, s) : dispatch_fwd_n<2, 16>(g, cg, info, P, locs, grid, out, s);
  return small ? dispatch_fwd_n<1, 5>(g, cg, info, P, locs, grid, out, s) : dispatch_fwd_n<1, 16>(g, cg, info, P, locs, grid, out, s);
}

// Launch grids have at most 65535 rows of batch groups. Wide 3D kernels
// stage fewer than 8 entries per group (their region would not fit shared
// memory), so a batch below TLGB_INTERP_MAX_BATCH can still need more rows:
// batch entries are independent, so such a batch is launched in parts.
int launch_fwd(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs, const void* grid,
               void* out, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  if (g.cplx && records_ok(g) && info->off_records > 0) return launch_gather_any(g, info, P, locs, grid, out, s, scratch, scratch_bytes);
  const int64_t per = (int64_t)65535 * fwd_cg(g);
  if (g.nbatch <= per) return launch_fwd_rows(g, info, P, locs, grid, out, s);
  const int64_t vs = value_size(g), vol = (int64_t)g.N[0] * g.N[1] * g.N[2];
  for (int64_t b0 = 0; b0 < g.nbatch; b0 += per) {
    Geo gc = g;
    gc.nbatch = std::min(per, (int64_t)g.nbatch - b0);
    TLGB_TRY(launch_fwd_rows(gc, info, P, locs, static_cast<const char*>(grid) + b0 * vol * vs,
                             static_cast<char*>(out) + b0 * g.npts * vs, s));
  }
  return TLGB_OK;
}

int launch_adj(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs, const void* vals,
               void* grid, void* scratch, cudaStream_t s) {
  // adj_cg is min(nbatch, 8): TLGB_INTERP_MAX_BATCH keeps the grid at <= 65535 rows
  if (cdiv(g.nbatch, adj_cg(g)) > 65535) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "interp adjoint: too many batch groups");
  if (on_blocks(g, info)) {
    if (g.ndim == 3)
      return g.nrow == 3 ? launch_adj_b3<3, 3>(g, info, P, locs, vals, grid, scratch, s)
                         : launch_adj_b3<3, 2>(g, info, P, locs, vals, grid, scratch, s);
    return g.nrow == 3 ? launch_adj_b3<2, 3>(g, info, P, locs, vals, grid, scratch, s)
                       : launch_adj_b3<2, 2>(g, info, P, locs, vals, grid, scratch, s);
  }
  const int cg = adj_cg(g);
  const bool small = ntb_for(g) == 5;
  if (g.ndim == 3) return small ? dispatch_adj_n<3, 5>(g, cg, info, P, locs, vals, grid, scratch, s) : dispatch_adj_n<3, 9>(g, cg, info, P, locs, vals, grid, scratch, s);
  if (g.ndim == 2) return small ? dispatch_adj_n<2, 5>(g, cg, info, P, locs, vals, grid, scratch, s) : dispatch_adj_n<2, 16>(g, cg, info, P, locs, vals, grid, scratch, s);
  return small ? dispatch_adj_n<1, 5>(g, cg, info, P, locs, vals, grid, scratch, s) : dispatch_adj_n<1, 16>(g, cg, info, P, locs, vals, grid, scratch, s);
}

int launch_grad2(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs, const void* grid,
                 const void* a, float* grad, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  if ((uintptr_t)P & 15) TLGB_FAIL(TLGB_ERR_INVALID, "trajectory gradient: the plan must be 16-byte aligned");
  const int64_t ncg = cdiv(g.nbatch, 8);
  int64_t nruns = grad2_runs(g, info);
  const size_t part = grad2_partial_bytes(g, info);
  if (nruns > 1 && (!scratch || scratch_bytes < part || ((uintptr_t)scratch & 7))) nruns = 1;
  const float2* at = nullptr;
  if (scratch && ((uintptr_t)scratch & 15) == 0 && grad2_scratch_bytes(g, info) > part && scratch_bytes >= grad2_scratch_bytes(g, info)) {
    float2* t = reinterpret_cast<float2*>(static_cast<char*>(scratch) + part);
    transpose_vals_kernel<<<dim3((unsigned)cdiv(g.npts, kTrPts), (unsigned)ncg), 256, 0, s>>>((const float2*)a, g.npts,
                                                                                              g.nbatch, t, nullptr);
    TLGB_CHECK_LAUNCH();
    at = t;
  }
  const int64_t run = cdiv(ncg, nruns), nunits = info->n_fwd_items * nruns;
  if (nunits >= (1ll << 31) - sm_count()) TLGB_FAIL(TLGB_ERR_UNSUPPORTED, "trajectory gradient: too many points and batch entries in one call");
  const long long n = (long long)g.npts * 2;
  float* partial = static_cast<float*>(scratch);
  if (nruns > 1 && info->n_home < g.npts)  // points without taps get no partial writes
    TLGB_CUDA(cudaMemsetAsync(partial, 0, (size_t)nruns * n * sizeof(float), s));
  CUtensorMap tmap;
  const int use_tma = region_map(g, grid, 20, 8, tmap);
  auto* k = at ? grad2_kernel<true> : grad2_kernel<false>;
  TLGB_TRY(set_smem(k, grad2_smem()));
  k<<<(unsigned)std::min<int64_t>(nunits, sm_count()), kGradWarps * 32 + kGatherProd, grad2_smem(), s>>>(
      tmap, use_tma, g, (const int4*)(P + info->off_fwd_items), (int)nruns, (int)run, (int)nunits,
      (const GatherRec<2, 4>*)(P + info->off_records), locs, (const float*)grid, at ? at : (const float2*)a, grad, partial);
  TLGB_CHECK_LAUNCH();
  if (nruns > 1) {
    grad_reduce_kernel<<<(unsigned)cdiv(n, 256), 256, 0, s>>>(partial, (int)nruns, n, grad);
    TLGB_CHECK_LAUNCH();
  }
  return TLGB_OK;
}

template <typename V, int NORM>
int launch_grad(const Geo& g, const tlgb_interp_plan_info* info, const char* P, const float* locs, const void* grid,
                const void* a, float* grad, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  if constexpr (std::is_same<V, float2>::value && NORM == 1)
    if (grad_on_ring(g, info) && ((uintptr_t)grad & 7) == 0)  // it stores a point's two components together
      return launch_grad2(g, info, P, locs, grid, a, grad, scratch, scratch_bytes, s);
  const int cg = grad_cg(g, sizeof(PTaps<true>));
  const size_t sm = grad_smem(g, cg, sizeof(PTaps<true>)) + kFwdChunk * 3 * sizeof(float);
  auto* k = interp_grad_kernel<V, NORM>;
  TLGB_TRY(set_smem(k, sm));
  int nsplit = grad_splits(g, info);
  const size_t need = grad_scratch_bytes(g, nsplit);
  if (!scratch || scratch_bytes < need) nsplit = 1;  // one pass over all coil groups per tile
  float* partial = static_cast<float*>(scratch);
  const long long n = (long long)g.npts * g.ndim;
  if (nsplit > 1 && info->n_home < g.npts)  // points without taps get no partial writes
    TLGB_CUDA(cudaMemsetAsync(partial, 0, need, s));
  dim3 grd((unsigned)info->n_fwd_items, (unsigned)nsplit);
  k<<<grd, NTHR, sm, s>>>(g, (const int4*)(P + info->off_fwd_items), (const int32_t*)(P + info->off_entries), locs,
                          (const V*)grid, (const V*)a, grad, cg, (int)kFwdChunk, partial);
  TLGB_CHECK_LAUNCH();
  if (nsplit > 1) {
    grad_reduce_kernel<<<(unsigned)cdiv(n, 256), 256, 0, s>>>(partial, nsplit, n, grad);
    TLGB_CHECK_LAUNCH();
  }
  return TLGB_OK;
}

}  // namespace
}  // namespace tlgb

extern "C" int tlgb_interp_forward_scratch_size(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info,
                                                size_t* bytes) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  if (!info || !bytes) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  *bytes = forward_scratch_bytes(g, info);
  return TLGB_OK;
}

extern "C" int tlgb_interp_forward_scratch(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info,
                                           const void* plan, const float* locs, const void* grid, void* out,
                                           void* scratch, size_t scratch_bytes, tlgb_stream_t stream) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  TLGB_TRY(check_plan(g, info, plan));
  if (g.npts == 0 || g.nbatch == 0) return TLGB_OK;
  if (!locs || !grid || !out) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  if (info->n_home < g.npts)  // points without a valid tap read as zero
    TLGB_CUDA(cudaMemsetAsync(out, 0, (size_t)g.nbatch * g.npts * value_size(g), s));
  if (info->n_fwd_items == 0) return TLGB_OK;
  const char* P = (const char*)plan;
  return launch_fwd(g, info, P, locs, grid, out, scratch, scratch_bytes, s);
}

extern "C" int tlgb_interp_forward(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info, const void* plan,
                                   const float* locs, const void* grid, void* out, tlgb_stream_t stream) {
  return tlgb_interp_forward_scratch(d, info, plan, locs, grid, out, nullptr, 0, stream);
}

extern "C" int tlgb_interp_adjoint(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info, const void* plan,
                                   const float* locs, const void* vals, void* grid, void* scratch,
                                   size_t scratch_bytes, tlgb_stream_t stream) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  TLGB_TRY(check_plan(g, info, plan));
  if (g.nbatch == 0) return TLGB_OK;
  if (!grid || (g.npts > 0 && (!locs || !vals))) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  size_t pb = 0, tb = 0;
  adj_scratch_parts(g, info, pb, tb);
  if (scratch_bytes < pb + tb || (pb + tb > 0 && !scratch)) TLGB_FAIL(TLGB_ERR_WORKSPACE, "adjoint scratch too small");
  g.tv_off = tb > 0 ? (long long)pb : -1;
  cudaStream_t s = (cudaStream_t)stream;
  const char* P = (const char*)plan;
  return launch_adj(g, info, P, locs, vals, grid, scratch, s);
}

extern "C" int tlgb_interp_grad_scratch_size(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info,
                                             size_t* bytes) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  if (!info || !bytes) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  *bytes = grad_on_ring(g, info) ? grad2_scratch_bytes(g, info) : grad_scratch_bytes(g, grad_splits(g, info));
  return TLGB_OK;
}

extern "C" int tlgb_interp_grad_locs(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info, const void* plan,
                                     const float* locs, const void* grid, const void* a, float* grad_locs,
                                     void* scratch, size_t scratch_bytes, tlgb_stream_t stream) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  TLGB_TRY(check_plan(g, info, plan));
  if (g.npts == 0) return TLGB_OK;
  if (!locs || !grid || !a || !grad_locs) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  if (info->n_home < g.npts || g.nbatch == 0)
    TLGB_CUDA(cudaMemsetAsync(grad_locs, 0, (size_t)g.npts * g.ndim * sizeof(float), s));
  if (g.nbatch == 0 || info->n_fwd_items == 0) return TLGB_OK;
  const char* P = (const char*)plan;
  if (g.cplx)
    return g.norm == 1 ? launch_grad<float2, 1>(g, info, P, locs, grid, a, grad_locs, scratch, scratch_bytes, s)
                       : launch_grad<float2, 2>(g, info, P, locs, grid, a, grad_locs, scratch, scratch_bytes, s);
  return g.norm == 1 ? launch_grad<float, 1>(g, info, P, locs, grid, a, grad_locs, scratch, scratch_bytes, s)
                     : launch_grad<float, 2>(g, info, P, locs, grid, a, grad_locs, scratch, scratch_bytes, s);
}

// ------------------------------------------------ gridding without allocation
//
// Some callers cannot allocate device memory at the moment they grid: a
// host framework that hands out memory only from a pool reserved at start-up
// (a scanner's real-time reconstruction loop, a service with a fixed memory
// budget), or an FFI caller (cgo, JNI) that has no allocator of its own and
// for which cudaMalloc would synchronise the device in the middle of a
// pipeline. For them tlgb_interp_adjoint_fixed takes the partial-tile scratch
// of dense tiles from this file-scope device buffer instead of from the
// caller. The buffer is part of the loaded module: every GPU that loads the
// library holds it until the process exits.

namespace tlgb {
namespace {
constexpr size_t kFixedScratchBytes = TLGB_ADJOINT_FIXED_SCRATCH_BYTES;
}  // namespace
}  // namespace tlgb

static __device__ __align__(256) unsigned char g_adjoint_fixed_scratch[tlgb::kFixedScratchBytes];

namespace tlgb {
namespace {

// The buffer's device address differs per CUDA context: the primary context
// of each device, and any context a caller made itself with the driver API
// (FFI hosts often do). The address is looked up once per context, with that
// context current, and remembered by the context's id (its handle may be given
// again, to a context in which the buffer lies elsewhere); the first lookup in a
// context may load the module there, which is when the buffer is allocated on
// that GPU.
std::mutex g_fixed_mu;
std::vector<std::pair<unsigned long long, void*>> g_fixed_addr;

// Device address of the fixed buffer in the current context.
int fixed_scratch_address(void** out) {
  unsigned long long ctx = context_id();
  std::lock_guard<std::mutex> lock(g_fixed_mu);
  for (const auto& e : g_fixed_addr)
    if (ctx != 0 && e.first == ctx) {
      *out = e.second;
      return TLGB_OK;
    }
  // with no context current, this first runtime call makes the current
  // device's primary context current on this thread
  TLGB_CUDA(cudaGetSymbolAddress(out, g_adjoint_fixed_scratch));
  if (ctx == 0) ctx = context_id();
  if (ctx == 0) return TLGB_OK;  // looked up again on the next call
  for (const auto& e : g_fixed_addr)
    if (e.first == ctx) return TLGB_OK;
  g_fixed_addr.emplace_back(ctx, *out);
  return TLGB_OK;
}

}  // namespace
}  // namespace tlgb

extern "C" int tlgb_interp_adjoint_fixed(const tlgb_interp_desc* d, const tlgb_interp_plan_info* info,
                                         const void* plan, const float* locs, const void* vals, void* grid,
                                         tlgb_stream_t stream) {
  Geo g;
  TLGB_TRY(make_geo(d, g));
  TLGB_TRY(check_plan(g, info, plan));
  if (g.nbatch == 0) return TLGB_OK;
  if (!grid || (g.npts > 0 && (!locs || !vals))) TLGB_FAIL(TLGB_ERR_INVALID, "null pointer");
  size_t need = 0, tb = 0;
  adj_scratch_parts(g, info, need, tb);
  if (need > kFixedScratchBytes && on_blocks(g, info)) {
    // narrow batches of a 2D grid need up to 12 times less room for the parts of
    // tiles: 10^6 points on 64^2 at width 6 3.4 MB, the parts of blocks 42 MB
    g.nrow = 0;
    adj_scratch_parts(g, info, need, tb);
  }
  if (need > kFixedScratchBytes)
    TLGB_FAIL(TLGB_ERR_WORKSPACE, "this plan needs " + std::to_string(need) +
                                      " bytes of partial-tile scratch, more than the fixed " +
                                      std::to_string(kFixedScratchBytes) +
                                      "-byte device buffer of tlgb_interp_adjoint_fixed; use "
                                      "tlgb_interp_adjoint with caller scratch");
  // the point-major copy of the values is used only when it fits as well
  g.tv_off = (tb > 0 && need + tb <= kFixedScratchBytes) ? (long long)need : -1;
  void* scratch = nullptr;
  if (need + (g.tv_off >= 0 ? tb : 0) > 0) TLGB_TRY(fixed_scratch_address(&scratch));
  return launch_adj(g, info, (const char*)plan, locs, vals, grid, scratch, (cudaStream_t)stream);
}

extern "C" int tlgb_test_skip_region_copy(int32_t on) {
  return tlgb::g_test_skip_copy.exchange(on == 2 ? 2 : (on ? 1 : 0));
}

extern "C" int tlgb_device_status(int32_t* status, int32_t clear) {
  if (status == nullptr) TLGB_FAIL(TLGB_ERR_INVALID, "status is NULL");
  int v = 0;
  TLGB_CUDA(cudaDeviceSynchronize());
  TLGB_CUDA(cudaMemcpyFromSymbol(&v, tlgb::g_tlgb_status, sizeof(int)));
  if (clear) {
    const int z = 0;
    TLGB_CUDA(cudaMemcpyToSymbol(tlgb::g_tlgb_status, &z, sizeof(int)));
  }
  int vc = 0;
  TLGB_TRY(tlgb::conv_device_status(&vc, clear));
  // debug builds: an index outside its range in a checked access (bit 4)
  int li = 0, lb = 0;
  TLGB_TRY(tlgb::checked_status(&li, clear));
  TLGB_TRY(tlgb::blocks_checked_status(&lb, clear));
  *status = v | vc | ((li | lb) ? 4 : 0);
  return TLGB_OK;
}
