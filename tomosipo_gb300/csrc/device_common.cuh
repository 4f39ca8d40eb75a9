// Device helpers shared by the projector kernels.
#pragma once

#include <cuda_runtime.h>

#include "tsgb_internal.h"

namespace tsgb {

// Per-layout description of a padded forward-projection volume copy, laid
// out [d][a][b] (b fastest) with kPad zero voxels on both sides of a and b.
struct LayoutDev {
  long long offset;
  int n_d, n_a, n_b;
  int o_d, o_a, o_b;
  int stride_d, stride_a;
};

struct LayoutTable {
  LayoutDev l[kMaxLayouts];
  int count;
};

__host__ inline LayoutTable make_layout_table(const tsgb_projector* p) {
  LayoutTable t{};
  const int anchors[3] = {p->g.oz, p->g.oy, p->g.ox};
  t.count = int(p->layouts.size());
  for (int i = 0; i < t.count; ++i) {
    const Layout& L = p->layouts[i];
    LayoutDev& D = t.l[i];
    D.offset = L.offset_elems;
    D.n_d = int(L.n_d);
    D.n_a = int(L.n_a);
    D.n_b = int(L.n_b);
    D.o_d = anchors[L.d];
    D.o_a = anchors[L.a];
    D.o_b = anchors[L.b];
    D.stride_a = int(L.n_b + 2 * kPad);
    D.stride_d = int((L.n_a + 2 * kPad) * (L.n_b + 2 * kPad));
  }
  return t;
}

// Ray through anchored pixel (ut, vt) for one angle: in-plane position on
// plane kt of the dominant axis is (Xa + kt ma, Xb + kt mb).
struct Ray {
  float Xa, ma, Xb, mb;
};

__device__ __forceinline__ Ray ray_general(const AngleParams& ap, float ut, float vt) {
  const float den = fmaf(ap.e[2], vt, fmaf(ap.e[1], ut, ap.e[0]));
  const float inv = 1.0f / den;
  Ray r;
  r.Xa = fmaf(ap.ca[2], vt, fmaf(ap.ca[1], ut, ap.ca[0])) * inv;
  r.ma = fmaf(ap.ma[2], vt, fmaf(ap.ma[1], ut, ap.ma[0])) * inv;
  r.Xb = fmaf(ap.cb[2], vt, fmaf(ap.cb[1], ut, ap.cb[0])) * inv;
  r.mb = fmaf(ap.mb[2], vt, fmaf(ap.mb[1], ut, ap.mb[0])) * inv;
  return r;
}

__device__ __forceinline__ Ray ray_column(const ColumnEntry& c, float vt) {
  Ray r;
  r.Xa = c.Xa;
  r.ma = c.ma;
  r.Xb = fmaf(vt, c.R, c.P);
  r.mb = fmaf(vt, c.S, c.Q);
  return r;
}

// Row or column of the source that covers row or column n of the projector's detector.
__device__ __forceinline__ unsigned source_pixel(const SinoSource& s, int n) {
  return __umulhi(unsigned(n), s.inv_d) >> s.shift;
}

// Pixel (iv, iu) of angle theta, on the detector.
template <bool kSpread>
__device__ __forceinline__ float sino_value(const SinoSource& s, const DeviceGeometry& g, int iv,
                                            int iu, int theta) {
  if (!kSpread) return __ldg(s.y + ((size_t)iv * g.nangles + theta) * g.cols + iu);
  return s.scale * __ldg(s.y + ((size_t)source_pixel(s, iv) * g.nangles + theta) *
                                   source_pixel(s, g.cols) + source_pixel(s, iu));
}

// World length of the ray between consecutive planes of the dominant axis.
__device__ __forceinline__ float ray_step(const AngleParams& ap, const Ray& r) {
  const float vd = ap.vs_d, va = ap.vs_a * r.ma, vb = ap.vs_b * r.mb;
  return sqrtf(fmaf(vd, vd, fmaf(va, va, vb * vb)));
}

// Job of block b in a multi-job launch: the j with start[j] <= b < start[j + 1]
// (start[0] = 0, n jobs).
__device__ __forceinline__ int multi_job_of(const long long* start, int n, long long b) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (b >= start[mid])
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ float tent(float t) { return fmaxf(0.0f, 1.0f - fabsf(t)); }

// Exact floor without the conversion unit: for |t| < 2^22, t + 1.5 * 2^23
// rounded toward -inf (__fadd_rd) is floor(t) + 1.5 * 2^23, an integer-valued
// float (floats there are spaced by 1) whose bit pattern is 0x4B400000 +
// floor(t). So floor(t) as a float is that sum minus kFloorMagic, and as an
// integer its bits minus kFloorBits: add and integer instructions, where
// floorf plus a float-to-int conversion would occupy the conversion (XU) pipe.
constexpr float kFloorMagic = 12582912.0f;
constexpr unsigned kFloorBits = 0x4B400000u;

// Clamp a detector coordinate to +-1e8 before an int conversion (NaN -> -1e8,
// +-inf -> +-1e8), so range bounds never overflow 32-bit integers.
__device__ __forceinline__ float clamp_coord(float c) { return fminf(fmaxf(c, -1.0e8f), 1.0e8f); }

__device__ __forceinline__ bool finite_ray(const Ray& r) {
  return isfinite(r.Xa) && isfinite(r.ma) && isfinite(r.Xb) && isfinite(r.mb);
}

// Narrow [klo, khi] (plane coordinates) to planes where X + k m lies in (lo, hi).
__device__ __forceinline__ void clip_planes(float X, float m, float lo, float hi, float& klo,
                                            float& khi) {
  if (m != 0.0f) {
    const float inv = 1.0f / m;
    const float t1 = (lo - X) * inv, t2 = (hi - X) * inv;
    klo = fmaxf(klo, fminf(t1, t2));
    khi = fminf(khi, fmaxf(t1, t2));
  } else if (!(X > lo && X < hi)) {
    klo = 1.0f;
    khi = 0.0f;
  }
}

// The detector columns whose rays cross a plane within an interval, for 32
// angles at a time with one lane per angle: lane l's angle has columns lo ..
// lo + cnt - 1, entries end - cnt .. end - 1 of the flattened list of all of them.
struct ColumnRanges {
  int lo, cnt, end, theta;
  int total;  // entries of all lanes
};

// solve: the pass's SolveEntry table (two float4 per angle), n the lane's angle;
// the ray of column u crosses plane kt at (A0 + A1 u) / (e0 + e1 u), solved for
// tl and th. Every lane of the warp calls it.
__device__ __forceinline__ ColumnRanges column_ranges(const float4* __restrict__ solve, int n,
                                                      int n_angles, float kt, float tl, float th,
                                                      const DeviceGeometry& g) {
  const int lane = threadIdx.x & 31;
  ColumnRanges r{0, 0, 0, 0, 0};
  if (n < n_angles) {
    const float4 s0 = __ldg(solve + 2 * n);      // ca0, ca1, ma0, ma1
    const float4 s1 = __ldg(solve + 2 * n + 1);  // e0, e1, theta, -
    const float A0 = fmaf(kt, s0.z, s0.x), A1 = fmaf(kt, s0.w, s0.y);
    const float u1 = __fdividef(fmaf(tl, s1.x, -A0), fmaf(-tl, s1.y, A1));
    const float u2 = __fdividef(fmaf(th, s1.x, -A0), fmaf(-th, s1.y, A1));
    r.lo = max(0, (int)floorf(clamp_coord(fminf(u1, u2))) + 1 + g.ou);
    const int hi = min(g.cols - 1, (int)ceilf(clamp_coord(fmaxf(u1, u2))) - 1 + g.ou);
    r.cnt = max(0, hi - r.lo + 1);
    r.theta = __float_as_int(s1.z);
  }
  r.end = r.cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, r.end, o);
    if (lane >= o) r.end += v;
  }
  r.total = __shfl_sync(0xffffffffu, r.end, 31);
  return r;
}

// Column iu of angle theta that list entry t stands for (t < total; else some
// valid or invalid column). Every lane of the warp calls it.
__device__ __forceinline__ void column_of(const ColumnRanges& r, int t, int& iu, int& theta) {
  int m = 0;  // the lane whose range holds t: the number of ranges that end at or before it
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1)
    if (__shfl_sync(0xffffffffu, r.end, m + o - 1) <= t) m += o;
  iu = __shfl_sync(0xffffffffu, r.lo - (r.end - r.cnt), m) + t;
  theta = __shfl_sync(0xffffffffu, r.theta, m);
}

// SIRT epilogue: residual W * (R * (y - A x)) of pixel idx, written where the
// backprojector reads it. s.res is the row-pair sinogram of bp_weight_kernel
// (kRowPad padding rows above and below the detector, zeroed once by the
// caller and never written): the pixel is the first value of its own row's
// pair and the second of the pair one row up. The plain recipe computes the
// same products with separate operations (y - A(x), times R, then the
// backprojector's W pass), rounded the same way.
// With s.zlayout the pairs are column-major (bp_weight_z_kernel): pixel
// (iv, theta, iu) is the first value of pair (theta, iu, iv + kRowPad) and the
// second of the pair before it. Without pairs (s.plain, parallel beams through
// flat.cu) the residual is a plain sinogram.
__device__ __forceinline__ void sirt_residual(const FpSirt& s, const DeviceGeometry& g,
                                              long long idx, float total, float W) {
  const float r = __fmul_rn(__fsub_rn(__ldg(s.y + idx), total), __ldg(s.R + idx));
  const float v = __fmul_rn(W, r);
  if (s.plain) {
    s.res[idx] = v;
    return;
  }
  if (s.zlayout) {
    const long long iu = idx % g.cols, rest = idx / g.cols;
    const long long theta = rest % g.nangles, iv = rest / g.nangles;
    float* e = s.res + 2 * ((theta * g.cols + iu) * (g.rows + 2 * kRowPad) + iv + kRowPad);
    e[0] = v;
    e[-1] = v;
    return;
  }
  const long long rs = (long long)g.nangles * g.cols;
  float* e = s.res + 2 * (idx + kRowPad * rs);
  e[0] = v;
  e[1 - 2 * rs] = v;
}

// Two fp32 values in one 64-bit register pair, and the packed operations on
// them (one issue slot for both halves; each half rounds as the scalar does).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 add2_rd(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Window accumulation: a column between voxels f0 and f0 + 1 of the window
// (f0 in -1 .. kX - 1) adds wl V(z) to voxel f0 and wr V(z) to voxel f0 + 1, for each of
// the kItems stacked items the warp works on, with V(z) of the lane's voxels along z in
// pairs: profile(item, jj). The uniform branch on f0 sits outside the z loop, so each
// profile pair goes straight into the two accumulators it feeds.
template <int kItems, int kX, int kPairs, int kM, typename F>
__device__ __forceinline__ void window_apply(f32x2 (&acc)[kItems][kX][kPairs], const F& profile,
                                             f32x2 wl2, f32x2 wr2) {
#pragma unroll
  for (int i = 0; i < kItems; ++i)
#pragma unroll
    for (int jj = 0; jj < kPairs; ++jj) {
      const f32x2 V = profile(i, jj);
      if constexpr (kM >= 0) acc[i][kM][jj] = fma2(wl2, V, acc[i][kM][jj]);
      if constexpr (kM + 1 < kX) acc[i][kM + 1][jj] = fma2(wr2, V, acc[i][kM + 1][jj]);
    }
}

// (kLo <= f0 < kHi: halves the candidates at each branch)
template <int kLo, int kHi, int kItems, int kX, int kPairs, typename F>
__device__ __forceinline__ void window_dispatch(f32x2 (&acc)[kItems][kX][kPairs], int f0,
                                                const F& profile, f32x2 wl2, f32x2 wr2) {
  if constexpr (kHi - kLo == 1) {
    window_apply<kItems, kX, kPairs, kLo>(acc, profile, wl2, wr2);
  } else {
    constexpr int kMid = kLo + (kHi - kLo) / 2;
    if (f0 < kMid)
      window_dispatch<kLo, kMid>(acc, f0, profile, wl2, wr2);
    else
      window_dispatch<kMid, kHi>(acc, f0, profile, wl2, wr2);
  }
}

// Tile (i, j) of linear block b of an ni x nj grid of tiles, run in patches of
// pi x pj tiles (i fastest inside a patch; only the last patches are smaller).
__device__ __forceinline__ void patch_tile(unsigned b, int ni, int nj, int pi, int pj, int& i,
                                           int& j) {
  const unsigned strip = unsigned(ni) * unsigned(pj);  // a full strip of patches
  const int s = int(b / strip);
  b -= unsigned(s) * strip;
  const int hj = min(pj, nj - s * pj);
  const int q = int(b / unsigned(pi * hj));
  b -= unsigned(q) * unsigned(pi * hj);
  const int wi = min(pi, ni - q * pi);
  i = q * pi + int(b % unsigned(wi));
  j = s * pj + int(b / unsigned(wi));
}

// ------------------------------------------------------------ FP tile order
// Tile (row block, column block, angle pair) of linear block b under s. The
// blocks of a group of pairs come first, inside a group the patches strip by
// strip, inside a patch the pairs and then the tiles with row blocks fastest.
// Only the last group, strip and patch can be smaller than the others, so
// each level's index is a plain quotient.
__device__ __forceinline__ void fp_schedule_tile(const FpSchedule& s, long long b, int& rb,
                                                 int& cb, int& pair) {
  const long long per_pair = (long long)s.row_blocks * s.col_blocks;
  const long long full_group = per_pair * s.group_pairs;
  const int grp = int(b / full_group);
  b -= grp * full_group;
  const int gsz = min(s.group_pairs, s.pairs - grp * s.group_pairs);
  const long long full_strip = (long long)gsz * s.patch_rows * s.col_blocks;
  const int pr = int(b / full_strip);
  b -= pr * full_strip;
  const int rsz = min(s.patch_rows, s.row_blocks - pr * s.patch_rows);
  const long long full_patch = (long long)gsz * rsz * s.patch_cols;
  const int pc = int(b / full_patch);
  b -= pc * full_patch;
  const int csz = min(s.patch_cols, s.col_blocks - pc * s.patch_cols);
  const long long tiles = (long long)rsz * csz;
  const long long q = b / tiles;
  pair = grp * s.group_pairs + int(q);
  const int t = int(b - q * tiles);
  rb = pr * s.patch_rows + t % rsz;
  cb = pc * s.patch_cols + t / rsz;
}

}  // namespace tsgb
