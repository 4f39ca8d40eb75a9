// Matched backprojection of separable angles with z-lane warps.
//
// The exact transpose of fp_ray_kernel for angles whose det_v runs along z
// (b = z: circular and helical cone and parallel scans), as bp_separable_kernel
// computes it, with the work laid out differently:
//
//  * The weighted sinogram is stored column-major: element (theta, iu, r) holds
//    the row pair (W y[v], W y[v+1]) of detector row v = r - kRowPad, rows
//    fastest (bp_weight_z_kernel). Padding pairs (v = -2, rows, rows + 1) and
//    the halves that fall off the detector are zero.
//  * A warp owns kX voxels along the in-plane axis a on one plane of the
//    dominant axis d, and 32 x kRun voxels along z: lane l holds z0 + l + 32 j
//    for j < kRun. On a plane, which detector columns reach a voxel and with
//    what in-plane weight depends only on its a-coordinate, so all 32 lanes
//    walk the same columns: the column loop is uniform (no divergence), and
//    each column's vertical profile V(z) is built once for the whole window
//    (kX + 1 voxel widths of columns per kX voxels). The columns come from a
//    list in shared memory that the lanes fill together, one entry each. The
//    lanes' row-pair loads of one column fall on about 23 consecutive rows: one
//    or two 128-byte lines per load.
//  * A column whose ray crosses the plane at q_a (window coordinates, floor f0,
//    fraction fa) adds (1 - fa) V to voxel f0 and fa V to voxel f0 + 1 (the
//    tents of the two voxels it lies between); a uniform branch on f0 picks the
//    accumulator registers.
//  * One launch runs both passes (angles whose in-plane axis is x, then y), each
//    into its own z-fastest scratch volume [y][x][z], so every store is a
//    coalesced 128-byte run and a small volume's passes fill the GPU together;
//    one tiled transpose (bp_zlane_out_kernel) then writes their sum to the
//    caller's [z][y][x] volume, setting, adding or applying the SIRT update.
//    Several stacked items (batched backprojection) share the launch.
//
// Measured (GB300; the matched backprojection, weight pass and transpose
// included): 512^3 / 1024 angles 92.0 ms, 256^3 / 360 4.14 ms (voxel-pair kernel 144
// and 6.5 ms). ncu at 256^3: 17 thread instructions per voxel-angle, issue, the
// FMA pipe and L1 each 65 % busy at 16 warps per SM (128 registers: 40 accumulators
// and two stages of loads), which bounds it: fixed-latency waits, 1.5 per issue.
//
// Arithmetic per (column, voxel) is bp_separable_kernel's: the two row tents
// of the fast path (|slope| >= 1 rows per voxel) as saturating adds from the
// exact row position, and the general row loop otherwise. Only the order in
// which each voxel's terms are summed differs (per angle, columns in order).
// Floors and float-to-int conversions of the inner loop avoid the conversion
// unit (see kFloorMagic), which a 512^3 profile showed half busy otherwise.
#include <cuda_runtime.h>

#include <algorithm>

#include "device_common.cuh"

namespace tsgb {
namespace {

constexpr float kMaxSlopeZ = 64.0f;  // must match fp.cu

// Plane step W of pixel (iv, iu) of an angle without column entries, 0 for rays the
// forward projector does not sample.
__device__ __forceinline__ float pixel_step_z(const AngleParams& ap, const DeviceGeometry& g,
                                              int iv, int iu) {
  const Ray r = ray_general(ap, float(iu - g.ou), float(iv - g.ov));
  const bool sampled =
      finite_ray(r) && fabsf(r.ma) <= kMaxSlopeZ && fabsf(r.mb) <= kMaxSlopeZ;
  return sampled ? ray_step(ap, r) : 0.0f;
}

// Column-major row-pair weighted sinogram. A block of 32 x 8 threads covers
// 32 detector columns x 32 padded pair rows of one angle: it computes the 33
// rows of W y it needs into shared memory (reads along u, coalesced), then
// writes the pairs along the rows (coalesced). Every padded pair is written,
// so the buffer needs no clearing. `out` points at the angle range's first
// column; blockIdx.z counts angles from `theta0`, over groups of kItems stacked
// sinograms: with kItems = 2 an element holds both items' pairs. (angles * groups
// fits 32 bits: an angle's tables take 256 bytes, and a batch's workspace is bounded.)
// DRAM bytes set its floor; what bounds it is issue (70-78 %) and the loads'
// latency, so each thread has 4 to 5 loads in flight and the column's part of W is
// taken out of the row loop (512^3 / 1024 angles 1.94 -> 1.26 ms, 0.72 at DRAM rate).
template <int kItems, bool kSpread>
__global__ void __launch_bounds__(256)
    bp_weight_z_kernel(const AngleParams* __restrict__ params,
                       const ColumnEntry* __restrict__ columns, SinoSource sino,
                       float2* __restrict__ out, long long group_pairs, DeviceGeometry g,
                       int theta0, int n_angles, int groups) {
  __shared__ float s[kItems][33][33];  // [item][row][column]
  const int iu0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int RP = g.rows + 2 * kRowPad;
  const int iu = iu0 + threadIdx.x;
  // the source's columns and elements between its rows (kSpread: a coarser detector)
  const int ys = kSpread ? int(source_pixel(sino, g.cols)) : g.cols;
  const size_t rs = (size_t)g.nangles * ys, item = rs * g.rows;
  for (unsigned b = blockIdx.z; b < unsigned(n_angles) * unsigned(groups); b += gridDim.z) {
    const unsigned group = groups == 1 ? 0 : b / unsigned(n_angles);
    const int n = int(b - group * unsigned(n_angles)), theta = theta0 + n;
    const AngleParams& ap = params[theta];
    {
      const int iv0 = r0 + int(threadIdx.y) - kRowPad;
      const float* y = sino.y + (size_t)group * kItems * item + (size_t)theta * ys +
                       (kSpread ? int(source_pixel(sino, iu)) : iu);
      if (!kSpread) y += (long long)iv0 * (long long)rs;
      float v[5][kItems];  // rows threadIdx.y + 8 q; the 33rd is the first warp's
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        const int iv = iv0 + 8 * q;
        const bool in = iu < g.cols && iv >= 0 && iv < g.rows && (q < 4 || threadIdx.y == 0);
        const size_t row = kSpread ? source_pixel(sino, iv) * rs : q * (8 * rs);
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
          const float x = in ? __ldg(y + i * item + row) : 0.0f;
          v[q][i] = kSpread ? sino.scale * x : x;
        }
      }
      const bool separable = ap.separable;
      ColumnEntry ce{};
      if (separable && iu < g.cols) ce = columns[(size_t)theta * g.cols + iu];
      const float vd = ap.vs_d, va = ap.vs_a * ce.ma, vs_b = ap.vs_b;
      const float vt0 = float(iv0 - g.ov);
      const bool column_sampled = isfinite(ce.Xa) && fabsf(ce.ma) <= kMaxSlopeZ;
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        if (q == 4 && threadIdx.y != 0) break;
        float W = 1.0f;
        if (separable) {  // as ray_column and ray_step, the column's part taken out
          const float vt = vt0 + float(8 * q);
          const float Xb = fmaf(vt, ce.R, ce.P), mb = fmaf(vt, ce.S, ce.Q), vb = vs_b * mb;
          W = sqrtf(fmaf(vd, vd, fmaf(va, va, vb * vb)));
          if (!column_sampled || !isfinite(Xb) || !(fabsf(mb) <= kMaxSlopeZ)) W = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kItems; ++i) s[i][threadIdx.y + 8 * q][threadIdx.x] = W * v[q][i];
      }
      if (!separable) {
#pragma unroll 1
        for (int k = threadIdx.y; k < 33; k += 8) {
          const float W = pixel_step_z(ap, g, r0 + k - kRowPad, iu);
#pragma unroll
          for (int i = 0; i < kItems; ++i) s[i][k][threadIdx.x] *= W;
        }
      }
    }
    __syncthreads();
    const int r = r0 + threadIdx.x, c0 = iu0 + int(threadIdx.y);
    float2* o = out + group * group_pairs + (((size_t)n * g.cols + c0) * RP + r) * kItems;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = int(threadIdx.y) + 8 * q;
      if (c0 + 8 * q >= g.cols || r >= RP) break;
      float2 v[kItems];
#pragma unroll
      for (int i = 0; i < kItems; ++i)
        v[i] = make_float2(s[i][threadIdx.x][c], s[i][threadIdx.x + 1][c]);
      if constexpr (kItems == 2)
        *reinterpret_cast<float4*>(o) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
      else
        *o = v[0];
      o += (size_t)(8 * kItems) * RP;
    }
    __syncthreads();
  }
}

// The row pairs of the kItems items at one element.
template <int kItems>
__device__ __forceinline__ void load_rows(const char* p, float2 (&y)[kItems]) {
  if constexpr (kItems == 2) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    y[0] = make_float2(v.x, v.y);
    y[1] = make_float2(v.z, v.w);
  } else {
    y[0] = __ldg(reinterpret_cast<const float2*>(p));
  }
}

// The columns of a list whose rows are at least a voxel apart (|Sl| >= 1).
// Row pair v0 = floor((z - B) / Sl) and v0 + 1 (tent half-width 1/|Sl| <= 1
// row). For voxel z: row v0's ray crosses the plane at t0 = v0 Sl + B - z from
// it, row v0+1's at t0 + Sl, so the tents are max(0, 1 - |t0|) and
// max(0, 1 - |Sl| + |t0|) (both at most 1: saturating adds). kClamp: rows are
// clamped to [vmin, vmax] (integers; NaN -> vmin), which clamps their floor;
// else every row is known to lie inside.
//
// A column's loads are issued before the column before it is added (stage,
// then finish), two stages of registers: without it a quarter of the warps'
// time was waiting for L1 and L2 at 256^3 (5.2 -> 4.6 ms per backprojection,
// although fewer warps fit). 16 voxels per lane leave no registers for this
// (116 ms at 512^3 / 1024 angles, against 100 ms for two ranges of 8).
template <bool kClamp, int kRun, int kItems, int kX>
__device__ __forceinline__ void zlane_columns(f32x2 (&acc)[kItems][kX][(kRun + 1) / 2],
                                              const float4 (&list)[34][4], int n, float zt,
                                              float vmin, float vmax) {
  constexpr int kPairs = (kRun + 1) / 2;
  constexpr size_t kElem = sizeof(float2) * kItems;
  struct Stage {
    f32x2 t[kPairs];
    float2 ya[kPairs][kItems], yb[kPairs][kItems];
  } st[2];
  const auto stage = [&](Stage& S, const float4(&entry)[4]) {
    const float4 e0 = entry[0], e1 = entry[1];
    const f32x2 Sl2 = pack2(e0.x, e0.y), Bl2 = pack2(e0.z, e0.w);
    const char* colb = reinterpret_cast<const char*>(
        size_t(__float_as_uint(e1.z)) | (size_t(__float_as_uint(e1.w)) << 32));
    const float C0 = e1.y - zt, vs0 = -C0 * e1.x, dv = 32.0f * e1.x;
#pragma unroll
    for (int jj = 0; jj < kPairs; ++jj) {
      // (an odd run's last pair repeats its voxel: the second half is not stored)
      const int ja = 2 * jj, jb = 2 * jj + 1 < kRun ? 2 * jj + 1 : 2 * jj;
      float ta = fmaf(float(ja), dv, vs0), tb = fmaf(float(jb), dv, vs0);
      if (kClamp) {
        ta = fminf(fmaxf(ta, vmin), vmax);
        tb = fminf(fmaxf(tb, vmin), vmax);
      }
      const f32x2 f = add2_rd(pack2(ta, tb), pack2(kFloorMagic, kFloorMagic));
      const f32x2 v0 = add2(f, pack2(-kFloorMagic, -kFloorMagic));
      S.t[jj] = add2(fma2(v0, Sl2, pack2(C0 - float(32 * ja), C0 - float(32 * jb))), Bl2);
      float fa, fb;
      unpack2(f, fa, fb);
      load_rows(colb + size_t(__float_as_uint(fa)) * kElem, S.ya[jj]);
      load_rows(colb + size_t(__float_as_uint(fb)) * kElem, S.yb[jj]);
    }
  };
  const auto finish = [&](const Stage& S, const float4(&entry)[4]) {
    const float4 e2 = entry[2];
    const float2 e3 = *reinterpret_cast<const float2*>(&entry[3]);
    f32x2 V[kItems][kPairs];
#pragma unroll
    for (int jj = 0; jj < kPairs; ++jj) {
      float ta, tb;
      unpack2(S.t[jj], ta, tb);
      ta = fabsf(ta);
      tb = fabsf(tb);
      const float wa0 = __saturatef(1.0f - ta), wa1 = __saturatef(e3.y + ta);
      const float wb0 = __saturatef(1.0f - tb), wb1 = __saturatef(e3.y + tb);
#pragma unroll
      for (int i = 0; i < kItems; ++i)
        V[i][jj] = pack2(fmaf(wa0, S.ya[jj][i].x, __fmul_rn(wa1, S.ya[jj][i].y)),
                         fmaf(wb0, S.yb[jj][i].x, __fmul_rn(wb1, S.yb[jj][i].y)));
    }
    const auto profile = [&](int i, int jj) { return V[i][jj]; };
    window_dispatch<-1, kX>(acc, __float_as_int(e3.x), profile, pack2(e2.x, e2.y),
                            pack2(e2.z, e2.w));
  };
  if (n == 0) return;
  const float4(*entry)[4] = list;
  stage(st[0], entry[0]);
  for (int k = 0; k < n; k += 2, entry += 2) {
    stage(st[1], entry[1]);
    finish(st[0], entry[0]);
    if (k + 1 < n) {
      stage(st[0], entry[2]);
      finish(st[1], entry[1]);
    }
  }
}

// The columns of a list with rows at least half a voxel apart (|Sl| >= 0.5), some
// less than one: a tent (half-width 1/|Sl| <= 2 rows) covers at most the four rows
// above its lower end. Row v0 (the one at or below that end) crosses the plane at t0
// = v0 Sl + B - z from voxel z, the four at t0 + Sl .. t0 + 4 Sl: two row-pair loads,
// each row weighted by its exact tent and added in increasing order (rows of weight 0
// add nothing). v0 is clamped so that both pairs lie in the padded column (rows off
// the detector hold zeros; a clamped window still covers the detector rows of the
// true one; NaN clamps to the low end). Loads a column ahead where the registers
// hold two stages (2 x 2 supersampled 128 x 160 x 160 / 200: 2.21 -> 1.95 ms per
// backprojection).
template <int kRun, int kItems, int kX>
__device__ __forceinline__ void zlane_fine_columns(f32x2 (&acc)[kItems][kX][(kRun + 1) / 2],
                                                   const float4 (&list)[34][4], int n, float zt,
                                                   float vmin, float vmax) {
  constexpr int kPairs = (kRun + 1) / 2, kN = 2 * kPairs;
  constexpr int kStages = kRun * kItems <= 4 ? 2 : 1;
  constexpr size_t kElem = sizeof(float2) * kItems;
  struct Stage {
    float t[kN];
    float2 y01[kN][kItems], y23[kN][kItems];
  } st[kStages];
  const auto stage = [&](Stage& S, const float4(&entry)[4]) {
    const float4 e0 = entry[0], e1 = entry[1];
    const char* colb = reinterpret_cast<const char*>(
        size_t(__float_as_uint(e1.z)) | (size_t(__float_as_uint(e1.w)) << 32));
    const float C0 = e1.y - zt, dv = 32.0f * e1.x;
    const float vs0 = fmaf(-C0, e1.x, -fabsf(e1.x));  // lower end of the tent of j = 0
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      const float t = fminf(fmaxf(fmaf(float(j), dv, vs0), vmin - 1.0f), vmax - 2.0f);
      const float f = __fadd_rd(t, kFloorMagic);
      const char* p = colb + size_t(__float_as_uint(f) + 1u) * kElem;
      S.t[j] = fmaf(f - kFloorMagic, e0.x, C0 - float(32 * j)) + e0.z;
      load_rows(p, S.y01[j]);
      load_rows(p + 2 * kElem, S.y23[j]);
    }
  };
  const auto finish = [&](const Stage& S, const float4(&entry)[4]) {
    const float Sl = entry[0].x;
    const float4 e2 = entry[2];
    const float f0 = entry[3].x;
    f32x2 V[kItems][kPairs];
#pragma unroll
    for (int jj = 0; jj < kPairs; ++jj) {
      float v[kItems][2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = 2 * jj + h;
        const float w0 = __saturatef(1.0f - fabsf(S.t[j] + Sl));
        const float w1 = __saturatef(1.0f - fabsf(fmaf(2.0f, Sl, S.t[j])));
        const float w2 = __saturatef(1.0f - fabsf(fmaf(3.0f, Sl, S.t[j])));
        const float w3 = __saturatef(1.0f - fabsf(fmaf(4.0f, Sl, S.t[j])));
#pragma unroll
        for (int i = 0; i < kItems; ++i)
          v[i][h] = fmaf(w3, S.y23[j][i].y,
                         fmaf(w2, S.y23[j][i].x,
                              fmaf(w1, S.y01[j][i].y, __fmul_rn(w0, S.y01[j][i].x))));
      }
#pragma unroll
      for (int i = 0; i < kItems; ++i) V[i][jj] = pack2(v[i][0], v[i][1]);
    }
    const auto profile = [&](int i, int jj) { return V[i][jj]; };
    window_dispatch<-1, kX>(acc, __float_as_int(f0), profile, pack2(e2.x, e2.y),
                            pack2(e2.z, e2.w));
  };
  if (n == 0) return;
  if constexpr (kStages == 1) {
    for (int k = 0; k < n; ++k) {
      stage(st[0], list[k]);
      finish(st[0], list[k]);
    }
  } else {
    const float4(*entry)[4] = list;
    stage(st[0], entry[0]);
    for (int k = 0; k < n; k += 2, entry += 2) {
      stage(st[1], entry[1]);
      finish(st[0], entry[0]);
      if (k + 1 < n) {
        stage(st[0], entry[2]);
        finish(st[1], entry[1]);
      }
    }
  }
}

// The columns of a list with rows less than half a voxel apart among them: every row
// whose tent reaches the voxel. The profile is built before the window's branch: inside
// it every branch held the row loops of all the lane's voxels (128 x 192^2 /
// 180 cone angles, 500 rows: 20.2 ms, now 7.2; the voxel-pair kernel 11.8).
// Scans without such rows (kHalfRows false; they get here with NaN row steps only) keep
// it inside where a lane holds 7 or 8 voxels: the compiler then schedules the common loop
// 1.3 % faster (256^3 / 360 angles 4.15 ms against 4.21).
template <bool kHalfRows, int kRun, int kItems, int kX>
__device__ __forceinline__ void zlane_any_columns(f32x2 (&acc)[kItems][kX][(kRun + 1) / 2],
                                                  const float4 (&list)[34][4], int n, float zt,
                                                  const DeviceGeometry& g) {
  constexpr int kPairs = (kRun + 1) / 2;
  for (int k = 0; k < n; ++k) {
    const float4 e0 = list[k][0], e1 = list[k][1], e2 = list[k][2], e3 = list[k][3];
    const float Sl = e0.x, inv = e1.x, C0 = (e1.y - zt) + e0.z;
    const float2* col = reinterpret_cast<const float2*>(  // anchored row 0
        (size_t(__float_as_uint(e1.z)) | (size_t(__float_as_uint(e1.w)) << 32)) +
        size_t(kFloorBits) * sizeof(float2) * kItems);
    const auto rows = [&](int i, int j) {
      const float Bj = C0 - float(32 * j);
      const float v1 = (-1.0f - Bj) * inv, v2 = (1.0f - Bj) * inv;
      const int iv_lo = max(0, (int)floorf(clamp_coord(fminf(v1, v2))) + g.ov);
      const int iv_hi = min(g.rows - 1, (int)ceilf(clamp_coord(fmaxf(v1, v2))) + g.ov);
      float V = 0.0f;
      for (int iv = iv_lo; iv <= iv_hi; ++iv)
        V = fmaf(tent(fmaf(float(iv - g.ov), Sl, Bj)), __ldg(col + (iv - g.ov) * kItems + i).x, V);
      return V;
    };
    const auto add = [&](const auto& profile) {
      window_dispatch<-1, kX>(acc, __float_as_int(e3.x), profile, pack2(e2.x, e2.y),
                              pack2(e2.z, e2.w));
    };
    if constexpr (kHalfRows || kRun < 7) {
      f32x2 V[kItems][kPairs];
#pragma unroll
      for (int i = 0; i < kItems; ++i)
#pragma unroll
        for (int jj = 0; jj < kPairs; ++jj)
          V[i][jj] = pack2(rows(i, 2 * jj), 2 * jj + 1 < kRun ? rows(i, 2 * jj + 1) : 0.0f);
      add([&](int i, int jj) { return V[i][jj]; });
    } else {
      add([&](int i, int jj) { return pack2(rows(i, 2 * jj), rows(i, 2 * jj + 1)); });
    }
  }
}

// One launch of the z-lane kernel: both passes (angles whose in-plane axis is
// x, then y) over `items` stacked sinograms.
struct ZlaneArgs {
  const SolveEntry* solve[2];  // pass 0: a = x, pass 1: a = y
  int n[2];                    // angles per pass
  int plane_blocks[2];
  unsigned blocks0;            // blocks of pass 0
  const ColumnEntry* columns;
  const float2* sinoz;         // column-major row pairs
  float* volt[2];              // [y][x][z] sum of each pass, z rows zs apart
  long long group_pairs, item_volt;  // strides: blockIdx.z (pairs), item (floats)
  int zs;
  DeviceGeometry g;
  bool half_rows;  // the projector's: which instantiation runs
};

// Block: kPlanes warps on adjacent planes of the dominant axis, same window of
// kX voxels along a and same z range. blockIdx.x = window * plane_blocks +
// plane block (pass 0 first, then pass 1), blockIdx.y = z range, blockIdx.z =
// item.
//
// What depends only on the angle or the detector column is computed with one
// lane per angle or column instead of by all lanes alike: 32 angles' column
// ranges at a time, then the ranges flattened into a list and each list entry's
// table entry, window position, row step and address by its own lane, kept in
// shared memory (a column is then three 16-byte broadcast reads and an 8-byte one). With
// all lanes alike this was 30 instructions per angle and 25 per column, which a run of
// few voxels along z does not hide.
//
// kItems = 2: a warp works on two stacked items at once (float4 elements): they share
// the columns, rows and weights, and an item then costs a multiply and three
// multiply-adds per voxel and column instead of the whole profile.
template <int kX, int kRun, int kPlanes, int kMinBlocks, int kItems, bool kHalfRows>
__global__ void __launch_bounds__(32 * kPlanes, kMinBlocks)
    bp_zlane_kernel(const __grid_constant__ ZlaneArgs A) {
  constexpr int kPairs = (kRun + 1) / 2;
  __shared__ float4 s_list[kPlanes][34][4];
  const DeviceGeometry& g = A.g;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int pass = blockIdx.x < A.blocks0 ? 0 : 1;
  const unsigned block = blockIdx.x - (pass ? A.blocks0 : 0u);
  const int n_p = pass ? g.nx : g.ny, n_a = pass ? g.ny : g.nx;
  const int ip = int(block % unsigned(A.plane_blocks[pass])) * kPlanes + w;  // plane (along d)
  const int i0 = int(block / unsigned(A.plane_blocks[pass])) * kX;          // window start (along a)
  if (ip >= n_p) return;  // whole warp (the block has no barriers)
  const int z0 = blockIdx.y * (32 * kRun) + lane;
  const float kt = float(ip - (pass ? g.ox : g.oy));
  const float i0t = float(i0 - (pass ? g.oy : g.ox));
  const float zt = float(z0 - g.oz), zw0 = float(int(blockIdx.y) * (32 * kRun) - g.oz);
  const int RP = g.rows + 2 * kRowPad;
  const float vmin = float(-kRowPad - g.ov), vmax = float(g.rows - g.ov);
  const int n_angles = A.n[pass];
  const float4* __restrict__ solve = reinterpret_cast<const float4*>(A.solve[pass]);
  const float4* __restrict__ col4 = reinterpret_cast<const float4*>(A.columns);
  const char* sino0 = reinterpret_cast<const char*>(A.sinoz + blockIdx.z * A.group_pairs +
                                                    (kRowPad + g.ov) * kItems);
  f32x2 acc[kItems][kX][kPairs];
#pragma unroll
  for (int i = 0; i < kItems; ++i)
#pragma unroll
    for (int m = 0; m < kX; ++m)
#pragma unroll
      for (int j = 0; j < kPairs; ++j) acc[i][m][j] = 0ull;

  for (int n0 = 0; n0 < n_angles; n0 += 32) {
    const ColumnRanges cr = column_ranges(solve, n0 + lane, n_angles, kt, i0t - 1.0f,
                                          i0t + float(kX), g);
    for (int t0 = 0; t0 < cr.total; t0 += 32) {
      const int t = t0 + lane;
      int iu, th;
      column_of(cr, t, iu, th);
      bool ok = t < cr.total;
      float4 e0, e1, e2, e3;
      int path = 0;
      if (ok) {
        const size_t ci = (size_t)th * g.cols + iu;
        const float4 c0 = __ldg(col4 + 2 * ci);      // Xa, ma, P, Q
        const float4 c1 = __ldg(col4 + 2 * ci + 1);  // R, S, -, -
        const float qa = fmaf(kt, c0.y, c0.x) - i0t;
        ok = qa > -1.0f && qa < float(kX);  // (NaN: no)
        const float fq = __fadd_rd(qa, kFloorMagic);
        const float fa = qa - (fq - kFloorMagic), wl = 1.0f - fa;
        // On this plane, q_b(vt) = B + vt * Sl; voxel z's rows lie near
        // (z - B) / Sl. A row v0 = floor(t) comes as kFloorMagic-biased bits: its
        // pair's address is the entry's (column minus kFloorBits pairs, 64-bit
        // wrap-around) + bits * 8.
        const float B = fmaf(kt, c0.w, c0.z), Sl = fmaf(kt, c1.y, c1.x);
        const float inv = __frcp_rn(Sl), aSl = fabsf(Sl);
        // rows are monotone in z: if the warp's first and last voxel (beyond the
        // volume's end too) select rows well inside [vmin, vmax], every voxel
        // does; else (NaN too) the path that clamps them
        const float ra = (zw0 - B) * inv, rb = (zw0 + float(32 * kRun - 1) - B) * inv;
        const float margin = fmaf(4e-7f, fabsf(ra) + fabsf(rb), 0.01f);
        const bool inside = fminf(ra, rb) >= vmin + margin && fmaxf(ra, rb) < vmax + 1.0f - margin;
        path = aSl >= 1.0f ? (inside ? 0 : 1) : aSl >= 0.5f ? 2 : 3;
        const size_t colb = reinterpret_cast<size_t>(sino0) +
                            (ci * RP - size_t(kFloorBits)) * sizeof(float2) * kItems;
        // B as a multiple of 2^-14 plus a remainder, so that B - z is exact
        const float Bh = (B + 768.0f) - 768.0f, Bl = B - Bh;
        e0 = make_float4(Sl, Sl, Bl, Bl);
        e1 = make_float4(inv, Bh, __uint_as_float(unsigned(colb)),
                         __uint_as_float(unsigned(colb >> 32)));
        e2 = make_float4(wl, wl, fa, fa);
        e3 = make_float4(__int_as_float(int(__float_as_uint(fq) - kFloorBits)), 1.0f - aSl,
                         __int_as_float(path), 0.0f);
      }
      const unsigned mask = __ballot_sync(0xffffffffu, ok);
      const int paths = __reduce_max_sync(0xffffffffu, ok ? path : 0);
      if (ok) {
        const int slot = __popc(mask & ((1u << lane) - 1u));
        s_list[w][slot][0] = e0;
        s_list[w][slot][1] = e1;
        s_list[w][slot][2] = e2;
        s_list[w][slot][3] = e3;
        if ((mask >> lane) == 1u) {  // the last: loads a column ahead find it again
          s_list[w][slot + 1][0] = s_list[w][slot + 2][0] = e0;
          s_list[w][slot + 1][1] = s_list[w][slot + 2][1] = e1;
        }
      }
      __syncwarp();
      const int columns_in = __popc(mask);
      if (paths == 0)
        zlane_columns<false, kRun>(acc, s_list[w], columns_in, zt, vmin, vmax);
      else if (paths == 1)
        zlane_columns<true, kRun>(acc, s_list[w], columns_in, zt, vmin, vmax);
      else if (paths == 2)
        zlane_fine_columns<kRun>(acc, s_list[w], columns_in, zt, vmin, vmax);
      else
        zlane_any_columns<kHalfRows, kRun>(acc, s_list[w], columns_in, zt, g);
      __syncwarp();  // the list is rewritten
    }
  }
  // [y][x][z] scratch: lanes along z, coalesced
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    float* __restrict__ volt = A.volt[pass] + (blockIdx.z * kItems + i) * A.item_volt;
#pragma unroll
    for (int m = 0; m < kX; ++m) {
      const int ia = i0 + m;
      if (ia >= n_a) break;
      float* out = volt + (pass ? (size_t)ia * g.nx + ip : (size_t)ip * g.nx + ia) * A.zs;
#pragma unroll
      for (int jj = 0; jj < kPairs; ++jj) {
        float va, vb;
        unpack2(acc[i][m][jj], va, vb);
        const int z = z0 + 64 * jj;
        if (z < g.nz) out[z] = va;
        if (2 * jj + 1 < kRun && z + 32 < g.nz) out[z + 32] = vb;
      }
    }
  }
}

// Epilogues of the transpose from the [y][x][z] scratch to the caller's volume.
enum ZlaneOut { kOutSet = 0, kOutAdd = 1, kOutSirt = 2 };

// vol[z][y][x] (=, +=) volt[y][x][z], or the SIRT update vol += C * volt with
// the plain recipe's rounding. volt is the sum of both passes' scratch volumes
// (volt1 may be null). 32 x 32 tiles of the (x, z) plane of one y through
// shared memory: reads along z and writes along x are both coalesced.
// The scratch volumes hold the slices first_z .. first_z + n_z - 1 (the others' sums
// are 0). blockIdx.x = item * z tiles + z tile.
template <int kOut>
__global__ void __launch_bounds__(256)
    bp_zlane_out_kernel(const float* __restrict__ volt0, const float* __restrict__ volt1,
                        long long item_volt, int zs, int first_z, int n_z,
                        float* __restrict__ vol, const float* __restrict__ C, DeviceGeometry g) {
  __shared__ float tile[32][33];  // [x][z]
  const int z_tiles = (g.nz + 31) / 32, item = blockIdx.x / z_tiles;
  const int z0 = (blockIdx.x - item * z_tiles) * 32, x0 = blockIdx.y * 32;
  volt0 += item * item_volt;
  if (volt1) volt1 += item * item_volt;
  vol += (size_t)item * g.nz * g.ny * g.nx;
  for (int y = blockIdx.z; y < g.ny; y += gridDim.z) {
    float v[4], v1[4], old[4], c[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = x0 + int(threadIdx.y) + 8 * q, z = z0 + int(threadIdx.x) - first_z;
      const size_t i = ((size_t)y * g.nx + x) * zs + z;
      const bool in = x < g.nx && z >= 0 && z < n_z;
      v[q] = in ? volt0[i] : 0.0f;
      v1[q] = in && volt1 ? volt1[i] : 0.0f;
    }
    if (kOut != kOutSet) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int z = z0 + int(threadIdx.y) + 8 * q, x = x0 + threadIdx.x;
        const size_t idx = ((size_t)z * g.ny + y) * g.nx + x;
        const bool in = x < g.nx && z < g.nz;
        old[q] = in ? vol[idx] : 0.0f;
        c[q] = kOut == kOutSirt && in ? __ldg(C + idx) : 0.0f;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      tile[threadIdx.y + 8 * q][threadIdx.x] = volt1 ? __fadd_rn(v[q], v1[q]) : v[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int z = z0 + int(threadIdx.y) + 8 * q, x = x0 + threadIdx.x;
      if (x >= g.nx || z >= g.nz) break;
      const float s = tile[threadIdx.x][threadIdx.y + 8 * q];
      vol[((size_t)z * g.ny + y) * g.nx + x] =
          kOut == kOutSet   ? s
          : kOut == kOutAdd ? __fadd_rn(old[q], s)
                            : __fadd_rn(old[q], __fmul_rn(s, c[q]));
    }
    __syncthreads();
  }
}

template <int kX, int kRun, int kPlanes, int kMinBlocks, int kItems = 1>
void launch_zlane_shape(ZlaneArgs& A, int groups, cudaStream_t stream) {
  const DeviceGeometry& g = A.g;
  unsigned blocks[2];
  for (int pass = 0; pass < 2; ++pass) {
    const int n_p = pass ? g.nx : g.ny, n_a = pass ? g.ny : g.nx;
    A.plane_blocks[pass] = (n_p + kPlanes - 1) / kPlanes;
    blocks[pass] = A.n[pass] > 0 ? unsigned(A.plane_blocks[pass]) * unsigned((n_a + kX - 1) / kX) : 0u;
  }
  A.blocks0 = blocks[0];
  const dim3 grid(blocks[0] + blocks[1], unsigned((g.nz + 32 * kRun - 1) / (32 * kRun)),
                  unsigned(groups));
  const auto kernel = kRun < 7 || A.half_rows
                          ? bp_zlane_kernel<kX, kRun, kPlanes, kMinBlocks, kItems, true>
                          : bp_zlane_kernel<kX, kRun, kPlanes, kMinBlocks, kItems, kRun < 7>;
  kernel<<<grid, 32 * kPlanes, 0, stream>>>(A);
}

// Warp shapes, by the voxels along z per lane (`run`, from the volume's nz: at
// most 8, ranges of near-equal length along z). Wider windows share a column's
// profile between more voxels ((kX + 1) / kX columns per voxel), as long as the
// accumulators and the two load stages fit the registers. Measured (GB300, window x
// warps per block; runs 3, 4, 6 and 8 when each was chosen, before later steps that
// serve all windows alike):
//   run 8, 512^3 / 1024 angles: 5 x 8 94.0 ms, 4 x 8 95.5, 3 x 8 101.0, 6 x 8 over 100
//   run 7, 224 x 224^2 / 200: 5 x 8 2.39 ms, 6 x 8 2.34, 4 x 8 2.41, 3 x 8 2.76;
//          224 x 100^2 / 120: 0.364 ms, 0.392, 0.395, 0.399
//   run 6, helical 170 x 190 x 181 / 257, forward projection included: 6 x 4 2.76 ms,
//          5 x 4 2.80, 4 x 4 2.88
//   run 5, 160 x 160^2 / 200: 6 x 4 1.02 ms, 5 x 4 1.07, 4 x 4 1.01, 8 x 4 1.01;
//          160 x 96^2 / 120: 0.284 ms, 0.273, 0.252, 0.235
//   run 4, 128^3 / 200: 6 x 4 0.407 ms, 8 x 4 0.431; 8 x 128^3: all within 2 %
//   run 3, SIRT at 96^3: 8 x 4 1.61 ms, 4 x 4 1.66, 6 x 4 1.71
//   run 2, 64^3 / 96: 4 x 8 66 us, 3 x 8 73, 6 x 8 87, 8 x 8 89; 64 x 192^2 / 180:
//          657 us, 675, 640, 617
//   run 1, 32 x 64^2 / 96: 4 x 8 64 us, 3 x 8 70, 6 x 8 83, 8 x 8 83; 32 x 192^2 / 180:
//          643 us, 659, 621, 600
// The tuning's bp_shape 3 and 4 force other windows for run 8, 5 and 6 cap the run at 4
// and 2; any other value takes this rule.
int zlane_run(const tsgb_projector* p) {
  const int shape = zlane_shape(p);
  const int most = shape == 5 ? 4 : shape == 6 ? 2 : 8;
  const int lanes = (p->g.nz + 31) / 32, ranges = (lanes + most - 1) / most;
  return (lanes + ranges - 1) / ranges;
}

void launch_zlane_passes(const tsgb_projector* p, ZlaneArgs& A, int items, cudaStream_t stream) {
  const int shape = zlane_shape(p);
  switch (zlane_run(p)) {
    case 1: return launch_zlane_shape<4, 1, 8, 4>(A, items, stream);
    case 2: return launch_zlane_shape<4, 2, 8, 4>(A, items, stream);
    case 3: return launch_zlane_shape<8, 3, 4, 4>(A, items, stream);
    case 4: return launch_zlane_shape<6, 4, 4, 5>(A, items, stream);
    case 5: return launch_zlane_shape<6, 5, 4, 4>(A, items, stream);
    case 6: return launch_zlane_shape<6, 6, 4, 4>(A, items, stream);
    case 7: return launch_zlane_shape<5, 7, 8, 2>(A, items, stream);
    default:
      if (shape == 3) return launch_zlane_shape<4, 8, 16, 1>(A, items, stream);
      if (shape == 4) return launch_zlane_shape<3, 8, 8, 2>(A, items, stream);
      return launch_zlane_shape<5, 8, 8, 2>(A, items, stream);
  }
}

// Two items per warp, where the registers hold both (runs of at most 4). The windows
// are those of launch_zlane_passes: which columns share a list decides how rows of
// about a voxel are summed, so other windows would round differently from an item
// alone. 8 x 128^3 / 128 angles: 1.70 -> 1.05 ms.
constexpr int kTwoItemRun = 4;

void launch_zlane_two(const tsgb_projector* p, ZlaneArgs& A, int groups, cudaStream_t stream) {
  switch (zlane_run(p)) {
    case 1: return launch_zlane_shape<4, 1, 8, 3, 2>(A, groups, stream);
    case 2: return launch_zlane_shape<4, 2, 8, 3, 2>(A, groups, stream);
    case 3: return launch_zlane_shape<8, 3, 4, 3, 2>(A, groups, stream);
    default: return launch_zlane_shape<6, 4, 4, 4, 2>(A, groups, stream);
  }
}

// A launch over both angle lists of p (offsets into p->d_sep_angles), without its
// sinogram and scratch volumes.
ZlaneArgs zlane_args(const tsgb_projector* p, int off_x, int n_ax, int off_y, int n_ay) {
  ZlaneArgs A{};
  A.solve[0] = p->d_solve + off_x;
  A.solve[1] = p->d_solve + off_y;
  A.n[0] = n_ax;
  A.n[1] = n_ay;
  A.columns = p->d_columns;
  A.zs = p->g.nz;
  A.g = p->g;
  A.half_rows = p->half_rows;
  return A;
}

template <int kItems>
void launch_weights(const tsgb_projector* p, SinoSource sino, float2* out, long long group_pairs,
                    int angle_begin, int n_angles, int groups, cudaStream_t stream) {
  const DeviceGeometry& g = p->g;
  const int RP = g.rows + 2 * kRowPad;
  const dim3 grid(unsigned((g.cols + 31) / 32), unsigned((RP + 31) / 32),
                  unsigned(std::min<long long>((long long)n_angles * groups, 65535)));
  if (kItems == 1 && sino.d > 1)
    bp_weight_z_kernel<1, true><<<grid, dim3(32, 8), 0, stream>>>(
        p->d_params, p->d_columns, sino, out, group_pairs, g, angle_begin, n_angles, groups);
  else
    bp_weight_z_kernel<kItems, false><<<grid, dim3(32, 8), 0, stream>>>(
        p->d_params, p->d_columns, sino, out, group_pairs, g, angle_begin, n_angles, groups);
}

}  // namespace

void launch_zlane_out(const DeviceGeometry& g, int mode, const float* volt0, const float* volt1,
                      long long item_volt, int zs, int first_z, int n_z, float* vol,
                      const float* C, int items, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const dim3 grid(unsigned((g.nz + 31) / 32) * items, unsigned((g.nx + 31) / 32),
                  unsigned(std::min(g.ny, 65535)));
  const dim3 block(32, 8);
  if (mode == kOutSet)
    bp_zlane_out_kernel<kOutSet><<<grid, block, 0, stream>>>(volt0, volt1, item_volt, zs, first_z,
                                                             n_z, vol, C, g);
  else if (mode == kOutAdd)
    bp_zlane_out_kernel<kOutAdd><<<grid, block, 0, stream>>>(volt0, volt1, item_volt, zs, first_z,
                                                             n_z, vol, C, g);
  else
    bp_zlane_out_kernel<kOutSirt><<<grid, block, 0, stream>>>(volt0, volt1, item_volt, zs, first_z,
                                                              n_z, vol, C, g);
}

int64_t bp_pairs_bytes(const DeviceGeometry& g) {
  return (int64_t(g.rows + 2 * kRowPad) * g.nangles * g.cols * 8 + 255) / 256 * 256;
}

int64_t bp_volume_bytes(const DeviceGeometry& g) {
  return (int64_t(g.nz) * g.ny * g.nx * 4 + 255) / 256 * 256;
}

int64_t bp_scratch_bytes(const tsgb_projector* p) {
  return bp_scratch_volumes(p) * bp_volume_bytes(p->g);
}

int launch_bp_weight_z(const tsgb_projector* p, SinoSource sino, float* sinoz,
                       int angle_begin, int angle_end, void* stream) {
  const DeviceGeometry& g = p->g;
  float2* out = reinterpret_cast<float2*>(sinoz) +
                (size_t)angle_begin * g.cols * (g.rows + 2 * kRowPad);
  if (angle_end > angle_begin)
    launch_weights<1>(p, sino, out, 0, angle_begin, angle_end - angle_begin, 1,
                      static_cast<cudaStream_t>(stream));
  return int(cudaGetLastError());
}

bool launch_bp_zlane_separable(const tsgb_projector* p, int off_x, int n_ax, int off_y, int n_ay,
                               const float* sinoz, float* volt, float* vol, int out_mode,
                               const float* C, void* stream) {
  if (n_ax + n_ay == 0) return false;
  ZlaneArgs A = zlane_args(p, off_x, n_ax, off_y, n_ay);
  A.sinoz = reinterpret_cast<const float2*>(sinoz);
  // each pass has its own scratch volume; the transpose adds them
  A.volt[0] = volt;
  A.volt[1] = n_ax > 0 ? volt + bp_volume_bytes(p->g) / 4 : volt;
  launch_zlane_passes(p, A, 1, static_cast<cudaStream_t>(stream));
  launch_zlane_out(p->g, out_mode, volt, n_ax > 0 && n_ay > 0 ? A.volt[1] : nullptr, 0, A.zs, 0,
                   p->g.nz, vol, C, 1, stream);
  return true;
}

int launch_bp_zlane_batch(const tsgb_projector* p, float* vol, const float* sino, int items,
                          bool additive, char* workspace, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const DeviceGeometry& g = p->g;
  const int n_ax = p->n_sep_ax, n_ay = p->n_separable_bp - n_ax;
  const size_t sino_floats = size_t(g.rows) * g.nangles * g.cols;
  const long long pairs = bp_pairs_bytes(g) / 8, volt = bp_volume_bytes(g) / 4;
  // weighted sinograms of all items (two items interleaved, as 16-byte elements, in a
  // workspace aligned to them), then the scratch volumes
  float2* sinoz = reinterpret_cast<float2*>(workspace);
  const bool aligned = reinterpret_cast<uintptr_t>(workspace) % sizeof(float4) == 0;
  const int two = aligned && zlane_run(p) <= kTwoItemRun ? items / 2 : 0, one = items - 2 * two;
  if (two > 0) launch_weights<2>(p, {sino}, sinoz, 2 * pairs, 0, g.nangles, two, stream);
  if (one > 0)
    launch_weights<1>(p, {sino + 2 * two * sino_floats}, sinoz + 2 * two * pairs, pairs, 0, g.nangles,
                      one, stream);
  ZlaneArgs A = zlane_args(p, 0, n_ax, n_ax, n_ay);
  A.item_volt = volt * bp_scratch_volumes(p);
  A.volt[0] = reinterpret_cast<float*>(workspace + items * bp_pairs_bytes(g));
  A.volt[1] = n_ax > 0 ? A.volt[0] + volt : A.volt[0];
  float* first = A.volt[0];
  const float* second = n_ax > 0 && n_ay > 0 ? A.volt[1] : nullptr;
  if (two > 0) {
    A.sinoz = sinoz;
    A.group_pairs = 2 * pairs;
    launch_zlane_two(p, A, two, stream);
  }
  if (one > 0) {
    A.sinoz = sinoz + 2 * two * pairs;
    A.group_pairs = pairs;
    A.volt[0] += 2 * two * A.item_volt;
    A.volt[1] += 2 * two * A.item_volt;
    launch_zlane_passes(p, A, one, stream);
  }
  launch_zlane_out(g, additive ? 1 : 0, first, second, A.item_volt, A.zs, 0, g.nz, vol, nullptr,
                   items, stream);
  return int(cudaGetLastError());
}

}  // namespace tsgb
