// Parallel beams whose rays stay in one volume slice (p->flat): no ray has a
// component along z, det_v runs along z and det_u has no z component, as in
// every circular parallel scan (tomosipo/geometry/parallel.py). Both projections are
// those of fp.cu and bp_zlane.cu (Joseph's method and its exact transpose), with
// the z direction taken out of the inner loops:
//
//  * A ray's position along z, q_b = P + v R, is the same on every plane, so its
//    plane sum over the four voxels around it is the z interpolation of two
//    in-slice line sums. fp_flat_kernel computes the line sums S[theta][u][z] of
//    every slice, two coalesced loads, a sample and its addition per plane and voxel
//    along z, from one z-fastest copy of the volume; fp_flat_rows_kernel
//    interpolates them to the detector rows. (Where the rows are few and lie far
//    apart fp.cu follows their rays instead: flat_lines_pay in plan.cpp.)
//  * The transpose: a detector column's vertical profile V(z) does not depend on
//    the plane, so flat_resample_kernel computes it once per (angle, column)
//    instead of once per plane, and bp_flat_kernel adds it to the voxels with
//    the in-slice weights alone.
//
// Lanes run along z with kV consecutive floats each, so every load is a full
// 128 to 512 bytes. The kernels see only the slices that some detector row
// interpolates: their geometry's nz and oz are those slices' (window below), the
// volume's own only where a caller's volume is addressed.
#include <cuda_runtime.h>

#include <algorithm>

#include "device_common.cuh"

namespace tsgb {
namespace {

// Floats between z columns of the flat buffers (16-byte aligned columns).
__host__ __device__ inline int flat_zs(const DeviceGeometry& g) { return (g.nz + 3) / 4 * 4; }

template <int kV>
struct Vec;
template <>
struct Vec<1> {
  using T = float;
};
template <>
struct Vec<2> {
  using T = float2;
};
template <>
struct Vec<4> {
  using T = float4;
};

// kV floats at p as packed pairs (kV = 1: the second half is 0). kConstant: memory that
// the kernel does not write.
template <int kV, bool kConstant = true>
__device__ __forceinline__ void load_pairs(const float* p, f32x2 (&v)[(kV + 1) / 2]) {
  using T = typename Vec<kV>::T;
  const T* q = reinterpret_cast<const T*>(p);
  const T x = kConstant ? __ldg(q) : *q;
  if constexpr (kV == 1) v[0] = pack2(x, 0.0f);
  if constexpr (kV == 2) v[0] = pack2(x.x, x.y);
  if constexpr (kV == 4) {
    v[0] = pack2(x.x, x.y);
    v[1] = pack2(x.z, x.w);
  }
}
template <int kV>
__device__ __forceinline__ void store_pairs(float* p, const f32x2 (&v)[(kV + 1) / 2]) {
  float a, b, c, d;
  unpack2(v[0], a, b);
  if constexpr (kV == 1) *p = a;
  if constexpr (kV == 2) *reinterpret_cast<float2*>(p) = make_float2(a, b);
  if constexpr (kV == 4) {
    unpack2(v[1], c, d);
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
  }
}

// ------------------------------------------------------------------ forward
// z-fastest copy of the volume with kPad zero voxels around each slice:
// element (y, x, z) at ((y + kPad) (nx + 2 kPad) + x + kPad) zs + z, z rows
// padded with zeros to zs. Each block transposes 32 x 32 tiles of the (x, z)
// plane through shared memory. blockIdx.x = item * z tiles + z tile.
__global__ void __launch_bounds__(256)
    flat_copy_kernel(const float* __restrict__ vol, long long item_vol, float* __restrict__ copy,
                     long long item_copy, DeviceGeometry g) {
  __shared__ float tile[32][33];  // [z][x]
  const int zs = flat_zs(g), nxp = g.nx + 2 * kPad, nyp = g.ny + 2 * kPad;
  const int z_tiles = (zs + 31) / 32, item = blockIdx.x / z_tiles;
  const int z0 = (blockIdx.x - item * z_tiles) * 32, x0 = blockIdx.y * 32;
  vol += item * item_vol;
  copy += item * item_copy;
  for (int yp = blockIdx.z; yp < nyp; yp += gridDim.z) {
    const int y = yp - kPad, x = x0 + int(threadIdx.x) - kPad;
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int z = z0 + int(threadIdx.y) + 8 * q;
      const bool in = z < g.nz && y >= 0 && y < g.ny && x >= 0 && x < g.nx;
      v[q] = in ? __ldg(vol + ((size_t)z * g.ny + y) * g.nx + x) : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) tile[threadIdx.y + 8 * q][threadIdx.x] = v[q];
    __syncthreads();
#pragma unroll
    for (int k = threadIdx.y, q = 0; q < 4; ++q, k += 8) {
      const int xp = x0 + k, z = z0 + threadIdx.x;
      if (xp < nxp && z < zs) copy[((size_t)yp * nxp + xp) * zs + z] = tile[threadIdx.x][k];
    }
    __syncthreads();
  }
}

// Tile order of the line sums: a block is kFlatCols columns x kFlatAngles
// adjacent angles (one warp each), whose lines overlap in L1; blocks run over
// patches of kPatchCols column groups x kPatchAngles angle groups, so that the
// part of the volume a patch crosses stays in L2.
constexpr int kFlatCols = 2, kFlatAngles = 4;
constexpr int kPatchCols = 16, kPatchAngles = 16;
constexpr int kFlatPlanes = 32;  // planes prepared at a time, one per lane

// Line sums of kR ranges of 32 kV voxels along z: per plane the line's two
// columns with the weights 1 - fa and fa. Positions, weights and offsets of 32
// planes at a time are computed with one lane per plane and read back from shared
// memory. Planes alternate between two partial sums.
// sums holds the angles from angle_begin on.
// blockIdx.x = tile, blockIdx.y = z range, blockIdx.z = item.
template <int kV, int kR>
__global__ void __launch_bounds__(256)
    fp_flat_kernel(const AngleParams* __restrict__ params, const ColumnEntry* __restrict__ columns,
                   const float* __restrict__ copy, float* __restrict__ sums, long long item_floats,
                   DeviceGeometry g, int angle_begin, int angle_end) {
  constexpr int kP = (kV + 1) / 2;
  __shared__ float4 s_plane[kFlatCols * kFlatAngles][kFlatPlanes];  // byte offset, 1 - fa, fa
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col_groups = (g.cols + kFlatCols - 1) / kFlatCols;
  const int ang_groups = (angle_end - angle_begin + kFlatAngles - 1) / kFlatAngles;
  // patch, then tile inside it (only the last patches are smaller)
  unsigned b = blockIdx.x;
  const int pa = int(b / unsigned(kPatchAngles * col_groups));
  b -= unsigned(pa) * unsigned(kPatchAngles * col_groups);
  const int asz = min(kPatchAngles, ang_groups - pa * kPatchAngles);
  const int pc = int(b / unsigned(asz * kPatchCols));
  b -= unsigned(pc) * unsigned(asz * kPatchCols);
  const int csz = min(kPatchCols, col_groups - pc * kPatchCols);
  const int iu = (pc * kPatchCols + int(b) % csz) * kFlatCols + w % kFlatCols;
  const int theta = angle_begin + (pa * kPatchAngles + int(b) / csz) * kFlatAngles + w / kFlatCols;
  if (iu >= g.cols || theta >= angle_end) return;  // whole warp (no block barriers)
  const AngleParams& ap = params[theta];
  const ColumnEntry& ce = columns[(size_t)theta * g.cols + iu];
  const float Xa = ce.Xa, ma = ce.ma;
  const int zs = flat_zs(g), nxp = g.nx + 2 * kPad;
  const bool ax = ap.a == 2;
  const int stride_a = ax ? zs : nxp * zs, stride_d = ax ? nxp * zs : zs;  // floats
  const int border = -((g.oy + kPad) * nxp + g.ox + kPad) * zs;
  const int z0 = blockIdx.y * (32 * kV * kR) + lane * kV;
  // anchored voxel (0, 0), this lane's z
  const char* base = reinterpret_cast<const char*>(
      copy + blockIdx.z * item_floats + ((long long)(g.oy + kPad) * nxp + g.ox + kPad) * zs + z0);
  // planes where the line passes within a voxel of the slice
  float klo = float(-ap.o_d), khi = float(ap.n_d - 1 - ap.o_d);
  clip_planes(Xa, ma, float(-1 - ap.o_a), float(ap.n_a - ap.o_a), klo, khi);
  const int k0 = klo <= khi ? (int)ceilf(klo) : 1, k1 = klo <= khi ? (int)floorf(khi) : 0;
  f32x2 acc[2][kR][kP];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
      for (int i = 0; i < kP; ++i) acc[q][r][i] = 0ull;
  for (int kb = k0; kb <= k1; kb += kFlatPlanes) {
    const int k = kb + lane;
    const float qa = fmaf(float(k), ma, Xa);
    const float fq = __fadd_rd(qa, kFloorMagic);
    const float fa = qa - (fq - kFloorMagic);
    const int i0 = int(__float_as_uint(fq) - kFloorBits);
    const bool in = k <= k1;
    // (planes past the last read the copy's zero border)
    s_plane[w][lane] = make_float4(__int_as_float(in ? k * stride_d + i0 * stride_a : border),
                                   in ? 1.0f - fa : 0.0f, in ? fa : 0.0f, 0.0f);
    __syncwarp();
    const int n = min(kFlatPlanes, k1 - kb + 1);
#pragma unroll 2
    for (int p = 0; p < n; p += 2) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 e = s_plane[w][p + q];
        const char* p0 = base + (long long)__float_as_int(e.x) * 4;
        const char* p1 = p0 + (long long)stride_a * 4;
        const f32x2 w0 = pack2(e.y, e.y), w1 = pack2(e.z, e.z);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          if (z0 + r * 32 * kV >= zs) break;
          f32x2 v0[kP], v1[kP];
          load_pairs<kV>(reinterpret_cast<const float*>(p0) + r * 32 * kV, v0);
          load_pairs<kV>(reinterpret_cast<const float*>(p1) + r * 32 * kV, v1);
#pragma unroll
          for (int i = 0; i < kP; ++i)
            // (the plane's sample, then the sum: one rounding of the sum per plane)
            acc[q][r][i] = add2(acc[q][r][i], fma2(w1, v1[i], mul2(w0, v0[i])));
        }
      }
    }
    __syncwarp();
  }
  float* out =
      sums + blockIdx.z * item_floats + ((size_t)(theta - angle_begin) * g.cols + iu) * zs + z0;
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    if (z0 + r * 32 * kV >= zs) break;
    f32x2 s[kP];
#pragma unroll
    for (int i = 0; i < kP; ++i) s[i] = add2(acc[0][r][i], acc[1][r][i]);
    store_pairs<kV>(out + r * 32 * kV, s);
  }
}

// Detector rows from the line sums: row v lies at q_b = P + v R along z, its sum
// is the linear interpolation of S there (0 outside the volume) times the plane
// step W. 32 x 32 tiles of (row, column) through shared memory: reads along z,
// writes along u. blockIdx.z counts items * angles of the range.
template <int kMode>  // 0 set, 1 add, 2 SIRT residual
__global__ void __launch_bounds__(256)
    fp_flat_rows_kernel(const AngleParams* __restrict__ params,
                        const ColumnEntry* __restrict__ columns, const float* __restrict__ sums,
                        long long item_floats, float* __restrict__ sino, DeviceGeometry g,
                        int angle_begin, int n_angles, int items, FpSirt sirt) {
  __shared__ float tile[32][33];  // [row][column]
  const int zs = flat_zs(g);
  const int u0 = blockIdx.x * 32, v0 = blockIdx.y * 32;
  for (unsigned b = blockIdx.z; b < unsigned(items) * unsigned(n_angles); b += gridDim.z) {
    const int item = items == 1 ? 0 : int(b / unsigned(n_angles));
    const int n = int(b - unsigned(item) * unsigned(n_angles)), theta = angle_begin + n;
    const AngleParams& ap = params[theta];
    const float P = ap.cb[0], R = ap.cb[2];
    const int iv = v0 + int(threadIdx.x);
    const float q = fmaf(float(iv - g.ov), R, P);
    const bool in = iv < g.rows && q > float(-1 - g.oz) && q < float(g.nz - g.oz);
    const float fl = floorf(in ? q : 0.0f), f = in ? q - fl : 0.0f;
    const int j = int(fl) + g.oz;
    const bool in_a = in && j >= 0, in_d = in && j + 1 < g.nz;
    const int c0 = u0 + int(threadIdx.y);
    const float* s = sums + item * item_floats + ((size_t)n * g.cols + c0) * zs + j;
    float a[4], d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool column = c0 + 8 * q < g.cols;
      a[q] = in_a && column ? __ldg(s + q * 8 * zs) : 0.0f;
      d[q] = in_d && column ? __ldg(s + q * 8 * zs + 1) : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      tile[threadIdx.x][threadIdx.y + 8 * q] = fmaf(f, d[q] - a[q], a[q]);
    __syncthreads();
    const int iu = u0 + int(threadIdx.x);
    if (iu < g.cols) {
      Ray r;
      r.Xa = r.Xb = r.mb = 0.0f;
      r.ma = columns[(size_t)theta * g.cols + iu].ma;
      const float W = ray_step(ap, r);
      const long long row = (long long)g.nangles * g.cols;
      long long idx = (v0 + int(threadIdx.y)) * row + (long long)theta * g.cols + iu;
      float* out = sino + item * (g.rows * row);
#pragma unroll
      for (int k = threadIdx.y, q = 0; q < 4; ++q, k += 8) {
        if (v0 + k >= g.rows) break;
        const float total = __fmul_rn(tile[k][threadIdx.x], W);
        if (kMode == 2)
          sirt_residual(sirt, g, idx, total, W);
        else
          out[idx] = kMode == 1 ? __fadd_rn(out[idx], total) : total;
        idx += 8 * row;
      }
    }
    __syncthreads();
  }
}


// --------------------------------------------------------------- backward
// V[theta][u][z] = sum over the detector rows of tent(P + v R - z) W y[v][theta][u]
// (W = 1 when kWeighted: a SIRT residual holds W y). Rows at least a voxel apart:
// the two rows around z, as saturating adds; else every row whose tent reaches z.
// 32 (z) x 32 (column) tiles through shared memory: reads along u, writes along z. out
// holds the angles from angle_begin on. blockIdx.x = column tile, blockIdx.y = z tile,
// blockIdx.z counts items * angles.
template <bool kWeighted, bool kSpread>
__global__ void __launch_bounds__(256)
    flat_resample_kernel(const AngleParams* __restrict__ params,
                         const ColumnEntry* __restrict__ columns, SinoSource sino,
                         float* __restrict__ out, long long item_floats, DeviceGeometry g,
                         int angle_begin, int n_angles, int items) {
  __shared__ float tile[32][33];  // [z][column]
  // per z: rows a voxel apart or more: both tents, the first row, which are on the
  // detector; else P - z, the first row from the anchor, the first row, how many
  __shared__ float4 s_z[32];
  const int zs = flat_zs(g);
  const int u0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
  const int iu = u0 + int(threadIdx.x);
  // the source's columns and elements between its rows (kSpread: a coarser detector)
  const int ys = kSpread ? int(source_pixel(sino, g.cols)) : g.cols;
  const size_t rs = (size_t)g.nangles * ys;
  const auto value = [&](const float* y, int iv) {
    if (!kSpread) return __ldg(y + (long long)iv * (long long)rs);
    return sino.scale * __ldg(y + source_pixel(sino, iv) * rs);
  };
  for (unsigned b = blockIdx.z; b < unsigned(items) * unsigned(n_angles); b += gridDim.z) {
    const int item = items == 1 ? 0 : int(b / unsigned(n_angles));
    const int angle = int(b - unsigned(item) * unsigned(n_angles)), theta = angle_begin + angle;
    const AngleParams& ap = params[theta];
    const float P = ap.cb[0], R = ap.cb[2], inv = __frcp_rn(R), aR = fabsf(R);
    // P as a multiple of 2^-14 plus a remainder, so that P - z is exact
    const float Ph = (P + 768.0f) - 768.0f, Pl = P - Ph;
    const float* y = sino.y + (size_t)item * g.rows * rs + (size_t)theta * ys +
                     (kSpread ? int(source_pixel(sino, iu)) : iu);
    float W = 1.0f;
    if (!kWeighted && iu < g.cols) {
      Ray r;
      r.Xa = r.Xb = r.mb = 0.0f;
      r.ma = columns[(size_t)theta * g.cols + iu].ma;
      W = ray_step(ap, r);
    }
    // the rows that reach each z, found by the first warp: the two around it and their
    // tents, or the first and last whose tent covers it
    if (threadIdx.y == 0) {
      const int z = z0 + int(threadIdx.x);
      const float C = Ph - float(z - g.oz);
      if (aR >= 1.0f) {
        const float v = floorf(clamp_coord(-(C + Pl) * inv));
        const float t = fabsf(fmaf(v, R, C) + Pl);
        const int iv = int(v) + g.ov;
        const int in0 = z < g.nz && iv >= 0 && iv < g.rows ? 1 : 0;
        const int in1 = z < g.nz && iv + 1 >= 0 && iv + 1 < g.rows ? 2 : 0;
        s_z[threadIdx.x] = make_float4(__saturatef(1.0f - t), __saturatef((1.0f - aR) + t),
                                       __int_as_float(iv), __int_as_float(in0 | in1));
      } else {
        const float B = C + Pl;
        // (widened by more than v1's and v2's rounding; a row more has weight 0)
        const float va = (-1.0f - B) * inv, vb = (1.0f - B) * inv;
        const float v1 = clamp_coord(fminf(va, vb)), v2 = clamp_coord(fmaxf(va, vb));
        const int lo = max(0, (int)ceilf(v1 - fmaf(fabsf(v1), 1e-6f, 0.01f)) + g.ov);
        const int hi = min(g.rows - 1, (int)floorf(v2 + fmaf(fabsf(v2), 1e-6f, 0.01f)) + g.ov);
        s_z[threadIdx.x] = make_float4(C, float(lo - g.ov), __int_as_float(lo),
                                       __int_as_float(z < g.nz ? hi - lo + 1 : 0));
      }
    }
    __syncthreads();
    float V[4];
    if (aR >= 1.0f) {
      float y0[4], y1[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 e = s_z[threadIdx.y + 8 * q];
        const int iv = __float_as_int(e.z), in = iu < g.cols ? __float_as_int(e.w) : 0;
        y0[q] = in & 1 ? value(y, iv) : 0.0f;
        y1[q] = in & 2 ? value(y, iv + 1) : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 e = s_z[threadIdx.y + 8 * q];
        V[q] = fmaf(e.x, W * y0[q], e.y * (W * y1[q]));
      }
    } else {
      // one row of each of the four z at a time (their loads in flight together)
      int n[4], most = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        n[q] = iu < g.cols ? __float_as_int(s_z[threadIdx.y + 8 * q].w) : 0;
        most = max(most, n[q]);
        V[q] = 0.0f;
      }
      for (int i = 0; i < most; ++i) {
        float yi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          yi[q] = i < n[q] ? value(y, __float_as_int(s_z[threadIdx.y + 8 * q].z) + i) : 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 e = s_z[threadIdx.y + 8 * q];
          if (i < n[q]) V[q] = fmaf(tent(fmaf(e.y + float(i), R, e.x) + Pl), W * yi[q], V[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) tile[threadIdx.y + 8 * q][threadIdx.x] = V[q];
    __syncthreads();
    const int z = z0 + int(threadIdx.x);
#pragma unroll
    for (int c = threadIdx.y, q = 0; q < 4; ++q, c += 8)
      if (z < zs && u0 + c < g.cols)
        out[item * item_floats + ((size_t)angle * g.cols + u0 + c) * zs + z] = tile[threadIdx.x][c];
    __syncthreads();
  }
}

struct FlatBpArgs {
  const SolveEntry* solve[2];  // pass 0: a = x, pass 1: a = y
  int n[2];
  int plane_blocks[2];
  unsigned blocks0;
  const ColumnEntry* columns;
  const float* profiles;       // V[theta][u][z] from column first_column (theta, u) on
  unsigned first_column;
  float* volt[2];              // [y][x][z] sum of each pass
  bool add[2];                 // onto what volt holds (angles of an earlier launch)
  long long item_floats;
  DeviceGeometry g;
};

constexpr int kFlatWarps = 8, kFlatX = 4;

// As bp_zlane_kernel (windows of kX voxels along a on one plane, one warp each;
// column lists built with one lane per column; loads a column ahead), with the
// profile read instead of computed. Lanes hold kR runs of kV consecutive voxels
// along z. blockIdx.x = window * plane_blocks + plane block (pass 0, then pass 1),
// blockIdx.y = z range, blockIdx.z = item.
template <int kX, int kV, int kR, int kMinBlocks, int kSplit>
__global__ void __launch_bounds__(32 * kFlatWarps, kMinBlocks)
    bp_flat_kernel(const __grid_constant__ FlatBpArgs A) {
  constexpr int kPlanes = kFlatWarps / kSplit;
  constexpr int kP = (kV + 1) / 2, kPairs = kP * kR;
  // column list: weights (1 - fa, 1 - fa, fa, fa) and (window position f0, column);
  // two slots past a full list are loaded from, never added
  __shared__ float4 s_weight[kFlatWarps][34];
  __shared__ int2 s_column[kFlatWarps][34];
  const DeviceGeometry& g = A.g;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int pass = blockIdx.x < A.blocks0 ? 0 : 1;
  const unsigned block = blockIdx.x - (pass ? A.blocks0 : 0u);
  const int n_p = pass ? g.nx : g.ny, n_a = pass ? g.ny : g.nx;
  const int ip = int(block % unsigned(A.plane_blocks[pass])) * kPlanes + w % kPlanes;
  const int i0 = int(block / unsigned(A.plane_blocks[pass])) * kX;
  if (kSplit == 1 && ip >= n_p) return;  // whole warp (no block barriers then)
  // this warp's angles (none where the plane lies outside the volume)
  const int n_all = ip < n_p ? A.n[pass] : 0;
  const int n_begin = n_all * (w / kPlanes) / kSplit, n_end = n_all * (w / kPlanes + 1) / kSplit;
  const int zs = flat_zs(g);
  const int z0 = blockIdx.y * (32 * kV * kR) + lane * kV;
  const float kt = float(ip - (pass ? g.ox : g.oy));
  const float i0t = float(i0 - (pass ? g.oy : g.ox));
  const float4* __restrict__ solve = reinterpret_cast<const float4*>(A.solve[pass]);
  const float4* __restrict__ col4 = reinterpret_cast<const float4*>(A.columns);
  const char* base = reinterpret_cast<const char*>(A.profiles + blockIdx.z * A.item_floats);
  unsigned zoff[kR];  // bytes from a column's start
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int z = z0 + r * 32 * kV;
    zoff[r] = (z < zs ? z : 0) * unsigned(sizeof(float));
  }
  f32x2 acc[1][kX][kPairs];
#pragma unroll
  for (int m = 0; m < kX; ++m)
#pragma unroll
    for (int j = 0; j < kPairs; ++j) acc[0][m][j] = 0ull;
  // (slots not filled yet stand for column 0)
  for (int k = lane; k < 34; k += 32) s_column[w][k] = make_int2(0, 0);
  __syncwarp();
  const unsigned column_bytes = unsigned(zs * sizeof(float));
  const auto stage = [&](f32x2(&V)[kPairs], int2 c) {
    const char* p = base + (size_t)unsigned(c.y) * column_bytes;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      // (lanes past the end of the column read its start; they are not stored)
      f32x2 x[kP];
      load_pairs<kV>(reinterpret_cast<const float*>(p + zoff[r]), x);
#pragma unroll
      for (int i = 0; i < kP; ++i) V[r * kP + i] = x[i];
    }
  };
  const auto finish = [&](const f32x2(&V)[kPairs], int2 c, float4 e) {
    const auto profile = [&](int, int j) { return V[j]; };
    window_dispatch<-1, kX>(acc, c.x, profile, pack2(e.x, e.y), pack2(e.z, e.w));
  };
  for (int n0 = n_begin; n0 < n_end; n0 += 32) {
    const ColumnRanges cr =
        column_ranges(solve, n0 + lane, n_end, kt, i0t - 1.0f, i0t + float(kX), g);
    for (int t0 = 0; t0 < cr.total; t0 += 32) {
      const int t = t0 + lane;
      int iu, th;
      column_of(cr, t, iu, th);
      bool ok = t < cr.total;
      float4 e;
      int2 c;
      if (ok) {
        const size_t ci = (size_t)th * g.cols + iu;
        const float4 c0 = __ldg(col4 + 2 * ci);  // Xa, ma, -, -
        const float qa = fmaf(kt, c0.y, c0.x) - i0t;
        ok = qa > -1.0f && qa < float(kX);  // (NaN: no)
        const float fq = __fadd_rd(qa, kFloorMagic);
        const float fa = qa - (fq - kFloorMagic);
        e = make_float4(1.0f - fa, 1.0f - fa, fa, fa);
        c = make_int2(int(__float_as_uint(fq) - kFloorBits), int(unsigned(ci) - A.first_column));
      }
      const unsigned mask = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        const int slot = __popc(mask & ((1u << lane) - 1u));
        s_weight[w][slot] = e;
        s_column[w][slot] = c;
      }
      __syncwarp();
      // A column's profile is loaded while the column before it is added, its
      // list entry a column earlier still.
      const int n = __popc(mask);
      const int2* lc = s_column[w];
      const float4* lw = s_weight[w];
      int2 cq[4];
      float4 eq[2];
      f32x2 v[2][kPairs];
      cq[0] = lc[0];
      cq[1] = lc[1];
      eq[0] = lw[0];
      stage(v[0], cq[0]);
      for (int k = 0; k < n; k += 4, lc += 4, lw += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (k + i >= n) break;
          cq[(i + 2) & 3] = lc[i + 2];
          eq[(i + 1) & 1] = lw[i + 1];
          stage(v[(i + 1) & 1], cq[(i + 1) & 3]);
          finish(v[i & 1], cq[i], eq[i & 1]);
        }
      }
      __syncwarp();  // the list is rewritten
    }
  }
  if constexpr (kSplit > 1) {
    // the splits' sums, in order
    __shared__ f32x2 s_sum[kPlanes][kX * kPairs][32];
    for (int split = 1; split < kSplit; ++split) {
      if (w / kPlanes == split) {
#pragma unroll
        for (int i = 0; i < kX * kPairs; ++i)
          s_sum[w % kPlanes][i][lane] = acc[0][i / kPairs][i % kPairs];
      }
      __syncthreads();
      if (w / kPlanes == 0) {
#pragma unroll
        for (int i = 0; i < kX * kPairs; ++i)
          acc[0][i / kPairs][i % kPairs] =
              add2(acc[0][i / kPairs][i % kPairs], s_sum[w % kPlanes][i][lane]);
      }
      __syncthreads();
    }
    if (w / kPlanes != 0 || ip >= n_p) return;
  }
  float* volt = A.volt[pass] + blockIdx.z * A.item_floats + z0;
#pragma unroll
  for (int m = 0; m < kX; ++m) {
    const int ia = i0 + m;
    if (ia >= n_a) break;
    float* out = volt + (pass ? (size_t)ia * g.nx + ip : (size_t)ip * g.nx + ia) * zs;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      if (z0 + r * 32 * kV >= zs) break;
      f32x2 x[kP];
#pragma unroll
      for (int i = 0; i < kP; ++i) x[i] = acc[0][m][r * kP + i];
      if (A.add[pass]) {
        f32x2 old[kP];
        load_pairs<kV, false>(out + r * 32 * kV, old);
#pragma unroll
        for (int i = 0; i < kP; ++i) x[i] = add2(old[i], x[i]);
      }
      store_pairs<kV>(out + r * 32 * kV, x);
    }
  }
}

template <int kV, int kR>
void launch_fp_tiles(const tsgb_projector* p, const float* copy, float* sums, long long item_floats,
                     const DeviceGeometry& g, int angle_begin, int angle_end, int items,
                     cudaStream_t stream) {
  const int zs = flat_zs(g);
  const unsigned tiles = unsigned((g.cols + kFlatCols - 1) / kFlatCols) *
                         unsigned((angle_end - angle_begin + kFlatAngles - 1) / kFlatAngles);
  const dim3 grid(tiles, unsigned((zs + 32 * kV * kR - 1) / (32 * kV * kR)), unsigned(items));
  fp_flat_kernel<kV, kR><<<grid, 32 * kFlatCols * kFlatAngles, 0, stream>>>(
      p->d_params, p->d_columns, copy, sums, item_floats, g, angle_begin, angle_end);
}

template <int kX, int kV, int kR, int kMinBlocks, int kSplit>
void launch_bp_windows(FlatBpArgs& A, int items, cudaStream_t stream) {
  const DeviceGeometry& g = A.g;
  const int zs = flat_zs(g);
  unsigned blocks[2];
  for (int pass = 0; pass < 2; ++pass) {
    const int n_p = pass ? g.nx : g.ny, n_a = pass ? g.ny : g.nx;
    A.plane_blocks[pass] = (n_p + kFlatWarps / kSplit - 1) / (kFlatWarps / kSplit);
    blocks[pass] = A.n[pass] > 0 ? unsigned(A.plane_blocks[pass]) * unsigned((n_a + kX - 1) / kX) : 0u;
  }
  A.blocks0 = blocks[0];
  const dim3 grid(blocks[0] + blocks[1], unsigned((zs + 32 * kV * kR - 1) / (32 * kV * kR)),
                  unsigned(items));
  bp_flat_kernel<kX, kV, kR, kMinBlocks, kSplit><<<grid, 32 * kFlatWarps, 0, stream>>>(A);
}

// Warps of one item that share a window's angles: where the windows alone are few
// for 152 SMs, 2 or 8 warps take a part of the angles each and add their sums.
// Measured (us per backprojection, split 1 / 2 / 8): 32^3 / 60 angles 27.9 / 19.3 /
// 13.2, 64^3 / 96 43.1 / 30.8 / 36.3, 128^3 / 200 195.6 / 190.2 / -, 192^3 / 300 887 /
// 965 / -. Windows of 4 voxels: 6 at 203 x 397 x 421 / 401 cost 10.4 ms (forward
// projection included) against 9.6, 3 and 5 9.7 and 10.3.
template <int kV, int kR, int kMinBlocks>
void launch_bp_split(FlatBpArgs& A, int items, cudaStream_t stream) {
  const DeviceGeometry& g = A.g;
  const int64_t ranges = (flat_zs(g) + 32 * kV * kR - 1) / (32 * kV * kR);
  const int64_t warps = int64_t(g.ny) * g.nx / kFlatX * ranges * ((A.n[0] > 0) + (A.n[1] > 0));
  if (warps < 1024)
    launch_bp_windows<kFlatX, kV, kR, kMinBlocks, 8>(A, items, stream);
  else if (warps < 16384)
    launch_bp_windows<kFlatX, kV, kR, kMinBlocks, 2>(A, items, stream);
  else
    launch_bp_windows<kFlatX, kV, kR, kMinBlocks, 1>(A, items, stream);
}

// Buffers start on 16 bytes in workspaces this package allocates. A caller's own may
// not: its copies and columns are then read one float at a time.
bool vectors_aligned(const void* workspace) {
  return reinterpret_cast<uintptr_t>(workspace) % sizeof(float4) == 0;
}

// The geometry of the slices p's rows interpolate. A detector of 32 rows over 512
// slices of 192^2 voxels, 180 angles: forward projection 933 -> 218 us, backprojection
// 1012 -> 329 (all slices against 64).
DeviceGeometry window(const tsgb_projector* p) {
  DeviceGeometry g = p->g;
  g.oz -= p->flat_z0;
  g.nz = p->flat_nz;
  return g;
}

int64_t round256(int64_t b) { return (b + 255) / 256 * 256; }
int64_t copy_bytes(const DeviceGeometry& g) {
  return round256(int64_t(g.ny + 2 * kPad) * (g.nx + 2 * kPad) * flat_zs(g) * 4);
}
// Angles whose line sums or profiles the kernels hold at a time: about 2 GiB of them
// (whole patches of angle groups), so that a long scan does not need its sinogram's size
// or more once again. Pieces cost their launches and, in the backprojection, a read of
// the scratch volumes each.
int line_angles(const DeviceGeometry& g) {
  constexpr int64_t kBudget = int64_t(2) << 30, kPatch = kFlatAngles * kPatchAngles;
  const int64_t fit = kBudget / (int64_t(g.cols) * flat_zs(g) * 4) / kPatch * kPatch;
  return int(std::min<int64_t>(g.nangles, std::max(fit, kPatch)));
}
int64_t line_bytes(const DeviceGeometry& g) {
  return round256(int64_t(line_angles(g)) * g.cols * flat_zs(g) * 4);
}
int64_t volt_bytes(const DeviceGeometry& g) {
  return round256(int64_t(g.ny) * g.nx * flat_zs(g) * 4);
}

}  // namespace

int64_t flat_fp_bytes(const tsgb_projector* p) {
  const DeviceGeometry g = window(p);
  return copy_bytes(g) + line_bytes(g);
}
int64_t flat_bp_bytes(const tsgb_projector* p) {
  const DeviceGeometry g = window(p);
  return line_bytes(g) + bp_scratch_volumes(p) * volt_bytes(g);
}
int flat_chunks(const tsgb_projector* p) {
  return (p->g.nangles - 1) / line_angles(window(p)) + 1;
}

int launch_flat_fp(const tsgb_projector* p, const float* vol, float* sino, bool additive,
                   float* workspace, void* stream_, const FpSirt* sirt, int angle_begin,
                   int angle_end, bool copies_ready, int items, int64_t item_bytes) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const DeviceGeometry g = window(p);
  const int zs = flat_zs(g), step = line_angles(g);
  const long long item_floats = item_bytes / 4;
  float* copy = workspace;
  float* sums = workspace + copy_bytes(g) / 4;
  if (!copies_ready) {
    const dim3 grid(unsigned((zs + 31) / 32) * unsigned(items),
                    unsigned((g.nx + 2 * kPad + 31) / 32),
                    unsigned(std::min(g.ny + 2 * kPad, 65535)));
    const long long slice = (long long)g.ny * g.nx;
    flat_copy_kernel<<<grid, dim3(32, 8), 0, stream>>>(vol + p->flat_z0 * slice, p->g.nz * slice,
                                                       copy, item_floats, g);
  }
  for (int a0 = angle_begin, a1; a0 < angle_end; a0 = a1) {
    a1 = int(std::min<int64_t>(int64_t(a0) + step, angle_end));
    if (zs <= 32 || !vectors_aligned(workspace))
      launch_fp_tiles<1, 1>(p, copy, sums, item_floats, g, a0, a1, items, stream);
    else if (zs <= 64)
      launch_fp_tiles<2, 1>(p, copy, sums, item_floats, g, a0, a1, items, stream);
    else if (zs <= 128)
      launch_fp_tiles<4, 1>(p, copy, sums, item_floats, g, a0, a1, items, stream);
    else
      launch_fp_tiles<4, 2>(p, copy, sums, item_floats, g, a0, a1, items, stream);
    const dim3 grid(unsigned((g.cols + 31) / 32), unsigned((g.rows + 31) / 32),
                    unsigned(std::min<long long>((long long)items * (a1 - a0), 65535)));
    const auto rows = sirt       ? fp_flat_rows_kernel<2>
                      : additive ? fp_flat_rows_kernel<1>
                                 : fp_flat_rows_kernel<0>;
    rows<<<grid, dim3(32, 8), 0, stream>>>(p->d_params, p->d_columns, sums, item_floats, sino, g, a0,
                                           a1 - a0, items, sirt ? *sirt : FpSirt{});
  }
  return int(cudaGetLastError());
}

int launch_flat_bp(const tsgb_projector* p, float* vol, SinoSource sino, bool weighted,
                   int out_mode, const float* C, float* workspace, void* stream_, int angle_begin,
                   int angle_end, int items, int64_t item_bytes) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const DeviceGeometry g = window(p);
  const int zs = flat_zs(g), step = line_angles(g);
  if (angle_end <= angle_begin) return int(cudaGetLastError());
  FlatBpArgs A{};
  A.columns = p->d_columns;
  A.profiles = workspace;
  A.item_floats = item_bytes / 4;
  A.g = g;
  // a pass's angles in [a0, a1): where they lie in its list (ids increase), how many
  const auto b = p->host_sep_angles.begin();
  const auto range = [&](int pass, int a0, int a1, int* n) {
    const auto lo = pass ? b + p->n_sep_ax : b, hi = pass ? p->host_sep_angles.end() : b + p->n_sep_ax;
    const auto first = std::lower_bound(lo, hi, a0);
    *n = int(std::lower_bound(first, hi, a1) - first);
    return p->d_solve + (first - b);
  };
  int all[2];
  for (int pass = 0; pass < 2; ++pass) range(pass, angle_begin, angle_end, &all[pass]);
  A.volt[0] = workspace + line_bytes(g) / 4;
  A.volt[1] = all[0] > 0 ? A.volt[0] + volt_bytes(g) / 4 : A.volt[0];
  for (int a0 = angle_begin, a1; a0 < angle_end; a0 = a1) {
    a1 = int(std::min<int64_t>(int64_t(a0) + step, angle_end));
    const dim3 grid(unsigned((g.cols + 31) / 32), unsigned((zs + 31) / 32),
                    unsigned(std::min<long long>((long long)items * (a1 - a0), 65535)));
    // (residuals are never spread)
    const auto resample = weighted     ? flat_resample_kernel<true, false>
                          : sino.d > 1 ? flat_resample_kernel<false, true>
                                       : flat_resample_kernel<false, false>;
    resample<<<grid, dim3(32, 8), 0, stream>>>(p->d_params, p->d_columns, sino, workspace,
                                               A.item_floats, g, a0, a1 - a0, items);
    A.first_column = unsigned(a0) * unsigned(g.cols);
    for (int pass = 0; pass < 2; ++pass) A.solve[pass] = range(pass, a0, a1, &A.n[pass]);
    if (zs <= 32 || !vectors_aligned(workspace))
      launch_bp_split<1, 1, 4>(A, items, stream);
    else if (zs <= 64)
      launch_bp_split<2, 1, 4>(A, items, stream);
    else if (zs <= 128)
      launch_bp_split<4, 1, 4>(A, items, stream);
    else if (192 * ((zs + 191) / 192) < 256 * ((zs + 255) / 256))
      // z ranges of 3 x 64 voxels leave fewer lanes idle than 2 x 128: nz = 140, 160, 192
      // and 300 of 192^2 to 256^2 columns 587 -> 547, 536 -> 470, 872 -> 826 and 1853 ->
      // 1750 us per backprojection (256, where they do not: 1702 -> 3012). The forward
      // projection gains nothing (437 -> 447 us at 160).
      launch_bp_split<2, 3, 3>(A, items, stream);
    else
      launch_bp_split<4, 2, 3>(A, items, stream);
    for (int pass = 0; pass < 2; ++pass) A.add[pass] = A.add[pass] || A.n[pass] > 0;
  }
  launch_zlane_out(p->g, out_mode, A.volt[0], all[0] > 0 && all[1] > 0 ? A.volt[1] : nullptr,
                   A.item_floats, zs, p->flat_z0, p->flat_nz, vol, C, items, stream);
  return int(cudaGetLastError());
}

}  // namespace tsgb
