// Bilinear (voxel-driven) backprojection of the angles whose projection keeps u
// and the depth constant along z (det_v along z: circular and helical scans),
// with the bilinear backprojector's weights or FDK's.
//
// All voxels of a column (x, y) read between the same two detector columns with
// the same weights, and their rows are linear in z. So a warp owns one voxel
// column, its lanes run along z (lane l: z0 + l + 32 j, j < kRun), and what
// depends only on the angle (columns, weights, depth, row step) is computed with
// one lane per angle, 32 angles at a time, and read back from shared memory.
// Per voxel and angle that leaves the row, two loads and the interpolation.
//
// The sinogram is copied to column-major row pairs (bilinear_pairs_kernel):
// element (angle, u, r) = (y[v], y[v+1]) of detector row v = r - kRowPad, rows
// fastest, kRowPad zero rows and kColPad zero columns around the detector. The
// lanes' loads of a column fall on about 23 consecutive pairs, and neighbouring
// voxel columns (the block's other warps) read the same detector columns from L1.
// Results go to a z-fastest scratch volume, which launch_zlane_out transposes.
//
// The two 8-byte loads per voxel bound it: 95 % of the L1 data pipe at 320^3 / 500 FDK
// angles, 10.6 ms against 14.5 for one thread per voxel column and 16-byte quads (14 ms
// before the blocks ran in patches: a quarter of the L2 reads missed).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "device_common.cuh"

namespace tsgb {
namespace {

__host__ __device__ inline int padded_cols(const DeviceGeometry& g) { return g.cols + 2 * kColPad; }
__host__ __device__ inline int padded_rows(const DeviceGeometry& g) { return g.rows + 2 * kRowPad; }

// Column-major row pairs of the sinogram. A block copies 32 padded columns x 32
// padded rows of one angle through shared memory (33 rows: a pair's second row).
__global__ void __launch_bounds__(256)
    bilinear_pairs_kernel(const float* __restrict__ sino, float2* __restrict__ out,
                          DeviceGeometry g) {
  __shared__ float s[33][33];  // [row][column]
  const int cp = padded_cols(g), rp = padded_rows(g);
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int theta = blockIdx.z; theta < g.nangles; theta += gridDim.z) {
    const int iu = c0 + int(threadIdx.x) - kColPad;
    float v[5];  // rows threadIdx.y + 8 q; the 33rd is the first warp's
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int k = int(threadIdx.y) + 8 * q, iv = r0 + k - kRowPad;
      const bool in = iu >= 0 && iu < g.cols && iv >= 0 && iv < g.rows && k < 33;
      v[q] = in ? __ldg(sino + ((size_t)iv * g.nangles + theta) * g.cols + iu) : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q)
      if (q < 4 || threadIdx.y == 0) s[threadIdx.y + 8 * q][threadIdx.x] = v[q];
    __syncthreads();
    const int r = r0 + threadIdx.x;
#pragma unroll
    for (int c = threadIdx.y, q = 0; q < 4; ++q, c += 8)
      if (r < rp && c0 + c < cp)
        out[((size_t)theta * cp + c0 + c) * rp + r] =
            make_float2(s[threadIdx.x][c], s[threadIdx.x + 1][c]);
    __syncthreads();
  }
}

// Block: kWX x kWY voxel columns, one warp each.
constexpr int kWX = 2, kWY = 2;
// Blocks run in square patches of this many blocks a side, about the number in
// flight, so that the detector columns they read stay in L2.
constexpr int kPatch = 24;

// An angle's part for one voxel column, as two (cone: three) 16-byte words:
// weights of the two detector columns (twice each: packed operands), row step dv
// and row at z = 0, and the address of the first column's anchored row 0 minus
// kFloorBits pairs; cone: the weight's horizontal part.
template <int kWeight>
constexpr int kWords = kWeight == kBilCone ? 3 : 2;

// Entries [0, n) added to the lane's voxels zt + 32 j. kClamp: rows are clamped
// into the zero padding (integers vmin .. vmax; NaN -> vmin), which clamps their
// floor; else every row is known to lie inside.
template <int kRun, int kWeight, bool kClamp>
__device__ __forceinline__ void add_angles(float (&acc)[kRun],
                                           const float4 (&list)[34][kWords<kWeight>], int n,
                                           float zt, float vz, float vmin, float vmax,
                                           unsigned column_bytes) {
  constexpr int kPairs = (kRun + 1) / 2;
  struct Stage {
    f32x2 fv[kPairs], a[kRun], b[kRun];
  } st[2];
  const auto stage = [&](Stage& S, const float4(&entry)[kWords<kWeight>]) {
    const float4 e1 = entry[1];
    const char* col = reinterpret_cast<const char*>(
        size_t(__float_as_uint(e1.z)) | (size_t(__float_as_uint(e1.w)) << 32));
    const char* next = col + column_bytes;
    const float t0 = fmaf(zt, e1.x, e1.y);
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      const int ja = 2 * q, jb = 2 * q + 1 < kRun ? 2 * q + 1 : 2 * q;
      float ta = fmaf(float(32 * ja), e1.x, t0), tb = fmaf(float(32 * jb), e1.x, t0);
      if (kClamp) {
        ta = fminf(fmaxf(ta, vmin), vmax);
        tb = fminf(fmaxf(tb, vmin), vmax);
      }
      const f32x2 f = add2_rd(pack2(ta, tb), pack2(kFloorMagic, kFloorMagic));
      // t - floor(t), exact
      S.fv[q] = fma2(add2(f, pack2(-kFloorMagic, -kFloorMagic)), pack2(-1.0f, -1.0f), pack2(ta, tb));
      float fa, fb;
      unpack2(f, fa, fb);
      const size_t ra = size_t(__float_as_uint(fa)) * sizeof(float2);
      S.a[ja] = __ldg(reinterpret_cast<const unsigned long long*>(col + ra));
      S.b[ja] = __ldg(reinterpret_cast<const unsigned long long*>(next + ra));
      if (jb != ja) {
        const size_t rb = size_t(__float_as_uint(fb)) * sizeof(float2);
        S.a[jb] = __ldg(reinterpret_cast<const unsigned long long*>(col + rb));
        S.b[jb] = __ldg(reinterpret_cast<const unsigned long long*>(next + rb));
      }
    }
  };
  const auto finish = [&](const Stage& S, const float4(&entry)[kWords<kWeight>]) {
    const float4 e0 = entry[0];
    float4 e2;
    if constexpr (kWeight == kBilCone) e2 = entry[2];
    const f32x2 w0 = pack2(e0.x, e0.y), w1 = pack2(e0.z, e0.w);
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
      // the two rows between the columns, then between the rows
      float r0, r1, fa, fb;
      unpack2(fma2(w1, S.b[j], mul2(w0, S.a[j])), r0, r1);
      unpack2(S.fv[j / 2], fa, fb);
      const float val = fmaf(j % 2 ? fb : fa, r1 - r0, r0);
      if constexpr (kWeight == kBilCone) {
        const float dz = fmaf(float(32 * j), vz, fmaf(zt, vz, e2.y));
        const float l2 = fmaf(dz, dz, e2.x);
        acc[j] = fmaf(l2 * rsqrtf(l2) * e2.z, val, acc[j]);
      } else {
        acc[j] += val;
      }
    }
  };
  if (n == 0) return;
  const float4(*entry)[kWords<kWeight>] = list;
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

template <int kRun, int kWeight, int kMinBlocks>
__global__ void __launch_bounds__(32 * kWX * kWY, kMinBlocks)
    bp_bilinear_zlane_kernel(const float4* __restrict__ table, int n_angles,
                             const float2* __restrict__ pairs, float* __restrict__ volt,
                             DeviceGeometry g, const float* __restrict__ angle_w) {
  __shared__ float4 s_list[kWX * kWY][34][kWords<kWeight>];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int bx, by;
  patch_tile(blockIdx.x, (g.nx + kWX - 1) / kWX, (g.ny + kWY - 1) / kWY, kPatch, kPatch, bx, by);
  const int x = bx * kWX + w % kWX, y = by * kWY + w / kWX;
  if (x >= g.nx || y >= g.ny) return;  // whole warp (the block has no barriers)
  const int z0 = blockIdx.y * (32 * kRun) + lane;
  const float xt = float(x - g.ox), yt = float(y - g.oy), zt = float(z0 - g.oz);
  const float zw0 = float(int(blockIdx.y) * (32 * kRun) - g.oz);
  const int cp = padded_cols(g), rp = padded_rows(g);
  const float vmin = float(-kRowPad - g.ov), vmax = float(g.rows - g.ov);
  float acc[kRun];
#pragma unroll
  for (int j = 0; j < kRun; ++j) acc[j] = 0.0f;
  for (int n0 = 0; n0 < n_angles; n0 += 32) {
    const int n = n0 + lane;
    bool ok = n < n_angles, inside = true;
    float4 e[3];
    if (ok) {
      const float4 t0 = __ldg(table + n), t1 = __ldg(table + n_angles + n);
      const float4 t2 = __ldg(table + 2 * (size_t)n_angles + n);
      const int theta = __float_as_int(t2.w);
      const float nw = fmaf(t1.w, yt, fmaf(t2.x, xt, t2.y));
      const float inw = 1.0f / nw;
      // (quotients, one rounding each, once per voxel column and angle: the positions'
      // errors are most of the result's)
      const float ut = fmaf(t0.x, yt, fmaf(t0.y, xt, t0.z)) / nw;
      const float fu0 = floorf(ut), fu = ut - fu0;
      // behind the source, or both columns off the detector: nothing to add
      ok = nw > 0.0f && fu0 >= float(-1 - g.ou) && fu0 <= float(g.cols - 1 - g.ou);
      const float dv = t0.w / nw;
      const float vb = fmaf(t1.x, yt, fmaf(t1.y, xt, t1.z)) / nw;  // row at z = 0
      // rows are monotone in z: inside if the warp's first and last voxel's are
      const float ra = fmaf(zw0, dv, vb), rb = fmaf(zw0 + float(32 * kRun - 1), dv, vb);
      const float margin = fmaf(4e-7f, fabsf(ra) + fabsf(rb), 0.01f);
      inside = fminf(ra, rb) >= vmin + margin && fmaxf(ra, rb) < vmax + 1.0f - margin;
      float K = t2.z;
      if (kWeight == kBilFdk) K = __ldg(angle_w + theta) * inw * inw;
      if (kWeight == kBilCone) {
        const float4 t3 = __ldg(table + 3 * (size_t)n_angles + n);
        const float dx = (xt - t3.z) * g.vs[2], dy = (yt - t3.y) * g.vs[1];
        e[2] = make_float4(fmaf(dx, dx, dy * dy), -t3.x * g.vs[0], K * inw * inw * inw, 0.0f);
        K = 1.0f;
      }
      const int iu = ok ? int(fu0) + g.ou : 0;
      const size_t col =
          reinterpret_cast<size_t>(pairs) +
          ((size_t(theta) * cp + size_t(iu + kColPad)) * rp + size_t(kRowPad + g.ov) -
           size_t(kFloorBits)) * sizeof(float2);
      const float wa = fmaf(-fu, K, K), wb = fu * K;
      e[0] = make_float4(wa, wa, wb, wb);
      e[1] = make_float4(dv, vb, __uint_as_float(unsigned(col)), __uint_as_float(unsigned(col >> 32)));
    }
    const unsigned mask = __ballot_sync(0xffffffffu, ok);
    const bool clamp = __any_sync(0xffffffffu, ok && !inside);
    if (ok) {
      const int slot = __popc(mask & ((1u << lane) - 1u));
#pragma unroll
      for (int i = 0; i < kWords<kWeight>; ++i) s_list[w][slot][i] = e[i];
      // the last: loads an angle ahead find it again
      if ((mask >> lane) == 1u) s_list[w][slot + 1][1] = s_list[w][slot + 2][1] = e[1];
    }
    __syncwarp();
    const unsigned column_bytes = unsigned(rp) * unsigned(sizeof(float2));
    if (clamp)
      add_angles<kRun, kWeight, true>(acc, s_list[w], __popc(mask), zt, g.vs[0], vmin, vmax, column_bytes);
    else
      add_angles<kRun, kWeight, false>(acc, s_list[w], __popc(mask), zt, g.vs[0], vmin, vmax, column_bytes);
    __syncwarp();  // the list is rewritten
  }
  float* out = volt + ((size_t)y * g.nx + x) * g.nz;
#pragma unroll
  for (int j = 0; j < kRun; ++j)
    if (z0 + 32 * j < g.nz) out[z0 + 32 * j] = acc[j];
}

template <int kRun, int kMinBlocks>
void launch_run(const tsgb_projector* p, const float2* pairs, float* volt, const float* angle_w,
                cudaStream_t stream) {
  const DeviceGeometry& g = p->g;
  const dim3 grid(unsigned((g.nx + kWX - 1) / kWX) * unsigned((g.ny + kWY - 1) / kWY),
                  unsigned((g.nz + 32 * kRun - 1) / (32 * kRun)));
  const float4* table = reinterpret_cast<const float4*>(p->d_bil_table);
  if (angle_w)
    bp_bilinear_zlane_kernel<kRun, kBilFdk, kMinBlocks><<<grid, 32 * kWX * kWY, 0, stream>>>(
        table, p->n_bil_fast, pairs, volt, g, angle_w);
  else if (g.kind == TSGB_CONE)
    bp_bilinear_zlane_kernel<kRun, kBilCone, kMinBlocks><<<grid, 32 * kWX * kWY, 0, stream>>>(
        table, p->n_bil_fast, pairs, volt, g, nullptr);
  else
    bp_bilinear_zlane_kernel<kRun, kBilParallel, kMinBlocks><<<grid, 32 * kWX * kWY, 0, stream>>>(
        table, p->n_bil_fast, pairs, volt, g, nullptr);
}

// Ranges along z and voxels per lane: at most 5, ranges of near-equal length.
int z_ranges(const DeviceGeometry& g) { return ((g.nz + 31) / 32 + 4) / 5; }
int z_run(const DeviceGeometry& g) {
  const int ranges = z_ranges(g);
  return ((g.nz + 31) / 32 + ranges - 1) / ranges;
}

int64_t pairs_bytes(const DeviceGeometry& g) {
  return (int64_t(padded_rows(g)) * padded_cols(g) * g.nangles * 8 + 255) / 256 * 256;
}

}  // namespace

// The times of this kernel over those of one thread per 16 voxels and quads, as factors:
//  * a voxel, cone 0.87, FDK 0.70, parallel 0.58 of the quads' time (256^3 / 360 angles:
//    5.63 / 6.35, 4.56 / 6.0 and 4.20 / 9.8 ms), 1.15 times that with 2 voxels a lane;
//  * lanes past the end of the volume and of the quads' runs of 16 (400 voxels take 480);
//  * rows finer than half a voxel: a load's 32 lanes spread over more lines (128 x 192^2 /
//    90 cone angles: 3, 4 and 6 rows a voxel 0.64 / 0.61, 0.75 / 0.67, 1.09 / 0.72 ms);
//  * the scratch volume, written and read once, as much as 4.7 angles (256^3, 1, 3, 16
//    and 64 cone angles: 110 / 35, 140 / 67, 337 / 277 and 1079 / 1117 us);
//  * the quad kernel's threads, too few for the GPU below about 3e5 (64^3 / 180: 85 / 474).
// Over 1140 sizes, angle counts and weights the faster of the two was missed by more than
// 5 % at 31, and by 27 % at most. Up to 32 voxels along z a wide slice keeps the quads
// (256^2 / 360: 16 voxels 0.79 ms against 1.09, 32 0.92 / 1.06); a slice or two on their
// own a less wide one (180 angles: 176^2 0.24 ms against 0.29, 150^2 0.24 / 0.21).
bool bilinear_zlane(const tsgb_projector* p, BilWeight weight) {
  const DeviceGeometry& g = p->g;
  if (thin_volume(p, 32, 1 << 15) || (g.nz <= 2 && int64_t(g.nx) * g.ny > 24000)) return false;
  const int run = z_run(g), quad_runs = (g.nz + 15) / 16;
  const double lanes = 32.0 * run * z_ranges(g) / (16.0 * quad_runs);
  const double voxel = (weight == kBilCone ? 0.87 : weight == kBilFdk ? 0.70 : 0.58) *
                       (run == 2 ? 1.15 : 1.0);
  const double rows = 1.0 + 0.37 * std::max(0.0, p->bil_row_step - 2.0);
  const double fill = std::min(1.0, std::cbrt(double(g.nx) * g.ny * quad_runs / 3e5));
  return fill * (voxel * lanes * rows + 4.7 / std::max(1, p->n_bil_fast)) < 1.0;
}

int64_t bilinear_bytes(const tsgb_projector* p) {
  // (a cone's projector serves the bilinear weights and FDK's)
  const bool cone = p->g.kind == TSGB_CONE;
  const bool a = bilinear_zlane(p, cone ? kBilCone : kBilParallel);
  const bool b = cone ? bilinear_zlane(p, kBilFdk) : a;
  const int64_t quads = int64_t(padded_rows(p->g)) * p->g.nangles * padded_cols(p->g) *
                        int64_t(4 * sizeof(float));
  return std::max(a && b ? int64_t(0) : quads,
                  a || b ? pairs_bytes(p->g) + bp_volume_bytes(p->g) : int64_t(0));
}

int launch_bilinear_zlane(const tsgb_projector* p, float* vol, const float* sino,
                          const float* angle_w, bool additive, float* workspace, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const DeviceGeometry& g = p->g;
  float2* pairs = reinterpret_cast<float2*>(workspace);
  float* volt = workspace + pairs_bytes(g) / 4;
  const dim3 grid(unsigned((padded_cols(g) + 31) / 32), unsigned((padded_rows(g) + 31) / 32),
                  unsigned(std::min(g.nangles, 65535)));
  bilinear_pairs_kernel<<<grid, dim3(32, 8), 0, stream>>>(sino, pairs, g);
  switch (z_run(g)) {
    case 1: launch_run<1, 12>(p, pairs, volt, angle_w, stream); break;
    case 2: launch_run<2, 10>(p, pairs, volt, angle_w, stream); break;
    case 3: launch_run<3, 8>(p, pairs, volt, angle_w, stream); break;
    case 4: launch_run<4, 8>(p, pairs, volt, angle_w, stream); break;
    default: launch_run<5, 8>(p, pairs, volt, angle_w, stream);
  }
  launch_zlane_out(g, additive ? 1 : 0, volt, nullptr, 0, g.nz, 0, g.nz, vol, nullptr, 1, stream);
  return int(cudaGetLastError());
}

}  // namespace tsgb
