// Detector supersampling (tomosipo/astra.py:80-98, doc/topics/operator.rst:69-86).
//
// With detector supersampling d the forward projection averages d x d rays
// per detector pixel, at sub-pixel offsets ((s + 0.5) / d - 0.5) pixels. Those
// are exactly the pixel centres of a d-times finer detector (rows * d x
// cols * d, pixel vectors det_v / d and det_u / d), so a supersampled
// projector runs its forward projection on that fine detector and bins each
// d x d block (times 1 / d^2); its matched backprojection spreads each pixel's
// value times 1 / d^2 over its block and backprojects on the fine detector,
// which is the exact transpose. The backprojection's first kernel spreads the
// values as it reads them (SinoSource).
#include <cuda_runtime.h>

#include <algorithm>

#include "tsgb_internal.h"

namespace tsgb {
namespace {

// coarse[iv][t][iu] (+)= sum over the d x d block of fine, times 1 / d^2. One warp
// per detector line of an angle: the line index is divided once, not once per pixel
// (a thread per pixel, with three 64-bit divisions, took 41 us for 160 x 200 x 304
// pixels of 2 x 2).
__global__ void __launch_bounds__(256)
    ss_bin_kernel(const float* __restrict__ fine, float* __restrict__ coarse, int rows,
                  int nangles, int cols, int d, float scale, int additive) {
  const long long lines = (long long)rows * nangles, fcols = (long long)cols * d;
  for (long long line = blockIdx.x * 8LL + threadIdx.y; line < lines; line += gridDim.x * 8LL) {
    const long long iv = line / nangles, t = line - iv * nangles;
    const float* first = fine + (iv * d * nangles + t) * fcols;
    float* out = coarse + line * cols;
    for (int iu = threadIdx.x; iu < cols; iu += 32) {
      float s = 0.0f;
      for (int s1 = 0; s1 < d; ++s1) {
        const float* row = first + s1 * nangles * fcols + (long long)iu * d;
        for (int s2 = 0; s2 < d; ++s2) s += __ldg(row + s2);
      }
      s *= scale;
      out[iu] = additive ? out[iu] + s : s;
    }
  }
}

}  // namespace

int launch_ss_bin(const tsgb_projector* p, const float* fine, float* coarse, bool additive,
                  void* stream) {
  const DeviceGeometry& g = p->g;
  const int d = p->det_ss;
  const long long blocks = ((long long)g.rows * g.nangles + 7) / 8;
  ss_bin_kernel<<<unsigned(std::min(blocks, 152LL * 64)), dim3(32, 8), 0,
                  static_cast<cudaStream_t>(stream)>>>(fine, coarse, g.rows, g.nangles, g.cols, d,
                                                       1.0f / float(d * d), additive ? 1 : 0);
  return int(cudaGetLastError());
}

}  // namespace tsgb
