// Distortion-correction remap on sm_100a.
//
// The reference models lens distortion with undistor
// (src/distortion_correction.cpp:20-61: Brown radial K1-K3 and tangential
// P1-P3 about (xc, yc), then a two-axis parallax scaling) and applies it to
// point coordinates only.  The tracking path here corrects whole frames: the
// corrected pixel (x, y) takes the distorted frame's value at the point xd
// with undistor(xd) = (x, y).  xd is found by 8 Newton steps from xd = (x, y)
// with a forward-difference Jacobian (step 1e-3 px), then sampled with the
// reference's cubic interpolant (src/interpol.cpp:42-86) and rounded half up.
//
// The inverse map depends only on the 14 parameters, so it is built once per
// parameter set into a resident FP64 map (16 bytes per pixel: 336 MB at
// 5616x3744, kept in HBM) and each frame is then a single gather pass.  This
// file is compiled with -fmad=false; the cos/sin of the two parallax angles
// come from the host.  With both, the device repeats the CPU restatement's
// FP64 operations exactly.
#include "ptk_cubic.cuh"
#include "ptk_internal.cuh"
#include "ptk_undistor.cuh"

namespace ptk {

__global__ void k_remap_build(Disto X, double2* map, int dimx, int dimy) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= dimx || y >= dimy) return;
  const double xu = (double)x, yu = (double)y;
  double xd = xu, yd = yu;
  const double h = 1e-3;
  for (int it = 0; it < 8; ++it) {
    double fx, fy, fx1, fy1, fx2, fy2;
    undistor_d(X, xd, yd, &fx, &fy);
    undistor_d(X, xd + h, yd, &fx1, &fy1);
    undistor_d(X, xd, yd + h, &fx2, &fy2);
    const double j11 = (fx1 - fx) / h, j21 = (fy1 - fy) / h;
    const double j12 = (fx2 - fx) / h, j22 = (fy2 - fy) / h;
    const double rx = fx - xu, ry = fy - yu;
    const double det = j11 * j22 - j12 * j21;
    xd = xd - (j22 * rx - j12 * ry) / det;
    yd = yd - (j11 * ry - j21 * rx) / det;
  }
  map[(size_t)y * dimx + x] = make_double2(xd, yd);
}

// One output row per blockIdx.y; a thread per output pixel.  The 4x4 support
// is gathered through the read-only path; rows of neighbouring threads are
// adjacent, so each warp's 16 loads touch a few cache lines.  Bound by the FP64
// and conversion pipes (57 and 13 operations a pixel, 120 and 104 cycles a warp;
// with every pixel and coordinate converted and the coefficients in FP64 about
// 105 and 23), then by the 22 bytes a pixel: 5616x3744, with the copy back, 248
// -> 168 us.
__global__ void k_remap_apply(const double2* __restrict__ map, const uint16_t* __restrict__ src,
                              uint16_t* __restrict__ dst, int pitch, int dimx, int dimy) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= dimx || y >= dimy) return;
  const double2 m = map[(size_t)y * dimx + x];
  int out = 0;
  if (m.x >= 1.0 && m.y >= 1.0 && m.x < (double)(dimx - 2) && m.y < (double)(dimy - 2)) {
    int ix, iy;
    const double x01 = split(m.x, &ix), y01 = split(m.y, &iy);
    const double y2 = y01 * y01;
    const uint16_t* p0 = src + (size_t)(iy - 1) * pitch + (ix - 1);
    const uint16_t *p1 = p0 + pitch, *p2 = p1 + pitch, *p3 = p2 + pitch;
    double arr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      arr[i] = cubic_px_twice(__ldg(p0 + i), __ldg(p1 + i), __ldg(p2 + i), __ldg(p3 + i), y01, y2);
    const int r = __double2int_rd(__fma_rn(0.5, cubic1_fast(arr[0], arr[1], arr[2], arr[3], x01), 0.5));
    out = min(max(r, 0), 65535);
  }
  dst[(size_t)y * pitch + x] = (uint16_t)out;
}

void launch_remap_build(const double* params14, const double* trig4, double2* map, int dimx, int dimy,
                        cudaStream_t s) {
  Disto X;
  for (int i = 0; i < 14; ++i) X.p[i] = params14[i];
  for (int i = 0; i < 4; ++i) X.trig[i] = trig4[i];
  dim3 grid((dimx + 127) / 128, dimy);
  k_remap_build<<<grid, 128, 0, s>>>(X, map, dimx, dimy);
}

void launch_remap_apply(const double2* map, const uint16_t* src, uint16_t* dst, int pitch, int dimx, int dimy,
                        cudaStream_t s) {
  dim3 grid((dimx + 127) / 128, dimy);
  k_remap_apply<<<grid, 128, 0, s>>>(map, src, dst, pitch, dimx, dimy);
}

}  // namespace ptk
