// Subpixel refinement on sm_100a: the NCC objective through image
// interpolation, its adjoint gradient, and a per-grain Powell minimiser.
//
// The objective (objective_exact) follows the reference's FP64 operations
// (src/p-tracker.cpp:1018-1088, src/interpol.cpp:19-144) in their order and
// without FMA contraction (this file is compiled with -fmad=false): the
// interpolated values are computed in parallel, and its sums are those of the
// reference's loops over the pattern points in point order, rounded after
// every point, computed by the whole block (ptk_seqsum.cuh); cos / sin come
// from ptk_crtrig.cuh.  Inside Powell the frame region under the grain is
// staged in shared memory.
//
// One CTA of kSubpixThreads refines one grain.  The Powell driver
// (follow_pattern_subpixel_xyR, src/p-tracker.cpp:1090-1128; the minimiser
// comes from the un-vendored toofus powell_nr3.hpp, src/p-tracker.hpp:51) runs
// redundantly on every thread with block-uniform control flow: each objective
// value is produced by a block reduction and broadcast, so every thread takes
// the same branches.  The algorithm is Powell's direction-set method with
// golden-ratio bracketing and Brent's parabolic line minimiser; its constants
// and tests match the CPU oracle's restatement exactly.
#include <climits>
#include <type_traits>

#include "ptk_crtrig.cuh"
#include "ptk_cubic.cuh"
#include "ptk_internal.cuh"
#include "ptk_seqsum.cuh"

namespace ptk {

namespace {

constexpr double kGold = 1.6180339887498949;
constexpr double kCGold = 0.3819660112501051;
constexpr double kLineRelTol = 1.0e-4;
constexpr double kLineAbsTol = 1.0e-10;
constexpr int kBracketMaxIter = 60;
constexpr int kBrentMaxIter = 100;
constexpr int kPowellMaxIter = 200;
constexpr double kTiny = 1.0e-25;

__device__ __forceinline__ double pixd(const FrameDev& f, int x, int y) {
  return (double)__ldg(&f.pix[(size_t)y * f.pitch + x]);
}

// CubicInterpolate, src/interpol.cpp:42-53
__device__ __forceinline__ double cubic1(double p0, double p1, double p2, double p3, double x) {
  const double f0 = p1, f1 = p2;
  const double fp0 = 0.5 * (p2 - p0);
  const double fp1 = 0.5 * (p3 - p1);
  const double d = f0, c = fp0;
  const double b = -3.0 * f0 + 3.0 * f1 - 2.0 * fp0 - fp1;
  const double a = 2.0 * f0 - 2.0 * f1 + fp0 + fp1;
  const double x2 = x * x;
  return (a * x2 * x + b * x2 + c * x + d);
}

// derivative of cubic1 with respect to x
__device__ __forceinline__ double cubic1_dx(double p0, double p1, double p2, double p3, double x) {
  const double f0 = p1, f1 = p2;
  const double fp0 = 0.5 * (p2 - p0);
  const double fp1 = 0.5 * (p3 - p1);
  const double c = fp0;
  const double b = -3.0 * f0 + 3.0 * f1 - 2.0 * fp0 - fp1;
  const double a = 2.0 * f0 - 2.0 * f1 + fp0 + fp1;
  return (3.0 * a * x * x + 2.0 * b * x + c);
}

// Catmull-Rom weight of control point k at x (cubic1 is linear in p)
__device__ __forceinline__ void cubic_weights(double x, double w[4]) {
  const double x2 = x * x, x3 = x2 * x;
  w[0] = -0.5 * x3 + x2 - 0.5 * x;
  w[1] = 1.5 * x3 - 2.5 * x2 + 1.0;
  w[2] = -1.5 * x3 + 2.0 * x2 + 0.5 * x;
  w[3] = 0.5 * x3 - 0.5 * x2;
}

// QuinticInterpolate, src/interpol.cpp:89-111
__device__ __forceinline__ double quintic1(double p0, double p1, double p2, double p3, double x) {
  const double f0 = p1, f1 = p2;
  const double fp0 = 0.5 * (p2 - p0);
  const double fp1 = 0.5 * (p3 - p1);
  const double fs0 = p0 - 2.0 * p1 + p2;
  const double fs1 = p1 - 2.0 * p2 + p3;
  const double f = f0, e = fp0, d = 0.5 * fs0;
  const double c = 0.5 * (fs1 - 8.0 * fp1 + 20.0 * f1 - 3.0 * fs0 - 12.0 * fp0 - 20.0 * f0);
  const double b = 15.0 * f0 + 8.0 * fp0 + 1.5 * fs0 - 15.0 * f1 + 7.0 * fp1 - fs1;
  const double a = f1 - b - c - 0.5 * fs0 - fp0 - f0;
  const double x2 = x * x, x4 = x2 * x2;
  return (a * x4 * x + b * x4 + c * x2 * x + d * x2 + e * x + f);
}

// Whether the cubic's 4x4 support of (x, y) lies in the frame.
__device__ __forceinline__ bool cubic_inside(const FrameDev& f, double x, double y) {
  return x >= 1.0 && y >= 1.0 && x < (double)(f.dimx - 2) && y < (double)(f.dimy - 2);
}

// image_interp*::getValue (src/interpol.cpp:21-39, 55-86, 113-144).  The
// reference reads out of bounds when the support leaves the frame; here the
// support is clamped into the frame and *clamped is set.
__device__ double interp(const FrameDev& f, int kind, double x, double y, bool* clamped) {
  if (kind == PTK_INTERP_CUBIC && cubic_inside(f, x, y)) {
    int ix, iy;
    const double x01 = split(x, &ix), y01 = split(y, &iy), y2 = y01 * y01;
    const uint16_t* p = f.pix + (size_t)(iy - 1) * f.pitch + (ix - 1);
    double arr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      arr[i] = cubic_px_twice(__ldg(p + i), __ldg(p + f.pitch + i), __ldg(p + 2 * f.pitch + i), __ldg(p + 3 * f.pitch + i),
                              y01, y2);
    return 0.5 * cubic1_fast(arr[0], arr[1], arr[2], arr[3], x01);
  }
  int ix = (int)floor(x);
  int iy = (int)floor(y);
  const double x01 = x - (double)ix;
  const double y01 = y - (double)iy;
  const int lo = kind == PTK_INTERP_LINEAR ? 0 : 1;
  const int hi = kind == PTK_INTERP_LINEAR ? 1 : 2;
  if (ix - lo < 0 || iy - lo < 0 || ix + hi >= f.dimx || iy + hi >= f.dimy || !(x == x) || !(y == y)) {
    *clamped = true;
    ix = min(max(ix, lo), f.dimx - 1 - hi);
    iy = min(max(iy, lo), f.dimy - 1 - hi);
  }
  if (kind == PTK_INTERP_LINEAR) {
    const double a0 = pixd(f, ix, iy), a1 = pixd(f, ix, iy + 1);
    const double b0 = pixd(f, ix + 1, iy), b1 = pixd(f, ix + 1, iy + 1);
    const double r0 = (a1 - a0) * y01 + a0;
    const double r1 = (b1 - b0) * y01 + b0;
    return (r1 - r0) * x01 + r0;
  }
  double arr[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int xx = ix - 1 + i;
    const double q0 = pixd(f, xx, iy - 1), q1 = pixd(f, xx, iy), q2 = pixd(f, xx, iy + 1), q3 = pixd(f, xx, iy + 2);
    arr[i] = kind == PTK_INTERP_QUINTIC ? quintic1(q0, q1, q2, q3, y01) : cubic1(q0, q1, q2, q3, y01);
  }
  return kind == PTK_INTERP_QUINTIC ? quintic1(arr[0], arr[1], arr[2], arr[3], x01)
                                    : cubic1(arr[0], arr[1], arr[2], arr[3], x01);
}

// Cubic value and its partial derivatives at (x, y).
__device__ double interp_cubic_grad(const FrameDev& f, double x, double y, double* gx, double* gy, bool* clamped) {
  if (cubic_inside(f, x, y)) {  // everything below on doubled values
    int ix, iy;
    const double x01 = split(x, &ix), y01 = split(y, &iy), y2 = y01 * y01;
    const uint16_t* p = f.pix + (size_t)(iy - 1) * f.pitch + (ix - 1);
    double arr[4], darr[4], w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      arr[i] = cubic_px_twice(__ldg(p + i), __ldg(p + f.pitch + i), __ldg(p + 2 * f.pitch + i), __ldg(p + 3 * f.pitch + i),
                              y01, y2, &darr[i]);
    cubic_weights(x01, w);
    *gx = 0.5 * cubic1_dx(arr[0], arr[1], arr[2], arr[3], x01);
    *gy = 0.5 * (w[0] * darr[0] + w[1] * darr[1] + w[2] * darr[2] + w[3] * darr[3]);
    return 0.5 * cubic1_fast(arr[0], arr[1], arr[2], arr[3], x01);
  }
  int ix = (int)floor(x);
  int iy = (int)floor(y);
  const double x01 = x - (double)ix;
  const double y01 = y - (double)iy;
  if (ix - 1 < 0 || iy - 1 < 0 || ix + 2 >= f.dimx || iy + 2 >= f.dimy || !(x == x) || !(y == y)) {
    *clamped = true;
    ix = min(max(ix, 1), f.dimx - 3);
    iy = min(max(iy, 1), f.dimy - 3);
  }
  double arr[4], darr[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int xx = ix - 1 + i;
    const double q0 = pixd(f, xx, iy - 1), q1 = pixd(f, xx, iy), q2 = pixd(f, xx, iy + 1), q3 = pixd(f, xx, iy + 2);
    arr[i] = cubic1(q0, q1, q2, q3, y01);
    darr[i] = cubic1_dx(q0, q1, q2, q3, y01);
  }
  double w[4];
  cubic_weights(x01, w);
  *gx = cubic1_dx(arr[0], arr[1], arr[2], arr[3], x01);
  *gy = w[0] * darr[0] + w[1] * darr[1] + w[2] * darr[2] + w[3] * darr[3];
  return cubic1(arr[0], arr[1], arr[2], arr[3], x01);
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < NT / 32; ++k) s += red[k];
  return s;
}

// Per-grain constants of the objective.
struct ObjGrain {
  int b, P;
  double xref, yref;  // (double)refcoord + d, in the reference's order
  double drot;
  double mean0, c0c0;
};

// One block's grain and its exact objective, in shared memory: everything an
// evaluation needs besides the point X.  The dynamic shared memory holds, per
// pattern point, the sample of the current evaluation and, where they fit, the
// centred reference value d0 = I0 - mean0 (doubles), and before them the
// current-frame region around the grain (uint16, row-major, staged once; w = 0:
// none).
struct ExactObj {
  const short2* pat0;  // the grain's pattern points
  const uint16_t* w0;  // and their reference values
  FrameDev cur;
  int interp, P;
  SeqPlan one, two;    // how the sums' terms are split
  double xref, yref, drot, mean0, c0c0, inv_num_pix;
  double disp_max, stiffness;
  int reach;           // every point lies within reach - 1 pixels of the pattern's origin
  int x0, y0, w, h;    // the staged region
  int v_at, d0_at;     // bytes from the start of the dynamic shared memory
  int clamped;
  double rot, c1, s1;  // the last rotation angle, its cosine and sine
  double X[3];         // the point to evaluate next
  int done;            // no further one
};
__device__ __forceinline__ ExactObj& exact_obj() {
  __shared__ ExactObj s;
  return s;
}
extern __shared__ __align__(16) unsigned char s_subpix[];
__device__ __forceinline__ double* obj_v(const ExactObj& ex) { return reinterpret_cast<double*>(s_subpix + ex.v_at); }
__device__ __forceinline__ double* obj_d0(const ExactObj& ex) { return reinterpret_cast<double*>(s_subpix + ex.d0_at); }

// Terms of the objective's sums, in point order (seq_sums).
struct SumV {  // sum v
  const double* v;
  struct Of {
    const double* v;
    __device__ __forceinline__ double operator()(int i) const { return v[i]; }
  };
  __device__ __forceinline__ Of of(int) const { return Of{v}; }
};
// d0 of a point: staged, or from the reference value in global memory
// (patterns whose values and d0 exceed the shared memory, and single
// evaluations, which would read each staged value only three times).
struct RefStaged {
  const double* d0;
  __device__ __forceinline__ explicit RefStaged(const ExactObj& ex) : d0(obj_d0(ex)) {}
  __device__ __forceinline__ double operator()(int i) const { return d0[i]; }
};
struct RefGlobal {
  const uint16_t* w0;
  double mean0;
  int last;
  __device__ __forceinline__ explicit RefGlobal(const ExactObj& ex) : w0(ex.w0), mean0(ex.mean0), last(ex.P - 1) {}
  __device__ __forceinline__ double operator()(int i) const { return u16d(w0[min(i, last)]) - mean0; }
};
template <class Ref>
struct SumC {  // sum d0 d1 and sum d1^2
  const double* d1;
  Ref d0;
  struct Of {
    const double* d1;
    Ref d0;
    int n;
    __device__ __forceinline__ double operator()(int i) const {
      const double d = d1[i];
      return (n == 0 ? d0(i) : d) * d;
    }
  };
  __device__ __forceinline__ Of of(int n) const { return Of{d1, d0, n}; }
};
template <>
struct SumC<RefStaged> {
  const double* d1;
  RefStaged d0;
  struct Of {
    const double *d1, *f;
    __device__ __forceinline__ double operator()(int i) const { return f[i] * d1[i]; }
  };
  __device__ __forceinline__ Of of(int n) const { return Of{d1, n == 0 ? d0.d0 : d1}; }
};
template <class Ref>
struct SumA {  // sum d0^2: C0C0 of do_precomputations (src/p-tracker.cpp:646-651)
  Ref d0;
  struct Of {
    Ref d0;
    __device__ __forceinline__ double operator()(int i) const {
      const double d = d0(i);
      return d * d;
    }
  };
  __device__ __forceinline__ Of of(int) const { return Of{d0}; }
};

// Samples of all points, by the block, where every 4x4 support lies in the
// staged region.  Two points per thread at a time (their chains of dependent
// operations, about 30 long, overlap), the next two's offsets loaded before.
template <int NT, int KIND>
__device__ __forceinline__ void sample_staged(const ExactObj& ex, double xpix1, double ypix1, double c1, double s1) {
  constexpr int kAt = 2;
  const uint16_t* patch = reinterpret_cast<const uint16_t*>(s_subpix);
  double* v = obj_v(ex);
  const short2* pat0 = ex.pat0;
  const int P = ex.P, w = ex.w, at0 = -(ex.y0 + 1) * w - (ex.x0 + 1);
  short2 q[kAt];
#pragma unroll
  for (int k = 0; k < kAt; ++k) q[k] = pat0[min((int)threadIdx.x + k * NT, P - 1)];
  for (int i = threadIdx.x; i < P; i += kAt * NT) {
    double x01[kAt], y01[kAt], val[kAt];
    const uint16_t* px[kAt];
#pragma unroll
    for (int k = 0; k < kAt; ++k) {
      const double x = (double)q[k].x, y = (double)q[k].y;
      const double xs = xpix1 + c1 * x + s1 * y;
      const double ys = ypix1 - s1 * x + c1 * y;
      int ix, iy;
      x01[k] = split(xs, &ix);
      y01[k] = split(ys, &iy);
      px[k] = patch + iy * w + ix + at0;  // the support's corner (ix - 1, iy - 1)
      q[k] = pat0[min(i + (kAt + k) * NT, P - 1)];
    }
#pragma unroll
    for (int k = 0; k < kAt; ++k) {
      const uint16_t* p = px[k];
      if constexpr (KIND == PTK_INTERP_LINEAR) {
        const double a0 = u16d(p[w + 1]), a1 = u16d(p[2 * w + 1]), b0 = u16d(p[w + 2]), b1 = u16d(p[2 * w + 2]);
        const double r0 = (a1 - a0) * y01[k] + a0;
        const double r1 = (b1 - b0) * y01[k] + b0;
        val[k] = (r1 - r0) * x01[k] + r0;
      } else if constexpr (KIND == PTK_INTERP_CUBIC) {
        const double y2 = y01[k] * y01[k];
        double arr[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          arr[j] = cubic_px_twice(p[j], p[w + j], p[2 * w + j], p[3 * w + j], y01[k], y2);
        val[k] = 0.5 * cubic1_fast(arr[0], arr[1], arr[2], arr[3], x01[k]);
      } else {
        double arr[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          arr[j] = quintic1(u16d(p[j]), u16d(p[w + j]), u16d(p[2 * w + j]), u16d(p[3 * w + j]), y01[k]);
        val[k] = quintic1(arr[0], arr[1], arr[2], arr[3], x01[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < kAt; ++k)
      if (i + k * NT < P) v[i + k * NT] = val[k];
  }
}

// NCC_to_minimize_xyR (src/p-tracker.cpp:1018-1088): the sample positions
// xpix1 + c1 x + s1 y and ypix1 - s1 x + c1 y and the interpolators in the
// reference's operations and order, every product and sum rounded separately
// (this file is compiled without FMA contraction), cos / sin correctly
// rounded (ptk_crtrig.cuh) where the host C library is within an ulp.  The
// block's threads interpolate the points in parallel into shared memory (66 FP64
// operations a point, and 18 conversions on their own pipe), then form the sums of the reference's two loops over them,
//     mean1 = (sum v) * (1 / P),  C0C1 = sum d0 (v - mean1),  C1C1 = sum (v - mean1)^2
// (d0 = I0 - mean0), each rounded after every point in point order as those
// loops round it (seq_sums), so that the value is the reference's bit for bit
// and Powell takes the reference's path even where the objective is flat.
// Called by every thread of the block, with X in exact_obj().X; the value is the
// first warp's return.  Not inlined: Powell calls it from a dozen places.
template <int NT, class Ref>
__device__ __noinline__ double objective_exact() {
  ExactObj& ex = exact_obj();
  const double X0 = ex.X[0], X1 = ex.X[1], X2 = ex.X[2];
  const int tid = threadIdx.x;
  const double xpix1 = ex.xref + X0;
  const double ypix1 = ex.yref + X1;
  const double rot = ex.drot + X2;
  if (!(rot == ex.rot)) {  // block-uniform: the line searches along x and y keep the angle
    __syncthreads();
    if (tid == 0) {
      ex.c1 = crtrig::cr_cos(rot);
      ex.rot = rot;
    }
    if (tid == 32) ex.s1 = crtrig::cr_sin(rot);
    __syncthreads();
  }
  const double c1 = ex.c1, s1 = ex.s1;
  // block-uniform: every sample's 4x4 support lies in the staged region
  const double reach = (double)ex.reach;
  const bool inside = xpix1 - reach >= (double)(ex.x0 + 1) && ypix1 - reach >= (double)(ex.y0 + 1) &&
                      xpix1 + reach <= (double)(ex.x0 + ex.w - 2) && ypix1 + reach <= (double)(ex.y0 + ex.h - 2);
  if (inside) {
    if (ex.interp == PTK_INTERP_CUBIC) sample_staged<NT, PTK_INTERP_CUBIC>(ex, xpix1, ypix1, c1, s1);
    else if (ex.interp == PTK_INTERP_LINEAR) sample_staged<NT, PTK_INTERP_LINEAR>(ex, xpix1, ypix1, c1, s1);
    else sample_staged<NT, PTK_INTERP_QUINTIC>(ex, xpix1, ypix1, c1, s1);
  } else {
    bool clamped = false;
    double* v = obj_v(ex);
    for (int i = tid; i < ex.P; i += NT) {
      const short2 q = ex.pat0[i];
      const double x = (double)q.x, y = (double)q.y;
      const double xs = xpix1 + c1 * x + s1 * y;
      const double ys = ypix1 - s1 * x + c1 * y;
      v[i] = interp(ex.cur, ex.interp, xs, ys, &clamped);
    }
    if (clamped) ex.clamped = 1;
  }
  __syncthreads();
  const SeqSumScratch<NT>& sc = seq_scratch<NT>();
  seq_sums<NT, 1>(ex.P, ex.one, SumV{obj_v(ex)});
  __syncthreads();
  const double mean1 = sc.out[0] * ex.inv_num_pix;
  {  // d1 = v - mean1 in v's place
    double* v = obj_v(ex);
    for (int i = tid; i < ex.P; i += NT) v[i] -= mean1;
  }
  __syncthreads();
  seq_sums<NT, 2>(ex.P, ex.two, SumC<Ref>{obj_v(ex), Ref(ex)});
  __syncthreads();
  if (tid >= 32) return 0.0;
  const double ncc = sc.out[0] / sqrt(ex.c0c0 * sc.out[1]);
  double W = 1.0;
  const double d2 = X0 * X0 + X1 * X1;
  if (!(ex.disp_max > 0.0 && d2 < 0.999999 * ex.disp_max * ex.disp_max)) {  // (well below it no root is needed)
    const double disp = sqrt(d2);
    if (disp > ex.disp_max) W = ex.stiffness * (disp - ex.disp_max) + 1.0;
  }
  return (1.0 - ncc) * W;
}

// Sets the block's grain up and forms C0C0 in the reference's order.
template <int NT, class Ref>
__device__ __forceinline__ void exact_begin(const ObjGrain& o, const GrainsDev& g, const FrameDev& cur,
                                            const SubpixParams& sp, int reach, int x0, int y0, int w, int h, int v_at,
                                            int d0_at) {
  ExactObj& ex = exact_obj();
  if (std::is_same<Ref, RefStaged>::value) {
    double* d0 = reinterpret_cast<double*>(s_subpix + d0_at);
    for (int i = threadIdx.x; i < o.P; i += NT) d0[i] = u16d(g.w0[o.b + i]) - o.mean0;
  }
  if (threadIdx.x == 0) {
    ex.pat0 = g.pat0 + o.b;
    ex.w0 = g.w0 + o.b;
    ex.mean0 = o.mean0;
    ex.cur = cur;
    ex.interp = sp.interp;
    ex.P = o.P;
    ex.one = seq_plan(o.P, kSeqThreads<NT, 1>);
    ex.two = seq_plan(o.P, kSeqThreads<NT, 2>);
    ex.xref = o.xref;
    ex.yref = o.yref;
    ex.drot = o.drot;
    ex.inv_num_pix = 1.0 / (double)o.P;
    ex.disp_max = sp.disp_max;
    ex.stiffness = sp.stiffness;
    ex.reach = reach;
    ex.x0 = x0;
    ex.y0 = y0;
    ex.w = w;
    ex.h = h;
    ex.v_at = v_at;
    ex.d0_at = d0_at;
    ex.clamped = 0;
    ex.done = 0;
    ex.rot = __longlong_as_double(0x7ff8000000000000ll);
  }
  __syncthreads();
  seq_sums<NT, 1>(o.P, ex.one, SumA<Ref>{Ref(ex)});
  __syncthreads();
  if (threadIdx.x == 0) ex.c0c0 = seq_scratch<NT>().out[0];
  __syncthreads();
}

// Objective and its gradient (adjoint through the cubic interpolant and the
// rotation; no reference counterpart).  dNCC/dv_i = (a_i - (C01/C11) b_i) / den
// with a, b the centred reference and current values; the mean terms cancel.
template <int NT>
__device__ double objective_grad(const GrainsDev& g, const FrameDev& cur, const SubpixParams& sp,
                                 const ObjGrain& o, const double X[3], double* vals, double* red, double grad[3],
                                 bool* clamped) {
  const double xpix1 = o.xref + X[0];
  const double ypix1 = o.yref + X[1];
  const double rot = o.drot + X[2];
  double s1, c1;
  sincos(rot, &s1, &c1);
  double* gxs = vals + o.P;
  double* gys = vals + 2 * o.P;
  double sum = 0.0;
  for (int i = threadIdx.x; i < o.P; i += NT) {
    const short2 q = g.pat0[o.b + i];
    const double x = (double)q.x, y = (double)q.y;
    const double xs = xpix1 + c1 * x + s1 * y;
    const double ys = ypix1 - s1 * x + c1 * y;
    double gx, gy;
    const double v = interp_cubic_grad(cur, xs, ys, &gx, &gy, clamped);
    vals[i] = v;
    gxs[i] = gx;
    gys[i] = gy;
    sum += v;
  }
  const double mean1 = block_sum<NT>(sum, red) * (1.0 / (double)o.P);
  double c01 = 0.0, c11 = 0.0;
  for (int i = threadIdx.x; i < o.P; i += NT) {
    const double d1 = vals[i] - mean1;
    const double d0 = (double)g.w0[o.b + i] - o.mean0;
    c01 += d0 * d1;
    c11 += d1 * d1;
  }
  c01 = block_sum<NT>(c01, red);
  c11 = block_sum<NT>(c11, red);
  const double den = sqrt(o.c0c0 * c11);
  const double ncc = c01 / den;
  const double ratio = c01 / c11;
  double G0 = 0.0, G1 = 0.0, G2 = 0.0;
  for (int i = threadIdx.x; i < o.P; i += NT) {
    const short2 q = g.pat0[o.b + i];
    const double x = (double)q.x, y = (double)q.y;
    const double d1 = vals[i] - mean1;
    const double d0 = (double)g.w0[o.b + i] - o.mean0;
    const double dn = (d0 - ratio * d1) / den;
    G0 += dn * gxs[i];
    G1 += dn * gys[i];
    G2 += dn * (gxs[i] * (-s1 * x + c1 * y) + gys[i] * (-c1 * x - s1 * y));
  }
  G0 = block_sum<NT>(G0, red);
  G1 = block_sum<NT>(G1, red);
  G2 = block_sum<NT>(G2, red);
  double W = 1.0, dW0 = 0.0, dW1 = 0.0;
  const double disp = sqrt(X[0] * X[0] + X[1] * X[1]);
  if (disp > sp.disp_max) {
    W = sp.stiffness * (disp - sp.disp_max) + 1.0;
    dW0 = sp.stiffness * X[0] / disp;
    dW1 = sp.stiffness * X[1] / disp;
  }
  const double f0 = 1.0 - ncc;
  grad[0] = -G0 * W + f0 * dW0;
  grad[1] = -G1 * W + f0 * dW1;
  grad[2] = -G2 * W;
  return f0 * W;
}

__device__ ObjGrain load_grain(const GrainsDev& g, int gi) {
  ObjGrain o;
  o.b = g.pstart[gi];
  o.P = g.pstart[gi + 1] - o.b;
  o.xref = (double)g.refx[gi] + g.dx[gi];
  o.yref = (double)g.refy[gi] + g.dy[gi];
  o.drot = g.drot[gi];
  o.mean0 = g.mean0[gi];
  o.c0c0 = g.c0c0[gi];
  return o;
}

// --- Powell on the device, block-uniform ----------------------------------
// The first warp runs Powell, the others take part in its evaluations only (the
// minimiser's scalar FP64 work, repeated by every warp, would compete with the
// samples of the other blocks on the SM).
template <int NT, class Ref>
struct PowellEval {
  __device__ __forceinline__ double operator()(const double X[3]) const {
    ExactObj& ex = exact_obj();
    if (threadIdx.x < 3) ex.X[threadIdx.x] = threadIdx.x == 0 ? X[0] : (threadIdx.x == 1 ? X[1] : X[2]);
    __syncthreads();
    return objective_exact<NT, Ref>();
  }
};

// f0: the objective at p, which is g(0): p + 0 dir is p bit for bit for finite
// directions (p itself was reached as p + alpha dir, with the same roundings).
template <class F>
__device__ double line_minimize(F& f, const double p[3], const double dir[3], double f0, double* gmin) {
  auto g = [&](double alpha) {
    double t[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) t[j] = p[j] + alpha * dir[j];
    return f(t);
  };
  double a = 0.0, b = 1.0;
  double ga = isfinite(dir[0]) && isfinite(dir[1]) && isfinite(dir[2]) ? f0 : g(a), gb = g(b);
  if (gb > ga) {
    double t = a;
    a = b;
    b = t;
    t = ga;
    ga = gb;
    gb = t;
  }
  double c = b + kGold * (b - a);
  double gc = g(c);
  int it = 0;
  while (gc < gb && it < kBracketMaxIter) {
    a = b;
    ga = gb;
    b = c;
    gb = gc;
    c = b + kGold * (b - a);
    gc = g(c);
    ++it;
  }
  double lo = a < c ? a : c;
  double hi = a < c ? c : a;
  double x = b, w = b, v = b;
  double fx = gb, fw = gb, fv = gb;
  double d = 0.0, e = 0.0;
  for (int iter = 0; iter < kBrentMaxIter; ++iter) {
    const double m = 0.5 * (lo + hi);
    const double tol1 = kLineRelTol * fabs(x) + kLineAbsTol;
    const double tol2 = 2.0 * tol1;
    if (fabs(x - m) <= tol2 - 0.5 * (hi - lo)) break;
    bool golden = true;
    if (fabs(e) > tol1) {
      double r = (x - w) * (fx - fv);
      double q = (x - v) * (fx - fw);
      double pp = (x - v) * q - (x - w) * r;
      q = 2.0 * (q - r);
      if (q > 0.0) pp = -pp;
      else q = -q;
      const double eprev = e;
      e = d;
      if (fabs(pp) < fabs(0.5 * q * eprev) && pp > q * (lo - x) && pp < q * (hi - x)) {
        d = pp / q;
        const double u = x + d;
        if (u - lo < tol2 || hi - u < tol2) d = (m - x) >= 0.0 ? tol1 : -tol1;
        golden = false;
      }
    }
    if (golden) {
      e = (x >= m) ? lo - x : hi - x;
      d = kCGold * e;
    }
    const double u = (fabs(d) >= tol1) ? x + d : x + (d >= 0.0 ? tol1 : -tol1);
    const double fu = g(u);
    if (fu <= fx) {
      if (u >= x) lo = x;
      else hi = x;
      v = w;
      fv = fw;
      w = x;
      fw = fx;
      x = u;
      fx = fu;
    } else {
      if (u < x) lo = u;
      else hi = u;
      if (fu <= fw || w == x) {
        v = w;
        fv = fw;
        w = u;
        fw = fu;
      } else if (fu <= fv || v == x || v == w) {
        v = u;
        fv = fu;
      }
    }
  }
  *gmin = fx;
  return x;
}

template <class F>
__device__ void powell_minimize(F& f, double p[3], const double step[3], double ftol, double* fret_out) {
  double dirs[3][3] = {{step[0], 0.0, 0.0}, {0.0, step[1], 0.0}, {0.0, 0.0, step[2]}};
  double pstart[3] = {p[0], p[1], p[2]};
  double fret = f(p);
  if (!isfinite(fret)) {  // flat window: NCC undefined, nothing to minimise
    *fret_out = fret;
    return;
  }
  for (int iter = 0; iter < kPowellMaxIter; ++iter) {
    const double fp = fret;
    int ibig = 0;
    double del = 0.0;
    for (int i = 0; i < 3; ++i) {
      const double fptt = fret;
      double gmin;
      const double alpha = line_minimize(f, p, dirs[i], fret, &gmin);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        dirs[i][j] *= alpha;
        p[j] += dirs[i][j];
      }
      fret = gmin;
      if (fptt - fret > del) {
        del = fptt - fret;
        ibig = i;
      }
    }
    if (2.0 * (fp - fret) <= ftol * (fabs(fp) + fabs(fret)) + kTiny) break;
    double ptt[3], xit[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      ptt[j] = 2.0 * p[j] - pstart[j];
      xit[j] = p[j] - pstart[j];
      pstart[j] = p[j];
    }
    const double fe = f(ptt);
    if (fe < fp) {
      const double t1 = fp - fret - del;
      const double t = 2.0 * (fp - 2.0 * fret + fe) * t1 * t1 - del * (fp - fe) * (fp - fe);
      if (t < 0.0) {
        double gmin;
        const double alpha = line_minimize(f, p, xit, fret, &gmin);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          xit[j] *= alpha;
          p[j] += xit[j];
        }
        fret = gmin;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          dirs[ibig][j] = dirs[2][j];
          dirs[2][j] = xit[j];
        }
      }
    }
  }
  *fret_out = fret;
}

}  // namespace

// Dynamic shared memory of the Powell kernel: the staged frame region (its
// cap in uint16 elements), then two doubles per pattern point.
struct PowellSmem {
  int patch_cap;   // elements of the staged frame region
  int max_points;  // largest pattern of the grains
  size_t bytes;
};

__host__ __device__ inline size_t powell_vals_offset(int patch_cap) {
  return ((size_t)patch_cap * sizeof(uint16_t) + 15) & ~(size_t)15;
}

// after the last point's values: what the sums' walk may read past them
constexpr size_t kTermPad = 4 * sizeof(double);

// what a block may use besides the kernels' static shared memory
constexpr size_t kPowellSmemMax = (227 - 20) * 1024;

// Margin of the staged frame region around the pattern (pixels): the moves of
// Powell's steps.  Samples further out read the frame.
constexpr int kPatchMargin = 6;

// follow_pattern_subpixel_xyR (src/p-tracker.cpp:1090-1128) for every grain,
// one block per grain, grains taken in `order` (decreasing pattern size) when
// given.  A grain takes 160-400 evaluations one after another, so an
// evaluation's latency counts: for 441 points 11.5k cycles (2.0k samples, 3.4k
// the first sum, 4.5k the other two, 0.4k cosine and sine, 1.3k Powell's own
// divisions and roots), against 33k with the sums and the cosine's series in one
// thread.  Of whole pairs: 12 grains of up to 530 points 3.57 -> 1.83 ms, 400 of
// 1,260-2,820 (8-bit frames of 2048x1536) 20.5 -> 7.6 ms, 2000 of up to 5,025
// (5616x3744) 47.7 -> 26.5 ms, of which the search took 9.2 then.
template <int NT, int BLOCKS, class Ref>
__global__ void __launch_bounds__(NT, BLOCKS) k_subpix_powell(GrainsDev g, FrameDev cur, SubpixParams sp,
                                                              int patch_cap, int max_points, const int* order,
                                                              const int* list_count) {
  __shared__ int s_m2;
  if (list_count && (int)blockIdx.x >= *list_count) return;
  const int gi = order ? order[blockIdx.x] : (int)blockIdx.x;
  if (g.masked[gi] || (g.flags[gi] & 3)) return;
  const ObjGrain o = load_grain(g, gi);
  if (o.P <= 0 || o.P > max_points) return;
  // stage the frame region under the pattern, with a margin for the Powell steps
  if (threadIdx.x == 0) s_m2 = 0;
  __syncthreads();
  const int v_at = (int)powell_vals_offset(patch_cap), d0_at = v_at + max_points * (int)sizeof(double);
  uint16_t* s_patch = reinterpret_cast<uint16_t*>(s_subpix);
  int m2 = 0;
  for (int i = threadIdx.x; i < o.P; i += NT) {
    const short2 q = g.pat0[o.b + i];
    m2 = max(m2, (int)q.x * q.x + (int)q.y * q.y);
  }
  atomicMax(&s_m2, m2);
  __syncthreads();
  const int reach = (int)ceil(sqrt((double)s_m2)) + 1;
  const int cx = (int)floor(o.xref), cy = (int)floor(o.yref);
  const int px0 = max(cx - reach - kPatchMargin, 0), py0 = max(cy - reach - kPatchMargin, 0);
  const int px1 = min(cx + reach + kPatchMargin + 3, cur.dimx), py1 = min(cy + reach + kPatchMargin + 3, cur.dimy);
  int pw = max(px1 - px0, 0), ph = max(py1 - py0, 0);
  if (pw * ph > patch_cap) ph = pw > 0 ? min(ph, patch_cap / pw) : 0;  // samples outside read the frame
  for (int e = threadIdx.x; e < pw * ph; e += NT) {
    const int yy = e / pw, xx = e - yy * pw;
    s_patch[e] = cur.pix[(size_t)(py0 + yy) * cur.pitch + (px0 + xx)];
  }
  exact_begin<NT, Ref>(o, g, cur, sp, reach, px0, py0, pw, ph, v_at, d0_at);
  ExactObj& ex = exact_obj();
  if (threadIdx.x >= 32) {
    for (;;) {
      __syncthreads();
      if (ex.done) return;
      objective_exact<NT, Ref>();
    }
  }
  const PowellEval<NT, Ref> f{};
  double X[3] = {0.0, 0.0, 0.0};
  double fret;
  powell_minimize(f, X, sp.init_dir, sp.tol, &fret);
  if (threadIdx.x == 0) {
    ex.done = 1;
    g.ncc_subpix[gi] = 1.0 - fret;
    g.upix[gi] += X[0];
    g.vpix[gi] += X[1];
    g.rot_inc[gi] += X[2];
    g.dx[gi] += X[0];
    g.dy[gi] += X[1];
    g.drot[gi] += X[2];
    if (ex.clamped) g.status[gi] |= PTK_ST_SUBPIX_CLAMPED;
  }
  __syncthreads();  // lets the other warps go
}

// Objective at caller-given X for every grain, as Powell evaluates it.
__global__ void __launch_bounds__(kSubpixThreads) k_objective(GrainsDev g, FrameDev cur, SubpixParams sp,
                                                                const double* Xall, double* f, int max_points,
                                                                const int* order) {
  const int gi = order[blockIdx.x];
  const ObjGrain o = load_grain(g, gi);
  if (o.P <= 0 || o.P > max_points) {
    if (threadIdx.x == 0) f[gi] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  // one evaluation: no frame region is staged
  exact_begin<kSubpixThreads, RefGlobal>(o, g, cur, sp, 0, 0, 0, 0, 0, 0, 0);
  if (threadIdx.x < 3) exact_obj().X[threadIdx.x] = Xall[3 * gi + threadIdx.x];
  __syncthreads();
  const double val = objective_exact<kSubpixThreads, RefGlobal>();
  if (threadIdx.x == 0) f[gi] = val;
}

// The objective's FP64 gradient (and value, in block order) at caller-given X
// for every grain.
__global__ void __launch_bounds__(kSubpixThreads) k_objective_grad(GrainsDev g, FrameDev cur, SubpixParams sp,
                                                                     const double* Xall, double* f, double* grad,
                                                                     int max_points, const int* order) {
  __shared__ double red[kSubpixThreads / 32];
  const int gi = order[blockIdx.x];
  const ObjGrain o = load_grain(g, gi);
  if (o.P <= 0 || o.P > max_points) {
    if (threadIdx.x == 0)
      f[gi] = grad[3 * gi] = grad[3 * gi + 1] = grad[3 * gi + 2] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const double X[3] = {Xall[3 * gi], Xall[3 * gi + 1], Xall[3 * gi + 2]};
  bool clamped = false;
  double G[3];
  const double val = objective_grad<kSubpixThreads>(g, cur, sp, o, X, reinterpret_cast<double*>(s_subpix), red, G,
                                                     &clamped);
  if (threadIdx.x == 0) {
    f[gi] = val;
    grad[3 * gi] = G[0];
    grad[3 * gi + 1] = G[1];
    grad[3 * gi + 2] = G[2];
  }
}

// `staged`: the centred reference values too (powell_staged).
static PowellSmem powell_smem(int max_points, int max_r, bool staged) {
  PowellSmem m;
  // the reach of a rotated and rounded pattern is at most max_r + 1
  const size_t side = (size_t)(2 * (max_r + 1) + 2 * kPatchMargin + 3);
  size_t patch = side * side;
  const size_t rest = (size_t)max_points * sizeof(double) * (staged ? 2 : 1);
  if (powell_vals_offset((int)patch) + rest > kPowellSmemMax)  // samples outside the region read the frame
    patch = rest < kPowellSmemMax ? (kPowellSmemMax - rest) / sizeof(uint16_t) - 8 : 0;
  m.patch_cap = (int)patch;
  m.max_points = max_points;
  m.bytes = powell_vals_offset(m.patch_cap) + rest + kTermPad;
  return m;
}

static bool powell_staged(int max_points) { return (size_t)max_points * 2 * sizeof(double) <= kPowellSmemMax - 32 * 1024; }

// The kernel of a launch.  128 threads a block, except where there are no more
// grains than SMs (each block has an SM to itself, and its evaluations' latency
// is the whole time) and patterns large enough to keep 256 or 512 busy.  Threads
// a block 128 / 256 / 512: 80 grains of up to 5,000 points (three frames with
// rescues) 18.9 / 18.2 / 16.4 ms, 40 of up to 2,100 2.72 / 2.70 / 2.76 ms, 12 of
// up to 530 1.88 / 2.03 / 2.6 ms; 400 of up to 2,820 7.8 / 8.6 / 11.1 ms, 2000 of
// up to 5,000 27.2 / 28.4 / 41 ms.
constexpr int kPowellWidestPoints = 3000;
typedef void (*PowellKernel)(GrainsDev, FrameDev, SubpixParams, int, int, const int*, const int*);
struct PowellLaunch {
  PowellKernel kernel;
  int threads;
  PowellSmem smem;
  PowellLaunch(int n, int max_points, int max_r, int num_sms, bool small) {
    const bool staged = powell_staged(max_points);
    threads = !staged ? 256 : (n > num_sms || max_points <= kPowellWidePoints ? 128 : (max_points <= kPowellWidestPoints ? 256 : 512));
    kernel = !staged         ? k_subpix_powell<256, 1, RefGlobal>
             : threads == 512 ? k_subpix_powell<512, 1, RefStaged>
             : threads == 256 ? k_subpix_powell<256, 2, RefStaged>
             : small          ? k_subpix_powell<128, 4, RefStaged>
                              : k_subpix_powell<128, 3, RefStaged>;
    smem = powell_smem(max_points, max_r, staged);
    ensure_smem((const void*)kernel, smem.bytes);
  }
  void operator()(int n, const GrainsDev& g, const FrameDev& cur, const SubpixParams& sp, const int* order,
                  const int* list_count, cudaStream_t s) const {
    kernel<<<n, threads, smem.bytes, s>>>(g, cur, sp, smem.patch_cap, smem.max_points, order, list_count);
  }
};

// One launch gives every block the shared memory of the largest pattern (5,000
// points: two blocks an SM).  With more grains than run at once, those of up to
// kPowellWidePoints points (29 KB: four blocks an SM) get a launch of their own,
// beside the others', and fill the SMs that these leave idle: 2000 grains of 300
// to 5,000 points, whole pair 26.4 -> 24.0 ms (five small blocks an SM: 23.9;
// the large ones with 256 threads: 24.4); 400 grains of 1,260 to 2,820, which
// all run at once, would take 6.88 instead of 6.65 ms.
bool powell_split(const PowellSizes& z, int num_sms) {
  return z.n > 3 * num_sms && z.n_large > 0 && z.n_large < z.n;
}

void prepare_subpix(const PowellSizes& z, int num_sms) {
  PowellLaunch(z.n, z.max_points, z.max_r, num_sms, false);
  if (powell_split(z, num_sms)) PowellLaunch(z.n, z.small_points, z.small_r, num_sms, true);
}

void launch_subpix_powell(const GrainsDev& g, const FrameDev& cur, const SubpixParams& sp, const PowellSizes& z,
                          int num_sms, const int* order, cudaStream_t s, const SideStream& side,
                          const int* list_count) {
  if (g.n <= 0) return;
  const PowellLaunch large(z.n, z.max_points, z.max_r, num_sms, false);
  if (list_count || !powell_split(z, num_sms)) {
    large(g.n, g, cur, sp, order, list_count, s);
    return;
  }
  const PowellLaunch small(z.n, z.small_points, z.small_r, num_sms, true);
  cudaEventRecord(side.fork, s);
  cudaStreamWaitEvent(side.stream, side.fork, 0);
  large(z.n_large, g, cur, sp, order, nullptr, s);
  small(z.n - z.n_large, g, cur, sp, order + z.n_large, nullptr, side.stream);
  cudaEventRecord(side.join, side.stream);
  cudaStreamWaitEvent(s, side.join, 0);
}

// One launch of the objective or gradient kernel over n grains of `order`.
static void launch_objective_class(int n, const GrainsDev& g, const FrameDev& cur, const SubpixParams& sp,
                                   const double* X, double* f, double* grad, int max_points, const int* order,
                                   cudaStream_t s) {
  // with the gradient: its samples too
  const size_t bytes = (size_t)max_points * sizeof(double) * (grad ? 3 : 1) + (grad ? 0 : kTermPad);
  if (grad) {
    if (bytes <= 227 * 1024) ensure_smem((const void*)k_objective_grad, bytes);
    k_objective_grad<<<n, kSubpixThreads, bytes, s>>>(g, cur, sp, X, f, grad, max_points, order);
  } else {
    ensure_smem((const void*)k_objective, bytes);
    k_objective<<<n, kSubpixThreads, bytes, s>>>(g, cur, sp, X, f, max_points, order);
  }
}

// With more grains than run at once, small patterns have a launch of their own
// beside the large ones' (as in launch_subpix_powell): 5,000 points leave one
// gradient block an SM (120 KB), 1,500 six.  2000 grains of 300 to 5,000 points:
// gradient 190 -> 101 us, the two calls together 362 -> 260 us.
int launch_objective(const GrainsDev& g, const FrameDev& cur, const SubpixParams& sp, const double* X, double* f,
                     double* grad, const PowellSizes& z, int num_sms, const int* order, cudaStream_t s,
                     const SideStream& side) {
  if (g.n <= 0) return 0;
  if (!powell_split(z, num_sms)) {
    launch_objective_class(g.n, g, cur, sp, X, f, grad, z.max_points, order, s);
    return 1;
  }
  cudaEventRecord(side.fork, s);
  cudaStreamWaitEvent(side.stream, side.fork, 0);
  launch_objective_class(z.n_large, g, cur, sp, X, f, grad, z.max_points, order, s);
  launch_objective_class(z.n - z.n_large, g, cur, sp, X, f, grad, z.small_points, order + z.n_large, side.stream);
  cudaEventRecord(side.join, side.stream);
  cudaStreamWaitEvent(s, side.join, 0);
  return 2;
}

}  // namespace ptk
