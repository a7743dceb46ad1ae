// Test harness (not part of the library): the correctly rounded cosine and sine
// (p-tracker_b200/csrc/ptk_crtrig.cuh on the host) with and without the quick
// phase, over arrays of angles.
#include "../p-tracker_b200/csrc/ptk_crtrig.cuh"

extern "C" {

// out[i]: cr_cos (which == 0) or cr_sin (1) of x[i]
void crt_eval(const double* x, long n, int which, double* out) {
  for (long i = 0; i < n; ++i) out[i] = ptk::crtrig::cr_trig(x[i], which);
}

// the double-double series alone, for |x| <= pi/4
void crt_series(const double* x, long n, int which, double* out) {
  using namespace ptk::crtrig;
  for (long i = 0; i < n; ++i) out[i] = which ? sin_dd(dd{x[i], 0.0}) : cos_dd(dd{x[i], 0.0});
}

// how many of the angles the quick phase leaves to the series
long crt_undecided(const double* x, long n, int which) {
  long k = 0;
  double out;
  for (long i = 0; i < n; ++i) k += ptk::crtrig::quick_trig(x[i], which, &out) ? 0 : 1;
  return k;
}
}
