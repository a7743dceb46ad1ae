// Sums in index order, rounded after every term, by a whole thread block.
//
// A running FP64 sum s_{i+1} = RN(s_i + t_i) looks serial: P dependent
// additions.  But while the running sum keeps its sign and binade, its spacing
// u is fixed, s_i is a whole multiple of u, and the increment s_{i+1} - s_i
// depends on s_i only through its last mantissa bit (which decides ties).  So a
// run of terms acts on the sum's bit pattern as a map of that bit alone,
//     bits(s) -> bits(s) + k[bits(s) & 1],
// and such maps compose.  Each thread takes one contiguous run of terms (a
// chunk), in four parts:
//   1. it adds the parts up; a block scan gives every part an approximate
//      starting value a and, with the sum of |t|, bounds on the running sum
//      inside it;
//   2. it runs each part from two values next to a, one with an even and one
//      with an odd last bit.  Where the bounds, widened by more than all
//      rounding errors, stay in one binade, the results give the part's map;
//      it is held as c[0], c[1] in terms of the sums' distances from the
//      approximate values, which fit 32 bits:
//          d = bits(s) - bits(a)  ->  d + c[d & 1]   (a with an even last bit);
//   3. a warp scan composes the maps between the parts that leave their binade,
//      and one thread walks over them, adding the terms of those parts - and of
//      a last chunk that is not full - one by one.
// The result is the serial loop's bit for bit, for any terms (a NaN or an
// infinity leaves no part with bounds, and the walk is then that loop).
//
// What bounds it: instruction latency in a few warps.  Dependent additions take
// 8.5 cycles: P / (4 threads) of them, twice, and the walk's, about
// log2(threads) parts for a growing sum, against P of them for one thread; a
// single warp issues an instruction every three cycles or so, which is why the
// loops carry no bounds checks (chunks are full, of 1 + 4 l terms), the maps are
// 32-bit and the walk's steps come as a list.
#pragma once

#include <cuda_runtime.h>

namespace ptk {

// One step of the walk: the map k[0], k[1] of the sum's bit pattern, then n
// terms from index `at`, then step `next` (negative: it was the last one).
struct __align__(16) SeqStep {
  long long k0, k1;
  int at, n, next, pad;
};

template <int NT>
struct SeqSumScratch {        // each warp works for one sum
  SeqStep list[NT / 32 * 33];  // 33 per warp: its steps, in order
  double wsum[NT / 32];       // per warp: sum of its chunks
  float wabs[NT / 32];        // per warp: sum of |t|, rounded up
  double out[2];              // the sums
};

// The block's scratch (a function, so that every use sees shared memory).
template <int NT>
__device__ __forceinline__ SeqSumScratch<NT>& seq_scratch() {
  __shared__ SeqSumScratch<NT> s;
  return s;
}

// 1 when some value of [lo, hi] may lie in another binade than the others.
__device__ __forceinline__ unsigned seq_leaves(double lo, double hi) {
  const unsigned a = (unsigned)__double2hiint(lo), b = (unsigned)__double2hiint(hi);
  return (unsigned)((a ^ b) >= 1u << 20) | (unsigned)(((a >> 20) & 0x7ffu) - 1u >= 0x7feu);
}
// (a0, a1), then (b0, b1)
__device__ __forceinline__ void seq_compose(int a0, int a1, int b0, int b1, int* c0, int* c1) {
  *c0 = a0 + ((a0 & 1) ? b1 : b0);
  *c1 = a1 + ((a1 & 1) ? b0 : b1);
}

// How P terms are split over G threads: chunks of 1 + 4 l terms, the first of
// the four parts one longer (an odd number, so that the threads' 8-byte terms at
// that stride lie in different banks), `full` of them.
struct SeqPlan {
  int l, full;
};
__device__ __forceinline__ SeqPlan seq_plan(int P, int G) {
  const int l = ((P + G - 1) / G + 2) / 4;
  return SeqPlan{l, P / (1 + 4 * l)};
}

// Threads of a block that form one of NS sums side by side: all of its share, up
// to 128, or 256 in the widest blocks, which have the largest patterns (more
// threads shorten the chunks less than they lengthen the scan).
template <int NT, int NS>
constexpr int kSeqThreads = NT >= 512 ? 256 : (NT / NS < 128 ? NT / NS : 128);

// NS = 1 or 2 sums of P terms, each by kSeqThreads<NT, NS> threads (plan:
// seq_plan(P, kSeqThreads<NT, NS>)).  terms.of(n) provides sum n's terms as a
// function of their index, which may be asked for up to three terms past the
// last one (any value will do).  The sums are in seq_scratch<NT>().out once the
// block has synchronised (the caller does).  Every thread must call it; the
// scratch must not be in use.
template <int NT, int NS, class Terms>
__device__ __forceinline__ void seq_sums(int P, const SeqPlan plan, const Terms& terms) {
  static_assert((NS == 1 || NS == 2) && NT % (32 * NS) == 0, "whole warps per sum");
  constexpr int G = kSeqThreads<NT, NS>;  // threads of one sum
  SeqSumScratch<NT>& sc = seq_scratch<NT>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = warp / (G / 32), tid = threadIdx.x - n * G, warp0 = n * (G / 32);
  const auto term = terms.of(n);
  const int l = plan.l, L = 1 + 4 * l, full = plan.full;
  const int beg = tid * L;
  const bool mine = n < NS && tid < full;
  double S[4], A[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) S[u] = A[u] = 0.0;
  if (mine) {
    S[0] = term(beg);
    A[0] = fabs(S[0]);
    for (int i = beg + 1; i <= beg + l; ++i) {
      double t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) t[u] = term(i + u * l);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        S[u] += t[u];
        A[u] += fabs(t[u]);
      }
    }
  }
  double inc = (S[0] + S[1]) + (S[2] + S[3]);
  float warp_abs = __double2float_ru((A[0] + A[1]) + (A[2] + A[3]));
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
    warp_abs = __fadd_ru(warp_abs, __shfl_xor_sync(0xffffffffu, warp_abs, o));
  }
  if (lane == 31) {
    sc.wsum[warp] = inc;
    sc.wabs[warp] = warp_abs;
  }
  const double before_me = __shfl_up_sync(0xffffffffu, inc, 1);
  __syncthreads();
  if (n < NS && 32 * (warp - warp0) < full) {  // (warp-uniform)
    double base = 0.0;
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < G / 32; ++w) {
      const double y = sc.wsum[warp0 + w];
      if (w < warp - warp0) base += y;
      total = __fadd_ru(total, sc.wabs[warp0 + w]);
    }
    // approximate sums before each part and after the last (which the next
    // thread forms by the same additions), with an even last bit.  Every partial
    // sum of full chunks, the serial one's and the ones here, is within
    // 2 * 16384 * 2^-53 * sum |t| of the exact value; with bounds that stay
    // 2^-14 sum |t| away from the binade's ends - and so from zero - that is
    // less than 2^30 spacings.
    double a[5];
    a[0] = lane > 0 ? base + before_me : base;
    a[1] = a[0] + S[0];
    a[2] = a[1] + S[1];
    a[3] = a[2] + S[2];
    a[4] = base + inc;
    // margin: the power of two above 2^-14 sum |t| (none for sums beyond FP32)
    const double mg = __hiloint2double(total < 1e38f ? ((__float_as_int(total) >> 23) + (1023 - 127 - 13)) << 20 : 0x7ff00000, 0);
    unsigned leaves = 0u, some[4];  // bit u: part u leaves its binade; whether it has terms that are not all zero
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double d = A[u] - S[u], e = A[u] + S[u], lo = a[u] - mg, hi = a[u] + mg;
      // (a part whose terms are all zero leaves any sum as it is)
      some[u] = (unsigned)(A[u] != 0.0);
      leaves |= (seq_leaves(__fma_rn(-0.5, d, lo), __fma_rn(0.5, e, hi)) & some[u]) << u;
    }
    double s0[4], s1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s0[u] = __longlong_as_double(__double_as_longlong(a[u]) & ~1ll);
      s1[u] = __longlong_as_double(__double_as_longlong(a[u]) | 1ll);
    }
    if (mine) {
      const double t0 = term(beg);
      s0[0] += t0;
      s1[0] += t0;
      for (int i = beg + 1; i <= beg + l; ++i) {
        double t[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) t[u] = term(i + u * l);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          s0[u] += t[u];
          s1[u] += t[u];
        }
      }
    }
    // maps of the parts before and after the one that leaves its binade (all of
    // them in `c` where none does); two such parts: the whole chunk is added
    // term by term.  A run of maps without terms that count changes nothing, but
    // its approximate sums may differ from the true one by more than 32 bits:
    // `some` tells.  Chunk 0, where the sum starts at zero, is added term by term.
    int b0 = 0, b1 = 0, c0 = 0, c1 = 0;
    double from = a[0], to = a[0];  // where the map c starts; the step's start
    int at = beg, cnt = 0;
    unsigned b_some = 0u, c_some = 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool out = (leaves >> u) & 1u;
      const int e = __double2loint(a[u + 1]) & ~1;
      int n0, n1;
      seq_compose(c0, c1, __double2loint(s0[u]) - e, __double2loint(s1[u]) - e - 1, &n0, &n1);
      b0 = out ? c0 : b0;
      b1 = out ? c1 : b1;
      b_some = out ? c_some : b_some;
      to = out ? a[u] : to;
      from = out ? a[u + 1] : from;
      at = out ? beg + u * l + (u > 0 ? 1 : 0) : at;
      cnt = out ? l + (u > 0 ? 0 : 1) : cnt;
      c0 = out ? 0 : n0;
      c1 = out ? 0 : n1;
      c_some = out ? 0u : c_some | some[u];
    }
    const bool many = (leaves & (leaves - 1u)) != 0u, head = tid == 0, whole = many | head;
    b0 = whole ? 0 : b0;
    b1 = whole ? 0 : b1;
    c0 = whole ? 0 : c0;
    c1 = whole ? 0 : c1;
    b_some = whole ? 0u : b_some;
    c_some = whole ? 0u : c_some;
    to = whole ? a[0] : to;
    from = whole ? a[4] : from;
    at = whole ? beg : at;
    cnt = whole ? L : cnt;
    const unsigned cut = __ballot_sync(0xffffffffu, cnt != 0), any = __ballot_sync(0xffffffffu, c_some != 0u);
    // first lane of the run of maps that ends before this lane's step (or, for
    // the last lane's final map, with it): the last lane with a step, or lane 0
    const unsigned below = cut & ((1u << lane) - 1u), upto = cut & (0xffffffffu >> (31 - lane));
    const int first = below ? 31 - __clz(below) : 0, own = upto ? 31 - __clz(upto) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int p0 = __shfl_up_sync(0xffffffffu, c0, o), p1 = __shfl_up_sync(0xffffffffu, c1, o);
      int n0, n1;
      seq_compose(p0, p1, c0, c1, &n0, &n1);
      if (lane - o >= own) {
        c0 = n0;
        c1 = n1;
      }
    }
    const int p0 = __shfl_up_sync(0xffffffffu, c0, 1), p1 = __shfl_up_sync(0xffffffffu, c1, 1);
    const long long from_bits = __double_as_longlong(from) & ~1ll;
    const long long first_bits = __shfl_sync(0xffffffffu, from_bits, first);
    const long long own_bits = __shfl_sync(0xffffffffu, from_bits, own);
    const int slot = 33 * warp;
    // In a run the sum's bits change by `to - from`, the approximate sums at its
    // ends, and by the map of the distances; a run without terms that count
    // changes nothing.
    if (cnt != 0) {
      int m0, m1;
      seq_compose(lane > 0 ? p0 : 0, lane > 0 ? p1 : 0, b0, b1, &m0, &m1);
      const bool run = (b_some | (unsigned)((any & ((1u << lane) - 1u) & ~((1u << first) - 1u)) != 0u)) != 0u;
      const long long by = (__double_as_longlong(to) & ~1ll) - (lane > 0 ? first_bits : __double_as_longlong(a[0]) & ~1ll);
      const int k = slot + __popc(below);
      sc.list[k] = SeqStep{run ? by + m0 : 0, run ? by + m1 : 0, at, cnt, k + 1, 0};
    }
    if (lane == 31) {  // the warp's last map, and what the full chunks leave of the terms
      const bool last = 32 * (warp - warp0 + 1) >= full;
      const bool run = (any & ~((1u << own) - 1u)) != 0u;
      const long long by = (__double_as_longlong(a[4]) & ~1ll) - own_bits;
      sc.list[slot + __popc(cut)] = SeqStep{run ? by + c0 : 0, run ? by + c1 : 0, full * L, last ? P - full * L : 0,
                                            last ? -1 : slot + 33, 0};
    }
  }
  __syncthreads();
  if (n < NS && tid == 0) {
    // The walk of sum n, four terms at a time (past a step's end: + 0, which
    // changes nothing: s is never -0).  Branches cost more than what they would
    // skip here: there is one, the loop's.
    SeqStep e = sc.list[33 * warp];
    if (full == 0) e = SeqStep{0, 0, 0, P, -1, 0};  // fewer terms than one chunk
    double s = 0.0, t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = term(e.at + u);
    bool more;
    do {
      const SeqStep f = sc.list[max(e.next, 0)];
      const long long b = __double_as_longlong(s);
      s = __longlong_as_double(b + ((b & 1) ? e.k1 : e.k0));
#pragma unroll
      for (int u = 0; u < 4; ++u) s += u < e.n ? t[u] : 0.0;
      const bool rest = e.n > 4;
      more = rest || e.next >= 0;
      e.at = rest ? e.at + 4 : f.at;
      e.n = rest ? e.n - 4 : f.n;
      e.next = rest ? e.next : f.next;
      e.k0 = rest ? 0 : f.k0;
      e.k1 = rest ? 0 : f.k1;
#pragma unroll
      for (int u = 0; u < 4; ++u) t[u] = term(e.at + u);
    } while (more);
    sc.out[n] = s;
  }
}

}  // namespace ptk
