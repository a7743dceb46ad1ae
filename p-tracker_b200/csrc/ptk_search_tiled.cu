// Register-tiled exact search (the plain form's fast kernel).
//
// Same results as k_search (every candidate's S1 = sum I1, S11 = sum I1^2 and
// S01 = sum I0*I1 exact, same ranking and tie rule), computed with far fewer
// instructions per pattern-pixel-candidate:
//
//  * The rotated pattern of a work item is scattered once into a dense
//    column-major map over its bounding box:
//        map(x, y) = sum over points at (x, y) of (I0 + 2^20)
//    i.e. the reference pixel sum plus 2^20 x the multiplicity M(x, y), added up
//    by 32-bit integer atomics and turned into FP64 numbers in place.
//  * For each map column, every thread (one x offset u, 8 consecutive y
//    offsets) streams its current-frame column in blocks of 8 values and
//    accumulates sum map(x, y) * (2^16 + I1(x+u, y+v)) with FP64 FMAs, 8 rows x
//    8 candidates per chunk: 2^16 + v is a bit pattern of v's, v alone would
//    take an FP64 subtraction.  All operands and partial sums are integers below
//    2^52, so every FMA is exact:  acc = S01 + 2^20 S1 + 2^16 sum(map), whose
//    last term every candidate shares.  Two 8-value register
//    blocks alternate (no register moves); the next block is loaded between
//    the two halves of a chunk's FMAs, hiding shared-memory latency.
//  * S1 and S11 come from the column's maximal runs of constant multiplicity:
//    with d = m (I1 after the run - I1 at its start), each y offset differs from
//    the next by d and by d (their sum).  The sums at the first y offset are
//    taken once per x offset, a column by one warp of its class.
//  * If a column has more runs than the per-column list holds (sparse custom
//    patterns), the work item takes the differences entry by entry instead.
//  * An FP32 estimate of each coefficient leaves the FP64 root and division to
//    those that may be a warp's best.
//
// What bounds it: FP64 FMAs (42 % of their peak) and the instructions around
// them (59 % of the issue slots).  A work item of 2,000 points takes 49 k cycles
// of FMAs and differences (+-8; 70 k at +-15) and some 30 k around them, two
// blocks a multiprocessor.  Windows slid per thread from a sum of its own, points
// rotated twice, FP64 atomics and a root and division per candidate, before:
// +-15, 2000 grains 9.14 -> 8.01 ms; +-8, 400 grains 1.45 -> 1.28 ms; +-6, 40
// grains 70 -> 68 us.
//
// Thread layout: 256 threads.  A tile of nu x nv candidates has nu * ceil(nv / 8)
// pairs of an x offset and 8 consecutive y offsets, a pair per lane; they take
// 1, 2 or 4 warps, and the 8, 4 or 2 classes of warps share the map columns
// (every 8th, 4th or 2nd), their sums added through shared memory at the end.
// So a small zone's columns are spread over the warps that a full 32x32 tile
// needs for its candidates: +-8 (17x17, 2 warps a class), 400 grains of 1,260 to
// 2,820 points 2.43 -> 1.46 ms; +-6, 40 grains 156 -> 70 us; +-15 (31x31, 4 warps
// a class as before), 2000 grains 9.23 -> 9.14 ms.  The patch pitch is
// a template constant so every shared-memory address in the inner loop is a
// register plus an immediate.
#include <climits>

#include "ptk_internal.cuh"

namespace ptk {

namespace {

constexpr int kTT = 8;               // candidates per thread (along y) = rows per chunk
constexpr int kTiledThreads = 256;   // 8 warps, in 2, 4 or 8 classes of map columns
constexpr int kHeld = 8;             // rotated points a thread keeps between its two passes over them
constexpr int kRunsPerCol = 8;
constexpr int kMultShift = 20;       // map entry = I0 sum + multiplicity * 2^20
constexpr double kMult = 1048576.0;

__device__ __forceinline__ short2 rotate_round_t(short2 p, double c, double s) {
  const double px = (double)p.x, py = (double)p.y;
  const double xr = __dadd_rn(__dmul_rn(c, px), __dmul_rn(s, py));
  const double yr = __dadd_rn(__dmul_rn(-s, px), __dmul_rn(c, py));
  return make_short2((short)round(xr), (short)round(yr));
}

// 2^16 + v of a 16-bit v: its bits stand at the top of the mantissa
__device__ __forceinline__ double u16_above(unsigned v) { return __hiloint2double((int)(0x40F00000u + (v << 4)), 0); }

__device__ __forceinline__ bool better_t(double ncc, int idx, double bn, int bi) {
  return ncc > 0.0 && (ncc > bn || (ncc == bn && idx < bi));
}

struct TiledGeom {
  int mw, mh;  // map columns / rows (rows padded for the chunk loop)
  int ph;      // patch rows (the pitch is the template constant)
};

__host__ __device__ inline TiledGeom tiled_geom(int max_r) {
  TiledGeom t;
  const int box = 2 * max_r + 1;
  t.mw = box;
  // a column's last chunk ends up to 7 rows below its last point; the last
  // thread's blocks of 8 rows go 24 + 16 rows further
  // (16 rows less in both than a chunk more each, so that offsets to +-61 fit
  // where +-59 did: at 60, 60 grains, 2.39 ms in the direct kernel, 0.51 here)
  t.mh = ((box + kTT - 1) / kTT) * kTT + kTT;
  t.ph = t.mh + kTileV + kTT;
  return t;
}

// (4 more than a multiple of 8: the columns of lanes 8 rows apart start 16 banks apart)
__host__ __device__ inline int tiled_pitch(int max_r) { return 2 * max_r + 1 + kTileU - 1 <= 132 ? 132 : 260; }

__host__ __device__ inline size_t tiled_map_bytes(int max_r) {
  const TiledGeom t = tiled_geom(max_r);
  size_t b = (size_t)t.mw * t.mh * 8;
  const size_t partial = (size_t)kTiledThreads * kTT * 20;  // column-class partial sums
  return b < partial ? partial : b;
}

__host__ __device__ inline size_t tiled_smem(int max_r) {
  const TiledGeom t = tiled_geom(max_r);
  size_t b = tiled_map_bytes(max_r);
  b += (size_t)t.mw * kRunsPerCol * 4;  // runs
  b += (size_t)t.mw * 4 * 2;            // column extent + run count
  b = (b + 15) & ~(size_t)15;
  b += (size_t)tiled_pitch(max_r) * t.ph * 2;  // patch
  return b + 16;
}

}  // namespace

template <int PITCH>
__global__ void __launch_bounds__(kTiledThreads, 2) k_search_tiled(SearchLaunch p, int max_r) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_item, s_bbox[4], s_overflow;
  __shared__ double s_rn[kTiledThreads / 32];
  __shared__ int s_ri[kTiledThreads / 32];
  const TiledGeom G = tiled_geom(max_r);
  const size_t map_bytes = tiled_map_bytes(max_r);
  double* s_map = reinterpret_cast<double*>(smem);
  unsigned* s_map32 = reinterpret_cast<unsigned*>(smem);  // (little-endian: an entry's low word is 2 e)
  int* s_runs = reinterpret_cast<int*>(smem + map_bytes);
  int* s_ext = s_runs + G.mw * kRunsPerCol;  // packed (lo | hi << 16), empty column: lo > hi
  int* s_nrun = s_ext + G.mw;
  const size_t pofs = (map_bytes + (size_t)G.mw * kRunsPerCol * 4 + (size_t)G.mw * 8 + 15) & ~(size_t)15;
  uint16_t* s_patch = reinterpret_cast<uint16_t*>(smem + pofs);
  // partial sums of all column classes but the first reuse the map region after the FMAs
  double* s_pacc = reinterpret_cast<double*>(smem);
  long long* s_p11 = reinterpret_cast<long long*>(smem + (size_t)kTiledThreads * kTT * 8);
  int* s_p1 = reinterpret_cast<int*>(smem + (size_t)kTiledThreads * kTT * 16);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int count = *p.list_count;
  const int per_grain = p.nrot * p.tiles_u * p.tiles_v;
  long long total = (long long)count * per_grain;
  if (total > p.max_items) total = p.max_items;
  const int NU = p.left + p.right + 1, NV = p.up + p.down + 1;
  const GrainsDev& g = p.g;

  int next = 0;  // thread 0: the item after this one
  if (tid == 0) next = atomicAdd(p.work_next, 1);
  for (;;) {
    if (tid == 0) {
      s_item = next;
      s_bbox[0] = s_bbox[2] = INT_MAX;
      s_bbox[1] = s_bbox[3] = INT_MIN;
      s_overflow = 0;
    }
    __syncthreads();
    const int item = s_item;
    if (item >= total) break;
    if (tid == 0) next = atomicAdd(p.work_next, 1);
    const int li = item / per_grain;
    const int rem = item - li * per_grain;
    const int r = rem / (p.tiles_u * p.tiles_v);
    const int t = rem - r * (p.tiles_u * p.tiles_v);
    const int tu = t / p.tiles_v, tv = t - tu * p.tiles_v;
    const int gi = p.list[li];
    const int b = g.pstart[gi], P = g.pstart[gi + 1] - b;
    if (g.masked[gi] || (g.flags[gi] & 2) || P <= 0 || P > kMaxPatternPoints) {
      if (tid == 0) p.best[item] = SearchBest{0.0, INT_MAX, 0};
      __syncthreads();
      continue;
    }
    short2 held[kHeld];
    uint16_t held_w[kHeld];
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
      const int i = tid + k * kTiledThreads;
      held[k] = make_short2(0, 0);
      held_w[k] = 0;
      if (i < P) {
        held[k] = g.pat[b + i];
        held_w[k] = g.w0[b + i];
      }
    }
    const double total_rot = (g.refrot[gi] + g.drot[gi]) + p.steps[r];
    double s1, c1;
    sincos(total_rot, &s1, &c1);
    const int gdx = (int)round(g.dx[gi]);
    const int gdy = (int)round(g.dy[gi]);

    // (a) bounding box of the rotated pattern
    int xmn = INT_MAX, xmx = INT_MIN, ymn = INT_MAX, ymx = INT_MIN;
    auto rotated = [&](short2 p0) {
      const short2 q = rotate_round_t(p0, c1, s1);
      xmn = min(xmn, (int)q.x);
      xmx = max(xmx, (int)q.x);
      ymn = min(ymn, (int)q.y);
      ymx = max(ymx, (int)q.y);
      return q;
    };
#pragma unroll
    for (int k = 0; k < kHeld; ++k)
      if (tid + k * kTiledThreads < P) held[k] = rotated(held[k]);
    for (int i = tid + kHeld * kTiledThreads; i < P; i += kTiledThreads) rotated(g.pat[b + i]);
    for (int o = 16; o > 0; o >>= 1) {
      xmn = min(xmn, __shfl_xor_sync(0xffffffffu, xmn, o));
      xmx = max(xmx, __shfl_xor_sync(0xffffffffu, xmx, o));
      ymn = min(ymn, __shfl_xor_sync(0xffffffffu, ymn, o));
      ymx = max(ymx, __shfl_xor_sync(0xffffffffu, ymx, o));
    }
    if (lane == 0) {
      atomicMin(&s_bbox[0], xmn);
      atomicMax(&s_bbox[1], xmx);
      atomicMin(&s_bbox[2], ymn);
      atomicMax(&s_bbox[3], ymx);
    }
    __syncthreads();
    const int bx0 = s_bbox[0], bx1 = s_bbox[1], by0 = s_bbox[2], by1 = s_bbox[3];
    const int bw = bx1 - bx0 + 1, bh = by1 - by0 + 1;
    const int u0 = -p.left + tu * kTileU, u1 = min(u0 + kTileU - 1, p.right);
    const int v0 = -p.up + tv * kTileV, v1 = min(v0 + kTileV - 1, p.down);
    // this thread's candidates: x offset ul, y offsets rb .. rb + 7 of the tile, over
    // the map columns of class `cls` (of `ncls`)
    const int nu = u1 - u0 + 1, nvg = (v1 - v0 + kTT) / kTT, pairs = nu * nvg;
    const int wpc = pairs <= 32 ? 1 : (pairs <= 64 ? 2 : 4), ncls = kTiledThreads / 32 / wpc;
    const int cls = warp / wpc, pair = (warp - cls * wpc) * 32 + lane;
    const bool active = pair < pairs;  // (the others repeat the first pair)
    const int vg = active ? pair / nu : 0, ul = active ? pair - vg * nu : 0, rb = kTT * vg;
    const int X0 = g.refx[gi] + gdx + bx0 + u0;
    const int Y0 = g.refy[gi] + gdy + by0 + v0;
    const int needw = bw + (u1 - u0), needh = bh + (v1 - v0);
    const bool oob = X0 < 0 || Y0 < 0 || X0 + needw > p.cur.dimx || Y0 + needh > p.cur.dimy;
    const int mh = ((bh + kTT - 1) / kTT) * kTT + kTT;  // rows of this item's map
    const bool fits = bw <= G.mw && mh <= G.mh && bw + kTileU - 1 <= PITCH;
    if (oob || !fits) {
      if (tid == 0) {
        if (oob) atomicOr(&g.flags[gi], 1);
        else atomicOr(&g.flags[gi], 4);  // does not fit the tiled layout (not expected: host sizes it)
        p.best[item] = SearchBest{0.0, INT_MAX, 0};
      }
      __syncthreads();
      continue;
    }

    // (b) zero the map, (c) scatter I0 + 2^20 per point: at most 16 points a pixel,
    // so the sums fit the 32 low bits of an entry, where integer atomics add them
    for (int e = tid; e < bw * mh / 2; e += kTiledThreads) reinterpret_cast<double2*>(s_map)[e] = make_double2(0.0, 0.0);
    __syncthreads();
    auto scatter = [&](short2 q, unsigned w) {
      atomicAdd(&s_map32[2 * ((q.x - bx0) * mh + (q.y - by0))], w + (1u << kMultShift));
    };
#pragma unroll
    for (int k = 0; k < kHeld; ++k)
      if (tid + k * kTiledThreads < P) scatter(held[k], held_w[k]);
    for (int i = tid + kHeld * kTiledThreads; i < P; i += kTiledThreads)
      scatter(rotate_round_t(g.pat[b + i], c1, s1), g.w0[b + i]);
    // (e) stage the patch: rows [0, needh) x columns [0, needw); the rest
    // (reached only by zero weights or by candidates outside the zone) is zero
    const int ph = mh + kTT * nvg + kTT;
    constexpr int kW = kTiledThreads / 32;
    constexpr int kRows = 8;  // rows' loads in flight
    for (int yy = warp; yy < ph; yy += kRows * kW)
      for (int xx = lane; xx < needw; xx += 32) {
        uint16_t v[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
          const int y = yy + k * kW;
          v[k] = y < needh ? p.cur.pix[(size_t)(Y0 + y) * p.cur.pitch + (X0 + xx)] : (uint16_t)0;
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k)
          if (yy + k * kW < ph) s_patch[(yy + k * kW) * PITCH + xx] = v[k];
      }
    __syncthreads();
    // (d) per column, by a warp: the entries as FP64 numbers, the extent of the
    // non-zero rows and the runs of constant multiplicity, whose ends are the rows (up to bh, where it is 0) at which it changes
    for (int x = warp; x < bw; x += kTiledThreads / 32) {
      double* col = s_map + x * mh;
      const unsigned* col32 = s_map32 + 2 * x * mh;
      int lo = INT_MAX, hi = -1, nr = 0, start = 0, before = 0;
      for (int y0 = 0; y0 <= bh; y0 += 64) {  // 64 rows a step, two per lane
        const int y[2] = {y0 + lane, y0 + 32 + lane};
        unsigned entry[2];
        int m[2], prev[2];
        bool change[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          entry[h] = y[h] < bh ? col32[2 * y[h]] : 0u;
          m[h] = (int)(entry[h] >> kMultShift);
          prev[h] = __shfl_up_sync(0xffffffffu, m[h], 1);
        }
        const int mid = __shfl_sync(0xffffffffu, m[0], 31), last = __shfl_sync(0xffffffffu, m[1], 31);
        if (lane == 0) {
          prev[0] = before;
          prev[1] = mid;
        }
        before = last;
        unsigned long long on = 0, changes = 0, ends = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          change[h] = m[h] != prev[h] && y[h] <= bh;
          on |= (unsigned long long)__ballot_sync(0xffffffffu, m[h] != 0) << (32 * h);
          changes |= (unsigned long long)__ballot_sync(0xffffffffu, change[h]) << (32 * h);
          ends |= (unsigned long long)__ballot_sync(0xffffffffu, change[h] && prev[h] != 0) << (32 * h);
          if (entry[h]) col[y[h]] = __hiloint2double(0x43300000, (int)entry[h]) - 4503599627370496.0;
        }
        if (on) {
          lo = min(lo, y0 + __ffsll((long long)on) - 1);
          hi = y0 + 63 - __clzll((long long)on);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const unsigned long long below = (1ull << (lane + 32 * h)) - 1ull;
          if (change[h] && prev[h] != 0) {
            const unsigned long long c = changes & below;
            const int s = c ? y0 + 63 - __clzll((long long)c) : start, k = nr + __popcll(ends & below);
            if (k < kRunsPerCol) s_runs[x * kRunsPerCol + k] = s | ((y[h] - 1) << 8) | (prev[h] << 16);
          }
        }
        nr += __popcll(ends);
        if (changes) start = y0 + 63 - __clzll((long long)changes);
      }
      if (lane == 0) {
        s_ext[x] = hi < 0 ? 1 : (lo | (hi << 16));
        s_nrun[x] = nr;
        if (nr > kRunsPerCol) atomicOr(&s_overflow, 1);
      }
    }
    __syncthreads();

    // (f) candidates: x offset u0 + ul, y offsets v0 + rb + 0..7, map columns of class `cls`
    double acc[kTT];
    int F1[kTT];        // S1(v + 1) - S1(v), S11(v + 1) - S11(v) for its y offsets v
    long long F11[kTT];
    unsigned base1 = 0;  // S1 and S11 at the tile's first y offset and x offset `lane`, of some columns
    unsigned long long base11 = 0;
#pragma unroll
    for (int k = 0; k < kTT; ++k) {
      acc[k] = 0.0;
      F1[k] = 0;
      F11[k] = 0;
    }
    const int turn = warp - cls * wpc, ub = min(lane, nu - 1);
    int nth = 0;
    const bool overflow = s_overflow != 0;
    for (int x = cls; x < bw; x += ncls) {
      const int ext = s_ext[x];
      const int lo = ext & 0xfffe, hi = ext >> 16;  // from an even row: the map is read in pairs
      if (hi == 0 && ext) continue;
      // column of this thread from row lo + rb, in blocks of 8 rows
      const uint16_t* cp = s_patch + (lo + rb) * PITCH + x + ul;
      const double* wp = s_map + x * mh + lo;
      double A[kTT], B[kTT];
#pragma unroll
      for (int k = 0; k < kTT; ++k) A[k] = u16_above(cp[k * PITCH]);
#pragma unroll
      for (int k = 0; k < kTT; ++k) B[k] = u16_above(cp[(kTT + k) * PITCH]);
      // chunk c uses (A, B) = row blocks c, c+1; block c+2 is loaded into A
      // between the FMAs that read A and those that read only B
      int nchunk = (hi - lo) / kTT + 1;
      for (;;) {
        {
          double w[kTT];
#pragma unroll
          for (int j = 0; j < kTT; j += 2) {
            const double2 two = *reinterpret_cast<const double2*>(wp + j);
            w[j] = two.x;
            w[j + 1] = two.y;
          }
#pragma unroll
          for (int j = 0; j < kTT; ++j)
#pragma unroll
            for (int k = 0; k < kTT; ++k)
              if (j + k < kTT) acc[k] = fma(w[j], A[j + k], acc[k]);
          cp += kTT * PITCH;
#pragma unroll
          for (int k = 0; k < kTT; ++k) A[k] = u16_above(cp[(kTT + k) * PITCH]);
#pragma unroll
          for (int j = 0; j < kTT; ++j)
#pragma unroll
            for (int k = 0; k < kTT; ++k)
              if (j + k >= kTT) acc[k] = fma(w[j], B[j + k - kTT], acc[k]);
          wp += kTT;
        }
        if (--nchunk == 0) break;
        {
          double w[kTT];
#pragma unroll
          for (int j = 0; j < kTT; j += 2) {
            const double2 two = *reinterpret_cast<const double2*>(wp + j);
            w[j] = two.x;
            w[j + 1] = two.y;
          }
#pragma unroll
          for (int j = 0; j < kTT; ++j)
#pragma unroll
            for (int k = 0; k < kTT; ++k)
              if (j + k < kTT) acc[k] = fma(w[j], B[j + k], acc[k]);
          cp += kTT * PITCH;
#pragma unroll
          for (int k = 0; k < kTT; ++k) B[k] = u16_above(cp[(kTT + k) * PITCH]);
#pragma unroll
          for (int j = 0; j < kTT; ++j)
#pragma unroll
            for (int k = 0; k < kTT; ++k)
              if (j + k >= kTT) acc[k] = fma(w[j], A[j + k - kTT], acc[k]);
          wp += kTT;
        }
        if (--nchunk == 0) break;
      }
      const uint16_t* colp = s_patch + rb * PITCH + x + ul;
      const uint16_t* basep = s_patch + x + ub;
      const bool mine = (nth++ & (wpc - 1)) == turn;  // this warp takes the column's base sums
      if (!overflow) {
        const int nr = s_nrun[x];
        for (int q = 0; q < nr; ++q) {
          const int rr = s_runs[x * kRunsPerCol + q];
          const int a = rr & 0xff, e = (rr >> 8) & 0xff, m = rr >> 16;
          if (mine) {
            unsigned sm = 0;
            unsigned long long s2 = 0;
#pragma unroll 4
            for (int y = a; y <= e; ++y) {
              const unsigned val = basep[y * PITCH];
              sm += val;
              s2 += (unsigned long long)val * val;
            }
            base1 += (unsigned)m * sm;
            base11 += (unsigned long long)m * s2;
          }
          const uint16_t* in = colp + (e + 1) * PITCH;
          const uint16_t* out = colp + a * PITCH;
#pragma unroll
          for (int k = 0; k < kTT; ++k) {
            const int vin = in[k * PITCH], vout = out[k * PITCH];
            const int d = m * (vin - vout);
            F1[k] += d;
            F11[k] += (long long)d * (vin + vout);
          }
        }
      } else {
        // entry by entry: every non-zero map entry of the column with its multiplicity
        const double* wcol = s_map + x * mh;
        for (int y = lo; y <= hi; ++y) {
          const int m = (int)(wcol[y] * (1.0 / kMult));
          if (!m) continue;
          if (mine) {
            const unsigned val = basep[y * PITCH];
            base1 += (unsigned)m * val;
            base11 += (unsigned long long)m * (val * val);
          }
          int vout = colp[y * PITCH];
#pragma unroll
          for (int k = 0; k < kTT; ++k) {
            const int vin = colp[(y + k + 1) * PITCH];
            const int d = m * (vin - vout);
            F1[k] += d;
            F11[k] += (long long)d * (vin + vout);
            vout = vin;
          }
        }
      }
    }
    // sum the column classes (the map is no longer needed)
    __syncthreads();
    if (cls > 0) {
      const int slot = (cls - 1) * 32 * wpc + pair;
#pragma unroll
      for (int k = 0; k < kTT; ++k) {
        s_pacc[k * kTiledThreads + slot] = acc[k];
        s_p11[k * kTiledThreads + slot] = F11[k];
        s_p1[k * kTiledThreads + slot] = F1[k];
      }
    }
    // (the slots of class 0, the last 32 wpc of each row, hold the base sums, a
    // row per warp, and in s_pacc the pairs' own sums of differences)
    s_p11[warp * kTiledThreads + kTiledThreads - 32 + lane] = (long long)base11;
    s_p1[warp * kTiledThreads + kTiledThreads - 32 + lane] = (int)base1;
    __syncthreads();
    long long* s_t11 = reinterpret_cast<long long*>(s_pacc) + kTiledThreads - 32 * wpc;
    long long* s_t1 = s_t11 + kTiledThreads;
    if (cls == 0) {
      long long t1 = 0, t11 = 0;
#pragma unroll
      for (int k = 0; k < kTT; ++k) {
        for (int c = 1; c < ncls; ++c) {
          const int slot = k * kTiledThreads + (c - 1) * 32 * wpc + pair;
          acc[k] += s_pacc[slot];
          F11[k] += s_p11[slot];
          F1[k] += s_p1[slot];
        }
        t1 += F1[k];
        t11 += F11[k];
      }
      s_t11[pair] = t11;
      s_t1[pair] = t1;
    }
    __syncthreads();
    double bn = 0.0;
    int bi = INT_MAX;
    if (cls == 0) {  // (the lanes without a pair of their own repeat the first one)
      const long long Pl = P, S0 = g.s0[gi];
      const double den1 = (double)(Pl * g.s00[gi] - S0 * S0);
      const long long above = (S0 + (Pl << kMultShift)) << 16;  // 2^16 x the map's sum
      const int u = u0 + ul;
      long long s1 = 0, s11 = 0;
      for (int w = 0; w < kTiledThreads / 32; ++w) {
        s1 += (unsigned)s_p1[w * kTiledThreads + kTiledThreads - 32 + ul];
        s11 += s_p11[w * kTiledThreads + kTiledThreads - 32 + ul];
      }
      for (int j = 0; j < vg; ++j) {
        s1 += s_t1[j * nu + ul];
        s11 += s_t11[j * nu + ul];
      }
      // An FP32 estimate first (its relative error is below 1e-6; den1 and d2 lie
      // below 2^60): the division and the root for those that may be the warp's best.
      long long num[kTT], d2[kTT];
      float est[kTT], top = 0.0f;
#pragma unroll
      for (int k = 0; k < kTT; ++k) {
        const long long s1k = s1, s11k = s11;
        s1 += F1[k];
        s11 += F11[k];
        const long long s01 = __double2ll_rn(acc[k]) - above - (s1k << kMultShift);
        num[k] = Pl * s01 - S0 * s1k;
        d2[k] = Pl * s11k - s1k * s1k;
        est[k] = v0 + rb + k <= v1 ? (float)num[k] * rsqrtf((float)den1 * (float)d2[k]) : -1.0f;
        if (est[k] < 2.0f) top = fmaxf(top, est[k]);
      }
      top = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(top)));  // (not negative)
#pragma unroll
      for (int k = 0; k < kTT; ++k) {
        const int v = v0 + rb + k;
        if (v > v1 || est[k] < top * 0.9999f) continue;
        const double ncc = (double)num[k] / sqrt(den1 * (double)d2[k]);
        const int idx = (r * NU + (u + p.left)) * NV + (v + p.up);
        if (better_t(ncc, idx, bn, bi)) {
          bn = ncc;
          bi = idx;
        }
      }
    }
    // the best of the warps that hold pairs: coefficients are not negative, so
    // they order as their bits do
    if (cls == 0) {
      const int hi = __reduce_max_sync(0xffffffffu, __double2hiint(bn));
      const bool at_hi = __double2hiint(bn) == hi;
      const unsigned lo = __reduce_max_sync(0xffffffffu, at_hi ? (unsigned)__double2loint(bn) : 0u);
      const int idx = __reduce_min_sync(0xffffffffu, at_hi && (unsigned)__double2loint(bn) == lo ? bi : INT_MAX);
      if (lane == 0) {
        s_rn[warp] = __hiloint2double(hi, (int)lo);
        s_ri[warp] = idx;
      }
    }
    __syncthreads();
    if (tid == 0) {
      double fn = 0.0;
      int fi = INT_MAX;
      for (int k = 0; k < wpc; ++k)
        if (better_t(s_rn[k], s_ri[k], fn, fi)) {
          fn = s_rn[k];
          fi = s_ri[k];
        }
      p.best[item] = SearchBest{fn, fi, 0};
    }
    __syncthreads();
  }
}

size_t search_tiled_smem(int max_r) { return tiled_smem(max_r); }

int search_tiled_occupancy(size_t smem, int max_r) {
  int blocks = 0;
  if (tiled_pitch(max_r) == 132) {
    ensure_smem((const void*)k_search_tiled<132>, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_search_tiled<132>, kTiledThreads, smem);
  } else {
    ensure_smem((const void*)k_search_tiled<260>, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_search_tiled<260>, kTiledThreads, smem);
  }
  return blocks;
}

void launch_search_tiled(const SearchLaunch& p, int max_r, int grid, size_t smem, cudaStream_t s) {
  search_tiled_occupancy(smem, max_r);
  if (tiled_pitch(max_r) == 132) k_search_tiled<132><<<grid, kTiledThreads, smem, s>>>(p, max_r);
  else k_search_tiled<260><<<grid, kTiledThreads, smem, s>>>(p, max_r);
}

}  // namespace ptk
