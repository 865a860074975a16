// fr_plane.cu -- the plane-column insertion kernel (gauss_2, gauss_5,
// trilinear).
//
// A slice's taps lie in a slab around its plane.  With A the axis along which
// the plane's normal is largest, B and C the other two, every tap column
// (b, c) crosses that slab in one short run of cells along A (at most 7 cells
// for the two-tap windows, 19 for gauss_5).  One lane owns one column of one
// slice: it walks the pixels whose window covers the column, sums their taps
// into the run, held in its own shared-memory words (gauss_5 keeps the six
// cells of the current window in registers), and at the end adds the run's
// sums to the volume, one reduction per touched cell, under the placement
// rules of add_complex_at_fast.  No lane ever shares a cell with another
// before that, so there are neither barriers nor shared-memory atomics, and a
// warp (an 8 x 4 patch of columns) depends on no other warp.
//
// Reductions are free while the volume fits L2 and cost a quarter of the time
// beyond it (gauss_2, d7, N = 384: 47.4 us a particle with two a cell, 37.0
// with the value's alone, 34.4 with none), by the request rather than by the
// byte.  So a large call's partial volume holds a cell's value and weight
// together, one 16-byte reduction (39.4, and 35.4 with the patches drawn), and
// a run's cells are addressed by a stride.  Walking eight neighbouring columns in step, which puts their
// reductions into one line, took more instructions than it saved (45.0).
//
// What bounds it: issue slots (68 % of cycles issue at gauss_5, whose registers
// leave 16 warps an SM, 78 % at gauss_2), at 69 % of lanes busy: the windows of
// a warp's columns hold unequal pixel counts.  A gauss_5 tap takes 36 thread
// instructions, 64 in the tile columns: a pixel's coordinates and window serve
// six taps, the weights go through packed operations, and a cell leaves the
// registers once.
// Measured on one B200, insertion alone (the kernels it took over from in
// parentheses): gauss_5, d7, N = 384, 64 particles 17.9 ms (46.8, tile columns
// with shared read-modify-writes), one particle 0.35 ms (1.32, an atomic per
// tap); gauss_2, c1, N = 192, 2048 particles 1.41 ms (2.12, tiles with shared
// atomics).  Blocks an SM: gauss_5 without spills (two of eight warps, 128
// registers) against three at 80, 20.1 against 21.6 ms with the patches dealt
// out; five or four of four warps 20.8 and 20.3.  The two-tap windows at three
// blocks 1.52 ms, two 1.70, four 1.60, five 1.71 (spills).
//
// Tap selection and weights are the reference's bit for bit (window start,
// exp-table index, radius); a cell's taps of one slice are summed before they
// reach the volume, so only the order of additions differs from one atomic
// per tap.
//
// Reference: do_insert_slice_work (libEM/reconstructor.cpp:1122-1210),
// insert_pixel (libEM/reconstructor_tools.cpp:128-230, 315-376),
// add_complex_at_fast (libEM/emdata_core.h:368-410).
#include <algorithm>
#include <climits>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

#include "fr_device.cuh"
#include "fr_internal.h"

namespace fr {
namespace plane {

constexpr float kDel = 0.02f;   // slack on the approximate plane geometry

// Taps of a window along one axis, its reach (a pixel at p covers tap t iff
// t - lo <= p < t + hi) and the most cells a column's run can hold: the
// plane's height over the (lo+hi)-wide square window varies by at most
// 2 (lo+hi), its slopes being at most 1 along the dominant axis.  EXP: the
// fast_exp entries kept in shared memory; gauss_5's largest r*h*50 is
// 36.75 * 0.949 * 50 < 1745, past the reference's 1000 entries (the rest read
// as 0 and are replaced), gauss_2's 3 * 2.468 * 50 < 371.
template <int MODE> struct Win;
template <> struct Win<MODE_GAUSS5> {
  static constexpr float lo = 2.5f, hi = 3.5f;
  static constexpr int K = 6, W = 20, EXP = 2048, NT = 256, CTAS = 2, DRAW = 2;
};
template <> struct Win<MODE_GAUSS2> {
  static constexpr float lo = 1.0f, hi = 1.0f;
  static constexpr int K = 2, W = 8, EXP = 512, NT = 256, CTAS = 3, DRAW = 8;
};
template <> struct Win<MODE_TRILINEAR> : Win<MODE_GAUSS2> {
  static constexpr int EXP = 0;
};

// What a warp's columns of one slice share, in the warp's own shared words.
// u*, v*: the first two rows of the rotation, components along A, B and C.
// The rest is linear in the column (tb, tc): the rows its window meets
// (ylo, yhi), the first cells its pixels can start at (alo, ahi), and per row
// y the x range [lo, hi] each of its two window constraints leaves, lo = L +
// tb * I + y * S and hi likewise from U (kDel wider than the window).
struct SliceGeom {
  float ua, ub, uc, w;
  float va, vb, vc, pad;
  float yb, yc, ylo, yhi;
  float ab, ac, alo, ahi;
  float Ib, Lb, Ub, Sb;
  float Ic, Lc, Uc, Sc;
};

struct Smem {
  const float *exp;     // [Win<MODE>::EXP]
  const float *rtab;    // [N+2]
  const short *xmax;    // [N]
  SliceGeom *geom;      // this warp's
  float2 *sv;           // [W][32] this warp's value sums, lane-minor
  float *sw;            // [W][32] this warp's weight sums
  int *ticket;          // the block's next patch
};

// Util::fast_exp's table entry for f = -y, y in [0, 41).  The reference's
// index (int)(y*50.0 + 0.5) (double) is floor(50y + 1/2): one multiply-add
// rounded down onto the spacing of [2^21, 2^22), 1/4, leaves four times that
// floor (and two lower bits) in the mantissa, which is the entry's byte
// offset.  Exact for every float y: the product and sum are not rounded before.
constexpr float kIndex = 2097152.5f;   // 2^21 + 1/2
__device__ __forceinline__ float exp_at(float t, const float *tab) {
  return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(tab) +
                                          (__float_as_int(t) & 0x1FFC));
}

// First tap of a pixel's window, as an integer-valued float: floor(p - 2.5)
// (gauss_5) or floor(p), by additions rounded down onto a spacing of 1/2 and
// then 1 (floor of a floor onto a finer grid), |p| < 2^20.
template <int MODE> __device__ __forceinline__ float win_start(float p, int &start) {
  float t;
  if (MODE == MODE_GAUSS5) t = __fadd_rd(__fadd_rd(p, 6291456.0f - 2.5f), 6291456.0f);
  else t = __fadd_rd(p, 12582912.0f);
  start = __float_as_int(t) - 0x4B400000;
  return __fsub_rn(t, 12582912.0f);
}

// Pairs of floats: one issue slot for two operations, each rounded as its
// scalar form.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(f2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// The squares of a pair, each rounded before it is added to: a packed product
// whose only use is a packed sum comes out of the assembler as one fused
// operation, .rn or not, so these two stay scalar.
__device__ __forceinline__ f2 square2(f2 v) {
  float a, b;
  unpack(v, a, b);
  return pack(__fmul_rn(a, a), __fmul_rn(b, b));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 fma2_rd(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Adds (re, im, w) to one cell of the run.
__device__ __forceinline__ void cell_add(const Smem &S, int at, float re, float im, float w) {
  float2 v = S.sv[at];
  v.x += re;
  v.y += im;
  S.sv[at] = v;
  S.sw[at] += w;
}

// Word of cell (i, j, l), i >= 0, in a centre copy of half-width c.
__device__ __forceinline__ int centre_cell(int c, int i, int j, int l) {
  return ((l + c) * (2 * c + 1) + j + c) * (c + 1) + i;
}

// add_tap_atomic's placement rules in a partial volume; launch_merge keeps the
// imaginary parts of the two self-conjugate cells zero.
__device__ __forceinline__ void quad_tap(float4 *quad, int N, int x, int y, int z, float re,
                                         float im, float w) {
  const int h = N >> 1, w2 = h + 1;
  if (abs(x) > h || abs(y) > h || abs(z) > h) return;
  float4 *mirror = quad + (size_t)((y <= 0 ? -y : N - y) + (z <= 0 ? -z : N - z) * N) * w2 + abs(x);
  if (x == 0 || abs(x) == h) {
    if (y == 0 && z == 0) {
      atomicAdd(mirror, make_float4(re, 0.0f, w, 0.0f));
      return;
    }
    atomicAdd(mirror, make_float4(re, -im, 0.0f, 0.0f));
  }
  if (x < 0) {
    atomicAdd(mirror, make_float4(re, -im, w, 0.0f));
    return;
  }
  atomicAdd(quad + (size_t)((y < 0 ? N + y : y) + (z < 0 ? N + z : z) * N) * w2 + x,
            make_float4(re, im, w, 0.0f));
}

// Adds the sums of tap cell (i, j, l) of a slice to the volume, or to the
// slice's copy of the cells near the origin (see plane_centre).
__device__ __forceinline__ void place(const InsertJob &J, float2 *cd, float *cn, int i, int j, int l,
                                      float re, float im, float w) {
  const int N = J.N, n2 = N >> 1, w2 = n2 + 1;
  const int ia = abs(i), c = J.centre;
  const bool near = cd && ia <= c && abs(j) <= c && abs(l) <= c;
  if (ia == 0 || ia >= n2) {
    if (near) {   // i = 0 (c < N/2): both mirror cells, the mirrored one without weight
      const int at = centre_cell(c, 0, j, l);
      const bool origin = j == 0 && l == 0;
      if (!origin) atomicAdd(cd + centre_cell(c, 0, -j, -l), make_float2(re, -im));
      atomicAdd(cd + at, make_float2(re, origin ? 0.0f : im));
      atomicAdd(cn + at, w);
    } else if (J.quad) {
      quad_tap(J.quad, N, i, j, l, re, im, w);
    } else {
      add_tap_atomic(J.data, J.norm, N, N, i, j, l, re, im, w);
    }
    return;
  }
  if (abs(j) > n2 || abs(l) > n2) return;
  // add_complex_at_fast away from the planes x = 0 and |x| = N/2: the cell,
  // or for x < 0 its mirror, conjugated
  if (i < 0) {
    j = -j;
    l = -l;
    im = -im;
  }
  size_t at;
  float2 *data = reinterpret_cast<float2 *>(J.data);
  float *norm = J.norm;
  if (near) {
    at = centre_cell(c, ia, j, l);
    data = cd;
    norm = cn;
  } else {
    at = (size_t)ia + (size_t)((j < 0 ? N + j : j) + (l < 0 ? N + l : l) * N) * w2;
    if (J.quad) {
      atomicAdd(J.quad + at, make_float4(re, im, w, 0.0f));
      return;
    }
  }
  atomicAdd(data + at, make_float2(re, im));
  atomicAdd(norm + at, w);
}

// One column (tb, tc) of the slice, a lane each.
template <int MODE>
__device__ __forceinline__ void column(const InsertJob &J, const Smem &S, int A, int tb, int tc,
                                       const float2 *__restrict__ sl, float h, float2 *cd,
                                       float *cn) {
  constexpr float LO = Win<MODE>::lo, HI = Win<MODE>::hi;
  const int N = J.N, n2 = N >> 1, w2 = n2 + 1;
  const int lane = threadIdx.x & 31;
  const float Nf = (float)N;
  const SliceGeom &G = *S.geom;
  const float tbf = (float)tb, tcf = (float)tc;
  // exact window bounds on the pixel's coordinates.  A gauss_5 pixel is
  // skipped whole when its window starts below -N/2-4
  // (libEM/reconstructor_tools.cpp:321), which only a column at -N/2 can meet.
  const float edge = (float)(-n2) - 1.5f;
  const float lob = MODE == MODE_GAUSS5 ? fmaxf(tbf - LO, edge) : tbf - LO, hib = tbf + HI;
  const float loc = MODE == MODE_GAUSS5 ? fmaxf(tcf - LO, edge) : tcf - LO, hic = tcf + HI;
  const float yv0 = fmaf(tbf, G.yb, tcf * G.yc), av0 = fmaf(tbf, G.ab, tcf * G.ac);
  const int r0 = max(-n2, __float2int_ru(yv0 + G.ylo)),
            r1 = min(n2 - 1, __float2int_rd(yv0 + G.yhi));
  const int kb = __float2int_rd(av0 + G.alo);
  const int nq = __float2int_rd(av0 + G.ahi) + Win<MODE>::K - kb;   // cells of the run
  const float Lb = fmaf(tbf, G.Ib, G.Lb), Ub = fmaf(tbf, G.Ib, G.Ub);
  const float Lc = fmaf(tcf, G.Ic, G.Lc), Uc = fmaf(tcf, G.Ic, G.Uc);
  const float Sb = G.Sb, Sc = G.Sc;
  const float ua = G.ua, ub = G.ub, uc = G.uc, w = G.w;
  const float vscale = MODE == MODE_TRILINEAR ? 1.0f : w;
  const int cell0 = lane - kb * 32;      // cell k of the run is word cell0 + 32 k

#pragma unroll 1
  for (int y = r0; y <= r1; y++) {
    const float yf = (float)y;
    const int xm = S.xmax[y + n2];
    const float xlo = fmaxf(fmaxf(fmaf(yf, Sb, Lb), fmaf(yf, Sc, Lc)), 0.0f);
    const float xhi = fminf(fminf(fmaf(yf, Sb, Ub), fmaf(yf, Sc, Uc)), (float)xm);
    const int c0 = __float2int_ru(xlo), c1 = __float2int_rd(xhi);
    if (c0 > c1) continue;
    const float ry = S.rtab[y + n2];
    const float qa = __fmul_rn(ry, G.va), qb = __fmul_rn(ry, G.vb), qc = __fmul_rn(ry, G.vc);
    const float2 *rowp = sl + (size_t)(y < 0 ? N + y : y) * w2;
    // heights rise along the walk, so gauss_5's window only moves up
    const int dx = ua < 0.0f ? -1 : 1;
    int x = ua < 0.0f ? c1 : c0;
    float ar[6], ai[6], aw[6];
    int cur = INT_MAX;     // gauss_5: the cell of ar[0], ...
    if (MODE == MODE_GAUSS5) {
#pragma unroll
      for (int t = 0; t < 6; t++) ar[t] = ai[t] = aw[t] = 0.0f;
    }
#pragma unroll 1
    for (int cnt = c1 - c0; cnt >= 0; cnt--, x += dx) {
      const float rx = S.rtab[x + n2];
      const float pb = __fmul_rn(__fadd_rn(__fmul_rn(rx, ub), qb), Nf);
      const float pc = __fmul_rn(__fadd_rn(__fmul_rn(rx, uc), qc), Nf);
      const float pa = __fmul_rn(__fadd_rn(__fmul_rn(rx, ua), qa), Nf);
      bool in;
      if (MODE == MODE_GAUSS5)
        in = lob <= pb && pb < hib && loc <= pc && pc < hic && pa >= edge;
      else
        in = lob <= pb && pb < hib && loc <= pc && pc < hic;
      if (!in) continue;
      float2 v = __ldg(rowp + x);
      if (x == 0 && y < 0) {   // reads (0, -y) conjugated
        v = __ldg(sl + (size_t)(-y) * w2);
        v.y = -v.y;
      }
      v.x *= vscale;
      v.y *= vscale;
      int a0;
      const float a0f = win_start<MODE>(pa, a0);
      const float db = __fsub_rn(tbf, pb), dc = __fsub_rn(tcf, pc);
      if (MODE == MODE_TRILINEAR) {
        // (libEM/reconstructor_tools.cpp:191-230): double products
        const double ob = 1.0 - fabs((double)db), oc = 1.0 - fabs((double)dc);
#pragma unroll
        for (int t = 0; t < 2; t++) {
          const double oa = 1.0 - fabs((double)__fsub_rn(a0f + (float)t, pa));
          const double q = A == 2 ? (ob * oc) * oa : (oa * ob) * oc;
          const float g = (float)(q * (double)w);
          cell_add(S, cell0 + (a0 + t) * 32, v.x * g, v.y * g, g);
        }
        continue;
      }
      // r = (dx^2 + dy^2) + dz^2 (libEM/util.h:816-819): with A = z the sum
      // of the other two comes first, else A's square is in the first sum
      float f0 = __fmul_rn(db, db), f1 = __fmul_rn(dc, dc);
      if (A == 2) {
        f0 = __fadd_rn(f0, f1);
        f1 = 0.0f;
      }
      const f2 npa = pack(-pa, -pa), f00 = pack(f0, f0), f11 = pack(f1, f1), hh = pack(h, h);
      const f2 c50 = pack(50.0f, 50.0f), cidx = pack(kIndex, kIndex), aa = pack(a0f, a0f);
      if (MODE == MODE_GAUSS2) {
        const f2 d = add2(add2(aa, pack(0.0f, 1.0f)), npa);
        const f2 r = add2(add2(square2(d), f00), f11);
        float t0, t1;
        unpack(fma2_rd(mul2(r, hh), c50, cidx), t0, t1);
        const float g0 = exp_at(t0, S.exp), g1 = exp_at(t1, S.exp);   // r <= 3: in the table
        const int at = cell0 + a0 * 32;
        float2 q0 = S.sv[at], q1 = S.sv[at + 32];
        float w0 = S.sw[at], w1 = S.sw[at + 32];
        q0.x = fmaf(v.x, g0, q0.x);
        q0.y = fmaf(v.y, g0, q0.y);
        q1.x = fmaf(v.x, g1, q1.x);
        q1.y = fmaf(v.y, g1, q1.y);
        S.sv[at] = q0;
        S.sv[at + 32] = q1;
        S.sw[at] = w0 + g0;
        S.sw[at + 32] = w1 + g1;
        continue;
      }
      // gauss_5: move the window up to a0 (at most one cell: heights change
      // by less than one a pixel), handing the cell below it over
      cur = min(cur, a0);
      if (cur < a0) {
        cell_add(S, cell0 + cur * 32, ar[0], ai[0], aw[0]);
#pragma unroll
        for (int t = 0; t < 5; t++) { ar[t] = ar[t + 1]; ai[t] = ai[t + 1]; aw[t] = aw[t + 1]; }
        ar[5] = ai[5] = aw[5] = 0.0f;
        cur = a0;
      }
      float yv[6], g[6];
#pragma unroll
      for (int t = 0; t < 6; t += 2) {
        const f2 d = add2(add2(aa, pack((float)t, (float)(t + 1))), npa);
        const f2 r = add2(add2(square2(d), f00), f11);
        const f2 yy = mul2(r, hh);
        float t0, t1;
        unpack(yy, yv[t], yv[t + 1]);
        unpack(fma2_rd(yy, c50, cidx), t0, t1);
        g[t] = exp_at(t0, S.exp);
        g[t + 1] = exp_at(t1, S.exp);
      }
      // past the table (y > 19.98, r > 21.05) the reference calls exp: d^2 is
      // at most 12.25 for the first tap and 6.25 for the others
      const float f01 = f0 + f1;
      if (f01 > 8.7f) {
        if (yv[0] > 19.98f) g[0] = expf(-yv[0]);
        if (f01 > 14.7f) {
#pragma unroll
          for (int t = 1; t < 6; t++)
            if (yv[t] > 19.98f) g[t] = expf(-yv[t]);
        }
      }
      const f2 vx = pack(v.x, v.x), vy = pack(v.y, v.y);
#pragma unroll
      for (int t = 0; t < 6; t += 2) {
        const f2 gg = pack(g[t], g[t + 1]);
        unpack(fma2(vx, gg, pack(ar[t], ar[t + 1])), ar[t], ar[t + 1]);
        unpack(fma2(vy, gg, pack(ai[t], ai[t + 1])), ai[t], ai[t + 1]);
        unpack(add2(gg, pack(aw[t], aw[t + 1])), aw[t], aw[t + 1]);
      }
    }
    if (MODE == MODE_GAUSS5 && cur != INT_MAX) {
#pragma unroll
      for (int t = 0; t < 6; t++) cell_add(S, cell0 + (cur + t) * 32, ar[t], ai[t], aw[t]);
    }
  }
  // the run into the volume; its words go back to zero for the next column
  const float wscale = MODE == MODE_TRILINEAR ? 1.0f : w;
  // Most runs stay clear of the planes x = 0 and N/2, of the row or slab where
  // indices wrap and of the centre copies: their cells are one stride apart,
  // and a run below x = 0 goes to its mirror cells, conjugated.
  const int ke = kb + nq - 1, reach = max(abs(tb), abs(tc)), side = A == 0 ? kb : tb;
  const int centre = cd ? J.centre : -1;
  if (max(reach, max(abs(kb), abs(ke))) < n2 && (kb > 0 || ke < 0) && side != 0 &&
      !(reach <= centre && min(abs(kb), abs(ke)) <= centre)) {
    const int sg = side < 0 ? -1 : 1;
    const int i = sg * side, j = sg * (A == 1 ? kb : (A == 0 ? tb : tc)), l = sg * (A == 2 ? kb : tc);
    const size_t at = (size_t)i + (size_t)((j < 0 ? N + j : j) + (l < 0 ? N + l : l) * N) * w2;
    const int step = sg * (A == 0 ? 1 : (A == 1 ? w2 : w2 * N));
    const float sgf = (float)sg;
    if (J.quad) {   // one reduction a cell
      float4 *pq = J.quad + at;
      float2 *pv = S.sv + lane;
      float *pw = S.sw + lane;
#pragma unroll 1
      for (int q = 0; q < nq; q++, pq += step, pv += 32, pw += 32) {
        const float2 v = *pv;
        const float s = *pw;
        if (v.x == 0.0f && v.y == 0.0f && s == 0.0f) continue;
        *pv = make_float2(0.0f, 0.0f);
        *pw = 0.0f;
        atomicAdd(pq, make_float4(v.x, sgf * v.y, s * wscale, 0.0f));
      }
      return;
    }
    float2 *pd = reinterpret_cast<float2 *>(J.data) + at;
    float *pn = J.norm + at;
    float2 *pv = S.sv + lane;
    float *pw = S.sw + lane;
#pragma unroll 1
    for (int q = 0; q < nq; q++, pd += step, pn += step, pv += 32, pw += 32) {
      const float2 v = *pv;
      const float s = *pw;
      if (v.x == 0.0f && v.y == 0.0f && s == 0.0f) continue;
      *pv = make_float2(0.0f, 0.0f);
      *pw = 0.0f;
      atomicAdd(pd, make_float2(v.x, sgf * v.y));
      atomicAdd(pn, s * wscale);
    }
    return;
  }
#pragma unroll 1
  for (int q = 0; q < nq; q++) {
    const int at = q * 32 + lane;
    const float2 v = S.sv[at];
    const float s = S.sw[at];
    if (v.x == 0.0f && v.y == 0.0f && s == 0.0f) continue;
    S.sv[at] = make_float2(0.0f, 0.0f);
    S.sw[at] = 0.0f;
    const int k = kb + q;
    const int i = A == 0 ? k : tb, j = A == 0 ? tb : (A == 1 ? k : tc), l = A == 2 ? k : tc;
    place(J, cd, cn, i, j, l, v.x, v.y, s * wscale);
  }
}

// x range lines of one window constraint t - lo <= x*u + y*v < t + hi.
__device__ __forceinline__ void band(float lo, float hi, float u, float v, float &I, float &L,
                                     float &U, float &S) {
  if (fabsf(u) > 1e-4f) {
    I = 1.0f / u;
    const float p = (-lo - kDel) * I, q = (hi + kDel) * I;
    L = fminf(p, q);
    U = fmaxf(p, q);
    S = -v * I;
  } else {   // nearly constant along the row: left to the exact window test
    I = S = 0.0f;
    L = -1e9f;
    U = 1e9f;
  }
}

// A block's `count` units of one job: u, u + step, ..., unit i being part i %
// parts of slice i / parts, which has that slice's patches i % parts + k parts.
// The warps draw them, DRAW at a time; the ticket starts at 0.  Dealt out
// beforehand they left the warps up to a quarter apart, patches at the disc's
// edge holding less (gauss_5, d7, N = 384, one particle: an SM busy 592,000
// cycles on average, 737,000 at most): one particle 423 us against 355 now,
// 128 307 against 280 each; gauss_2, d7, N = 384 39.4 against 35.3.
template <int MODE, int DRAW>
__device__ __forceinline__ void run_units(const InsertJob &J, const Smem &S, int u, int step,
                                          int count, int parts, float h,
                                          const float *__restrict__ table) {
  constexpr float LO = Win<MODE>::lo, HI = Win<MODE>::hi;
  constexpr float E = 0.5f * (LO + HI) + kDel, C = 0.5f * (HI - LO);
  constexpr float OFF = MODE == MODE_GAUSS5 ? 2.5f : 0.0f;
  const int N = J.N, n2 = N >> 1, w2 = n2 + 1;
  const int lane = threadIdx.x & 31;
  // the farthest column of the half disk x >= 0, |p| <= R
  const float R = J.corners ? n2 * 1.4143f + 1.0f : n2 + 0.52f;
  const int share = ((N / 8 + 1) * (N / 4 + 1) + parts * DRAW - 1) / (parts * DRAW);
  // what the warp's tickets of one unit share
  int cur = -1, part = 0, A = 0, b0 = 0, c0 = 0, nb = 1, total = 0;
  float ub = 0, uc = 0, vb = 0, vc = 0, idet = 0, ex = 0, ey = 0;
  const float2 *sl = nullptr;
  float2 *cd = nullptr;
  float *cn = nullptr;
#pragma unroll 1
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(S.ticket, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    const int i = t / share, k = t - i * share;
    if (i >= count) break;
    if (i != cur) {
      cur = i;
      const int v = u + i * step, s = v / parts;
      part = v - s * parts;
      const int p = s / J.nsym;
      const float w = __ldg(&J.pw[p]);
      float M[6];
#pragma unroll
      for (int e = 0; e < 6; e++) M[e] = __ldg(&J.t3d[9 * (size_t)s + e]);
      sl = J.slices + (size_t)p * N * w2;
      const float lu = M[0] * M[0] + M[1] * M[1] + M[2] * M[2];
      const float lv = M[3] * M[3] + M[4] * M[4] + M[5] * M[5];
      const float uv = M[0] * M[3] + M[1] * M[4] + M[2] * M[5];
      total = w == 0.0f ? 0
              : fabsf(lu - 1.0f) < 0.01f && fabsf(lv - 1.0f) < 0.01f && fabsf(uv) < 0.01f
                  ? 1
                  : -1;   // not a rotation (a caller's own matrix)
      if (total > 0) {
        const float nx = M[1] * M[5] - M[2] * M[4], ny = M[2] * M[3] - M[0] * M[5],
                    nz = M[0] * M[4] - M[1] * M[3];
        const float ax = fabsf(nx), ay = fabsf(ny), az = fabsf(nz);
        A = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
        const float ua = A == 0 ? M[0] : (A == 1 ? M[1] : M[2]),
                    va = A == 0 ? M[3] : (A == 1 ? M[4] : M[5]);
        ub = A == 0 ? M[1] : M[0];
        uc = A == 2 ? M[1] : M[2];
        vb = A == 0 ? M[4] : M[3];
        vc = A == 2 ? M[4] : M[5];
        idet = 1.0f / (ub * vc - uc * vb);
        // (pb, pc) -> y and the plane's height pa, over the windows' extent
        SliceGeom G;
        G.ua = ua; G.ub = ub; G.uc = uc; G.w = w;
        G.va = va; G.vb = vb; G.vc = vc; G.pad = 0.0f;
        G.yb = -uc * idet;
        G.yc = ub * idet;
        const float y0 = C * (G.yb + G.yc), yy = E * (fabsf(G.yb) + fabsf(G.yc));
        G.ylo = y0 - yy;
        G.yhi = y0 + yy;
        G.ab = (vc * ua - uc * va) * idet;
        G.ac = (ub * va - vb * ua) * idet;
        const float a0 = C * (G.ab + G.ac) - OFF, ea = E * (fabsf(G.ab) + fabsf(G.ac)) + kDel;
        G.alo = a0 - ea;
        G.ahi = a0 + ea;
        band(LO, HI, ub, vb, G.Ib, G.Lb, G.Ub, G.Sb);
        band(LO, HI, uc, vc, G.Ic, G.Lc, G.Uc, G.Sc);
        __syncwarp();
        if (lane == 0) *S.geom = G;
        __syncwarp();
        // the tap columns that the half disk reaches
        const float hb = R * sqrtf(ub * ub + vb * vb), gb = R * fabsf(vb);
        const float hc = R * sqrtf(uc * uc + vc * vc), gc = R * fabsf(vc);
        b0 = max(-n2, __float2int_ru((ub < 0 ? -hb : -gb) - HI - kDel));
        c0 = max(-n2, __float2int_ru((uc < 0 ? -hc : -gc) - HI - kDel));
        const int b1 = min(n2, __float2int_rd((ub < 0 ? gb : hb) + LO + kDel));
        const int c1 = min(n2, __float2int_rd((uc < 0 ? gc : hc) + LO + kDel));
        nb = ((b1 - b0) >> 3) + 1;
        total = b1 < b0 || c1 < c0 ? 0 : nb * (((c1 - c0) >> 2) + 1);
        ex = (fabsf(vc) * (E + 3.5f) + fabsf(vb) * (E + 1.5f)) * fabsf(idet);
        ey = (fabsf(ub) * (E + 1.5f) + fabsf(uc) * (E + 3.5f)) * fabsf(idet);
        cd = nullptr;
        if (J.cdata) {
          const size_t cells = (size_t)(J.centre + 1) * (2 * J.centre + 1) * (2 * J.centre + 1);
          cd = reinterpret_cast<float2 *>(J.cdata) + (s % J.copies) * cells;
          cn = J.cdata + 2 * J.copies * cells + (s % J.copies) * cells;
        }
      }
    }
    if (total < 0) {   // tap by tap
      const int s = (u + i * step) / parts;
      const float w = __ldg(&J.pw[s / J.nsym]);
      float M[6];
#pragma unroll
      for (int e = 0; e < 6; e++) M[e] = __ldg(&J.t3d[9 * (size_t)s + e]);
      for (int e = (part * share + k) * 32 + lane; e < N * w2; e += parts * share * 32) {
        const int x = e % w2, y = e / w2 - n2;
        if (x > S.xmax[y + n2]) continue;
        float xx, yy, zz;
        pixel_coords(S.rtab[x + n2], S.rtab[y + n2], M, (float)N, xx, yy, zz);
        const float2 v = slice_value(sl, N, x, y);
        insert_pixel_atomic<MODE>(J.data, J.norm, N, N, xx, yy, zz, v.x, v.y, w, h, table, false);
      }
      continue;
    }
    int q = part + k * DRAW * parts;
    if (q >= total) {   // the unit is done
      if (lane == 0) atomicMax(S.ticket, (i + 1) * share);
      continue;
    }
    const int dqc = DRAW > 1 ? parts / nb : 0, dqb = parts - dqc * nb;
    int qc = q / nb, qb = q - qc * nb;
#pragma unroll 1
    for (int d = 0; d < DRAW && q < total; d++, q += parts) {
      if (d > 0) {
        qc += dqc;
        qb += dqb;
        if (qb >= nb) {
          qb -= nb;
          qc++;
        }
      }
      const int tb0 = b0 + qb * 8, tc0 = c0 + qc * 4;
      // the patch's windows in slice coordinates: any pixel of the half disk?
      const float pb = tb0 + 3.5f + C, pc = tc0 + 1.5f + C;
      const float xc = (pb * vc - pc * vb) * idet, yc = (ub * pc - uc * pb) * idet;
      const float dx = fmaxf(0.0f, fabsf(xc) - ex), dy = fmaxf(0.0f, fabsf(yc) - ey);
      if (xc + ex < -kDel || dx * dx + dy * dy > R * R) continue;
      const int tb = tb0 + (lane & 7), tc = tc0 + (lane >> 3);
      if (tb <= n2 && tc <= n2) column<MODE>(J, S, A, tb, tc, sl, h, cd, cn);
      __syncwarp();
    }
  }
}

template <int MODE>
__device__ __forceinline__ void smem_layout(Smem &S, unsigned char *dyn, int maxN, float *&exp,
                                            float *&rtab, short *&xmax) {
  constexpr int W = Win<MODE>::W, NW = Win<MODE>::NT / 32;
  const int warp = threadIdx.x >> 5;
  S.geom = reinterpret_cast<SliceGeom *>(dyn) + warp;
  float2 *sv = reinterpret_cast<float2 *>(dyn + NW * sizeof(SliceGeom));
  float *sw = reinterpret_cast<float *>(sv + NW * W * 32);
  exp = sw + NW * W * 32;
  rtab = exp + Win<MODE>::EXP;
  xmax = reinterpret_cast<short *>(rtab + maxN + 2);
  S.sv = sv + warp * W * 32;
  S.sw = sw + warp * W * 32;
  S.exp = exp;
  S.rtab = rtab;
  S.xmax = xmax;
}

template <int MODE> size_t smem_bytes(int maxN) {
  constexpr int NW = Win<MODE>::NT / 32;
  return NW * sizeof(SliceGeom) + (size_t)NW * Win<MODE>::W * 32 * 12 + Win<MODE>::EXP * 4 +
         4 * (size_t)(maxN + 2) + 2 * (size_t)maxN;
}

template <int MODE>
__device__ __forceinline__ void smem_init(const Smem &S, float *exp,
                                          const float *__restrict__ table) {
  for (int i = threadIdx.x; i < Win<MODE>::EXP; i += Win<MODE>::NT) exp[i] = i < 1000 ? __ldg(&table[i]) : 0.0f;
  for (int i = threadIdx.x & 31; i < Win<MODE>::W * 32; i += 32) {
    S.sv[i] = make_float2(0.0f, 0.0f);
    S.sw[i] = 0.0f;
  }
}

__device__ __forceinline__ void load_geometry(const InsertJob &J, float *rtab, short *xmax) {
  for (int i = threadIdx.x; i < J.N + 2; i += blockDim.x) rtab[i] = __ldg(&J.rtab[i]);
  for (int i = threadIdx.x; i < J.N; i += blockDim.x) xmax[i] = (short)__ldg(&J.xmax[i]);
}

}  // namespace plane

// One job: unit u is part u % parts of slice u / parts.
template <int MODE, int DRAW>
__global__ void __launch_bounds__(plane::Win<MODE>::NT, plane::Win<MODE>::CTAS)
    k_plane(InsertJob J, int units, int parts, float h, const float *__restrict__ table) {
  extern __shared__ __align__(16) unsigned char dyn[];
  plane::Smem S;
  float *exp, *rtab;
  short *xmax;
  __shared__ int s_ticket;
  plane::smem_layout<MODE>(S, dyn, J.N, exp, rtab, xmax);
  plane::smem_init<MODE>(S, exp, table);
  plane::load_geometry(J, rtab, xmax);
  S.ticket = &s_ticket;
  if (threadIdx.x == 0) s_ticket = 0;
  __syncthreads();
  const int u = blockIdx.x, step = gridDim.x;
  plane::run_units<MODE, DRAW>(J, S, u, step, (units - u + step - 1) / step, parts, h, table);
}

// Several jobs of one mode: job segs[i].job has the units from segs[i].first on.
template <int MODE, int DRAW>
__global__ void __launch_bounds__(plane::Win<MODE>::NT, plane::Win<MODE>::CTAS)
    k_plane_multi(const InsertJob *__restrict__ jobs, const PlaneSeg *__restrict__ segs, int nsegs,
                  int units, int maxN, float h, const float *__restrict__ table) {
  extern __shared__ __align__(16) unsigned char dyn[];
  plane::Smem S;
  float *exp, *rtab;
  short *xmax;
  plane::smem_layout<MODE>(S, dyn, maxN, exp, rtab, xmax);
  plane::smem_init<MODE>(S, exp, table);
  __shared__ int s_ticket;
  S.ticket = &s_ticket;
  const int step = gridDim.x;
  for (int u = blockIdx.x; u < units;) {
    int lo = 0, hi = nsegs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (segs[mid].first <= u) lo = mid;
      else hi = mid - 1;
    }
    const PlaneSeg g = segs[lo];
    const int end = lo + 1 < nsegs ? segs[lo + 1].first : units;
    const int count = (end - u + step - 1) / step;   // the block's units of this job
    const InsertJob J = jobs[g.job];
    __syncthreads();
    plane::load_geometry(J, rtab, xmax);
    if (threadIdx.x == 0) s_ticket = 0;
    __syncthreads();
    plane::run_units<MODE, DRAW>(J, S, u - g.first, step, count, g.parts, h, table);
    u += count * step;
  }
}

// Adds a job's partial volume to its accumulators and clears it.  One block
// per row; cells farther than the pixels and their windows reach are skipped.
// The two self-conjugate cells keep a zero imaginary part once touched.
__global__ void __launch_bounds__(128)
    k_merge(float2 *__restrict__ data, float *__restrict__ norm, float4 *__restrict__ quad, int N,
            float reach) {
  const int w2 = N / 2 + 1;
  const int y = blockIdx.x, z = blockIdx.y;
  const float fy = (float)(y <= N / 2 ? y : y - N), fz = (float)(z <= N / 2 ? z : z - N);
  const float left = reach * reach - fy * fy - fz * fz;
  if (left < 0.0f) return;
  const int n = min(w2, (int)sqrtf(left) + 2);
  const size_t row = ((size_t)z * N + y) * w2;
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    const float4 v = quad[row + x];
    // (an x = 0 cell may hold conjugate values and no weight)
    if (v.z == 0.0f && v.x == 0.0f && v.y == 0.0f) continue;
    float2 d = data[row + x];
    d.x += v.x;
    d.y += v.y;
    if (y == 0 && z == 0 && (x == 0 || x == w2 - 1)) d.y = 0.0f;
    data[row + x] = d;
    norm[row + x] += v.z;
    quad[row + x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// Adds a job's centre copies to its accumulators and clears them: grid.y =
// job, one thread per cell.
__global__ void __launch_bounds__(256)
    k_merge_centre(const InsertJob *__restrict__ jobs, const InsertJob one, int mode) {
  const InsertJob &J = jobs ? jobs[blockIdx.y] : one;
  if (!J.cdata || J.mode != mode) return;
  const int c = J.centre, side = 2 * c + 1, N = J.N, w2 = N / 2 + 1;
  const int cells = (c + 1) * side * side;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= cells) return;
  float2 *cd = reinterpret_cast<float2 *>(J.cdata) + q;
  float *cn = J.cdata + 2 * (size_t)J.copies * cells + q;
  double re = 0.0, im = 0.0, w = 0.0;
  bool any = false;
  for (int k = 0; k < J.copies; k++, cd += cells, cn += cells) {
    const float2 v = *cd;
    const float s = *cn;
    if (v.x == 0.0f && v.y == 0.0f && s == 0.0f) continue;
    any = true;
    re += v.x;
    im += v.y;
    w += s;
    *cd = make_float2(0.0f, 0.0f);
    *cn = 0.0f;
  }
  if (!any) return;
  const int i = q % (c + 1), j = (q / (c + 1)) % side - c, l = q / ((c + 1) * side) - c;
  const size_t at = (size_t)i + (size_t)((j < 0 ? N + j : j) + (l < 0 ? N + l : l) * N) * w2;
  float2 *d = reinterpret_cast<float2 *>(J.data) + at;
  float2 v = *d;
  v.x += (float)re;
  v.y = (i == 0 && j == 0 && l == 0) ? 0.0f : v.y + (float)im;
  *d = v;
  J.norm[at] += (float)w;
}

// Patches drawn at a time: enough that a draw costs little beside them (gauss_5,
// d7, N = 384, 128 particles one 293 us each, two 280; gauss_2, c1, N = 192,
// 2048, one 1.58 ms, four 1.43, eight 1.41, sixteen 1.41 and 111 us a single
// particle of N = 384, d7 instead of 89), but one by one where the warps get
// fewer than four each (gauss_5, c1, N = 192, one slice 74 us, 99 by two).
long plane_patches(int N, long slices) {
  return slices * ((long)(N / 8 + 2) * (N / 4 + 3) * 3 / 4);
}
static bool draw_one(long patches) { return patches < 4 * 148 * 16; }

static int plane_parts(int N, int mode, long slices) {
  // 8 x 4 patches of the bounding box of a slice's columns (at most, about
  // N x N/2 * sqrt 2), one to a warp at a time: a unit (a block's share) is
  // small enough to balance the blocks and large enough to pay for its set-up
  const int warps = 8, per = mode == MODE_GAUSS5 ? 8 : 32;
  const long patches = plane_patches(N, 1);
  const long most = std::max(1L, (patches + warps - 1) / warps);
  const long fine = std::max(1L, (patches + warps * per - 1) / (warps * per));
  const long fill = (148L * 12 + slices - 1) / std::max(1L, slices);
  return (int)std::min(most, std::max(fine, fill));
}

int plane_seg(const InsertJob &j, int job, int first, long slices, PlaneSeg &out) {
  out.job = job;
  out.first = first;
  out.parts = plane_parts(j.N, j.mode, slices);
  const long end = first + (long)j.np * j.nsym * out.parts;
  return end > INT_MAX ? -1 : (int)end;
}

// Blocks that fit the device at once, for a kernel and its shared memory
// (looked up once: the query costs a small call a few microseconds).
static int resident(const void *func, int threads, size_t smem, cudaError_t *e) {
  int dev = 0;
  cudaGetDevice(&dev);
  static std::mutex mu;
  static std::map<std::tuple<const void *, int, size_t>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  int &n = known[std::make_tuple(func, dev, smem)];
  *e = cudaSuccess;
  if (n) return n;
  *e = set_max_smem(func, smem);
  if (*e != cudaSuccess) return 0;
  int sms = 148, per_sm = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  *e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, func, threads, smem);
  if (*e != cudaSuccess) return 0;
  return n = sms * std::max(1, per_sm);
}

template <int MODE>
static cudaError_t launch_t(const InsertJob &j, float h, const float *table, cudaStream_t st) {
  const long slices = (long)j.np * j.nsym;
  const int parts = plane_parts(j.N, j.mode, slices);
  if (slices * parts > INT_MAX) return cudaErrorInvalidValue;
  const int units = (int)(slices * parts);
  const size_t smem = plane::smem_bytes<MODE>(j.N);
  cudaError_t e;
  constexpr int DRAW = plane::Win<MODE>::DRAW;
  auto *kernel = k_plane<MODE, DRAW>;
  if constexpr (MODE == MODE_GAUSS5)
    if (draw_one(plane_patches(j.N, slices))) kernel = k_plane<MODE, 1>;
  const int fit = resident((const void *)kernel, plane::Win<MODE>::NT, smem, &e);
  if (e != cudaSuccess) return e;
  note_launch();
  kernel<<<std::min(units, fit), plane::Win<MODE>::NT, smem, st>>>(j, units, parts, h, table);
  return cudaGetLastError();
}

cudaError_t launch_plane_tables(const InsertJob &j, const float *table, float h, cudaStream_t st) {
  const long slices = (long)j.np * j.nsym;
  if (slices == 0) return cudaSuccess;
  switch (j.mode) {
    case MODE_GAUSS2: return launch_t<MODE_GAUSS2>(j, h, table, st);
    case MODE_GAUSS5: return launch_t<MODE_GAUSS5>(j, h, table, st);
    case MODE_TRILINEAR: return launch_t<MODE_TRILINEAR>(j, h, table, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_plane(const InsertJob &j, cudaStream_t st) {
  const Consts &c = consts();
  return launch_plane_tables(j, c.d_exp, j.mode == MODE_GAUSS5 ? c.h5 : c.h2, st);
}

template <int MODE>
static cudaError_t launch_multi_t(const InsertJob *d_jobs, const PlaneSeg *d_segs, int nsegs,
                                  int units, int maxN, long patches, cudaStream_t st) {
  const Consts &c = consts();
  const size_t smem = plane::smem_bytes<MODE>(maxN);
  cudaError_t e;
  constexpr int DRAW = plane::Win<MODE>::DRAW;
  auto *kernel = k_plane_multi<MODE, DRAW>;
  if constexpr (MODE == MODE_GAUSS5)
    if (draw_one(patches)) kernel = k_plane_multi<MODE, 1>;
  const int fit = resident((const void *)kernel, plane::Win<MODE>::NT, smem, &e);
  if (e != cudaSuccess) return e;
  note_launch();
  kernel<<<std::min(units, fit), plane::Win<MODE>::NT, smem, st>>>(
      d_jobs, d_segs, nsegs, units, maxN, MODE == MODE_GAUSS5 ? c.h5 : c.h2, c.d_exp);
  return cudaGetLastError();
}

cudaError_t launch_plane_multi(const InsertJob *d_jobs, const PlaneSeg *d_segs, int nsegs,
                               int units, int mode, int maxN, long patches, cudaStream_t st) {
  if (units == 0) return cudaSuccess;
  switch (mode) {
    case MODE_GAUSS2: return launch_multi_t<MODE_GAUSS2>(d_jobs, d_segs, nsegs, units, maxN, patches, st);
    case MODE_GAUSS5: return launch_multi_t<MODE_GAUSS5>(d_jobs, d_segs, nsegs, units, maxN, patches, st);
    case MODE_TRILINEAR:
      return launch_multi_t<MODE_TRILINEAR>(d_jobs, d_segs, nsegs, units, maxN, patches, st);
    default: return cudaErrorInvalidValue;
  }
}

size_t plane_centre(int N, long slices, int &half, int &copies) {
  half = std::min(15, N / 2 - 1);
  copies = (int)std::min(32L, (std::min(slices, (long)kPlaneTurn) + 63) / 64);
  return slices < 16 ? 0 : 12 * (size_t)copies * (half + 1) * (2 * half + 1) * (2 * half + 1);
}

cudaError_t launch_merge_centre(const InsertJob *d_jobs, int njobs, const InsertJob *one, int mode,
                                int half, cudaStream_t st) {
  const int cells = (half + 1) * (2 * half + 1) * (2 * half + 1);
  note_launch();
  k_merge_centre<<<dim3((cells + 255) / 256, njobs), 256, 0, st>>>(d_jobs, one ? *one : InsertJob(),
                                                                   mode);
  return cudaGetLastError();
}

cudaError_t launch_merge(const InsertJob &j, cudaStream_t st) {
  // the farthest pixel (the kernel takes matrices within 1 % of a rotation)
  // and the corner of its window
  const float reach = 1.01f * (j.corners ? 0.7072f * j.N + 1.0f : 0.5f * j.N + 0.52f) + 3.5f * 1.7321f;
  note_launch();
  k_merge<<<dim3(j.N, j.N), 128, 0, st>>>(reinterpret_cast<float2 *>(j.data), j.norm, j.quad, j.N,
                                          reach);
  return cudaGetLastError();
}

}  // namespace fr
