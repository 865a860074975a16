// fr_slice.cu -- the whole per-particle preparation in one launch, for images
// whose padded size fits one SM's shared memory.
//
// The pipeline of fr_prologue.cu (edge mean, zero-padded clip, CTF phase flip
// through a 2-D FFT and back, edge mean, bilinear shift, phase origin to
// corner, r2c FFT) reads and writes its images in HBM at every stage.  Here a
// block owns one particle and its padded image never leaves shared memory
// between the raw pixels and the finished slice.
//
// What bounds it: instructions between barriers (55 % of cycles issue; some
// twenty passes over the image in shared memory, 8 per value and pass).  With
// their insertion's fixed cost, particles with a CTF: box 128 (N = 192), 2,048
// in 1.13 ms against 1.83 in nine launches whose transforms move 1.2 GB each;
// box 64 (N = 96), 2,000 in 0.36 against 0.83; box 160 (N = 240), 600 in 0.63
// against 1.24.
//
// Layout.  Two image rows make one complex row: z[j][n] = (row 2j, row 2j+1)
// at n, rows N + 1 apart so that lanes over j hit distinct banks.  An N-point
// FFT along a row is two passes of radices R1 and R2 (N = R1 R2, R2 even) held
// in registers, in place: frequency k = k1 + R1 k2 ends at position k1 R2 + k2,
// rotated by k1 within its block of R2 so that lanes over consecutive k hit
// distinct banks.  The two rows' half spectra X0, X1 then replace the pair's
// spectrum, X0[k] at k's position and X1[k] at (N-k)'s, 0 < k < N/2; columns 0
// and N/2 are real along a row and share one complex column, column 0's value
// as the real part.  So an N x N image and its half spectrum both take N^2
// floats, and a column's even rows sit at k's position, its odd rows at
// (N-k)'s.  Along y the passes are the same, rows in place of positions.  The
// inverse runs the passes backwards.  The phase origin's move to the corner
// (a shift by N/2, N even) is the sign (-1)^(kx+ky) of the spectrum.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "fr_ctf.cuh"
#include "fr_device.cuh"
#include "fr_fft.cuh"
#include "fr_handle.h"

namespace fr {
namespace slc {

using namespace fft;

// ------------------------------------------------------------------ passes
struct Shape {
  int N, R1, R2;          // N = R1 * R2, R2 even
  int ld;                 // N + 1
  unsigned inv1;          // k / R1 = k * inv1 >> 16 for k < 256
  const float2 *tw;       // [N] (cos, sin) of 2 pi i / N
};

// Columns c = k1 R2/2 + k2 of the half spectrum, in shared memory: the
// positions of the even rows (frequency k = k1 + R1 k2) and of the odd rows
// (N - k; c = 0: N/2), k itself, and the column of each k.
struct Cols {
  unsigned short *even, *odd, *kx, *at;   // [N/2] each
};

__device__ __forceinline__ float2 twiddle(const Shape &s, int i, int dir) {
  const float2 w = __ldg(&s.tw[i]);
  return make_float2(w.x, dir * w.y);
}

// Position of frequency (k1, k2) in a row.
__device__ __forceinline__ int place_of(const Shape &s, int k1, int k2) {
  const int r = k2 + k1 % s.R2;
  return k1 * s.R2 + (r >= s.R2 ? r - s.R2 : r);
}
// Walks (slow, fast) pairs, fast in [0, nf), one per thread.
struct Walk {
  int fast, slow, df, ds, nf;
  __device__ __forceinline__ Walk(int nf_) : nf(nf_) {
    slow = threadIdx.x / nf;
    fast = threadIdx.x - slow * nf;
    ds = blockDim.x / nf;
    df = blockDim.x - ds * nf;
  }
  __device__ __forceinline__ void next() {
    fast += df;
    slow += ds;
    if (fast >= nf) {
      fast -= nf;
      slow++;
    }
  }
};

// Rows, radix R1, between n = n1 R2 + n' and (k1, n'); lanes over row pairs.
// The inverse leaves the image times `scale`.
template <int R, int DIR>
__device__ __noinline__ void row_outer(float2 *z, Shape s, float scale) {
  for (Walk w(s.N / 2); w.slow < s.R2; w.next()) {
    float2 *p = z + w.fast * s.ld + w.slow;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = p[r * s.R2];
    if (DIR > 0) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float2 e = twiddle(s, r * w.slow, DIR);
        v[r] = cmul(v[r], e.x, e.y);
      }
    }
    dft<R, DIR>(v);
    if (DIR < 0) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float2 e = twiddle(s, r * w.slow, DIR);
        v[r] = cmul(v[r], e.x, e.y);
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (DIR > 0) v[r] = make_float2(__fmul_rn(v[r].x, scale), __fmul_rn(v[r].y, scale));
      p[r * s.R2] = v[r];
    }
  }
}

// Rows, radix R2, between (k1, n') and (k1, k2) (rotated by k1).
template <int R, int DIR> __device__ __noinline__ void row_inner(float2 *z, Shape s) {
  for (Walk w(s.N / 2); w.slow < s.R1; w.next()) {
    float2 *p = z + w.fast * s.ld + w.slow * R;
    const int k1 = w.slow % R;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int q = DIR < 0 ? r : (r + k1 >= R ? r + k1 - R : r + k1);
      v[r] = p[q];
    }
    dft<R, DIR>(v);
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int q = DIR > 0 ? r : (r + k1 >= R ? r + k1 - R : r + k1);
      p[q] = v[r];
    }
  }
}

// Columns, radix R1, between rows y = n1 R2 + n' and (k1, n'); lanes over
// columns.  R2 is even, so a butterfly's rows share their parity.
template <int R, int DIR> __device__ __noinline__ void col_outer(float2 *z, Shape s, Cols t) {
  const int step = (s.R2 / 2) * s.ld;
  for (Walk w(s.N / 2); w.slow < s.R2; w.next()) {
    float2 *p = z + (w.slow >> 1) * s.ld + ((w.slow & 1) ? t.odd : t.even)[w.fast];
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = p[r * step];
    if (DIR > 0) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float2 e = twiddle(s, r * w.slow, DIR);
        v[r] = cmul(v[r], e.x, e.y);
      }
    }
    dft<R, DIR>(v);
    if (DIR < 0) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float2 e = twiddle(s, r * w.slow, DIR);
        v[r] = cmul(v[r], e.x, e.y);
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) p[r * step] = v[r];
  }
}

// Columns, radix R2, between (k1, n') and (k1, k2).  MODE 0: forward.  1:
// forward, times the CTF's sign, and straight back (the packed column 0 only
// forward: col0_flip has its signs).  2: back, column 0 alone.
template <int R, int MODE>
__device__ __noinline__ void col_inner(float2 *z, Shape s, Cols t, const CtfDev *ctf) {
  const int n2 = s.N / 2;
  const int nc = MODE == 2 ? 1 : n2;
  for (Walk w(nc); w.slow < s.R1; w.next()) {
    float2 *pe = z + w.slow * (R / 2) * s.ld + t.even[w.fast];
    float2 *po = z + w.slow * (R / 2) * s.ld + t.odd[w.fast];
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r += 2) {
      v[r] = pe[(r >> 1) * s.ld];
      v[r + 1] = po[(r >> 1) * s.ld];
    }
    if (MODE != 2) dft<R, -1>(v);
    if (MODE == 1 && w.fast != 0) {
      const int kx = t.kx[w.fast];
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int ky = w.slow + s.R1 * r;
        const float sg = ctf_sign(*ctf, kx, ky < n2 ? ky : ky - s.N);
        v[r].x *= sg;
        v[r].y *= sg;
      }
    }
    if (MODE == 2 || (MODE == 1 && w.fast != 0)) dft<R, 1>(v);
#pragma unroll
    for (int r = 0; r < R; r += 2) {
      pe[(r >> 1) * s.ld] = v[r];
      po[(r >> 1) * s.ld] = v[r + 1];
    }
  }
}

// The value of column 0 at row position q.
__device__ __forceinline__ float2 &packed(float2 *z, const Shape &s, int q, int nyq) {
  return z[(q >> 1) * s.ld + ((q & 1) ? nyq : 0)];
}
__device__ __forceinline__ int row_place(const Shape &s, int ky) {
  const int k2 = (int)((unsigned)ky * s.inv1 >> 16);
  return (ky - k2 * s.R1) * s.R2 + k2;
}

// The CTF's signs on the packed column: C = F0 + i Fn of the real columns 0
// and N/2, whose transforms are F(-ky) = conj F(ky).  With astigmatism the
// signs at ky and -ky may differ; the inverse real FFT keeps the real part of
// such a column, which is what their mean leaves.
__device__ void col0_flip(float2 *z, const Shape &s, const CtfDev &ctf) {
  const int n2 = s.N / 2, nyq = place_of(s, 0, s.R2 / 2);
  for (int ky = threadIdx.x; ky <= n2; ky += blockDim.x) {
    const int q = row_place(s, ky), m = row_place(s, ky == 0 ? 0 : s.N - ky);
    const float2 a = packed(z, s, q, nyq), b = packed(z, s, m, nyq);
    const int y = ky < n2 ? ky : -n2, ym = ky < n2 ? -ky : -n2;
    const float h0 = 0.25f * (ctf_sign(ctf, 0, y) + ctf_sign(ctf, 0, ym)),
                hn = 0.25f * (ctf_sign(ctf, n2, y) + ctf_sign(ctf, n2, ym));
    const float2 f = make_float2(h0 * (a.x + b.x), h0 * (a.y - b.y));   // F0
    const float2 g = make_float2(hn * (a.y + b.y), hn * (b.x - a.x));   // Fn
    packed(z, s, q, nyq) = make_float2(f.x - g.y, f.y + g.x);
    packed(z, s, m, nyq) = make_float2(f.x + g.y, g.x - f.y);
  }
}

// Pair spectrum <-> the two rows' half spectra.
template <int DIR> __device__ void split_rows(float2 *z, const Shape &s, const Cols &t) {
  const int n2 = s.N / 2;
  for (Walk w(n2); w.slow < n2; w.next()) {   // lanes over row pairs
    float2 &a = z[w.fast * s.ld + t.even[w.slow]], &b = z[w.fast * s.ld + t.odd[w.slow]];
    if (w.slow == 0) {
      const float2 u = a, v = b;
      a = make_float2(u.x, v.x);
      b = make_float2(u.y, v.y);
      continue;
    }
    const float2 u = a, v = b;
    if (DIR < 0) {   // Z[k], Z[N-k] -> X0[k], X1[k]
      a = make_float2(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
      b = make_float2(0.5f * (u.y + v.y), 0.5f * (v.x - u.x));
    } else {         // X0 + i X1, conj X0 + i conj X1
      a = make_float2(u.x - v.y, u.y + v.x);
      b = make_float2(u.x + v.y, v.x - u.y);
    }
  }
}

// R1's cases.  17 and 19 have a kernel of their own (BIG): with them among the
// others those took more registers (N = 240, 600 particles 656 against 637 us).
#define FR_RADIX(R, CALL)             \
  if constexpr (BIG) {                \
    if (R == 17) CALL(17);            \
    else CALL(19);                    \
  } else switch (R) {                 \
    case 2: CALL(2); break;           \
    case 3: CALL(3); break;           \
    case 4: CALL(4); break;           \
    case 5: CALL(5); break;           \
    case 6: CALL(6); break;           \
    case 7: CALL(7); break;           \
    case 8: CALL(8); break;           \
    case 9: CALL(9); break;           \
    case 10: CALL(10); break;         \
    case 11: CALL(11); break;         \
    case 12: CALL(12); break;         \
    case 13: CALL(13); break;         \
    case 14: CALL(14); break;         \
    case 15: CALL(15); break;         \
    default: CALL(16); break;         \
  }
#define FR_EVEN_RADIX(R, CALL)        \
  switch (R) {                        \
    case 2: CALL(2); break;           \
    case 4: CALL(4); break;           \
    case 6: CALL(6); break;           \
    case 8: CALL(8); break;           \
    case 10: CALL(10); break;         \
    case 12: CALL(12); break;         \
    case 14: CALL(14); break;         \
    default: CALL(16); break;         \
  }

// Image -> half spectrum, last column pass left to the caller.
template <bool BIG>
__device__ __forceinline__ void forward(float2 *z, const Shape &s, const Cols &t) {
#define CALL(R) row_outer<R, -1>(z, s, 1.0f)
  FR_RADIX(s.R1, CALL)
#undef CALL
  __syncthreads();
#define CALL(R) row_inner<R, -1>(z, s)
  FR_EVEN_RADIX(s.R2, CALL)
#undef CALL
  __syncthreads();
  split_rows<-1>(z, s, t);
  __syncthreads();
#define CALL(R) col_outer<R, -1>(z, s, t)
  FR_RADIX(s.R1, CALL)
#undef CALL
  __syncthreads();
}

// EMData::get_edge_mean, 2-D branch (libEM/emdata_metadata.cpp:713-735): pairs
// of opposite edge values added in float, the pairs in double.
// at(y, x): the image's value.
// The warps' sums wait in the padding at the rows' ends (there are at least as
// many row pairs as warps: slice_threads).
template <class F>
__device__ __forceinline__ float edge_mean(int n, float2 *z, const Shape &s, F at) {
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    acc += (double)__fadd_rn(at(0, i), at(n - 1, i));
    acc += (double)__fadd_rn(at(i, 0), at(i, n - 1));
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  auto slot = [&](int i) { return reinterpret_cast<double *>(z + i * s.ld + s.N); };
  if ((threadIdx.x & 31) == 0) *slot(threadIdx.x >> 5) = acc;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += *slot(i);
  __syncthreads();
  return __fdiv_rn((float)t, (float)(n * 4));
}

// Bilinear translation in place (TransformProcessor::transform, 2-D real
// branch, libEM/processor.cpp:11025-11080) of v - mean, times scale_out.
// Output rows read rows on one side only, so groups of rows are done in that
// order: a group's results wait in registers until all of it has been read.
// A thread keeps one column; the blockDim / N threads of a column take its
// row pairs in turn.
constexpr int kHold = 4;   // row pairs a thread holds at a time
__device__ __forceinline__ void translate(float2 *z, const Shape &s, float tx, float ty, float mean,
                                          float scale_out) {
  const int N = s.N, n2 = N / 2, h = n2;
  if (fabsf(tx) < 1e-6f && fabsf(ty) < 1e-6f) {   // Transform::is_identity: copied
    for (Walk w(N); w.slow < n2; w.next()) {
      float2 &v = z[w.slow * s.ld + w.fast];
      v = make_float2(__fmul_rn(__fsub_rn(v.x, mean), scale_out),
                      __fmul_rn(__fsub_rn(v.y, mean), scale_out));
    }
    __syncthreads();
    return;
  }
  const int lines = blockDim.x / N, line = threadIdx.x / N, x = threadIdx.x - line * N;
  const bool on = line < lines;
  const float x2 = __fadd_rn(__fadd_rn((float)(x - h), tx), (float)h);
  const bool okx = !(x2 < 0 || x2 >= N);   // a NaN shift is not outside: its slice is NaN
  const int ix = okx ? (int)x2 : 0, dx = ix == N - 1 ? 0 : 2;   // to the next column, in floats
  const float t = __fsub_rn(x2, (float)ix), omt = __fsub_rn(1.0f, t);
  const float *col = reinterpret_cast<const float *>(z) + 2 * ix;
  auto value = [&](int y) {
    const float y2 = __fadd_rn(__fadd_rn((float)(y - h), ty), (float)h);
    if (!okx || y2 < 0 || y2 >= N) return 0.0f;
    const int iy = (int)y2, jy = iy == N - 1 ? iy : iy + 1;
    const float u = __fsub_rn(y2, (float)iy), omu = __fsub_rn(1.0f, u);
    const float *p = col + 2 * (iy >> 1) * s.ld + (iy & 1), *q = col + 2 * (jy >> 1) * s.ld + (jy & 1);
    float a = __fmul_rn(__fmul_rn(omt, omu), __fsub_rn(p[0], mean));
    a = __fadd_rn(a, __fmul_rn(__fmul_rn(t, omu), __fsub_rn(p[dx], mean)));
    a = __fadd_rn(a, __fmul_rn(__fmul_rn(omt, u), __fsub_rn(q[0], mean)));
    a = __fadd_rn(a, __fmul_rn(__fmul_rn(t, u), __fsub_rn(q[dx], mean)));
    return __fmul_rn(a, scale_out);
  };
  const bool up = ty >= 0.0f;
  for (int g = 0; g < n2; g += lines * kHold) {
    float2 hold[kHold];
    const int first = g + line;
#pragma unroll
    for (int q = 0; q < kHold; q++) {
      const int i = first + q * lines, j = up ? i : n2 - 1 - i;
      if (on && i < n2) hold[q] = make_float2(value(2 * j), value(2 * j + 1));
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kHold; q++) {
      const int i = first + q * lines, j = up ? i : n2 - 1 - i;
      if (on && i < n2) z[j * s.ld + x] = hold[q];
    }
    __syncthreads();
  }
}

// The half spectrum in natural order to global memory, times (-1)^(kx+ky).  A
// thread keeps one kx; columns 0 and N/2 come out of their shared column.
__device__ __forceinline__ void store(float2 *z, const Shape &s, const Cols &t,
                                      float2 *__restrict__ out) {
  const int N = s.N, n2 = N / 2, w2 = n2 + 1;
  const int lines = blockDim.x / n2, line = threadIdx.x / n2, kx = threadIdx.x - line * n2;
  if (line < lines && kx > 0) {
    const int c = t.at[kx];
    const float2 *even = z + t.even[c], *odd = z + t.odd[c];
    float2 *o = out + kx;
#pragma unroll 4
    for (int ky = line; ky < N; ky += lines) {
      const int q = row_place(s, ky);
      float2 v = ((q & 1) ? odd : even)[(q >> 1) * s.ld];
      if ((kx + ky) & 1) v = make_float2(-v.x, -v.y);
      o[(size_t)ky * w2] = v;
    }
  }
  const int nyq = t.odd[0];
  for (int ky = threadIdx.x; ky < N; ky += blockDim.x) {
    const float2 a = packed(z, s, row_place(s, ky), nyq),
                 b = packed(z, s, row_place(s, ky == 0 ? 0 : N - ky), nyq);
    const float h0 = (ky & 1) ? -0.5f : 0.5f, hn = (ky + n2) & 1 ? -0.5f : 0.5f;
    out[(size_t)ky * w2] = make_float2(h0 * (a.x + b.x), h0 * (a.y - b.y));
    out[(size_t)ky * w2 + n2] = make_float2(hn * (a.y + b.y), hn * (b.x - a.x));
  }
}

struct Args {
  const float *raw;                 // contiguous images, or
  const float *const *src_tab;      // one pointer per particle
  int box;
  const CtfDev *ctf;                // null: no phase flip
  const float *txy;                 // null: no shift
  const float *rot, *sym;           // null rot: no composition
  float *t3d;
  const PartSym *psym;
  int nsym;
  int means;                        // subtract the edge means
  float scale_out;
  float2 *out;                      // [n][N][N/2+1]
};

}  // namespace slc

template <bool BIG> __global__ void __launch_bounds__(768, 1) k_slice(slc::Args a, slc::Shape s) {
  using namespace slc;
  extern __shared__ __align__(16) unsigned char dyn[];
  const int N = s.N, n2 = N / 2, box = a.box, p = blockIdx.x;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  Cols t;
  t.even = reinterpret_cast<unsigned short *>(z + n2 * s.ld);
  t.odd = t.even + n2;
  t.kx = t.odd + n2;
  t.at = t.kx + n2;
  for (int c = threadIdx.x; c < n2; c += blockDim.x) {
    const int half = s.R2 / 2, k1 = c / half, k2 = c - k1 * half, k = k1 + s.R1 * k2;
    t.even[c] = (unsigned short)place_of(s, k1, k2);
    t.odd[c] = (unsigned short)(c == 0    ? place_of(s, 0, half)
                                : k1 == 0 ? place_of(s, 0, s.R2 - k2)
                                          : place_of(s, s.R1 - k1, s.R2 - 1 - k2));
    t.kx[c] = (unsigned short)k;
    t.at[k] = (unsigned short)c;
  }
  if (a.rot) {   // the particle's symmetry copies (libEM/transform.cpp:1384-1395)
    const float *sy = a.sym;
    int ns = a.nsym;
    size_t s0 = (size_t)p * a.nsym;
    if (a.psym) {
      const PartSym ps = a.psym[p];
      sy = ps.sym;
      ns = ps.nsym;
      s0 = (size_t)ps.slice0;
    }
    for (int e = threadIdx.x; e < ns * 9; e += blockDim.x)
      a.t3d[s0 * 9 + e] = compose_element(a.rot + 9 * (size_t)p, sy + 9 * (e / 9), e % 9);
  }
  const float *src = a.src_tab ? a.src_tab[p] : a.raw + (size_t)p * box * box;
  float mean = 0.0f;
  if (a.means) mean = edge_mean(box, z, s, [&](int y, int x) { return __ldg(&src[(size_t)y * box + x]); });
  // Region origin (box - N) // 2 (Python floor division)
  const int o = (box - N) >= 0 ? (box - N) / 2 : -((N - box + 1) / 2);
  {
    // a thread keeps one column; its loads go out four row pairs at a time
    const int lines = blockDim.x / N, line = threadIdx.x / N, c = threadIdx.x - line * N;
    const bool in = c + o >= 0 && c + o < box;
    const float *col = src + c + o;
    for (int j0 = line; line < lines && j0 < n2; j0 += 4 * lines) {
      float2 v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int j = j0 + q * lines, y = 2 * j + o;
        const float *at = col + (long)y * box;
        v[q].x = in && j < n2 && (unsigned)y < (unsigned)box ? __ldg(at) : mean;
        v[q].y = in && j < n2 && (unsigned)(y + 1) < (unsigned)box ? __ldg(at + box) : mean;
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int j = j0 + q * lines;
        if (j < n2) z[j * s.ld + c] = make_float2(__fsub_rn(v[q].x, mean), __fsub_rn(v[q].y, mean));
      }
    }
  }
  __syncthreads();
  if (a.ctf && a.ctf[p].on != 0.0f) {
    const CtfDev ctf = a.ctf[p];
    const float scale_in = 1.0f / ((float)N * (float)N);   // do_ift's
    forward<BIG>(z, s, t);
#define CALL(R) col_inner<R, 1>(z, s, t, &ctf)
    FR_EVEN_RADIX(s.R2, CALL)
#undef CALL
    __syncthreads();
    col0_flip(z, s, ctf);
    __syncthreads();
#define CALL(R) col_inner<R, 2>(z, s, t, &ctf)
    FR_EVEN_RADIX(s.R2, CALL)
#undef CALL
    __syncthreads();
#define CALL(R) col_outer<R, 1>(z, s, t)
    FR_RADIX(s.R1, CALL)
#undef CALL
    __syncthreads();
    split_rows<1>(z, s, t);
    __syncthreads();
#define CALL(R) row_inner<R, 1>(z, s)
    FR_EVEN_RADIX(s.R2, CALL)
#undef CALL
    __syncthreads();
#define CALL(R) row_outer<R, 1>(z, s, scale_in)
    FR_RADIX(s.R1, CALL)
#undef CALL
    __syncthreads();
  }
  mean = 0.0f;
  if (a.means) {
    const float *zf = reinterpret_cast<const float *>(z);
    mean = edge_mean(N, z, s, [&](int y, int x) {
      return zf[2 * ((y >> 1) * s.ld + x) + (y & 1)];
    });
  }
  translate(z, s, a.txy ? a.txy[2 * (size_t)p] : 0.0f, a.txy ? a.txy[2 * (size_t)p + 1] : 0.0f,
            mean, a.scale_out);
  forward<BIG>(z, s, t);
#define CALL(R) col_inner<R, 0>(z, s, t, nullptr)
  FR_EVEN_RADIX(s.R2, CALL)
#undef CALL
  __syncthreads();
  store(z, s, t, a.out + (size_t)p * N * (n2 + 1));
}

// N = R1 * R2 with R2 even, both among the radices above and as close as they
// come; false where there is no such pair or the image does not fit.
static size_t slice_smem(int N) {
  return sizeof(float2) * (size_t)(N / 2) * (N + 1) + sizeof(short) * 2 * N;
}
static bool slice_radices(int N, int &R1, int &R2) {
  if (N < 16 || slice_smem(N) > 232448) return false;
  const int all[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 19};
  int best = 1 << 30;
  for (int a : all)
    for (int b : all) {
      if (a * b != N || b % 2 || b > 16) continue;
      const int worst = std::max(a, b);
      if (worst < best || (worst == best && b < R2)) {
        best = worst;
        R1 = a;
        R2 = b;
      }
    }
  return best < (1 << 30);
}
// A block takes its particle 26 us (N = 96, no CTF) to 87 us (N = 192, CTF),
// however few there are, where the line preparation takes 28 to 46 us for up to
// a dozen.  With a CTF, us a call, against it: N = 88, 1 particle 44, 44; N =
// 112, 1 55, 46; N = 96, 16 53, 45 and 24 53, 67; N = 144, 48 75, 68 and 64
// 102, 105; N = 192, 64 115, 132.  Against the library's transforms (sizes with
// a radix of 17 or 19): N = 152, 1 85, 50 and 48 90, 128.
bool slice_fits(int N, int n, bool ctf) {
  int a = 0, b = 0;
  if (!slice_radices(N, a, b)) return false;
  if (std::max(a, b) > 16) return n >= 24;
  return n >= 56 || (ctf && (N <= 88 || (N <= 112 && n >= 20)));
}
// Threads of a block: several blocks share an SM at the smaller sizes
// (2,000 particles: N = 96 0.33, 0.37, 0.48 ms with 256, 384, 768 threads;
// N = 144 0.77, 0.66, 0.81; N = 192 1.77, 1.46, 1.20).
static int slice_threads(int N) { return N <= 112 ? 256 : N <= 160 ? 384 : 768; }

// (cos, sin)(2 pi i / N) on the current device.
static int slice_twiddles(int N, const float2 **out) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, float2 *> known;
  int dev = 0;
  CU(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  float2 *&t = known[std::make_pair(dev, N)];
  if (!t) {
    std::vector<float2> h(N);
    for (int i = 0; i < N; i++) {
      const double w = 2.0 * M_PI * i / N;
      h[i] = make_float2((float)std::cos(w), (float)std::sin(w));
    }
    float2 *d = nullptr;
    if (device_malloc((void **)&d, sizeof(float2) * N) != cudaSuccess) {
      cudaGetLastError();
      return fail(FR_ENOMEM, "device allocation of %zu bytes failed", sizeof(float2) * N);
    }
    CU(cudaMemcpy(d, h.data(), sizeof(float2) * N, cudaMemcpyHostToDevice));
    CU(cudaStreamSynchronize(nullptr));   // a copy from pageable memory may still be on its way
    t = d;
  }
  *out = t;
  return FR_OK;
}

int launch_slice(const float *d_raw, const float *const *d_src, int n, int box, int N,
                 const void *d_ctf, const float *d_txy, bool means, const float *d_rot,
                 const float *d_sym, int nsym, float *d_t3d, const PartSym *d_psym,
                 float scale_out, float2 *d_out, cudaStream_t st) {
  if (n == 0) return FR_OK;
  slc::Shape s;
  s.N = N;
  s.ld = N + 1;
  if (!slice_radices(N, s.R1, s.R2))
    return fail(FR_EUNSUPPORTED, "size %d does not take the one-launch preparation", N);
  s.inv1 = (65536 + s.R1 - 1) / s.R1;
  TRY(slice_twiddles(N, &s.tw));
  slc::Args a;
  a.raw = d_raw;
  a.src_tab = d_src;
  a.box = box;
  a.ctf = reinterpret_cast<const CtfDev *>(d_ctf);
  a.txy = d_txy;
  a.rot = d_rot;
  a.sym = d_sym;
  a.t3d = d_t3d;
  a.psym = d_psym;
  a.nsym = nsym;
  a.means = means ? 1 : 0;
  a.scale_out = scale_out;
  a.out = d_out;
  const size_t smem = slice_smem(N);
  auto *kernel = s.R1 > 16 ? k_slice<true> : k_slice<false>;
  CU(set_max_smem((const void *)kernel, smem));
  note_launch();
  kernel<<<n, slice_threads(N), smem, st>>>(a, s);
  CU(cudaGetLastError());
  return FR_OK;
}

}  // namespace fr
