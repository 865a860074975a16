// fr_lines.cu -- the per-particle preparation as five launches over lines (rows
// or columns) of every particle: calls of few particles, and images larger
// than one SM's shared memory (fr_slice.cu gives a block a whole particle,
// which pays from some tens of particles on).
//
//   rows:    edge mean, zero-padded clip, FFT along x          (CTF particles)
//   columns: FFT along y, CTF sign, FFT back                   (CTF particles)
//   rows:    FFT back along x, the image                       (CTF particles)
//   rows:    edge mean, bilinear shift, FFT along x
//   columns: FFT along y, phase origin to corner, the slice
//
// A block takes up to sixteen lines (128 bytes of a row) into shared memory,
// transforms them there and writes them out, so a stage reads and writes its
// image once; the half spectra live in the slices' own buffer.  Two real rows
// make one complex line.
//
// What bounds it: for one particle, launches and each block's load, two or
// three dependent passes and store, some 8 us a stage however little there is
// to do; that is why the stages are five and not ten, why a block then has as
// few as two lines, and why a stage's blocks start while the one before it
// drains.  For many, instructions (56 % of cycles issue) at four blocks an SM.
// A call with a CTF, against the ten launches with the library's transforms
// (fr_prologue.cu), us: N = 192, 1 particle 46 (62), 16 61 (73); N = 256, 128
// particles 224 (249); N = 384, 1 47 (60), 64 287 (373), 512 1930 (2420); N =
// 480, 512 3416 (3611).  Three blocks an SM and eight lines a block: N = 384,
// 512 2199; loads one at a time: 3305.
//
// The line FFT: up to three passes of radices in registers, decimation in
// frequency, in place: pass i takes blocks of L = R M points, butterflies over
// points M apart, and leaves frequency k = k0 + R0 (k1 + R1 k2) at position
// k0 M0 + k1 M1 + k2 (a table).  Every 16 points are padded by one, so that
// lanes R points apart hit distinct banks.
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
namespace lines {

using namespace fft;

struct Plan {
  int N, P, ld;
  int R[3], M[3];
  unsigned minv[3];            // b / M = umulhi(b, minv), M > 1
  const float2 *tw;            // [N] (cos, sin) of 2 pi i / N
  const unsigned short *pos;   // [N] position of each frequency
};

__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }

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

// store(slow, fast, load(slow, fast)) over w's pairs, slow < count, U loads at
// a time: one by one each would wait for memory.
template <int U, class L, class S>
__device__ __forceinline__ void batched(Walk w, int count, L load, S store) {
  while (w.slow < count) {
    int f[U], s[U];
    float2 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      f[u] = w.fast;
      s[u] = w.slow;
      v[u] = load(min(s[u], count - 1), f[u]);
      w.next();
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (s[u] < count) store(s[u], f[u], v[u]);
  }
}

// Pass i of `count` lines.
template <int R, int DIR>
__device__ __noinline__ void line_pass(float2 *z, int count, const Plan &p, int i) {
  const int M = p.M[i], step = p.N / (R * M);
  for (Walk w(p.N / R); w.slow < count; w.next()) {
    const int block = M > 1 ? (int)__umulhi((unsigned)w.fast, p.minv[i]) : w.fast;
    const int j = w.fast - block * M;
    float2 *q = z + w.slow * p.ld;
    const int base = block * M * R + j;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = q[pad(base + r * M)];
    if (DIR > 0 && M > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float2 e = __ldg(&p.tw[r * j * step]);
        v[r] = cmul(v[r], e.x, e.y);
      }
    }
    dft<R, DIR>(v);
    if (DIR < 0 && M > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float2 e = __ldg(&p.tw[r * j * step]);
        v[r] = cmul(v[r], e.x, -e.y);
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) q[pad(base + r * M)] = v[r];
  }
}

// All passes of `count` lines; barriers before the first and after the last.
template <int DIR> __device__ __forceinline__ void transform(float2 *z, int count, const Plan &p) {
#pragma unroll 1
  for (int q = 0; q < p.P; q++) {
    const int i = DIR < 0 ? q : p.P - 1 - q;
    __syncthreads();
    switch (p.R[i]) {
      case 2: line_pass<2, DIR>(z, count, p, i); break;
      case 3: line_pass<3, DIR>(z, count, p, i); break;
      case 4: line_pass<4, DIR>(z, count, p, i); break;
      case 5: line_pass<5, DIR>(z, count, p, i); break;
      case 6: line_pass<6, DIR>(z, count, p, i); break;
      case 7: line_pass<7, DIR>(z, count, p, i); break;
      case 8: line_pass<8, DIR>(z, count, p, i); break;
      case 9: line_pass<9, DIR>(z, count, p, i); break;
      case 10: line_pass<10, DIR>(z, count, p, i); break;
      case 11: line_pass<11, DIR>(z, count, p, i); break;
      case 12: line_pass<12, DIR>(z, count, p, i); break;
      case 13: line_pass<13, DIR>(z, count, p, i); break;
      case 14: line_pass<14, DIR>(z, count, p, i); break;
      case 15: line_pass<15, DIR>(z, count, p, i); break;
      default: line_pass<16, DIR>(z, count, p, i); break;
    }
  }
  __syncthreads();
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
  float *img;                       // [n][N][N]: the images after the phase flip,
  double *edge;                     // and their blocks' edge sums, [n][gridDim.y]
  float2 *spec;                     // [n][N][N/2+1]: half spectra, then the slices
};

__device__ __forceinline__ bool has_ctf(const Args &a, int p) {
  return a.ctf && a.ctf[p].on != 0.0f;
}

__device__ __forceinline__ double block_sum(double v, double *s_red) {
  for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += s_red[i];
  return t;
}

// EMData::get_edge_mean, 2-D branch (libEM/emdata_metadata.cpp:713-735): pairs
// of opposite edge values added in float, the pairs in double; every block of
// a particle gets the same value.
template <class F> __device__ __forceinline__ float edge_mean(int n, double *s_red, F at) {
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    acc += (double)__fadd_rn(at(0, i), at(n - 1, i));
    acc += (double)__fadd_rn(at(i, 0), at(i, n - 1));
  }
  return __fdiv_rn((float)block_sum(acc, s_red), (float)(n * 4));
}

// The padded raw image less its edge mean.
struct Padded {
  const float *src;
  int box, o;
  float mean;
  __device__ __forceinline__ float operator()(int y, int x) const {
    y += o;
    x += o;
    if ((unsigned)y >= (unsigned)box || (unsigned)x >= (unsigned)box) return 0.0f;
    return __fsub_rn(__ldg(&src[(size_t)y * box + x]), mean);
  }
};
// The image after the phase flip.  A stage runs beside the one before it until
// its grid dependency is resolved, so what that one writes (these images, their
// edge sums, the half spectra) is never read through the non-coherent path.
struct Image {
  const float *img;
  int N;
  __device__ __forceinline__ float operator()(int y, int x) const {
    return img[(size_t)y * N + x];
  }
};

__device__ __forceinline__ Padded padded(const Args &a, int N, int p, double *s_red, bool means) {
  Padded s;
  s.src = a.src_tab ? a.src_tab[p] : a.raw + (size_t)p * a.box * a.box;
  s.box = a.box;
  // Region origin (box - N) // 2 (Python floor division)
  s.o = (a.box - N) >= 0 ? (a.box - N) / 2 : -((N - a.box + 1) / 2);
  s.mean = 0.0f;
  if (means)
    s.mean = edge_mean(a.box, s_red,
                       [&](int y, int x) { return __ldg(&s.src[(size_t)y * s.box + x]); });
  return s;
}

// Bilinear translation (TransformProcessor::transform, 2-D real branch,
// libEM/processor.cpp:11025-11080) of at - mean, times scale: the part that
// one column's outputs share, then one output.
struct Shift {
  float tx, ty, mean, scale;
  int N;
  bool copy;   // Transform::is_identity
};
struct Column {
  int ix, jx;
  float t, omt;
  bool in;
};
__device__ __forceinline__ Column column_of(const Shift &c, int x) {
  const int h = c.N / 2;
  const float x2 = __fadd_rn(__fadd_rn((float)(x - h), c.tx), (float)h);
  Column k;
  k.in = !(x2 < 0 || x2 >= c.N);   // a NaN shift is not outside: its slice is NaN
  k.ix = c.copy ? x : k.in ? (int)x2 : 0;
  k.jx = k.ix == c.N - 1 ? k.ix : k.ix + 1;
  k.t = __fsub_rn(x2, (float)k.ix);
  k.omt = __fsub_rn(1.0f, k.t);
  return k;
}
template <class F>
__device__ __forceinline__ float shifted(const F &at, const Shift &c, const Column &k, int y) {
  if (c.copy) return __fmul_rn(__fsub_rn(at(y, k.ix), c.mean), c.scale);
  const int h = c.N / 2;
  const float y2 = __fadd_rn(__fadd_rn((float)(y - h), c.ty), (float)h);
  // outside: 0, after loads that wait for no test
  const bool in = k.in && !(y2 < 0 || y2 >= c.N);
  const int iy = in ? (int)y2 : 0, jy = iy == c.N - 1 ? iy : iy + 1;
  const float u = __fsub_rn(y2, (float)iy), omu = __fsub_rn(1.0f, u);
  const float a = at(iy, k.ix), b = at(iy, k.jx), d = at(jy, k.ix), e = at(jy, k.jx);
  float v = __fmul_rn(__fmul_rn(k.omt, omu), __fsub_rn(a, c.mean));
  v = __fadd_rn(v, __fmul_rn(__fmul_rn(k.t, omu), __fsub_rn(b, c.mean)));
  v = __fadd_rn(v, __fmul_rn(__fmul_rn(k.omt, u), __fsub_rn(d, c.mean)));
  v = __fadd_rn(v, __fmul_rn(__fmul_rn(k.t, u), __fsub_rn(e, c.mean)));
  return in ? __fmul_rn(v, c.scale) : 0.0f;
}

extern __shared__ __align__(16) unsigned char dyn[];

// What a stage can do before the stage it reads has finished: lets the next
// one start, takes the position table (behind the lines in shared memory),
// has the twiddles fetched.  Then waits for the stage before.
__device__ __forceinline__ unsigned short *begin(float2 *z, int count, const Plan &p) {
  cudaTriggerProgrammaticLaunchCompletion();
  unsigned short *pos = reinterpret_cast<unsigned short *>(z + count * p.ld);
  for (int i = threadIdx.x; i < p.N; i += blockDim.x) pos[i] = __ldg(&p.pos[i]);
  for (int i = 16 * threadIdx.x; i < p.N; i += 16 * blockDim.x)
    asm volatile("{.reg .f32 x;\n ld.global.nc.f32 x, [%0];}" ::"l"(p.tw + i));
  cudaGridDependencySynchronize();
  return pos;
}

// The block's lines (row pairs j0 .. j0+count) transformed and their two rows'
// half spectra written.
__device__ __forceinline__ void rows_out(float2 *z, int count, int j0, const Plan &p,
                                         const unsigned short *pos, float2 *__restrict__ out) {
  const int N = p.N, w2 = N / 2 + 1;
  transform<-1>(z, count, p);
  for (Walk w(w2); w.slow < count; w.next()) {
    const float2 *q = z + w.slow * p.ld;
    const int k = w.fast;
    const float2 a = q[pad(pos[k])], b = q[pad(pos[k ? N - k : 0])];
    float2 *o = out + (size_t)(2 * (j0 + w.slow)) * w2 + k;
    o[0] = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
    o[w2] = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
  }
}

// First rows of the phase flip.
__global__ void __launch_bounds__(256, 4) k_rows_pad(Args a, Plan p, int per) {
  __shared__ double s_red[8];
  const int q = blockIdx.x, N = p.N, j0 = blockIdx.y * per, count = min(per, N / 2 - j0);
  if (!has_ctf(a, q)) return;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = begin(z, per, p);
  // rows outside the box are zero whatever its edge mean
  const int o = (a.box - N) >= 0 ? (a.box - N) / 2 : -((N - a.box + 1) / 2);
  const bool blank = 2 * (j0 + count) + o <= 0 || 2 * j0 + o >= a.box;
  const Padded at = padded(a, N, q, s_red, a.means && !blank);
  batched<4>(
      Walk(N), count,
      [&](int s, int x) { return make_float2(at(2 * (j0 + s), x), at(2 * (j0 + s) + 1, x)); },
      [&](int s, int x, float2 v) { z[s * p.ld + pad(x)] = v; });
  rows_out(z, count, j0, p, pos, a.spec + (size_t)q * N * (N / 2 + 1));
}

// Columns there and back with the CTF's sign between.
__global__ void __launch_bounds__(256, 4) k_cols_flip(Args a, Plan p, int per) {
  const int q = blockIdx.x, N = p.N, w2 = N / 2 + 1, c0 = blockIdx.y * per,
            count = min(per, w2 - c0);
  if (!has_ctf(a, q)) return;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = begin(z, per, p);
  float2 *spec = a.spec + (size_t)q * N * w2 + c0;
  batched<8>(
      Walk(count), N, [&](int y, int c) { return spec[(size_t)y * w2 + c]; },
      [&](int y, int c, float2 v) { z[c * p.ld + pad(y)] = v; });
  transform<-1>(z, count, p);
  const CtfDev k = a.ctf[q];
  for (Walk w(N); w.slow < count; w.next()) {
    float2 &v = z[w.slow * p.ld + pad(pos[w.fast])];
    const float sg = ctf_sign(k, c0 + w.slow, w.fast < N / 2 ? w.fast : w.fast - N);
    v = make_float2(v.x * sg, v.y * sg);
  }
  transform<1>(z, count, p);
  for (Walk w(count); w.slow < N; w.next())
    spec[(size_t)w.slow * w2 + w.fast] = z[w.fast * p.ld + pad(w.slow)];
}

// Rows back to the image, scaled as do_ift scales it.
__global__ void __launch_bounds__(256, 4) k_rows_back(Args a, Plan p, int per) {
  __shared__ double s_red[8];
  const int q = blockIdx.x, N = p.N, n2 = N / 2, w2 = n2 + 1, j0 = blockIdx.y * per,
            count = min(per, n2 - j0);
  if (!has_ctf(a, q)) return;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = begin(z, per, p);
  const float2 *spec = a.spec + (size_t)q * N * w2;
  __syncthreads();
  for (Walk w(w2); w.slow < count;) {
    float2 us[4], vs[4];
    int ks[4], rows[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
      ks[g] = w.fast;
      rows[g] = w.slow;
      const float2 *r = spec + (size_t)(2 * (j0 + min(w.slow, count - 1))) * w2 + w.fast;
      us[g] = r[0];
      vs[g] = r[w2];
      w.next();
    }
#pragma unroll
    for (int g = 0; g < 4; g++) {
      if (rows[g] >= count) break;
      const int k = ks[g];
      const float2 u = us[g], v = vs[g];
      float2 *o = z + rows[g] * p.ld;
      if (k == 0 || k == n2) {   // real along the row: an inverse real FFT reads no more
        o[pad(pos[k])] = make_float2(u.x, v.x);
      } else {
        o[pad(pos[k])] = make_float2(u.x - v.y, u.y + v.x);
        o[pad(pos[N - k])] = make_float2(u.x + v.y, v.x - u.y);
      }
    }
  }
  transform<1>(z, count, p);
  const float inv = 1.0f / ((float)N * (float)N);
  float *img = a.img + (size_t)q * N * N;
  double edge = 0.0;   // the block's share of the edge sum, for the next stage
  for (Walk w(N); w.slow < count; w.next()) {
    const float2 v = z[w.slow * p.ld + pad(w.fast)];
    const int y = 2 * (j0 + w.slow), x = w.fast;
    const float u0 = __fmul_rn(v.x, inv), u1 = __fmul_rn(v.y, inv);
    float *o = img + (size_t)y * N + x;
    o[0] = u0;
    o[N] = u1;
    if (x == 0 || x == N - 1) edge += (double)u0 + (double)u1;
    if (y == 0) edge += u0;
    if (y == N - 2) edge += u1;
  }
  edge = block_sum(edge, s_red);
  if (threadIdx.x == 0) a.edge[(size_t)q * gridDim.y + blockIdx.y] = edge;
}

// Rows of the shifted image (or, without a phase flip, of the padded raw one).
__global__ void __launch_bounds__(256, 4) k_rows_shift(Args a, Plan p, int per) {
  __shared__ double s_red[8];
  const int q = blockIdx.x, N = p.N, j0 = blockIdx.y * per, count = min(per, N / 2 - j0);
  if (a.rot && blockIdx.y == 0) {   // the particle's symmetry copies (libEM/transform.cpp:1384-1395)
    const float *sy = a.sym;
    int ns = a.nsym;
    size_t s0 = (size_t)q * a.nsym;
    if (a.psym) {
      const PartSym ps = a.psym[q];
      sy = ps.sym;
      ns = ps.nsym;
      s0 = (size_t)ps.slice0;
    }
    for (int e = threadIdx.x; e < ns * 9; e += blockDim.x)
      a.t3d[s0 * 9 + e] = compose_element(a.rot + 9 * (size_t)q, sy + 9 * (e / 9), e % 9);
  }
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = begin(z, per, p);
  const float tx = a.txy ? a.txy[2 * (size_t)q] : 0.0f, ty = a.txy ? a.txy[2 * (size_t)q + 1] : 0.0f;
  Shift c;
  c.tx = tx;
  c.ty = ty;
  c.scale = a.scale_out;
  c.N = N;
  c.copy = fabsf(tx) < 1e-6f && fabsf(ty) < 1e-6f;
  auto rows = [&](const auto &at, float mean) {
    c.mean = mean;
    // a thread keeps a column for all of the block's rows
    const int lines = max(1, (int)blockDim.x / N), line = lines > 1 ? threadIdx.x / N : 0;
    if (line >= lines) return;
    for (int x = threadIdx.x - line * N; x < N; x += blockDim.x) {
      const Column k = column_of(c, x);
      for (int s0 = line; s0 < count; s0 += 2 * lines) {
        float2 v[2];
#pragma unroll
        for (int g = 0; g < 2; g++) {
          const int y = 2 * (j0 + min(s0 + g * lines, count - 1));
          v[g] = make_float2(shifted(at, c, k, y), shifted(at, c, k, y + 1));
        }
#pragma unroll
        for (int g = 0; g < 2; g++)
          if (s0 + g * lines < count) z[(s0 + g * lines) * p.ld + pad(x)] = v[g];
      }
    }
  };
  if (has_ctf(a, q)) {
    const Image at{a.img + (size_t)q * N * N, N};
    double t = 0.0;   // the edge mean from the blocks' sums (same grid)
    if (a.means) {
      for (int i = threadIdx.x; i < (int)gridDim.y; i += blockDim.x)
        t += a.edge[(size_t)q * gridDim.y + i];
      t = block_sum(t, s_red);
    }
    rows(at, a.means ? __fdiv_rn((float)t, (float)(N * 4)) : 0.0f);
  } else {
    const Padded at = padded(a, N, q, s_red, a.means);
    // a frame of zeros has the edge mean 0
    const bool framed = at.o < 0 && a.box - at.o < N;
    rows(at, a.means && !framed ? edge_mean(N, s_red, at) : 0.0f);
  }
  rows_out(z, count, j0, p, pos, a.spec + (size_t)q * N * (N / 2 + 1));
}

// Last columns: the slice in natural order, the phase origin moved to the
// corner (a shift by N/2, N even) by the sign (-1)^(kx+ky).
__global__ void __launch_bounds__(256, 4) k_cols_out(Args a, Plan p, int per) {
  const int q = blockIdx.x, N = p.N, w2 = N / 2 + 1, c0 = blockIdx.y * per,
            count = min(per, w2 - c0);
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = begin(z, per, p);
  float2 *spec = a.spec + (size_t)q * N * w2 + c0;
  batched<8>(
      Walk(count), N, [&](int y, int c) { return spec[(size_t)y * w2 + c]; },
      [&](int y, int c, float2 v) { z[c * p.ld + pad(y)] = v; });
  transform<-1>(z, count, p);
  for (Walk w(count); w.slow < N; w.next()) {
    float2 v = z[w.fast * p.ld + pad(pos[w.slow])];
    if ((c0 + w.fast + w.slow) & 1) v = make_float2(-v.x, -v.y);
    spec[(size_t)w.slow * w2 + w.fast] = v;
  }
}

// Up to three radices of 2 to 16 whose product is N, as few as it takes and the
// largest as small as it goes; false where there are none.
static bool factor(int N, std::vector<int> &out) {
  if (N < 2 || N > 4096) return false;
  if (N <= 16) {
    out = {N};
    return true;
  }
  int best = 17;
  for (int a = 2; a <= 16; a++)
    if (N % a == 0 && N / a >= 2 && std::max(a, N / a) < best) {
      best = std::max(a, N / a);
      out = {a, N / a};
    }
  if (best <= 16) return true;
  for (int a = 2; a <= 16; a++)
    for (int b = 2; b <= 16; b++) {
      const int c = N / (a * b), worst = std::max(a, std::max(b, c));
      if (N % (a * b) == 0 && c >= 2 && worst < best) {
        best = worst;
        out = {a, b, c};
      }
    }
  return best <= 16;
}

// The plan's tables on the current device, made once per size.
static int get_plan(int N, Plan &out) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, Plan> known;
  int dev = 0;
  CU(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find(std::make_pair(dev, N));
  if (it != known.end()) {
    out = it->second;
    return FR_OK;
  }
  std::vector<int> R;
  if (!factor(N, R)) return fail(FR_EUNSUPPORTED, "size %d does not take the line preparation", N);
  Plan p;
  memset(&p, 0, sizeof p);
  p.N = N;
  p.P = (int)R.size();
  p.ld = (N + N / 16 + 1) | 1;
  int M = N;
  for (int i = 0; i < p.P; i++) {
    M /= R[i];
    p.R[i] = R[i];
    p.M[i] = M;
    p.minv[i] = M > 1 ? (unsigned)((0x100000000ull + M - 1) / M) : 0;
  }
  std::vector<float2> tw(N);
  std::vector<unsigned short> pos(N);
  for (int k = 0; k < N; k++) {
    tw[k] = make_float2((float)std::cos(2.0 * M_PI * k / N), (float)std::sin(2.0 * M_PI * k / N));
    int rest = k, at = 0;
    for (int i = 0; i < p.P; i++) {
      at += rest % R[i] * p.M[i];
      rest /= R[i];
    }
    pos[k] = (unsigned short)at;
  }
  unsigned char *d = nullptr;
  const size_t tb = sizeof(float2) * N;
  if (device_malloc((void **)&d, tb + sizeof(short) * N) != cudaSuccess) {
    cudaGetLastError();
    return fail(FR_ENOMEM, "device allocation of %zu bytes failed", tb + sizeof(short) * N);
  }
  CU(cudaMemcpy(d, tw.data(), tb, cudaMemcpyHostToDevice));
  CU(cudaMemcpy(d + tb, pos.data(), sizeof(short) * N, cudaMemcpyHostToDevice));
  CU(cudaStreamSynchronize(nullptr));   // a copy from pageable memory may still be on its way
  p.tw = reinterpret_cast<const float2 *>(d);
  p.pos = reinterpret_cast<const unsigned short *>(d + tb);
  known[std::make_pair(dev, N)] = p;
  out = p;
  return FR_OK;
}

}  // namespace lines

size_t lines_edge_bytes(int N, int n) { return sizeof(double) * (size_t)n * (N / 2); }

// Sizes of up to three radices; others take the library's transforms, and so do
// many large images with a CTF, whose columns no longer come by whole 128-byte
// lines: N = 1024, 16 511 against 516 us, 64 1882 against 1699; N = 2048, 4 600
// against 777, 16 2260 against 2015.
bool lines_fits(int N, int n, bool ctf) {
  std::vector<int> r;
  return !(ctf && N >= 1000 && (long)n * N > 16384) && lines::factor(N, r);
}

int launch_lines(const float *d_raw, const float *const *d_src, int n, int box, int N,
                 const void *d_ctf, const float *d_txy, bool means, const float *d_rot,
                 const float *d_sym, int nsym, float *d_t3d, const PartSym *d_psym,
                 float scale_out, float *d_img, double *d_edge, float2 *d_out, cudaStream_t st) {
  if (n == 0) return FR_OK;
  lines::Plan p;
  TRY(lines::get_plan(N, p));
  lines::Args a;
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
  a.img = d_img;
  a.edge = d_edge;
  a.spec = d_out;
  // lines per block: few when the call has few, so that it reaches every SM,
  // and no more than let four blocks share one
  const int n2 = N / 2, w2 = n2 + 1;
  const size_t line = sizeof(float2) * p.ld;
  int per = 16;
  while (per > 2 && ((long)n * n2 < 148L * 2 * per || line * per > 60000)) per /= 2;
  while (per > 1 && line * per + sizeof(short) * N > 220000) per /= 2;
  const size_t smem = line * per + sizeof(short) * N;
  const dim3 rows(n, (n2 + per - 1) / per), cols(n, (w2 + per - 1) / per);
  // the shift's threads keep a column, or as many as it takes
  const int turns = (N + 255) / 256, shift = N > 128 ? ((N + turns - 1) / turns + 31) / 32 * 32 : 256;
  bool first = true;
  auto go = [&](void (*k)(lines::Args, lines::Plan, int), dim3 grid, int threads) {
    cudaError_t e = set_max_smem((const void *)k, smem);
    if (e != cudaSuccess) return e;
    note_launch();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    // each stage after the first may start while the one before it drains
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &early;
    cfg.numAttrs = first ? 0 : 1;
    first = false;
    return cudaLaunchKernelEx(&cfg, k, a, p, per);
  };
  if (d_ctf) {
    CU(go(lines::k_rows_pad, rows, 256));
    CU(go(lines::k_cols_flip, cols, 256));
    CU(go(lines::k_rows_back, rows, 256));
  }
  CU(go(lines::k_rows_shift, rows, shift));
  CU(go(lines::k_cols_out, cols, 256));
  return FR_OK;
}

}  // namespace fr
