// fr_lines.cu -- the per-particle preparation as five launches over lines (rows
// or columns) of every particle, for calls of few particles (fr_slice.cu gives
// a block a whole particle, which pays from some tens of particles on).
//
//   rows:    edge mean, zero-padded clip, FFT along x          (CTF particles)
//   columns: FFT along y, CTF sign, FFT back                   (CTF particles)
//   rows:    FFT back along x, the image                       (CTF particles)
//   rows:    edge mean, bilinear shift, FFT along x
//   columns: FFT along y, phase origin to corner, the slice
//
// A block takes a few lines into shared memory, transforms them there and
// writes them out, so a stage reads and writes its image once; the half spectra
// live in the slices' own buffer.  Two real rows make one complex line.  What
// bounds it: launch latency, and each block's load, few dependent passes and
// store, some 8 us a stage however little there is to do.  That is why the
// stages are five and not ten, and why a block has as few as two lines: one
// particle with a CTF at N = 192 47 us (62 in ten launches with the library's
// transforms, two of which are its own rows and columns), N = 384 55 (59).
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
struct Image {
  const float *img;
  int N;
  __device__ __forceinline__ float operator()(int y, int x) const {
    return __ldg(&img[(size_t)y * N + x]);
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
// libEM/processor.cpp:11025-11080) of at - mean, times scale: one output.
template <class F>
__device__ __forceinline__ float shifted(const F &at, int N, int y, int x, float tx, float ty,
                                         bool copy, float mean, float scale) {
  if (copy) return __fmul_rn(__fsub_rn(at(y, x), mean), scale);   // Transform::is_identity
  const int h = N / 2;
  const float x2 = __fadd_rn(__fadd_rn((float)(x - h), tx), (float)h);
  const float y2 = __fadd_rn(__fadd_rn((float)(y - h), ty), (float)h);
  if (!(x2 >= 0 && x2 < N && y2 >= 0 && y2 < N)) return 0.0f;
  const int ix = (int)x2, iy = (int)y2;
  const int jx = ix == N - 1 ? ix : ix + 1, jy = iy == N - 1 ? iy : iy + 1;
  const float t = __fsub_rn(x2, (float)ix), u = __fsub_rn(y2, (float)iy);
  const float omt = __fsub_rn(1.0f, t), omu = __fsub_rn(1.0f, u);
  float v = __fmul_rn(__fmul_rn(omt, omu), __fsub_rn(at(iy, ix), mean));
  v = __fadd_rn(v, __fmul_rn(__fmul_rn(t, omu), __fsub_rn(at(iy, jx), mean)));
  v = __fadd_rn(v, __fmul_rn(__fmul_rn(omt, u), __fsub_rn(at(jy, ix), mean)));
  v = __fadd_rn(v, __fmul_rn(__fmul_rn(t, u), __fsub_rn(at(jy, jx), mean)));
  return __fmul_rn(v, scale);
}

extern __shared__ __align__(16) unsigned char dyn[];

// Shared memory: the lines, then the position table.
__device__ __forceinline__ unsigned short *load_pos(float2 *z, int count, const Plan &p) {
  unsigned short *pos = reinterpret_cast<unsigned short *>(z + count * p.ld);
  for (int i = threadIdx.x; i < p.N; i += blockDim.x) pos[i] = __ldg(&p.pos[i]);
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
__global__ void __launch_bounds__(256) k_rows_pad(Args a, Plan p, int per) {
  __shared__ double s_red[8];
  const int q = blockIdx.x, N = p.N, j0 = blockIdx.y * per, count = min(per, N / 2 - j0);
  if (!has_ctf(a, q)) return;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = load_pos(z, per, p);
  // rows outside the box are zero whatever its edge mean
  const int o = (a.box - N) >= 0 ? (a.box - N) / 2 : -((N - a.box + 1) / 2);
  const bool blank = 2 * (j0 + count) + o <= 0 || 2 * j0 + o >= a.box;
  const Padded at = padded(a, N, q, s_red, a.means && !blank);
  for (Walk w(N); w.slow < count; w.next()) {
    const int y = 2 * (j0 + w.slow);
    z[w.slow * p.ld + pad(w.fast)] = make_float2(at(y, w.fast), at(y + 1, w.fast));
  }
  rows_out(z, count, j0, p, pos, a.spec + (size_t)q * N * (N / 2 + 1));
}

// Columns there and back with the CTF's sign between.
__global__ void __launch_bounds__(256) k_cols_flip(Args a, Plan p, int per) {
  const int q = blockIdx.x, N = p.N, w2 = N / 2 + 1, c0 = blockIdx.y * per,
            count = min(per, w2 - c0);
  if (!has_ctf(a, q)) return;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = load_pos(z, per, p);
  float2 *spec = a.spec + (size_t)q * N * w2 + c0;
  for (Walk w(count); w.slow < N; w.next())
    z[w.fast * p.ld + pad(w.slow)] = spec[(size_t)w.slow * w2 + w.fast];
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
__global__ void __launch_bounds__(256) k_rows_back(Args a, Plan p, int per) {
  __shared__ double s_red[8];
  const int q = blockIdx.x, N = p.N, n2 = N / 2, w2 = n2 + 1, j0 = blockIdx.y * per,
            count = min(per, n2 - j0);
  if (!has_ctf(a, q)) return;
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = load_pos(z, per, p);
  const float2 *spec = a.spec + (size_t)q * N * w2;
  __syncthreads();
  for (Walk w(w2); w.slow < count; w.next()) {
    const int k = w.fast;
    const float2 *r = spec + (size_t)(2 * (j0 + w.slow)) * w2 + k;
    const float2 u = r[0], v = r[w2];
    float2 *o = z + w.slow * p.ld;
    if (k == 0 || k == n2) {   // real along the row: an inverse real FFT reads no more
      o[pad(pos[k])] = make_float2(u.x, v.x);
    } else {
      o[pad(pos[k])] = make_float2(u.x - v.y, u.y + v.x);
      o[pad(pos[N - k])] = make_float2(u.x + v.y, v.x - u.y);
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
__global__ void __launch_bounds__(256) k_rows_shift(Args a, Plan p, int per) {
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
  const unsigned short *pos = load_pos(z, per, p);
  const float tx = a.txy ? a.txy[2 * (size_t)q] : 0.0f, ty = a.txy ? a.txy[2 * (size_t)q + 1] : 0.0f;
  const bool copy = fabsf(tx) < 1e-6f && fabsf(ty) < 1e-6f;
  auto rows = [&](const auto &at, float mean) {
    for (Walk w(N); w.slow < count; w.next()) {
      const int y = 2 * (j0 + w.slow), x = w.fast;
      z[w.slow * p.ld + pad(x)] =
          make_float2(shifted(at, N, y, x, tx, ty, copy, mean, a.scale_out),
                      shifted(at, N, y + 1, x, tx, ty, copy, mean, a.scale_out));
    }
  };
  if (has_ctf(a, q)) {
    const Image at{a.img + (size_t)q * N * N, N};
    double t = 0.0;   // the edge mean from the blocks' sums (same grid)
    for (int i = 0; i < (int)gridDim.y; i++) t += __ldg(&a.edge[(size_t)q * gridDim.y + i]);
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
__global__ void __launch_bounds__(256) k_cols_out(Args a, Plan p, int per) {
  const int q = blockIdx.x, N = p.N, w2 = N / 2 + 1, c0 = blockIdx.y * per,
            count = min(per, w2 - c0);
  float2 *z = reinterpret_cast<float2 *>(dyn);
  const unsigned short *pos = load_pos(z, per, p);
  float2 *spec = a.spec + (size_t)q * N * w2 + c0;
  for (Walk w(count); w.slow < N; w.next())
    z[w.fast * p.ld + pad(w.slow)] = spec[(size_t)w.slow * w2 + w.fast];
  transform<-1>(z, count, p);
  for (Walk w(count); w.slow < N; w.next()) {
    float2 v = z[w.fast * p.ld + pad(pos[w.slow])];
    if ((c0 + w.fast + w.slow) & 1) v = make_float2(-v.x, -v.y);
    spec[(size_t)w.slow * w2 + w.fast] = v;
  }
}

// Up to three radices whose product is N, the largest as small as it goes.
static bool factor(int N, std::vector<int> &out) {
  static const int all[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16};
  int best = 1 << 30;
  for (int passes = 1; passes <= 3 && best == 1 << 30; passes++)
    for (int a : all)
      for (int b : all)
        for (int c : all) {
          if (passes < 3 && c != 2) break;
          if (passes < 2 && b != 2) break;
          const int p = a * (passes > 1 ? b : 1) * (passes > 2 ? c : 1);
          if (p != N) continue;
          std::vector<int> r{a};
          if (passes > 1) r.push_back(b);
          if (passes > 2) r.push_back(c);
          const int worst = *std::max_element(r.begin(), r.end());
          if (worst < best) {
            best = worst;
            out = r;
          }
        }
  return best < (1 << 30);
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
  if (cudaMalloc(&d, tb + sizeof(short) * N) != cudaSuccess) {
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

// Few particles only: five short launches against ten, a call of one particle
// with a CTF N = 192 47 against 62 us, N = 384 55 against 59; from about
// eight on, or four of the larger sizes, the library's transforms over many
// lines at once win (N = 192, 4: 51 against 63, 8: 70 against 63; N = 384, 2:
// 57 against 65, 4: 87 against 70).
bool lines_fits(int N, int n) {
  std::vector<int> r;
  return n <= (N <= 240 ? 6 : 2) && lines::factor(N, r);
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
  // lines per block: few when the call has few, so that it reaches every SM
  const int n2 = N / 2, w2 = n2 + 1;
  const size_t line = sizeof(float2) * p.ld;
  int per = 8;
  while (per > 2 && ((long)n * n2 < 148L * 2 * per || line * per > 60000)) per /= 2;
  while (per > 1 && line * per + sizeof(short) * N > 220000) per /= 2;
  const size_t smem = line * per + sizeof(short) * N;
  const dim3 rows(n, (n2 + per - 1) / per), cols(n, (w2 + per - 1) / per);
  const int threads = 256;
  auto go = [&](void (*k)(lines::Args, lines::Plan, int), dim3 grid) {
    cudaError_t e = set_max_smem((const void *)k, smem);
    if (e != cudaSuccess) return e;
    note_launch();
    k<<<grid, threads, smem, st>>>(a, p, per);
    return cudaGetLastError();
  };
  if (d_ctf) {
    CU(go(lines::k_rows_pad, rows));
    CU(go(lines::k_cols_flip, cols));
    CU(go(lines::k_rows_back, rows));
  }
  CU(go(lines::k_rows_shift, rows));
  CU(go(lines::k_cols_out, cols));
  return FR_OK;
}

}  // namespace fr
