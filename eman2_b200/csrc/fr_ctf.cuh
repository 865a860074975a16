// fr_ctf.cuh -- the CTF phase flip's sign and the composition of rotations,
// shared by the preparation kernels.
#pragma once
#include <cuda_runtime.h>

namespace fr {

// Per-particle CTF constants, formed on the host (ctf_constants,
// fr_prologue.cu) exactly as EMAN2Ctf::compute_2d_complex forms them.
struct CtfDev { float g1, g2, acac, ds, defocus, dfdiff, dfang, on; };

// Sign of cos(a) for a float a, as the correctly rounded float cosine has it
// (0 or above: +1).  With t = a / pi to float accuracy, the sign is the parity
// of the nearest integer unless t is close to half-way between two of them or
// large; then a double cosine decides.
static __device__ __noinline__ float cos_sign_exact(float a) {
  return cos((double)a) < 0.0 ? -1.0f : 1.0f;
}
__device__ __forceinline__ float cos_sign(float a) {
  const float t = a * 0.31830988618379067f;
  const float r = rintf(t);
  if (fabsf(t - r) < 0.4995f && fabsf(t) < 1000.0f) return ((int)r & 1) ? -1.0f : 1.0f;
  return cos_sign_exact(a);
}

// The defocus along the direction of (x, y), with astigmatism.
static __device__ __noinline__ float ctf_defocus(const CtfDev &k, int x, int y) {
  const float ang = atan2f((float)y, (float)x);
  const double a2 = (double)__fmul_rn(2.0f, ang) - 2.0 * 3.14159265358979323846 / 180.0f * (double)k.dfang;
  return (float)((double)k.defocus + (double)(k.dfdiff / 2.0f) * cos(a2));
}

// CTF_SIGN at frequency (x, y), y in [-N/2, N/2) (EMAN2Ctf::compute_2d_complex,
// libEM/ctf.cpp:1076-1090).  |(x, y)| is Util::hypot_fast's: the root of an
// integer below 2^24 rounded once to float (a double root rounded again to
// float is the same).
__device__ __forceinline__ float ctf_sign(const CtfDev &k, int x, int y) {
  const float s = __fmul_rn(__fsqrt_rn((float)(x * x + y * y)), k.ds);
  const float t1 = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(-k.g1, s), s), s), s);
  const float df = k.dfdiff != 0.0f ? ctf_defocus(k, x, y) : k.defocus;
  const float gam = __fadd_rn(t1, __fmul_rn(__fmul_rn(__fmul_rn(k.g2, df), s), s));
  return cos_sign(__fsub_rn(gam, k.acac));
}

// Element e of a * b (row-major 3 x 3), in float with the products and sums
// rounded in the reference's order (libEM/transform.cpp:1384-1395).
__device__ __forceinline__ float compose_element(const float *__restrict__ a,
                                                 const float *__restrict__ b, int e) {
  const int i = e / 3, j = e % 3;
  float v = __fmul_rn(a[3 * i + 0], b[j]);
  v = __fadd_rn(v, __fmul_rn(a[3 * i + 1], b[3 + j]));
  return __fadd_rn(v, __fmul_rn(a[3 * i + 2], b[6 + j]));
}

}  // namespace fr
