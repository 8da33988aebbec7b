// Double-precision functions of the FP64 path kernel's coefficients, from tables.
//
// FP64 issues at 1/64 of the FP32 rate on this GPU (a warp instruction holds
// its scheduler for 64 cycles), so what a function costs is its number of
// FP64 instructions.  These take fewer than the math library's by reading
// more from tables (built once per context, each entry correctly rounded but
// for rare ties): the argument that is left is so small that the higher
// terms of its series, relative to the result below 2^-28, can be formed in
// FP32 without touching the last bit by more than a fraction; widening and
// narrowing between the formats are integer operations.  The method is the
// usual table-driven one (P. T. P. Tang, "Table-driven implementation of the
// exponential / logarithm function in IEEE floating-point arithmetic", ACM
// TOMS 15(2), 1989, and 16(4), 1990).
//
//                       FP64 instructions   largest (rms) error, ulp   CUDA's
//   sin and cos of pi x   8                 1.30 (0.28)                1.41 (0.34)
//   sin and cos of x      8                 1.18 (0.28)                1.35 (0.35)
//   exp, |x| < 708        9                 0.50 (0.29)                0.81 (0.30)
// (on the arguments of tests/test_gpu_device_math.py)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dev_common.cuh"

namespace pdds {

// sin and cos at i/65536 of a right angle, i = 0 .. 65536, with what the
// doubles leave out and the FP32 factors of the angle's second-order terms.
struct __align__(16) TrigEntry {
  double s, c;
  float sl, cl;  // sin - s, cos - c
  float hs, hc;  // -s/2, -c/2
};
constexpr int F64_TRIG = 65536;   // entries per right angle
constexpr int F64_EXP = 4096;     // entries per octave

struct Fast64 {
  const TrigEntry* trig;  // [F64_TRIG + 1]
  const double* ex;       // [F64_EXP]: 2^(i / 4096)
  const float* exl;       // what ex leaves out
};

namespace f64 {

// ------------------------------------------------------------ formats
// FP32 of a double by truncation; 0 for magnitudes below 2^-120.
__device__ __forceinline__ float narrow(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned b = __funnelshift_l(lo, hi, 3) - 0xC0000000u;
  const unsigned ok = (hi & 0x7ff00000u) >= ((1023u - 120u) << 20) ? (b & 0x7fffffffu) | (hi & 0x80000000u) : 0u;
  return __uint_as_float(ok);
}
// Double of an FP32 value; 0 below 2^-126.
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f);
  const int hi = (int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u));
  return b & 0x7f800000u ? __hiloint2double(hi, (int)(b << 29)) : 0.0;
}

// ------------------------------------------------------------ sin, cos
// sin and cos of (angle of table entry idx) + d, |d| <= 1.2e-5, d32 = d:
// s + c d + (d^2 (-s/2 - c d / 6) + sl), the last term below 2^-33.
__device__ __forceinline__ void sincos_at(const Fast64& T, int idx, double d, float d32, double& sn, double& cs) {
  const double2 sc = __ldg(reinterpret_cast<const double2*>(T.trig + idx));
  const float4 h = __ldg(reinterpret_cast<const float4*>(T.trig + idx) + 1);
  const float d2 = d32 * d32, d6 = d32 * 0.33333334f;
  const float ws = fmaf(d2, fmaf(h.w, d6, h.z), h.x), wc = fmaf(d2, fmaf(-h.z, d6, h.w), h.y);
  sn = sc.x + fma(sc.y, d, widen(ws));
  cs = sc.y + fma(-sc.x, d, widen(wc));
}
// rotation by q right angles
__device__ __forceinline__ void quadrant(int q, double& sn, double& cs) {
  const double a = q & 1 ? cs : sn, b = q & 1 ? sn : cs;
  sn = __hiloint2double(__double2hiint(a) ^ ((q & 2) << 30), __double2loint(a));
  cs = __hiloint2double(__double2hiint(b) ^ (((q + 1) & 2) << 30), __double2loint(b));
}
constexpr double MAGIC = 6755399441055744.0;  // 1.5 2^52: rounds to an integer in the low word

// sin and cos of pi x
__device__ __forceinline__ void sincospi(const Fast64& T, double x, double& sn, double& cs) {
  if (((unsigned)__double2hiint(x) & 0x7ff00000u) >= ((1023u + 12u) << 20)) {  // |x| >= 4096, or not finite
    ::sincospi(x, &sn, &cs);
    return;
  }
  const double t = fma(x, 2.0 * F64_TRIG, MAGIC);
  const int k = __double2loint(t);
  const double r = fma(t - MAGIC, -0.5 / F64_TRIG, x);
  const float r32 = narrow(r);
  const double d = fma(r, 3.141592653589793, widen(r32 * 1.2246468e-16f));  // pi r, pi in two parts
  sincos_at(T, k & (F64_TRIG - 1), d, r32 * 3.1415927f, sn, cs);
  quadrant(k >> 16, sn, cs);
}
// sin and cos of x.  From |x| = 16 on, and where x is not finite, the math
// library's: the angle that is left is off by up to 2^-123 per table step, and
// the further out, the nearer to a zero of the sine or cosine a double can lie.
__device__ __forceinline__ void sincos(const Fast64& T, double x, double& sn, double& cs) {
  if (((unsigned)__double2hiint(x) & 0x7ff00000u) >= ((1023u + 4u) << 20)) {
    ::sincos(x, &sn, &cs);
    return;
  }
  const double t = fma(x, 41721.51340188181, MAGIC);  // 65536 / (pi / 2)
  const int k = __double2loint(t);
  const double kd = t - MAGIC;
  // (pi / 2) / 65536 in two parts
  const double d = fma(-kd, 9.343313592127634e-22, fma(-kd, 2.3968449810713143e-05, x));
  sincos_at(T, k & (F64_TRIG - 1), d, narrow(d), sn, cs);
  quadrant(k >> 16, sn, cs);
}

// ------------------------------------------------------------ exp
__device__ __forceinline__ double exp(const Fast64& T, double a) {
  if (((unsigned)__double2hiint(a) & 0x7fffffffu) >= 0x40862000u) return ::exp(a);  // |a| >= 708, or not finite
  const double t = fma(a, 5909.278887481194, MAGIC);  // 4096 / ln2
  const int k = __double2loint(t);
  const double kd = t - MAGIC;
  // ln2 / 4096 in two parts
  const double r = fma(-kd, 5.661735385366942e-21, fma(-kd, 0.0001692253858788929, a));
  // e^r - 1 = (r + r^2/2) + (r^3/6 + r^4/24), |r| <= 8.5e-5
  const float r32 = narrow(r), v = r32 * r32 * r32 * fmaf(r32, 0.041666668f, 0.16666667f);
  const double q = fma(r * 0.5, r, r) + widen(v);
  const int i = k & (F64_EXP - 1);
  const double b = __ldg(T.ex + i);
  const double e = b + fma(b, q, widen(__ldg(T.exl + i)));
  return __hiloint2double(__double2hiint(e) + ((k >> 12) << 20), __double2loint(e));
}

}  // namespace f64

// Bytes of the tables, and the kernel that fills them (k_fast64.cu).
size_t fast64_bytes();
Fast64 fast64_view(const void* block);
cudaError_t launch_fast64_tables(void* block, cudaStream_t s);

}  // namespace pdds
