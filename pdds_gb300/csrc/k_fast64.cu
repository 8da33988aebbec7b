// Fills the tables of fast64.cuh.  Entries are formed with unevaluated sums
// of two doubles (about 100 bits) from nested Taylor series and rounded once,
// so an entry is the correctly rounded value but for rare ties.
#include "fast64.cuh"

namespace pdds {

namespace {

// hi + lo, |lo| <= ulp(hi) / 2
struct dd {
  double h, l;
};
__device__ dd fast_two(double a, double b) {  // |a| >= |b|
  const double s = a + b;
  return {s, b - (s - a)};
}
__device__ dd two(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
__device__ dd add(dd a, dd b) {
  const dd s = two(a.h, b.h);
  return fast_two(s.h, s.l + (a.l + b.l));
}
__device__ dd mul(dd a, dd b) {
  const double p = a.h * b.h;
  return fast_two(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__device__ dd div(dd a, double d) {
  const double q = a.h / d;
  return fast_two(q, (fma(-q, d, a.h) + a.l) / d);
}
__device__ dd scale(dd a, double k) {  // k an integer of few bits
  const double p = a.h * k;
  return fast_two(p, fma(a.h, k, -p) + a.l * k);
}
__device__ dd one_minus(dd a) { return add({1.0, 0.0}, {-a.h, -a.l}); }

const int TERMS = 12;  // (pi/4)^25 / 25! and 0.7^24 / 24! are below 2^-90

__global__ void k_fast64_tables(TrigEntry* trig, double* ex, float* exl) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const dd PIO2 = {1.5707963267948966, 6.123233995736766e-17}, LN2 = {0.6931471805599453, 2.3190468138462996e-17};
  if (t <= F64_TRIG / 2) {
    // sin x = x (1 - x^2/(2 3) (1 - x^2/(4 5) (...))), cos x likewise, x <= pi / 4
    dd x = scale(PIO2, (double)t);
    x.h /= F64_TRIG;
    x.l /= F64_TRIG;
    const dd x2 = mul(x, x);
    dd s = {1.0, 0.0}, c = {1.0, 0.0};
    for (int k = TERMS; k >= 1; k--) {
      s = one_minus(div(mul(x2, s), (double)((2 * k) * (2 * k + 1))));
      c = one_minus(div(mul(x2, c), (double)((2 * k - 1) * (2 * k))));
    }
    s = mul(x, s);
    const float hs = (float)(-0.5 * s.h), hc = (float)(-0.5 * c.h);
    trig[t] = {s.h, c.h, (float)s.l, (float)c.l, hs, hc};
    trig[F64_TRIG - t] = {c.h, s.h, (float)c.l, (float)s.l, hc, hs};
    return;
  }
  const int u = t - (F64_TRIG / 2 + 1);
  if (u < F64_EXP) {
    // e^x = 1 + x (1 + x/2 (1 + x/3 (...)))
    dd x = scale(LN2, (double)u);
    x.h /= F64_EXP;
    x.l /= F64_EXP;
    dd e = {1.0, 0.0};
    for (int k = 2 * TERMS; k >= 1; k--) e = add({1.0, 0.0}, div(mul(x, e), (double)k));
    ex[u] = e.h;
    exl[u] = (float)e.l;
  }
}

size_t up256(size_t n) { return (n + 255) & ~size_t(255); }
const size_t TRIG_BYTES = up256((F64_TRIG + 1) * sizeof(TrigEntry));
const size_t EXP_BYTES = up256(F64_EXP * sizeof(double));
const size_t EXPL_BYTES = up256(F64_EXP * sizeof(float));

}  // namespace

size_t fast64_bytes() { return TRIG_BYTES + EXP_BYTES + EXPL_BYTES; }

Fast64 fast64_view(const void* block) {
  const unsigned char* b = static_cast<const unsigned char*>(block);
  Fast64 t;
  t.trig = reinterpret_cast<const TrigEntry*>(b);
  b += TRIG_BYTES;
  t.ex = reinterpret_cast<const double*>(b);
  b += EXP_BYTES;
  t.exl = reinterpret_cast<const float*>(b);
  return t;
}

cudaError_t launch_fast64_tables(void* block, cudaStream_t s) {
  const Fast64 t = fast64_view(block);
  const int n = F64_TRIG / 2 + 1 + F64_EXP;
  k_fast64_tables<<<(n + 63) / 64, 64, 0, s>>>(const_cast<TrigEntry*>(t.trig), const_cast<double*>(t.ex),
                                               const_cast<float*>(t.exl));
  return cudaGetLastError();
}

}  // namespace pdds
