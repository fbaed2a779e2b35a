// quotient.cuh -- the divisions of the FVT kernels: the quotient itself, quotients by a shared
// denominator, and the limiter's ratios (limiterBJ.f90:42-81).
//
// FP64 results are those of the plain expressions, bit for bit, so that the stage kernels
// keep the reference's roundings; a case that cannot be answered so says it.
#pragma once

namespace storm {
namespace {

constexpr double kZero = 0.0;
constexpr double kHalf = 0.5;
constexpr double kOne = 1.0;
constexpr double kOneThird = 1.0 / 3.0;
constexpr double kG = 9.81;
constexpr double kFmachp = 2.220446049250313e-16;   // EPSILON(zero)
constexpr double kVsmall = 2.2250738585072014e-308; // TINY(zero)
constexpr double kVlarge = 1.7976931348623157e+308; // HUGE(zero)
#define SMALL_F ((double)1.0e-9f)                   // REAL(mp) :: small = 1.0E-9

__device__ __forceinline__ double fmin2(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double fmax2(double a, double b) { return (b > a) ? b : a; }

// The IEEE quotient a / b, with a zero numerator answered without the division: for
// a nonzero b that is not a NaN, a signed zero divided by b is the zero whose sign is
// the exclusive or of the two signs, which is exactly what the division returns.  A
// zero quotient is rare in general code but common here (dry cells, still water, a
// limiter ratio whose numerator is the cell's own extremum, axis-aligned normals),
// and the division's own handling of that case costs far more than this test.
__device__ __forceinline__ double qdiv(double a, double b) {
  double r;
  if (a == 0.0 && b != 0.0 && b == b)
    r = __longlong_as_double((__double_as_longlong(a) ^ __double_as_longlong(b)) &
                             (long long)0x8000000000000000ULL);
  else
    r = a / b;
  return r;
}
// The mixed path's FP32 quotients: the approximate reciprocal-multiply division
// (__fdividef, within 2 ulp for |b| in [2^-126, 2^126]; the denominators here are
// determinants, celerities, wave-speed spans and limiter increments of ordinary
// magnitude), whose error is far below the FP32 rounding the path already accepts.
__device__ __forceinline__ float qdiv(float a, float b) { return __fdividef(a, b); }

// Quotients by one denominator, without the division's slow path inline.
//
// FP64, from P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990.  The reciprocal: Newton's iteration
// y <- y + y (1 - b y), two fused multiply-adds a step, which squares the error 1 - b y.  The
// seed instruction looks at 20 bits of b's fraction and gives 20 bits of the result's, an
// error below 2^-17; two steps square that to 2^-68, so that rounding is what is left and y
// is within one unit in the last place of 1/b.  From there the third gives the correctly
// rounded 1/b, except where b's significand is all ones (Markstein's theorem on the
// reciprocal).  The quotient: a y is within two units of a/b, a correction
// q <- q + (a - b q) y brings it within one, and the second, its residual then being exact,
// rounds it correctly (his theorem on the quotient): the bits of a / b.
// Neither theorem holds where a quotient or a residual overflows or becomes subnormal; for
// operands outside 2^-450 .. 2^451, and for a significand of all ones, `bad` is set and the
// caller takes the division itself.  A zero numerator's quotient is a y exactly.
template <class R>
struct Den;
template <>
struct Den<double> {
  double b, y;
  __device__ __forceinline__ static bool ordinary(double x) {
    return (unsigned)((__double2hiint(x) & 0x7fffffff) - 0x23d00000) < 0x38500000u;  // 2^-450 .. 2^451
  }
  __device__ __forceinline__ static double seed(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
  }
  __device__ __forceinline__ Den(double b_, bool* bad) : b(b_), y(seed(b_)) {
#pragma unroll
    for (int step = 0; step < 3; step++) y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    const bool ones = (__double2hiint(b) & 0xfffff) == 0xfffff && __double2loint(b) == -1;
    *bad = *bad || !ordinary(b) || ones;
  }
  __device__ __forceinline__ double quot(double a, bool* bad) const {
    const double q0 = a * y;
    double q = __fma_rn(__fma_rn(-b, q0, a), y, q0);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    const bool zero = a == kZero;
    *bad = *bad || !(zero || ordinary(a));
    return zero ? q0 : q;
  }
};
template <>
struct Den<float> {
  float b;
  __device__ __forceinline__ Den(float b_, bool*) : b(b_) {}
  __device__ __forceinline__ float quot(float a, bool*) const { return qdiv(a, b); }
};

// equals.f90:1-27
__device__ __forceinline__ bool equals(double a, double b) {
  double eps = fabs(a) * kFmachp;
  if (eps == kZero) eps = kVsmall;
  return !(fabs(a - b) > eps);
}

// The limiter's ratio at one face (beta = one).
__device__ __forceinline__ double limited_r(double q0, double qn, double g_x, double g_y, double rx, double ry) {
  const double qmin = fmin2(q0, qn);
  const double qmax = fmax2(q0, qn);
  const double qj = q0 + g_x * rx + g_y * ry;
  const double delq = qj - q0;
  double rj;
  if (equals(delq, kZero)) rj = kOne;
  else {
    // r = (qmin-q0)/delq for delq < 0, (qmax-q0)/delq otherwise; both are >= 0.
    // When |num| > |delq| the exact quotient exceeds one, so the rounded one is
    // >= 1 and the limiter's min(r,1) is 1: the division is skipped, same bits.
    const double num = (delq < 0) ? (qmin - q0) : (qmax - q0);
    rj = (fabs(num) > fabs(delq)) ? kOne : qdiv(num, delq);
  }
  const double a = fmin2(kOne * rj, kOne);
  const double b = fmin2(rj, kOne);
  return fmax2(a, b);
}
__device__ __forceinline__ float limited_r(double q0, double qn, float g_x, float g_y, float rx, float ry) {
  const float dmin = (float)(fmin2(q0, qn) - q0), dmax = (float)(fmax2(q0, qn) - q0);
  const float delq = g_x * rx + g_y * ry;
  if (fabsf(delq) <= 1e-30f) return 1.0f;
  const float num = (delq < 0) ? dmin : dmax;
  return (fabsf(num) >= fabsf(delq)) ? 1.0f : qdiv(num, delq);
}

// The limiter of one field over its three faces (min of limited_r), a face at a time.
// FP64: the ratios num/delq are compared by cross products, which order them beyond
// doubt when the products differ by more than their rounding (rounding is monotonic, so
// the smallest exact ratio has the smallest rounded one), and only the smallest is
// divided.  Products too close to tell, subnormal or not finite set `bad`.
template <class R>
struct Limit3;
template <>
struct Limit3<double> {
  double n = kOne, d = kOne;  // the smallest ratio so far
  bool any = false;
  __device__ __forceinline__ void face(double q0, double qn, double gx, double gy, double rx, double ry, bool* bad) {
    const double delq = (q0 + gx * rx + gy * ry) - q0;
    const double num = ((delq < 0 ? qn < q0 : qn > q0) ? qn : q0) - q0;
    const double an = fabs(num), ad = fabs(delq);
    // the ratio counts as one if equals(delq, zero), which holds up to 2^-1023 and for
    // infinities and NaN, or if it exceeds one
    constexpr double kTiny = 1.1125369292536007e-308;
    const bool cnt = ad > kTiny && ad <= kVlarge && !(an > ad);
    const double p = fabs(num * d), q = fabs(n * delq);
    constexpr double kBelow = 1.0 - 1.0e-15;
    const bool less = p < q * kBelow, more = q < p * kBelow;
    const bool cmp = any && cnt && n != kZero;
    *bad = *bad || (cmp && !((less && q > 1.0e-290) || (more && p > 1.0e-290))) || (cnt && !(an <= ad));
    const bool take = any ? cmp && less : cnt;
    n = take ? num : n;
    d = take ? delq : d;
    any = any || cnt;
  }
  __device__ __forceinline__ double value(bool* bad) const {
    const double r = Den<double>(d, bad).quot(n, bad);  // 1/1 if no ratio counts
    return any ? r : kOne;
  }
};
template <>
struct Limit3<float> {
  float r = 0.f;
  bool any = false;
  __device__ __forceinline__ void face(double q0, double qn, float gx, float gy, float rx, float ry, bool*) {
    const float x = limited_r(q0, qn, gx, gy, rx, ry);
    r = any ? fmin2(r, x) : x;
    any = true;
  }
  __device__ __forceinline__ float value(bool*) const { return r; }
};

}  // namespace
}  // namespace storm
