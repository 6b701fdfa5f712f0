// Precision-generic device math and warp reductions (float -> CUDA single
// precision library functions, double -> double precision ones).
#pragma once
#include <cuda_runtime.h>
#include <limits>

namespace wamgpu {

__device__ __forceinline__ float dsqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double dsqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float dexp(float x) { return expf(x); }
__device__ __forceinline__ double dexp(double x) { return exp(x); }
__device__ __forceinline__ float dlog(float x) { return logf(x); }
__device__ __forceinline__ double dlog(double x) { return log(x); }
__device__ __forceinline__ float dlog10(float x) { return log10f(x); }
__device__ __forceinline__ double dlog10(double x) { return log10(x); }
__device__ __forceinline__ float dpow(float x, float y) { return powf(x, y); }
__device__ __forceinline__ double dpow(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float dsin(float x) { return sinf(x); }
__device__ __forceinline__ double dsin(double x) { return sin(x); }
__device__ __forceinline__ float dcos(float x) { return cosf(x); }
__device__ __forceinline__ double dcos(double x) { return cos(x); }
__device__ __forceinline__ float dtanh(float x) { return tanhf(x); }
__device__ __forceinline__ double dtanh(double x) { return tanh(x); }
__device__ __forceinline__ float dsinh(float x) { return sinhf(x); }
__device__ __forceinline__ double dsinh(double x) { return sinh(x); }
__device__ __forceinline__ float dcosh(float x) { return coshf(x); }
__device__ __forceinline__ double dcosh(double x) { return cosh(x); }
__device__ __forceinline__ float datan2(float y, float x) { return atan2f(y, x); }
__device__ __forceinline__ double datan2(double y, double x) { return atan2(y, x); }
__device__ __forceinline__ float dabs(float x) { return fabsf(x); }
__device__ __forceinline__ double dabs(double x) { return fabs(x); }
// Fortran MAX/MIN semantics for ordered operands
// a / b through the hardware reciprocal path for FP32 (at most 2 ulp,
// |b| in [2^-126, 2^126]); the precise division for FP64.  Used where the
// divisor is bounded, as max(1, ...) is.
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }

// Separately rounded products and sums (never contracted into an FMA), for
// the expressions whose last bit decides an integer on the reference's
// separate-operation arithmetic: the spectral integrals behind the cut-off
// index, the stress sums of the LFACTOR iteration, the drag law of u*.
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
// a * b + c rounded once.
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
// Two single-precision operations per instruction (fma.rn.f32x2 and the like):
// each half rounds as the scalar operation does, but the compiler fuses an add2
// of a mul2 into one rounding, .rn or not (seen on sm_100a, CUDA 12.9): sums of
// products that must round twice stay scalar.  A packed operation issues in one
// slot and takes the FP32 pipe two cycles (B200): it saves issue slots only.
struct F2 {
  unsigned long long v;
  __device__ F2() {}
  __device__ F2(float x, float y) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y)); }
  __device__ float x() const { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return a; }
  __device__ float y() const { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return b; }
};
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
// Quotients a / b for one divisor b, each rounded as the IEEE division
// rounds it, without a division per quotient.  In single precision the
// quotient is the float rounding of a times the double reciprocal of b.  That
// product is within 2^-52 (relative) of a/b, while a/b lies more than 2^-49
// (relative) from every midpoint between two floats: a midpoint m has an odd
// 25-bit significand, so a - m*b is a nonzero multiple of 2^-25 ulp(a).  Both
// therefore round to the same float.  Branch-free, unlike the division's
// special-operand paths.  In double precision it is the division itself.
template <typename R> struct RecipDiv;
template <> struct RecipDiv<float> {
  double y;
  __device__ explicit RecipDiv(float b) : y(1.0 / (double)b) {}
  __device__ float operator()(float a) const { return __double2float_rn(__dmul_rn((double)a, y)); }
  __device__ F2 operator()(F2 a) const { return F2((*this)(a.x()), (*this)(a.y())); }
};
template <> struct RecipDiv<double> {
  double b;
  __device__ explicit RecipDiv(double b_) : b(b_) {}
  __device__ double operator()(double a) const { return a / b; }
};
// The same quotients without leaving single precision: with y the correctly
// rounded reciprocal of b, two corrections by the exact residual a - q*b end in
// the correctly rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990), as
// long as the residual is exact, which holds for a = 0 and for |a| >= LO
// (b and the quotient in the normal range).  The caller checks that and takes
// RecipDiv otherwise.  Why: the conversions to and from double run at 1/8 of
// the FP32 rate; a RecipDiv quotient takes 4.2 cycles per warp and SM, this 1.4
// (B200).
struct MarksteinDiv {
  static constexpr float LO = 1e-28f;  // 2^-100 and room for a divisor of a hundred in between
  float b, y;
  __device__ explicit MarksteinDiv(float b_) : b(b_), y(1.0f / b_) {}
  __device__ float operator()(float a) const {
    float q = __fmul_rn(a, y);
    q = __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
    return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
  }
  __device__ F2 operator()(F2 a) const {
    const F2 y2(y, y), nb(-b, -b);
    F2 q = mul2(a, y2);
    q = fma2(fma2(q, nb, a), y2, q);
    return fma2(fma2(q, nb, a), y2, q);
  }
};
// Running test of the numerators: bits - 1 of |a| as an unsigned number is
// smallest for the smallest nonzero |a| (zero wraps to the largest).
__device__ __forceinline__ unsigned num_bits(float a) { return (__float_as_uint(a) & 0x7fffffffu) - 1u; }

// Correctly rounded single-precision transcendentals (evaluated in double,
// rounded once) for the same per-point values: the cut-off index's LOG10 /
// LOG, the LFACTOR exponentials and wind-direction cosines, and WAVNU2's
// dispersion relation.  The CPU oracle evaluates them the same way, so equal
// inputs give equal integer decisions.  In double precision they are the
// functions themselves.
__device__ __forceinline__ float crlog10(float x) { return (float)log10((double)x); }
__device__ __forceinline__ double crlog10(double x) { return log10(x); }
__device__ __forceinline__ float crlog(float x) { return (float)log((double)x); }
__device__ __forceinline__ double crlog(double x) { return log(x); }
__device__ __forceinline__ float crexp(float x) { return (float)exp((double)x); }
__device__ __forceinline__ double crexp(double x) { return exp(x); }
__device__ __forceinline__ float crcos(float x) { return (float)cos((double)x); }
__device__ __forceinline__ double crcos(double x) { return cos(x); }
__device__ __forceinline__ float crsin(float x) { return (float)sin((double)x); }
__device__ __forceinline__ double crsin(double x) { return sin(x); }
__device__ __forceinline__ float crtanh(float x) { return (float)tanh((double)x); }
__device__ __forceinline__ double crtanh(double x) { return tanh(x); }
__device__ __forceinline__ float crcosh(float x) { return (float)cosh((double)x); }
__device__ __forceinline__ double crcosh(double x) { return cosh(x); }
__device__ __forceinline__ float crsinh(float x) { return (float)sinh((double)x); }
__device__ __forceinline__ double crsinh(double x) { return sinh(x); }

template <typename R> __device__ __forceinline__ R dmax(R a, R b) { return a < b ? b : a; }
template <typename R> __device__ __forceinline__ R dmin(R a, R b) { return b < a ? b : a; }

template <typename R> __device__ __forceinline__ R warp_sum(R v) {
  for (int o = 16; o > 0; o >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Four consecutive reals from a 16-byte aligned address.
template <typename R> struct Quad { R a, b, c, d; };
__device__ __forceinline__ Quad<float> ld4(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Quad<double> ld4(const double* p) {
  const double2 u = *reinterpret_cast<const double2*>(p), v = *reinterpret_cast<const double2*>(p + 2);
  return {u.x, u.y, v.x, v.y};
}
template <typename R> __device__ __forceinline__ R warp_max(R v) {
  for (int o = 16; o > 0; o >>= 1) v = dmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace wamgpu
