// Math policies for the generated CellML right-hand sides.
//
// fdm_math_exact:  exp/log as the model file writes them.  FP64 uses the CUDA double-precision
//                  functions; FP32 uses the SFU (ex2/lg2) intrinsics, the FP32-reaction mode's
//                  precision contract being "Vm within 0.1 mV of the FP64 oracle".
// fdm_math_approx: the reference's "approximateExponentialFunction" helpers
//                  (core/src/cellml/source_code_generator/03_generator_vc.cpp:385-407, :436-490):
//                  exp(x) ~ (1 + x/1024)^1024 and a piecewise Taylor log refined by one Newton step.
//                  In FP64 the squaring chain is evaluated literally, giving the reference's rounding.
//                  In FP32 ten squarings would amplify the rounding of 1 + x/1024 by 1024, so the
//                  same function is evaluated as exp(1024*log1p(x/1024)), with log1p from its power
//                  series (alternating terms (-1)^(k+1) s^k / k, s = x/1024) and the SFU exponential;
//                  arguments beyond the series' range fall back to the FP64 squaring chain.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

// single SFU instructions for the FP32 form of the right-hand sides (relative error ~2^-22):
// 2^x, 1/x and log2(x), flushing denormals (the FP32 reaction is compiled with -ftz=true)
__device__ __forceinline__ float fdm_ex2(float x)
{
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float fdm_rcp(float x)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float fdm_lg2(float x)
{
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// --------------------------------------------------------------------------------------------
// fdm_f2: two FP32 values (two nodes) evaluated by one packed sm_100 instruction (FADD2 / FMUL2 /
// FFMA2 through __fadd2_rn / __fmul2_rn / __ffma2_rn).  The generated paired right-hand side
// (rates_fast2) is the FP32 form written over this type, so one instruction stream advances two
// nodes.  A product is kept unevaluated (fdm_f2_prod) until it meets an addend, so a*b + c becomes
// one FFMA2 as a scalar a*b + c becomes one FFMA.  Transcendentals (ex2, rcp, lg2) have no packed
// form and run per component.
// --------------------------------------------------------------------------------------------
struct fdm_f2 {
  float2 v;
  __device__ __forceinline__ fdm_f2() {}
  __device__ __forceinline__ explicit fdm_f2(double c) : v(make_float2((float)c, (float)c)) {}
  __device__ __forceinline__ explicit fdm_f2(float c) : v(make_float2(c, c)) {}
  __device__ __forceinline__ fdm_f2(float a, float b) : v(make_float2(a, b)) {}
  __device__ __forceinline__ fdm_f2(float2 x) : v(x) {}
};
struct fdm_f2_prod {
  float2 a, b;
  __device__ __forceinline__ operator fdm_f2() const { return fdm_f2(__fmul2_rn(a, b)); }
};
struct fdm_b2 {
  bool x, y;
};

// a - b as one packed subtraction (PTX sub.f32x2; there is no packed-subtract intrinsic)
__device__ __forceinline__ float2 fdm_sub2(float2 a, float2 b)
{
  unsigned long long ra, rb, rd;
  memcpy(&ra, &a, 8);
  memcpy(&rb, &b, 8);
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
  float2 d;
  memcpy(&d, &rd, 8);
  return d;
}
// -a: one packed subtraction from zero (two scalar negations would cost two instructions)
__device__ __forceinline__ float2 fdm_neg2(float2 a) { return fdm_sub2(make_float2(0.f, 0.f), a); }
__device__ __forceinline__ fdm_f2 operator-(fdm_f2 a) { return fdm_f2(fdm_neg2(a.v)); }
__device__ __forceinline__ fdm_f2 operator+(fdm_f2 a) { return a; }
__device__ __forceinline__ fdm_f2_prod operator-(fdm_f2_prod p) { return fdm_f2_prod{fdm_neg2(p.a), p.b}; }
__device__ __forceinline__ fdm_f2_prod operator*(fdm_f2 a, fdm_f2 b) { return fdm_f2_prod{a.v, b.v}; }
__device__ __forceinline__ fdm_f2 operator+(fdm_f2 a, fdm_f2 b) { return fdm_f2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ fdm_f2 operator-(fdm_f2 a, fdm_f2 b) { return fdm_f2(fdm_sub2(a.v, b.v)); }
__device__ __forceinline__ fdm_f2 operator+(fdm_f2_prod p, fdm_f2 c) { return fdm_f2(__ffma2_rn(p.a, p.b, c.v)); }
__device__ __forceinline__ fdm_f2 operator+(fdm_f2 c, fdm_f2_prod p) { return fdm_f2(__ffma2_rn(p.a, p.b, c.v)); }
// a b - c and c - a b: a product and a packed subtraction (the negated operand of a fused form would
// cost a separate instruction as well); the generator writes constant subtrahends as negative addends
__device__ __forceinline__ fdm_f2 operator-(fdm_f2_prod p, fdm_f2 c) { return fdm_f2(fdm_sub2(__fmul2_rn(p.a, p.b), c.v)); }
__device__ __forceinline__ fdm_f2 operator-(fdm_f2 c, fdm_f2_prod p) { return fdm_f2(fdm_sub2(c.v, __fmul2_rn(p.a, p.b))); }
__device__ __forceinline__ fdm_f2 operator+(fdm_f2_prod p, fdm_f2_prod q) { return p + fdm_f2(q); }
__device__ __forceinline__ fdm_f2 operator-(fdm_f2_prod p, fdm_f2_prod q) { return p - fdm_f2(q); }
__device__ __forceinline__ fdm_f2& operator+=(fdm_f2& a, fdm_f2 b) { return a = a + b; }
__device__ __forceinline__ fdm_f2& operator+=(fdm_f2& a, fdm_f2_prod p) { return a = p + a; }
__device__ __forceinline__ fdm_f2 fdm_ex2(fdm_f2 x) { return fdm_f2(fdm_ex2(x.v.x), fdm_ex2(x.v.y)); }
__device__ __forceinline__ fdm_f2 fdm_rcp(fdm_f2 x) { return fdm_f2(fdm_rcp(x.v.x), fdm_rcp(x.v.y)); }
__device__ __forceinline__ fdm_f2 fdm_lg2(fdm_f2 x) { return fdm_f2(fdm_lg2(x.v.x), fdm_lg2(x.v.y)); }
__device__ __forceinline__ fdm_f2 operator/(fdm_f2 a, fdm_f2 b) { return a * fdm_rcp(b); }
__device__ __forceinline__ fdm_f2 fabs(fdm_f2 x) { return fdm_f2(fabsf(x.v.x), fabsf(x.v.y)); }
__device__ __forceinline__ fdm_f2 sqrt(fdm_f2 x) { return fdm_f2(sqrtf(x.v.x), sqrtf(x.v.y)); }
__device__ __forceinline__ fdm_f2 fdm_powf_pair(fdm_f2 x, fdm_f2 y)
{
  return fdm_f2(__powf(x.v.x, y.v.x), __powf(x.v.y, y.v.y));
}
#define FDM_F2_CMP(op)                                                                                   \
  __device__ __forceinline__ fdm_b2 operator op(fdm_f2 a, fdm_f2 b) { return fdm_b2{a.v.x op b.v.x, a.v.y op b.v.y}; }
FDM_F2_CMP(<)
FDM_F2_CMP(<=)
FDM_F2_CMP(>)
FDM_F2_CMP(>=)
FDM_F2_CMP(==)
FDM_F2_CMP(!=)
#undef FDM_F2_CMP
__device__ __forceinline__ fdm_b2 operator&&(fdm_b2 a, fdm_b2 b) { return fdm_b2{a.x && b.x, a.y && b.y}; }
__device__ __forceinline__ fdm_b2 operator||(fdm_b2 a, fdm_b2 b) { return fdm_b2{a.x || b.x, a.y || b.y}; }
__device__ __forceinline__ fdm_b2 operator!(fdm_b2 a) { return fdm_b2{!a.x, !a.y}; }
// per-component select (the paired form of c ? a : b; both operands are evaluated)
__device__ __forceinline__ fdm_f2 fdm_sel(fdm_b2 c, fdm_f2 a, fdm_f2 b)
{
  return fdm_f2(c.x ? a.v.x : b.v.x, c.y ? a.v.y : b.v.y);
}

// --------------------------------------------------------------------------------------------
// Batched reciprocals (simultaneous inversion): with q = d0 d1 [d2] one SFU reciprocal gives
// 1/d_k = (1/q) * (product of the other factors), three multiplications per saved reciprocal.
// Valid while q stays inside the FP32 range: for the Hodgkin-Huxley denominators
// exp(-(Vm+k)/10) c -/+ 1 that holds for Vm > -340 mV.  Outside it q is inf or 0 and the
// reciprocals become NaN, which the solver's non-finite check reports (FDM_ERR_NAN); the
// FP32-reaction mode is specified for physiological potentials.  No range test is made: a
// branch inside the right-hand side costs more than the reciprocals it saves.
// --------------------------------------------------------------------------------------------
// 1 - 2^t without cancellation and never exactly 0, for the FP32 form of 1 - exp(u) (t = u log2 e): for
// |t| < 2^-6 the series -x (1 + x/2 + x^2/6), x = t ln 2 (relative error below 2^-26 there), else 1 - ex2(t);
// t = 0 gives the smallest normal float instead of 0, so a removable singularity x / (1 - e^-ax) at x = 0
// evaluates to 0 rather than 0/0
__device__ __forceinline__ float fdm_1mexp2(float t)
{
  const float x = t * 0.69314718055994531f;
  const float series = -x * (1.f + x * (0.5f + x * (1.f / 6.f)));
  float d = fabsf(t) < 0.015625f ? series : 1.f - fdm_ex2(t);
  return d == 0.f ? 1.17549435e-38f : d;
}
__device__ __forceinline__ fdm_f2 fdm_1mexp2(fdm_f2 t) { return fdm_f2(fdm_1mexp2(t.v.x), fdm_1mexp2(t.v.y)); }
__device__ __forceinline__ double fdm_1mexp2(double t)
{
  const double d = -expm1(t * 0.69314718055994531);
  return d == 0.0 ? 2.2250738585072014e-308 : d;
}

template<class R>
__device__ __forceinline__ void fdm_rcp_batch(R d0, R d1, R& r0, R& r1)
{
  const R iv = fdm_rcp(R(d0 * d1));
  r0 = iv * d1;
  r1 = iv * d0;
}

template<class R>
__device__ __forceinline__ void fdm_rcp_batch(R d0, R d1, R d2, R& r0, R& r1, R& r2)
{
  const R q1 = d0 * d1;
  const R iv = fdm_rcp(R(q1 * d2));
  r2 = iv * q1;
  const R t = iv * d2; // 1/(d0 d1)
  r0 = t * d1;
  r1 = t * d0;
}

// --------------------------------------------------------------------------------------------
// FP64 exponential and division of the FP64 right-hand sides (rates_f64 and the fast adjoint forms).  A right-hand side
// strings a few of them together, and one thread's chain of them is what bounds small problems: CUDA's exp takes 150
// cycles here, its division 120, and their branches for special arguments keep the compiler from interleaving independent
// ones.  These have no branches, only selects: with CUDA's exp for its three single exponentials a Hodgkin-Huxley
// right-hand side takes 304 ns instead of 189 with one warp per SM, 440 instead of 358 with 8, 1171 instead of 1131 with 24.
// --------------------------------------------------------------------------------------------
// The argument c x of an exponential with a constant c, reduced without being formed: c x = k ln 2 + c R with R = x - k
// (ln 2/c), so that its rounding error is that of c R (at most 0.35), not that of c x.  hi: ln 2/c rounded to 42 bits (k hi
// is exact); lo: what hi leaves of ln 2, (ln 2/c - hi) c; l2e = c / ln 2.  c_lo: what c as a double leaves of c.
struct fdm_exp_scale {
  double c, c_lo, l2e, hi, lo;
};
// exp(c x) = 2^k exp(r), |r| <= ln 2 / 2, with ln 2/c in two parts (Cody and Waite), k from the rounding of the sum
// with 1.5 2^52; exp(r) = 1 + r + r^2 Q(r) with the degree-9 interpolation of Q at the Chebyshev nodes (relative error
// 3.4e-17), evaluated by Estrin's scheme.
struct fdm_exp_reduced {
  double t, r;   // k as a double, r
  int k;
  __device__ __forceinline__ fdm_exp_reduced(double x, double l2e)
  {
    const double magic = 6755399441055744.0;
    t = fma(x, l2e, magic);
    k = __double2loint(t);
    t -= magic;
  }
  // r^2 Q(r) + small
  __device__ __forceinline__ double poly(double small) const
  {
    const double r2 = r * r, r4 = r2 * r2;
    const double a0 = fma(0x1.5555555555555p-3, r, 0.5), a1 = fma(0x1.11111111109adp-7, r, 0x1.5555555553d4fp-5);
    const double a2 = fma(0x1.a01a01a7c8d47p-13, r, 0x1.6c16c17893833p-10);
    const double a3 = fma(0x1.71de0d9c145d0p-19, r, 0x1.a019b8ef67c6cp-16);
    const double a4 = fma(0x1.af38d53857513p-26, r, 0x1.2891a8c1d838dp-22);
    const double q = fma(fma(a4, r4, fma(a3, r2, a2)), r4, fma(a1, r2, a0));
    return fma(r2, q, small);
  }
};
// The ends of the range: 0 below -708 (the result would be subnormal), infinite (SAT: 2^1020, for divisors) from where
// the result would be within 3e-6 of the largest number; NaN for NaN.
constexpr double FDM_EXP_MAX = 709.78271, FDM_EXP_MIN = -708.0;
template<bool SAT>
__device__ __forceinline__ double fdm_exp_ends(double e, bool over, bool under)
{
  const int hi = over ? (SAT ? (1023 + 1020) << 20 : 0x7ff00000) : (under ? 0 : __double2hiint(e));
  return __hiloint2double(hi, over || under ? 0 : __double2loint(e));
}
__device__ __forceinline__ double fdm_exp_times_2k(double e, int k)
{
  return __hiloint2double(__double2hiint(e) + (k << 20), __double2loint(e));
}
// exp(x): 1 + r is rounded once and what that loses is added to the small terms.  At most 0.87 ulp and 0.253 on average
// of 4 million arguments (CUDA's exp: 0.88 and 0.258).
template<bool SAT = false>
__device__ __forceinline__ double fdm_exp64(double x)
{
  constexpr double ln2_lo = 0x1.ef35793c76730p-45;
  fdm_exp_reduced z(x, 0x1.71547652b82fep+0);
  const double rh = fma(z.t, -0x1.62e42fefa3800p-1, x);
  z.r = fma(z.t, -ln2_lo, rh);
  const double s = 1.0 + rh;
  const double e = s + z.poly(fma(z.t, -ln2_lo, rh - (s - 1.0)));
  return fdm_exp_ends<SAT>(fdm_exp_times_2k(e, z.k), x > FDM_EXP_MAX, x < FDM_EXP_MIN);
}
// exp(c x) with a constant c.  Of exp(r) at most 1.2 ulp and 0.27 on average; with the argument's rounding the
// exponential of a product rounded first has 1 to 9 halves of an ulp where |c x| is 1 to 6, this at most 2.4.
template<bool SAT = false>
__device__ __forceinline__ double fdm_exp64(double x, const fdm_exp_scale& f)
{
  fdm_exp_reduced z(x, f.l2e);
  z.r = fma(z.t, -f.lo, f.c * fma(z.t, -f.hi, x));
  const double e = 1.0 + z.poly(z.r);
  const double top = FDM_EXP_MAX / f.c, bottom = FDM_EXP_MIN / f.c;   // constants
  return fdm_exp_ends<SAT>(fdm_exp_times_2k(e, z.k), f.c > 0.0 ? x > top : x < top, f.c > 0.0 ? x < bottom : x > bottom);
}
// exp(c x) - 1 without the cancellation: 2^k (exp(r) - 1) + (2^k - 1), halved on the way so that k = 1024 has a 2^k.
// exp minus 1 loses 1/|exp(x) - 1| of exp's accuracy: 1.0 ulp on average for |x| <= 5 and 135 at 1e-2, this 0.27 and
// 0.25 (at most 2).
template<bool SAT = false>
__device__ __forceinline__ double fdm_expm1_64(double x, const fdm_exp_scale& f)
{
  fdm_exp_reduced z(x, f.l2e);
  z.r = fma(z.t, -f.lo, f.c * fma(z.t, -f.hi, x));
  const double s = __hiloint2double((1022 + z.k) << 20, 0);
  const double h = fma(s, z.poly(z.r), s - 0.5);
  const double y = h + h;
  const double top = FDM_EXP_MAX / f.c, bottom = FDM_EXP_MIN / f.c;
  const bool over = f.c > 0.0 ? x > top : x < top, under = f.c > 0.0 ? x < bottom : x > bottom;
  return over ? __hiloint2double(SAT ? (1023 + 1020) << 20 : 0x7ff00000, 0) : (under ? -1.0 : y);
}
template<bool SAT = false>
__device__ __forceinline__ double fdm_expm1_64(double x)
{
  return fdm_expm1_64<SAT>(x, fdm_exp_scale{1.0, 0.0, 0x1.71547652b82fep+0, 0x1.62e42fefa3800p-1, 0x1.ef35793c76730p-45});
}
// exp(c x + b) and exp(c x + b) - 1 for several small b (|b| <= 2) from one reduction: exp(c x) = 2^k (s + p) with s =
// 1 + c R rounded and p the rest, whose error is some 2^-56 of the sum, times e^b in two parts.  For divisors: the
// argument is held in [-700, 700].  With exp(c x + b) - 1 near 0 the error is 0.3 of the 2^-53 that an exponential
// rounded first leaves there, as long as x is exact (a sum V + d near -V is).  5 to 6 FP64 instructions each instead of
// about 20.
struct fdm_exp_offset {
  double e, e_lo;   // e^b and what it leaves of e^b
};
struct fdm_exp_group {
  double s, p, two_k;
  int k;
  __device__ __forceinline__ fdm_exp_group(double x, const fdm_exp_scale& f)
  {
    const double end = fabs(700.0 / f.c);   // a constant
    x = x > end ? end : x;
    x = x < -end ? -end : x;
    fdm_exp_reduced z(x, f.l2e);
    const double R = fma(z.t, -f.hi, x);
    z.r = fma(z.t, -f.lo, f.c * R);
    s = fma(f.c, R, 1.0);
    p = z.poly(fma(z.t, -f.lo, fma(f.c, R, 1.0 - s)));
    k = z.k;
    two_k = __hiloint2double((1023 + k) << 20, 0);
  }
  __device__ __forceinline__ double expm1() const { return fma(two_k, p, fma(two_k, s, -1.0)); }
  __device__ __forceinline__ double exp() const { return fdm_exp_times_2k(s + p, k); }
  __device__ __forceinline__ double expm1(const fdm_exp_offset& o) const
  {
    const double h = __dmul_rn(s, o.e);
    return fma(two_k, rest(h, o), fma(two_k, h, -1.0));
  }
  __device__ __forceinline__ double exp(const fdm_exp_offset& o) const
  {
    const double h = __dmul_rn(s, o.e);
    return fdm_exp_times_2k(__dadd_rn(h, rest(h, o)), k);
  }
  // (s + p) e^b - h
  __device__ __forceinline__ double rest(double h, const fdm_exp_offset& o) const
  {
    return fma(p, o.e, fma(s, o.e_lo, fma(s, o.e, -h)));
  }
};
// 1/d by one Halley step (cubic) from the hardware's approximation: 0.507 ulp; a/b with one residual correction of a
// (1/b), correctly rounded in 4 million quotients.  For b normal and finite (beyond 2^1022 in magnitude the quotient is
// 0), a and the quotient finite; b = 0, subnormal or infinite, and a quotient that overflows, give NaN.
__device__ __forceinline__ double fdm_rcp_approx(double d)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  return y;
}
__device__ __forceinline__ double fdm_halley(double d, double y)
{
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double fdm_rcp64(double d) { return fdm_halley(d, fdm_rcp_approx(d)); }
__device__ __forceinline__ double fdm_div64(double a, double b)
{
  const double y = fdm_rcp64(b);
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ bool fdm_is_nan(double x) { return (__double2hiint(x) & 0x7fffffff) > 0x7ff00000; }
// a/b as IEEE arithmetic has it for every a and b.  A divisor that is subnormal or at least 2^1021 is scaled together
// with the dividend; the hardware's approximation of 1/b is infinite for b = 0 and 0 for infinite b and stays as it is
// then; what the correction turns into NaN (such b, infinite a, a quotient that overflows) is a (1/b) itself.  Shorten
// (36 x 1481 nodes, 4 steps) with 26 of them took 5.76 ms, with CUDA's division in their place 6.55.
__device__ __forceinline__ double fdm_div64_any(double a, double b)
{
  const int exponent = __double2hiint(b) & 0x7ff00000;
  const int scale = exponent == 0 ? (1023 + 54) << 20 : (exponent >= 2044 << 20 ? (1023 - 54) << 20 : 1023 << 20);
  a *= __hiloint2double(scale, 0);
  b *= __hiloint2double(scale, 0);
  const double y0 = fdm_rcp_approx(b);
  const unsigned ye = (unsigned)__double2hiint(y0) & 0x7ff00000u;
  const double y = ye - (1u << 20) < (2046u << 20) ? fdm_halley(b, y0) : y0;
  const double q = a * y;
  const double c = fma(fma(-b, q, a), y, q);
  return fdm_is_nan(c) ? q : c;
}
// 1/d for every d: where the step would give NaN or the result is not normal, the hardware's approximation, infinite
// for d = 0 and subnormal d, 0 for infinite d and from 2^1022 on.
__device__ __forceinline__ double fdm_rcp64_any(double d)
{
  const double y = fdm_rcp_approx(d);
  const unsigned exponent = (unsigned)__double2hiint(d) & 0x7ff00000u;
  return exponent - (1u << 20) < (2044u << 20) ? fdm_halley(d, y) : y;
}

struct fdm_math_exact {
  // the branch-free FP64 forms above, for the FP64 right-hand sides
  // (exp(c x) with a constant c has a form of its own; _sat: finite, for divisors)
  __device__ __forceinline__ static double fast_exp(double x) { return fdm_exp64(x); }
  __device__ __forceinline__ static double fast_exp(double x, const fdm_exp_scale& f) { return fdm_exp64(x, f); }
  __device__ __forceinline__ static double fast_exp_sat(double x) { return fdm_exp64<true>(x); }
  __device__ __forceinline__ static double fast_exp_sat(double x, const fdm_exp_scale& f) { return fdm_exp64<true>(x, f); }
  __device__ __forceinline__ static double fast_expm1(double x) { return fdm_expm1_64(x); }
  __device__ __forceinline__ static double fast_expm1(double x, const fdm_exp_scale& f) { return fdm_expm1_64(x, f); }
  __device__ __forceinline__ static double fast_expm1_sat(double x) { return fdm_expm1_64<true>(x); }
  __device__ __forceinline__ static double fast_expm1_sat(double x, const fdm_exp_scale& f)
  {
    return fdm_expm1_64<true>(x, f);
  }
  __device__ __forceinline__ static double fast_div(double a, double b) { return fdm_div64(a, b); }
  __device__ __forceinline__ static double fast_div0(double x, double e) { return fdm_div64(x, e); }
  __device__ __forceinline__ static double fast_div_any(double a, double b) { return fdm_div64_any(a, b); }
  __device__ __forceinline__ static double fast_rcp(double d) { return fdm_rcp64_any(d); }
  // exp(c x + b) of a group: g from the group's base; x, f: the argument as a product c x by itself
  using exp_group = fdm_exp_group;
  __device__ __forceinline__ static double group_exp(const exp_group& g, double, const fdm_exp_scale&) { return g.exp(); }
  __device__ __forceinline__ static double group_expm1(const exp_group& g, double, const fdm_exp_scale&) { return g.expm1(); }
  __device__ __forceinline__ static double group_exp(const exp_group& g, const fdm_exp_offset& o, double, const fdm_exp_scale&)
  {
    return g.exp(o);
  }
  // (exactly 0 where the argument is)
  __device__ __forceinline__ static double group_expm1(const exp_group& g, const fdm_exp_offset& o, double x,
                                                       const fdm_exp_scale&)
  {
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0 ? 0.0 : g.expm1(o);
  }
  // derivatives for the adjoint: d exp(x)/dx = exp(x), d log(x)/dx = 1/x
  template<class R>
  __device__ __forceinline__ static R dexp(R x, R ex) { (void)x; return ex; }
  template<class R>
  __device__ __forceinline__ static R dlog(R x, R lx) { (void)lx; return (R)1 / x; }
  __device__ __forceinline__ static double exp(double x) { return ::exp(x); }
  __device__ __forceinline__ static float exp(float x) { return __expf(x); }
  __device__ __forceinline__ static double log(double x) { return ::log(x); }
  __device__ __forceinline__ static float log(float x) { return __logf(x); }
  __device__ __forceinline__ static double pow(double x, double y) { return ::pow(x, y); }
  __device__ __forceinline__ static float pow(float x, float y) { return __powf(x, y); }
};

__device__ __forceinline__ double fdm_approx_exp_d(double x)
{
  double y = 1.0 + x / 1024.;
#pragma unroll
  for (int i = 0; i < 10; i++)
    y *= y;
  return y;
}

__device__ __forceinline__ float fdm_approx_exp_f(float x)
{
  // 1024*log1p(x/1024) = x - x^2/2048 + x^3/(3*1024^2) - x^4/(4*1024^3) + ...; the truncation
  // after the x^7 term is below 3e-9 for |x| <= 40.
  if (fabsf(x) > 40.f)
    return (float)fdm_approx_exp_d((double)x);
  const float c2 = -1.f / 2048.f;
  const float c3 = 1.f / (3.f * 1048576.f);
  const float c4 = -1.f / (4.f * 1073741824.f);
  const float c5 = 1.f / (5.f * 1099511627776.f);
  const float c6 = -1.f / (6.f * 1125899906842624.f);
  const float c7 = 1.f / (7.f * 1152921504606846976.f);
  float p = fmaf(x, c7, c6);
  p = fmaf(x, p, c5);
  p = fmaf(x, p, c4);
  p = fmaf(x, p, c3);
  p = fmaf(x, p, c2);
  p = fmaf(x, p, 1.f);
  return __expf(x * p);
}

template<class R>
__device__ __forceinline__ R fdm_approx_log_poly(R x)
{
  const R t1 = x - R(1);
  const R t1_2 = t1 * t1;
  const R t1_4 = t1_2 * t1_2;
  const R t1_6 = t1_4 * t1_2;
  const R r1 = t1 - R(0.5) * t1_2 + R(1. / 3) * t1_2 * t1 - R(0.25) * t1_4 + R(0.2) * t1_4 * t1 - R(1. / 6) * t1_6;
  const R t3 = x - R(3);
  const R t3_2 = t3 * t3;
  const R t3_4 = t3_2 * t3_2;
  const R r3 = R(1.0986122886681098) + R(1. / 3) * t3 - R(0.05555555555555555) * t3_2
               + R(0.012345679012345678) * t3_2 * t3 - R(0.0030864197530864196) * t3_4;
  const R t9 = x - R(9);
  const R t9_2 = t9 * t9;
  const R t9_4 = t9_2 * t9_2;
  const R r9 = R(2.1972245773362196) + R(1. / 9) * t9 - R(0.006172839506172839) * t9_2
               + R(0.0004572473708276177) * t9_2 * t9 - R(3.8103947568968146e-05) * t9_4;
  R r = r1;
  if (x >= R(2) && x < R(6))
    r = r3;
  else if (x >= R(6))
    r = r9;
  return r;
}

struct fdm_math_approx {
  // c x with the product's and the constant's rounding errors added: the quotient by 1/c to an ulp
  __device__ __forceinline__ static double scaled(double x, const fdm_exp_scale& f) { return fma(x, f.c, x * f.c_lo); }
  __device__ __forceinline__ static double fast_exp(double x) { return exp(x); }
  __device__ __forceinline__ static double fast_exp(double x, const fdm_exp_scale& f) { return exp(scaled(x, f)); }
  __device__ __forceinline__ static double fast_exp_sat(double x)
  {
    const double y = exp(x);
    return y > 0x1p1020 ? 0x1p1020 : y;
  }
  __device__ __forceinline__ static double fast_exp_sat(double x, const fdm_exp_scale& f) { return fast_exp_sat(scaled(x, f)); }
  __device__ __forceinline__ static double fast_expm1(double x) { return exp(x) - 1.0; }
  __device__ __forceinline__ static double fast_expm1(double x, const fdm_exp_scale& f) { return fast_exp(x, f) - 1.0; }
  __device__ __forceinline__ static double fast_expm1_sat(double x) { return fast_exp_sat(x) - 1.0; }
  __device__ __forceinline__ static double fast_expm1_sat(double x, const fdm_exp_scale& f) { return fast_exp_sat(x, f) - 1.0; }
  __device__ __forceinline__ static double fast_div(double a, double b) { return fdm_div64(a, b); }
  // the approximation minus 1 is 0 in a neighbourhood of 0
  __device__ __forceinline__ static double fast_div0(double x, double e) { return fdm_div64_any(x, e); }
  __device__ __forceinline__ static double fast_div_any(double a, double b) { return fdm_div64_any(a, b); }
  __device__ __forceinline__ static double fast_rcp(double d) { return fdm_rcp64_any(d); }
  // (not multiplicative: every member by itself)
  struct exp_group {
    __device__ __forceinline__ exp_group(double, const fdm_exp_scale&) {}
  };
  __device__ __forceinline__ static double group_exp(const exp_group&, double x, const fdm_exp_scale& f)
  {
    return fast_exp_sat(x, f);
  }
  __device__ __forceinline__ static double group_expm1(const exp_group&, double x, const fdm_exp_scale& f)
  {
    return fast_expm1_sat(x, f);
  }
  __device__ __forceinline__ static double group_exp(const exp_group&, const fdm_exp_offset&, double x, const fdm_exp_scale& f)
  {
    return fast_exp_sat(x, f);
  }
  __device__ __forceinline__ static double group_expm1(const exp_group&, const fdm_exp_offset&, double x,
                                                       const fdm_exp_scale& f)
  {
    return fast_expm1_sat(x, f);
  }
  // d/dx (1 + x/1024)^1024 = (1 + x/1024)^1023; the log approximation is differentiated as 1/x
  template<class R>
  __device__ __forceinline__ static R dexp(R x, R ex) { return ex / ((R)1 + x / (R)1024); }
  template<class R>
  __device__ __forceinline__ static R dlog(R x, R lx) { (void)lx; return (R)1 / x; }
  __device__ __forceinline__ static double exp(double x) { return fdm_approx_exp_d(x); }
  __device__ __forceinline__ static float exp(float x) { return fdm_approx_exp_f(x); }
  __device__ __forceinline__ static double log(double x)
  {
    double r = fdm_approx_log_poly<double>(x);
    r -= (1 - x / fdm_approx_exp_d(r));
    return r;
  }
  __device__ __forceinline__ static float log(float x)
  {
    float r = fdm_approx_log_poly<float>(x);
    r -= (1.f - __fdividef(x, fdm_approx_exp_f(r)));
    return r;
  }
  __device__ __forceinline__ static double pow(double x, double y) { return ::pow(x, y); }
  __device__ __forceinline__ static float pow(float x, float y) { return __powf(x, y); }
};
