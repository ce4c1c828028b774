// Generated by opendihu_b200/cellml.py from the OpenCOR C export hodgkin_huxley_1952.c; do not edit.
// parametersUsedAsAlgebraic = [], parametersUsedAsConstant = [2, 3, 4]
#pragma once
#include "../fdm_math.cuh"

struct fdm_model_hodgkin_huxley_1952_anone_c2_3_4 {
  static constexpr int nStates = 4;
  static constexpr int nAlgebraics = 9;
  static constexpr int nParameters = 3;
  static constexpr bool usesTime = false;
  static constexpr const char* name = "hodgkin_huxley_1952";
  static constexpr double statesInitialValues[4] = {-0x1.2c00000000000p+6, 0x1.999999999999ap-5, 0x1.3333333333333p-1, 0x1.4cccccccccccdp-2};
  static constexpr double parameterDefaults[3] = {0.0, 0x1.e000000000000p+6, 0x1.2000000000000p+5};
  template<class R> __device__ __forceinline__ static R fdm_pow2(R x) { return x*x; }
  template<class R> __device__ __forceinline__ static R fdm_pow3(R x) { return x*(fdm_pow2(x)); }
  template<class R> __device__ __forceinline__ static R fdm_pow4(R x) { return fdm_pow2(x)*fdm_pow2(x); }
  template<class R, class M>
  __device__ __forceinline__ static void rates(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, R* __restrict__ RATES, R* __restrict__ ALGEBRAIC)
  {
    (void)VOI; (void)PARAMS;
#define FDM_EXP(x) M::exp(x)
#define FDM_LOG(x) M::log(x)
#define FDM_POWF(x, y) M::pow(x, y)
#define FDM_ABS(x) fabs(x)
#define FDM_SQRT(x) sqrt(x)
#define FDM_POW2(x) fdm_pow2(x)
#define FDM_POW3(x) fdm_pow3(x)
#define FDM_POW4(x) fdm_pow4(x)
    ALGEBRAIC[1] = (((-((R)0.100000)) * (STATES[0] + ((R)50.0000))) / (FDM_EXP(((-(STATES[0] + ((R)50.0000))) / ((R)10.0000))) - ((R)1.00000)));
    ALGEBRAIC[5] = (((R)4.00000) * FDM_EXP(((-(STATES[0] + ((R)75.0000))) / ((R)18.0000))));
    RATES[1] = ((ALGEBRAIC[1] * (((R)1.00000) - STATES[1])) - (ALGEBRAIC[5] * STATES[1]));
    ALGEBRAIC[2] = (((R)0.0700000) * FDM_EXP(((-(STATES[0] + ((R)75.0000))) / ((R)20.0000))));
    ALGEBRAIC[6] = (((R)1.00000) / (FDM_EXP(((-(STATES[0] + ((R)45.0000))) / ((R)10.0000))) + ((R)1.00000)));
    RATES[2] = ((ALGEBRAIC[2] * (((R)1.00000) - STATES[2])) - (ALGEBRAIC[6] * STATES[2]));
    ALGEBRAIC[3] = (((-((R)0.0100000)) * (STATES[0] + ((R)65.0000))) / (FDM_EXP(((-(STATES[0] + ((R)65.0000))) / ((R)10.0000))) - ((R)1.00000)));
    ALGEBRAIC[7] = (((R)0.125000) * FDM_EXP(((STATES[0] + ((R)75.0000)) / ((R)80.0000))));
    RATES[3] = ((ALGEBRAIC[3] * (((R)1.00000) - STATES[3])) - (ALGEBRAIC[7] * STATES[3]));
    ALGEBRAIC[0] = (((PARAMS[1] * FDM_POW3(STATES[1])) * STATES[2]) * (STATES[0] - ((R)0x1.4000000000000p+5)));
    ALGEBRAIC[4] = ((PARAMS[2] * FDM_POW4(STATES[3])) * (STATES[0] - ((R)-0x1.5c00000000000p+6)));
    ALGEBRAIC[8] = (((R)0x1.3333333333333p-2) * (STATES[0] - ((R)-0x1.018c49ba5e354p+6)));
    RATES[0] = ((-((((-PARAMS[0]) + ALGEBRAIC[0]) + ALGEBRAIC[4]) + ALGEBRAIC[8])) / ((R)0x1.0000000000000p+0));
#undef FDM_POW2
#undef FDM_POW3
#undef FDM_POW4
#undef FDM_EXP
#undef FDM_LOG
#undef FDM_POWF
#undef FDM_ABS
#undef FDM_SQRT
  }
  // FP64 form: constants collected into one factor per product, divisions by constants as
  // multiplications, exp(u) - 1 by a function of its own
  template<class R, class M>
  __device__ __forceinline__ static void rates_f64(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, R* __restrict__ RATES, R* __restrict__ ALGEBRAIC)
  {
    (void)VOI; (void)PARAMS;
#define FDM_EXP(...) M::fast_exp(__VA_ARGS__)
#define FDM_EXPM1(...) M::fast_expm1(__VA_ARGS__)
#define FDM_EXP_SAT(...) M::fast_exp_sat(__VA_ARGS__)
#define FDM_EXPM1_SAT(...) M::fast_expm1_sat(__VA_ARGS__)
#define FDM_EXP_OF(...) M::group_exp(__VA_ARGS__)
#define FDM_EXPM1_OF(...) M::group_expm1(__VA_ARGS__)
#define FDM_DIV(x, y) M::fast_div(x, y)
#define FDM_DIV0(x, y) M::fast_div0(x, y)
#define FDM_DIV_ANY(x, y) M::fast_div_any(x, y)
#define FDM_LOG(x) M::log(x)
#define FDM_POWF(x, y) M::pow(x, y)
#define FDM_ABS(x) fabs(x)
#define FDM_SQRT(x) sqrt(x)
#define FDM_POW2(x) fdm_pow2(x)
#define FDM_POW3(x) fdm_pow3(x)
#define FDM_POW4(x) fdm_pow4(x)
    const typename M::exp_group fdm_g0((STATES[0] + ((R)0x1.9000000000000p+5)), fdm_exp_scale{-0x1.999999999999ap-4, 0x1.999999999999ap-58, -0x1.2776c50ef9bfep-3, -0x1.bb9d3beb8c800p+2, 0x1.566f7e8b7365ap-47});
    ALGEBRAIC[1] = FDM_DIV0((((R)-0x1.999999999999ap-4) * (STATES[0] + ((R)0x1.9000000000000p+5))), FDM_EXPM1_OF(fdm_g0, (STATES[0] + ((R)0x1.9000000000000p+5)), fdm_exp_scale{-0x1.999999999999ap-4, 0x1.999999999999ap-58, -0x1.2776c50ef9bfep-3, -0x1.bb9d3beb8c800p+2, 0x1.566f7e8b7365ap-47}));
    ALGEBRAIC[5] = (((R)0x1.0000000000000p+2) * FDM_EXP((STATES[0] + ((R)0x1.2c00000000000p+6)), fdm_exp_scale{-0x1.c71c71c71c71cp-5, -0x1.c71c71c71c71cp-59, -0x1.484b13d7c02a9p-4, -0x1.8f40b5ed98000p+3, 0x1.0ba74058e83a2p-45}));
    RATES[1] = ((ALGEBRAIC[1] * (((R)0x1.0000000000000p+0) - STATES[1])) - (ALGEBRAIC[5] * STATES[1]));
    ALGEBRAIC[2] = (((R)0x1.1eb851eb851ecp-4) * FDM_EXP((STATES[0] + ((R)0x1.2c00000000000p+6)), fdm_exp_scale{-0x1.999999999999ap-5, 0x1.999999999999ap-59, -0x1.2776c50ef9bfep-4, -0x1.bb9d3beb8c800p+3, 0x1.566f7e8b7365ap-47}));
    ALGEBRAIC[6] = FDM_DIV(((R)0x1.0000000000000p+0), (FDM_EXP_OF(fdm_g0, fdm_exp_offset{0x1.a61298e1e069cp+0, -0x1.b4690082a4906p-55}, (STATES[0] + ((R)0x1.6800000000000p+5)), fdm_exp_scale{-0x1.999999999999ap-4, 0x1.999999999999ap-58, -0x1.2776c50ef9bfep-3, -0x1.bb9d3beb8c800p+2, 0x1.566f7e8b7365ap-47}) + ((R)0x1.0000000000000p+0)));
    RATES[2] = ((ALGEBRAIC[2] * (((R)0x1.0000000000000p+0) - STATES[2])) - (ALGEBRAIC[6] * STATES[2]));
    ALGEBRAIC[3] = FDM_DIV0((((R)-0x1.47ae147ae147bp-7) * (STATES[0] + ((R)0x1.0400000000000p+6))), FDM_EXPM1_OF(fdm_g0, fdm_exp_offset{0x1.c8f87724b5c1dp-3, 0x1.91afa497dc416p-57}, (STATES[0] + ((R)0x1.0400000000000p+6)), fdm_exp_scale{-0x1.999999999999ap-4, 0x1.999999999999ap-58, -0x1.2776c50ef9bfep-3, -0x1.bb9d3beb8c800p+2, 0x1.566f7e8b7365ap-47}));
    ALGEBRAIC[7] = (((R)0x1.0000000000000p-3) * FDM_EXP((STATES[0] + ((R)0x1.2c00000000000p+6)), fdm_exp_scale{0x1.999999999999ap-7, -0x1.999999999999ap-61, 0x1.2776c50ef9bfep-6, 0x1.bb9d3beb8c800p+5, 0x1.566f7e8b7365ap-47}));
    RATES[3] = ((ALGEBRAIC[3] * (((R)0x1.0000000000000p+0) - STATES[3])) - (ALGEBRAIC[7] * STATES[3]));
    ALGEBRAIC[0] = (((PARAMS[1] * FDM_POW3(STATES[1])) * STATES[2]) * (STATES[0] - ((R)0x1.4000000000000p+5)));
    ALGEBRAIC[4] = ((PARAMS[2] * FDM_POW4(STATES[3])) * (STATES[0] - ((R)-0x1.5c00000000000p+6)));
    ALGEBRAIC[8] = (((R)0x1.3333333333333p-2) * (STATES[0] - ((R)-0x1.018c49ba5e354p+6)));
    RATES[0] = (-((((-PARAMS[0]) + ALGEBRAIC[0]) + ALGEBRAIC[4]) + ALGEBRAIC[8]));
#undef FDM_POW2
#undef FDM_POW3
#undef FDM_POW4
#undef FDM_EXP
#undef FDM_EXPM1
#undef FDM_EXP_SAT
#undef FDM_EXPM1_SAT
#undef FDM_EXP_OF
#undef FDM_EXPM1_OF
#undef FDM_DIV
#undef FDM_DIV0
#undef FDM_DIV_ANY
#undef FDM_LOG
#undef FDM_POWF
#undef FDM_ABS
#undef FDM_SQRT
  }
  // FP32 form: exponentials exp(a.x + b_k) that share a.x are evaluated once as exp(a.x) * e^{b_k};
  // exponentials, logarithms and reciprocals as single SFU instructions (fdm_ex2/fdm_lg2/fdm_rcp)
  static constexpr int nSharedExponentials = 1;
  template<class R, class M>
  __device__ __forceinline__ static void rates_fast(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, R* __restrict__ RATES, R* __restrict__ ALGEBRAIC)
  {
    (void)VOI; (void)PARAMS;
#define FDM_EXP(x) M::exp(x)
#define FDM_LOG(x) M::log(x)
#define FDM_POWF(x, y) M::pow(x, y)
#define FDM_ABS(x) fabs(x)
#define FDM_SQRT(x) sqrt(x)
#define FDM_POW2(x) fdm_pow2(x)
#define FDM_POW3(x) fdm_pow3(x)
#define FDM_POW4(x) fdm_pow4(x)
    const R fdm_e0 = fdm_ex2(((R)-0x1.2776c50ef9bffp-3) * STATES[0]);
    const R fdm_d0 = ((fdm_e0 * ((R)0x1.b993fe00d5376p-8)) + ((R)-0x1.0000000000000p+0));
    const R fdm_d1 = ((fdm_e0 * ((R)0x1.6c0504695c417p-7)) + ((R)1.00000));
    const R fdm_d2 = ((fdm_e0 * ((R)0x1.8a1e18a954ffap-10)) + ((R)-0x1.0000000000000p+0));
    R fdm_r0, fdm_r1, fdm_r2;
    fdm_rcp_batch(fdm_d0, fdm_d1, fdm_d2, fdm_r0, fdm_r1, fdm_r2);
    ALGEBRAIC[1] = ((((R)-0x1.999999999999ap-4) * STATES[0] + ((R)-0x1.4000000000000p+2)) * fdm_r0);
    ALGEBRAIC[5] = fdm_ex2(((R)-0x1.484b13d7c02a9p-4) * STATES[0] + ((R)-0x1.00b7fb40d531ep+2));
    RATES[1] = (ALGEBRAIC[1] - (ALGEBRAIC[1] + ALGEBRAIC[5]) * STATES[1]);
    ALGEBRAIC[2] = fdm_ex2(((R)-0x1.2776c50ef9bffp-4) * STATES[0] + ((R)-0x1.27e435c543615p+3));
    ALGEBRAIC[6] = fdm_r1;
    RATES[2] = (ALGEBRAIC[2] - (ALGEBRAIC[2] + ALGEBRAIC[6]) * STATES[2]);
    ALGEBRAIC[3] = ((((R)-0x1.47ae147ae147bp-7) * STATES[0] + ((R)-0x1.4cccccccccccdp-1)) * fdm_r2);
    ALGEBRAIC[7] = fdm_ex2(((R)0x1.2776c50ef9bffp-6) * STATES[0] + ((R)-0x1.a5c0d11273531p+0));
    RATES[3] = (ALGEBRAIC[3] - (ALGEBRAIC[3] + ALGEBRAIC[7]) * STATES[3]);
    ALGEBRAIC[0] = (((PARAMS[1] * FDM_POW3(STATES[1])) * STATES[2]) * (STATES[0] - ((R)0x1.4000000000000p+5)));
    ALGEBRAIC[4] = ((PARAMS[2] * FDM_POW4(STATES[3])) * (STATES[0] - ((R)-0x1.5c00000000000p+6)));
    ALGEBRAIC[8] = (((R)0x1.3333333333333p-2) * STATES[0] + ((R)0x1.350ebedfa43fep+4));
    RATES[0] = (((PARAMS[0] - ALGEBRAIC[0]) - ALGEBRAIC[4]) - ALGEBRAIC[8]);
#undef FDM_POW2
#undef FDM_POW3
#undef FDM_POW4
#undef FDM_EXP
#undef FDM_LOG
#undef FDM_POWF
#undef FDM_ABS
#undef FDM_SQRT
  }
  // paired FP32 form: the FP32 form over two nodes at once (fdm_f2, packed FP32 instructions)
  template<class M>
  __device__ __forceinline__ static void rates_fast2(const fdm_f2 VOI, const fdm_f2* __restrict__ STATES, const fdm_f2* __restrict__ PARAMS, fdm_f2* __restrict__ RATES, fdm_f2* __restrict__ ALGEBRAIC)
  {
    typedef fdm_f2 R;
    (void)VOI; (void)PARAMS;
#define FDM_POWF(x, y) fdm_powf_pair(x, y)
#define FDM_ABS(x) fabs(x)
#define FDM_SQRT(x) sqrt(x)
#define FDM_POW2(x) fdm_pow2(x)
#define FDM_POW3(x) fdm_pow3(x)
#define FDM_POW4(x) fdm_pow4(x)
    const R fdm_h0 = fdm_ex2(((R)-0x1.2776c50ef9bffp-4) * STATES[0] + ((R)-0x1.27e435c543615p+3));
    const R fdm_e0 = fdm_h0 * fdm_h0;
    const R fdm_d0 = ((fdm_e0 * ((R)0x1.36c724ec76f8fp+11)) + ((R)-0x1.0000000000000p+0));
    const R fdm_d1 = ((fdm_e0 * ((R)0x1.00316d3b6c10ap+12)) + ((R)1.00000));
    const R fdm_d2 = ((fdm_e0 * ((R)0x1.15602daa0de7fp+9)) + ((R)-0x1.0000000000000p+0));
    R fdm_r0, fdm_r1, fdm_r2;
    fdm_rcp_batch(fdm_d0, fdm_d1, fdm_d2, fdm_r0, fdm_r1, fdm_r2);
    ALGEBRAIC[1] = ((((R)-0x1.999999999999ap-4) * STATES[0] + ((R)-0x1.4000000000000p+2)) * fdm_r0);
    ALGEBRAIC[5] = fdm_ex2(((R)-0x1.484b13d7c02a9p-4) * STATES[0] + ((R)-0x1.00b7fb40d531ep+2));
    RATES[1] = (ALGEBRAIC[1] - (ALGEBRAIC[1] + ALGEBRAIC[5]) * STATES[1]);
    ALGEBRAIC[2] = fdm_h0;
    ALGEBRAIC[6] = fdm_r1;
    RATES[2] = (ALGEBRAIC[2] - (ALGEBRAIC[2] + ALGEBRAIC[6]) * STATES[2]);
    ALGEBRAIC[3] = ((((R)-0x1.47ae147ae147bp-7) * STATES[0] + ((R)-0x1.4cccccccccccdp-1)) * fdm_r2);
    ALGEBRAIC[7] = fdm_ex2(((R)0x1.2776c50ef9bffp-6) * STATES[0] + ((R)-0x1.a5c0d11273531p+0));
    RATES[3] = (ALGEBRAIC[3] - (ALGEBRAIC[3] + ALGEBRAIC[7]) * STATES[3]);
    ALGEBRAIC[0] = (((PARAMS[1] * FDM_POW3(STATES[1])) * STATES[2]) * (STATES[0] - ((R)0x1.4000000000000p+5)));
    ALGEBRAIC[4] = ((PARAMS[2] * FDM_POW4(STATES[3])) * (STATES[0] - ((R)-0x1.5c00000000000p+6)));
    ALGEBRAIC[8] = (((R)0x1.3333333333333p-2) * STATES[0] + ((R)0x1.350ebedfa43fep+4));
    RATES[0] = ((((PARAMS[2] * FDM_POW4(STATES[3]))) * (((R)-0x1.5c00000000000p+6) - STATES[0]) + ((((PARAMS[1] * FDM_POW3(STATES[1])) * STATES[2])) * (((R)0x1.4000000000000p+5) - STATES[0]) + PARAMS[0])) - ALGEBRAIC[8]);
#undef FDM_POW2
#undef FDM_POW3
#undef FDM_POW4
#undef FDM_POWF
#undef FDM_ABS
#undef FDM_SQRT
  }
  // vector-Jacobian product: LAM_STATES += J^T LAM_RATES, LAM_PARAMS += (dRATES/dPARAMS)^T LAM_RATES
  template<class R, class M>
  __device__ __forceinline__ static void rates_vjp(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, const R* __restrict__ LAM_RATES, R* __restrict__ LAM_STATES, R* __restrict__ LAM_PARAMS)
  {
    (void)VOI; (void)PARAMS;
#define FDM_POW2(x) fdm_pow2(x)
#define FDM_POW3(x) fdm_pow3(x)
#define FDM_POW4(x) fdm_pow4(x)
    R ALG[9];
    (void)ALG;
    const R t0 = (-((R)0.100000));
    const R t1 = (STATES[0] + ((R)50.0000));
    const R t2 = (t0 * t1);
    const R t3 = (STATES[0] + ((R)50.0000));
    const R t4 = (-t3);
    const R t5 = (t4 / ((R)10.0000));
    const R t6 = M::exp(t5);
    const R t7 = (t6 - ((R)1.00000));
    const R t8 = (t2 / t7);
    ALG[1] = t8;
    const R t9 = (STATES[0] + ((R)75.0000));
    const R t10 = (-t9);
    const R t11 = (t10 / ((R)18.0000));
    const R t12 = M::exp(t11);
    const R t13 = (((R)4.00000) * t12);
    ALG[5] = t13;
    const R t14 = (((R)1.00000) - STATES[1]);
    const R t15 = (t8 * t14);
    const R t16 = (t13 * STATES[1]);
    const R t17 = (t15 - t16);
    const R t18 = (STATES[0] + ((R)75.0000));
    const R t19 = (-t18);
    const R t20 = (t19 / ((R)20.0000));
    const R t21 = M::exp(t20);
    const R t22 = (((R)0.0700000) * t21);
    ALG[2] = t22;
    const R t23 = (STATES[0] + ((R)45.0000));
    const R t24 = (-t23);
    const R t25 = (t24 / ((R)10.0000));
    const R t26 = M::exp(t25);
    const R t27 = (t26 + ((R)1.00000));
    const R t28 = (((R)1.00000) / t27);
    ALG[6] = t28;
    const R t29 = (((R)1.00000) - STATES[2]);
    const R t30 = (t22 * t29);
    const R t31 = (t28 * STATES[2]);
    const R t32 = (t30 - t31);
    const R t33 = (-((R)0.0100000));
    const R t34 = (STATES[0] + ((R)65.0000));
    const R t35 = (t33 * t34);
    const R t36 = (STATES[0] + ((R)65.0000));
    const R t37 = (-t36);
    const R t38 = (t37 / ((R)10.0000));
    const R t39 = M::exp(t38);
    const R t40 = (t39 - ((R)1.00000));
    const R t41 = (t35 / t40);
    ALG[3] = t41;
    const R t42 = (STATES[0] + ((R)75.0000));
    const R t43 = (t42 / ((R)80.0000));
    const R t44 = M::exp(t43);
    const R t45 = (((R)0.125000) * t44);
    ALG[7] = t45;
    const R t46 = (((R)1.00000) - STATES[3]);
    const R t47 = (t41 * t46);
    const R t48 = (t45 * STATES[3]);
    const R t49 = (t47 - t48);
    const R t50 = FDM_POW3(STATES[1]);
    const R t51 = (PARAMS[1] * t50);
    const R t52 = (t51 * STATES[2]);
    const R t53 = (STATES[0] - ((R)0x1.4000000000000p+5));
    const R t54 = (t52 * t53);
    ALG[0] = t54;
    const R t55 = FDM_POW4(STATES[3]);
    const R t56 = (PARAMS[2] * t55);
    const R t57 = (STATES[0] - ((R)-0x1.5c00000000000p+6));
    const R t58 = (t56 * t57);
    ALG[4] = t58;
    const R t59 = (STATES[0] - ((R)-0x1.018c49ba5e354p+6));
    const R t60 = (((R)0x1.3333333333333p-2) * t59);
    ALG[8] = t60;
    const R t61 = (-PARAMS[0]);
    const R t62 = (t61 + t54);
    const R t63 = (t62 + t58);
    const R t64 = (t63 + t60);
    const R t65 = (-t64);
    const R t66 = (t65 / ((R)0x1.0000000000000p+0));
    R a_t0 = (R)0;
    R a_t1 = (R)0;
    R a_t2 = (R)0;
    R a_t3 = (R)0;
    R a_t4 = (R)0;
    R a_t5 = (R)0;
    R a_t6 = (R)0;
    R a_t7 = (R)0;
    R a_t8 = (R)0;
    R a_t9 = (R)0;
    R a_t10 = (R)0;
    R a_t11 = (R)0;
    R a_t12 = (R)0;
    R a_t13 = (R)0;
    R a_t14 = (R)0;
    R a_t15 = (R)0;
    R a_t16 = (R)0;
    R a_t17 = (R)0;
    R a_t18 = (R)0;
    R a_t19 = (R)0;
    R a_t20 = (R)0;
    R a_t21 = (R)0;
    R a_t22 = (R)0;
    R a_t23 = (R)0;
    R a_t24 = (R)0;
    R a_t25 = (R)0;
    R a_t26 = (R)0;
    R a_t27 = (R)0;
    R a_t28 = (R)0;
    R a_t29 = (R)0;
    R a_t30 = (R)0;
    R a_t31 = (R)0;
    R a_t32 = (R)0;
    R a_t33 = (R)0;
    R a_t34 = (R)0;
    R a_t35 = (R)0;
    R a_t36 = (R)0;
    R a_t37 = (R)0;
    R a_t38 = (R)0;
    R a_t39 = (R)0;
    R a_t40 = (R)0;
    R a_t41 = (R)0;
    R a_t42 = (R)0;
    R a_t43 = (R)0;
    R a_t44 = (R)0;
    R a_t45 = (R)0;
    R a_t46 = (R)0;
    R a_t47 = (R)0;
    R a_t48 = (R)0;
    R a_t49 = (R)0;
    R a_t50 = (R)0;
    R a_t51 = (R)0;
    R a_t52 = (R)0;
    R a_t53 = (R)0;
    R a_t54 = (R)0;
    R a_t55 = (R)0;
    R a_t56 = (R)0;
    R a_t57 = (R)0;
    R a_t58 = (R)0;
    R a_t59 = (R)0;
    R a_t60 = (R)0;
    R a_t61 = (R)0;
    R a_t62 = (R)0;
    R a_t63 = (R)0;
    R a_t64 = (R)0;
    R a_t65 = (R)0;
    R a_t66 = (R)0;
    a_t66 += LAM_RATES[0];
    a_t17 += LAM_RATES[1];
    a_t32 += LAM_RATES[2];
    a_t49 += LAM_RATES[3];
    a_t65 += a_t66 / ((R)0x1.0000000000000p+0);
    a_t64 += -a_t65;
    a_t63 += a_t64;
    a_t60 += a_t64;
    a_t62 += a_t63;
    a_t58 += a_t63;
    a_t61 += a_t62;
    a_t54 += a_t62;
    LAM_PARAMS[0] += -a_t61;
    a_t59 += a_t60 * ((R)0x1.3333333333333p-2);
    LAM_STATES[0] += a_t59;
    a_t56 += a_t58 * t57;
    a_t57 += a_t58 * t56;
    LAM_STATES[0] += a_t57;
    LAM_PARAMS[2] += a_t56 * t55;
    a_t55 += a_t56 * PARAMS[2];
    LAM_STATES[3] += a_t55 * ((R)4 * FDM_POW3(STATES[3]));
    a_t52 += a_t54 * t53;
    a_t53 += a_t54 * t52;
    LAM_STATES[0] += a_t53;
    a_t51 += a_t52 * STATES[2];
    LAM_STATES[2] += a_t52 * t51;
    LAM_PARAMS[1] += a_t51 * t50;
    a_t50 += a_t51 * PARAMS[1];
    LAM_STATES[1] += a_t50 * ((R)3 * FDM_POW2(STATES[1]));
    a_t47 += a_t49;
    a_t48 += -a_t49;
    a_t45 += a_t48 * STATES[3];
    LAM_STATES[3] += a_t48 * t45;
    a_t41 += a_t47 * t46;
    a_t46 += a_t47 * t41;
    LAM_STATES[3] += -a_t46;
    a_t44 += a_t45 * ((R)0.125000);
    a_t43 += a_t44 * M::dexp(t43, t44);
    a_t42 += a_t43 / ((R)80.0000);
    LAM_STATES[0] += a_t42;
    a_t35 += a_t41 / t40;
    a_t40 += -a_t41 * t41 / t40;
    a_t39 += a_t40;
    a_t38 += a_t39 * M::dexp(t38, t39);
    a_t37 += a_t38 / ((R)10.0000);
    a_t36 += -a_t37;
    LAM_STATES[0] += a_t36;
    a_t33 += a_t35 * t34;
    a_t34 += a_t35 * t33;
    LAM_STATES[0] += a_t34;
    a_t30 += a_t32;
    a_t31 += -a_t32;
    a_t28 += a_t31 * STATES[2];
    LAM_STATES[2] += a_t31 * t28;
    a_t22 += a_t30 * t29;
    a_t29 += a_t30 * t22;
    LAM_STATES[2] += -a_t29;
    a_t27 += -a_t28 * t28 / t27;
    a_t26 += a_t27;
    a_t25 += a_t26 * M::dexp(t25, t26);
    a_t24 += a_t25 / ((R)10.0000);
    a_t23 += -a_t24;
    LAM_STATES[0] += a_t23;
    a_t21 += a_t22 * ((R)0.0700000);
    a_t20 += a_t21 * M::dexp(t20, t21);
    a_t19 += a_t20 / ((R)20.0000);
    a_t18 += -a_t19;
    LAM_STATES[0] += a_t18;
    a_t15 += a_t17;
    a_t16 += -a_t17;
    a_t13 += a_t16 * STATES[1];
    LAM_STATES[1] += a_t16 * t13;
    a_t8 += a_t15 * t14;
    a_t14 += a_t15 * t8;
    LAM_STATES[1] += -a_t14;
    a_t12 += a_t13 * ((R)4.00000);
    a_t11 += a_t12 * M::dexp(t11, t12);
    a_t10 += a_t11 / ((R)18.0000);
    a_t9 += -a_t10;
    LAM_STATES[0] += a_t9;
    a_t2 += a_t8 / t7;
    a_t7 += -a_t8 * t8 / t7;
    a_t6 += a_t7;
    a_t5 += a_t6 * M::dexp(t5, t6);
    a_t4 += a_t5 / ((R)10.0000);
    a_t3 += -a_t4;
    LAM_STATES[0] += a_t3;
    a_t0 += a_t2 * t1;
    a_t1 += a_t2 * t0;
    LAM_STATES[0] += a_t1;
  }
  static constexpr int nTape = 67;
  template<class R, class M>
  __device__ __forceinline__ static void rates_tape(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, R* __restrict__ RATES, R* __restrict__ TAPE)
  {
    (void)VOI; (void)PARAMS;
    R ALG[9];
    (void)ALG;
    const R t0 = (-((R)0.100000));
    TAPE[0] = t0;
    const R t1 = (STATES[0] + ((R)50.0000));
    TAPE[1] = t1;
    const R t2 = (t0 * t1);
    TAPE[2] = t2;
    const R t3 = (STATES[0] + ((R)50.0000));
    TAPE[3] = t3;
    const R t4 = (-t3);
    TAPE[4] = t4;
    const R t5 = (t4 / ((R)10.0000));
    TAPE[5] = t5;
    const R t6 = M::exp(t5);
    TAPE[6] = t6;
    const R t7 = (t6 - ((R)1.00000));
    TAPE[7] = t7;
    const R t8 = (t2 / t7);
    TAPE[8] = t8;
    ALG[1] = t8;
    const R t9 = (STATES[0] + ((R)75.0000));
    TAPE[9] = t9;
    const R t10 = (-t9);
    TAPE[10] = t10;
    const R t11 = (t10 / ((R)18.0000));
    TAPE[11] = t11;
    const R t12 = M::exp(t11);
    TAPE[12] = t12;
    const R t13 = (((R)4.00000) * t12);
    TAPE[13] = t13;
    ALG[5] = t13;
    const R t14 = (((R)1.00000) - STATES[1]);
    TAPE[14] = t14;
    const R t15 = (t8 * t14);
    TAPE[15] = t15;
    const R t16 = (t13 * STATES[1]);
    TAPE[16] = t16;
    const R t17 = (t15 - t16);
    TAPE[17] = t17;
    const R t18 = (STATES[0] + ((R)75.0000));
    TAPE[18] = t18;
    const R t19 = (-t18);
    TAPE[19] = t19;
    const R t20 = (t19 / ((R)20.0000));
    TAPE[20] = t20;
    const R t21 = M::exp(t20);
    TAPE[21] = t21;
    const R t22 = (((R)0.0700000) * t21);
    TAPE[22] = t22;
    ALG[2] = t22;
    const R t23 = (STATES[0] + ((R)45.0000));
    TAPE[23] = t23;
    const R t24 = (-t23);
    TAPE[24] = t24;
    const R t25 = (t24 / ((R)10.0000));
    TAPE[25] = t25;
    const R t26 = M::exp(t25);
    TAPE[26] = t26;
    const R t27 = (t26 + ((R)1.00000));
    TAPE[27] = t27;
    const R t28 = (((R)1.00000) / t27);
    TAPE[28] = t28;
    ALG[6] = t28;
    const R t29 = (((R)1.00000) - STATES[2]);
    TAPE[29] = t29;
    const R t30 = (t22 * t29);
    TAPE[30] = t30;
    const R t31 = (t28 * STATES[2]);
    TAPE[31] = t31;
    const R t32 = (t30 - t31);
    TAPE[32] = t32;
    const R t33 = (-((R)0.0100000));
    TAPE[33] = t33;
    const R t34 = (STATES[0] + ((R)65.0000));
    TAPE[34] = t34;
    const R t35 = (t33 * t34);
    TAPE[35] = t35;
    const R t36 = (STATES[0] + ((R)65.0000));
    TAPE[36] = t36;
    const R t37 = (-t36);
    TAPE[37] = t37;
    const R t38 = (t37 / ((R)10.0000));
    TAPE[38] = t38;
    const R t39 = M::exp(t38);
    TAPE[39] = t39;
    const R t40 = (t39 - ((R)1.00000));
    TAPE[40] = t40;
    const R t41 = (t35 / t40);
    TAPE[41] = t41;
    ALG[3] = t41;
    const R t42 = (STATES[0] + ((R)75.0000));
    TAPE[42] = t42;
    const R t43 = (t42 / ((R)80.0000));
    TAPE[43] = t43;
    const R t44 = M::exp(t43);
    TAPE[44] = t44;
    const R t45 = (((R)0.125000) * t44);
    TAPE[45] = t45;
    ALG[7] = t45;
    const R t46 = (((R)1.00000) - STATES[3]);
    TAPE[46] = t46;
    const R t47 = (t41 * t46);
    TAPE[47] = t47;
    const R t48 = (t45 * STATES[3]);
    TAPE[48] = t48;
    const R t49 = (t47 - t48);
    TAPE[49] = t49;
    const R t50 = FDM_POW3(STATES[1]);
    TAPE[50] = t50;
    const R t51 = (PARAMS[1] * t50);
    TAPE[51] = t51;
    const R t52 = (t51 * STATES[2]);
    TAPE[52] = t52;
    const R t53 = (STATES[0] - ((R)0x1.4000000000000p+5));
    TAPE[53] = t53;
    const R t54 = (t52 * t53);
    TAPE[54] = t54;
    ALG[0] = t54;
    const R t55 = FDM_POW4(STATES[3]);
    TAPE[55] = t55;
    const R t56 = (PARAMS[2] * t55);
    TAPE[56] = t56;
    const R t57 = (STATES[0] - ((R)-0x1.5c00000000000p+6));
    TAPE[57] = t57;
    const R t58 = (t56 * t57);
    TAPE[58] = t58;
    ALG[4] = t58;
    const R t59 = (STATES[0] - ((R)-0x1.018c49ba5e354p+6));
    TAPE[59] = t59;
    const R t60 = (((R)0x1.3333333333333p-2) * t59);
    TAPE[60] = t60;
    ALG[8] = t60;
    const R t61 = (-PARAMS[0]);
    TAPE[61] = t61;
    const R t62 = (t61 + t54);
    TAPE[62] = t62;
    const R t63 = (t62 + t58);
    TAPE[63] = t63;
    const R t64 = (t63 + t60);
    TAPE[64] = t64;
    const R t65 = (-t64);
    TAPE[65] = t65;
    const R t66 = (t65 / ((R)0x1.0000000000000p+0));
    TAPE[66] = t66;
    RATES[0] = t66;
    RATES[1] = t17;
    RATES[2] = t32;
    RATES[3] = t49;
  }
  template<class R, class M>
  __device__ __forceinline__ static void rates_vjp_tape(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, const R* __restrict__ TAPE, const R* __restrict__ LAM_RATES, R* __restrict__ LAM_STATES, R* __restrict__ LAM_PARAMS)
  {
    (void)VOI; (void)PARAMS; (void)STATES;
    const R t0 = TAPE[0];
    const R t1 = TAPE[1];
    const R t2 = TAPE[2];
    const R t3 = TAPE[3];
    const R t4 = TAPE[4];
    const R t5 = TAPE[5];
    const R t6 = TAPE[6];
    const R t7 = TAPE[7];
    const R t8 = TAPE[8];
    const R t9 = TAPE[9];
    const R t10 = TAPE[10];
    const R t11 = TAPE[11];
    const R t12 = TAPE[12];
    const R t13 = TAPE[13];
    const R t14 = TAPE[14];
    const R t15 = TAPE[15];
    const R t16 = TAPE[16];
    const R t17 = TAPE[17];
    const R t18 = TAPE[18];
    const R t19 = TAPE[19];
    const R t20 = TAPE[20];
    const R t21 = TAPE[21];
    const R t22 = TAPE[22];
    const R t23 = TAPE[23];
    const R t24 = TAPE[24];
    const R t25 = TAPE[25];
    const R t26 = TAPE[26];
    const R t27 = TAPE[27];
    const R t28 = TAPE[28];
    const R t29 = TAPE[29];
    const R t30 = TAPE[30];
    const R t31 = TAPE[31];
    const R t32 = TAPE[32];
    const R t33 = TAPE[33];
    const R t34 = TAPE[34];
    const R t35 = TAPE[35];
    const R t36 = TAPE[36];
    const R t37 = TAPE[37];
    const R t38 = TAPE[38];
    const R t39 = TAPE[39];
    const R t40 = TAPE[40];
    const R t41 = TAPE[41];
    const R t42 = TAPE[42];
    const R t43 = TAPE[43];
    const R t44 = TAPE[44];
    const R t45 = TAPE[45];
    const R t46 = TAPE[46];
    const R t47 = TAPE[47];
    const R t48 = TAPE[48];
    const R t49 = TAPE[49];
    const R t50 = TAPE[50];
    const R t51 = TAPE[51];
    const R t52 = TAPE[52];
    const R t53 = TAPE[53];
    const R t54 = TAPE[54];
    const R t55 = TAPE[55];
    const R t56 = TAPE[56];
    const R t57 = TAPE[57];
    const R t58 = TAPE[58];
    const R t59 = TAPE[59];
    const R t60 = TAPE[60];
    const R t61 = TAPE[61];
    const R t62 = TAPE[62];
    const R t63 = TAPE[63];
    const R t64 = TAPE[64];
    const R t65 = TAPE[65];
    const R t66 = TAPE[66];
    R a_t0 = (R)0;
    R a_t1 = (R)0;
    R a_t2 = (R)0;
    R a_t3 = (R)0;
    R a_t4 = (R)0;
    R a_t5 = (R)0;
    R a_t6 = (R)0;
    R a_t7 = (R)0;
    R a_t8 = (R)0;
    R a_t9 = (R)0;
    R a_t10 = (R)0;
    R a_t11 = (R)0;
    R a_t12 = (R)0;
    R a_t13 = (R)0;
    R a_t14 = (R)0;
    R a_t15 = (R)0;
    R a_t16 = (R)0;
    R a_t17 = (R)0;
    R a_t18 = (R)0;
    R a_t19 = (R)0;
    R a_t20 = (R)0;
    R a_t21 = (R)0;
    R a_t22 = (R)0;
    R a_t23 = (R)0;
    R a_t24 = (R)0;
    R a_t25 = (R)0;
    R a_t26 = (R)0;
    R a_t27 = (R)0;
    R a_t28 = (R)0;
    R a_t29 = (R)0;
    R a_t30 = (R)0;
    R a_t31 = (R)0;
    R a_t32 = (R)0;
    R a_t33 = (R)0;
    R a_t34 = (R)0;
    R a_t35 = (R)0;
    R a_t36 = (R)0;
    R a_t37 = (R)0;
    R a_t38 = (R)0;
    R a_t39 = (R)0;
    R a_t40 = (R)0;
    R a_t41 = (R)0;
    R a_t42 = (R)0;
    R a_t43 = (R)0;
    R a_t44 = (R)0;
    R a_t45 = (R)0;
    R a_t46 = (R)0;
    R a_t47 = (R)0;
    R a_t48 = (R)0;
    R a_t49 = (R)0;
    R a_t50 = (R)0;
    R a_t51 = (R)0;
    R a_t52 = (R)0;
    R a_t53 = (R)0;
    R a_t54 = (R)0;
    R a_t55 = (R)0;
    R a_t56 = (R)0;
    R a_t57 = (R)0;
    R a_t58 = (R)0;
    R a_t59 = (R)0;
    R a_t60 = (R)0;
    R a_t61 = (R)0;
    R a_t62 = (R)0;
    R a_t63 = (R)0;
    R a_t64 = (R)0;
    R a_t65 = (R)0;
    R a_t66 = (R)0;
    a_t66 += LAM_RATES[0];
    a_t17 += LAM_RATES[1];
    a_t32 += LAM_RATES[2];
    a_t49 += LAM_RATES[3];
    a_t65 += a_t66 / ((R)0x1.0000000000000p+0);
    a_t64 += -a_t65;
    a_t63 += a_t64;
    a_t60 += a_t64;
    a_t62 += a_t63;
    a_t58 += a_t63;
    a_t61 += a_t62;
    a_t54 += a_t62;
    LAM_PARAMS[0] += -a_t61;
    a_t59 += a_t60 * ((R)0x1.3333333333333p-2);
    LAM_STATES[0] += a_t59;
    a_t56 += a_t58 * t57;
    a_t57 += a_t58 * t56;
    LAM_STATES[0] += a_t57;
    LAM_PARAMS[2] += a_t56 * t55;
    a_t55 += a_t56 * PARAMS[2];
    LAM_STATES[3] += a_t55 * ((R)4 * FDM_POW3(STATES[3]));
    a_t52 += a_t54 * t53;
    a_t53 += a_t54 * t52;
    LAM_STATES[0] += a_t53;
    a_t51 += a_t52 * STATES[2];
    LAM_STATES[2] += a_t52 * t51;
    LAM_PARAMS[1] += a_t51 * t50;
    a_t50 += a_t51 * PARAMS[1];
    LAM_STATES[1] += a_t50 * ((R)3 * FDM_POW2(STATES[1]));
    a_t47 += a_t49;
    a_t48 += -a_t49;
    a_t45 += a_t48 * STATES[3];
    LAM_STATES[3] += a_t48 * t45;
    a_t41 += a_t47 * t46;
    a_t46 += a_t47 * t41;
    LAM_STATES[3] += -a_t46;
    a_t44 += a_t45 * ((R)0.125000);
    a_t43 += a_t44 * M::dexp(t43, t44);
    a_t42 += a_t43 / ((R)80.0000);
    LAM_STATES[0] += a_t42;
    a_t35 += a_t41 / t40;
    a_t40 += -a_t41 * t41 / t40;
    a_t39 += a_t40;
    a_t38 += a_t39 * M::dexp(t38, t39);
    a_t37 += a_t38 / ((R)10.0000);
    a_t36 += -a_t37;
    LAM_STATES[0] += a_t36;
    a_t33 += a_t35 * t34;
    a_t34 += a_t35 * t33;
    LAM_STATES[0] += a_t34;
    a_t30 += a_t32;
    a_t31 += -a_t32;
    a_t28 += a_t31 * STATES[2];
    LAM_STATES[2] += a_t31 * t28;
    a_t22 += a_t30 * t29;
    a_t29 += a_t30 * t22;
    LAM_STATES[2] += -a_t29;
    a_t27 += -a_t28 * t28 / t27;
    a_t26 += a_t27;
    a_t25 += a_t26 * M::dexp(t25, t26);
    a_t24 += a_t25 / ((R)10.0000);
    a_t23 += -a_t24;
    LAM_STATES[0] += a_t23;
    a_t21 += a_t22 * ((R)0.0700000);
    a_t20 += a_t21 * M::dexp(t20, t21);
    a_t19 += a_t20 / ((R)20.0000);
    a_t18 += -a_t19;
    LAM_STATES[0] += a_t18;
    a_t15 += a_t17;
    a_t16 += -a_t17;
    a_t13 += a_t16 * STATES[1];
    LAM_STATES[1] += a_t16 * t13;
    a_t8 += a_t15 * t14;
    a_t14 += a_t15 * t8;
    LAM_STATES[1] += -a_t14;
    a_t12 += a_t13 * ((R)4.00000);
    a_t11 += a_t12 * M::dexp(t11, t12);
    a_t10 += a_t11 / ((R)18.0000);
    a_t9 += -a_t10;
    LAM_STATES[0] += a_t9;
    a_t2 += a_t8 / t7;
    a_t7 += -a_t8 * t8 / t7;
    a_t6 += a_t7;
    a_t5 += a_t6 * M::dexp(t5, t6);
    a_t4 += a_t5 / ((R)10.0000);
    a_t3 += -a_t4;
    LAM_STATES[0] += a_t3;
    a_t0 += a_t2 * t1;
    a_t1 += a_t2 * t0;
    LAM_STATES[0] += a_t1;
  }
#undef FDM_POW2
#undef FDM_POW3
#undef FDM_POW4
  // the same in the fast form (exact exponentials): shared exponentials, reciprocals
  template<class R, class M>
  __device__ __forceinline__ static void rates_vjp_fast(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, const R* __restrict__ LAM_RATES, R* __restrict__ LAM_STATES, R* __restrict__ LAM_PARAMS)
  {
    (void)VOI; (void)PARAMS;
#define FDM_POW2(x) fdm_pow2(x)
#define FDM_POW3(x) fdm_pow3(x)
#define FDM_POW4(x) fdm_pow4(x)
    R ALG[9];
    (void)ALG;
    const R t0 = (-((R)0.100000));
    const R t1 = (STATES[0] + ((R)50.0000));
    const R t2 = (t0 * t1);
    const R t3 = (((R)-0x1.999999999999ap-4) * STATES[0]);
    const R t4 = M::fast_exp(t3);
    const R t5 = (t4 * ((R)0x1.b993fe00d5376p-8));
    const R t6 = (t5 - ((R)1.00000));
    const R t7 = M::fast_rcp(t6);
    const R t8 = (t2 * t7);
    ALG[1] = t8;
    const R t9 = (STATES[0] + ((R)75.0000));
    const R t10 = (-t9);
    const R t11 = (t10 * ((R)0x1.c71c71c71c71cp-5));
    const R t12 = M::fast_exp(t11);
    const R t13 = (((R)4.00000) * t12);
    ALG[5] = t13;
    const R t14 = (((R)1.00000) - STATES[1]);
    const R t15 = (t8 * t14);
    const R t16 = (t13 * STATES[1]);
    const R t17 = (t15 - t16);
    const R t18 = (STATES[0] + ((R)75.0000));
    const R t19 = (-t18);
    const R t20 = (t19 * ((R)0x1.999999999999ap-5));
    const R t21 = M::fast_exp(t20);
    const R t22 = (((R)0.0700000) * t21);
    ALG[2] = t22;
    const R t23 = (t4 * ((R)0x1.6c0504695c417p-7));
    const R t24 = (t23 + ((R)1.00000));
    const R t25 = M::fast_rcp(t24);
    const R t26 = (((R)1.00000) * t25);
    ALG[6] = t26;
    const R t27 = (((R)1.00000) - STATES[2]);
    const R t28 = (t22 * t27);
    const R t29 = (t26 * STATES[2]);
    const R t30 = (t28 - t29);
    const R t31 = (-((R)0.0100000));
    const R t32 = (STATES[0] + ((R)65.0000));
    const R t33 = (t31 * t32);
    const R t34 = (t4 * ((R)0x1.8a1e18a954ffap-10));
    const R t35 = (t34 - ((R)1.00000));
    const R t36 = M::fast_rcp(t35);
    const R t37 = (t33 * t36);
    ALG[3] = t37;
    const R t38 = (STATES[0] + ((R)75.0000));
    const R t39 = (t38 * ((R)0x1.999999999999ap-7));
    const R t40 = M::fast_exp(t39);
    const R t41 = (((R)0.125000) * t40);
    ALG[7] = t41;
    const R t42 = (((R)1.00000) - STATES[3]);
    const R t43 = (t37 * t42);
    const R t44 = (t41 * STATES[3]);
    const R t45 = (t43 - t44);
    const R t46 = FDM_POW3(STATES[1]);
    const R t47 = (PARAMS[1] * t46);
    const R t48 = (t47 * STATES[2]);
    const R t49 = (STATES[0] - ((R)0x1.4000000000000p+5));
    const R t50 = (t48 * t49);
    ALG[0] = t50;
    const R t51 = FDM_POW4(STATES[3]);
    const R t52 = (PARAMS[2] * t51);
    const R t53 = (STATES[0] - ((R)-0x1.5c00000000000p+6));
    const R t54 = (t52 * t53);
    ALG[4] = t54;
    const R t55 = (STATES[0] - ((R)-0x1.018c49ba5e354p+6));
    const R t56 = (((R)0x1.3333333333333p-2) * t55);
    ALG[8] = t56;
    const R t57 = (-PARAMS[0]);
    const R t58 = (t57 + t50);
    const R t59 = (t58 + t54);
    const R t60 = (t59 + t56);
    const R t61 = (-t60);
    const R t62 = (t61 * ((R)0x1.0000000000000p+0));
    R a_t0 = (R)0;
    R a_t1 = (R)0;
    R a_t2 = (R)0;
    R a_t3 = (R)0;
    R a_t4 = (R)0;
    R a_t5 = (R)0;
    R a_t6 = (R)0;
    R a_t7 = (R)0;
    R a_t8 = (R)0;
    R a_t9 = (R)0;
    R a_t10 = (R)0;
    R a_t11 = (R)0;
    R a_t12 = (R)0;
    R a_t13 = (R)0;
    R a_t14 = (R)0;
    R a_t15 = (R)0;
    R a_t16 = (R)0;
    R a_t17 = (R)0;
    R a_t18 = (R)0;
    R a_t19 = (R)0;
    R a_t20 = (R)0;
    R a_t21 = (R)0;
    R a_t22 = (R)0;
    R a_t23 = (R)0;
    R a_t24 = (R)0;
    R a_t25 = (R)0;
    R a_t26 = (R)0;
    R a_t27 = (R)0;
    R a_t28 = (R)0;
    R a_t29 = (R)0;
    R a_t30 = (R)0;
    R a_t31 = (R)0;
    R a_t32 = (R)0;
    R a_t33 = (R)0;
    R a_t34 = (R)0;
    R a_t35 = (R)0;
    R a_t36 = (R)0;
    R a_t37 = (R)0;
    R a_t38 = (R)0;
    R a_t39 = (R)0;
    R a_t40 = (R)0;
    R a_t41 = (R)0;
    R a_t42 = (R)0;
    R a_t43 = (R)0;
    R a_t44 = (R)0;
    R a_t45 = (R)0;
    R a_t46 = (R)0;
    R a_t47 = (R)0;
    R a_t48 = (R)0;
    R a_t49 = (R)0;
    R a_t50 = (R)0;
    R a_t51 = (R)0;
    R a_t52 = (R)0;
    R a_t53 = (R)0;
    R a_t54 = (R)0;
    R a_t55 = (R)0;
    R a_t56 = (R)0;
    R a_t57 = (R)0;
    R a_t58 = (R)0;
    R a_t59 = (R)0;
    R a_t60 = (R)0;
    R a_t61 = (R)0;
    R a_t62 = (R)0;
    a_t62 += LAM_RATES[0];
    a_t17 += LAM_RATES[1];
    a_t30 += LAM_RATES[2];
    a_t45 += LAM_RATES[3];
    a_t61 += a_t62 * ((R)0x1.0000000000000p+0);
    a_t60 += -a_t61;
    a_t59 += a_t60;
    a_t56 += a_t60;
    a_t58 += a_t59;
    a_t54 += a_t59;
    a_t57 += a_t58;
    a_t50 += a_t58;
    LAM_PARAMS[0] += -a_t57;
    a_t55 += a_t56 * ((R)0x1.3333333333333p-2);
    LAM_STATES[0] += a_t55;
    a_t52 += a_t54 * t53;
    a_t53 += a_t54 * t52;
    LAM_STATES[0] += a_t53;
    LAM_PARAMS[2] += a_t52 * t51;
    a_t51 += a_t52 * PARAMS[2];
    LAM_STATES[3] += a_t51 * ((R)4 * FDM_POW3(STATES[3]));
    a_t48 += a_t50 * t49;
    a_t49 += a_t50 * t48;
    LAM_STATES[0] += a_t49;
    a_t47 += a_t48 * STATES[2];
    LAM_STATES[2] += a_t48 * t47;
    LAM_PARAMS[1] += a_t47 * t46;
    a_t46 += a_t47 * PARAMS[1];
    LAM_STATES[1] += a_t46 * ((R)3 * FDM_POW2(STATES[1]));
    a_t43 += a_t45;
    a_t44 += -a_t45;
    a_t41 += a_t44 * STATES[3];
    LAM_STATES[3] += a_t44 * t41;
    a_t37 += a_t43 * t42;
    a_t42 += a_t43 * t37;
    LAM_STATES[3] += -a_t42;
    a_t40 += a_t41 * ((R)0.125000);
    a_t39 += a_t40 * M::dexp(t39, t40);
    a_t38 += a_t39 * ((R)0x1.999999999999ap-7);
    LAM_STATES[0] += a_t38;
    a_t33 += a_t37 * t36;
    a_t36 += a_t37 * t33;
    a_t35 += -a_t36 * t36 * t36;
    a_t34 += a_t35;
    a_t4 += a_t34 * ((R)0x1.8a1e18a954ffap-10);
    a_t31 += a_t33 * t32;
    a_t32 += a_t33 * t31;
    LAM_STATES[0] += a_t32;
    a_t28 += a_t30;
    a_t29 += -a_t30;
    a_t26 += a_t29 * STATES[2];
    LAM_STATES[2] += a_t29 * t26;
    a_t22 += a_t28 * t27;
    a_t27 += a_t28 * t22;
    LAM_STATES[2] += -a_t27;
    a_t25 += a_t26 * ((R)1.00000);
    a_t24 += -a_t25 * t25 * t25;
    a_t23 += a_t24;
    a_t4 += a_t23 * ((R)0x1.6c0504695c417p-7);
    a_t21 += a_t22 * ((R)0.0700000);
    a_t20 += a_t21 * M::dexp(t20, t21);
    a_t19 += a_t20 * ((R)0x1.999999999999ap-5);
    a_t18 += -a_t19;
    LAM_STATES[0] += a_t18;
    a_t15 += a_t17;
    a_t16 += -a_t17;
    a_t13 += a_t16 * STATES[1];
    LAM_STATES[1] += a_t16 * t13;
    a_t8 += a_t15 * t14;
    a_t14 += a_t15 * t8;
    LAM_STATES[1] += -a_t14;
    a_t12 += a_t13 * ((R)4.00000);
    a_t11 += a_t12 * M::dexp(t11, t12);
    a_t10 += a_t11 * ((R)0x1.c71c71c71c71cp-5);
    a_t9 += -a_t10;
    LAM_STATES[0] += a_t9;
    a_t2 += a_t8 * t7;
    a_t7 += a_t8 * t2;
    a_t6 += -a_t7 * t7 * t7;
    a_t5 += a_t6;
    a_t4 += a_t5 * ((R)0x1.b993fe00d5376p-8);
    a_t3 += a_t4 * M::dexp(t3, t4);
    LAM_STATES[0] += a_t3 * ((R)-0x1.999999999999ap-4);
    a_t0 += a_t2 * t1;
    a_t1 += a_t2 * t0;
    LAM_STATES[0] += a_t1;
  }
  static constexpr int nTapeFast = 63;
  template<class R, class M>
  __device__ __forceinline__ static void rates_tape_fast(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, R* __restrict__ RATES, R* __restrict__ TAPE)
  {
    (void)VOI; (void)PARAMS;
    R ALG[9];
    (void)ALG;
    const R t0 = (-((R)0.100000));
    TAPE[0] = t0;
    const R t1 = (STATES[0] + ((R)50.0000));
    TAPE[1] = t1;
    const R t2 = (t0 * t1);
    TAPE[2] = t2;
    const R t3 = (((R)-0x1.999999999999ap-4) * STATES[0]);
    TAPE[3] = t3;
    const R t4 = M::fast_exp(t3);
    TAPE[4] = t4;
    const R t5 = (t4 * ((R)0x1.b993fe00d5376p-8));
    TAPE[5] = t5;
    const R t6 = (t5 - ((R)1.00000));
    TAPE[6] = t6;
    const R t7 = M::fast_rcp(t6);
    TAPE[7] = t7;
    const R t8 = (t2 * t7);
    TAPE[8] = t8;
    ALG[1] = t8;
    const R t9 = (STATES[0] + ((R)75.0000));
    TAPE[9] = t9;
    const R t10 = (-t9);
    TAPE[10] = t10;
    const R t11 = (t10 * ((R)0x1.c71c71c71c71cp-5));
    TAPE[11] = t11;
    const R t12 = M::fast_exp(t11);
    TAPE[12] = t12;
    const R t13 = (((R)4.00000) * t12);
    TAPE[13] = t13;
    ALG[5] = t13;
    const R t14 = (((R)1.00000) - STATES[1]);
    TAPE[14] = t14;
    const R t15 = (t8 * t14);
    TAPE[15] = t15;
    const R t16 = (t13 * STATES[1]);
    TAPE[16] = t16;
    const R t17 = (t15 - t16);
    TAPE[17] = t17;
    const R t18 = (STATES[0] + ((R)75.0000));
    TAPE[18] = t18;
    const R t19 = (-t18);
    TAPE[19] = t19;
    const R t20 = (t19 * ((R)0x1.999999999999ap-5));
    TAPE[20] = t20;
    const R t21 = M::fast_exp(t20);
    TAPE[21] = t21;
    const R t22 = (((R)0.0700000) * t21);
    TAPE[22] = t22;
    ALG[2] = t22;
    const R t23 = (t4 * ((R)0x1.6c0504695c417p-7));
    TAPE[23] = t23;
    const R t24 = (t23 + ((R)1.00000));
    TAPE[24] = t24;
    const R t25 = M::fast_rcp(t24);
    TAPE[25] = t25;
    const R t26 = (((R)1.00000) * t25);
    TAPE[26] = t26;
    ALG[6] = t26;
    const R t27 = (((R)1.00000) - STATES[2]);
    TAPE[27] = t27;
    const R t28 = (t22 * t27);
    TAPE[28] = t28;
    const R t29 = (t26 * STATES[2]);
    TAPE[29] = t29;
    const R t30 = (t28 - t29);
    TAPE[30] = t30;
    const R t31 = (-((R)0.0100000));
    TAPE[31] = t31;
    const R t32 = (STATES[0] + ((R)65.0000));
    TAPE[32] = t32;
    const R t33 = (t31 * t32);
    TAPE[33] = t33;
    const R t34 = (t4 * ((R)0x1.8a1e18a954ffap-10));
    TAPE[34] = t34;
    const R t35 = (t34 - ((R)1.00000));
    TAPE[35] = t35;
    const R t36 = M::fast_rcp(t35);
    TAPE[36] = t36;
    const R t37 = (t33 * t36);
    TAPE[37] = t37;
    ALG[3] = t37;
    const R t38 = (STATES[0] + ((R)75.0000));
    TAPE[38] = t38;
    const R t39 = (t38 * ((R)0x1.999999999999ap-7));
    TAPE[39] = t39;
    const R t40 = M::fast_exp(t39);
    TAPE[40] = t40;
    const R t41 = (((R)0.125000) * t40);
    TAPE[41] = t41;
    ALG[7] = t41;
    const R t42 = (((R)1.00000) - STATES[3]);
    TAPE[42] = t42;
    const R t43 = (t37 * t42);
    TAPE[43] = t43;
    const R t44 = (t41 * STATES[3]);
    TAPE[44] = t44;
    const R t45 = (t43 - t44);
    TAPE[45] = t45;
    const R t46 = FDM_POW3(STATES[1]);
    TAPE[46] = t46;
    const R t47 = (PARAMS[1] * t46);
    TAPE[47] = t47;
    const R t48 = (t47 * STATES[2]);
    TAPE[48] = t48;
    const R t49 = (STATES[0] - ((R)0x1.4000000000000p+5));
    TAPE[49] = t49;
    const R t50 = (t48 * t49);
    TAPE[50] = t50;
    ALG[0] = t50;
    const R t51 = FDM_POW4(STATES[3]);
    TAPE[51] = t51;
    const R t52 = (PARAMS[2] * t51);
    TAPE[52] = t52;
    const R t53 = (STATES[0] - ((R)-0x1.5c00000000000p+6));
    TAPE[53] = t53;
    const R t54 = (t52 * t53);
    TAPE[54] = t54;
    ALG[4] = t54;
    const R t55 = (STATES[0] - ((R)-0x1.018c49ba5e354p+6));
    TAPE[55] = t55;
    const R t56 = (((R)0x1.3333333333333p-2) * t55);
    TAPE[56] = t56;
    ALG[8] = t56;
    const R t57 = (-PARAMS[0]);
    TAPE[57] = t57;
    const R t58 = (t57 + t50);
    TAPE[58] = t58;
    const R t59 = (t58 + t54);
    TAPE[59] = t59;
    const R t60 = (t59 + t56);
    TAPE[60] = t60;
    const R t61 = (-t60);
    TAPE[61] = t61;
    const R t62 = (t61 * ((R)0x1.0000000000000p+0));
    TAPE[62] = t62;
    RATES[0] = t62;
    RATES[1] = t17;
    RATES[2] = t30;
    RATES[3] = t45;
  }
  template<class R, class M>
  __device__ __forceinline__ static void rates_vjp_tape_fast(const R VOI, const R* __restrict__ STATES, const R* __restrict__ PARAMS, const R* __restrict__ TAPE, const R* __restrict__ LAM_RATES, R* __restrict__ LAM_STATES, R* __restrict__ LAM_PARAMS)
  {
    (void)VOI; (void)PARAMS; (void)STATES;
    const R t0 = TAPE[0];
    const R t1 = TAPE[1];
    const R t2 = TAPE[2];
    const R t3 = TAPE[3];
    const R t4 = TAPE[4];
    const R t5 = TAPE[5];
    const R t6 = TAPE[6];
    const R t7 = TAPE[7];
    const R t8 = TAPE[8];
    const R t9 = TAPE[9];
    const R t10 = TAPE[10];
    const R t11 = TAPE[11];
    const R t12 = TAPE[12];
    const R t13 = TAPE[13];
    const R t14 = TAPE[14];
    const R t15 = TAPE[15];
    const R t16 = TAPE[16];
    const R t17 = TAPE[17];
    const R t18 = TAPE[18];
    const R t19 = TAPE[19];
    const R t20 = TAPE[20];
    const R t21 = TAPE[21];
    const R t22 = TAPE[22];
    const R t23 = TAPE[23];
    const R t24 = TAPE[24];
    const R t25 = TAPE[25];
    const R t26 = TAPE[26];
    const R t27 = TAPE[27];
    const R t28 = TAPE[28];
    const R t29 = TAPE[29];
    const R t30 = TAPE[30];
    const R t31 = TAPE[31];
    const R t32 = TAPE[32];
    const R t33 = TAPE[33];
    const R t34 = TAPE[34];
    const R t35 = TAPE[35];
    const R t36 = TAPE[36];
    const R t37 = TAPE[37];
    const R t38 = TAPE[38];
    const R t39 = TAPE[39];
    const R t40 = TAPE[40];
    const R t41 = TAPE[41];
    const R t42 = TAPE[42];
    const R t43 = TAPE[43];
    const R t44 = TAPE[44];
    const R t45 = TAPE[45];
    const R t46 = TAPE[46];
    const R t47 = TAPE[47];
    const R t48 = TAPE[48];
    const R t49 = TAPE[49];
    const R t50 = TAPE[50];
    const R t51 = TAPE[51];
    const R t52 = TAPE[52];
    const R t53 = TAPE[53];
    const R t54 = TAPE[54];
    const R t55 = TAPE[55];
    const R t56 = TAPE[56];
    const R t57 = TAPE[57];
    const R t58 = TAPE[58];
    const R t59 = TAPE[59];
    const R t60 = TAPE[60];
    const R t61 = TAPE[61];
    const R t62 = TAPE[62];
    R a_t0 = (R)0;
    R a_t1 = (R)0;
    R a_t2 = (R)0;
    R a_t3 = (R)0;
    R a_t4 = (R)0;
    R a_t5 = (R)0;
    R a_t6 = (R)0;
    R a_t7 = (R)0;
    R a_t8 = (R)0;
    R a_t9 = (R)0;
    R a_t10 = (R)0;
    R a_t11 = (R)0;
    R a_t12 = (R)0;
    R a_t13 = (R)0;
    R a_t14 = (R)0;
    R a_t15 = (R)0;
    R a_t16 = (R)0;
    R a_t17 = (R)0;
    R a_t18 = (R)0;
    R a_t19 = (R)0;
    R a_t20 = (R)0;
    R a_t21 = (R)0;
    R a_t22 = (R)0;
    R a_t23 = (R)0;
    R a_t24 = (R)0;
    R a_t25 = (R)0;
    R a_t26 = (R)0;
    R a_t27 = (R)0;
    R a_t28 = (R)0;
    R a_t29 = (R)0;
    R a_t30 = (R)0;
    R a_t31 = (R)0;
    R a_t32 = (R)0;
    R a_t33 = (R)0;
    R a_t34 = (R)0;
    R a_t35 = (R)0;
    R a_t36 = (R)0;
    R a_t37 = (R)0;
    R a_t38 = (R)0;
    R a_t39 = (R)0;
    R a_t40 = (R)0;
    R a_t41 = (R)0;
    R a_t42 = (R)0;
    R a_t43 = (R)0;
    R a_t44 = (R)0;
    R a_t45 = (R)0;
    R a_t46 = (R)0;
    R a_t47 = (R)0;
    R a_t48 = (R)0;
    R a_t49 = (R)0;
    R a_t50 = (R)0;
    R a_t51 = (R)0;
    R a_t52 = (R)0;
    R a_t53 = (R)0;
    R a_t54 = (R)0;
    R a_t55 = (R)0;
    R a_t56 = (R)0;
    R a_t57 = (R)0;
    R a_t58 = (R)0;
    R a_t59 = (R)0;
    R a_t60 = (R)0;
    R a_t61 = (R)0;
    R a_t62 = (R)0;
    a_t62 += LAM_RATES[0];
    a_t17 += LAM_RATES[1];
    a_t30 += LAM_RATES[2];
    a_t45 += LAM_RATES[3];
    a_t61 += a_t62 * ((R)0x1.0000000000000p+0);
    a_t60 += -a_t61;
    a_t59 += a_t60;
    a_t56 += a_t60;
    a_t58 += a_t59;
    a_t54 += a_t59;
    a_t57 += a_t58;
    a_t50 += a_t58;
    LAM_PARAMS[0] += -a_t57;
    a_t55 += a_t56 * ((R)0x1.3333333333333p-2);
    LAM_STATES[0] += a_t55;
    a_t52 += a_t54 * t53;
    a_t53 += a_t54 * t52;
    LAM_STATES[0] += a_t53;
    LAM_PARAMS[2] += a_t52 * t51;
    a_t51 += a_t52 * PARAMS[2];
    LAM_STATES[3] += a_t51 * ((R)4 * FDM_POW3(STATES[3]));
    a_t48 += a_t50 * t49;
    a_t49 += a_t50 * t48;
    LAM_STATES[0] += a_t49;
    a_t47 += a_t48 * STATES[2];
    LAM_STATES[2] += a_t48 * t47;
    LAM_PARAMS[1] += a_t47 * t46;
    a_t46 += a_t47 * PARAMS[1];
    LAM_STATES[1] += a_t46 * ((R)3 * FDM_POW2(STATES[1]));
    a_t43 += a_t45;
    a_t44 += -a_t45;
    a_t41 += a_t44 * STATES[3];
    LAM_STATES[3] += a_t44 * t41;
    a_t37 += a_t43 * t42;
    a_t42 += a_t43 * t37;
    LAM_STATES[3] += -a_t42;
    a_t40 += a_t41 * ((R)0.125000);
    a_t39 += a_t40 * M::dexp(t39, t40);
    a_t38 += a_t39 * ((R)0x1.999999999999ap-7);
    LAM_STATES[0] += a_t38;
    a_t33 += a_t37 * t36;
    a_t36 += a_t37 * t33;
    a_t35 += -a_t36 * t36 * t36;
    a_t34 += a_t35;
    a_t4 += a_t34 * ((R)0x1.8a1e18a954ffap-10);
    a_t31 += a_t33 * t32;
    a_t32 += a_t33 * t31;
    LAM_STATES[0] += a_t32;
    a_t28 += a_t30;
    a_t29 += -a_t30;
    a_t26 += a_t29 * STATES[2];
    LAM_STATES[2] += a_t29 * t26;
    a_t22 += a_t28 * t27;
    a_t27 += a_t28 * t22;
    LAM_STATES[2] += -a_t27;
    a_t25 += a_t26 * ((R)1.00000);
    a_t24 += -a_t25 * t25 * t25;
    a_t23 += a_t24;
    a_t4 += a_t23 * ((R)0x1.6c0504695c417p-7);
    a_t21 += a_t22 * ((R)0.0700000);
    a_t20 += a_t21 * M::dexp(t20, t21);
    a_t19 += a_t20 * ((R)0x1.999999999999ap-5);
    a_t18 += -a_t19;
    LAM_STATES[0] += a_t18;
    a_t15 += a_t17;
    a_t16 += -a_t17;
    a_t13 += a_t16 * STATES[1];
    LAM_STATES[1] += a_t16 * t13;
    a_t8 += a_t15 * t14;
    a_t14 += a_t15 * t8;
    LAM_STATES[1] += -a_t14;
    a_t12 += a_t13 * ((R)4.00000);
    a_t11 += a_t12 * M::dexp(t11, t12);
    a_t10 += a_t11 * ((R)0x1.c71c71c71c71cp-5);
    a_t9 += -a_t10;
    LAM_STATES[0] += a_t9;
    a_t2 += a_t8 * t7;
    a_t7 += a_t8 * t2;
    a_t6 += -a_t7 * t7 * t7;
    a_t5 += a_t6;
    a_t4 += a_t5 * ((R)0x1.b993fe00d5376p-8);
    a_t3 += a_t4 * M::dexp(t3, t4);
    LAM_STATES[0] += a_t3 * ((R)-0x1.999999999999ap-4);
    a_t0 += a_t2 * t1;
    a_t1 += a_t2 * t0;
    LAM_STATES[0] += a_t1;
  }
#undef FDM_POW2
#undef FDM_POW3
#undef FDM_POW4
};
