// The FP64 arithmetic of the right-hand sides on host arrays, for tests: the functions of fdm_math.cuh, and the right-hand
// side of a model as the kernels evaluate it.  test_model.cuh: the generated model, TEST_MODEL its name, TEST_SCALE and
// TEST_OFFSET the constants of exp(-x/10 - 3/2).
#include "fdm_kernels.cuh"
#include "test_model.cuh"

namespace {

__global__ void function_kernel(int f, int64_t n, const double* x, const double* y, double* out)
{
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  switch (f) {
  case 0: out[i] = fdm_math_exact::fast_exp(x[i]); break;
  case 1: out[i] = fdm_math_exact::fast_rcp(x[i]); break;
  case 2: out[i] = fdm_math_exact::fast_div(x[i], y[i]); break;
  case 11: out[i] = fdm_math_exact::fast_div_any(x[i], y[i]); break;
  case 3: out[i] = fdm_math_exact::fast_expm1(x[i]); break;
  case 4: out[i] = fdm_math_exact::fast_exp(x[i], TEST_SCALE); break;
  case 5: out[i] = fdm_math_exact::fast_expm1(x[i], TEST_SCALE); break;
  case 6: out[i] = fdm_math_exact::fast_exp_sat(x[i]); break;
  case 7: out[i] = fdm_exp_group(x[i], TEST_SCALE).exp(TEST_OFFSET); break;
  case 8: out[i] = fdm_exp_group(x[i], TEST_SCALE).expm1(TEST_OFFSET); break;
  case 9: out[i] = fdm_exp_group(x[i], TEST_SCALE).exp(); break;
  case 10: out[i] = fdm_exp_group(x[i], TEST_SCALE).expm1(); break;
  }
}

template<class Math>
__global__ void rates_kernel(int64_t n, double t, const double* states, const double* params, double* rates)
{
  using M = TEST_MODEL;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  double y[M::nStates], p[M::nParameters > 0 ? M::nParameters : 1], r[M::nStates], alg[M::nAlgebraics];
  for (int s = 0; s < M::nStates; s++)
    y[s] = states[s * n + i];
  for (int q = 0; q < M::nParameters; q++)
    p[q] = params[q * n + i];
  fdm::model_rates<M, double, Math>(t, y, p, r, alg);
  for (int s = 0; s < M::nStates; s++)
    rates[s * n + i] = r[s];
}

// device copy of a host array, freed at the end of the call
struct Array {
  double* d = nullptr;
  double* host;
  size_t bytes;
  Array(const double* h, int64_t n) : host((double*)h), bytes(sizeof(double) * (size_t)(n > 0 ? n : 1))
  {
    if (cudaMalloc((void**)&d, bytes) == cudaSuccess && host)
      cudaMemcpy(d, host, bytes, cudaMemcpyHostToDevice);
  }
  ~Array() { cudaFree(d); }
};

} // namespace

extern "C" int eval_function(int f, int64_t n, const double* x, const double* y, double* out)
{
  Array X(x, n), Y(y, n), O(out, n);
  if (!X.d || !Y.d || !O.d)
    return 1;
  function_kernel<<<(unsigned)((n + 255) / 256), 256>>>(f, n, X.d, Y.d, O.d);
  return (int)cudaMemcpy(out, O.d, O.bytes, cudaMemcpyDeviceToHost);
}

extern "C" int eval_rates(int approximate, int64_t n, double t, const double* states, const double* params, double* rates)
{
  using M = TEST_MODEL;
  Array S(states, n * M::nStates), P(params, n * M::nParameters), R(rates, n * M::nStates);
  if (!S.d || !P.d || !R.d)
    return 1;
  const unsigned blocks = (unsigned)((n + 127) / 128);
  if (approximate)
    rates_kernel<fdm_math_approx><<<blocks, 128>>>(n, t, S.d, P.d, R.d);
  else
    rates_kernel<fdm_math_exact><<<blocks, 128>>>(n, t, S.d, P.d, R.d);
  return (int)cudaMemcpy(rates, R.d, R.bytes, cudaMemcpyDeviceToHost);
}
