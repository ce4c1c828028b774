// Split-path kernels (reaction, diffusion, stimulation schedule) and the model table.
#define FDM_COMMON_KERNELS_TU
#include <algorithm>
#include <atomic>
#include <mutex>

#include "fdm_internal.h"
#include "fdm_diffusion.cuh"
#include "fdm_equilibrium.cuh"
#include "fdm_model_launch.cuh"

#include "generated/hodgkin_huxley_1952_anone_c2_3_4.cuh"
#include "generated/shorten_ocallaghan_davidson_soboleva_2007_a32_c65.cuh"

namespace fdm {

using HH = fdm_model_hodgkin_huxley_1952_anone_c2_3_4;
using SH = fdm_model_shorten_ocallaghan_davidson_soboleva_2007_a32_c65;

static const ModelDesc g_models[] = {
  {HH::name, HH::nStates, HH::nAlgebraics, HH::nParameters, HH::statesInitialValues, HH::parameterDefaults, true},
  {SH::name, SH::nStates, SH::nAlgebraics, SH::nParameters, SH::statesInitialValues, SH::parameterDefaults, false},
};

constexpr int kBuiltinModels = (int)(sizeof(g_models) / sizeof(g_models[0]));
constexpr int kMaxModules = 64;

// run-time model modules, appended by register_model_module and never removed (their libraries stay loaded)
static ModelModule g_modules[kMaxModules];
static std::atomic<int> g_n_modules{0};
static std::mutex g_modules_mu;

int n_models() { return kBuiltinModels + g_n_modules.load(std::memory_order_acquire); }

static const ModelModule* module_of(int model)
{
  const int k = model - kBuiltinModels;
  return (k >= 0 && k < g_n_modules.load(std::memory_order_acquire)) ? &g_modules[k] : nullptr;
}

const ModelDesc* model_desc(int model)
{
  if (model >= 0 && model < kBuiltinModels)
    return &g_models[model];
  const ModelModule* m = module_of(model);
  return m ? &m->desc : nullptr;
}

int register_model_module(const ModelModule& m)
{
  std::lock_guard<std::mutex> lock(g_modules_mu);
  const int k = g_n_modules.load(std::memory_order_relaxed);
  if (k >= kMaxModules || m.abi != FDM_MODEL_MODULE_ABI)
    return -1;
  g_modules[k] = m;
  g_modules[k].desc.fused_supported = false;   // modules carry the split-path, equilibrium and adjoint kernels
  g_n_modules.store(k + 1, std::memory_order_release);
  return kBuiltinModels + k;
}

cudaError_t launch_reaction(int model, RealKind rk, MathKind mk, const ReactionArgs& a, cudaStream_t s)
{
  switch (model) {
  case 0: return reaction_model<HH>(rk, mk, a, s);
  case 1: return reaction_model<SH>(rk, mk, a, s);
  default: {
    const ModelModule* m = module_of(model);
    return m ? m->reaction(rk, mk, a, s) : cudaErrorInvalidValue;
  }
  }
}

cudaError_t launch_cellml_rhs(int model, MathKind mk, int64_t n, double t, const double* states, const double* params,
                              double* rates, double* algebraics, cudaStream_t s)
{
  if (n == 0)
    return cudaSuccess;
  switch (model) {
  case 0: return cellml_rhs_model<HH>(mk, n, t, states, params, rates, algebraics, s);
  case 1: return cellml_rhs_model<SH>(mk, n, t, states, params, rates, algebraics, s);
  default: {
    const ModelModule* m = module_of(model);
    return m ? m->cellml_rhs(mk, n, t, states, params, rates, algebraics, s) : cudaErrorInvalidValue;
  }
  }
}

cudaError_t launch_equilibrium_search(int model, MathKind mk, double* u, const double* u0, const double* params,
                               EquilibriumSearch* es, int64_t max_iterations, cudaStream_t s)
{
  switch (model) {
  case 0: return equilibrium_search_model<HH>(mk, u, u0, params, es, max_iterations, s);
  case 1: return equilibrium_search_model<SH>(mk, u, u0, params, es, max_iterations, s);
  default: {
    const ModelModule* m = module_of(model);
    return m ? m->equilibrium_search(mk, u, u0, params, es, max_iterations, s) : cudaErrorInvalidValue;
  }
  }
}

cudaError_t launch_schedule(const StimArgs& a, const SplitStep* steps, int n_steps, cudaStream_t s)
{
  if (a.n_fibers == 0)
    return cudaSuccess;
  const int fibers = SCHEDULE_T / 32;   // a warp per fiber
  stimulation_schedule_kernel<<<(a.n_fibers + fibers - 1) / fibers, SCHEDULE_T, 0, s>>>(a, steps, n_steps);
  return cudaGetLastError();
}

template<int WHAT>
static cudaError_t factor_launch(int n_fibers, int tile, const int64_t* fiber_offsets, const double* element_lengths,
                                 const double* prefactor, double dt, int implicit_euler, double* coef, int64_t stride,
                                 double* vm, double* scratch, cudaStream_t s)
{
  if (n_fibers == 0)
    return cudaSuccess;
  // the limit is the largest tile's, whatever this launch asks for: other solvers of the device, in other host threads,
  // launch the kernel with tiles of their own
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = set_smem_once(diffusion_factor_kernel<WHAT>, factor_smem_bytes(FACTOR_TILE), attr_done);
  if (e != cudaSuccess)
    return e;
  diffusion_factor_kernel<WHAT><<<(unsigned)n_fibers, FACTOR_T, factor_smem_bytes(tile), s>>>(
      fiber_offsets, element_lengths, prefactor, dt, implicit_euler, coef, stride, vm, scratch, tile);
  return cudaGetLastError();
}

cudaError_t launch_coefficients(int n_fibers, const int64_t* fiber_offsets, const double* element_lengths,
                                const double* prefactor, double dt, int implicit_euler, double* coef, int64_t stride,
                                int64_t max_fiber_len, cudaStream_t s)
{
  // shared memory for the longest fiber only: more CTAs per SM
  const int tile = (int)std::min<int64_t>(FACTOR_TILE, std::max<int64_t>(max_fiber_len, 1));
  return factor_launch<FACTOR>(n_fibers, tile, fiber_offsets, element_lengths, prefactor, dt, implicit_euler, coef,
                               stride, nullptr, nullptr, s);
}

cudaError_t launch_diffusion_operator(int n_fibers, int64_t n_nodes, const int64_t* fiber_offsets,
                                      const double* element_lengths, const double* prefactor, double dt,
                                      int implicit_euler, double* vm, double* scratch, cudaStream_t s)
{
  return factor_launch<FACTOR_SOLVE>(n_fibers, FACTOR_TILE, fiber_offsets, element_lengths, prefactor, dt,
                                     implicit_euler, nullptr, n_nodes, vm, scratch, s);
}

__global__ void __launch_bounds__(256) states_to_pairs_kernel(const double* __restrict__ x, float* __restrict__ hi,
                                                              float* __restrict__ lo, int64_t n)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = x[i];
    const float h = __double2float_rn(v);
    hi[i] = h;
    lo[i] = __double2float_rn(__dsub_rn(v, (double)h));
  }
}

__global__ void __launch_bounds__(256) pairs_to_states_kernel(const float* __restrict__ hi,
                                                              const float* __restrict__ lo, double* __restrict__ x,
                                                              int64_t n)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = __dadd_rn((double)hi[i], (double)lo[i]);
}

static unsigned elementwise_blocks(int64_t n)
{
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16));
}

cudaError_t launch_states_to_pairs(const double* x, float* hi, float* lo, int64_t n, cudaStream_t s)
{
  if (n <= 0)
    return cudaSuccess;
  states_to_pairs_kernel<<<elementwise_blocks(n), 256, 0, s>>>(x, hi, lo, n);
  return cudaGetLastError();
}

cudaError_t launch_pairs_to_states(const float* hi, const float* lo, double* x, int64_t n, cudaStream_t s)
{
  if (n <= 0)
    return cudaSuccess;
  pairs_to_states_kernel<<<elementwise_blocks(n), 256, 0, s>>>(hi, lo, x, n);
  return cudaGetLastError();
}

// from this many fibers on a warp per fiber can fill the GPU (four warps on each of 148 SMs): launch_diffusion takes it
// for short fibers and for fibers too long for registers, launch_adjoint_diffusion for all
constexpr int DIFFUSION_BLOCK_MAX_FIBERS = 4 * 148;

template<int M>
static cudaError_t diffusion_reg_launch(int n_fibers, const int64_t* fiber_offsets, const double* coef, int64_t stride,
                                        double* vm, cudaStream_t s, const int* eq_counter, const int* eq_nbuf,
                                        int n_ranks)
{
  diffusion_reg_kernel<M><<<(unsigned)n_fibers, DIFFUSION_T, 0, s>>>(fiber_offsets, coef, stride, vm, eq_counter,
                                                                     eq_nbuf, n_ranks);
  return cudaGetLastError();
}

cudaError_t launch_diffusion(int n_fibers, const int64_t* fiber_offsets, const double* coef, int64_t stride,
                                  double* vm, double* scratch, int64_t max_fiber_len, cudaStream_t s,
                                  const int* eq_counter, const int* eq_nbuf, int n_ranks)
{
  if (n_fibers == 0)
    return cudaSuccess;
  const int nr = n_ranks > 0 ? n_ranks : 1;
  // many short fibers: a warp per fiber, as half of a CTA's threads would have no node (4096 fibers: of 100 nodes
  // 12.5 us against 18.5 us with a CTA each, of 200 nodes 20.6 against 18.5; 592 fibers of 100 nodes: 6.2 us both)
  const bool many = n_fibers >= DIFFUSION_BLOCK_MAX_FIBERS;
  if (!(many && max_fiber_len <= DIFFUSION_T / 2)) {
    switch ((max_fiber_len + 2 * DIFFUSION_T - 1) / (2 * DIFFUSION_T)) {
    case 1: return diffusion_reg_launch<2>(n_fibers, fiber_offsets, coef, stride, vm, s, eq_counter, eq_nbuf, nr);
    case 2: return diffusion_reg_launch<4>(n_fibers, fiber_offsets, coef, stride, vm, s, eq_counter, eq_nbuf, nr);
    case 3: return diffusion_reg_launch<6>(n_fibers, fiber_offsets, coef, stride, vm, s, eq_counter, eq_nbuf, nr);
    case 4: return diffusion_reg_launch<8>(n_fibers, fiber_offsets, coef, stride, vm, s, eq_counter, eq_nbuf, nr);
    case 5: return diffusion_reg_launch<10>(n_fibers, fiber_offsets, coef, stride, vm, s, eq_counter, eq_nbuf, nr);
    default: break;
    }
  }
  if (!many) {
    // fibers too long for registers
    diffusion_block_kernel<256><<<(unsigned)n_fibers, 256, 0, s>>>(fiber_offsets, coef, stride, vm, scratch,
                                                                   eq_counter, eq_nbuf, nr);
    return cudaGetLastError();
  }
  const int T = 128;
  const int64_t threads = (int64_t)n_fibers * 32;
  diffusion_warp_kernel<<<(unsigned)((threads + T - 1) / T), T, 0, s>>>(n_fibers, fiber_offsets, coef, stride, vm,
                                                                        scratch, eq_counter, eq_nbuf, nr);
  return cudaGetLastError();
}

// Clusters stay within a group of SMs that share a network port, and the groups' sizes differ: on a B200 there is room
// for 15 clusters of 8 CTAs, 22 of 6, 26 of 5, 33 of 4, 45 of 3, 74 of 2 with an SM for every CTA (the shared memory
// asked for leaves none for a second one).
__global__ void own_sm_probe_kernel()
{
}

int clusters_with_own_sms(int csize)
{
  constexpr int HALF_SM = 120 * 1024;
  int n = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)csize);
  cfg.blockDim = dim3(WINDOW_T);
  cfg.dynamicSmemBytes = HALF_SM;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(own_sm_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, HALF_SM) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, own_sm_probe_kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// The few fibers a window kernel is for: a CTA for at most WINDOW_T nodes and an SM for every CTA; the most CTAs per
// fiber (at most 8, down to 128 nodes each) with which that holds.  Where CTAs share an SM, the launches cost less than that:
// per step of 5 substeps a half step 16 fibers of 1481 nodes take 12.6 us with clusters of 6, 24.3 with clusters of 8
// (one more than fit) and 15.1 with a launch per half step and solve; 24 fibers 24.4 with clusters of 6 (22 fit) and
// 15.6.
int window_cluster_size(int model, int n_fibers, int64_t max_fiber_len)
{
  const int least = (int)std::min<int64_t>((max_fiber_len + WINDOW_T - 1) / WINDOW_T, FDM_MAX_CLUSTER + 1);
  const int most = (int)std::min<int64_t>((max_fiber_len + 127) / 128, FDM_MAX_CLUSTER);
  if (model != 0 || n_fibers < 1)
    return 0;
  for (int c = most; c >= std::max(least, 1); c--)
    if (clusters_with_own_sms(c) >= n_fibers)
      return c;
  return 0;
}

template<class Math, int M>
static cudaError_t window_launch(const ReactionArgs& a, int n_fibers, int csize, const int64_t* fiber_offsets,
                                 const double* coef, int n_steps, cudaStream_t s)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n_fibers * csize));
  cfg.blockDim = dim3(WINDOW_T);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, window_cluster_kernel<HH, Math, M>, a, fiber_offsets, coef, n_steps);
}

template<class Math>
static cudaError_t window_shape(const ReactionArgs& a, int n_fibers, int csize, int64_t max_fiber_len,
                                const int64_t* fiber_offsets, const double* coef, int n_steps, cudaStream_t s)
{
  switch ((max_fiber_len + 2 * WINDOW_T - 1) / (2 * WINDOW_T)) {
  case 1: return window_launch<Math, 2>(a, n_fibers, csize, fiber_offsets, coef, n_steps, s);
  case 2: return window_launch<Math, 4>(a, n_fibers, csize, fiber_offsets, coef, n_steps, s);
  case 3: return window_launch<Math, 6>(a, n_fibers, csize, fiber_offsets, coef, n_steps, s);
  case 4: return window_launch<Math, 8>(a, n_fibers, csize, fiber_offsets, coef, n_steps, s);
  default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_window(int model, MathKind mk, const ReactionArgs& a, int n_fibers, int csize, int64_t max_fiber_len,
                          const int64_t* fiber_offsets, const double* coef, int n_steps, cudaStream_t s)
{
  if (model != 0 || csize < 1)
    return cudaErrorInvalidValue;
  return mk == MATH_EXACT
             ? window_shape<fdm_math_exact>(a, n_fibers, csize, max_fiber_len, fiber_offsets, coef, n_steps, s)
             : window_shape<fdm_math_approx>(a, n_fibers, csize, max_fiber_len, fiber_offsets, coef, n_steps, s);
}

// ---- equilibrium skip ----
cudaError_t launch_equilibrium_half(int model, RealKind rk, MathKind mk, const ReactionArgs& a, const EqLayout& L,
                                    const EqSpec& e, int n_states, int* n_launches, cudaStream_t s)
{
  cudaError_t ce = cudaSuccess;
  switch (model) {
  case 0: ce = reaction_eq_model<HH>(rk, mk, a, L, e, s); break;
  case 1: ce = reaction_eq_model<SH>(rk, mk, a, L, e, s); break;
  default: {
    const ModelModule* m = module_of(model);
    if (!m)
      return cudaErrorInvalidValue;
    ce = m->reaction_eq(rk, mk, a, L, e, s);
  }
  }
  if (ce != cudaSuccess || L.n_buffers == 0)
    return ce;
  *n_launches += 2;
  if (!L.in_warp) {
    const int T = 128;
    const unsigned bb = (unsigned)((L.n_buffers + T - 1) / T);
    if (rk == REAL_F64)
      eq_changed_kernel<double><<<bb, T, 0, s>>>(a, L, e, n_states);
    else
      eq_changed_kernel<float><<<bb, T, 0, s>>>(a, L, e, n_states);
    eq_scan_block_kernel<<<(unsigned)((L.n_buffers + EQ_SCAN_T - 1) / EQ_SCAN_T), EQ_SCAN_T, 0, s>>>(L);
    *n_launches += 2;
  }
  const unsigned blocks = (unsigned)((L.n_buffers * L.W + EQ_T - 1) / EQ_T);
  if (rk == REAL_F64)
    eq_commit_kernel<double><<<blocks, EQ_T, 0, s>>>(a, L, e, n_states);
  else
    eq_commit_kernel<float><<<blocks, EQ_T, 0, s>>>(a, L, e, n_states);
  return cudaGetLastError();
}

cudaError_t launch_adjoint_half(int model, MathKind mk, const AdjointArgs& a, cudaStream_t s)
{
  switch (model) {
  case 0: return adjoint_model<HH>(mk, a, s);
  case 1: return adjoint_model<SH>(mk, a, s);
  default: {
    const ModelModule* m = module_of(model);
    return m ? m->adjoint_half(mk, a, s) : cudaErrorInvalidValue;
  }
  }
}

template<int T, int M>
static cudaError_t adjoint_diffusion_block(int n_fibers, const int64_t* fiber_offsets, const double* element_lengths,
                                           const double* coef, int64_t stride, double* lam, const double* u,
                                           const double* x, int implicit_euler, double* grad_prefactor,
                                           cudaStream_t s)
{
  adjoint_diffusion_block_kernel<T, M><<<(unsigned)n_fibers, T, 0, s>>>(fiber_offsets, element_lengths, coef, stride,
                                                                       lam, u, x, implicit_euler, grad_prefactor);
  return cudaGetLastError();
}

cudaError_t launch_adjoint_diffusion(int n_fibers, const int64_t* fiber_offsets, const double* element_lengths,
                                     const double* coef, int64_t stride, double* lam, const double* u, const double* x,
                                     int implicit_euler, double* grad_prefactor, double* scratch, double* mu,
                                     int64_t max_fiber_len, cudaStream_t s)
{
  if (n_fibers == 0)
    return cudaSuccess;
  // few fibers: one CTA per fiber (block-wide scans); many fibers: one warp per fiber fills the GPU
  if (n_fibers < DIFFUSION_BLOCK_MAX_FIBERS) {
    if (max_fiber_len <= 512)
      return adjoint_diffusion_block<128, 4>(n_fibers, fiber_offsets, element_lengths, coef, stride, lam, u, x,
                                             implicit_euler, grad_prefactor, s);
    if (max_fiber_len <= 1024)
      return adjoint_diffusion_block<256, 4>(n_fibers, fiber_offsets, element_lengths, coef, stride, lam, u, x,
                                             implicit_euler, grad_prefactor, s);
    if (max_fiber_len <= 1536)
      return adjoint_diffusion_block<256, 6>(n_fibers, fiber_offsets, element_lengths, coef, stride, lam, u, x,
                                             implicit_euler, grad_prefactor, s);
    if (max_fiber_len <= 2048)
      return adjoint_diffusion_block<256, 8>(n_fibers, fiber_offsets, element_lengths, coef, stride, lam, u, x,
                                             implicit_euler, grad_prefactor, s);
    if (max_fiber_len <= 4096)
      return adjoint_diffusion_block<512, 8>(n_fibers, fiber_offsets, element_lengths, coef, stride, lam, u, x,
                                             implicit_euler, grad_prefactor, s);
  }
  const int T = 128;
  const int64_t threads = (int64_t)n_fibers * 32;
  adjoint_diffusion_warp_kernel<<<(unsigned)((threads + T - 1) / T), T, 0, s>>>(
      n_fibers, fiber_offsets, element_lengths, coef, stride, lam, u, x, implicit_euler, grad_prefactor, scratch, mu);
  return cudaGetLastError();
}

__global__ void count_nonfinite_kernel(const double* __restrict__ x, int64_t n, int* count)
{
  int local = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    local += isfinite(x[i]) ? 0 : 1;
  local = __reduce_add_sync(0xffffffffu, local);
  if ((threadIdx.x & 31) == 0 && local)
    atomicAdd(count, local);
}

cudaError_t launch_count_nonfinite(const double* x, int64_t n, int* count, cudaStream_t s)
{
  if (n == 0)
    return cudaSuccess;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 8)
    blocks = 148 * 8;
  count_nonfinite_kernel<<<blocks, 256, 0, s>>>(x, n, count);
  return cudaGetLastError();
}

} // namespace fdm
