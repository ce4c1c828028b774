// Diffusion kernels of the split path: the factorization of every fiber's tridiagonal system, its solve with a
// stored factorization, and both in one pass for the standalone operator (compute.tpp:256-507).
//   IE: (K - M/dt) u+ = -M/dt u            CN: (K/2 - M/dt) u+ = (-K/2 - M/dt) u
// following the element loops of compute.tpp:336-449, and its LU factors for
//   d'_i = mulF_i d'_{i-1} + inv_i d_i,     x_i = d'_i - cp_i x_{i+1}
// Per node the six doubles are stored as coef[k*stride + node], k = 0..5 = mulF, inv, cp, l, m, r
// with d_i = l_i u_{i-1} + m_i u_i + r_i u_{i+1}.
#pragma once
#include "fdm_kernels.cuh"

namespace fdm {

// Elements of a fiber as the assembly needs them: k = pf/h and m = h/6 (the mass entries are m and 2 m = h/3), both
// 0 where there is no element.
struct ElementTerms {
  double idt, theta;   // 1/dt; 1 (IE) or 1/2 (CN)
  int ie;
  __device__ __forceinline__ ElementTerms(double dt, int implicit_euler)
      : idt(1 / dt), theta(implicit_euler ? 1.0 : 0.5), ie(implicit_euler)
  {
  }
  __device__ __forceinline__ double off(double k, double m) const { return theta * k - idt * m; }
  __device__ __forceinline__ double diag(double k, double m) const { return -theta * k - idt * (2.0 * m); }
  __device__ __forceinline__ double rhs_off(double k, double m) const
  {
    return ie ? -idt * m : -0.5 * k - idt * m;
  }
  __device__ __forceinline__ double rhs_diag(double k, double m) const
  {
    return ie ? -idt * (2.0 * m) : 0.5 * k - idt * (2.0 * m);
  }
};

// One CTA per fiber.  The factorization is the serial chain cp_i = c_i / (b_i - a_i cp_{i-1}), one division after the
// other along the fiber.  Its dependence on the entering value shrinks by a_i c_i / den_i^2 < 1 per node (about 0.01
// for the usual steps), so each thread runs its chunk of nodes from FACTOR_WARMUP nodes earlier with a guessed
// entering value of 0 and reaches the chain's own value, bit for bit.  That is checked: a thread whose entering value
// differs in any bit from the last value of the chunk before it repeats its chunk from that one, until no thread
// differs, so the result is the serial chain's whatever the step width.
//   WHAT == FACTOR: the coefficients are written; FACTOR_SOLVE: they stay on chip and vm is solved in place.
// A tile of FACTOR_TILE nodes lives in shared memory (longer fibers: tile after tile, in FACTOR_SOLVE with d' and cp
// in scratch between the two sweeps).  Threads hold an odd number of consecutive nodes, so that their shared-memory
// accesses, that many doubles apart, meet no bank twice.
// Bound by FP64 work (two divisions per element, two to three per node with the warm-up) and latency, so what counts is
// that three CTAs share an SM: three arrays of a tile in shared memory, the reciprocals of the chain's divisions kept for
// the sweeps, the branch-free division.  A thread per fiber, with six divisions and six uncoalesced stores per node, took
// 2519 us for the factorization of 4096 fibers of 500 to 2500 nodes and a solve 524 us more; FACTOR_SOLVE does both in
// 169 us (214 with four arrays, CUDA's division and another reciprocal per node).  (Factorization of 64 fibers of 1481
// nodes: 1129 us, now 8.)
constexpr int FACTOR_T = 256;
constexpr int FACTOR_M = 11;          // most nodes per thread (odd)
constexpr int FACTOR_TILE = 2560;
constexpr int FACTOR_WARMUP = 12;
enum FactorWhat { FACTOR, FACTOR_SOLVE };

constexpr int FACTOR_PER = FACTOR_TILE / FACTOR_T;   // most nodes per thread of the assembly

inline size_t factor_smem_bytes(int tile) { return sizeof(double) * (size_t)(2 * (tile + 1) + tile); }

template<int WHAT>
__global__ void __launch_bounds__(FACTOR_T, 3) diffusion_factor_kernel(
    const int64_t* __restrict__ fiber_offsets, const double* __restrict__ element_lengths,
    const double* __restrict__ prefactor, double dt, int implicit_euler, double* __restrict__ coef, int64_t stride,
    double* __restrict__ vm, double* __restrict__ scratch, int tile)
{
  extern __shared__ double smem[];
  double* so = smem;             // tile + 1: off-diagonal of the element left of local node i at i (first its k)
  double* sb = so + tile + 1;    // tile + 1: diagonal of node i (first the element's m)
  double* sr = sb + tile + 1;    // tile: FACTOR_SOLVE: right-hand side, then d', then the solution; FACTOR: cp
  __shared__ double sexit[FACTOR_T];
  __shared__ double sF[2 * (FACTOR_T / 32)], sG[2 * (FACTOR_T / 32)];
  const int f = blockIdx.x;
  const int tid = threadIdx.x;
  const int64_t o = fiber_offsets[f];
  const int64_t n = fiber_offsets[f + 1] - o;
  const double* h = element_lengths + (o - f); // fiber f's elements follow the previous fibers' n-1 each
  const double pf = prefactor[f];
  const ElementTerms et(dt, implicit_euler);
  double carry_cp = 0.0, carry_d = 0.0;
  double cp[FACTOR_M], inv[FACTOR_M];
  for (int64_t base = 0; base < n; base += tile) {
    const int cnt = (int)min((int64_t)tile, n - base);
    const int m = ((cnt + FACTOR_T - 1) / FACTOR_T) | 1;
    for (int e = tid; e <= cnt; e += FACTOR_T) {
      const int64_t g = base - 1 + e;
      const bool ok = g >= 0 && g < n - 1;
      const double hh = ok ? h[g] : 1.0;
      so[e] = ok ? fdm_rcp64(hh) * pf : 0.0;
      sb[e] = ok ? fdm_div64(hh, 6.0) : 0.0;
    }
    __syncthreads();
    double off[FACTOR_PER], diag[FACTOR_PER];
    double last_off = 0.0;
#pragma unroll
    for (int j = 0; j < FACTOR_PER; j++) {
      const int i = tid + j * FACTOR_T;
      if (i >= cnt)
        continue;
      const double k0 = so[i], m0 = sb[i], k1 = so[i + 1], m1 = sb[i + 1];
      off[j] = et.off(k0, m0);
      diag[j] = et.diag(k0, m0) + et.diag(k1, m1);
      if (i == cnt - 1)
        last_off = et.off(k1, m1);
      const double l = et.rhs_off(k0, m0), c = et.rhs_diag(k0, m0) + et.rhs_diag(k1, m1), r = et.rhs_off(k1, m1);
      const int64_t v = base + i;
      if (WHAT == FACTOR) {
        coef[3 * stride + o + v] = l;
        coef[4 * stride + o + v] = c;
        coef[5 * stride + o + v] = r;
      } else {
        const double um = v > 0 ? vm[o + v - 1] : 0.0, up = v < n - 1 ? vm[o + v + 1] : 0.0;
        sr[i] = l * um + c * vm[o + v] + r * up;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < FACTOR_PER; j++) {
      const int i = tid + j * FACTOR_T;
      if (i >= cnt)
        continue;
      so[i] = off[j];
      sb[i] = diag[j];
      if (i == cnt - 1)
        so[cnt] = last_off;
    }
    __syncthreads();
    // the chunk [lo, hi) of this thread
    const int lo = min(tid * m, cnt), hi = min(lo + m, cnt);
    auto link = [&](int i, double before, double& reciprocal) -> double {
      const double d = sb[i] - before * so[i], c = so[i + 1];
      reciprocal = fdm_rcp64(d);
      const double q = c * reciprocal;
      return fma(fma(-d, q, c), reciprocal, q);   // c / d as fdm_div64
    };
    auto chunk = [&](double x) -> double {
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi) {
          x = link(lo + j, x, inv[j]);
          cp[j] = x;
        }
      return x;
    };
    double entry = lo <= FACTOR_WARMUP ? carry_cp : 0.0;
    for (int i = max(0, lo - FACTOR_WARMUP); i < lo; i++) {
      double r;
      entry = link(i, entry, r);
    }
    sexit[tid] = chunk(entry);
    __syncthreads();
    for (int round = 0; round <= FACTOR_T; round++) { // a round finishes at least the first chunk that differs
      const double prev = tid > 0 ? sexit[tid - 1] : carry_cp;
      const bool differs = lo < hi && __double_as_longlong(prev) != __double_as_longlong(entry);
      if (!__syncthreads_or(differs))
        break;
      if (differs) {
        entry = prev;
        sexit[tid] = chunk(entry);
      }
      __syncthreads();
    }
    const double last_cp = sexit[(cnt - 1) / m];
    if (WHAT == FACTOR) {
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi)
          sr[lo + j] = cp[j];
      __syncthreads();
      for (int i = tid; i < cnt; i += FACTOR_T) {
        const int64_t g = o + base + i;
        const double a = so[i];
        const double r = fdm_rcp64(sb[i] - (i > 0 ? sr[i - 1] : carry_cp) * a);
        coef[0 * stride + g] = base + i > 0 ? -a * r : 0.0;
        coef[1 * stride + g] = r;
        coef[2 * stride + g] = base + i < n - 1 ? sr[i] : 0.0;
      }
    } else {
      // forward sweep
      Affine acc{1.0, 0.0};
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi)
          acc = compose(acc, Affine{-so[lo + j] * inv[j], inv[j] * sr[lo + j]});
      Affine total;
      const Affine pre = block_scan_map<FACTOR_T, false>(acc, sF, sG, &total);
      double d = fma(pre.F, carry_d, pre.G);
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi) {
          d = -so[lo + j] * inv[j] * d + inv[j] * sr[lo + j];
          sr[lo + j] = d;
        }
      carry_d = fma(total.F, carry_d, total.G);
      if (n > tile) {
#pragma unroll
        for (int j = 0; j < FACTOR_M; j++)
          if (lo + j < hi) {
            scratch[o + base + lo + j] = sr[lo + j];
            scratch[stride + o + base + lo + j] = cp[j];
          }
      }
    }
    carry_cp = last_cp;
    if (n > tile)
      __syncthreads(); // the tile's shared arrays and scan slots are free
  }
  if (WHAT == FACTOR_SOLVE && n > 0) {
    // back substitution, from the last tile (its d' and cp still in place) to the first
    double carry_x = 0.0;
    for (int64_t base = (n - 1) / tile * tile; base >= 0; base -= tile) {
      const int cnt = (int)min((int64_t)tile, n - base);
      const int m = ((cnt + FACTOR_T - 1) / FACTOR_T) | 1;
      const int lo = min(tid * m, cnt), hi = min(lo + m, cnt);
      if (base + cnt < n) {
#pragma unroll
        for (int j = 0; j < FACTOR_M; j++)
          if (lo + j < hi) {
            sr[lo + j] = scratch[o + base + lo + j];
            cp[j] = scratch[stride + o + base + lo + j];
          }
      }
      Affine acc{1.0, 0.0};
#pragma unroll
      for (int j = FACTOR_M - 1; j >= 0; j--)
        if (lo + j < hi)
          acc = compose(acc, Affine{-cp[j], sr[lo + j]});
      Affine total;
      const Affine pre =
          block_scan_map<FACTOR_T, true>(acc, sF + FACTOR_T / 32, sG + FACTOR_T / 32, &total);
      double x = fma(pre.F, carry_x, pre.G);
#pragma unroll
      for (int j = FACTOR_M - 1; j >= 0; j--)
        if (lo + j < hi) {
          x = -cp[j] * x + sr[lo + j];
          sr[lo + j] = x;
        }
      carry_x = fma(total.F, carry_x, total.G);
      __syncthreads();
      for (int i = tid; i < cnt; i += FACTOR_T)
        vm[o + base + i] = sr[i];
      if (n > tile)
        __syncthreads();
    }
  }
}

// One diffusion solve per fiber with a stored factorization, one CTA per fiber of at most DIFFUSION_T * M nodes.  Each
// thread owns ceil(n / DIFFUSION_T) consecutive nodes and reads all it needs of them at once, so that the loads
// overlap; the right-hand side, d' and the factors stay in registers and the two sweeps are block-wide scans.  The
// partition follows from the fiber's own length alone: a fiber's result does not depend on the fibers beside it.
// eq_counter / eq_nbuf (or null): the equilibrium skip's per-rank count of inactive buffers and number of
// buffers; a fiber of a rank whose buffers are all counted inactive is not solved (compute.tpp:261-265)
// Bound by the latency of the loads and the two scans for few fibers (16 x 1481: 6.5 us with a loop over the nodes
// and d' in memory, now 4.4), by memory for many (1024 fibers of 500 to 2500 nodes: 156 us with a warp per fiber and
// its uncoalesced chunks, now 31.7; 100 MB, 0.5 of the measured copy rate).
constexpr int DIFFUSION_T = 256;

// the stored factorization of a thread's chunk of a fiber, and the solve of the CTA's fiber with it
template<int M>
struct DiffusionChunk {
  int n, lo, cnt;               // nodes of the fiber, the thread's first node and number of nodes
  double F[M], C[M], inv[M], cl[M], cm[M], cr[M];
  __device__ __forceinline__ void load(const double* __restrict__ coef, int64_t stride, int64_t o, int nodes)
  {
    n = nodes;
    const int L = (n + DIFFUSION_T - 1) / DIFFUSION_T;
    lo = min((int)threadIdx.x * L, n);
    cnt = min(L, n - lo);
    const double* c0 = coef + o + lo;
#pragma unroll
    for (int j = 0; j < M; j++) {
      const bool on = j < cnt;
      F[j] = on ? c0[j] : 1.0;   // beyond the chunk the identity map
      C[j] = on ? c0[2 * stride + j] : -1.0;
      inv[j] = on ? c0[stride + j] : 0.0;
      cl[j] = on ? c0[3 * stride + j] : 0.0;
      cm[j] = on ? c0[4 * stride + j] : 0.0;
      cr[j] = on ? c0[5 * stride + j] : 0.0;
    }
  }
  // v: the fiber's Vm (global or shared memory), solved in place; sF, sG: 2 * DIFFUSION_T / 32 slots
  __device__ __forceinline__ void solve(double* v, double* sF, double* sG) const
  {
    double u[M + 2], G[M];
#pragma unroll
    for (int j = 0; j < M + 2; j++)
      u[j] = (j <= cnt + 1 && lo + j >= 1 && lo + j <= n) ? v[lo + j - 1] : 0.0;
#pragma unroll
    for (int j = 0; j < M; j++)
      G[j] = inv[j] * (cl[j] * u[j] + cm[j] * u[j + 1] + cr[j] * u[j + 2]);
    Affine acc{1.0, 0.0};
#pragma unroll
    for (int j = 0; j < M; j++)
      acc = compose(acc, Affine{F[j], G[j]});
    // its barrier follows every read of the old Vm
    double d = block_scan_incoming<DIFFUSION_T, false>(acc, sF, sG);
    Affine bacc{1.0, 0.0};
#pragma unroll
    for (int j = 0; j < M; j++) {
      d = F[j] * d + G[j];
      G[j] = j < cnt ? d : 0.0;
    }
#pragma unroll
    for (int j = M - 1; j >= 0; j--)
      bacc = compose(bacc, Affine{-C[j], G[j]});
    double x = block_scan_incoming<DIFFUSION_T, true>(bacc, sF + DIFFUSION_T / 32, sG + DIFFUSION_T / 32);
#pragma unroll
    for (int j = M - 1; j >= 0; j--) {
      x = -C[j] * x + G[j];
      if (j < cnt)
        v[lo + j] = x;
    }
  }
};

template<int M>
__global__ void __launch_bounds__(DIFFUSION_T) diffusion_reg_kernel(const int64_t* __restrict__ fiber_offsets,
                                                                    const double* __restrict__ coef, int64_t stride,
                                                                    double* __restrict__ vm,
                                                                    const int* __restrict__ eq_counter,
                                                                    const int* __restrict__ eq_nbuf, int n_ranks)
{
  __shared__ double sF[2 * (DIFFUSION_T / 32)], sG[2 * (DIFFUSION_T / 32)];
  const int f = blockIdx.x;
  if (eq_counter && eq_counter[f % n_ranks] == eq_nbuf[f % n_ranks])
    return; // the whole CTA: the rank's buffers are all inactive
  const int64_t o = fiber_offsets[f];
  DiffusionChunk<M> chunk;
  chunk.load(coef, stride, o, (int)(fiber_offsets[f + 1] - o));
  chunk.solve(vm + o, sF, sG);
}

// A whole window of split steps of few fibers in one launch, FP64: a fiber per thread-block cluster, a thread per node.
// With a launch per half step and per solve the launches, the passes over the states and the start of every kernel
// take about half of a step that has some hundred nodes per SM.  Here the states stay in registers for the window; the
// CTAs send their Vm to the cluster's first one, which solves the fiber's diffusion as diffusion_reg_kernel does, with
// the factors in registers, and the others fetch theirs back: two cluster barriers per step.  Same functions and
// partition as the kernels it stands in for, and the same values, bit for bit, whichever form the number of fibers
// leads to. Bound by the FP64 work of the Heun substeps at 8 warps per SM, 2.0 us of the 2.7 + 2.0 n0 us per step at n0
// substeps a half step.  Per step of 5 substeps a half step, with launches and so: 16 fibers of 1481 nodes (clusters of
// 6) 15.1 and 12.6 us; one of 101 nodes 9.4 and 6.8; 74 of 500 14.1 and 10.6.
constexpr int WINDOW_T = DIFFUSION_T;

template<class Model, class Math, int M>
__global__ void __launch_bounds__(WINDOW_T, 1) window_cluster_kernel(ReactionArgs a,
                                                                     const int64_t* __restrict__ fiber_offsets,
                                                                     const double* __restrict__ coef, int n_steps)
{
  constexpr int NS = Model::nStates;
  constexpr int NP = Model::nParameters > 0 ? Model::nParameters : 1;
  constexpr int NSM = NS > 1 ? NS - 1 : 1;
  __shared__ double vs[WINDOW_T * M];
  __shared__ double sF[2 * (WINDOW_T / 32)], sG[2 * (WINDOW_T / 32)];
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank(), csize = (int)cluster.num_blocks();
  const int f = blockIdx.x / csize;
  const int64_t o = fiber_offsets[f];
  const int n = (int)(fiber_offsets[f + 1] - o);
  const int npc = (n + csize - 1) / csize;   // nodes per CTA, at most WINDOW_T
  const int q = crank * npc + (int)threadIdx.x;
  const bool ok = (int)threadIdx.x < npc && q < n;
  const int64_t i = o + (ok ? q : 0);
  double* home = cluster.map_shared_rank(vs, 0);
  double* st = (double*)a.states;
  const double* pr = (const double*)a.params;
  double V = a.vm[i], S[NSM], Lo[NSM], P[NP], Pstim[NP];
#pragma unroll
  for (int s = 1; s < NS; s++) {
    S[s - 1] = st[(s - 1) * a.stride + i];
    Lo[s - 1] = 0.0;
  }
#pragma unroll
  for (int p = 0; p < Model::nParameters; p++) {
    P[p] = pr[p * a.stride + i];
    Pstim[p] = (a.stimulus_mode == 1 && p == a.stimulus_parameter) ? a.stimulus_value : P[p];
  }
  const int cf = ok ? a.clamp_fiber[i] : -1;
  const int slot = ok && a.trace_slot ? a.trace_slot[i] : -1;
  DiffusionChunk<M> chunk;
  chunk.load(coef, a.stride, o, crank == 0 ? n : 0);
#pragma unroll 1
  for (int hs = 0; hs < 2 * n_steps; hs++) {
    const SplitStep s = a.steps[hs >> 1];
    const double t0 = (hs & 1) ? s.mid : s.t;
    const int base = hs * a.nsub_stride;
    const int first = a.gate ? gate_first(a.gate_start, a.gate_stride, a.gate[i], hs) : 0;
    const bool store = a.store_alg && hs == 2 * n_steps - 1;
    if (ok) {
#pragma unroll 1
      for (int k = first; k < s.n0; k++) {
        const double t = xadd(t0, xmul((double)k, s.dt0));
        const bool stim = cf >= 0 && stim_bit(a.flags, a.words_per_fiber, cf, base + k);
        const bool vclamp = stim && a.stimulus_mode == 0;
        double Pk[NP];
#pragma unroll
        for (int p = 0; p < NP; p++)
          Pk[p] = (stim && a.stimulus_mode == 1) ? Pstim[p] : P[p];
        if (store && k == s.n0 - 1) {
          double alg[Model::nAlgebraics];
          heun_step<Model, double, Math, true>(V, S, Lo, Pk, t, s.dt0, vclamp, a.vstim, alg);
          store_algebraics<Model>(alg, a.n_alg_out, a.alg_indices, a.alg_out, a.n_nodes, i);
        } else {
          heun_step<Model, double, Math, false>(V, S, Lo, Pk, t, s.dt0, vclamp, a.vstim, nullptr);
        }
      }
    }
    if (hs & 1) {
      if (slot >= 0)
        record_trace(a.trace, a.n_trace, a.trace_capacity, a.act, slot, s.global_no, V);
      continue;
    }
    // (a slot of home is read back by the thread that fills it: no barrier is needed before the next fill)
    if (ok)
      home[q] = V;
    cluster.sync();
    if (crank == 0)
      chunk.solve(vs, sF, sG);
    cluster.sync();
    if (ok)
      V = home[q];
  }
  if (ok) {
    a.vm[i] = V;
#pragma unroll
    for (int s = 1; s < NS; s++)
      st[(s - 1) * a.stride + i] = S[s - 1];
  }
  cluster.sync();   // the first CTA's shared memory outlives the others' reads
}

} // namespace fdm
