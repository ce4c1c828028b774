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
// Bound by FP64 work (two divisions per element, two to three per node with the warm-up) and latency; a thread per
// fiber, with six divisions and six uncoalesced stores per node, took 2519 us for the factorization of 4096 fibers of
// 500 to 2500 nodes and a solve 524 us more; FACTOR_SOLVE does both in 214 us.  (64 fibers of 1481 nodes: 1129 us,
// now 8.)
constexpr int FACTOR_T = 256;
constexpr int FACTOR_M = 11;          // most nodes per thread (odd)
constexpr int FACTOR_TILE = 2560;
constexpr int FACTOR_WARMUP = 12;
enum FactorWhat { FACTOR, FACTOR_SOLVE };

inline size_t factor_smem_bytes(int tile) { return sizeof(double) * (size_t)(2 * (tile + 1) + 2 * tile); }

template<int WHAT>
__global__ void __launch_bounds__(FACTOR_T) diffusion_factor_kernel(
    const int64_t* __restrict__ fiber_offsets, const double* __restrict__ element_lengths,
    const double* __restrict__ prefactor, double dt, int implicit_euler, double* __restrict__ coef, int64_t stride,
    double* __restrict__ vm, double* __restrict__ scratch, int tile)
{
  extern __shared__ double smem[];
  double* ek = smem;             // tile + 1: element left of local node i at i, right of it at i + 1
  double* em = ek + tile + 1;    // tile + 1
  double* sb = em + tile + 1;    // tile: diagonal (FACTOR_SOLVE: then the solution)
  double* sr = sb + tile;        // tile: right-hand side (FACTOR: then cp)
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
  double cp[FACTOR_M], den[FACTOR_M];
  for (int64_t base = 0; base < n; base += tile) {
    const int cnt = (int)min((int64_t)tile, n - base);
    const int m = ((cnt + FACTOR_T - 1) / FACTOR_T) | 1;
    for (int e = tid; e <= cnt; e += FACTOR_T) {
      const int64_t g = base - 1 + e;
      const bool ok = g >= 0 && g < n - 1;
      const double hh = ok ? h[g] : 1.0;
      ek[e] = ok ? 1. / hh * pf : 0.0;
      em[e] = ok ? hh / 6 : 0.0;
    }
    __syncthreads();
    for (int i = tid; i < cnt; i += FACTOR_T) {
      sb[i] = et.diag(ek[i], em[i]) + et.diag(ek[i + 1], em[i + 1]);
      if (WHAT == FACTOR_SOLVE) {
        const int64_t v = base + i;
        const double um = v > 0 ? vm[o + v - 1] : 0.0, up = v < n - 1 ? vm[o + v + 1] : 0.0;
        sr[i] = et.rhs_off(ek[i], em[i]) * um +
                (et.rhs_diag(ek[i], em[i]) + et.rhs_diag(ek[i + 1], em[i + 1])) * vm[o + v] +
                et.rhs_off(ek[i + 1], em[i + 1]) * up;
      }
    }
    __syncthreads();
    // the chunk [lo, hi) of this thread
    const int lo = min(tid * m, cnt), hi = min(lo + m, cnt);
    auto link = [&](int i, double before, double& d) -> double {
      d = sb[i] - before * et.off(ek[i], em[i]);
      return et.off(ek[i + 1], em[i + 1]) / d;
    };
    auto chunk = [&](double x) -> double {
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi) {
          x = link(lo + j, x, den[j]);
          cp[j] = x;
        }
      return x;
    };
    double entry = lo <= FACTOR_WARMUP ? carry_cp : 0.0;
    for (int i = max(0, lo - FACTOR_WARMUP); i < lo; i++) {
      double d;
      entry = link(i, entry, d);
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
        const double a = et.off(ek[i], em[i]);
        const double inv = 1.0 / (sb[i] - (i > 0 ? sr[i - 1] : carry_cp) * a);
        coef[0 * stride + g] = base + i > 0 ? -a * inv : 0.0;
        coef[1 * stride + g] = inv;
        coef[2 * stride + g] = base + i < n - 1 ? sr[i] : 0.0;
        coef[3 * stride + g] = et.rhs_off(ek[i], em[i]);
        coef[4 * stride + g] = et.rhs_diag(ek[i], em[i]) + et.rhs_diag(ek[i + 1], em[i + 1]);
        coef[5 * stride + g] = et.rhs_off(ek[i + 1], em[i + 1]);
      }
    } else {
      // forward sweep: den becomes d'
      Affine acc{1.0, 0.0};
      double mf[FACTOR_M];
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi) {
          const double inv = 1.0 / den[j];
          mf[j] = -et.off(ek[lo + j], em[lo + j]) * inv;
          den[j] = inv * sr[lo + j];
          acc = compose(acc, Affine{mf[j], den[j]});
        }
      Affine total;
      const Affine pre = block_scan_map<FACTOR_T, false>(acc, sF, sG, &total);
      double d = fma(pre.F, carry_d, pre.G);
#pragma unroll
      for (int j = 0; j < FACTOR_M; j++)
        if (lo + j < hi) {
          d = mf[j] * d + den[j];
          den[j] = d;
        }
      carry_d = fma(total.F, carry_d, total.G);
      if (n > tile) {
#pragma unroll
        for (int j = 0; j < FACTOR_M; j++)
          if (lo + j < hi) {
            scratch[o + base + lo + j] = den[j];
            scratch[stride + o + base + lo + j] = cp[j];
          }
      }
    }
    carry_cp = last_cp;
    if (n > tile)
      __syncthreads(); // the tile's shared arrays and scan slots are free
  }
  if (WHAT == FACTOR_SOLVE && n > 0) {
    // back substitution, from the last tile (still in registers) to the first
    double carry_x = 0.0;
    for (int64_t base = (n - 1) / tile * tile; base >= 0; base -= tile) {
      const int cnt = (int)min((int64_t)tile, n - base);
      const int m = ((cnt + FACTOR_T - 1) / FACTOR_T) | 1;
      const int lo = min(tid * m, cnt), hi = min(lo + m, cnt);
      if (base + cnt < n) {
#pragma unroll
        for (int j = 0; j < FACTOR_M; j++)
          if (lo + j < hi) {
            den[j] = scratch[o + base + lo + j];
            cp[j] = scratch[stride + o + base + lo + j];
          }
      }
      Affine acc{1.0, 0.0};
#pragma unroll
      for (int j = FACTOR_M - 1; j >= 0; j--)
        if (lo + j < hi)
          acc = compose(acc, Affine{-cp[j], den[j]});
      Affine total;
      const Affine pre =
          block_scan_map<FACTOR_T, true>(acc, sF + FACTOR_T / 32, sG + FACTOR_T / 32, &total);
      double x = fma(pre.F, carry_x, pre.G);
#pragma unroll
      for (int j = FACTOR_M - 1; j >= 0; j--)
        if (lo + j < hi) {
          x = -cp[j] * x + den[j];
          sb[lo + j] = x;
        }
      carry_x = fma(total.F, carry_x, total.G);
      __syncthreads();
      for (int i = tid; i < cnt; i += FACTOR_T)
        vm[o + base + i] = sb[i];
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
  const int n = (int)(fiber_offsets[f + 1] - o);
  const int L = (n + DIFFUSION_T - 1) / DIFFUSION_T;
  const int lo = min((int)threadIdx.x * L, n);
  const int cnt = min(L, n - lo);
  const double* c0 = coef + o + lo;
  double* v = vm + o + lo;
  double F[M], G[M], C[M];
  double u[M + 2];
#pragma unroll
  for (int j = 0; j < M + 2; j++)
    u[j] = (j <= cnt + 1 && lo + j >= 1 && lo + j <= n) ? v[j - 1] : 0.0;
#pragma unroll
  for (int j = 0; j < M; j++) {
    if (j < cnt) {
      F[j] = c0[j];
      C[j] = c0[2 * stride + j];
      G[j] = c0[stride + j] *
             (c0[3 * stride + j] * u[j] + c0[4 * stride + j] * u[j + 1] + c0[5 * stride + j] * u[j + 2]);
    } else {
      F[j] = 1.0;   // the identity map
      C[j] = -1.0;
      G[j] = 0.0;
    }
  }
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
      v[j] = x;
  }
}

} // namespace fdm
