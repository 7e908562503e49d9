// hq_kernels.cu -- the smaller sm_100a kernels of the batched DQMC sweep (FP64) and the
// shared-memory limits of every per-chain kernel. The large kernels have files of their own:
//  hq_interval.cu : k_interval (wrap + Metropolis flips with DMMA-flushed delayed updates)
//  hq_udt.cu      : k_udt (UDV factorisation of a stack push)
//  hq_invert.cu   : k_invert (blocked Gauss-Jordan inverse of the G builders)
//  hq_gemm.cu     : k_gemm (batched DMMA GEMM of the G builders)
// This file holds:
//  k_bchain    : B-matrix chain of one interval applied to U_top*D_top
//                (src/dqmc_core.cpp:190, :251 + the (M*U)*S product of svd_stack.hpp:144).
//  k_measure   : equal-time estimators + snapshot of a freshly built G.
//  k_dyn_*     : time-displaced propagation and estimators (src/dqmc_core.cpp:291-390,
//                include/observable_methods.hpp:84-195).
//  k_adj_*     : adjoint of log|det(1 + B...B)| (no counterpart in the reference).
#include <algorithm>
#include <mutex>

#include "hq_phases.cuh"

namespace hq {

// ---------------------------------------------------------------------------------
//  k_bchain: X <- (U_top diag(D_top) or 1), then the B products of interval b:
//   up  : X <- B(t) X = e^{V_t} E X, t ascending            (src/dqmc_core.cpp:190)
//   down: X <- B(t)^T X = E e^{V_t} X, t descending           (src/dqmc_core.cpp:251)
//  dir UP pushes onto the left stack, DOWN onto the right stack; that stack holds b
//  entries before the push (top entry b-1, none when b = 0).
//  init: the right stack at initialisation (src/dqmc_core.cpp:67-87) is the down
//  direction without updates.
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(HQ_INT_THREADS, 1)
k_bchain(const HqChain* __restrict__ chains, int nchains, int dir, int b, int resident) {
  extern __shared__ __align__(16) double smem[];
  __shared__ HqChain ch;
  const int c = blockIdx.x;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  if (!ch.active || b >= ch.n_stab) return;
  bchain_body(ch, dir, b, resident != 0, smem);
}

// ---------------------------------------------------------------------------------
//  k_measure: estimators + snapshot of G after a stabilisation (slice `lslice`
//  computed from the interval), the last slice of every interval.
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(HQ_THREADS)
k_measure(const HqChain* __restrict__ chains, int nchains, int dir, int b, int flags) {
  __shared__ HqChain ch;
  __shared__ double red[96];
  const int c = blockIdx.x;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  if (!ch.active || b >= ch.n_stab) return;
  measure_body(ch, dir, b, flags, red);
}

// ---------------------------------------------------------------------------------
//  Dynamic (time-displaced) sweep, src/dqmc_core.cpp:291-390. Per slice t:
//    G(t,t) <- B G B^-1 ; G(t,0) <- B G(t,0) ; G(0,t) <- G(0,t) B^-1
//  k_dyn_slices applies this for the interval's slices to one of the three matrices per
//  CTA (blockIdx.y = 0: G(t,t), 1: G(t,0), 2: G(0,t)), except for the last slice which
//  is rebuilt by the boundary step, and stores the per-slice results.
// ---------------------------------------------------------------------------------
template <bool RES>
__device__ __forceinline__ void dyn_step(const HqChain& ch, double* M, int ld, int which, const double* vp, const double* vm,
                                         double* stage) {
  if (which != 2) apply_side<LEFT_B, RES>(ch, M, ld, vp, stage);      // left multiplication by B(l) = e^V E
  if (which != 1) apply_side<RIGHT_BINV, RES>(ch, M, ld, vm, stage);  // right multiplication by B(l)^-1
}

__global__ void __launch_bounds__(HQ_INT_THREADS, 1)
k_dyn_slices(const HqChain* __restrict__ chains, int nchains, int b, int flags, int resident) {
  extern __shared__ __align__(16) double smem[];
  __shared__ HqChain ch;
  const int c = blockIdx.x, which = blockIdx.y;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  if (!ch.active || b >= ch.n_stab) return;
  const int N = ch.N;
  int t_lo, t_hi;
  interval_range(ch.nt, ch.pace, ch.n_stab, HQ_UP, b, t_lo, t_hi);
  double* src = which == 0 ? ch.G : (which == 1 ? ch.Gt0 : ch.G0t);
  double* snap = which == 0 ? ch.snap_tt : (which == 1 ? ch.snap_t0 : ch.snap_0t);
  double* M;
  int ld;
  double* p = smem;
  if (resident) { M = p; ld = interval_ld(N); p += (size_t)N * ld; load_mat_async(M, ld, src, N, N); }
  else { M = src; ld = N; }
  double* stage = p;
  double* vp = stage + 8 * (pad16(N) + 4);
  double* vm = vp + N;
  __syncthreads();
  const int nsl = t_hi - t_lo + 1;
  // the next slice's fields are on their way while a slice is worked on
  auto field = [&](int t) {
    return t <= t_hi && (int)threadIdx.x < N ? ch.fields[(size_t)(t % ch.nt) * N + threadIdx.x] : (int8_t)0;
  };
  int8_t next = field(t_lo);
  for (int step = 0; step < nsl; ++step) {
    const int t = t_lo + step;
    const int l = t % ch.nt;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const bool pos = (i == (int)threadIdx.x ? next : ch.fields[(size_t)l * N + i]) > 0;
      vp[i] = pos ? ch.ev_p : ch.ev_m;
      vm[i] = pos ? ch.ev_m : ch.ev_p;
    }
    next = field(t + 1);
    __syncthreads();
    if (resident) dyn_step<true>(ch, M, ld, which, vp, vm, stage);
    else dyn_step<false>(ch, M, ld, which, vp, vm, stage);
    if (step < nsl - 1 && snap) copy_mat(snap + (size_t)l * N * N, N, M, ld, N);
    __syncthreads();
  }
  if (resident) copy_mat(src, N, M, ld, N);
}

// G(t,0) <- G(t,t) and G(0,t) <- G(t,t) - 1 at the start of a dynamic sweep
// (src/dqmc_core.cpp:302-303)
__global__ void k_dyn_start(const HqChain* __restrict__ chains, int nchains) {
  const int c = blockIdx.x;
  if (c >= nchains) return;
  const HqChain& ch = chains[c];
  if (!ch.active) return;
  const int N = ch.N;
  for (int idx = threadIdx.x; idx < N * N; idx += blockDim.x) {
    const int i = idx % N, j = idx / N;
    const double v = ch.G[idx];
    ch.Gt0[idx] = v;
    ch.G0t[idx] = v - (i == j ? 1.0 : 0.0);
  }
}

// dynamic estimators of one slice l from G(t,0), G(0,t) (include/observable_methods.hpp:
// 110-120, 178-195) and the displacement-summed g(d) = sum_i G(t,0)[i+d, i] for G(k,t)
// (:84-103). dyn_acc layout: [0][nt] spin, [1][nt] ldos, [2 + d][nt] g(d) for d < N.
__device__ void dyn_measure(const HqChain& ch, const double* Gt0, const double* G0t, int l, double* red) {
  const int N = ch.N, L = ch.L;
  double sp = 0.0, ld = 0.0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const double a = Gt0[i + (size_t)i * N], b = G0t[i + (size_t)i * N];
    sp -= 2.0 * a * b;
    ld += a;
  }
  sp = block_sum(sp, red);
  ld = block_sum(ld, red);
  if (threadIdx.x == 0) {
    ch.dyn_acc[0 * ch.nt + l] += sp / (2.0 * N);
    ch.dyn_acc[1 * ch.nt + l] += ld / N;
  }
  // g(d): d = dx + L dy, sum over i of G[(xi+dx, yi+dy), i]
  for (int d = threadIdx.x; d < N; d += blockDim.x) {
    const int dx = d % L, dy = d / L;
    double acc = 0.0;
    for (int i = 0; i < N; ++i) {
      const int xi = i % L, yi = i / L;
      const int j = (xi + dx) % L + L * ((yi + dy) % L);
      acc += Gt0[j + (size_t)i * N];
    }
    ch.dyn_acc[(size_t)(2 + d) * ch.nt + l] += acc;
  }
}

// measure the dynamic estimators of every slice of interval b from the snapshots
// (slices of the interval other than the last) or from the fresh G's (the last one): one CTA per
// slice (blockIdx.y), whose sums are its own
__global__ void __launch_bounds__(HQ_THREADS)
k_dyn_measure(const HqChain* __restrict__ chains, int nchains, int b) {
  __shared__ HqChain ch;
  __shared__ double red[32];
  const int c = blockIdx.x;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  if (!ch.active || b >= ch.n_stab) return;
  const int N = ch.N;
  int t_lo, t_hi;
  interval_range(ch.nt, ch.pace, ch.n_stab, HQ_UP, b, t_lo, t_hi);
  const size_t NN = (size_t)N * N;
  for (int t = t_lo + (int)blockIdx.y; t <= t_hi; t += (int)gridDim.y) {
    const int l = t % ch.nt;
    const double* gt0;
    const double* g0t;
    if (t == t_hi) { gt0 = ch.Gt0; g0t = ch.G0t; }
    else { gt0 = ch.snap_t0 + l * NN; g0t = ch.snap_0t + l * NN; }
    dyn_measure(ch, gt0, g0t, l, red);
    __syncthreads();
  }
}

// at a dynamic boundary: commit the freshly built G(t,t), G(t,0), G(0,t) (in W3, W0, W4) after
// recording the signed wrap errors (src/dqmc_core.cpp:334-344), and store them into the snapshots of
// the boundary slice with the tau = 0 convention (src/dqmc_core.cpp:379-387). A chain's elements are
// spread over gridDim.y CTAs.
__global__ void __launch_bounds__(HQ_THREADS) k_dyn_commit(const HqChain* __restrict__ chains, int nchains, int b) {
  __shared__ double red[32];
  const int c = blockIdx.x;
  if (c >= nchains) return;
  const HqChain& ch = chains[c];
  if (!ch.active || b >= ch.n_stab) return;
  const int N = ch.N, NN = N * N;
  int t_lo, t_hi;
  interval_range(ch.nt, ch.pace, ch.n_stab, HQ_UP, b, t_lo, t_hi);
  const int l = t_hi % ch.nt;
  const size_t at = (size_t)l * NN;
  double ett = -INFINITY, edyn = -INFINITY;
  for (int idx = blockIdx.y * blockDim.x + threadIdx.x; idx < NN; idx += gridDim.y * blockDim.x) {
    const double ftt = ch.W3[idx];
    double ft0 = ch.W0[idx], f0t = ch.W4[idx];
    ett = fmax(ett, ftt - ch.G[idx]);
    edyn = fmax(edyn, fmax(ft0 - ch.Gt0[idx], f0t - ch.G0t[idx]));
    if (l == 0) {
      // at tau = beta the stored pair is G(0,0), G(0,0) - 1; the propagated matrices
      // are replaced likewise
      ft0 = ftt;
      f0t = ftt - (idx % N == idx / N ? 1.0 : 0.0);
    }
    ch.G[idx] = ftt;
    ch.Gt0[idx] = ft0;
    ch.G0t[idx] = f0t;
    if (ch.snap_tt) ch.snap_tt[at + idx] = ftt;
    if (ch.snap_t0) ch.snap_t0[at + idx] = ft0;
    if (ch.snap_0t) ch.snap_0t[at + idx] = f0t;
  }
  ett = block_max(ett, red);
  edyn = block_max(edyn, red);
  if (threadIdx.x == 0) {
    atomic_max_double(ch.acc + HQ_ACC_WRAP_TT, ett);
    atomic_max_double(ch.acc + HQ_ACC_WRAP_DYN, edyn);
  }
}

// ---------------------------------------------------------------------------------
//  Adjoint of log|det(1 + B(nt-1)...B(0))| (no counterpart in the reference).
//  With G_l = (1 + B_l..B_1 B_nt..B_{l+1})^-1 the G of the up sweep after slice l:
//    d/dmu    = dt sum_l tr(1 - G_l)
//    d/dalpha = sum_l sum_i s_li (1 - G_l)_ii
//    d/dE     : tr(dE E^-1 D),  D = sum_l e^{-V_l} (1 - G_l) e^{V_l}
//  A no-update up pass wraps G slice by slice and is rebuilt from the stacks every
//  `pace` slices (the checkpoints), so no slice is stored. D accumulates in W4.
// ---------------------------------------------------------------------------------
__device__ void adj_accum(const HqChain& ch, const double* G, int ld, const int8_t* s, double* red) {
  const int N = ch.N;
  double tr = 0.0, sa = 0.0;
  for (int idx = threadIdx.x; idx < N * N; idx += blockDim.x) {
    const int i = idx % N, j = idx / N;
    const double one_m = (i == j ? 1.0 : 0.0) - G[i + (size_t)j * ld];
    const double f = (s[i] > 0 ? ch.ev_m : ch.ev_p) * (s[j] > 0 ? ch.ev_p : ch.ev_m);
    ch.W4[idx] += one_m * f;
    if (i == j) { tr += one_m; sa += (s[i] > 0 ? one_m : -one_m); }
  }
  tr = block_sum(tr, red);
  sa = block_sum(sa, red);
  if (threadIdx.x == 0) {
    ch.acc[HQ_ACC_DMU] += ch.dt * tr;
    ch.acc[HQ_ACC_DALPHA] += sa;
  }
}

__global__ void __launch_bounds__(HQ_INT_THREADS, 1)
k_adj_interval(const HqChain* __restrict__ chains, int nchains, int b, int resident) {
  extern __shared__ __align__(16) double smem[];
  __shared__ HqChain ch;
  __shared__ double red[32];
  __shared__ int8_t s[HQ_MAX_N];
  const int c = blockIdx.x;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  if (!ch.active || b >= ch.n_stab) return;
  const int N = ch.N;
  int t_lo, t_hi;
  interval_range(ch.nt, ch.pace, ch.n_stab, HQ_UP, b, t_lo, t_hi);
  double* G;
  int ld;
  double* p = smem;
  if (resident) { G = p; ld = interval_ld(N); p += (size_t)N * ld; load_mat_async(G, ld, ch.G, N, N); }
  else { G = ch.G; ld = N; }
  double* stage = p;
  double* vp = stage + 8 * (pad16(N) + 4);
  double* vm = vp + N;
  __syncthreads();
  const int nsl = t_hi - t_lo + 1;
  for (int step = 0; step < nsl; ++step) {
    const int t = t_lo + step;
    const int l = t % ch.nt;
    for (int i = threadIdx.x; i < N; i += blockDim.x) s[i] = ch.fields[(size_t)l * N + i];
    __syncthreads();
    slice_factors(ch, s, vp, vm);
    __syncthreads();
    if (resident) wrap_slice<true>(ch, G, ld, vp, vm, HQ_UP, stage);
    else wrap_slice<false>(ch, G, ld, vp, vm, HQ_UP, stage);
    if (step < nsl - 1) adj_accum(ch, G, ld, s, red);
    __syncthreads();
  }
  if (resident) copy_mat(ch.G, N, G, ld, N);
}

// the last slice of interval b, after the boundary rebuilt G
__global__ void __launch_bounds__(HQ_THREADS) k_adj_last(const HqChain* __restrict__ chains, int nchains, int b) {
  __shared__ HqChain ch;
  __shared__ double red[32];
  __shared__ int8_t s[HQ_MAX_N];
  const int c = blockIdx.x;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  if (!ch.active || b >= ch.n_stab) return;
  const int N = ch.N;
  int t_lo, t_hi;
  interval_range(ch.nt, ch.pace, ch.n_stab, HQ_UP, b, t_lo, t_hi);
  const int l = t_hi % ch.nt;
  for (int i = threadIdx.x; i < N; i += blockDim.x) s[i] = ch.fields[(size_t)l * N + i];
  __syncthreads();
  adj_accum(ch, ch.G, N, s, red);
}


// zeroes D (W4) and the scalar accumulators of every chain
__global__ void __launch_bounds__(HQ_THREADS) k_adj_begin(const HqChain* __restrict__ chains, int nchains) {
  const int c = blockIdx.x;
  if (c >= nchains) return;
  const HqChain& ch = chains[c];
  for (int idx = threadIdx.x; idx < ch.N * ch.N; idx += blockDim.x) ch.W4[idx] = 0.0;
  if (threadIdx.x == 0) ch.acc[HQ_ACC_DMU] = ch.acc[HQ_ACC_DALPHA] = 0.0;
}

// log|det(1 + U D Vt)| = sum log max(D, 1) + log|det W1|, W1 = dmax^-1 U^T + dmin Vt of the full left
// stack: LU with partial pivoting (the largest |entry| of a column, the smallest row among equals),
// one CTA per chain, W1 in shared memory where it fits (it is overwritten otherwise). Bound by the
// latency of the N pivots (search, row exchange, multipliers, rank-1 update: a barrier each);
// 100 x 100: 0.1 ms for 64 chains at once, where the host's loops took 0.4 ms per chain.
__global__ void __launch_bounds__(HQ_INT_THREADS, 1)
k_logdet(const HqChain* __restrict__ chains, int nchains, double* out, int resident) {
  extern __shared__ __align__(16) double smem[];
  __shared__ HqChain ch;
  __shared__ int piv;
  const int c = blockIdx.x;
  if (c >= nchains) return;
  if (threadIdx.x == 0) ch = chains[c];
  __syncthreads();
  const int N = ch.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* f = smem;  // multipliers of a step
  double* A = resident ? smem + N : ch.W1;
  const int ld = resident ? smem_ld(N) : N;
  if (resident) load_mat_async(A, ld, ch.W1, N, N);
  const double* D = ch.stackD + (size_t)(ch.n_stab - 1) * N;
  double sum = 0.0;
  for (int k = 0; k < N; ++k) sum += threadIdx.x == 0 ? log(fmax(D[k], 1.0)) : 0.0;
  __syncthreads();
  for (int k = 0; k < N; ++k) {
    if (warp == 0) {
      double best = -1.0;
      int bi = k;
      for (int r = k + lane; r < N; r += 32) {
        const double v = fabs(A[r + (size_t)k * ld]);
        if (v > best) { best = v; bi = r; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      if (lane == 0) piv = bi;
    }
    __syncthreads();
    const int p = piv;
    if (p != k)
      for (int j = k + threadIdx.x; j < N; j += blockDim.x) {
        const double t = A[k + (size_t)j * ld];
        A[k + (size_t)j * ld] = A[p + (size_t)j * ld];
        A[p + (size_t)j * ld] = t;
      }
    __syncthreads();
    const double pv = A[k + (size_t)k * ld];
    if (threadIdx.x == 0) sum += log(fabs(pv));
    for (int r = k + 1 + threadIdx.x; r < N; r += blockDim.x) f[r] = A[r + (size_t)k * ld] / pv;
    __syncthreads();
    for (int j = k + 1 + warp; j < N; j += nw) {
      const double akj = A[k + (size_t)j * ld];
      for (int r = k + 1 + lane; r < N; r += 32) A[r + (size_t)j * ld] -= f[r] * akj;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[c] = sum;
}

// W3 = Phi o W2^T, Phi the divided differences of exp(-dt w) at the eigenvalues w of K:
// Phi_ij = (f_i - f_j) / (w_i - w_j) as f_j expm1(-dt (w_i - w_j)) / (w_i - w_j), -dt (f_i + f_j) / 2 where
// the eigenvalues coincide
__global__ void __launch_bounds__(HQ_THREADS)
k_adj_divided(const HqChain* __restrict__ chains, int nchains, const double* const* __restrict__ eig) {
  const int c = blockIdx.x;
  if (c >= nchains) return;
  const HqChain& ch = chains[c];
  const int N = ch.N;
  const double dt = ch.dt, *w = eig[c], *M = ch.W2;
  double* P = ch.W3;
  for (int j = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5); j < N; j += gridDim.y * (blockDim.x >> 5)) {
    const double wj = w[j], fj = exp(-dt * wj);
    for (int i = threadIdx.x & 31; i < N; i += 32) {
      const double d = w[i] - wj;
      const double phi = fabs(d) > 1e-10 ? fj * expm1(-dt * d) / d : -dt * 0.5 * (exp(-dt * w[i]) + fj);
      P[i + (size_t)j * N] = phi * M[j + (size_t)i * N];
    }
  }
}

// the caller's layout: per chain dmu, dalpha, dK (W3, N x N) at off[c]
__global__ void __launch_bounds__(HQ_THREADS)
k_adj_gather(const HqChain* __restrict__ chains, int nchains, const long long* __restrict__ off, double* out) {
  const int c = blockIdx.x;
  if (c >= nchains) return;
  const HqChain& ch = chains[c];
  double* o = out + off[c];
  const int stride = blockDim.x * gridDim.y, t0 = blockIdx.y * blockDim.x + threadIdx.x;
  if (t0 == 0) {
    o[0] = ch.acc[HQ_ACC_DMU];
    o[1] = ch.acc[HQ_ACC_DALPHA];
  }
  for (int idx = t0; idx < ch.N * ch.N; idx += stride) o[2 + idx] = ch.W3[idx];
}

}  // namespace hq

// =====================================================================================
//  launch wrappers (host)
// =====================================================================================
namespace hq {

size_t smem_interval_bytes(int Nmax, int kmax, bool resident) {
  return interval_smem_doubles(Nmax, kmax, resident) * sizeof(double);
}
size_t smem_udt_bytes(int Nmax, bool resident) {
  return smem_matrix_bytes(Nmax, resident, 2 * kQB * panel_ld(Nmax) + 2 * kQB * kQB + 3 * Nmax +
                                               ((Nmax - 1) / kQB) * kQB * kQB);
}
size_t smem_invert_bytes(int Nmax, bool resident) {
  return smem_matrix_bytes(Nmax, resident, 2 * kGJ * panel_ld(Nmax) + 3 * Nmax + 64);
}
// a matrix in the padded layout of the wrap, the stage of the dense exp(-dt K) and two words per site
static size_t smem_wrap_bytes(int Nmax, bool resident) {
  const size_t mat = resident ? (size_t)Nmax * interval_ld(Nmax) : 0;
  return (mat + 8 * (pad16(Nmax) + 4) + 2 * (size_t)Nmax + 64) * sizeof(double);
}
// the B chain's matrix, the stage and one word per site
static size_t smem_bchain_bytes(int Nmax, bool resident) {
  return smem_matrix_bytes(Nmax, resident, 8 * (pad16(Nmax) + 4) + Nmax + 64);
}
static size_t smem_logdet_bytes(int Nmax, bool resident) {
  return ((resident ? (size_t)Nmax * smem_ld(Nmax) : 0) + Nmax) * sizeof(double);
}
size_t smem_matrix_bytes(int Nmax, bool resident, int extra_doubles) {
  const size_t mat = resident ? (size_t)Nmax * smem_ld(Nmax) : 0;
  return (mat + (size_t)extra_doubles) * sizeof(double);
}

// The dynamic shared-memory limit of a kernel is a per-device property of the function
// shared by every context of the process: it is only ever raised, so that preparing a
// context of small chains never lowers the limit an existing context of larger chains
// launches with.
constexpr int kMaxTrackedDevices = 64;
constexpr int kTrackedKernels = 10;
static size_t g_smem_set[kMaxTrackedDevices][kTrackedKernels];
static std::mutex g_smem_mutex;  // contexts may be created by several threads at once

static cudaError_t raise_smem(int slot, const void* fn, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_smem_mutex);
  if (dev >= 0 && dev < kMaxTrackedDevices && g_smem_set[dev][slot] >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && dev >= 0 && dev < kMaxTrackedDevices) g_smem_set[dev][slot] = bytes;
  return e;
}

// sets the dynamic shared-memory limits of every per-chain kernel (outside any stream
// capture) so that chains of up to Nmax sites can be launched
// dynamic shared memory that kernel fn can take next to its own static shared memory under the
// device's per-block opt-in limit optin
static size_t smem_room(const void* fn, size_t optin) {
  cudaFuncAttributes a;
  const size_t st = cudaFuncGetAttributes(&a, fn) == cudaSuccess ? a.sharedSizeBytes : 16384;  // conservative
  return optin > st ? optin - st : 0;
}

bool interval_fits(int Nmax, int kmax, bool resident, size_t optin) {
  return smem_interval_bytes(Nmax, kmax, resident) <= smem_room(fn_interval(), optin);
}

bool matrices_fit(int Nmax, size_t optin) {
  const size_t wrap = smem_wrap_bytes(Nmax, true);
  return interval_fits(Nmax, 4, true, optin) && smem_bchain_bytes(Nmax, true) <= smem_room((const void*)k_bchain, optin) &&
         wrap <= smem_room((const void*)k_dyn_slices, optin) && wrap <= smem_room((const void*)k_adj_interval, optin) &&
         smem_invert_bytes(Nmax, true) <= smem_room(fn_invert(), optin) &&
         smem_udt_bytes(Nmax, true) <= smem_room(fn_udt(), optin);
}

cudaError_t prepare_kernels(int Nmax, int kmax, bool resident) {
  const size_t wrap = smem_wrap_bytes(Nmax, resident);
  cudaError_t e;
  if ((e = raise_smem(0, fn_interval(), smem_interval_bytes(Nmax, kmax, resident))) != cudaSuccess) return e;
  if ((e = raise_smem(1, (const void*)k_bchain, smem_bchain_bytes(Nmax, resident))) != cudaSuccess) return e;
  if ((e = raise_smem(2, fn_udt(), smem_udt_bytes(Nmax, resident))) != cudaSuccess) return e;
  if ((e = raise_smem(3, fn_invert(), smem_invert_bytes(Nmax, resident))) != cudaSuccess) return e;
  if ((e = raise_smem(4, (const void*)k_dyn_slices, wrap)) != cudaSuccess) return e;
  if ((e = raise_smem(5, (const void*)k_adj_interval, wrap)) != cudaSuccess) return e;
  return raise_smem(8, (const void*)k_logdet, smem_logdet_bytes(Nmax, resident));
}

cudaError_t prepare_interval_cl() {
  const cudaError_t e = raise_smem(6, fn_interval_cl(), smem_interval_cl_bytes());
  if (e != cudaSuccess) return e;
  return raise_smem(7, fn_bchain_cols(), smem_bchain_cols_bytes());
}

cudaError_t prepare_sweep(int Nmax, int kmax) { return raise_smem(9, fn_sweep(), smem_sweep_bytes(Nmax, kmax)); }

cudaError_t launch_bchain(const HqChain* chains, int n, int dir, int b, int Nmax, bool resident, cudaStream_t st) {
  const size_t bytes = smem_bchain_bytes(Nmax, resident);
  k_bchain<<<n, HQ_INT_THREADS, bytes, st>>>(chains, n, dir, b, resident ? 1 : 0);
  return cudaGetLastError();
}
cudaError_t launch_measure(const HqChain* chains, int n, int dir, int b, int flags, cudaStream_t st) {
  k_measure<<<n, HQ_THREADS, 0, st>>>(chains, n, dir, b, flags);
  return cudaGetLastError();
}
cudaError_t launch_dyn_start(const HqChain* chains, int n, cudaStream_t st) {
  k_dyn_start<<<n, 256, 0, st>>>(chains, n);
  return cudaGetLastError();
}
cudaError_t launch_dyn_slices(const HqChain* chains, int n, int b, int flags, int Nmax, bool resident, cudaStream_t st) {
  const size_t bytes = smem_wrap_bytes(Nmax, resident);
  dim3 grid(n, 3);
  k_dyn_slices<<<grid, HQ_INT_THREADS, bytes, st>>>(chains, n, b, flags, resident ? 1 : 0);
  return cudaGetLastError();
}
cudaError_t launch_dyn_measure(const HqChain* chains, int n, int b, int pace, cudaStream_t st) {
  k_dyn_measure<<<dim3(n, std::min(pace, 32)), HQ_THREADS, 0, st>>>(chains, n, b);
  return cudaGetLastError();
}
cudaError_t launch_adj_interval(const HqChain* chains, int n, int b, int Nmax, bool resident, cudaStream_t st) {
  const size_t bytes = smem_wrap_bytes(Nmax, resident);
  k_adj_interval<<<n, HQ_INT_THREADS, bytes, st>>>(chains, n, b, resident ? 1 : 0);
  return cudaGetLastError();
}
cudaError_t launch_adj_begin(const HqChain* chains, int n, cudaStream_t st) {
  k_adj_begin<<<n, HQ_THREADS, 0, st>>>(chains, n);
  return cudaGetLastError();
}
cudaError_t launch_logdet(const HqChain* chains, int n, double* out, int Nmax, bool resident, cudaStream_t st) {
  k_logdet<<<n, HQ_INT_THREADS, smem_logdet_bytes(Nmax, resident), st>>>(chains, n, out, resident ? 1 : 0);
  return cudaGetLastError();
}
cudaError_t launch_adj_divided(const HqChain* chains, int n, const double* const* eig, cudaStream_t st) {
  k_adj_divided<<<dim3(n, 4), HQ_THREADS, 0, st>>>(chains, n, eig);
  return cudaGetLastError();
}
cudaError_t launch_adj_gather(const HqChain* chains, int n, const long long* off, double* out, cudaStream_t st) {
  k_adj_gather<<<dim3(n, 4), HQ_THREADS, 0, st>>>(chains, n, off, out);
  return cudaGetLastError();
}
cudaError_t launch_adj_last(const HqChain* chains, int n, int b, cudaStream_t st) {
  k_adj_last<<<n, HQ_THREADS, 0, st>>>(chains, n, b);
  return cudaGetLastError();
}
cudaError_t launch_dyn_commit(const HqChain* chains, int n, int b, int Nmax, cudaStream_t st) {
  const int parts = std::max(1, std::min(8, Nmax * Nmax / 4096));
  k_dyn_commit<<<dim3(n, parts), HQ_THREADS, 0, st>>>(chains, n, b);
  return cudaGetLastError();
}

// Copies every chain's accumulator block into one chain-major buffer, so that a single
// device-to-host copy reads the estimators of all chains.
__global__ void k_gather_acc(const HqChain* chains, int n, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * HQ_ACC_COUNT) return;
  const int c = i / HQ_ACC_COUNT;
  out[i] = chains[c].acc[i - c * HQ_ACC_COUNT];
}
cudaError_t launch_gather_acc(const HqChain* chains, int n, double* out, cudaStream_t st) {
  const int total = n * HQ_ACC_COUNT;
  k_gather_acc<<<(total + 255) / 256, 256, 0, st>>>(chains, n, out);
  return cudaGetLastError();
}

}  // namespace hq

