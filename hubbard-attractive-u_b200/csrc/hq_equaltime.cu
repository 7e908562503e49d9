// hq_equaltime.cu -- k_equaltime: the equal-time G(0,0) = (1 + B(nt-1)...B(0))^-1 of one chain of up to
// 64 sites in ONE launch (src/dqmc_core.cpp:67-97, include/utils/stable_numerics.hpp:186-239), for
// the entry point that allocates nothing.
#include <atomic>

#include "hq_cta_gemm.cuh"
#include "hq_invert.cuh"
#include "hq_phases.cuh"
#include "hq_udt.cuh"

namespace hq {

// One CTA of 16 warps does what the launch sequence of hq_init_stacks_and_g does, phase after phase,
// with the same arithmetic: per interval the B chain, the UDV push (X stays in shared memory) and the
// cumulative V^T; then the builder with an empty left stack, whose products with the identity are
// left out (they change no bit): W1 = U_R drmax^-1 + Vt_R^T drmin, its inverse, G = U_R drmax^-1 W1^-1.
// What bounds it: the latency of one chain's reflectors, pivots and passes on one SM. As 4 + 3 n_stab
// launches with six uploads a 4x4, nt = 40 call took 215 us, 111 us this way.
constexpr int kEqMaxN = 64;
constexpr size_t kEqSmem =
    sizeof(double) * (cta_gemm_doubles(kEqMaxN, kEqMaxN) > (size_t)kEqMaxN * smem_ld(kEqMaxN) + 2 * kQB * panel_ld(kEqMaxN) +
                                                               2 * kQB * kQB + 3 * kEqMaxN + 4 * kQB * kQB + 64
                          ? cta_gemm_doubles(kEqMaxN, kEqMaxN)
                          : (size_t)kEqMaxN * smem_ld(kEqMaxN) + 2 * kQB * panel_ld(kEqMaxN) + 2 * kQB * kQB + 3 * kEqMaxN +
                                4 * kQB * kQB + 64);

__global__ void __launch_bounds__(HQ_THREADS, 1) k_equaltime(const __grid_constant__ HqChain chain) {
  extern __shared__ __align__(16) double smem[];
  __shared__ HqChain ch;
  __shared__ PivotMoves mv;
  __shared__ double red[96];
  __shared__ double pv[2];
  __shared__ HqGemmJob job;
  if (threadIdx.x == 0) {
    ch = chain;
    HqGemmJob j{};
    j.M = j.Nc = j.K = j.lda = j.ldb = j.ldc = chain.N;
    j.alpha = 1.0;
    j.active = 1;
    job = j;
  }
  if (threadIdx.x < HQ_ACC_COUNT) chain.acc[threadIdx.x] = 0.0;
  __syncthreads();
  const int N = ch.N;
  const size_t NN = (size_t)N * N;
  double* Vt = ch.stackVt + (size_t)ch.n_stab * NN;  // the right stack
  for (int b = 0; b < ch.n_stab; ++b) {
    bchain_body(ch, HQ_DOWN, b, true, smem, true);
    __syncthreads();
    udt_body<1>(ch, 1, b, true, smem, mv, true);
    __syncthreads();
    if (b == 0) {
      for (int k = threadIdx.x; k < N * N; k += blockDim.x) Vt[k] = ch.W0[k];
    } else {
      if (threadIdx.x == 0) {
        job.A = ch.W0;
        job.B = Vt + (b - 1) * NN;
        job.C = Vt + b * NN;
      }
      __syncthreads();
      gemm_cta(job, smem, red);
    }
    __syncthreads();
  }
  const size_t top = (size_t)ch.n_stab + ch.n_stab - 1;
  const double *UR = ch.stackU + top * NN, *DR = ch.stackD + top * N, *VR = ch.stackVt + top * NN;
  for (int j = threadIdx.x >> 5; j < N; j += blockDim.x >> 5) {
    const double dmax = vscale(DR, 2, j), dmin = vscale(DR, 3, j);
    for (int i = threadIdx.x & 31; i < N; i += 32)
      ch.W1[i + (size_t)j * N] = __dadd_rn(__dmul_rn(UR[i + (size_t)j * N], dmax), __dmul_rn(VR[j + (size_t)i * N], dmin));
  }
  __syncthreads();
  invert_body<1>(ch, 0, true, smem, pv);
  if (threadIdx.x == 0) {
    job.A = UR;
    job.B = ch.W1;
    job.C = ch.G;
    job.ks = DR;
    job.ks_mode = 2;
  }
  __syncthreads();
  gemm_cta(job, smem, red);
}

cudaError_t launch_equaltime(const HqChain& chain, cudaStream_t st) {
  static std::atomic<bool> ready[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !ready[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute((const void*)k_equaltime, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEqSmem);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) ready[dev].store(true, std::memory_order_release);
  }
  k_equaltime<<<1, HQ_THREADS, kEqSmem, st>>>(chain);
  return cudaGetLastError();
}

}  // namespace hq
