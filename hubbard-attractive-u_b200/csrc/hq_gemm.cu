// hq_gemm.cu -- k_gemm, the batched FP64 DMMA GEMM of the G builders
// (include/utils/stable_numerics.hpp:186-324) with the wrap-error epilogue (:37-48).
#include "hq_common.cuh"

namespace hq {

// ---------------------------------------------------------------------------------
//  k_gemm: batched C = alpha op(A) diag(ks) op(B) (row / column scalings, beta, wrap-error
//  epilogue), one CTA per T x T tile of one job; K streams through shared memory in chunks of 16
//  with cp.async double buffering. Shared layouts keep the fragment loads free of bank conflicts
//  for either transpose:
//    op(A) = A   : sA[k * ldm + m]     op(A) = A^T : sA[m * ldk + k]     ldm, ldk = 4 (mod 16)
//    op(B) = B   : sB[n * ldk + k]     op(B) = B^T : sB[k * ldm + n]
//  One copy of the body per transpose case and with or without k-scalings: with the cases decided
//  inside the inner loop, its address selections took as long as its DMMAs (256 products of 144^3,
//  plain: 116 us, 72 us now, 21.2 of 35.5 TFLOP/s). Four CTAs of the 48 x 48 tile per SM spill a few words in the
//  epilogue and are faster all the same (4.5 against 5.2 ms a sweep of 256 12 x 12 chains with three).
//  Tiles: 48 x 48 with six warps of 16 x 24 (144 = 3 x 48), or 64 x 64 with eight warps of 16 x 32
//  where that pads the matrices less (launch_gemm): 256 products of 64^3 12.6 against 20.8 us, 32 of
//  256^3 55.6 against 59.7 us; larger tiles and fewer, larger warp blocks were slower for 144^3 (48 x 72
//  92 us, 48 x 96 97 us, two warps of 48 x 24 116 us).
// ---------------------------------------------------------------------------------
constexpr int kGKc = 16, kGLdk = kGKc + 4;

// copies 2 doubles (16 B) with zero fill of the invalid part; both addresses 16-byte aligned
__device__ __forceinline__ void cp_async_pair(double* dst, const double* src, int nvalid) {
  const unsigned saddr = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  const int nbytes = nvalid <= 0 ? 0 : (nvalid >= 2 ? 16 : 8);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(src), "r"(nbytes));
}

// stages the chunk [k0, k0 + 16) x [r0, r0 + T) of op(X) (r = m for A, n for B; R rows).
// KMAJ: op(X) is contiguous along k in memory (A^T or B) -> layout [r][k]; otherwise
// contiguous along r -> layout [k][r]. `pair` selects 16-byte copies (even ld, aligned base).
template <bool KMAJ, int T, int NTH>
__device__ __forceinline__ void g_stage(const double* X, int ldx, int R, int K, int r0, int k0, double* sX, bool pair) {
  constexpr int LDM = panel_ld(T);
  if (pair) {
#pragma unroll
    for (int idx = threadIdx.x; idx < T * (kGKc / 2); idx += NTH) {
      const int r = KMAJ ? idx / (kGKc / 2) : 2 * (idx % (T / 2)), k = KMAJ ? 2 * (idx % (kGKc / 2)) : idx / (T / 2);
      const int nv = KMAJ ? ((r0 + r < R) ? min(2, K - (k0 + k)) : 0) : ((k0 + k < K) ? min(2, R - (r0 + r)) : 0);
      const size_t go = KMAJ ? (k0 + k) + (size_t)(r0 + r) * ldx : (r0 + r) + (size_t)(k0 + k) * ldx;
      cp_async_pair(KMAJ ? sX + r * kGLdk + k : sX + k * LDM + r, nv > 0 ? X + go : X, nv);
    }
  } else {
    for (int idx = threadIdx.x; idx < T * kGKc; idx += NTH) {
      const int r = KMAJ ? idx / kGKc : idx % T, k = KMAJ ? idx % kGKc : idx / T;
      const bool ok = k0 + k < K && r0 + r < R;
      const size_t go = KMAJ ? (k0 + k) + (size_t)(r0 + r) * ldx : (r0 + r) + (size_t)(k0 + k) * ldx;
      cp_async_8(KMAJ ? sX + r * kGLdk + k : sX + k * LDM + r, ok ? X + go : X, ok);
    }
  }
}

template <int T>
struct GemmTile;
template <>
struct GemmTile<48> { static constexpr int WM = 3, WN = 2, CTAS = 4; };  // warps along m, n; CTAs per SM
template <>
struct GemmTile<64> { static constexpr int WM = 4, WN = 2, CTAS = 2; };
template <int T>
constexpr int kGThreads = GemmTile<T>::WM* GemmTile<T>::WN * 32;
template <int T>
constexpr int kGStage = (panel_ld(T) * kGKc > T * kGLdk) ? panel_ld(T) * kGKc : T * kGLdk;  // doubles

template <int T, bool AMAJ, bool BMAJ, bool KS>
__device__ __forceinline__ void gemm_tile(const HqGemmJob& J, int m0, int n0, double* sA, double* sB, double* sK, double* red) {
  constexpr int NTH = kGThreads<T>, NI = T / GemmTile<T>::WN / 8, LDM = panel_ld(T), SX = kGStage<T>;
  const bool pa = (J.lda % 2 == 0) && ((reinterpret_cast<uintptr_t>(J.A) & 15) == 0);
  const bool pb = (J.ldb % 2 == 0) && ((reinterpret_cast<uintptr_t>(J.B) & 15) == 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int wm = (warp % GemmTile<T>::WM) * 16, wn = (warp / GemmTile<T>::WM) * 8 * NI;
  double acc[NI][4];
#pragma unroll
  for (int j = 0; j < NI; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
  const int nchunks = (J.K + kGKc - 1) / kGKc;
  auto stage = [&](int c) {
    if (c < nchunks) {
      const int k0 = c * kGKc, buf = c & 1;
      g_stage<AMAJ, T, NTH>(J.A, J.lda, J.M, J.K, m0, k0, sA + buf * SX, pa);
      g_stage<BMAJ, T, NTH>(J.B, J.ldb, J.Nc, J.K, n0, k0, sB + buf * SX, pb);
      if (KS && threadIdx.x < kGKc)
        sK[buf * kGKc + threadIdx.x] = (k0 + (int)threadIdx.x < J.K) ? vscale(J.ks, J.ks_mode, k0 + threadIdx.x) : 0.0;
    }
    cp_async_commit();
  };
  stage(0);
  for (int c = 0; c < nchunks; ++c) {
    stage(c + 1);
    cp_async_wait<1>();
    __syncthreads();
    const double* A_ = sA + (c & 1) * SX + (AMAJ ? (wm + g) * kGLdk + q : q * LDM + wm + g);
    const double* B_ = sB + (c & 1) * SX + (BMAJ ? (wn + g) * kGLdk + q : q * LDM + wn + g);
    const double* K_ = sK + (c & 1) * kGKc + q;
#pragma unroll
    for (int kk = 0; kk < kGKc; kk += 4) {
      double a0 = AMAJ ? A_[kk] : A_[kk * LDM];
      double a1 = AMAJ ? A_[8 * kGLdk + kk] : A_[kk * LDM + 8];
      if (KS) {
        a0 *= K_[kk];
        a1 *= K_[kk];
      }
#pragma unroll
      for (int j = 0; j < NI; ++j) dmma_16x8x4(acc[j], a0, a1, BMAJ ? B_[8 * j * kGLdk + kk] : B_[kk * LDM + 8 * j]);
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  // epilogue: alpha, row / column scalings, beta, wrap-error maximum. A thread's two rows and 2 NI
  // columns take one scaling each (divisions among them) instead of a pair per element, and the old
  // values are loaded before the first store.
  double emax = -INFINITY;
  double rsv[2], old[NI][4];
  const bool load_old = J.beta != 0.0 || J.epi == 1;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int gm = m0 + wm + g + 8 * h;
    rsv[h] = gm < J.M ? vscale(J.rs, J.rs_mode, gm) : 0.0;
  }
#pragma unroll
  for (int j = 0; j < NI; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int gm = m0 + wm + g + ((e & 2) ? 8 : 0);
      const int gn = n0 + wn + j * 8 + 2 * q + (e & 1);
      old[j][e] = (load_old && gm < J.M && gn < J.Nc) ? J.C[gm + (size_t)gn * J.ldc] : 0.0;
    }
#pragma unroll
  for (int j = 0; j < NI; ++j) {
    double csv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int gn = n0 + wn + j * 8 + 2 * q + h;
      csv[h] = gn < J.Nc ? vscale(J.cs, J.cs_mode, gn) : 0.0;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int gm = m0 + wm + g + ((e & 2) ? 8 : 0);
      const int gn = n0 + wn + j * 8 + 2 * q + (e & 1);
      if (gm < J.M && gn < J.Nc) {
        double v = J.alpha * acc[j][e] * rsv[e >> 1] * csv[e & 1];
        if (J.beta != 0.0) v = fma(J.beta, old[j][e], v);
        if (J.epi == 1) emax = fmax(emax, v - old[j][e]);
        J.C[gm + (size_t)gn * J.ldc] = v;
      }
    }
  }
  if (J.epi == 1 && J.err_out) {
    emax = block_max(emax, red);
    if (threadIdx.x == 0) atomic_max_double(J.err_out, emax);
  }
}

// Up to three job lists of n jobs each in one launch (products that do not depend on each other: the
// push with the first builder product, the displaced builder's in two rounds), so that a sweep's
// interval has four instead of five of these launches and a dynamic one five instead of eight.
template <int T>
__global__ void __launch_bounds__(kGThreads<T>, GemmTile<T>::CTAS)
k_gemm(HqGemmLists lists, int tiles_n) {
  __shared__ __align__(16) double sA[2 * kGStage<T>];
  __shared__ __align__(16) double sB[2 * kGStage<T>];
  __shared__ double sK[2 * kGKc];
  __shared__ double red[32];
  __shared__ HqGemmJob J;
  static_assert(sizeof(HqGemmJob) == 128, "16 words of 8 bytes");
  const int li = blockIdx.z, jb = blockIdx.y;
  if (threadIdx.x < 16) {
    const HqGemmJob* src = (li == 0 ? lists.l[0] : (li == 1 ? lists.l[1] : lists.l[2])) + jb;
    reinterpret_cast<unsigned long long*>(&J)[threadIdx.x] = reinterpret_cast<const unsigned long long*>(src)[threadIdx.x];
  }
  __syncthreads();
  if (!J.active) return;
  const int m0 = (blockIdx.x / tiles_n) * T, n0 = (blockIdx.x % tiles_n) * T;
  if (m0 >= J.M || n0 >= J.Nc) return;
  // op(A) = A^T and op(B) = B are contiguous along k
  auto run = [&](auto am, auto bm) {
    constexpr bool AM = decltype(am)::value != 0, BM = decltype(bm)::value != 0;
    if (J.ks_mode != 0) gemm_tile<T, AM, BM, true>(J, m0, n0, sA, sB, sK, red);
    else gemm_tile<T, AM, BM, false>(J, m0, n0, sA, sB, sK, red);
  };
  if (J.ta) {
    if (J.tb == 0) run(IntC<1>{}, IntC<1>{});
    else run(IntC<1>{}, IntC<0>{});
  } else {
    if (J.tb == 0) run(IntC<0>{}, IntC<1>{});
    else run(IntC<0>{}, IntC<0>{});
  }
}

cudaError_t launch_gemm(const HqGemmLists& lists, int nlists, int njobs, int Mmax, int Nmax, cudaStream_t st) {
  if (njobs <= 0 || nlists <= 0) return cudaSuccess;
  // the tile that pads the largest matrix least, 48 at equal padding
  auto padded = [&](int t) { return ((Mmax + t - 1) / t) * t * (((Nmax + t - 1) / t) * t); };
  const int t = padded(64) < padded(48) ? 64 : 48;
  const int tm = (Mmax + t - 1) / t, tn = (Nmax + t - 1) / t;
  const dim3 grid(tm * tn, njobs, nlists);  // up to 65535 jobs per list
  if (t == 64) k_gemm<64><<<grid, kGThreads<64>, 0, st>>>(lists, tn);
  else k_gemm<48><<<grid, kGThreads<48>, 0, st>>>(lists, tn);
  return cudaGetLastError();
}
cudaError_t launch_gemm(const HqGemmJob* jobs, int njobs, int Mmax, int Nmax, cudaStream_t st) {
  return launch_gemm(HqGemmLists{{jobs, nullptr, nullptr}}, 1, njobs, Mmax, Nmax, st);
}

}  // namespace hq
