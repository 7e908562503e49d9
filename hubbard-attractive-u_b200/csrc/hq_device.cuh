// hq_device.cuh -- device helpers of the sm_100a DQMC kernels:
//   * the reference's random stream (std::default_random_engine = minstd_rand0 and
//     std::bernoulli_distribution / generate_canonical<double,53> of libstdc++),
//     replayed exactly with jump-ahead so every site of a slice gets its uniform at once;
//   * FP64 tensor-core (DMMA, mma.sync m16n8k4 .f64) fragment helpers;
//   * the dense (DMMA) exp(-dt K) application;
//   * block reductions.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "hq_types.h"

namespace hq {

// ------------------------------------------------------------------------------------
//  minstd_rand0: x <- 16807 x mod (2^31 - 1)   (libstdc++ default_random_engine,
//  src/random.cpp:14). generate_canonical<double, 53> draws two values:
//     sum = (x1 - 1) + (x2 - 1) * R ;  ret = sum / round(R*R) ;  R = 2147483646
//  with plain IEEE double operations (no contraction), clamped below 1.
// ------------------------------------------------------------------------------------
constexpr uint32_t kMinstdA = 16807u;
constexpr uint32_t kMinstdM = 2147483647u;

// a * x mod m for a, x < m = 2^31 - 1, exactly, without a division: with t = a x =
// hi 2^31 + lo and 2^31 = 1 (mod m), t = lo + hi (mod m); two folds leave a value <= m + 1
__host__ __device__ inline uint32_t minstd_mulmod(uint64_t a, uint64_t x) {
  const uint64_t t = a * x;
  uint64_t r = (t & kMinstdM) + (t >> 31);
  r = (r & kMinstdM) + (r >> 31);
  return static_cast<uint32_t>(r >= kMinstdM ? r - kMinstdM : r);
}
// a^k mod m
__host__ __device__ inline uint32_t minstd_pow(uint64_t k) {
  uint64_t result = 1, base = kMinstdA;
  while (k) {
    if (k & 1) result = minstd_mulmod(result, base);
    base = minstd_mulmod(base, base);
    k >>= 1;
  }
  return static_cast<uint32_t>(result);
}

__device__ inline double canonical_from_pair(uint32_t x1, uint32_t x2) {
  const double R = 2147483646.0;
  const double RR = __dmul_rn(R, R);
  const double sum = __dadd_rn((double)(x1 - 1u), __dmul_rn((double)(x2 - 1u), R));
  double r = __ddiv_rn(sum, RR);
  if (r >= 1.0) r = 0.99999999999999988898;  // nextafter(1.0, 0.0)
  return r;
}

// ------------------------------------------------------------------------------------
//  DMMA m16n8k4 (FP64). Fragment ownership (lane = 4*g + q):
//    A (16x4, row): a0 = A[g][q], a1 = A[g+8][q]
//    B (4x8,  col): b0 = B[q][g]
//    C (16x8)     : c0 = C[g][2q], c1 = C[g][2q+1], c2 = C[g+8][2q], c3 = C[g+8][2q+1]
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void dmma_16x8x4(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// the warp's index as a value the compiler knows to be the same in all its lanes, so that branches
// on it need no reconvergence
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// ------------------------------------------------------------------------------------
//  Reductions
// ------------------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// block-wide sum; red must hold >= 32 doubles; result valid in all threads
__device__ inline double block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double t = (lane < nw) ? red[lane] : 0.0;
  t = warp_sum(t);
  return t;
}
__device__ inline double block_max(double v, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double t = (lane < nw) ? red[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

// three block-wide sums in one reduction round (2 barriers)
__device__ inline void block_sum3(double& a, double& b, double& c, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  a = warp_sum(a); b = warp_sum(b); c = warp_sum(c);
  __syncthreads();
  if (lane == 0) { red[w] = a; red[32 + w] = b; red[64 + w] = c; }
  __syncthreads();
  a = warp_sum(lane < nw ? red[lane] : 0.0);
  b = warp_sum(lane < nw ? red[32 + lane] : 0.0);
  c = warp_sum(lane < nw ? red[64 + lane] : 0.0);
}

// adds one slice's equal-time estimators to acc from this thread's partial sums of
// tr = sum_i G_ii, dd = sum_i (1 - G_ii)^2 and sq = sum_ij G_ij^2 (include/observable_methods.hpp:39-83)
__device__ inline void measure_commit(double tr, double dd, double sq, int N, double* acc, double* red) {
  block_sum3(tr, dd, sq, red);
  if (threadIdx.x == 0) {
    acc[HQ_ACC_FILLING] += 2.0 - 2.0 * tr / N;
    acc[HQ_ACC_DOCC] += dd / N;
    acc[HQ_ACC_SWAVE] += (2.0 * sq - 2.0 * tr + N) / N;
    acc[HQ_ACC_NSLICE] += 1.0;
  }
}

// Element loops over an N x N column-major matrix without integer division: warps walk
// the columns, lanes the rows (consecutive lanes touch consecutive addresses).
#define HQ_FOR_EACH_ELEM(N, i, j)                                                      \
  for (int j = (int)(threadIdx.x >> 5); j < (N); j += (int)(blockDim.x >> 5))          \
    for (int i = (int)(threadIdx.x & 31); i < (N); i += 32)

// atomic max on doubles (ordered-int trick; values may be negative)
__device__ inline void atomic_max_double(double* addr, double val) {
  unsigned long long* p = reinterpret_cast<unsigned long long*>(addr);
  unsigned long long old = *p, assumed;
  do {
    assumed = old;
    if (__longlong_as_double(assumed) >= val) return;
    old = atomicCAS(p, assumed, __double_as_longlong(val));
  } while (old != assumed);
}

// ------------------------------------------------------------------------------------
//  Dense exp(-dt K) application with DMMA, M in shared (or global) memory, E in global
//  (L2-resident: shared by every chain of the same parameters).
//  dense_apply:       M <- E M, by column blocks (E M[:, blk] needs only blk)
//  dense_apply_right: M <- M E, by row blocks    (M[blk, :] E needs only blk)
//  E is symmetric here (K real symmetric), so op(E) = E in both cases.
//  stage: shared scratch of >= 2 * (N16 * 8) doubles used to stage k-chunks of E.
//  The output of a block is accumulated in registers (<= kMaxFrag fragments per warp).
// ------------------------------------------------------------------------------------
constexpr int kMaxFrag = 8;

__device__ inline void dense_apply(double* M, int ld, int N, const double* __restrict__ E, double* stage) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int N16 = (N + 15) & ~15;       // padded row count
  const int mt = N16 / 16;              // 16-row tiles
  const int max_tiles = kMaxFrag * nwarps;
  int cb8 = max_tiles / mt;             // 8-wide column tiles per block
  if (cb8 < 1) cb8 = 1;
  const int nt8 = (N + 7) / 8;
  if (cb8 > nt8) cb8 = nt8;
  const int CB = cb8 * 8;
  const int lds = N16 + 4;              // stage leading dimension
  for (int c0 = 0; c0 < N; c0 += CB) {
    const int tiles = mt * cb8;
    double acc[kMaxFrag][4];
#pragma unroll
    for (int f = 0; f < kMaxFrag; ++f) acc[f][0] = acc[f][1] = acc[f][2] = acc[f][3] = 0.0;
    for (int k0 = 0; k0 < N; k0 += 8) {
      // stage[kk * lds + r] = E[r, k0 + kk]
      __syncthreads();
      for (int kk = threadIdx.x >> 5; kk < 8; kk += blockDim.x >> 5)
        for (int r = threadIdx.x & 31; r < N16; r += 32) {
          const int k = k0 + kk;
          stage[kk * lds + r] = (r < N && k < N) ? E[r + (size_t)k * N] : 0.0;
        }
      __syncthreads();
#pragma unroll
      for (int f = 0; f < kMaxFrag; ++f) {
        const int tile = warp + f * nwarps;
        if (tile < tiles) {
          const int tm = tile % mt, tn = tile / mt;
          const int r = tm * 16 + g;
          const int cc = c0 + tn * 8 + g;
#pragma unroll
          for (int ks = 0; ks < 8; ks += 4) {
            const int k = k0 + ks + q;
            const double a0 = stage[(ks + q) * lds + r];
            const double a1 = stage[(ks + q) * lds + r + 8];
            const double b0 = (k < N && cc < N) ? M[k + (size_t)cc * ld] : 0.0;
            dmma_16x8x4(acc[f], a0, a1, b0);
          }
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int f = 0; f < kMaxFrag; ++f) {
      const int tile = warp + f * nwarps;
      if (tile < tiles) {
        const int tm = tile % mt, tn = tile / mt;
        const int r = tm * 16 + g, c = c0 + tn * 8 + 2 * q;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int rr = r + ((e & 2) ? 8 : 0), cc = c + (e & 1);
          if (rr < N && cc < N && cc < c0 + CB) M[rr + (size_t)cc * ld] = acc[f][e];
        }
      }
    }
    __syncthreads();
  }
}

// side-1 dense application uses row blocks of height CB where the tiles enumerate
// (8-col tiles over all N) x (16-row tiles inside the block); keep the block height a
// multiple of 16 and the tile count within kMaxFrag * nwarps.
__device__ inline void dense_apply_right(double* M, int ld, int N, const double* __restrict__ E, double* stage) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int N8 = (N + 7) & ~7;
  const int nt8 = N8 / 8;                // 8-col tiles over all columns
  const int max_tiles = kMaxFrag * nwarps;
  int rb16 = max_tiles / nt8;            // 16-row tiles per block
  if (rb16 < 1) rb16 = 1;
  const int mt16 = (N + 15) / 16;
  if (rb16 > mt16) rb16 = mt16;
  const int RB = rb16 * 16;
  const int lds = N8 + 4;
  for (int r0 = 0; r0 < N; r0 += RB) {
    const int tiles = nt8 * rb16;
    double acc[kMaxFrag][4];
#pragma unroll
    for (int f = 0; f < kMaxFrag; ++f) acc[f][0] = acc[f][1] = acc[f][2] = acc[f][3] = 0.0;
    for (int k0 = 0; k0 < N; k0 += 8) {
      __syncthreads();
      // stage[kk * lds + c] = E[k0+kk, c]
      for (int kk = threadIdx.x >> 5; kk < 8; kk += blockDim.x >> 5)
        for (int c = threadIdx.x & 31; c < N8; c += 32) {
          const int k = k0 + kk;
          stage[kk * lds + c] = (c < N && k < N) ? E[k + (size_t)c * N] : 0.0;
        }
      __syncthreads();
#pragma unroll
      for (int f = 0; f < kMaxFrag; ++f) {
        const int tile = warp + f * nwarps;
        if (tile < tiles) {
          const int tc = tile % nt8, tr = tile / nt8;
#pragma unroll
          for (int ks = 0; ks < 8; ks += 4) {
            const int k = k0 + ks + q;
            const int r = r0 + tr * 16 + g;
            const double a0 = (r < N && k < N) ? M[r + (size_t)k * ld] : 0.0;
            const double a1 = (r + 8 < N && k < N) ? M[r + 8 + (size_t)k * ld] : 0.0;
            const double b0 = stage[(ks + q) * lds + tc * 8 + g];
            dmma_16x8x4(acc[f], a0, a1, b0);
          }
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int f = 0; f < kMaxFrag; ++f) {
      const int tile = warp + f * nwarps;
      if (tile < tiles) {
        const int tc = tile % nt8, tr = tile / nt8;
        const int r = r0 + tr * 16 + g, c = tc * 8 + 2 * q;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int rr = r + ((e & 2) ? 8 : 0), cc = c + (e & 1);
          if (rr < N && cc < N && rr < r0 + RB) M[rr + (size_t)cc * ld] = acc[f][e];
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace hq
