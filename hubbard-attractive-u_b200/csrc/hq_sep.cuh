// hq_sep.cuh -- the separable exp(-dt K) of the L x L torus, exp(-dt K) = e^{dt mu} A (x) A with A
// circulant (src/square_lattice.cpp:30-61, src/hubbard.cpp:41-47), applied to a matrix by length-L
// circular convolutions along x and along y, with the diagonal e^{+-V} and the equal-time
// estimators riding on the passes.
#pragma once
#include "hq_device.cuh"

namespace hq {

// ------------------------------------------------------------------------------------
//  A pass applies the L-point circulant to the fibres of one lattice direction of one side:
//    side 0 (rows):    sites are rows,    a fibre is L rows of one column
//    side 1 (columns): sites are columns, a fibre is L columns of one row
//    pass 0: along x (sites L o + e), pass 1: along y (sites o + L e)
//  What bounds it: at 12 x 12 a pass reads and writes 20736 doubles of shared memory (2 x 1300
//  cycles at 128 B per clock) and takes 144 multiply-adds per fibre (3900 cycles of the SM's FP64
//  pipe). Two rows per thread move as 16-byte words, which at a leading dimension = 2 (mod 16) are
//  free of bank conflicts also where the lanes walk columns, and N and the leading dimension are
//  compile-time values: the four passes of a 12 x 12 wrap take 28k cycles (8 warps), 40k with both
//  known only at run time and 8-byte words.
//  Every output is a sum over its fibre in ascending order of the inputs, whatever the layout: the
//  sums are not regrouped (an even-odd split of the circulant saves a third of the products but
//  rounds differently, and a wrapped G amplifies differences of rounding by up to 1e12 before
//  the next stabilisation at large beta).
// ------------------------------------------------------------------------------------

// v <- A v for one fibre
template <int L>
__device__ __forceinline__ void sep_conv(const double (&a)[L], double (&v)[L]) {
  double acc[L];
#pragma unroll
  for (int e = 0; e < L; ++e) acc[e] = fma(a[e], v[0], 0.0);
#pragma unroll
  for (int f = 1; f < L; ++f)
#pragma unroll
    for (int e = 0; e < L; ++e) acc[e] = fma(a[(e - f + L) % L], v[f], acc[e]);
#pragma unroll
  for (int e = 0; e < L; ++e) v[e] = acc[e];
}

// estimator sums of a thread (see measure_commit)
struct SepMeas {
  double tr = 0.0, dd = 0.0, sq = 0.0;
  __device__ __forceinline__ void add(double v, bool diag) {
    sq = fma(v, v, sq);
    if (diag) { tr += v; dd += (1.0 - v) * (1.0 - v); }
  }
};

// One pass over the NCOL columns [0, NCOL) of M (leading dimension LD, or ld where LD = 0; N = L L
// rows). Pass 1 multiplies its results by c. SC scales on load (1) or on store (2), after c: with
// sl null by sc[i] at site i, otherwise by the product sl[line] sc[i], line the index on the other
// side. MEAS adds the estimator sums of the matrix as loaded (1) or as stored (2). Side 1 in pass 0
// needs NCOL a multiple of L, in pass 1 all N columns; side-1 sites and side-0 lines are indexed
// inside the block of columns.
template <int L, int LD, int SIDE, int PASS, int SC, int MEAS, int NCOL = L * L>
__device__ __forceinline__ void sep_pass(double* M, int ld, const double (&a)[L], double c, const double* sc,
                                         const double* sl, SepMeas& ms) {
  constexpr int N = L * L;
  const int LDv = LD > 0 ? LD : ld;
  constexpr bool kPair = LD > 0 && LD % 2 == 0 && L % 2 == 0;  // 16-byte words: even rows, aligned columns
  constexpr int ST = PASS == 0 ? 1 : L;                         // site step along the fibre
  if constexpr (SIDE == 1 || PASS == 1) {
    // W neighbouring fibres per thread, whose elements are neighbours in memory: rows i, i + 1 of
    // side 1, or the rows o, o + 1 of side 0's y-fibres
    constexpr int W = kPair ? 2 : 1;
    constexpr int LINES = SIDE == 1 ? N / W : NCOL;  // lanes walk rows (side 1) or columns (side 0)
    constexpr int FIB = SIDE == 1 ? (PASS == 0 ? NCOL / L : L) : L / W;
    for (int f = threadIdx.x; f < LINES * FIB; f += blockDim.x) {
      const int o = f / LINES, line = f - o * LINES;
      const int site0 = SIDE == 1 ? (PASS == 0 ? L * o : o) : W * o;  // first site of the (first) fibre
      double* p = SIDE == 1 ? M + W * line + (size_t)site0 * LDv : M + site0 + (size_t)line * LDv;
      const size_t st = SIDE == 1 ? (size_t)ST * LDv : (size_t)ST;
      double v[W][L], lf[W];
#pragma unroll
      for (int w = 0; w < W; ++w) lf[w] = (SC && sl) ? sl[SIDE == 1 ? W * line + w : line] : 1.0;
#pragma unroll
      for (int e = 0; e < L; ++e) {
        if constexpr (W == 2) {
          const double2 t = *reinterpret_cast<const double2*>(p + e * st);
          v[0][e] = t.x;
          v[1][e] = t.y;
        } else {
          v[0][e] = p[e * st];
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
          // the site of this element and the index of its line on the other side
          const int site = SIDE == 1 ? site0 + e * ST : site0 + w + e * ST;
          if (MEAS == 1) ms.add(v[w][e], SIDE == 1 ? site == W * line + w : site == line);
          if (SC == 1) v[w][e] *= lf[w] * sc[site];
        }
      }
#pragma unroll
      for (int w = 0; w < W; ++w) sep_conv<L>(a, v[w]);
#pragma unroll
      for (int e = 0; e < L; ++e) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int site = SIDE == 1 ? site0 + e * ST : site0 + w + e * ST;
          if (PASS == 1) v[w][e] *= c;
          if (SC == 2) v[w][e] *= lf[w] * sc[site];
          if (MEAS == 2) ms.add(v[w][e], SIDE == 1 ? site == W * line + w : site == line);
        }
        if constexpr (W == 2) *reinterpret_cast<double2*>(p + e * st) = make_double2(v[0][e], v[1][e]);
        else p[e * st] = v[0][e];
      }
    }
  } else {
    // x-fibres of side 0: L contiguous rows, lanes walk the columns
    for (int f = threadIdx.x; f < NCOL * L; f += blockDim.x) {
      const int o = f / NCOL, line = f - o * NCOL;
      double* p = M + L * o + (size_t)line * LDv;
      const double lf = (SC && sl) ? sl[line] : 1.0;
      double v[L];
      if constexpr (kPair) {
#pragma unroll
        for (int e = 0; e < L; e += 2) {
          const double2 t = *reinterpret_cast<const double2*>(p + e);
          v[e] = t.x;
          v[e + 1] = t.y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < L; ++e) v[e] = p[e];
      }
#pragma unroll
      for (int e = 0; e < L; ++e) {
        if (MEAS == 1) ms.add(v[e], L * o + e == line);
        if (SC == 1) v[e] *= lf * sc[L * o + e];
      }
      sep_conv<L>(a, v);
#pragma unroll
      for (int e = 0; e < L; ++e) {
        if (SC == 2) v[e] *= lf * sc[L * o + e];
        if (MEAS == 2) ms.add(v[e], L * o + e == line);
      }
      if constexpr (kPair) {
#pragma unroll
        for (int e = 0; e < L; e += 2) *reinterpret_cast<double2*>(p + e) = make_double2(v[e], v[e + 1]);
      } else {
#pragma unroll
        for (int e = 0; e < L; ++e) p[e] = v[e];
      }
    }
  }
}

// M <- c (A (x) A) M (side 0) or c M (A (x) A) (side 1), coefficients coef; a barrier after each
// pass. SC = 1: scaled before it, 2: after it (see sep_pass). MEAS as in sep_pass (1: first pass, 2:
// last).
template <int L, int LD, int SIDE, int SC, int MEAS = 0, int NCOL = L * L>
__device__ __forceinline__ void sep_side(double* M, int ld, const double* coef, double c, const double* sc, const double* sl,
                                         SepMeas& ms) {
  double a[L];
#pragma unroll
  for (int d = 0; d < L; ++d) a[d] = coef[d];
  sep_pass<L, LD, SIDE, 0, SC == 1 ? 1 : 0, MEAS == 1 ? 1 : 0, NCOL>(M, ld, a, c, sc, sl, ms);
  __syncthreads();
  sep_pass<L, LD, SIDE, 1, SC == 2 ? 2 : 0, MEAS == 2 ? 2 : 0, NCOL>(M, ld, a, c, sc, sl, ms);
  __syncthreads();
}

// The wrap of the whole matrix by one slice (see wrap_slice). vp = e^{V}, vm = e^{-V} of the slice's
// sites; the product of an element's two factors rides on the last pass's stores (up) or the first
// pass's loads (down). With MEAS the estimators of the matrix before (up) or after (down) the wrap
// are added to acc. LD > 0: M in dynamic shared memory; the factors always are.
template <int L, int LD, int UPDIR, int MEAS>
__device__ __noinline__ void sep_wrap(double* M, int ld, const HqChain& ch, const double* vp, const double* vm, double* acc,
                                      double* red) {
  SepMeas ms;
  if constexpr (LD > 0) M = as_shared(M);
  vp = as_shared(vp);
  vm = as_shared(vm);
  if constexpr (UPDIR) {
    sep_side<L, LD, 0, 0, MEAS ? 1 : 0>(M, ld, ch.sep_a, ch.sep_c, nullptr, nullptr, ms);
    sep_side<L, LD, 1, 2>(M, ld, ch.sep_ai, ch.sep_ci, vm, vp, ms);
  } else {
    sep_side<L, LD, 0, 1>(M, ld, ch.sep_ai, ch.sep_ci, vm, vp, ms);
    sep_side<L, LD, 1, 0, MEAS ? 2 : 0>(M, ld, ch.sep_a, ch.sep_c, nullptr, nullptr, ms);
  }
  if (MEAS) measure_commit(ms.tr, ms.dd, ms.sq, L * L, acc, red);
}

// One side alone, scaled before (SC = 1) or after (SC = 2) it
template <int L, int LD, int SIDE, int SC>
__device__ __noinline__ void sep_one(double* M, int ld, const double* coef, double c, const double* sc) {
  SepMeas ms;
  if constexpr (LD > 0) M = as_shared(M);
  sep_side<L, LD, SIDE, SC>(M, ld, coef, c, as_shared(sc), nullptr, ms);
}

// calls f(integral constant L) for the lattice size L in [1, HQ_MAX_L]
template <class F>
__device__ __forceinline__ void for_lattice(int L, F&& f) {
  switch (L) {
#define HQ_L_CASE(n) case n: f(IntC<n>{}); break;
    HQ_L_CASE(1) HQ_L_CASE(2) HQ_L_CASE(3) HQ_L_CASE(4) HQ_L_CASE(5) HQ_L_CASE(6) HQ_L_CASE(7) HQ_L_CASE(8)
    HQ_L_CASE(9) HQ_L_CASE(10) HQ_L_CASE(11) HQ_L_CASE(12) HQ_L_CASE(13) HQ_L_CASE(14) HQ_L_CASE(15)
#undef HQ_L_CASE
    default: f(IntC<16>{}); break;
  }
}

}  // namespace hq
