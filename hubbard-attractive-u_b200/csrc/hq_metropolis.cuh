// hq_metropolis.cuh -- building blocks of the submatrix Metropolis update shared by the
// interval kernels (one CTA per chain, and the thread-block-cluster variant for chains whose G
// spans several SMs): the acceptance test, the warp walk of a site block, the panels of its
// accepted flips and the DMMA flush.
#pragma once
#include "hq_common.cuh"

namespace hq {

// ---------------------------------------------------------------------------------
//  Metropolis sweep over the N sites of one slice: submatrix (block-delayed) updates.
//
//  The reference visits i = 0..N-1 in order, draws one uniform per site, and on
//  acceptance applies G -= gamma G[:,i] (e_i^T - G[i,:]), gamma = Delta/(1+(1-G_ii)Delta)
//  (src/hubbard.cpp:123-139). Here the sites are taken in blocks of up to 16 consecutive
//  sites (E. Gull, P. Staar, S. Fuchs et al., Submatrix updates for the continuous-time
//  auxiliary-field algorithm, Phys. Rev. B 83, 075122 (2011), applied to the Ising HS
//  field):
//   1. the walk: one warp holds g = G[B, B] in registers and visits the block's sites in order
//      with the reference's acceptance test and rank-1 updates of g alone (every later
//      decision of the block reads only g's diagonal). For the a accepted flips
//      j_0 < j_1 < ... it records gamma_m, X[B, m] = gamma_m g[:, j_m] and
//      Y[m, B] = g[j_m, :] - e_{j_m}^T (g before flip m);
//   2. the a flips become the panels of G_new = G + X Y,
//        X[:, m] = gamma_m (G[:, j_m] + sum_{m'<m} X[:, m'] Y[m', j_m])
//        Y[m, :] = G[j_m, :] - e_{j_m}^T + sum_{m'<m} X[j_m, m'] Y[m', :]
//      one row of X and one column of Y per thread, with the coefficients X[B, :] and
//      Y[:, B] from the walk's records;
//   3. G += X Y by DMMA (rank a <= 16).
//  On lattices of 81 sites and more with G in shared memory, warps 1 .. 7 flush while warp 0 takes the
//  next block's g = G[B', B'] + X[B', :] Y[:, B'] (the same DMMA steps, so the same bits as the flush
//  leaves) and walks it.
//  Measured at 12 x 12, 8 warps, thousands of cycles per slice (walk, panels, flush): 42, 17, 46 one
//  after the other; 56, 28 and 85 with predicated record stores in the walk, a branch per flip in the
//  panels, and a flush that checked every element against the edge.
//  The walk and the panels are bound by the latency of one dependency chain, the flush by the DMMA
//  pipe. With the walks beside the flushes a round trip of 200 slices at 12 x 12 takes 256 chains
//  48.2 ms instead of 51.1 (launches), one chain 23.6 instead of 25.3.
// ---------------------------------------------------------------------------------
constexpr int kLdR = 18;  // leading dimension of the walk's records: 16-byte rows whose stores spread over the banks

struct MetroShared {
  double* dl;     // Delta of each site [N]
  double* thr;    // u (1 + Delta) of each site [N]
  double* u;      // uniforms [N]
  double* rr;     // visit-time ratio of each site [N] (ratio log)
  int8_t* s;      // fields of the slice [N]
  int8_t* flip;   // accepted flags [N]
  double* X;      // N x 16 panel (column-major)
  double* Y;      // 16 x N panel (row-major)
  double* xt;     // X[B_s, m] of the block at xt[s kLdR + m], for sites visited after flip m (16-byte aligned)
  double* yt;     // Y[m, B_s] of the block at yt[s kLdR + m], likewise
  double* qg;     // gamma of each panel column [16], then 16 words that idle lanes of the walk write to
  int* ired;      // >= 2 ints: accepted counts of alternate blocks
  uint32_t* pw;   // a^(2i+1) mod m of each site [N]: the jump-ahead to site i's first draw
  int* qj;        // position inside the block of each accepted site, in order [16] (16-byte aligned)
};

// The acceptance ratio exactly as the reference evaluates it (src/hubbard.cpp:123-130):
// r = (1 + (1 - G_ii) Delta)^2 / (1 + Delta), each operation rounded on its own (no FMA
// contraction), the square as one product.
__device__ __forceinline__ double reference_ratio(double gii, double dl) {
  const double a = __dadd_rn(1.0, __dmul_rn(__dadd_rn(1.0, -gii), dl));
  return __ddiv_rn(__dmul_rn(a, a), __dadd_rn(1.0, dl));
}

// The walk of the nb <= 16 sites [b0, b0 + nb) by one warp, from their tile g of G. Lane 8 rg + cg
// holds the entries (4 rg + a, 2 cg + b), a < 4, b < 2, of g: a step needs column s at the lane's four rows, row s at its
// two columns and the diagonal entry, 7 shuffles. Entries of rows and columns already visited are
// not read again; they are left to run along.
//
// The decision of src/dqmc_core.cpp:110 is accept iff u < min(1, |r|). The fast walk tests
// u (1 + Delta) < a^2 (1 + Delta > 0), which needs no division on its dependency chain and equals
// the reference's test except when the two sides lie within a few rounding errors of each other.
// It only records whether that happened (warp-uniform; probability ~1e-12 per proposal): the
// return value. The caller then walks the block again, from its unchanged g, with EXACT: every
// decision in the reference's own form, u < min(1, |r|) with r as the reference evaluates it.
// The one warp issues in order, so the walk is straight code: every lane stores its records (lanes
// without any to a spare word), of accepted sites and others alike (the next site's overwrite them),
// because predicated stores became branches with a reconvergence each (5.5k instead of 3.2k cycles
// per block); the sites' constants are in registers before the first store (3.2k -> 2.9k); and
// NBC = 16 fixes nb at compile time (NBC = 0 takes nb). LOGT false compiles the ratio log out.
template <bool EXACT, bool LOGT, int NBC>
__device__ __forceinline__ bool walk_block16(const double* g, int ld, const MetroShared& sh, int b0, int nbr, int slot) {
  constexpr int NB = 16;
  const int nb = NBC > 0 ? NBC : nbr;
  const int lane = threadIdx.x & 31;
  const int rg = lane >> 3, cg = lane & 7;
  double r[4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int row = 4 * rg + a, col = 2 * cg + b;
      r[a][b] = (row < nb && col < nb) ? g[row + (size_t)col * ld] : 0.0;
    }
  __syncwarp();
  double dls[NB], thrs[NB];
#pragma unroll
  for (int s = 0; s < NB; ++s) {
    dls[s] = s < nb ? sh.dl[b0 + s] : 0.0;
    thrs[s] = s < nb ? sh.thr[b0 + s] : 0.0;
  }
  // this lane's record row is 4 rg + cg (cg < 4), its record column 2 cg + rg (rg < 2)
  double* xrec = cg < 4 ? sh.xt + (4 * rg + cg) * kLdR : sh.qg + 16;
  double* yrec = rg < 2 ? sh.yt + (2 * cg + rg) * kLdR : sh.qg + 16;
  double myr = 0.0;
  unsigned mask = 0u;
  bool near = false;
  int m = 0;  // flips accepted so far
#pragma unroll
  for (int s = 0; s < NB; ++s) {
    if (s < nb) {
      const double dl = dls[s], thr = thrs[s];
      // g_ss (lane 8 (s/4) + s/2); column s at the lane's rows (lane 8 rg + s/2, slot s&1); row s at
      // the lane's columns (lane 8 (s/4) + cg, slot s&3)
      const double dg = __shfl_sync(0xffffffffu, r[s & 3][s & 1], 8 * (s >> 2) + (s >> 1));
      double col[4], row[2];
#pragma unroll
      for (int a = 0; a < 4; ++a) col[a] = __shfl_sync(0xffffffffu, r[a][s & 1], 8 * rg + (s >> 1));
#pragma unroll
      for (int b = 0; b < 2; ++b) row[b] = __shfl_sync(0xffffffffu, r[s & 3][b], 8 * (s >> 2) + cg);
      const double av = fma(-dg, dl, 1.0 + dl);  // 1 + (1 - g_ss) Delta
      const double rc = __drcp_rn(av);
      const double gam = dl * rc;                // gamma = Delta / av
      if (LOGT && lane == s) myr = reference_ratio(dg, dl);
      bool acc;
      if (EXACT) {
        acc = sh.u[b0 + s] < fmin(1.0, fabs(reference_ratio(dg, dl)));
      } else {
        const double a2 = av * av;
        near = near || fabs(thr - a2) <= 1e-12 * a2;
        acc = thr < a2;
      }
      // the records of the flip, read for sites visited later
      const double xs = (cg & 1) ? ((cg & 2) ? col[3] : col[1]) : ((cg & 2) ? col[2] : col[0]);
      xrec[m] = gam * xs;
      yrec[m] = (rg & 1) ? row[1] : row[0];
      sh.qj[m] = s;
      sh.qg[m] = gam;
      const double gr = acc ? rc : 0.0;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const double f = gr * (dl * col[a]);
#pragma unroll
        for (int b = 0; b < 2; ++b) r[a][b] = fma(f, row[b], r[a][b]);
      }
      mask |= acc ? (1u << s) : 0u;
      m += acc ? 1 : 0;
    }
  }
  if (!EXACT && near) return true;
  if (lane < nb) {
    sh.flip[b0 + lane] = (mask >> lane) & 1u;
    if (LOGT) sh.rr[b0 + lane] = myr;
  }
  if (lane == 0) sh.ired[slot] = m;
  return false;
}

// The walks of the ratio log, of near ties and of short blocks, out of line behind one call each: their
// code and registers do not weigh on the fast walk's (a call of its own per length cost 1 % at 8x8). Blocks
// of 4 and 8 sites (the smaller delay depths, last blocks such as those of 36 and 100 sites) and single
// last sites (49, 81, 225 sites) have their steps and loads fixed at compile time. Round trips of 40
// slices, launches, nb at run time / fixed, ms: 64 chains of 8x8 at depth 4 5.59 / 3.99, at 8 4.46 / 3.73; 128
// of 12x12 16.3 / 13.7, 13.3 / 11.9; 16 of 14x14 76.6 / 71.4, 55.2 / 52.8; 64 of 6x6 at depth 16 2.70 / 2.53.
template <bool EXACT, bool LOGT>
__device__ __noinline__ bool walk_rare(const double* g, int ld, const MetroShared sh, int b0, int nb, int slot) {
  if constexpr (!EXACT && !LOGT) {
    if (nb == 1) return walk_block16<EXACT, LOGT, 1>(g, ld, sh, b0, nb, slot);
    if (nb == 4) return walk_block16<EXACT, LOGT, 4>(g, ld, sh, b0, nb, slot);
    if (nb == 8) return walk_block16<EXACT, LOGT, 8>(g, ld, sh, b0, nb, slot);
  }
  return walk_block16<EXACT, LOGT, 0>(g, ld, sh, b0, nb, slot);
}
// the walk with the reference's form of every decision where the fast one came near a tie; again()
// restores g before a second walk, if the first one's records overwrote it
template <class F>
__device__ __forceinline__ void walk(const double* g, int ld, const MetroShared& sh, int b0, int nb, bool log, int slot, F&& again) {
  if (log) {
    if (walk_rare<false, true>(g, ld, sh, b0, nb, slot)) again(), walk_rare<true, true>(g, ld, sh, b0, nb, slot);
  } else if (nb == 16) {
    if (walk_block16<false, false, 16>(g, ld, sh, b0, nb, slot)) again(), walk_rare<true, false>(g, ld, sh, b0, nb, slot);
  } else {
    if (walk_rare<false, false>(g, ld, sh, b0, nb, slot)) again(), walk_rare<true, false>(g, ld, sh, b0, nb, slot);
  }
}
// the walk of a tile that lies in G
__device__ __forceinline__ void walk(const double* g, int ld, const MetroShared& sh, int b0, int nb, bool log, int slot) {
  walk(g, ld, sh, b0, nb, log, slot, [] {});
}

// The next block's tile for the walk beside the flush, in DMMA accumulators of warp 0: the nb x nb
// entries at g, loaded before the flush touches G; then the flush's own k-steps (the block's rows of
// X, its columns of Y); then into shared memory, where it takes the place of the records xt: the walk has
// read it before its first record is written (a tile of its own would take 2.3 KB from the L1 cache).
struct NextTile {
  double v[2][4];
  __device__ __forceinline__ void load(const double* g, int ld, int nb) {
    const int gr = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = gr + ((e & 2) ? 8 : 0), col = 8 * t + 2 * q + (e & 1);
        v[t][e] = (row < nb && col < nb) ? g[row + (size_t)col * ld] : 0.0;
      }
  }
  template <int KA>
  __device__ __forceinline__ void update(const double* Xr, int ldx, const double* Yc, int ldy) {
    const int gr = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
    for (int s = 0; s < KA; ++s) {
      const double a0 = Xr[gr + (4 * s + q) * ldx], a1 = Xr[gr + 8 + (4 * s + q) * ldx];
#pragma unroll
      for (int t = 0; t < 2; ++t) dmma_16x8x4(v[t], a0, a1, Yc[(4 * s + q) * ldy + 8 * t + gr]);
    }
  }
  __device__ __forceinline__ void store(double* tile) const {
    const int gr = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) tile[gr + ((e & 2) ? 8 : 0) + (8 * t + 2 * q + (e & 1)) * kLdR] = v[t][e];
    __syncwarp();
  }
};

// W lines of a panel for a flips, 4 (KA - 1) < a <= 4 KA, in the thread's registers,
//   v[m] = w_m (g[m] + sum_{m'<m} c[j_m][m'] v[m']):
// rows of X (ISX: g[m] = G[p, j_m], c = the records yt, w = gamma) or columns of Y (g[m] = G[j_m, p] less
// 1 where p = j_m, c = xt, w = 1); entry of flip m at g[w] + q_m gs, delta[w] the position q_m of the 1.
// The sums run over the even and the odd m' apart. There is no branch on a (flips past a come out
// as zero), so the loads run ahead of the recurrences; two lines per thread share the coefficients,
// whose broadcast loads are most of the shared-memory traffic.
template <int KA, int W, bool ISX>
__device__ __forceinline__ void panel_lines(const double* const (&g)[W], size_t gs, const int (&delta)[W], const MetroShared& sh,
                                            int a, double (&v)[W][4 * KA]) {
  constexpr int K = 4 * KA;
  int qm[K];
#pragma unroll
  for (int k = 0; k < KA; ++k) {
    const int4 t = *reinterpret_cast<const int4*>(sh.qj + 4 * k);
    qm[4 * k] = t.x; qm[4 * k + 1] = t.y; qm[4 * k + 2] = t.z; qm[4 * k + 3] = t.w;
  }
#pragma unroll
  for (int m = 0; m < K; ++m) {
    qm[m] = m < a ? qm[m] : 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      v[w][m] = g[w][qm[m] * gs];
      if (!ISX) v[w][m] -= (qm[m] == delta[w] ? 1.0 : 0.0);
    }
  }
  const double* rec = ISX ? sh.yt : sh.xt;
#pragma unroll
  for (int m = 0; m < K; ++m) {
    const double* c = rec + qm[m] * kLdR;
    double s0[W], s1[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      s0[w] = v[w][m];
      s1[w] = 0.0;
    }
#pragma unroll
    for (int m2 = 0; m2 + 1 < m; m2 += 2) {
      const double2 t = *reinterpret_cast<const double2*>(c + m2);
#pragma unroll
      for (int w = 0; w < W; ++w) {
        s0[w] = fma(v[w][m2], t.x, s0[w]);
        s1[w] = fma(v[w][m2 + 1], t.y, s1[w]);
      }
    }
    const double cl = (m & 1) ? c[m - 1] : 0.0;
    const double sc = ISX ? sh.qg[m] : 1.0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      if (m & 1) s0[w] = fma(v[w][m - 1], cl, s0[w]);
      const double t = ISX ? sc * (s0[w] + s1[w]) : s0[w] + s1[w];
      v[w][m] = m < a ? t : 0.0;
    }
  }
}
// rows t and t + ceil(N / 2) of X (t + ... past the last row repeats it) by threads 0 .. 127
template <int KA>
__device__ __forceinline__ void panel_rows(const double* Gb, int ld, int N, const MetroShared& sh, int a, int ldx) {
  const int H = (N + 1) / 2;
  for (int t = threadIdx.x & 127; t < H; t += 128) {
    const int p1 = min(t + H, N - 1);
    const double* g[2] = {Gb + t, Gb + p1};
    const int none[2] = {-1, -1};
    double v[2][4 * KA];
    panel_lines<KA, 2, true>(g, ld, none, sh, a, v);
#pragma unroll
    for (int m = 0; m < 4 * KA; ++m) {
      sh.X[t + m * ldx] = v[0][m];
      sh.X[p1 + m * ldx] = v[1][m];
    }
  }
}
// columns t and t + ceil(nc / 2) of Y by threads 128 .. 255: Gr = the block's first row of the nc
// columns, the first of them column c0 of G
template <int KA>
__device__ __forceinline__ void panel_cols(const double* Gr, int ld, int nc, int c0, const MetroShared& sh, int a, int b0,
                                           int ldy) {
  const int H = (nc + 1) / 2;
  for (int t = threadIdx.x & 127; t < H; t += 128) {
    const int p1 = min(t + H, nc - 1);
    const double* g[2] = {Gr + (size_t)t * ld, Gr + (size_t)p1 * ld};
    const int delta[2] = {c0 + t - b0, c0 + p1 - b0};
    double v[2][4 * KA];
    panel_lines<KA, 2, false>(g, 1, delta, sh, a, v);
#pragma unroll
    for (int m = 0; m < 4 * KA; ++m) {
      sh.Y[m * ldy + t] = v[0][m];
      sh.Y[m * ldy + p1] = v[1][m];
    }
  }
}
// both panels of the block at b0 on one CTA
template <int KA>
__device__ __forceinline__ void build_panels(const double* G, int ld, int N, const MetroShared& sh, int ldp, int a, int b0) {
  static_assert(HQ_INT_THREADS == 256, "half the threads take X, half Y");
  if (threadIdx.x < 128) panel_rows<KA>(G + (size_t)b0 * ld, ld, N, sh, a, ldp);
  else panel_cols<KA>(G + b0, ld, N, 0, sh, a, b0, ldp);
}

// G[0:M, 0:Nc] += X[:, 0:k] Y[0:k, :] (k <= 16) with every element
// checked against the edge: 48 x 32 warp tiles (3 x 4 DMMA tiles sharing their fragments). For G in
// global memory, whose columns are not padded.
__device__ __forceinline__ void rank_update48(double* G, int ld, int M, int Nc, const MetroShared& sh, int ldx, int ldy, int k) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int mt = (M + 47) / 48, ns = (Nc + 31) / 32;
  const int ksteps = (k + 3) >> 2;
  for (int st = warp; st < mt * ns; st += nw) {
    const int r0 = (st % mt) * 48, c0 = (st / mt) * 32;
    double acc[3][4][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int r = r0 + 16 * i + g, c = c0 + t * 8 + 2 * q;
        acc[i][t][0] = (r < M && c < Nc) ? G[r + (size_t)c * ld] : 0.0;
        acc[i][t][1] = (r < M && c + 1 < Nc) ? G[r + (size_t)(c + 1) * ld] : 0.0;
        acc[i][t][2] = (r + 8 < M && c < Nc) ? G[r + 8 + (size_t)c * ld] : 0.0;
        acc[i][t][3] = (r + 8 < M && c + 1 < Nc) ? G[r + 8 + (size_t)(c + 1) * ld] : 0.0;
      }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (s < ksteps) {
        const int m = 4 * s + q;
        const bool mk = m < k;
        const double* Xp = sh.X + m * ldx;
        double fa[3][2], fb[4];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int r = r0 + 16 * i + g;
          fa[i][0] = (r < M && mk) ? Xp[r] : 0.0;
          fa[i][1] = (r + 8 < M && mk) ? Xp[r + 8] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int cb = c0 + t * 8 + g;
          fb[t] = (cb < Nc && mk) ? sh.Y[m * ldy + cb] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int t = 0; t < 4; ++t) dmma_16x8x4(acc[i][t], fa[i][0], fa[i][1], fb[t]);
      }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int r = r0 + 16 * i + g, c = c0 + t * 8 + 2 * q;
        if (r < M && c < Nc) G[r + (size_t)c * ld] = acc[i][t][0];
        if (r < M && c + 1 < Nc) G[r + (size_t)(c + 1) * ld] = acc[i][t][1];
        if (r + 8 < M && c < Nc) G[r + 8 + (size_t)c * ld] = acc[i][t][2];
        if (r + 8 < M && c + 1 < Nc) G[r + 8 + (size_t)(c + 1) * ld] = acc[i][t][3];
      }
  }
}

// G[0:16 MT, 0:8 T] += X[:, 0:4 KS] Y[0:4 KS, :] on storage that is padded to whole DMMA tiles, so that
// nothing is checked: 16 x 8 NT strips, NT = 3 or 2, whichever divides T (tile_cols). Pad rows and
// columns hold any values; they only reach pad rows and columns.
// Bound by the DMMA pipe (12 x 12, rank 12: 162 tiles x 3 steps x 8 cycles = 3.9k of 5.2k
// measured); strips of 16 x 24 keep eight warps evenly loaded (54 strips), 48 x 32 tiles took 7.1k.
template <int MT, int T, int KS>
__device__ __forceinline__ void rank_strips(double* G, int ld, const MetroShared& sh, int ldx, int ldy, int warp, int nw) {
  constexpr int NT = T % 3 == 0 ? 3 : 2;
  static_assert(T % NT == 0, "tile_cols pads the columns to whole strips");
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const double* Xq = sh.X + q * ldx + g;
  const double* Yq = sh.Y + q * ldy + g;
#pragma unroll 1
  for (int st = warp; st < MT * (T / NT); st += nw) {
    const int r0 = (st % MT) * 16, t0 = (st / MT) * NT;
    double* Gp = G + r0 + g + (size_t)(8 * t0 + 2 * q) * ld;
    const double* Yp = Yq + 8 * t0;
    double acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      acc[t][0] = Gp[(8 * t) * ld];
      acc[t][1] = Gp[(8 * t + 1) * ld];
      acc[t][2] = Gp[8 + (8 * t) * ld];
      acc[t][3] = Gp[8 + (8 * t + 1) * ld];
    }
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      const double a0 = Xq[4 * s * ldx + r0], a1 = Xq[4 * s * ldx + r0 + 8];
#pragma unroll
      for (int t = 0; t < NT; ++t) dmma_16x8x4(acc[t], a0, a1, Yp[4 * s * ldy + 8 * t]);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      Gp[(8 * t) * ld] = acc[t][0];
      Gp[(8 * t + 1) * ld] = acc[t][1];
      Gp[8 + (8 * t) * ld] = acc[t][2];
      Gp[8 + (8 * t + 1) * ld] = acc[t][3];
    }
  }
}

// calls f(integral constant ceil(a / 4)) for 1 <= a <= 16 flips
template <class F>
__device__ __forceinline__ void for_ksteps(int a, F&& f) {
  switch ((a + 3) >> 2) {
    case 1: f(IntC<1>{}); break;
    case 2: f(IntC<2>{}); break;
    case 3: f(IntC<3>{}); break;
    default: f(IntC<4>{}); break;
  }
}

}  // namespace hq
