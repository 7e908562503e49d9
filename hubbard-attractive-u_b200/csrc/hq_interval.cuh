// hq_interval.cuh -- the body of one stabilisation interval of one chain: G(tau,tau) resident in
// shared memory while the slices of the interval are wrapped (src/dqmc_core.cpp:142-161) and
// updated by Metropolis flips with delayed rank-k updates flushed by DMMA
// (src/dqmc_core.cpp:102-119, src/hubbard.cpp:123-139); fused equal-time estimators
// (include/observable_methods.hpp:39-151) and optional per-slice snapshots. Used by k_interval
// (one launch per interval) and by the persistent sweep kernel.
#pragma once
#include "hq_metropolis.cuh"

namespace hq {

// the interval body's shared-memory words of chain size N (see IntervalLayout)
__device__ __forceinline__ MetroShared metro_shared(double* smem, const IntervalLayout& o, int N) {
  MetroShared sh;
  sh.X = smem + o.work;
  sh.Y = smem + o.Y;
  sh.xt = smem + o.rec;
  sh.yt = sh.xt + 16 * kLdR;
  sh.qg = sh.yt + 16 * kLdR;
  sh.dl = smem + o.dl;
  sh.thr = smem + o.thr;
  sh.u = smem + o.u;
  sh.rr = smem + o.rr;
  sh.s = reinterpret_cast<int8_t*>(smem + o.fields);
  sh.flip = sh.s + N;
  sh.pw = reinterpret_cast<uint32_t*>(smem + o.pw);
  sh.ired = reinterpret_cast<int*>(smem + o.ints);
  sh.qj = sh.ired + 4;
  return sh;
}

// The Metropolis visits of one slice's N sites (see hq_metropolis.cuh) from the random state rng;
// returns the accepted flips (thread 0). L > 0: G in shared memory in the padded layout
// (interval_ld, tile_cols) of the lattice size L; L = 0: G in global memory, any N, checked against
// the edge. NB = the chain's delay depth: sites per block (4, 8 or 16). Every thread calls it. A
// function of its own per lattice size: registers and code of one size do not weigh on the others.
template <int L>
__device__ __noinline__ int metropolis_slice(const HqChain& ch, uint32_t rng, int flags, long long log_base) {
  extern __shared__ __align__(16) double smem[];
  // Warp 0 walks the next block beside the flush where the flush is long enough to lose a warp: round
  // trips with / without, ms: 48 chains of 9 x 9 6.33 / 6.53, one of 8 x 8 13.6 / 13.2, 32 of 7 x 7 (dense)
  // 5.67 / 5.46. With G in global memory the flush is so long that the warp it lacks costs more than
  // the walk beside it saves (16 chains of 14 x 14, interval kernel: 17.9 / 16.7 ms a sweep).
  constexpr bool kAhead = L >= 9;
  const int N = L > 0 ? L * L : ch.N;
  const IntervalLayout lay = interval_layout(N, L > 0 ? 16 : ch.kmax, L > 0);
  const MetroShared sh = metro_shared(smem, lay, N);
  double* G = L > 0 ? smem + lay.G : ch.G;
  const int ld = L > 0 ? interval_ld(N) : N;
  const int ldp = panel_ld(pad16(N));
  const int NB = ch.kmax;
  const int tid = threadIdx.x, warp = kAhead ? warp_index() : tid >> 5;
  const bool log = (flags & HQ_F_LOG_RATIOS) && ch.ratios;
  // uniforms of this slice: site i consumes engine draws 2i+1, 2i+2 after the current state
  for (int i = tid; i < N; i += blockDim.x) {
    const uint32_t x1 = minstd_mulmod(sh.pw[i], rng);
    const uint32_t x2 = minstd_mulmod(kMinstdA, x1);
    const double u = canonical_from_pair(x1, x2), dl = sh.s[i] > 0 ? ch.delta_p : ch.delta_m;
    sh.u[i] = u;
    sh.dl[i] = dl;
    sh.thr[i] = u * (1.0 + dl);
  }
  __syncthreads();
  int acc_count = 0;
  if constexpr (kAhead) {
    // bn: the block to walk; the one before it is to flush. The walk stands in the code once (with a copy
    // per flip count the instruction cache ate half of the gain).
    for (int bn = 0, bi = 0;; bn += NB, ++bi) {
      const bool more = bn < N, ahead = more && warp == 0;
      int a = 0;
      if (bn > 0) {
        __syncthreads();  // the previous block's walk and the flush before it are done
        // the count alternates between two words: with no flush (a == 0) no barrier follows,
        // and warp 0 writes the next block's count while other warps may still read this one
        a = sh.ired[(bi - 1) & 1];
        acc_count += a;
      }
      NextTile next;
      if (ahead) next.load(G + bn + (size_t)bn * ld, ld, min(NB, N - bn));
      if (a > 0)
        for_ksteps(a, [&](auto kc) {
          constexpr int KA = decltype(kc)::value;
          build_panels<KA>(G, ld, N, sh, ldp, a, bn - NB);
          __syncthreads();
          if (ahead) next.update<KA>(sh.X + bn, ldp, sh.Y + bn, ldp);
          else rank_strips<pad16(L * L) / 16, tile_cols(L * L), KA>(G, ld, sh, ldp, ldp, more ? warp - 1 : warp, more ? 7 : 8);
        });
      if (!more) break;
      if (ahead) {
        next.store(sh.xt);
        walk(sh.xt, kLdR, sh, bn, min(NB, N - bn), log, bi & 1, [&] { next.store(sh.xt); });
      }
    }
    __syncthreads();
  } else {
    for (int b0 = 0, bi = 0; b0 < N; b0 += NB, ++bi) {
      if (warp == 0) walk(G + b0 + (size_t)b0 * ld, ld, sh, b0, min(NB, N - b0), log, bi & 1);
      __syncthreads();
      const int a = sh.ired[bi & 1];  // alternating words, as above
      acc_count += a;
      if (a == 0) continue;
      for_ksteps(a, [&](auto kc) {
        constexpr int KA = decltype(kc)::value;
        build_panels<KA>(G, ld, N, sh, ldp, a, b0);
        __syncthreads();
        if constexpr (L > 0) rank_strips<pad16(L * L) / 16, tile_cols(L * L), KA>(G, ld, sh, ldp, ldp, tid >> 5, HQ_INT_THREADS / 32);
      });
      if constexpr (L == 0) rank_update48(G, ld, N, N, sh, ldp, ldp, a);
      __syncthreads();
    }
  }
  // apply the flips of this slice and optionally log the visit-time ratios
  for (int i = tid; i < N; i += blockDim.x) {
    if (sh.flip[i]) sh.s[i] = -sh.s[i];
    if (log && log_base + i < ch.ratio_cap) ch.ratios[log_base + i] = sh.rr[i];
  }
  __syncthreads();
  return acc_count;
}
template <bool RES>
__device__ __forceinline__ int metropolis_dispatch(const HqChain& ch, uint32_t rng, int flags, long long log_base) {
  int a = 0;
  if constexpr (RES) {
    for_lattice(ch.L, [&](auto lc) {
      constexpr int L = decltype(lc)::value;
      if constexpr (L <= 12) a = metropolis_slice<L>(ch, rng, flags, log_base);
    });
  } else {
    a = metropolis_slice<0>(ch, rng, flags, log_base);
  }
  return a;
}

// Shared-memory words of the interval body besides its dynamic region: reductions and the barrier
// of the bulk load of G (initialised for one arrival).
struct IntervalScratch {
  double* red;     // 96 doubles
  double* est;     // 4 doubles: the chain's estimator sums while its slices are worked on
  uint64_t* gbar;
};
constexpr int kIntervalScratchBytes = (96 + 4 + 2) * 8;

// Places the interval scratch at `p` (16-byte aligned, kIntervalScratchBytes long).
__device__ __forceinline__ IntervalScratch interval_scratch_at(void* p) {
  double* d = reinterpret_cast<double*>(p);
  return {d, d + 96, reinterpret_cast<uint64_t*>(d + 100)};
}

// The update (or no-update) slices of stabilisation interval b of chain `ch` in direction dir.
// `smem` is the block's dynamic shared memory (interval_smem_doubles(N, kmax, RES) doubles); gpar is the
// phase parity of sc.gbar for this interval's bulk load of G. Every thread of the block calls
// it; the chain is active and b < n_stab.
template <bool RES>
__device__ __forceinline__ void interval_body(const HqChain& ch, int dir, int b, int flags, double* smem,
                                              const IntervalScratch& sc, unsigned gpar) {
  const int N = ch.N;
  int t_lo, t_hi;
  interval_range(ch.nt, ch.pace, ch.n_stab, dir, b, t_lo, t_hi);

  // the resident G moves in and out by bulk copies of its columns (cp.async per element where the
  // columns are not 16-byte multiples)
  const IntervalLayout lay = interval_layout(N, ch.kmax, RES);
  double* G = RES ? smem + lay.G : ch.G;
  const int ld = RES ? interval_ld(N) : N;
  bool bulk = false;
  if (RES) {
    bulk = bulk_columns_ok(ch.G, N, ld);
    if (bulk) load_mat_bulk(G, ld, ch.G, N, sc.gbar, ch.acc + HQ_ACC_STATUS, gpar);
    else load_mat_async(G, ld, ch.G, N, N);
  }
  const MetroShared sh = metro_shared(smem, lay, N);
  double *work = sh.X, *vp = smem + lay.vp, *vm = smem + lay.vm;
  for (int i = threadIdx.x; i < N; i += blockDim.x) sh.pw[i] = minstd_pow(2ull * i + 1);
  const uint64_t slice_jump = minstd_pow(2ull * N);  // the engine's state after a slice's 2 N draws
  uint32_t rng = *ch.rng;
  double n_acc = 0.0, n_prop = 0.0;
  long long log_base = (flags & HQ_F_LOG_RATIOS) && ch.ratio_count ? *ch.ratio_count : 0;
  // the estimator sums stay in shared memory for the interval: a round trip to global memory per
  // slice is longer than a small lattice's passes
  static_assert(HQ_ACC_FILLING == 0 && HQ_ACC_DOCC == 1 && HQ_ACC_SWAVE == 2 && HQ_ACC_NSLICE == 3, "the first four");
  if (threadIdx.x < 4) sc.est[threadIdx.x] = ch.acc[threadIdx.x];
  __syncthreads();

  const int nsl = t_hi - t_lo + 1;
  // up / down sweeps in separable mode measure inside the wrap (up: slice t's G in the wrap of
  // slice t+1; down: in the wrap of slice t itself); the last slice of the interval is
  // measured after stabilisation
  const bool fused = (flags & HQ_F_MEASURE) && ch.expk_mode == HQK_EXPK_SEPARABLE && wrap_measures<RES>(ch.L) &&
                     (dir == HQ_UP || dir == HQ_DOWN);
  // the next slice's fields are on their way while a slice is worked on
  auto field = [&](int step) {
    const int l = ((dir == HQ_DOWN) ? (t_hi - step) : (t_lo + step)) % ch.nt;
    return step < nsl && (int)threadIdx.x < N ? ch.fields[(size_t)l * N + threadIdx.x] : (int8_t)0;
  };
  int8_t next = field(0);
  for (int step = 0; step < nsl; ++step) {
    const int t = (dir == HQ_DOWN) ? (t_hi - step) : (t_lo + step);
    const int l = t % ch.nt;
    if ((int)threadIdx.x < N) sh.s[threadIdx.x] = next;
    for (int i = threadIdx.x + blockDim.x; i < N; i += blockDim.x) sh.s[i] = ch.fields[(size_t)l * N + i];
    next = field(step + 1);
    __syncthreads();
    if (dir != HQ_DOWN) {
      slice_factors(ch, sh.s, vp, vm);
      __syncthreads();
      wrap_slice<RES>(ch, G, ld, vp, vm, HQ_UP, work, (fused && step > 0) ? sc.est : nullptr, sc.red);
    }
    if (dir == HQ_UP || dir == HQ_DOWN) {
      n_acc += metropolis_dispatch<RES>(ch, rng, flags, log_base);
      rng = minstd_mulmod(slice_jump, rng);
      n_prop += N;
      log_base += N;
    }
    if (dir == HQ_DOWN) {
      slice_factors(ch, sh.s, vp, vm);
      __syncthreads();
      wrap_slice<RES>(ch, G, ld, vp, vm, HQ_DOWN, work, (fused && step < nsl - 1) ? sc.est : nullptr, sc.red);
    }
    for (int i = threadIdx.x; i < N; i += blockDim.x) ch.fields[(size_t)l * N + i] = sh.s[i];
    if (step < nsl - 1) {
      const int lm = (dir == HQ_DOWN) ? ((t - 1) % ch.nt) : l;
      if ((flags & HQ_F_MEASURE) && !fused) measure_slice(G, ld, N, sc.est, sc.red);
      if ((flags & HQ_F_SNAPSHOT) && ch.snap_tt) copy_mat(ch.snap_tt + (size_t)lm * N * N, N, G, ld, N);
    }
    __syncthreads();
  }
  if (RES) {
    if (bulk) store_mat_bulk(ch.G, G, ld, N);
    else copy_mat(ch.G, N, G, ld, N);
  }
  if (threadIdx.x == 0) {
    for (int k = 0; k < 4; ++k) ch.acc[k] = sc.est[k];
    *ch.rng = rng;
    ch.acc[HQ_ACC_PROPOSED] += n_prop;
    ch.acc[HQ_ACC_ACCEPTED] += n_acc;
    if ((flags & HQ_F_LOG_RATIOS) && ch.ratio_count) *ch.ratio_count = log_base;
  }
}

}  // namespace hq
