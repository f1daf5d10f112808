// pf_persist.cuh -- building blocks of the persistent Krylov kernels: one
// cooperative launch runs many iterations, its CTAs keep the vectors of their
// own slots on chip, and the two inner products of an iteration double as the
// grid-wide barriers.
//
// Why.  An iteration of a pressure solve on a small grid moves little (at
// 48^3: 100k unknowns, 14 MB, all in L2), but as three launches it costs three
// launch gaps and three last-CTA reductions in series: 21 us at 24^3, 25 us at
// 48^3, 29 us at 64^3 and 80 us at 128^3, most of it waiting.
//
// Reduction.  A virtual CTA is what a CTA of the three-kernel path is: slots
// b, b + nred, b + 2 nred, ... with one thread per cell, nred = min(nslots,
// kMaxRedBlocks).  CTA c of the persistent grid owns slots c, c + kPsGrid,
// c + 2 kPsGrid, ..., which are whole virtual CTAs because kMaxRedBlocks is a
// multiple of kPsGrid.  Every virtual CTA's partial is formed by the same tree
// and published in an entry of its own; every CTA then reads all of them and
// sums them in the order of the three-kernel path's last CTA.  So every sum
// has the bits of the three-kernel path, on every CTA, without a broadcast.
// A maximum has the same bits in any order: one entry per CTA.
//
// Barrier.  A CTA stores its entries, then adds 1 to a counter, and one thread
// polls the counter until every CTA has arrived; only then are the entries
// read.  (148 CTAs whose threads poll the entries themselves take 6600 cycles
// a barrier, 8500 with 8 entries a CTA; with the counter first 2400 and 3500:
// the polls of many lines by every SM hold up the stores they wait for.)  The
// counter alone orders nothing: an entry is a 16-byte pair of the value and a
// tag, stored and loaded as one access, and a reader that finds another tag
// reads again.  Tags grow over the context's life, so nothing is ever cleared.
// A barrier that hands over other global memory (ps_barrier) adds a release
// fence before the arrival and an acquire fence after it (+1000 cycles and the
// time its writes take to land).
// Each reduction has two sets of entries, used alternately: a CTA that writes
// a set again has passed the reduction in between, so every CTA has read it.
//
// One launch holds every SM: a kernel of another stream (an asynchronous upload's
// unpacking, another context's work, the caller's own) starts only when it ends.
// So a launch runs no more than kPsTurns iterations of the resident kernels, and
// kPsStreamTurns / k where they take about 1.8 k us for the k slots of a CTA: 16 ms
// or less (2000 iterations in one launch held 11 ms at 48^3, 99 at 128^3, 173 at
// 148^3).  A launch more costs 15 us up to 64^3 and 50 at 128^3: 128^3 to 1e-6 takes
// 0.4 % longer than in launches of 2048, and would take 0.8 % in 8 ms.
//
// Every wait is bounded (kPsPolls polls); a CTA that runs out of them sets
// SolveCtl::aux[0] and leaves, and the host returns an error.
#pragma once

#include <algorithm>

#include "pf_solver.cuh"

namespace pf {

constexpr int kPsVirt = kMaxRedBlocks / kPsGrid;    // virtual CTAs of one CTA, at most
constexpr int kPsTurns = 2048, kPsStreamTurns = 4 * kPsTurns;
constexpr unsigned kPsPolls = 1u << 22;
constexpr int kPsWarps = PF_TV / 32;                // warps of a virtual CTA
constexpr int kPsFace = 6 * 64;                     // face values of a slot

static_assert(kMaxRedBlocks % kPsGrid == 0, "a CTA must own whole virtual CTAs");
static_assert(kPsWarps == 16, "half a warp folds one virtual CTA");

// iterations of the next launch: check_every if the caller gives it, else by_time
inline int ps_turns(int check_every, int by_time, int left) {
  const int n = check_every > 0 ? std::min(check_every, kPsTurns) : by_time;
  return std::min(n, left);
}

// a value and its tag, as one 16-byte access
__device__ __forceinline__ void ps_store(PsPair* p, double v, unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(tag)
      : "memory");
}
__device__ __forceinline__ void ps_load(const PsPair* p, double& v, unsigned long long& tag) {
  long long b;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(b), "=l"(tag)
               : "l"(p)
               : "memory");
  v = __longlong_as_double(b);
}
// loads until the tag is there; false when the polls ran out
__device__ __forceinline__ bool ps_await(const PsPair* p, double& v, unsigned long long& have,
                                         unsigned long long tag) {
  for (unsigned polls = 0; have != tag; ++polls) {
    if (polls > kPsPolls) return false;
    ps_load(p, v, have);
  }
  return true;
}
__device__ __forceinline__ void ps_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Warp sums of N values at once (N a power of two up to 8), each by the tree
// of warp_sum: at the first levels half of the lanes hand over one half of the
// values and half the other, so N values take N + 4 - log2 N exchanges instead
// of 5 N.  Returns the sum of value ps_owner<N>(lane).
template <int N>
__device__ __forceinline__ double warp_sum_many(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int h = N / 2; h > 0; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int q = 16 / N; q > 0; q >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], q);
  return v[0];
}
template <int N>
__device__ __forceinline__ int ps_owner(int lane) {
  return N == 1 ? 0 : N == 2 ? lane >> 4 : N == 4 ? ((lane >> 4) << 1) | ((lane >> 3) & 1)
                    : ((lane >> 4) << 2) | (((lane >> 3) & 1) << 1) | ((lane >> 2) & 1);
}

// Shared scratch of the reductions.
struct PsShared {
  double loc[kPsVirt][kPsWarps];  // warp sums of each virtual CTA
  double wmax[32];                // warp maxima of the CTA
  double glob[kPsWarps], gmax[8];
};

// The published entries of a context: [2 reductions][2 parities][kMaxRedBlocks]
// sums, [2 parities][kPsGrid] maxima, and the arrival counter on a line of its
// own.
struct PsBar {
  PsPair* e;
  unsigned long long* counter;
  __device__ __forceinline__ PsPair* sums(int which, int parity) const {
    return e + (size_t)(2 * which + parity) * kMaxRedBlocks;
  }
  __device__ __forceinline__ PsPair* maxima(int parity) const {
    return e + 4 * (size_t)kMaxRedBlocks + parity * kPsGrid;
  }
};

// Waits until the counter reaches `target` arrivals (one thread of the CTA).
__device__ __forceinline__ bool ps_poll(const unsigned long long* counter, unsigned long long target) {
  for (unsigned polls = 0; polls <= kPsPolls; ++polls) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(counter) : "memory");
    if (v >= target) return true;
  }
  return false;
}
__device__ __forceinline__ void ps_arrive(unsigned long long* counter) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(counter), "l"(1ull) : "memory");
}

// A barrier that hands over global memory: every write of the grid before it
// is visible to every thread after it.  False when the wait ran out.
__device__ __forceinline__ bool ps_barrier(const PsBar& bar, unsigned long long target) {
  int dead = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    ps_fence();
    ps_arrive(bar.counter);
    dead = !ps_poll(bar.counter, target);
    ps_fence();
  }
  return !__syncthreads_or(dead);
}

// First half of a reduction: the warp sums of the CTA's nvirt virtual CTAs are
// in sh.loc and (kMax) the warp maxima of its nwarps warps in sh.wmax, written
// by any thread.  Warp 0 folds them -- each virtual CTA by the tree of
// block_sum_max, half a warp each -- stores the entries and arrives.  The other
// warps go on at once.  Every thread of the CTA calls it.
template <bool kMax>
__device__ __forceinline__ void ps_publish(PsShared& sh, const PsBar& bar, int which, int parity,
                                           unsigned long long tag, int nvirt) {
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int i = threadIdx.x & 15, h = threadIdx.x >> 4;
  double a[kPsVirt / 2];
#pragma unroll
  for (int r = 0; r < kPsVirt / 2; ++r) a[r] = 2 * r + h < nvirt ? sh.loc[2 * r + h][i] : 0.0;
  double m = 0.0;
  if (kMax) m = warp_max_nonneg((int)threadIdx.x < (int)(blockDim.x >> 5) ? sh.wmax[threadIdx.x] : 0.0);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
#pragma unroll
    for (int r = 0; r < kPsVirt / 2; ++r) a[r] += __shfl_xor_sync(0xffffffffu, a[r], o);
  if (i == 0) {
#pragma unroll
    for (int r = 0; r < kPsVirt / 2; ++r)
      if (2 * r + h < nvirt) ps_store(bar.sums(which, parity) + blockIdx.x + kPsGrid * (2 * r + h), a[r], tag);
    if (kMax && h == 0) ps_store(bar.maxima(parity) + blockIdx.x, m, tag);
  }
  __syncwarp();
  if (threadIdx.x == 0) ps_arrive(bar.counter);
}

// Second half: waits for the `target`-th arrival, then every thread gets the
// grid's sum (and maximum).  `hook` runs once all CTAs have arrived, before the
// sums are formed, and returns false when a wait of its own ran out.  Returns
// false when any wait ran out.
template <bool kMax, typename Hook>
__device__ __forceinline__ bool ps_wait(PsShared& sh, const PsBar& bar, int which, int parity,
                                        unsigned long long tag, int nred, unsigned long long target, double& S,
                                        double& M, Hook hook) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int dead = 0;
  if (threadIdx.x == 0) dead = !ps_poll(bar.counter, target);
  dead = __syncthreads_or(dead);
  if (dead) return false;
  if (threadIdx.x < PF_TV) {
    // thread q sums entries q, q + 512, ... in that order
    const PsPair* e = bar.sums(which, parity);
    constexpr int kPer = (kMaxRedBlocks + PF_TV - 1) / PF_TV;
    const bool has_max = kMax && threadIdx.x < gridDim.x;
    double v[kPer], m = 0.0;
    unsigned long long have[kPer], hm = tag;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      v[u] = 0.0;
      have[u] = tag;
      if (threadIdx.x + u * PF_TV < nred) ps_load(e + threadIdx.x + u * PF_TV, v[u], have[u]);
    }
    if (has_max) ps_load(bar.maxima(parity) + threadIdx.x, m, hm);
    if (!hook()) dead = 1;
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (!ps_await(e + threadIdx.x + u * PF_TV, v[u], have[u], tag)) dead = 1;
      if (threadIdx.x + u * PF_TV < nred) s += v[u];
    }
    if (kMax) {
      if (!ps_await(bar.maxima(parity) + threadIdx.x, m, hm, tag)) dead = 1;
      static_assert(kPsGrid <= 8 * 32, "gmax holds one maximum per warp that loads them");
      if (wid < 8) {
        m = warp_max_nonneg(m);
        if (lane == 0) sh.gmax[wid] = m;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sh.glob[wid] = s;
  } else if (!hook()) {
    dead = 1;
  }
  dead = __syncthreads_or(dead);
  double s = sh.glob[lane & 15];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  S = s;
  if (kMax) M = warp_max_nonneg(sh.gmax[lane & 7]);
  return !dead;
}

// index of the cell that face value q (0..63) of face d touches: the
// neighbour's boundary cell
__device__ __forceinline__ int halo_cell(int d, int q) {
  const int a = q & 7, b = q >> 3;
  switch (d) {
    case 0: return (a << 3) | (b << 6);          // +x neighbour, its x = 0
    case 1: return 7 | (a << 3) | (b << 6);
    case 2: return a | (b << 6);                 // +y neighbour, its y = 0
    case 3: return a | 56 | (b << 6);
    case 4: return a | (b << 3);
    default: return a | (b << 3) | 448;
  }
}

// The scalars of a solve, advanced alike by every thread of the grid (the
// rules of finalize_stage, kStagePAp and kStageUpdate).  A launch ends when done is
// set: by its last iteration too (a loop bound of its own took a register and 0.04 us
// of the 7.7 at 64^3), which end_launch takes back while max_iter is not reached.
struct PsScalars {
  double alpha, beta, rz, res, tol;
  int it, stop, done;
  __device__ __forceinline__ PsScalars(const SolveCtl* c, int turns)
      : alpha(0.0), beta(c->beta), rz(c->rz), res(c->res), tol(c->tol), it(c->it), stop(c->it + turns),
        done(c->done) {}
  __device__ __forceinline__ void after_pap(double S) {
    if (!isfinite(S)) done = 4;
    else if (fabs(S) < 1e-30 || !isfinite(rz / S)) done = 2;
    else alpha = rz / S;
  }
  __device__ __forceinline__ void after_update(double S, double M) {
    it += 1;
    res = M;
    if (!isfinite(M) || !isfinite(S)) done = 4;
    else if (M < tol) done = 1;
    else {
      beta = S / rz;
      rz = S;
      if (it >= stop) done = 3;
    }
  }
  __device__ __forceinline__ void end_launch(int max_iter) {
    if (done == 3 && it < max_iter) done = 0;
  }
  __device__ __forceinline__ void store(SolveCtl* c) const {
    c->alpha = alpha;
    c->beta = beta;
    c->rz = rz;
    c->res = res;
    c->it = it;
    c->done = done;
  }
};

}  // namespace pf
