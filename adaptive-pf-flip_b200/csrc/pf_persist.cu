// pf_persist.cu -- the PLAIN pressure solve as one persistent kernel (see
// pf_persist.cuh for the reductions and the grid-wide barriers).
//
// Two kernels, by the slots a CTA owns (k = ceil(nslots / 148)): k_plain_resident
// for k <= 6 (up to 888 slots, e.g. 71^3 cells), k_plain_stream while a slot's
// 4.6 KB of shared memory fit (k <= 49, e.g. 150^3); larger systems, and a device
// that refuses the cooperative launch, take the three kernels of pf_pcg.cu.  Every operation rounds as there and the sums run
// in the same order, so x, the iteration count and the residuals have the same
// bits.  Per iteration, before (three launches) and now: 24^3 cells 21 -> 4.4 us,
// 48^3 25 -> 5.6, 64^3 28.6 -> 7.7, 128^3 80 -> 51.  Where the streaming kernel
// ends, 148^3 takes 87 us and the three kernels at 152^3 101: 93 for as many cells.
// Where the resident one ends (tiles: us resident, streaming): 544: 6.4, 10.4; 704:
// 7.7, 11.1; 810: 8.7, 12.7; with a kernel of eight slots, which spills, 900: 14.1,
// 13.2; 972: 13.1, 12.9; 1000: 14.6, 13.5.
#include <algorithm>

#include "pf_ctx.h"
#include "pf_persist.cuh"
#include "pf_quotient.cuh"

namespace pf {
namespace {

struct PsPlain {
  int nslots, nred;
  SolveCtl* ctl;
  const uint8_t* kind;
  const int* nbr;
  double *x, *r, *p0, *z;
  const double *diag, *cx, *cy, *cz;
  double scale;
  PsBar bar;
  PsPair* faces;  // [2][nslots][6][64]
  unsigned long long tag;
  int turns, max_iter;  // iterations of this launch, at most, and of the solve
};

// ---- everything on chip ---------------------------------------------------

// Two phases between two reductions:
//   phase 1  p = z + beta p, Ap, p.Ap
//   phase 2  r -= alpha Ap, z = r / diag, r.z, max|r|; then x += alpha p
// A cell's neighbours form their new direction themselves from its z and old
// p, so p needs no barrier of its own: the values are the ones the owner forms.
// The CTAs hand over nothing but the z of their slots' faces, as tagged pairs.
// Thread l owns cell l of each of the CTA's slots u = 0 .. U-1 (slot c +
// 148 u, a virtual CTA of its own).  Shared memory holds p (7 KB a slot with
// its six neighbour faces), the couplings (13.5 KB with the high faces') and x
// (4 KB).  512 threads: more would leave under 128 registers, and the U independent
// slots of a thread hide its latencies as well as more warps would.
constexpr int kResSlots = 6;
constexpr int kResSlotDoubles = 2 * PF_TV + kPsFace + 3 * PF_TV + 3 * 64;

template <int U>
__global__ void __launch_bounds__(PF_TV, 1) k_plain_resident(PsPlain A) {
  extern __shared__ double sm[];
  __shared__ PsShared sh;
  __shared__ int s_nbr[8 * U];
  const int c = blockIdx.x, l = threadIdx.x, lane = l & 31, wid = l >> 5;
  const int k = (A.nslots - c + kPsGrid - 1) / kPsGrid;
  double* s_p = sm;                        // [U][512]
  double* s_hp = s_p + U * PF_TV;          // [U][6][64]: p of the neighbours' faces
  double* s_c = s_hp + U * kPsFace;        // [U][3][512]
  double* s_hc = s_c + U * 3 * PF_TV;      // [U][3][64]: couplings across the high faces
  double* s_x = s_hc + U * 3 * 64;         // [U][512]
  const int lx = l & 7, ly = (l >> 3) & 7, lz = l >> 6;
  // this cell's place in the faces: x faces (y, z), y faces (x, z), z faces (x, y)
  const int fx = ly | (lz << 3), fy = lx | (lz << 3), fz = lx | (ly << 3);

  // and the entries of the slot's faces it fills, one per axis at most
  const int at_x = lx == 7 ? fx : lx == 0 ? 64 + fx : -1;
  const int at_y = ly == 7 ? 128 + fy : ly == 0 ? 192 + fy : -1;
  const int at_z = lz == 7 ? 256 + fz : lz == 0 ? 320 + fz : -1;

  PsScalars sc(A.ctl, A.turns);
  double r[U], za[U], dg[U], inv[U], hz[U];  // za: z, and Ap between the two phases
  unsigned live = 0, pinned = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    r[u] = za[u] = dg[u] = inv[u] = hz[u] = 0.0;
    if (u >= k) continue;
    const int s = c + kPsGrid * u;
    const size_t o = (size_t)s * PF_TV + l;
    const uint8_t kd = A.kind[o];
    if (kd) live |= 1u << u;
    if (kd == 2) pinned |= 1u << u;
    if (l < 6) s_nbr[8 * u + l] = A.nbr[6 * (size_t)s + l];
    s_x[u * PF_TV + l] = A.x[o];
    r[u] = A.r[o];
    za[u] = A.z[o];
    dg[u] = A.diag[o];
    inv[u] = inv_of(kd == 2 ? 1.0 : __dmul_rn(A.scale, dg[u]));
    s_p[u * PF_TV + l] = A.p0[o];
    s_c[(3 * u + 0) * PF_TV + l] = A.cx[o];
    s_c[(3 * u + 1) * PF_TV + l] = A.cy[o];
    s_c[(3 * u + 2) * PF_TV + l] = A.cz[o];
    if (l < kPsFace) {
      const int nb = A.nbr[6 * (size_t)s + (l >> 6)];
      const size_t h = (size_t)(nb >= 0 ? nb : 0) * PF_TV + halo_cell(l >> 6, l & 63);
      s_hp[u * kPsFace + l] = nb >= 0 ? A.p0[h] : 0.0;
      hz[u] = nb >= 0 ? A.z[h] : 0.0;
    }
    if (l < 3 * 64) {
      const int a = l >> 6, nb = A.nbr[6 * (size_t)s + 2 * a];
      const double* cc = a == 0 ? A.cx : a == 1 ? A.cy : A.cz;
      s_hc[u * 192 + l] = nb >= 0 ? cc[(size_t)nb * PF_TV + halo_cell(2 * a, l & 63)] : 0.0;
    }
  }
  __syncthreads();

  constexpr int N = U <= 1 ? 1 : U <= 2 ? 2 : U <= 4 ? 4 : 8;  // sums formed at once
  const int own = ps_owner<N>(lane);
  const bool writes = (lane & (32 / N - 1)) == 0;
  bool alive = true;
  unsigned long long arrivals = 0;
  for (int turn = 0; !sc.done; ++turn) {
    const int par = turn & 1;
    const unsigned long long tag = A.tag + turn;
    // ---- phase 1
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (l < kPsFace) s_hp[u * kPsFace + l] = __dadd_rn(hz[u], __dmul_rn(sc.beta, s_hp[u * kPsFace + l]));
      if ((live >> u) & 1u) s_p[u * PF_TV + l] = __dadd_rn(za[u], __dmul_rn(sc.beta, s_p[u * PF_TV + l]));
    }
    __syncthreads();
    double acc[N];
#pragma unroll
    for (int u = 0; u < N; ++u) acc[u] = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!((live >> u) & 1u)) continue;
      const double* sp = s_p + u * PF_TV + l;
      const double* hp = s_hp + u * kPsFace;
      const double* sc0 = s_c + 3 * u * PF_TV + l;
      const double* hc = s_hc + u * 192;
      const double p0 = sp[0];
      const double pn[6] = {lx < 7 ? sp[1] : hp[fx],        lx > 0 ? sp[-1] : hp[64 + fx],
                            ly < 7 ? sp[8] : hp[128 + fy],  ly > 0 ? sp[-8] : hp[192 + fy],
                            lz < 7 ? sp[64] : hp[256 + fz], lz > 0 ? sp[-64] : hp[320 + fz]};
      // +x -x +y -y +z -z, the reference's face order
      const double cf[6] = {lx < 7 ? sc0[1] : hc[fx],
                            sc0[0],
                            ly < 7 ? sc0[PF_TV + 8] : hc[64 + fy],
                            sc0[PF_TV],
                            lz < 7 ? sc0[2 * PF_TV + 64] : hc[128 + fz],
                            sc0[2 * PF_TV]};
      double off = 0.0;
#pragma unroll
      for (int d = 0; d < 6; ++d)
        if (cf[d] != 0.0) off = __dadd_rn(off, __dmul_rn(cf[d], pn[d]));
      const double ap =
          (pinned >> u) & 1u ? p0 : __dmul_rn(A.scale, __dsub_rn(__dmul_rn(dg[u], p0), off));
      za[u] = ap;
      acc[u] = __dmul_rn(p0, ap);
    }
    const double pap = warp_sum_many(acc);
    if (writes && own < U) sh.loc[own][wid] = pap;
    double S = 0.0, M = 0.0;
    ps_publish<false>(sh, A.bar, 0, par, tag, k);
    arrivals += gridDim.x;
    alive = ps_wait<false>(sh, A.bar, 0, par, tag, A.nred, arrivals, S, M, [] { return true; });
    if (!alive) break;
    sc.after_pap(S);
    if (sc.done) break;
    // ---- phase 2
    double rmax = 0.0;
#pragma unroll
    for (int u = 0; u < N; ++u) acc[u] = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!((live >> u) & 1u)) continue;
      r[u] = __dsub_rn(r[u], __dmul_rn(sc.alpha, za[u]));
      const double d = (pinned >> u) & 1u ? 1.0 : __dmul_rn(A.scale, dg[u]);
      const double z = quotient(r[u], d, inv[u]);
      za[u] = z;
      acc[u] = __dmul_rn(r[u], z);
      rmax = fmax(rmax, fabs(r[u]));
    }
    const double rzs = warp_sum_many(acc);
    rmax = warp_max_nonneg(rmax);
    if (writes && own < U) sh.loc[own][wid] = rzs;
    if (lane == 0) sh.wmax[wid] = rmax;
    ps_publish<true>(sh, A.bar, 1, par, tag, k);
    arrivals += gridDim.x;
    // while the other CTAs arrive: the faces (the arrival promises nothing
    // about them, their tags do) and x
    PsPair* out = A.faces + (size_t)par * A.nslots * kPsFace;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= k) continue;
      PsPair* f = out + (size_t)(c + kPsGrid * u) * kPsFace;
      if (at_x >= 0) ps_store(f + at_x, za[u], tag);
      if (at_y >= 0) ps_store(f + at_y, za[u], tag);
      if (at_z >= 0) ps_store(f + at_z, za[u], tag);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((live >> u) & 1u)
        s_x[u * PF_TV + l] = __dadd_rn(s_x[u * PF_TV + l], __dmul_rn(sc.alpha, s_p[u * PF_TV + l]));
    alive = ps_wait<true>(sh, A.bar, 1, par, tag, A.nred, arrivals, S, M, [&] {
      // the z of the neighbours' faces: face d of a slot is face d ^ 1 of the neighbour
      bool ok = true;
      if (l < kPsFace) {
        const PsPair* f[U];
        unsigned long long have[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int nb = u < k ? s_nbr[8 * u + (l >> 6)] : -1;
          f[u] = out + (size_t)max(nb, 0) * kPsFace + (((l >> 6) ^ 1) << 6) + (l & 63);
          hz[u] = 0.0;
          have[u] = tag;
          if (nb >= 0) ps_load(f[u], hz[u], have[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) ok = ok && ps_await(f[u], hz[u], have[u], tag);
      }
      return ok;
    });
    if (!alive) break;
    sc.after_update(S, M);
  }
  sc.end_launch(A.max_iter);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!((live >> u) & 1u)) continue;
    const size_t o = (size_t)(c + kPsGrid * u) * PF_TV + l;
    A.x[o] = s_x[u * PF_TV + l];
    if (sc.done) continue;  // else the next launch goes on from here
    A.r[o] = r[u];
    A.z[o] = za[u];
    A.p0[o] = s_p[u * PF_TV + l];
  }
  if (c == 0 && l == 0 && alive) sc.store(A.ctl);
  if (!alive && l == 0) A.ctl->aux[0] = 1.0;
}

// ---- larger systems ---------------------------------------------------------

// p, the couplings and the diagonal stay in global memory; z and Ap (never
// needed at once, and only by their own cell) share a place in shared memory,
// and r, then x, are kept there for as many of the CTA's slots as fit.  With z
// on chip the direction needs a pass of its own and a third barrier, which is
// the only one that hands over global memory:
//   direction  x += alpha p, p = z + beta p      barrier D (release / acquire)
//   phase 1    Ap, p.Ap                          reduction A
//   phase 2    r -= alpha Ap, z = r / diag       reduction B
// 96 bytes a cell and iteration with nothing kept (p 24, x 16, couplings 24,
// diagonal 16, r 16) against the three-kernel path's 139, 64 with r and x kept.
// (Forming the neighbours' p from their z instead, as the kernel above does,
// saves the barrier but loads 22 values a cell where this loads 14: 63 us an
// iteration at 128^3, long-scoreboard stalls.)
constexpr int kStreamThreads = 2 * PF_TV;  // two halves take alternate virtual CTAs
constexpr size_t ps_slot_bytes() { return PF_TV * sizeof(double) + PF_TV + 8 * sizeof(int); }

__global__ void __launch_bounds__(kStreamThreads, 1) k_plain_stream(PsPlain A, int kr, int kx) {
  extern __shared__ double sm[];
  __shared__ PsShared sh;
  const int c = blockIdx.x;
  const int l = threadIdx.x & (PF_TV - 1), half = threadIdx.x / PF_TV;
  const int lane = threadIdx.x & 31, wid = l >> 5;
  const int k = (A.nslots - c + kPsGrid - 1) / kPsGrid;  // slots of this CTA
  const int nvirt = min(k, kPsVirt);
  kr = min(kr, k);
  kx = min(kx, k);
  double* s_za = sm;                              // [k][512]
  double* s_r = s_za + (size_t)k * PF_TV;         // [kr][512]
  double* s_x = s_r + (size_t)kr * PF_TV;         // [kx][512]
  int* s_nbr = reinterpret_cast<int*>(s_x + (size_t)kx * PF_TV);  // [k][8]
  uint8_t* s_kind = reinterpret_cast<uint8_t*>(s_nbr + 8 * k);    // [k][512]
  PsScalars sc(A.ctl, A.max_iter - A.ctl->it);  // its loop bound ends the launch
  double* P = A.p0;
  for (int m = half; m < k; m += 2) {
    const int s = c + kPsGrid * m, q = m * PF_TV + l;
    const size_t o = (size_t)s * PF_TV + l;
    s_kind[q] = A.kind[o];
    if (l < 8) s_nbr[8 * m + l] = l < 6 ? A.nbr[6 * (size_t)s + l] : -1;
    s_za[q] = A.z[o];
    if (m < kr) s_r[q] = A.r[o];
    if (m < kx) s_x[q] = A.x[o];
  }
  __syncthreads();

  // Phase 1 gives a quarter of the CTA a slot and a thread two x neighbours: half
  // the load instructions of one cell per thread, twice the bytes in flight.  Per
  // iteration 88^3 cells 19.7 -> 16.7 us, 104^3 25.8 -> 22.4; 128^3 stays at 51,
  // where 220 MB per iteration pass through L2 and 100 MB of them to or from DRAM.
  // Phase 2 and the direction lost by it (17.4, 23.0 and 53.3 us with all three).
  const int quarter = threadIdx.x / kPairNT, l2 = 2 * (threadIdx.x % kPairNT);
  const int px = l2 & 7, py = (l2 >> 3) & 7, pz = l2 >> 6;
  constexpr int N = kPsVirt / 2;  // a thread's virtual CTAs are half, half + 2, ...
  const int own = half + 2 * ps_owner<N>(lane);
  const bool writes = (lane & (32 / N - 1)) == 0 && own < nvirt;
  bool pend = false, alive = true;
  unsigned long long arrivals = 0;
  // turns count up to a constant, from where leaves A.turns (a bound in a register
  // changed the allocation of phase 1: 0.5 % at 128^3)
  for (int turn = kPsTurns - A.turns; turn < kPsTurns && !sc.done; ++turn) {
    const int par = turn & 1;
    const unsigned long long tag = A.tag + turn;
    // ---- direction
    constexpr int kD = 4;
    for (int m0 = half; m0 < k; m0 += 2 * kD) {
      double po[kD], xo[kD];
#pragma unroll
      for (int u = 0; u < kD; ++u) {
        const int m = m0 + 2 * u;
        po[u] = xo[u] = 0.0;
        if (m < k) {
          const size_t o = (size_t)(c + kPsGrid * m) * PF_TV + l;
          po[u] = P[o];
          if (m >= kx && pend) xo[u] = A.x[o];
        }
      }
#pragma unroll
      for (int u = 0; u < kD; ++u) {
        const int m = m0 + 2 * u, q = m * PF_TV + l;
        if (m >= k || !s_kind[q]) continue;
        const size_t o = (size_t)(c + kPsGrid * m) * PF_TV + l;
        P[o] = __dadd_rn(s_za[q], __dmul_rn(sc.beta, po[u]));
        if (!pend) continue;
        if (m < kx) s_x[q] = __dadd_rn(s_x[q], __dmul_rn(sc.alpha, po[u]));
        else A.x[o] = __dadd_rn(xo[u], __dmul_rn(sc.alpha, po[u]));
      }
    }
    pend = false;
    arrivals += gridDim.x;
    alive = ps_barrier(A.bar, arrivals);
    if (!alive) break;
    // ---- phase 1: two cells per thread, four slots at a time
    {
      double sum[2][2];  // [virtual CTA quarter + 4 v][even, odd cells]
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        sum[v][0] = sum[v][1] = 0.0;
        for (int m = quarter + 4 * v; m < k; m += kPsVirt) {
          const int q = m * PF_TV + l2, s = c + kPsGrid * m, o = s * PF_TV + l2;
          const uchar2 kd = *reinterpret_cast<const uchar2*>(s_kind + q);
          if (!kd.x && !kd.y) continue;
          const int* nb = s_nbr + 8 * m;
          // the pair's neighbours; -1 where there is none
          auto across = [&](int d, int cell) {
            const int t = nb[d];
            return t >= 0 ? t * PF_TV + cell : -1;
          };
          const int xp = px < 6 ? o + 2 : across(0, l2 & ~7), xm = px > 0 ? o - 1 : across(1, l2 | 7),
                    yp = py < 7 ? o + 8 : across(2, l2 & ~56), ym = py > 0 ? o - 8 : across(3, l2 | 56),
                    zp = pz < 7 ? o + 64 : across(4, l2 & ~448), zm = pz > 0 ? o - 64 : across(5, l2 | 448);
          const double2 zero = make_double2(0.0, 0.0);
          const double2 p = ld_pair(P + o), dg = ld_pair(A.diag + o), cx = ld_pair(A.cx + o);
          const double2 cym = ym >= 0 ? ld_pair(A.cy + o) : zero, czm = zm >= 0 ? ld_pair(A.cz + o) : zero;
          const double2 cyp = yp >= 0 ? ld_pair(A.cy + yp) : zero, czp = zp >= 0 ? ld_pair(A.cz + zp) : zero;
          const double cxp = xp >= 0 ? A.cx[xp] : 0.0, cxm = xm >= 0 ? cx.x : 0.0;
          const double pxp = P[xp >= 0 ? xp : o], pxm = P[xm >= 0 ? xm : o];
          const double2 pyp = ld_pair(P + (yp >= 0 ? yp : o)), pym = ld_pair(P + (ym >= 0 ? ym : o));
          const double2 pzp = ld_pair(P + (zp >= 0 ? zp : o)), pzm = ld_pair(P + (zm >= 0 ? zm : o));
          double2 off = zero;  // each cell's faces in the reference's order, +x -x +y -y +z -z
          auto face = [](double& sum, double cf, double pn) {
            if (cf != 0.0) sum = __dadd_rn(sum, __dmul_rn(cf, pn));
          };
          face(off.x, cx.y, p.y);
          face(off.y, cxp, pxp);
          face(off.x, cxm, pxm);
          face(off.y, cx.y, p.x);
          face(off.x, cyp.x, pyp.x);
          face(off.y, cyp.y, pyp.y);
          face(off.x, cym.x, pym.x);
          face(off.y, cym.y, pym.y);
          face(off.x, czp.x, pzp.x);
          face(off.y, czp.y, pzp.y);
          face(off.x, czm.x, pzm.x);
          face(off.y, czm.y, pzm.y);
          double2 ap;
          ap.x = kd.x == 2 ? p.x : __dmul_rn(A.scale, __dsub_rn(__dmul_rn(dg.x, p.x), off.x));
          ap.y = kd.y == 2 ? p.y : __dmul_rn(A.scale, __dsub_rn(__dmul_rn(dg.y, p.y), off.y));
          *reinterpret_cast<double2*>(s_za + q) = ap;
          if (kd.x) sum[v][0] = __dadd_rn(sum[v][0], __dmul_rn(p.x, ap.x));
          if (kd.y) sum[v][1] = __dadd_rn(sum[v][1], __dmul_rn(p.y, ap.y));
        }
      }
      // sixteen threads hold the 32 cells of a warp of phase 2; the same tree
#pragma unroll
      for (int w = 8; w > 0; w >>= 1)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          sum[v][0] += __shfl_xor_sync(0xffffffffu, sum[v][0], w);
          sum[v][1] += __shfl_xor_sync(0xffffffffu, sum[v][1], w);
        }
      if ((lane & 15) == 0)
#pragma unroll
        for (int v = 0; v < 2; ++v) sh.loc[quarter + 4 * v][l2 >> 5] = sum[v][0] + sum[v][1];
    }
    double S = 0.0, M = 0.0;
    // No fence: the sums depend on every p read above, and the owners overwrite
    // p only with a value that depends on the sums.
    ps_publish<false>(sh, A.bar, 0, par, tag, nvirt);
    arrivals += gridDim.x;
    alive = ps_wait<false>(sh, A.bar, 0, par, tag, A.nred, arrivals, S, M, [] { return true; });
    if (!alive) break;
    sc.after_pap(S);
    if (sc.done) break;
    // ---- phase 2
    double acc[N], rmax = 0.0;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      acc[u] = 0.0;
#pragma unroll 2
      for (int m = half + 2 * u; m < k; m += kPsVirt) {
        const int q = m * PF_TV + l;
        const size_t o = (size_t)(c + kPsGrid * m) * PF_TV + l;
        const uint8_t kd = s_kind[q];
        if (!kd) continue;
        const double dg = A.diag[o];
        const double ro = m < kr ? s_r[q] : A.r[o];
        const double r = __dsub_rn(ro, __dmul_rn(sc.alpha, s_za[q]));
        if (m < kr) s_r[q] = r;
        else A.r[o] = r;
        const double d = kd == 2 ? 1.0 : __dmul_rn(A.scale, dg);
        const double z = d > 0.0 ? __ddiv_rn(r, d) : 0.0;
        s_za[q] = z;
        acc[u] = __dadd_rn(acc[u], __dmul_rn(r, z));
        rmax = fmax(rmax, fabs(r));
      }
    }
    const double rzs = warp_sum_many(acc);
    rmax = warp_max_nonneg(rmax);
    if (writes) sh.loc[own][wid] = rzs;
    if (lane == 0) sh.wmax[threadIdx.x >> 5] = rmax;
    ps_publish<true>(sh, A.bar, 1, par, tag, nvirt);
    arrivals += gridDim.x;
    alive = ps_wait<true>(sh, A.bar, 1, par, tag, A.nred, arrivals, S, M, [] { return true; });
    if (!alive) break;
    pend = true;
    sc.after_update(S, M);
  }
  // x's last update, and the state of the next launch when this one's turns are over
  for (int m = half; m < k; m += 2) {
    const int q = m * PF_TV + l;
    const size_t o = (size_t)(c + kPsGrid * m) * PF_TV + l;
    if (!s_kind[q]) continue;
    const double x = m < kx ? s_x[q] : A.x[o];
    A.x[o] = pend ? __dadd_rn(x, __dmul_rn(sc.alpha, P[o])) : x;
    if (sc.done) continue;
    if (m < kr) A.r[o] = s_r[q];
    A.z[o] = s_za[q];
  }
  if (c == 0 && threadIdx.x == 0 && alive) sc.store(A.ctl);
  if (!alive && threadIdx.x == 0) A.ctl->aux[0] = 1.0;
}

template <int U>
int launch_resident(pf_ctx* ctx, PsPlain& a, int grid, bool* refused) {
  const size_t smem = (size_t)U * kResSlotDoubles * sizeof(double);
  void* args[] = {&a};
  return ps_launch(ctx, (const void*)k_plain_resident<U>, grid, PF_TV, args, smem, smem, refused);
}

int launch_resident(pf_ctx* ctx, PsPlain& a, int k, int grid, bool* refused) {
  switch (k) {
    case 1: return launch_resident<1>(ctx, a, grid, refused);
    case 2: return launch_resident<2>(ctx, a, grid, refused);
    case 3: return launch_resident<3>(ctx, a, grid, refused);
    case 4: return launch_resident<4>(ctx, a, grid, refused);
    default: return launch_resident<kResSlots>(ctx, a, grid, refused);
  }
}

// room: what a CTA of this kernel may take
int launch_stream(pf_ctx* ctx, PsPlain& a, int k, int grid, size_t room, bool* refused) {
  const size_t v = PF_TV * sizeof(double), base = k * ps_slot_bytes();
  int kr = (int)std::min<size_t>(k, (room - base) / v);
  int kx = (int)std::min<size_t>(k, (room - base - kr * v) / v);
  void* args[] = {&a, &kr, &kx};
  return ps_launch(ctx, (const void*)k_plain_stream, grid, kStreamThreads, args, room, base + (size_t)(kr + kx) * v,
                   refused);
}

}  // namespace

int ps_launch(pf_ctx* ctx, const void* kernel, int grid, int threads, void** args, size_t smem_max, size_t smem,
              bool* refused) {
  *refused = false;
  PF_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
  PF_CUDA_TRY(cudaMemsetAsync(ctx->ps_counter, 0, sizeof(unsigned long long), ctx->stream));
  const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, smem, ctx->stream);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported || e == cudaErrorLaunchOutOfResources) {
    cudaGetLastError();  // not an error of the solve: leave none behind for the next check
    *refused = true;
    return PF_OK;
  }
  PF_CUDA_TRY(e);
  ++ctx->launches;
  return PF_OK;
}

int plain_persist(pf_ctx* ctx, int nslots, const uint8_t* kind, const int* nbr, PcgVec<double> v, double scale,
                  int max_iter, int check_every, SolveCtl* out, int* launched) {
  *launched = 0;
  if (nslots <= 0 || ctx->num_sms < kPsGrid) return PF_OK;
  const int grid = std::min(nslots, kPsGrid), k = (nslots + kPsGrid - 1) / kPsGrid;
  const size_t room = ctx->smem_optin - sizeof(PsShared) - 64;
  const bool resident = k <= kResSlots;
  if (!resident && k * ps_slot_bytes() > room) return PF_OK;
  PsPlain a{nslots, std::min(nslots, kMaxRedBlocks), ctx->ctl, kind, nbr, v.x, v.r, v.p, v.z, v.diag, v.cx, v.cy,
            v.cz, scale, PsBar{ctx->ps_entries, ctx->ps_counter}, ctx->ps_faces, 0, 0, max_iter};
  while (!out->done && *launched < max_iter) {
    a.turns = ps_turns(check_every, resident ? kPsTurns : kPsStreamTurns / k, max_iter - *launched);
    a.tag = ctx->ps_tag + 1 - (resident ? 0 : kPsTurns - a.turns);  // the tag of turn 0
    ctx->ps_tag += a.turns;
    bool refused = false;
    const int rc = resident ? launch_resident(ctx, a, k, grid, &refused) : launch_stream(ctx, a, k, grid, room, &refused);
    if (rc || refused) return rc;
    PF_CUDA_TRY(cudaMemcpyAsync(ctx->h_ctl, ctx->ctl, sizeof(SolveCtl), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    *out = *ctx->h_ctl;
    if (out->aux[0] != 0.0) return set_error(ctx, PF_ERR_CUDA, "pressure solve: a grid-wide wait ran out");
    *launched += a.turns;
  }
  return PF_OK;
}

}  // namespace pf
