// pf_persist_mixed.cu -- the MIXED mode's inner solve (Jacobi-PCG on A' in
// FP32, couplings and direction FP32 or BF16, FP64 inner products) as one
// persistent kernel, built like k_plain_resident (pf_persist.cu): the vectors
// stay on chip, the CTAs hand over the z of their slots' faces as tagged pairs.
// Roundings, fused multiply-adds and the order of the sums are those of the
// three kernels per iteration it replaces (pf_pcg.cu), so z and the iteration
// count have the same bits.  An inner iteration, three launches and here: 51 x 64
// x 45 cells (three slots a CTA) 25 and 5.5 us, 704 tiles (five) 25.4 and 8.0, 900
// (seven) 31.3 and 9.9, 1000 31.5 and 10.1 (BF16 couplings 33.6 and 10.1).  Eight
// slots are what the partial sums' scratch holds.
#include <cuda_bf16.h>

#include <algorithm>

#include "pf_ctx.h"
#include "pf_persist.cuh"

namespace pf {
namespace {

struct PsMixed {
  int nslots, nred, first;  // first: a fresh start (the direction is z)
  int cc16, cp16;           // couplings / direction in BF16
  SolveCtl* ctl;
  const uint8_t* kind;
  const int* nbr;
  float *e, *r;
  const float* d;
  void* p;
  const void* c[3];
  PsBar bar;
  PsPair* faces;
  unsigned long long tag;
  int turns, max_iter;  // iterations of this launch, at most, and of the solve
};

__device__ __forceinline__ float ld16(const void* a, int is16, size_t i) {
  return is16 ? __bfloat162float(((const __nv_bfloat16*)a)[i]) : ((const float*)a)[i];
}

// Thread l owns cell l of each of the CTA's slots; shared memory holds p with
// the six neighbour faces (3.5 KB a slot) and the couplings (6.8 KB).
constexpr int kMixSlotFloats = PF_TV + kPsFace + 3 * PF_TV + 3 * 64;

template <int U>
__global__ void __launch_bounds__(PF_TV, 1) k_mixed_resident(PsMixed A) {
  extern __shared__ float smf[];
  __shared__ PsShared sh;
  __shared__ int s_nbr[8 * U];
  const int c = blockIdx.x, l = threadIdx.x, lane = l & 31, wid = l >> 5;
  const int k = (A.nslots - c + kPsGrid - 1) / kPsGrid;
  float* s_p = smf;                     // [U][512]
  float* s_hp = s_p + U * PF_TV;        // [U][6][64]: p of the neighbours' faces
  float* s_c = s_hp + U * kPsFace;      // [U][3][512]
  float* s_hc = s_c + U * 3 * PF_TV;    // [U][3][64]: couplings across the high faces
  const int lx = l & 7, ly = (l >> 3) & 7, lz = l >> 6;
  const int fx = ly | (lz << 3), fy = lx | (lz << 3), fz = lx | (ly << 3);
  const int at_x = lx == 7 ? fx : lx == 0 ? 64 + fx : -1;
  const int at_y = ly == 7 ? 128 + fy : ly == 0 ? 192 + fy : -1;
  const int at_z = lz == 7 ? 256 + fz : lz == 0 ? 320 + fz : -1;

  PsScalars sc(A.ctl, A.turns);
  if (A.first) sc.beta = 0.0;
  float e[U], r[U], za[U], dg[U], hz[U];  // za: z, and A'p between the two phases
  unsigned live = 0, pinned = 0, has = 0;  // has: this thread's neighbours across a face exist, 3 bits a slot
#pragma unroll
  for (int u = 0; u < U; ++u) {
    e[u] = r[u] = za[u] = dg[u] = hz[u] = 0.0f;
    if (u >= k) continue;
    const int s = c + kPsGrid * u;
    const size_t o = (size_t)s * PF_TV + l;
    const uint8_t kd = A.kind[o];
    if (kd) live |= 1u << u;
    if (kd == 2) pinned |= 1u << u;
    const int* nb = A.nbr + 6 * (size_t)s;
    if (l < 6) s_nbr[8 * u + l] = nb[l];
    if (nb[lx == 7 ? 0 : 1] >= 0 || (lx > 0 && lx < 7)) has |= 1u << (3 * u);
    if (nb[ly == 7 ? 2 : 3] >= 0 || (ly > 0 && ly < 7)) has |= 2u << (3 * u);
    if (nb[lz == 7 ? 4 : 5] >= 0 || (lz > 0 && lz < 7)) has |= 4u << (3 * u);
    e[u] = A.e[o];
    r[u] = A.r[o];
    dg[u] = A.d[o];
    za[u] = dg[u] > 0.0f ? r[u] / dg[u] : 0.0f;
    s_p[u * PF_TV + l] = ld16(A.p, A.cp16, o);
#pragma unroll
    for (int a = 0; a < 3; ++a) s_c[(3 * u + a) * PF_TV + l] = ld16(A.c[a], A.cc16, o);
    if (l < kPsFace) {
      const int t = nb[l >> 6];
      const size_t h = (size_t)(t >= 0 ? t : 0) * PF_TV + halo_cell(l >> 6, l & 63);
      const float hd = A.d[h], hr = A.r[h];
      s_hp[u * kPsFace + l] = t >= 0 ? ld16(A.p, A.cp16, h) : 0.0f;
      hz[u] = t >= 0 && hd > 0.0f ? hr / hd : 0.0f;
    }
    if (l < 3 * 64) {
      const int a = l >> 6, t = nb[2 * a];
      s_hc[u * 192 + l] = t >= 0 ? ld16(A.c[a], A.cc16, (size_t)t * PF_TV + halo_cell(2 * a, l & 63)) : 0.0f;
    }
  }
  __syncthreads();

  constexpr int N = U <= 1 ? 1 : U <= 2 ? 2 : U <= 4 ? 4 : 8;
  const int own = ps_owner<N>(lane);
  const bool writes = (lane & (32 / N - 1)) == 0;
  bool alive = true;
  unsigned long long arrivals = 0;
  for (int turn = 0; !sc.done; ++turn) {
    const int par = turn & 1;
    const unsigned long long tag = A.tag + turn;
    // ---- phase 1: p = z + beta p, A'p
    const float beta = (float)sc.beta;
    auto direction = [&](float z, float p) {
      const float v = __fmaf_rn(beta, p, z);
      return A.cp16 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
    };
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (l < kPsFace) s_hp[u * kPsFace + l] = direction(hz[u], s_hp[u * kPsFace + l]);
      if ((live >> u) & 1u) s_p[u * PF_TV + l] = direction(za[u], s_p[u * PF_TV + l]);
    }
    __syncthreads();
    double acc[N];
#pragma unroll
    for (int u = 0; u < N; ++u) acc[u] = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!((live >> u) & 1u)) continue;
      const float* sp = s_p + u * PF_TV + l;
      const float* hp = s_hp + u * kPsFace;
      const float* cc = s_c + 3 * u * PF_TV + l;
      const float* hc = s_hc + u * 192;
      const float p0 = sp[0];
      const bool ex = (has >> (3 * u)) & 1u, ey = (has >> (3 * u)) & 2u, ez = (has >> (3 * u)) & 4u;
      float off = 0.0f;  // +x -x +y -y +z -z; a neighbour whose tile is not pooled adds nothing
      if (lx < 7 || ex) off = __fmaf_rn(lx < 7 ? cc[1] : hc[fx], lx < 7 ? sp[1] : hp[fx], off);
      if (lx > 0 || ex) off = __fmaf_rn(cc[0], lx > 0 ? sp[-1] : hp[64 + fx], off);
      if (ly < 7 || ey) off = __fmaf_rn(ly < 7 ? cc[PF_TV + 8] : hc[64 + fy], ly < 7 ? sp[8] : hp[128 + fy], off);
      if (ly > 0 || ey) off = __fmaf_rn(cc[PF_TV], ly > 0 ? sp[-8] : hp[192 + fy], off);
      if (lz < 7 || ez) off = __fmaf_rn(lz < 7 ? cc[2 * PF_TV + 64] : hc[128 + fz], lz < 7 ? sp[64] : hp[256 + fz], off);
      if (lz > 0 || ez) off = __fmaf_rn(cc[2 * PF_TV], lz > 0 ? sp[-64] : hp[320 + fz], off);
      const float ap = (pinned >> u) & 1u ? p0 : __fmaf_rn(dg[u], p0, -off);
      za[u] = ap;
      acc[u] = (double)p0 * (double)ap;
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
    // ---- phase 2: r, z
    const float alpha = (float)sc.alpha;
    double rmax = 0.0;
#pragma unroll
    for (int u = 0; u < N; ++u) acc[u] = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!((live >> u) & 1u)) continue;
      r[u] = __fmaf_rn(-alpha, za[u], r[u]);
      const float z = dg[u] > 0.0f ? r[u] / dg[u] : 0.0f;
      za[u] = z;
      acc[u] = (double)r[u] * (double)z;
      rmax = fmax(rmax, (double)fabsf(r[u]));
    }
    const double rzs = warp_sum_many(acc);
    rmax = warp_max_nonneg(rmax);
    if (writes && own < U) sh.loc[own][wid] = rzs;
    if (lane == 0) sh.wmax[wid] = rmax;
    ps_publish<true>(sh, A.bar, 1, par, tag, k);
    arrivals += gridDim.x;
    // while the other CTAs arrive: the faces and e
    PsPair* out = A.faces + (size_t)par * A.nslots * kPsFace;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= k) continue;
      PsPair* f = out + (size_t)(c + kPsGrid * u) * kPsFace;
      if (at_x >= 0) ps_store(f + at_x, (double)za[u], tag);
      if (at_y >= 0) ps_store(f + at_y, (double)za[u], tag);
      if (at_z >= 0) ps_store(f + at_z, (double)za[u], tag);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((live >> u) & 1u) e[u] = __fmaf_rn(alpha, s_p[u * PF_TV + l], e[u]);
    alive = ps_wait<true>(sh, A.bar, 1, par, tag, A.nred, arrivals, S, M, [&] {
      bool ok = true;
      if (l < kPsFace) {
        const PsPair* f[U];
        unsigned long long have[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int nb = u < k ? s_nbr[8 * u + (l >> 6)] : -1;
          f[u] = out + (size_t)max(nb, 0) * kPsFace + (((l >> 6) ^ 1) << 6) + (l & 63);
          v[u] = 0.0;
          have[u] = tag;
          if (nb >= 0) ps_load(f[u], v[u], have[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          ok = ok && ps_await(f[u], v[u], have[u], tag);
          hz[u] = (float)v[u];
        }
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
    A.e[o] = e[u];
    if (sc.done) continue;  // else the next launch goes on from here
    A.r[o] = r[u];
    if (A.cp16) ((__nv_bfloat16*)A.p)[o] = __float2bfloat16_rn(s_p[u * PF_TV + l]);
    else ((float*)A.p)[o] = s_p[u * PF_TV + l];
  }
  if (c == 0 && l == 0 && alive) sc.store(A.ctl);
  if (!alive && l == 0) A.ctl->aux[0] = 1.0;
}

template <int U>
int launch_mixed(pf_ctx* ctx, PsMixed& a, int grid, bool* refused) {
  const size_t smem = (size_t)U * kMixSlotFloats * sizeof(float);
  void* args[] = {&a};
  return ps_launch(ctx, (const void*)k_mixed_resident<U>, grid, PF_TV, args, smem, smem, refused);
}

int launch_mixed(pf_ctx* ctx, PsMixed& a, int k, int grid, bool* refused) {
  switch (k) {
    case 1: return launch_mixed<1>(ctx, a, grid, refused);
    case 2: return launch_mixed<2>(ctx, a, grid, refused);
    case 3: return launch_mixed<3>(ctx, a, grid, refused);
    case 4: return launch_mixed<4>(ctx, a, grid, refused);
    case 5: case 6: return launch_mixed<6>(ctx, a, grid, refused);
    default: return launch_mixed<8>(ctx, a, grid, refused);
  }
}

}  // namespace

int mixed_persist(pf_ctx* ctx, int nslots, const uint8_t* kind, const int* nbr, float* e, float* r, const float* d,
                  void* p, bool cp16, const void* const c[3], bool cc16, int max_iter, int check_every,
                  SolveCtl* out, int* launched) {
  const int k = (nslots + kPsGrid - 1) / kPsGrid, grid = std::min(nslots, kPsGrid);
  *launched = 0;
  if (nslots <= 0 || ctx->num_sms < kPsGrid || k > kPsVirt) return PF_OK;
  PsMixed a{nslots, std::min(nslots, kMaxRedBlocks), 1, cc16, cp16, ctx->ctl, kind, nbr, e, r, d, p,
            {c[0], c[1], c[2]}, PsBar{ctx->ps_entries, ctx->ps_counter}, ctx->ps_faces, 0, 0, max_iter};
  while (!out->done && *launched < max_iter) {
    a.turns = ps_turns(check_every, kPsTurns, max_iter - *launched);
    a.tag = ctx->ps_tag + 1;
    ctx->ps_tag += a.turns;
    bool refused = false;
    const int rc = launch_mixed(ctx, a, k, grid, &refused);
    if (rc || refused) return rc;
    PF_CUDA_TRY(cudaMemcpyAsync(ctx->h_ctl, ctx->ctl, sizeof(SolveCtl), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    *out = *ctx->h_ctl;
    if (out->aux[0] != 0.0) return set_error(ctx, PF_ERR_CUDA, "pressure solve: a grid-wide wait ran out");
    a.first = 0;
    *launched += a.turns;
  }
  return PF_OK;
}

}  // namespace pf
