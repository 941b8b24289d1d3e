// The mixed-precision CG's FP32 iterations between two reliable updates as one
// cooperative kernel, for boxes whose iterations are short (the verified
// mirror-symmetric stencil only).
//
// In the graph (mfe_mixed.cu) an iteration is three kernels of a few
// microseconds each.  Here the blocks stay resident, hold their share of r, p,
// x32 and Ap in shared memory (p is also written out, for the other blocks) and
// meet at three barriers per iteration; every block evaluates alpha, beta and
// the update decision from the same sums.  The kernel returns when a reliable
// update is due or the solve ends; the update's kernels and the bookkeeping
// (k_mx_after) follow as in the eager loop.
//
// Rows as in the FP64 loop's stencil (mfe_cg_loop.cu): a warp per 30 rows of the
// x-padded vectors, a column's nine entries per lane, the sides by shuffles.
// Dots in double-float per thread, FP64 from there.
//
// Measured, us per iteration of whole solves, graph against loop: 24^3 18.4 /
// 13.6, 64^3 18.8 / 14.0, 97 x 64 x 130 22.2 / 18.5, 124^3 29.1 / 27.7.  What
// bounds it: the barriers and sums (9 us, mfe_cg_loop.cu); from 80^3 on, the
// instructions per row (about 90 for 30 rows' share of a warp).
#include "mfe_gridloop.cuh"
#include "mfe_mixstate.cuh"

namespace mfe {

namespace {

struct MixLoopParams {
  int64_t n;  // length of the padded vectors
  float* r;
  float* p;
  float* x;
  float* Ap;
  MixState* st;
  double* partials;   // two sets of one per block: p.Ap, r.r
  GridSync sync;
  int held, span;     // vectors held (r, p, x, Ap in this order), floats of each
  int Nx, Ny, Nz, Nxp, NP;
  float w[8], dd;
};

// The stencil operator times p for the warp's rows first .. first + 29, lane l
// at row first + l - 1 (p has zero rows around it; padding entries are zero).
__device__ __forceinline__ float mx_rows(const MixLoopParams& P, int first, float* pr)
{
  const int r = min(max(first + (int)(threadIdx.x & 31) - 1, 0), (int)P.n - 1);
  const int iz = r / P.NP, rem = r - iz * P.NP, iy = rem / P.Nxp, ix = rem - iy * P.Nxp;
  const float* pc = P.p + r;
  const bool row = ix > 0 && ix < P.Nx - 1 && iy > 0 && iy < P.Ny - 1 && iz > 0 && iz < P.Nz - 1;
  float q[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int dz = k / 3 - 1, dy = k % 3 - 1;
    const bool in = (dy < 0 ? iy > 1 : dy > 0 ? iy < P.Ny - 2 : true) &&
                    (dz < 0 ? iz > 1 : dz > 0 ? iz < P.Nz - 2 : true);
    q[k] = k == 4 || (row && in) ? pc[dz * P.NP + dy * P.Nxp] : 0.0f;
  }
  *pr = q[4];
  const float a = row ? q[4] : 0.0f, b = q[3] + q[5], c = q[1] + q[7], d = (q[0] + q[2]) + (q[6] + q[8]);
  const float centre = fmaf(P.w[6], d, fmaf(P.w[4], c, fmaf(P.w[2], b, P.w[0] * a)));
  const float side = fmaf(P.w[7], d, fmaf(P.w[5], c, fmaf(P.w[3], b, P.w[1] * a)));
  const float l = __shfl_up_sync(~0u, side, 1), u = __shfl_down_sync(~0u, side, 1);
  return row ? centre + (l + u) : P.dd * q[4];
}

template <int NT>
__global__ void __launch_bounds__(NT, 1) k_mx_loop(const __grid_constant__ MixLoopParams P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  float* const held = reinterpret_cast<float*>(smem);
  __shared__ MixState S;
  __shared__ float s_alpha;
  __shared__ double s_v[NT];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned G = gridDim.x;
  if (tid == 0) S = *P.st;
  __syncthreads();
  if (!S.cont || S.gate || S.err) return;
  const int64_t c0 = share<4>(P.n, blockIdx.x, G);
  const int m = (int)(share<4>(P.n, blockIdx.x + 1, G) - c0), h = m / 4;  // n is a multiple of 4
  float4* const rg = reinterpret_cast<float4*>(P.r + c0);
  float4* const pg = reinterpret_cast<float4*>(P.p + c0);
  float4* const xg = reinterpret_cast<float4*>(P.x + c0);
  float4* const ag = reinterpret_cast<float4*>(P.Ap + c0);
  float4* const r4 = P.held > 0 ? reinterpret_cast<float4*>(held) : rg;
  float4* const p4 = P.held > 1 ? reinterpret_cast<float4*>(held + P.span) : pg;
  float4* const x4 = P.held > 2 ? reinterpret_cast<float4*>(held + 2 * P.span) : xg;
  float4* const a4 = P.held > 3 ? reinterpret_cast<float4*>(held + 3 * P.span) : ag;
  float* const a1 = reinterpret_cast<float*>(a4);
  // (every entry is filled, updated and written back by the same thread)
  for (int i = tid; i < h; i += NT) {
    if (P.held > 0) r4[i] = rg[i];
    if (P.held > 1) p4[i] = pg[i];
    if (P.held > 2) x4[i] = xg[i];
  }
  unsigned target = 0;
  bool ok = true;
  for (;;) {
    // p = r or r + beta p, after the last iteration's x32 += alpha p (k_mx_p)
    const bool first = S.first != 0, addx = !first && S.x_pending != 0;
    const float beta = (float)S.beta, ap = (float)S.alpha_prev;
#pragma unroll 2
    for (int i = tid; i < h; i += NT) {
      float4 pv = r4[i];
      if (!first) {
        const float4 po = p4[i];
        if (addx) {
          float4 xv = x4[i];
          xv.x = fmaf(ap, po.x, xv.x);
          xv.y = fmaf(ap, po.y, xv.y);
          xv.z = fmaf(ap, po.z, xv.z);
          xv.w = fmaf(ap, po.w, xv.w);
          x4[i] = xv;
        }
        pv.x = fmaf(beta, po.x, pv.x);
        pv.y = fmaf(beta, po.y, pv.y);
        pv.z = fmaf(beta, po.z, pv.z);
        pv.w = fmaf(beta, po.w, pv.w);
      }
      pg[i] = pv;
      if (P.held > 1) p4[i] = pv;
    }
    if (!(ok = grid_barrier(P.sync, target += G))) break;
    DFAcc dot;
    for (int f = 30 * warp; f < m; f += 30 * (NT / 32)) {
      const int i = f + lane - 1;
      float pr;
      const float y = mx_rows(P, (int)c0 + f, &pr);
      if (lane > 0 && lane < 31 && i < m) {
        a1[i] = y;
        dot.add_product(y, pr);
      }
    }
    ok = grid_sum<NT>(dot.value(), s_v, P.partials, P.sync, target += G, [&](double total) {
      S.pAp = total;
      s_alpha = total > 0.0 ? (float)(S.rr / total) : 0.0f;
    });
    if (!ok) break;
    // r -= alpha Ap, r.r (k_mx_update)
    const float alpha = s_alpha;
    DFAcc acc;
#pragma unroll 2
    for (int i = tid; i < h; i += NT) {
      float4 rv = r4[i];
      const float4 av = a4[i];
      rv.x = fmaf(-alpha, av.x, rv.x);
      rv.y = fmaf(-alpha, av.y, rv.y);
      rv.z = fmaf(-alpha, av.z, rv.z);
      rv.w = fmaf(-alpha, av.w, rv.w);
      r4[i] = rv;
      acc.add_product(rv.x, rv.x);
      acc.add_product(rv.y, rv.y);
      acc.add_product(rv.z, rv.z);
      acc.add_product(rv.w, rv.w);
    }
    ok = grid_sum<NT>(acc.value(), s_v, P.partials + G, P.sync, target += G, [&](double total) {
      S.rr_new = total;
      S.alpha_prev = alpha;
      S.x_pending = 1;
      S.k += 1;
      S.since += 1;
      S.first = 0;
      if (S.record && blockIdx.x == 0) S.history[S.k] = sqrt(total);
      if (!(S.pAp > 0.0)) S.status = MFE_BREAKDOWN;  // cg_solve.hpp:187
      S.gate = S.status == 0 && (S.since >= S.refine_k || total < S.delta2 * S.rr_at_update ||
                                 total <= S.tol_abs * S.tol_abs || S.k >= S.max_iter);
      if (!S.gate && S.status == 0) {
        S.beta = total / S.rr;
        S.rr = total;
      }
    });
    if (!ok || S.gate || S.status != 0) break;
  }
  // what the reliable update reads
  for (int i = tid; i < h; i += NT) {
    if (P.held > 0) rg[i] = r4[i];
    if (P.held > 2) xg[i] = x4[i];
  }
  if (!ok) {
    if (tid == 0) atomicOr(&P.st->err, ERR_WAIT_TIMEOUT);
  } else if (blockIdx.x == 0 && tid == 0) {
    store_state(P.st, S);
  }
}

template <int NT>
mfe_status run_mx_loop(mfe_ctx* ctx, MixLoopParams& P)
{
  static std::atomic<int> ready[64];
  constexpr size_t kMost = kRoom - 2048;  // its state and a double per thread
  // half of the SMs while they take 1,024 entries each: 76 blocks against 152, us per
  // iteration, 20^3 13.3 / 13.3, 40^3 12.5 / 12.5, 48^3 13.1 / 12.2
  const int g = loop_blocks(ctx, P.n, 128, 512 * (int64_t)ctx->sm_count);
  const size_t bytes = plan_held(P.n, g, sizeof(float), kMost, 4, &P.span, &P.held);
  void* args[] = {&P};
  return coop_launch<kMost>(ctx, (const void*)k_mx_loop<NT>, g, NT, 1, bytes, ready, args);
}

}  // namespace

mfe_status launch_mixed_loop(mfe_ctx* ctx, const mfe_csr* A, const float* coef, float* r, float* p, float* x32,
                             float* Ap, void* st)
{
  MixLoopParams P;
  P.n = stencil_rows(A);
  P.r = r;
  P.p = p;
  P.x = x32;
  P.Ap = Ap;
  P.st = static_cast<MixState*>(st);
  P.Nx = A->box_nx + 1;
  P.Ny = A->box_ny + 1;
  P.Nz = A->box_nz + 1;
  P.Nxp = stencil_pitch(A);
  P.NP = P.Nxp * P.Ny;
  if (!stencil_mirror_classes(coef, P.w))
    return fail(ctx, MFE_NOT_SUPPORTED, "the loop takes mirror-symmetric stencils");
  P.dd = coef[27];
  double* ws = static_cast<double*>(workspace(ctx, "mixed.loop", sizeof(double) * 4096 + 16));
  if (!ws) return fail(ctx, MFE_OOM, "mixed solver workspace allocation failed");
  P.partials = ws;
  MFE_TRY(start_sync(ctx, reinterpret_cast<unsigned*>(ws + 4096), &P.sync));
  // 512 threads against 1024, us per iteration: 64^3 14.0 / 14.9, 97 x 64 x 130
  // 18.5 / 18.6, 110^3 24.5 / 23.3, 124^3 30.1 / 27.7
  return P.n <= 6000 * (int64_t)ctx->sm_count ? run_mx_loop<512>(ctx, P) : run_mx_loop<1024>(ctx, P);
}

}  // namespace mfe
