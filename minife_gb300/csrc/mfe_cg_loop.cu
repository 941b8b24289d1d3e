// The FP64 CG's whole iteration loop as one cooperative kernel, for systems
// whose iterations are short.
//
// As a CUDA graph an iteration is two or three kernels in a while node, and on
// a small box their launches, drains and the node's own test cost 30 us
// whatever the kernels do.  Here the blocks stay resident and meet at three
// grid barriers per iteration (p complete; p.Ap; r.r), about 1.5 us each.  Every
// block sums the blocks' partial dots itself, in block order, and evaluates
// alpha, beta and the loop test from them, so no scalar has to be sent out.
// The arithmetic is the graph kernels' (mfe_cg.cu): the same FMAs per entry
// and, for the CSR values, the box kernel's two partial sums per row; only the
// dots' order of summation differs.
//
// Three forms of the product: the CSR values of a box matrix (a thread per
// row, columns in closed form, values through L1 / L2), the stencil operator in
// FP64 (a thread per row) and in fixed point (mfe_fixed64.cuh).
//
// Every wait is bounded: a block that waits longer than kWaitLimitNs records
// ERR_WAIT_TIMEOUT and leaves, and so do the others.
//
// Measured, us per iteration, graph against loop (N(0, 1) right-hand sides):
// CSR values 30^3 26.4 / 14.7, 48 x 40 x 56 30.6 / 21.7, 80^3 60.4 / 55.0;
// stencil 30^3 34.9 / 15.1, 97 x 64 x 83 41.3 / 32.9.  What bounds a small
// iteration: a barrier takes 1.2 us with 152 blocks (one counter; flags that
// every block polls took 5.1, a value and its sequence number in one 16-byte
// store 3.0), a dot with it 3.4 us (the fence after the block's stores, two
// rounds through L2 and two five-step sums at 120 clocks a step), three rows
// of 27 FMAs per FP64 pipe 1.3 us.
#include <atomic>

#include "mfe_box.cuh"
#include "mfe_cgstate.cuh"
#include "mfe_fixed64.cuh"

namespace mfe {

namespace {

struct LoopParams {
  int64_t n;
  double* x;
  double* r;
  double* p;
  double* Ap;
  int x_vec;               // x is 16-byte aligned
  CgState* st;
  double* partials;        // two sets of one per block: p.Ap, r.r
  unsigned* arrived;       // blocks arrived at the barriers so far (0 at launch)
  const double* vals;      // CSR operator: box values
  int Nx, Ny, Nz;
  double w[8], dd;         // stencil operator in FP64: class weights, Dirichlet diagonal
};

// The calling thread's block arrives at a barrier of all blocks and waits;
// false after the time limit.
__device__ __forceinline__ bool arrive_and_wait(unsigned* arrived, unsigned target)
{
  __threadfence();
  atomicAdd(arrived, 1u);
  auto there = [&] {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
    return (int)(v - target) >= 0;
  };
  if (there()) return true;
  const uint64_t t0 = global_ns();
  for (unsigned i = 1; !there(); ++i)
    if ((i & 255u) == 0 && global_ns() - t0 > kWaitLimitNs) return false;
  return true;
}

// All blocks; false (in every thread of the block) after the time limit.
__device__ __forceinline__ bool grid_barrier(unsigned* arrived, unsigned target)
{
  __shared__ bool s_ok;
  __syncthreads();
  if (threadIdx.x == 0) s_ok = arrive_and_wait(arrived, target);
  __syncthreads();
  return s_ok;
}

// The sum of v over all threads of all blocks, given to then(total) in thread 0
// of every block before a block barrier.  The FP64 pipe takes one warp's
// addition in 17 clocks, so a reduction by shuffles in every warp would cost
// more than the rest: one warp adds the block's values from shared memory, and
// after the grid barrier the blocks' sums in block order.
template <int NT, typename Then>
__device__ __forceinline__ bool grid_sum(double v, double* slots, unsigned* arrived, unsigned target, Then&& then)
{
  __shared__ double s_v[NT];
  __shared__ bool s_ok;
  s_v[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) a[i & 3] += s_v[i * 32 + threadIdx.x];
    const double bt = warp_sum((a[0] + a[1]) + (a[2] + a[3]));
    bool ok = true;
    if (threadIdx.x == 0) {
      __stcg(slots + blockIdx.x, bt);
      ok = arrive_and_wait(arrived, target);
    }
    __syncwarp();
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (unsigned i = threadIdx.x, j = 0; i < gridDim.x; i += 32, ++j) t[j & 3] += __ldcg(slots + i);
    const double total = warp_sum((t[0] + t[1]) + (t[2] + t[3]));
    if (threadIdx.x == 0) {
      s_ok = ok;
      then(total);
    }
  }
  __syncthreads();
  return s_ok;
}

// row r of the box CSR times p: k_spmv_box's two sums over the 27 slots
__device__ __forceinline__ double csr_box_row(const LoopParams& P, int r, double* pr)
{
  const int NxNy = P.Nx * P.Ny;
  const int iz = r / NxNy, rem = r - iz * NxNy, iy = rem / P.Nx, ix = rem - iy * P.Nx;
  const double* rowv = P.vals + row_offset(ix, iy, iz, P.Nx, P.Ny, P.Nz);
  const double* pc = P.p + r;
  const bool xm = ix > 0, xp = ix < P.Nx - 1, ym = iy > 0, yp = iy < P.Ny - 1, zm = iz > 0, zp = iz < P.Nz - 1;
  double v[27], q[27];
  if (__all_sync(__activemask(), xm && xp && ym && yp && zm && zp)) {
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        v[3 * j + d] = __ldg(rowv + 3 * j + d);
        q[3 * j + d] = __ldcg(pc + (j / 3 - 1) * NxNy + (j % 3 - 1) * P.Nx + d - 1);
      }
  } else {
    // the row's entries before those at dz, dy and dx
    const int cx = 1 + xm + xp, cxy = cx * (1 + ym + yp);
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int dz = j / 3 - 1, dy = j % 3 - 1, dx = d - 1;
        const bool in = (dx < 0 ? xm : dx > 0 ? xp : true) && (dy < 0 ? ym : dy > 0 ? yp : true) &&
                        (dz < 0 ? zm : dz > 0 ? zp : true);
        const int k = (dz < 0 ? 0 : dz == 0 ? (int)zm : zm + 1) * cxy +
                      (dy < 0 ? 0 : dy == 0 ? (int)ym : ym + 1) * cx + (dx < 0 ? 0 : dx == 0 ? (int)xm : xm + 1);
        v[3 * j + d] = in ? __ldg(rowv + k) : 0.0;
        q[3 * j + d] = in ? __ldcg(pc + dz * NxNy + dy * P.Nx + dx) : 0.0;
      }
  }
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    if (k & 1) s1 = fma(v[k], q[k], s1);
    else s0 = fma(v[k], q[k], s0);
  }
  *pr = q[13];
  return s0 + s1;
}

// row r of the stencil operator times p in FP64: the class sums over the 27
// neighbours (Dirichlet ones zeroed), or dd * p
__device__ __forceinline__ double stencil_row(const LoopParams& P, int r, double* pr)
{
  const int NxNy = P.Nx * P.Ny;
  const int iz = r / NxNy, rem = r - iz * NxNy, iy = rem / P.Nx, ix = rem - iy * P.Nx;
  const double* pc = P.p + r;
  const bool row = ix > 0 && ix < P.Nx - 1 && iy > 0 && iy < P.Ny - 1 && iz > 0 && iz < P.Nz - 1;
  const bool xm = ix > 1, xp = ix < P.Nx - 2, ym = iy > 1, yp = iy < P.Ny - 2, zm = iz > 1, zp = iz < P.Nz - 2;
  double q[27];
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const int dz = k / 9 - 1, dy = k / 3 % 3 - 1, dx = k % 3 - 1;
    const bool in = (dx < 0 ? xm : dx > 0 ? xp : true) && (dy < 0 ? ym : dy > 0 ? yp : true) &&
                    (dz < 0 ? zm : dz > 0 ? zp : true);
    q[k] = k == 13 || (row && in) ? __ldcg(pc + dz * NxNy + dy * P.Nx + dx) : 0.0;
  }
  *pr = q[13];
  if (!row) return P.dd * q[13];
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int az = 0; az < 2; ++az) {
    double g[9];  // the planes at |dz| = az
#pragma unroll
    for (int t = 0; t < 9; ++t) g[t] = az ? q[t] + q[18 + t] : q[9 + t];
    s0 = fma(P.w[4 * az], g[4], s0);
    s1 = fma(P.w[4 * az + 1], g[3] + g[5], s1);
    s0 = fma(P.w[4 * az + 2], g[1] + g[7], s0);
    s1 = fma(P.w[4 * az + 3], (g[0] + g[2]) + (g[6] + g[8]), s1);
  }
  return s0 + s1;
}

// product(): the block's rows of Ap; returns the thread's terms of p.Ap.
template <int NT, typename Op>
__device__ __forceinline__ void cg_loop(const LoopParams& P, Op&& product)
{
  // the CG state: every block keeps the same copy, thread 0 evaluates the
  // scalars, block 0 writes it back
  __shared__ CgState S;
  __shared__ double s_alpha, s_normr;
  const int tid = threadIdx.x;
  const unsigned G = gridDim.x;
  if (tid == 0) S = *P.st;
  __syncthreads();
  if (!S.cont || S.check_pending) return;
  // the block's rows of the vector updates: an even range
  const int64_t c0 = (P.n * blockIdx.x / G) & ~(int64_t)1;
  const int64_t c1 = blockIdx.x == G - 1 ? P.n : (P.n * (blockIdx.x + 1) / G) & ~(int64_t)1;
  const int64_t h0 = c0 / 2, h1 = c1 / 2;  // as pairs; an odd n leaves the last block's last entry
  const bool tail = (c1 & 1) && tid == 0;
  double2* const r2 = reinterpret_cast<double2*>(P.r);
  double2* const p2 = reinterpret_cast<double2*>(P.p);
  const double2* const a2 = reinterpret_cast<const double2*>(P.Ap);
  double2* const x2 = reinterpret_cast<double2*>(P.x);
  unsigned target = 0;
  bool ok = true;
  for (;;) {
    // normr of this iteration's top, beside the p update (cg_solve.hpp:163)
    if (tid == NT - 1) {
      s_normr = S.num_iters ? sqrt(S.rtrans) : S.normr;
      if (S.record && S.num_iters && blockIdx.x == 0) S.history[S.k] = s_normr;
    }
    // p = r, or r + beta p (cg_solve.hpp:153-161)
    const bool first = S.k == 1 || S.p_reset;
    const double beta = S.beta;
    if (first) {
      for (int64_t i = h0 + tid; i < h1; i += NT) p2[i] = r2[i];
      if (tail) P.p[c1 - 1] = P.r[c1 - 1];
    } else {
#pragma unroll 2
      for (int64_t i = h0 + tid; i < h1; i += NT) {
        const double2 rv = r2[i];
        double2 pv = p2[i];
        pv.x = fma(beta, pv.x, rv.x);
        pv.y = fma(beta, pv.y, rv.y);
        p2[i] = pv;
      }
      if (tail) P.p[c1 - 1] = fma(beta, P.p[c1 - 1], P.r[c1 - 1]);
    }
    if (!(ok = grid_barrier(P.arrived, target += G))) break;
    // Ap, p.Ap and the breakdown pre-test (cg_solve.hpp:179-198)
    const double dot = product();
    ok = grid_sum<NT>(dot, P.partials, P.arrived, target += G, [&](double total) {
      S.pAp = total;
      if (total < S.brkdown_tol) S.check_pending = 1;
      s_alpha = S.rtrans / total;
    });
    if (!ok) break;
    if (S.check_pending) {
      // breakdown() (cg_solve.hpp:49-67): |p.Ap| <= 100 ||Ap|| ||p|| eps.  Near
      // an absolute stop the pre-test fires every few iterations; a breakdown
      // itself is left to the host.
      double pp = 0.0, aa = 0.0;
      for (int64_t i = c0 + tid; i < c1; i += NT) {
        const double pv = P.p[i], av = __ldcg(P.Ap + i);
        pp = fma(pv, pv, pp);
        aa = fma(av, av, aa);
      }
      ok = grid_sum<NT>(aa, P.partials + G, P.arrived, target += G, [&](double total) { s_alpha = total; });
      if (!ok) break;
      ok = grid_sum<NT>(pp, P.partials, P.arrived, target += G, [&](double total) {
        const double pAp = S.pAp;
        if (!(pAp < 0 || fabs(pAp) <= 100 * sqrt(s_alpha) * sqrt(total) * 2.220446049250313e-16)) {
          S.check_pending = 0;
          S.brkdown_tol = 0.1 * pAp;
          s_alpha = S.rtrans / pAp;
        }
      });
      if (!ok || S.check_pending) break;
    }
    // x += alpha p, r -= alpha Ap, r.r (cg_solve.hpp:201-213 + :158)
    const double alpha = s_alpha;
    double acc = 0.0;
    if (P.x_vec) {
#pragma unroll 2
      for (int64_t i = h0 + tid; i < h1; i += NT) {
        double2 xv = x2[i], rv = r2[i];
        const double2 pv = p2[i], av = __ldcg(a2 + i);
        xv.x = fma(alpha, pv.x, xv.x);
        xv.y = fma(alpha, pv.y, xv.y);
        rv.x = fma(-alpha, av.x, rv.x);
        rv.y = fma(-alpha, av.y, rv.y);
        x2[i] = xv;
        r2[i] = rv;
        acc = fma(rv.x, rv.x, acc);
        acc = fma(rv.y, rv.y, acc);
      }
    } else {
      for (int64_t i = h0 + tid; i < h1; i += NT) {
        double2 rv = r2[i];
        const double2 pv = p2[i], av = __ldcg(a2 + i);
        P.x[2 * i] = fma(alpha, pv.x, P.x[2 * i]);
        P.x[2 * i + 1] = fma(alpha, pv.y, P.x[2 * i + 1]);
        rv.x = fma(-alpha, av.x, rv.x);
        rv.y = fma(-alpha, av.y, rv.y);
        r2[i] = rv;
        acc = fma(rv.x, rv.x, acc);
        acc = fma(rv.y, rv.y, acc);
      }
    }
    if (tail) {
      const int64_t t = c1 - 1;
      P.x[t] = fma(alpha, P.p[t], P.x[t]);
      const double rv = fma(-alpha, __ldcg(P.Ap + t), P.r[t]);
      P.r[t] = rv;
      acc = fma(rv, rv, acc);
    }
    // the loop test of iteration k + 1 with the normr of the top of iteration
    // k (cg_solve.hpp:152-163)
    ok = grid_sum<NT>(acc, P.partials + G, P.arrived, target += G, [&](double total) {
      S.rr_new = total;
      S.num_iters = S.k;
      S.p_reset = 0;
      S.normr = s_normr;
      S.cont = (S.k + 1 <= S.max_iter) && (S.normr > S.tol_abs);
      if (S.cont) {
        S.beta = total / S.rtrans;
        S.oldrtrans = S.rtrans;
        S.rtrans = total;
        S.k += 1;
      }
    });
    if (!ok || !S.cont) break;
  }
  if (!ok) {
    if (tid == 0) atomicOr(&P.st->err, ERR_WAIT_TIMEOUT);
  } else if (blockIdx.x == 0 && tid == 0) {
    if (S.check_pending) S.normr = s_normr;
    *P.st = S;
  }
}

// a thread per row; ST: the stencil operator in FP64, else the CSR values
template <int NT, bool ST>
__global__ void __launch_bounds__(NT, 1) k_cg_loop_rows(const __grid_constant__ LoopParams P)
{
  const int c0 = (int)(P.n * blockIdx.x / gridDim.x), c1 = (int)(P.n * (blockIdx.x + 1) / gridDim.x);
  cg_loop<NT>(P, [&] {
    double d = 0.0;
    for (int r = c0 + threadIdx.x; r < c1; r += NT) {
      double pr;
      const double y = ST ? stencil_row(P, r, &pr) : csr_box_row(P, r, &pr);
      __stcg(P.Ap + r, y);
      d = fma(y, pr, d);
    }
    return d;
  });
}

template <int NT, int CM, int NB, bool SEG>
__global__ void __launch_bounds__(NT, NB)
    k_cg_loop_fixed(const __grid_constant__ LoopParams P, const __grid_constant__ FxParams F)
{
  extern __shared__ __align__(16) unsigned char smem[];
  cg_loop<NT>(P, [&] {
    double d[kKP] = {};
    fx_sweep<NT, CM, SEG, true>(F, blockIdx.x, gridDim.x, smem, d);
    return (d[0] + d[1]) + (d[2] + d[3]);
  });
}

// blocks per SM that a cooperative launch can count on (the attribute set, the
// occupancy asked for, once per kernel and device)
mfe_status coop_blocks(mfe_ctx* ctx, const void* kern, int threads, size_t smem, int* per_sm)
{
  MFE_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  MFE_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, threads, smem));
  return MFE_OK;
}

template <int NT, bool ST>
mfe_status run_rows(mfe_ctx* ctx, LoopParams& P)
{
  const void* kern = (const void*)k_cg_loop_rows<NT, ST>;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(P.n, 64), ctx->sm_count));
  void* args[] = {&P};
  MFE_CUDA_TRY(ctx, cudaLaunchCooperativeKernel(kern, dim3(g), dim3(NT), args, 0, ctx->stream));
  return MFE_OK;
}

template <int NT, int CM, int NB, bool SEG>
mfe_status run_fixed(mfe_ctx* ctx, LoopParams& P, FxParams& F, int g)
{
  const void* kern = (const void*)k_cg_loop_fixed<NT, CM, NB, SEG>;
  constexpr size_t smem = FxShape<NT, CM, SEG>::kSmem;
  static std::atomic<int> per_sm[64];
  int have = per_sm[ctx->device & 63].load(std::memory_order_acquire);
  if (have == 0) {
    MFE_TRY(coop_blocks(ctx, kern, NT, smem, &have));
    per_sm[ctx->device & 63].store(have, std::memory_order_release);
  }
  if (have < NB) return fail(ctx, MFE_NOT_SUPPORTED, "the CG loop kernel does not fit the device");
  void* args[] = {&P, &F};
  MFE_CUDA_TRY(ctx, cudaLaunchCooperativeKernel(kern, dim3(g), dim3(NT), args, smem, ctx->stream));
  return MFE_OK;
}

}  // namespace

mfe_status launch_cg_loop(mfe_ctx* ctx, const mfe_csr* A, const CgLoopArgs& a)
{
  LoopParams P;
  P.n = A->nrows;
  P.x = a.x;
  P.r = a.r;
  P.p = a.p;
  P.Ap = a.Ap;
  P.x_vec = (reinterpret_cast<uintptr_t>(a.x) & 15u) == 0;
  P.st = static_cast<CgState*>(a.st);
  P.vals = static_cast<const double*>(A->vals);
  P.Nx = A->box_nx + 1;
  P.Ny = A->box_ny + 1;
  P.Nz = A->box_nz + 1;
  double* ws = static_cast<double*>(workspace(ctx, "cg.loop", sizeof(double) * 4096 + 16));
  if (!ws) return fail(ctx, MFE_OOM, "CG workspace allocation failed");
  P.partials = ws;
  P.arrived = reinterpret_cast<unsigned*>(ws + 4096);
  MFE_CUDA_TRY(ctx, cudaMemsetAsync(P.arrived, 0, sizeof(unsigned), ctx->stream));
  const bool narrow = P.n <= 256 * (int64_t)ctx->sm_count;  // a row per thread in the smaller block
  if (a.w8 == nullptr) return narrow ? run_rows<256, false>(ctx, P) : run_rows<512, false>(ctx, P);
  // The fixed-point sweep has 12 us of work per iteration whatever the size
  // (planes staged for runs of a step or two), the rows in FP64 27 operations
  // each: 48 x 40 x 56 elements 20.2 us per iteration in FP64 against 27.3,
  // 56^3 25.7 / 26.4, 60^3 28.4 / 27.1, 70^3 36.0 / 31.2.
  if (P.n <= 200000) {
    for (int c = 0; c < 8; ++c) P.w[c] = a.w8[c];
    P.dd = a.dd;
    return narrow ? run_rows<256, true>(ctx, P) : run_rows<512, true>(ctx, P);
  }
  FxParams F;
  int g;
  switch (fx_setup(ctx, A, a.w8, a.dd, a.p, a.Ap, F, &g)) {
    case FX_256X2: return run_fixed<256, 6, 2, false>(ctx, P, F, g);
    case FX_512: return run_fixed<512, 6, 1, false>(ctx, P, F, g);
    default: return run_fixed<256, 13, 1, true>(ctx, P, F, g);
  }
}

}  // namespace mfe
