// The FP64 CG's whole iteration loop as one cooperative kernel, for systems
// whose iterations are short.
//
// As a CUDA graph an iteration is two or three kernels in a while node, and on
// a small box their launches, drains and the node's own test cost 30 us
// whatever the kernels do.  Here the blocks stay resident and meet at three
// grid barriers per iteration (p complete; p.Ap; r.r), about 1.5 us each.  Every
// block sums the blocks' partial dots itself, in block order, and evaluates
// alpha, beta and the loop test from them, so no scalar has to be sent out.
// The arithmetic is the graph kernels' (mfe_cg.cu): for the CSR values the box
// kernel's two partial sums per row, for the stencil the same entries grouped by
// column; the dots' order of summation differs.
//
// A block's share of r, p, x and Ap stays in its shared memory as far as there is
// room (only p is also written out, for the other blocks), and with the CSR
// values so do the values of its first rows.
//
// Three forms of the product: the CSR values of a box matrix (a thread per row,
// columns in closed form), the stencil operator in FP64 (a warp per 30 rows) and
// in fixed point (mfe_fixed64.cuh).
//
// Every wait is bounded: a block that waits longer than kWaitLimitNs records
// ERR_WAIT_TIMEOUT and leaves, and so do the others.
//
// Measured, us per iteration, graph against loop (N(0, 1) right-hand sides):
// CSR values 30^3 24.9 / 11.3, 48 x 40 x 56 29.0 / 17.2, 80^3 60.4 / 45.3, 98^3
// 85.5 / 76.1; stencil 30^3 34.9 / 11.4, 64^3 40 / 22.2, 97 x 64 x 83 41.3 /
// 32.5.  With the vectors and values in global memory the loop took 14.7, 21.7
// and 55.0 (CSR) and, every thread summing its own 27 entries, 15.1 (stencil
// 30^3).  What bounds a small iteration: a barrier takes 1.2 us with 152 blocks
// (one counter; flags that every block polls took 5.1, a value and its sequence
// number in one 16-byte store 3.0), a dot with it 2.8 us (two rounds through L2
// and two five-step sums at 120 clocks a step), seven warps' 27 FMAs on an SM's
// FP64 pipe 1.7 us; from 64^3 on the FP64 pipe: 32 operations per row with the
// CSR values, 22 with the stencil.
#include "mfe_box.cuh"
#include "mfe_cgstate.cuh"
#include "mfe_fixed64.cuh"
#include "mfe_gridloop.cuh"

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
  GridSync sync;
  int held;                // vectors that a block holds in shared memory (r, p, x, Ap in this order)
  int span;                // doubles of each
  int held_chunks;         // CSR operator: chunks of 32 rows whose values the block holds too
  const double* vals;      // CSR operator: box values
  int Nx, Ny, Nz;
  double w[8], dd;         // stencil operator in FP64: class weights, Dirichlet diagonal
};

// row r of the box CSR times p: k_spmv_box's two sums over the 27 slots; vals:
// the values of the warp's 32 rows, from the first lane's row; taken() when
// they are in registers
template <typename Taken>
__device__ __forceinline__ double csr_box_row(const LoopParams& P, int r, const double* vals, double* pr, Taken&& taken)
{
  const int NxNy = P.Nx * P.Ny;
  const int iz = r / NxNy, rem = r - iz * NxNy, iy = rem / P.Nx, ix = rem - iy * P.Nx;
  // row_offset in 32 bits (27 entries of a million rows)
  auto before = [](int i, int n) { return i + max(i - 1, 0) + min(i, n - 1); };
  const int Sx = 3 * P.Nx - 2, nz = nbr(iz, P.Nz);
  const int off = (before(iz, P.Nz) * (3 * P.Ny - 2) + nz * before(iy, P.Ny)) * Sx +
                  nz * nbr(iy, P.Ny) * before(ix, P.Nx);
  const double* rowv = vals + (off - __shfl_sync(~0u, off, 0));
  const double* pc = P.p + r;
  const bool xm = ix > 0, xp = ix < P.Nx - 1, ym = iy > 0, yp = iy < P.Ny - 1, zm = iz > 0, zp = iz < P.Nz - 1;
  double v[27], q[27];
  if (__all_sync(~0u, xm && xp && ym && yp && zm && zp)) {
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
      for (int d = 0; d < 3; ++d) v[3 * j + d] = rowv[3 * j + d];
    taken();
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
      for (int d = 0; d < 3; ++d) q[3 * j + d] = pc[(j / 3 - 1) * NxNy + (j % 3 - 1) * P.Nx + d - 1];
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
        v[3 * j + d] = in ? rowv[k] : 0.0;
        q[3 * j + d] = in ? pc[dz * NxNy + dy * P.Nx + dx] : 0.0;
      }
    taken();
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

// The stencil operator times p in FP64 for the warp's rows first .. first + 29,
// lane l at row first + l - 1.  A lane sums its column's nine entries (Dirichlet
// ones zeroed) by class, weighs them as a centre column and as a side column,
// and takes the sides from its neighbours: 16 FP64 operations per row, where a
// thread that forms its whole row needs 28.  Lanes 0 and 31 are sides only; a
// line's end is a Dirichlet column, whose side is zero.
__device__ __forceinline__ double stencil_rows(const LoopParams& P, int first, double* pr)
{
  const int r = min(max(first + (int)(threadIdx.x & 31) - 1, 0), (int)P.n - 1);
  const int NxNy = P.Nx * P.Ny;
  const int iz = r / NxNy, rem = r - iz * NxNy, iy = rem / P.Nx, ix = rem - iy * P.Nx;
  const double* pc = P.p + r;
  const bool row = ix > 0 && ix < P.Nx - 1 && iy > 0 && iy < P.Ny - 1 && iz > 0 && iz < P.Nz - 1;
  double q[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int dz = k / 3 - 1, dy = k % 3 - 1;
    const bool in = (dy < 0 ? iy > 1 : dy > 0 ? iy < P.Ny - 2 : true) &&
                    (dz < 0 ? iz > 1 : dz > 0 ? iz < P.Nz - 2 : true);
    q[k] = k == 4 || (row && in) ? pc[dz * NxNy + dy * P.Nx] : 0.0;
  }
  *pr = q[4];
  const double a = row ? q[4] : 0.0, b = q[3] + q[5], c = q[1] + q[7], d = (q[0] + q[2]) + (q[6] + q[8]);
  const double centre = fma(P.w[6], d, fma(P.w[4], c, fma(P.w[2], b, P.w[0] * a)));
  const double side = fma(P.w[7], d, fma(P.w[5], c, fma(P.w[3], b, P.w[1] * a)));
  const double l = __shfl_up_sync(~0u, side, 1), u = __shfl_down_sync(~0u, side, 1);
  return row ? centre + (l + u) : P.dd * q[4];
}

// product(Ap): the block's rows of Ap (Ap: where the block keeps its own share);
// returns the thread's terms of p.Ap.  held: the shared memory for P.held vectors.
template <int NT, typename Op>
__device__ __forceinline__ void cg_loop(const LoopParams& P, double* held, Op&& product)
{
  // the CG state: every block keeps the same copy, thread 0 evaluates the
  // scalars, block 0 writes it back
  __shared__ CgState S;
  __shared__ double s_alpha, s_normr, s_v[NT];
  const int tid = threadIdx.x;
  const unsigned G = gridDim.x;
  if (tid == 0) S = *P.st;
  __syncthreads();
  if (!S.cont || S.check_pending) return;
  const int64_t c0 = share<2>(P.n, blockIdx.x, G);
  const int m = (int)(share<2>(P.n, blockIdx.x + 1, G) - c0), h = m / 2;
  const bool tail = (m & 1) && tid == 0;  // an odd n leaves the last block's last entry
  // the share's vectors where the block keeps them, and p where the others read it
  double* const r1 = P.held > 0 ? held : P.r + c0;
  double* const p1 = P.held > 1 ? held + P.span : P.p + c0;
  double* const x1 = P.held > 2 ? held + 2 * P.span : P.x + c0;
  double* const a1 = P.held > 3 ? held + 3 * P.span : P.Ap + c0;
  const bool x_vec = P.x_vec || P.held > 2;
  double2* const r2 = reinterpret_cast<double2*>(r1);
  double2* const p2 = reinterpret_cast<double2*>(p1);
  double2* const x2 = reinterpret_cast<double2*>(x1);
  const double2* const a2 = reinterpret_cast<const double2*>(a1);
  double2* const pg = reinterpret_cast<double2*>(P.p + c0);
  // (every entry is filled, updated and written back by the same thread)
  if (P.held > 0)
    for (int i = tid; i < h; i += NT) r2[i] = reinterpret_cast<const double2*>(P.r + c0)[i];
  if (P.held > 1)
    for (int i = tid; i < h; i += NT) p2[i] = pg[i];
  if (P.held > 2)
    for (int i = tid; i < h; i += NT) {
      x1[2 * i] = P.x[c0 + 2 * i];
      x1[2 * i + 1] = P.x[c0 + 2 * i + 1];
    }
  if (tail) {
    if (P.held > 0) r1[m - 1] = P.r[c0 + m - 1];
    if (P.held > 1) p1[m - 1] = P.p[c0 + m - 1];
    if (P.held > 2) x1[m - 1] = P.x[c0 + m - 1];
  }
  unsigned target = 0;
  bool ok = true;
  for (;;) {
    // p = r, or r + beta p (cg_solve.hpp:153-161)
    const bool first = S.k == 1 || S.p_reset;
    const double beta = S.beta;
#pragma unroll 2
    for (int i = tid; i < h; i += NT) {
      double2 pv = r2[i];
      if (!first) {
        const double2 po = p2[i];
        pv.x = fma(beta, po.x, pv.x);
        pv.y = fma(beta, po.y, pv.y);
      }
      pg[i] = pv;
      if (P.held > 1) p2[i] = pv;
    }
    if (tail) {
      const double pv = first ? r1[m - 1] : fma(beta, p1[m - 1], r1[m - 1]);
      P.p[c0 + m - 1] = pv;
      if (P.held > 1) p1[m - 1] = pv;
    }
    if (!(ok = grid_barrier(P.sync, target += G))) break;
    // Ap, p.Ap and the breakdown pre-test (cg_solve.hpp:179-198)
    const double dot = product(a1);
    ok = grid_sum<NT>(
        dot, s_v, P.partials, P.sync, target += G,
        [&](double total) {
          S.pAp = total;
          if (total < S.brkdown_tol) S.check_pending = 1;
          s_alpha = S.rtrans / total;
        },
        // normr of this iteration's top (cg_solve.hpp:163)
        [&] {
          s_normr = S.num_iters ? sqrt(S.rtrans) : S.normr;
          if (S.record && S.num_iters && blockIdx.x == 0) S.history[S.k] = s_normr;
        });
    if (!ok) break;
    if (S.check_pending) {
      // breakdown() (cg_solve.hpp:49-67): |p.Ap| <= 100 ||Ap|| ||p|| eps.  Near
      // an absolute stop the pre-test fires every few iterations; a breakdown
      // itself is left to the host.
      double pp = 0.0, aa = 0.0;
      for (int i = tid; i < m; i += NT) {
        const double pv = p1[i], av = a1[i];
        pp = fma(pv, pv, pp);
        aa = fma(av, av, aa);
      }
      ok = grid_sum<NT>(aa, s_v, P.partials + G, P.sync, target += G, [&](double total) { s_alpha = total; });
      if (!ok) break;
      ok = grid_sum<NT>(pp, s_v, P.partials, P.sync, target += G, [&](double total) {
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
    if (x_vec) {
#pragma unroll 2
      for (int i = tid; i < h; i += NT) {
        double2 xv = x2[i], rv = r2[i];
        const double2 pv = p2[i], av = a2[i];
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
      for (int i = tid; i < h; i += NT) {
        double2 rv = r2[i];
        const double2 pv = p2[i], av = a2[i];
        x1[2 * i] = fma(alpha, pv.x, x1[2 * i]);
        x1[2 * i + 1] = fma(alpha, pv.y, x1[2 * i + 1]);
        rv.x = fma(-alpha, av.x, rv.x);
        rv.y = fma(-alpha, av.y, rv.y);
        r2[i] = rv;
        acc = fma(rv.x, rv.x, acc);
        acc = fma(rv.y, rv.y, acc);
      }
    }
    if (tail) {
      x1[m - 1] = fma(alpha, p1[m - 1], x1[m - 1]);
      const double rv = fma(-alpha, a1[m - 1], r1[m - 1]);
      r1[m - 1] = rv;
      acc = fma(rv, rv, acc);
    }
    // the loop test of iteration k + 1 with the normr of the top of iteration
    // k (cg_solve.hpp:152-163)
    ok = grid_sum<NT>(acc, s_v, P.partials + G, P.sync, target += G, [&](double total) {
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
  // what the host's breakdown test, a restart and the caller read
  for (int i = tid; i < h; i += NT) {
    if (P.held > 0) reinterpret_cast<double2*>(P.r + c0)[i] = r2[i];
    if (P.held > 2) {
      P.x[c0 + 2 * i] = x1[2 * i];
      P.x[c0 + 2 * i + 1] = x1[2 * i + 1];
    }
    if (P.held > 3) reinterpret_cast<double2*>(P.Ap + c0)[i] = a2[i];
  }
  if (tail) {
    P.r[c0 + m - 1] = r1[m - 1];
    P.x[c0 + m - 1] = x1[m - 1];
    P.Ap[c0 + m - 1] = a1[m - 1];
  }
  if (!ok) {
    if (tid == 0) atomicOr(&P.st->err, ERR_WAIT_TIMEOUT);
  } else if (blockIdx.x == 0 && tid == 0) {
    if (S.check_pending) S.normr = s_normr;
    store_state(P.st, S);
  }
}

// the stencil operator in FP64, a warp per 30 rows
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_loop_stencil(const __grid_constant__ LoopParams P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int c0 = (int)share<2>(P.n, blockIdx.x, gridDim.x), c1 = (int)share<2>(P.n, blockIdx.x + 1, gridDim.x);
  cg_loop<NT>(P, reinterpret_cast<double*>(smem), [&](double* Ap) {
    double d = 0.0;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int f = c0 + 30 * w; f < c1; f += 30 * (NT / 32)) {
      const int r = f + lane - 1;
      double pr;
      const double y = stencil_rows(P, f, &pr);
      if (lane > 0 && lane < 31 && r < c1) {
        Ap[r - c0] = y;
        d = fma(y, pr, d);
      }
    }
    return d;
  });
}

constexpr int kChunk = 27 * 32;   // most values of 32 rows
constexpr int kMostChunks = 511;  // of a block

// The CSR values of a box, a warp per chunk of 32 rows.  A block's first chunks
// stay in shared memory; the others' values come through a buffer per warp, the
// next chunk's on their way while the warp computes, updates vectors or waits
// at a barrier.
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_cg_loop_csr(const __grid_constant__ LoopParams P)
{
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NW = NT / 32;
  const int c0 = (int)share<2>(P.n, blockIdx.x, gridDim.x), c1 = (int)share<2>(P.n, blockIdx.x + 1, gridDim.x);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (c1 - c0 + 31) / 32, held = min(P.held_chunks, chunks);
  double* const hv = reinterpret_cast<double*>(smem) + P.held * P.span;
  double* const buf = hv + P.held_chunks * kChunk + w * kChunk;
  __shared__ int s_off[kMostChunks + 1];  // CSR offset of each chunk
  for (int c = threadIdx.x; c <= chunks; c += NT)
    s_off[c] = (int)row_offset_of(min(c0 + 32 * c, c1), P.Nx, P.Ny, P.Nz);
  __syncthreads();
  auto fetch = [&](int c, double* to) {
    const int lo = s_off[c], hi = s_off[c + 1];
    const unsigned s = (unsigned)__cvta_generic_to_shared(to);
#pragma unroll 9
    for (int i = lane; i < hi - lo; i += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s + 8u * i), "l"(P.vals + lo + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // this warp's chunks through the buffer, over and over: first, first + NW, ...
  const int first = w + (held - w + NW - 1) / NW * NW;
  const bool streams = first < chunks;
  for (int c = w; c < held; c += NW) fetch(c, hv + c * kChunk);
  if (streams) fetch(first, buf);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  cg_loop<NT>(P, reinterpret_cast<double*>(smem), [&](double* Ap) {
    double d = 0.0;
    for (int c = w; c < chunks; c += NW) {
      const bool streamed = c >= held;
      if (streamed) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
      }
      const int r = c0 + 32 * c + lane;
      double pr;
      const double y = csr_box_row(P, min(r, c1 - 1), streamed ? buf : hv + c * kChunk, &pr, [&] {
        __syncwarp();
        if (streamed) fetch(c + NW < chunks ? c + NW : first, buf);
      });
      if (r < c1) {
        Ap[r - c0] = y;
        d = fma(y, pr, d);
      }
    }
    return d;
  });
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int NT, int CM, int NB, bool SEG>
__global__ void __launch_bounds__(NT, NB)
    k_cg_loop_fixed(const __grid_constant__ LoopParams P, const __grid_constant__ FxParams F)
{
  extern __shared__ __align__(16) unsigned char smem[];
  double* const held = reinterpret_cast<double*>(smem + FxShape<NT, CM, SEG>::kSmem);
  cg_loop<NT>(P, held, [&](double*) {
    double d[kKP] = {};
    fx_sweep<NT, CM, SEG, true>(F, blockIdx.x, gridDim.x, smem, d);
    return (d[0] + d[1]) + (d[2] + d[3]);
  });
}

// Half of the SMs while they take 128 rows each: 76 blocks against 152, us per
// iteration, CSR values / stencil, 18^3 10.5, 11.6 / 11.5, 12.6; 21^3 10.6, 11.2 / 10.9,
// 11.7; 24^3 11.4, 12.4 / 10.8, 11.6.
int fp64_blocks(const mfe_ctx* ctx, int64_t n) { return loop_blocks(ctx, n, 64, 64 * (int64_t)ctx->sm_count); }

template <int NT>
mfe_status run_stencil(mfe_ctx* ctx, LoopParams& P)
{
  static std::atomic<int> ready[64];
  const int g = fp64_blocks(ctx, P.n);
  const size_t smem = plan_held(P.n, g, sizeof(double), kRoom, 4, &P.span, &P.held);
  void* args[] = {&P};
  return coop_launch<kRoom>(ctx, (const void*)k_cg_loop_stencil<NT>, g, NT, 1, smem, ready, args);
}

template <int NT>
mfe_status run_csr(mfe_ctx* ctx, LoopParams& P)
{
  static std::atomic<int> ready[64];
  constexpr size_t kChunkBytes = kChunk * sizeof(double), kBuffers = NT / 32 * kChunkBytes;
  const int g = fp64_blocks(ctx, P.n);
  // all values beside all vectors, or the buffers, then vectors, then values
  size_t smem = plan_held(P.n, g, sizeof(double), kRoom, 4, &P.span, &P.held);
  const int chunks = (P.span + 31) / 32;
  if (chunks > kMostChunks) return fail(ctx, MFE_NOT_SUPPORTED, "the CG loop kernel does not fit the device");
  if (P.held == 4 && smem + chunks * kChunkBytes <= kRoom) {
    P.held_chunks = chunks;
    smem += chunks * kChunkBytes;
  } else {
    smem = plan_held(P.n, g, sizeof(double), kRoom - kBuffers, 4, &P.span, &P.held) + kBuffers;
    P.held_chunks = (int)((kRoom - smem) / kChunkBytes);
    smem += P.held_chunks * kChunkBytes;
  }
  void* args[] = {&P};
  return coop_launch<kRoom>(ctx, (const void*)k_cg_loop_csr<NT>, g, NT, 1, smem, ready, args);
}

template <int NT, int CM, int NB, bool SEG>
mfe_status run_fixed(mfe_ctx* ctx, LoopParams& P, FxParams& F, int g)
{
  static std::atomic<int> ready[64];
  constexpr size_t kSweep = FxShape<NT, CM, SEG>::kSmem, kRoom = 227 * 1024 / NB - kReserved;
  static_assert(kSweep <= kRoom, "the sweep's planes");
  const size_t smem = kSweep + plan_held(P.n, g, sizeof(double), kRoom - kSweep, 3, &P.span, &P.held);
  void* args[] = {&P, &F};
  return coop_launch<kRoom>(ctx, (const void*)k_cg_loop_fixed<NT, CM, NB, SEG>, g, NT, NB, smem, ready, args);
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
  P.held_chunks = 0;
  P.x_vec = (reinterpret_cast<uintptr_t>(a.x) & 15u) == 0;
  P.st = static_cast<CgState*>(a.st);
  P.vals = static_cast<const double*>(A->vals);
  P.Nx = A->box_nx + 1;
  P.Ny = A->box_ny + 1;
  P.Nz = A->box_nz + 1;
  double* ws = static_cast<double*>(workspace(ctx, "cg.loop", sizeof(double) * 4096 + 16));
  if (!ws) return fail(ctx, MFE_OOM, "CG workspace allocation failed");
  P.partials = ws;
  MFE_TRY(start_sync(ctx, reinterpret_cast<unsigned*>(ws + 4096), &P.sync));
  // 256 threads while they leave room for most values, else 384, us per
  // iteration: 48 x 40 x 56 17.2 / 16.9, 56^3 22.2 / 24.0, 64^3 31.1 / 28.8,
  // 80^3 48.5 / 45.3 (512: 50.2).
  if (a.w8 == nullptr) return P.n <= 1400 * (int64_t)ctx->sm_count ? run_csr<256>(ctx, P) : run_csr<384>(ctx, P);
  // FP64 against fixed point, us per iteration: 64^3 22.2 / 29.9, 72^3 27.3 /
  // 30.9, 80^3 32.4 / 32.7, 98^3 50.8 / 45.2: the sweep in fixed point takes
  // 12 us whatever the size (planes staged for runs of a step or two), the rows
  // in FP64 16 operations each.  256 threads against 384: 30^3 11.4 / 11.7,
  // 40^3 12.8 / 13.2, 48 x 40 x 56 15.7 / 15.2.
  if (P.n <= 500000) {
    for (int c = 0; c < 8; ++c) P.w[c] = a.w8[c];
    P.dd = a.dd;
    return P.n <= 600 * (int64_t)ctx->sm_count ? run_stencil<256>(ctx, P) : run_stencil<384>(ctx, P);
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
