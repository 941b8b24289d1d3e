// The FP64 CG's product with the verified stencil operator as a kernel of its
// own (the method: mfe_fixed64.cuh).
#include <atomic>

#include "mfe_cgstate.cuh"
#include "mfe_fixed64.cuh"

namespace mfe {

namespace {

template <int NT, int CM, int NB, bool SEG>
__global__ void __launch_bounds__(NT, NB)
    k_spmv_fixed(const __grid_constant__ FxParams P, double* partials, unsigned* ticket, CgState* st)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[32];
  double dacc[kKP] = {};  // p.Ap of the thread's rows, one chain per row written out
  fx_sweep<NT, CM, SEG, false>(P, blockIdx.x, gridDim.x, smem, dacc);
  const double bt = block_sum((dacc[0] + dacc[1]) + (dacc[2] + dacc[3]), red);
  double total;
  if (grid_reduce_last(bt, partials, ticket, red, &total) && threadIdx.x == 0) {
    st->pAp = total;
    if (total < st->brkdown_tol) st->check_pending = 1;
  }
}

template <int NT, int CM, int NB, bool SEG>
mfe_status fx_launch(mfe_ctx* ctx, const FxParams& P, int grid, const DotSink* sink, CgState* st)
{
  const void* kern = (const void*)k_spmv_fixed<NT, CM, NB, SEG>;
  constexpr size_t smem = FxShape<NT, CM, SEG>::kSmem;
  static std::atomic<bool> set[64];
  if (!set[ctx->device & 63].load(std::memory_order_acquire)) {
    MFE_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set[ctx->device & 63].store(true, std::memory_order_release);
  }
  k_spmv_fixed<NT, CM, NB, SEG><<<grid, NT, smem, ctx->stream>>>(P, sink->partials, sink->ticket, st);
  return check_launch(ctx, "k_spmv_fixed");
}

}  // namespace

mfe_status launch_cg_fixed(mfe_ctx* ctx, const mfe_csr* A, const double* w8, double dd, const double* p,
                           double* Ap, const DotSink* sink, void* cg_state)
{
  FxParams P;
  CgState* st = static_cast<CgState*>(cg_state);
  int g;
  switch (fx_setup(ctx, A, w8, dd, p, Ap, P, &g)) {
    case FX_256X2: return fx_launch<256, 6, 2, false>(ctx, P, g, sink, st);
    case FX_512: return fx_launch<512, 6, 1, false>(ctx, P, g, sink, st);
    default: return fx_launch<256, 13, 1, true>(ctx, P, g, sink, st);
  }
}

}  // namespace mfe
