// C ABI entry points (include/minife_gb300.h): context, memory, argument
// checking, and dispatch to the kernels of mfe_assemble.cu, mfe_spmv.cu and
// mfe_cg.cu.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstdint>
#include <cstring>
#include <tuple>
#include <atomic>
#include <mutex>
#include <map>
#include <thread>
#include <vector>

#include <sched.h>

#include "mfe_box.cuh"
#include "mfe_internal.h"

namespace mfe {

mfe_status fail(mfe_ctx* ctx, mfe_status st, const std::string& msg)
{
  if (ctx) ctx->err = msg;
  return st;
}

mfe_status cuda_fail(mfe_ctx* ctx, cudaError_t e, const char* where)
{
  std::string m = std::string(where) + ": " + cudaGetErrorString(e);
  if (e == cudaErrorMemoryAllocation) return fail(ctx, MFE_OOM, m);
  return fail(ctx, MFE_CUDA_ERR, m);
}

mfe_status check_launch(mfe_ctx* ctx, const char* where)
{
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, where);
  return MFE_OK;
}

void* workspace(mfe_ctx* ctx, const char* name, size_t bytes)
{
  mfe_ctx::Buf& b = ctx->ws[name];
  if (b.bytes >= bytes && b.ptr) return b.ptr;
  if (b.ptr) {
    // the old buffer may still be in use by queued work
    cudaStreamSynchronize(ctx->stream);
    cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
  }
  void* p = nullptr;
  if (cudaMalloc(&p, std::max<size_t>(bytes, 256)) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  b.ptr = p;
  b.bytes = std::max<size_t>(bytes, 256);
  return p;
}

void* host_scratch(mfe_ctx* ctx, size_t bytes)
{
  if (ctx->host_scratch_bytes >= bytes) return ctx->host_scratch;
  if (ctx->host_scratch) {
    cudaStreamSynchronize(ctx->stream);
    cudaFreeHost(ctx->host_scratch);
  }
  ctx->host_scratch = nullptr;
  ctx->host_scratch_bytes = 0;
  const size_t sz = std::max<size_t>(bytes, 4096);
  if (cudaMallocHost(&ctx->host_scratch, sz) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  ctx->host_scratch_bytes = sz;
  return ctx->host_scratch;
}

static mfe_status set_device(mfe_ctx* ctx)
{
  MFE_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  return MFE_OK;
}

static bool box_ok(int nx, int ny, int nz)
{
  if (nx < 1 || ny < 1 || nz < 1) return false;
  return box_nnz(nx, ny, nz) < ((int64_t)1 << 31);
}

static mfe_status check_csr(mfe_ctx* ctx, const mfe_csr* A)
{
  if (!A) return fail(ctx, MFE_BAD_ARG, "null matrix");
  if (A->nrows < 0 || A->nnz < 0 || A->nnz >= ((int64_t)1 << 31) || A->nrows >= ((int64_t)1 << 31))
    return fail(ctx, MFE_BAD_ARG, "matrix sizes out of range for 32-bit indices");
  if (A->nrows > 0 && (!A->row_offsets || (A->nnz > 0 && (!A->cols || !A->vals))))
    return fail(ctx, MFE_BAD_ARG, "null matrix array");
  if (A->dtype != MFE_F64 && A->dtype != MFE_F32) return fail(ctx, MFE_BAD_ARG, "bad dtype");
  return MFE_OK;
}

int resident_blocks(mfe_ctx* ctx, const void* kernel, int threads, size_t smem)
{
  static std::map<std::tuple<const void*, int, int, size_t>, int> cache;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(kernel, ctx->device, threads, smem);
  auto it = cache.find(key);
  if (it == cache.end()) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) != cudaSuccess) b = 4;
    it = cache.emplace(key, std::max(b, 1)).first;
  }
  return it->second * ctx->sm_count;
}

}  // namespace mfe

using namespace mfe;

extern "C" {

int mfe_abi_version(void) { return MFE_ABI_VERSION; }

const char* mfe_status_string(mfe_status s)
{
  switch (s) {
    case MFE_OK: return "ok";
    case MFE_BAD_ARG: return "bad argument";
    case MFE_OOM: return "out of device memory";
    case MFE_CUDA_ERR: return "CUDA error";
    case MFE_BREAKDOWN: return "numerical breakdown";
    case MFE_MAXITER: return "iteration limit reached";
    case MFE_TIMEOUT: return "device wait timed out";
    case MFE_NOT_SUPPORTED: return "not supported";
  }
  return "unknown status";
}

mfe_status mfe_ctx_create(int device, mfe_ctx** out)
{
  if (!out) return MFE_BAD_ARG;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    cudaGetLastError();
    return MFE_CUDA_ERR;
  }
  if (device < 0 || device >= count) return MFE_BAD_ARG;
  mfe_ctx* ctx = new mfe_ctx();
  ctx->device = device;
  if (cudaSetDevice(device) != cudaSuccess ||
      cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device) !=
          cudaSuccess ||
      cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&ctx->ev0) != cudaSuccess || cudaEventCreate(&ctx->ev1) != cudaSuccess) {
    cudaGetLastError();
    delete ctx;
    return MFE_CUDA_ERR;
  }
  ctx->stream = ctx->own_stream;
  // the products' error word starts at zero (memory may come with what another
  // context left in it)
  void* err = workspace(ctx, "spmv.err", sizeof(unsigned));
  if (!err || cudaMemsetAsync(err, 0, sizeof(unsigned), ctx->stream) != cudaSuccess ||
      cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
    cudaGetLastError();
    mfe_ctx_destroy(ctx);
    return MFE_CUDA_ERR;
  }
  *out = ctx;
  return MFE_OK;
}

mfe_status mfe_ctx_destroy(mfe_ctx* ctx)
{
  if (!ctx) return MFE_OK;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  cg_graph_destroy(ctx->cg_graph);
  for (auto& kv : ctx->ws)
    if (kv.second.ptr) cudaFree(kv.second.ptr);
  if (ctx->f32_copy.owned) {
    cudaFree(ctx->f32_copy.vals);
  }
  if (ctx->host_scratch) cudaFreeHost(ctx->host_scratch);
  if (ctx->side_stream) {
    cudaStreamSynchronize(ctx->side_stream);
    cudaStreamDestroy(ctx->side_stream);
  }
  if (ctx->ev_side) cudaEventDestroy(ctx->ev_side);
  if (ctx->side_pinned) cudaFreeHost(ctx->side_pinned);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
  delete ctx;
  return MFE_OK;
}

static void switch_stream(mfe_ctx* ctx, cudaStream_t s)
{
  if (s != ctx->stream) {
    // work already queued on the old stream completes before the switch
    cudaStreamSynchronize(ctx->stream);
    ctx->stream = s;
  }
}

mfe_status mfe_set_stream(mfe_ctx* ctx, void* stream)
{
  if (!ctx) return MFE_BAD_ARG;
  switch_stream(ctx, static_cast<cudaStream_t>(stream));
  return MFE_OK;
}

mfe_status mfe_use_own_stream(mfe_ctx* ctx)
{
  if (!ctx) return MFE_BAD_ARG;
  switch_stream(ctx, ctx->own_stream);
  return MFE_OK;
}

mfe_status mfe_synchronize(mfe_ctx* ctx)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  // error word of the standalone SpMV/SpMM launches since the last call
  return take_spmv_error(ctx);
}

const char* mfe_last_error_string(const mfe_ctx* ctx)
{
  return ctx ? ctx->err.c_str() : "null context";
}

int mfe_device_sm_count(const mfe_ctx* ctx) { return ctx ? ctx->sm_count : 0; }

mfe_status mfe_device_alloc(mfe_ctx* ctx, size_t bytes, void** out)
{
  if (!ctx || !out) return MFE_BAD_ARG;
  MFE_TRY(set_device(ctx));
  *out = nullptr;
  MFE_CUDA_TRY(ctx, cudaMalloc(out, std::max<size_t>(bytes, 16)));
  return MFE_OK;
}

mfe_status mfe_device_free(mfe_ctx* ctx, void* ptr)
{
  if (!ctx) return MFE_BAD_ARG;
  if (!ptr) return MFE_OK;
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  MFE_CUDA_TRY(ctx, cudaFree(ptr));
  return MFE_OK;
}

mfe_status mfe_memcpy_h2d(mfe_ctx* ctx, void* dst, const void* src, size_t bytes)
{
  if (!ctx || (bytes && (!dst || !src))) return MFE_BAD_ARG;
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
  return MFE_OK;
}

mfe_status mfe_memcpy_d2h(mfe_ctx* ctx, void* dst, const void* src, size_t bytes)
{
  if (!ctx || (bytes && (!dst || !src))) return MFE_BAD_ARG;
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  // error word of the standalone SpMV/SpMM launches since the last call
  return take_spmv_error(ctx);
}

mfe_status mfe_csr_alloc(mfe_ctx* ctx, int64_t nrows, int64_t nnz, mfe_dtype dtype, mfe_csr* out)
{
  if (!ctx || !out || nrows < 0 || nnz < 0 || nnz >= ((int64_t)1 << 31) ||
      (dtype != MFE_F64 && dtype != MFE_F32))
    return fail(ctx, MFE_BAD_ARG, "mfe_csr_alloc: bad arguments");
  MFE_TRY(set_device(ctx));
  memset(out, 0, sizeof(*out));
  const size_t vb = dtype == MFE_F64 ? 8 : 4;
  void *ro = nullptr, *cols = nullptr, *vals = nullptr;
  // values and columns are padded to a 16-byte multiple (bulk-copy granule)
  if (cudaMalloc(&ro, sizeof(int32_t) * (size_t)(nrows + 1)) != cudaSuccess ||
      cudaMalloc(&cols, sizeof(int32_t) * (size_t)(nnz + 4)) != cudaSuccess ||
      cudaMalloc(&vals, vb * (size_t)(nnz + 4)) != cudaSuccess) {
    cudaGetLastError();
    if (ro) cudaFree(ro);
    if (cols) cudaFree(cols);
    if (vals) cudaFree(vals);
    return fail(ctx, MFE_OOM, "mfe_csr_alloc: device allocation failed");
  }
  out->nrows = nrows;
  out->ncols = nrows;
  out->nnz = nnz;
  out->row_offsets = static_cast<int32_t*>(ro);
  out->cols = static_cast<int32_t*>(cols);
  out->vals = vals;
  out->dtype = dtype;
  out->owned = 1;
  return MFE_OK;
}

mfe_status mfe_csr_free(mfe_ctx* ctx, mfe_csr* A)
{
  if (!ctx || !A) return MFE_BAD_ARG;
  if (!A->owned) return fail(ctx, MFE_BAD_ARG, "matrix was not allocated by mfe_csr_alloc");
  cudaStreamSynchronize(ctx->stream);
  if (A->row_offsets) cudaFree(A->row_offsets);
  if (A->cols) cudaFree(A->cols);
  if (A->vals) cudaFree(A->vals);
  memset(A, 0, sizeof(*A));
  return MFE_OK;
}

mfe_status mfe_box_dims(int nx, int ny, int nz, int64_t* nrows, int64_t* nnz)
{
  if (!box_ok(nx, ny, nz)) return MFE_BAD_ARG;
  if (nrows) *nrows = (int64_t)(nx + 1) * (ny + 1) * (nz + 1);
  if (nnz) *nnz = box_nnz(nx, ny, nz);
  return MFE_OK;
}

static mfe_status check_box_matrix(mfe_ctx* ctx, int nx, int ny, int nz, const mfe_csr* A)
{
  if (!box_ok(nx, ny, nz)) return fail(ctx, MFE_BAD_ARG, "box dimensions must be >= 1 and give < 2^31 nonzeros");
  MFE_TRY(check_csr(ctx, A));
  int64_t n, nnz;
  mfe_box_dims(nx, ny, nz, &n, &nnz);
  if (A->nrows != n || A->nnz != nnz)
    return fail(ctx, MFE_BAD_ARG, "matrix is not sized for this box (see mfe_box_dims)");
  return MFE_OK;
}

mfe_status mfe_generate_structure(mfe_ctx* ctx, int nx, int ny, int nz, mfe_csr* A)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_box_matrix(ctx, nx, ny, nz, A));
  MFE_TRY(set_device(ctx));
  MFE_TRY(launch_structure(ctx, nx, ny, nz, A->row_offsets, A->cols));
  const size_t vb = A->dtype == MFE_F64 ? 8 : 4;
  MFE_CUDA_TRY(ctx, cudaMemsetAsync(A->vals, 0, vb * (size_t)A->nnz, ctx->stream));
  A->max_row_len = 27;  // upper bound of the 27-point rows
  A->box_nx = nx;
  A->box_ny = ny;
  A->box_nz = nz;
  return MFE_OK;
}

mfe_status mfe_assemble(mfe_ctx* ctx, int nx, int ny, int nz, const double* kappa, mfe_csr* A,
                        double* b, int impose_bc)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_box_matrix(ctx, nx, ny, nz, A));
  if (A->dtype != MFE_F64) return fail(ctx, MFE_BAD_ARG, "assembly needs an FP64 matrix");
  if (!b) return fail(ctx, MFE_BAD_ARG, "null b");
  MFE_TRY(set_device(ctx));
  MFE_TRY(launch_structure(ctx, nx, ny, nz, A->row_offsets, A->cols));
  MFE_TRY(launch_assemble(ctx, nx, ny, nz, kappa, A->row_offsets, static_cast<double*>(A->vals),
                          b, impose_bc));
  A->max_row_len = 27;  // upper bound of the 27-point rows
  A->box_nx = nx;
  A->box_ny = ny;
  A->box_nz = nz;
  return MFE_OK;
}

mfe_status mfe_impose_dirichlet(mfe_ctx* ctx, mfe_csr* A, double* b, double value,
                                const int32_t* bc_rows, int64_t n_bc)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, A));
  if (A->dtype != MFE_F64) return fail(ctx, MFE_BAD_ARG, "impose_dirichlet needs an FP64 matrix");
  if (!b || n_bc < 0 || (n_bc > 0 && !bc_rows)) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  return launch_impose_dirichlet(ctx, A, b, value, bc_rows, n_bc);
}

mfe_status mfe_box_bc_rows(mfe_ctx* ctx, int nx, int ny, int nz, int which, int32_t* rows,
                           int64_t* count_out)
{
  if (!ctx || !count_out || (which != 0 && which != 1)) return MFE_BAD_ARG;
  if (!box_ok(nx, ny, nz)) return fail(ctx, MFE_BAD_ARG, "bad box");
  const int Nx = nx + 1, Ny = ny + 1, Nz = nz + 1;
  // simple_mesh_description.hpp:62-224 on one rank, ascending (std::set order)
  std::vector<int32_t> v;
  for (int iz = 0; iz < Nz; ++iz)
    for (int iy = 0; iy < Ny; ++iy)
      for (int ix = 0; ix < Nx; ++ix) {
        const bool in = which == 1 ? (ix == Nx - 1)
                                   : (ix == 0 || iy == 0 || iz == 0 || iy == Ny - 1 || iz == Nz - 1);
        if (in) v.push_back((int32_t)(ix + (int64_t)Nx * (iy + (int64_t)Ny * iz)));
      }
  *count_out = (int64_t)v.size();
  if (rows && !v.empty()) {
    MFE_TRY(set_device(ctx));
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(rows, v.data(), sizeof(int32_t) * v.size(),
                                      cudaMemcpyHostToDevice, ctx->stream));
    MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return MFE_OK;
}

mfe_status mfe_csr_convert_f32(mfe_ctx* ctx, const mfe_csr* src, mfe_csr* dst)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, src));
  if (!dst || src->dtype != MFE_F64 || dst->dtype != MFE_F32 || dst->nnz != src->nnz ||
      dst->nrows != src->nrows || !dst->vals)
    return fail(ctx, MFE_BAD_ARG, "mfe_csr_convert_f32: dst must be an FP32 CSR of src's size");
  MFE_TRY(set_device(ctx));
  if (dst->row_offsets != src->row_offsets)
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(dst->row_offsets, src->row_offsets,
                                      sizeof(int32_t) * (size_t)(src->nrows + 1),
                                      cudaMemcpyDeviceToDevice, ctx->stream));
  if (dst->cols != src->cols)
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(dst->cols, src->cols, sizeof(int32_t) * (size_t)src->nnz,
                                      cudaMemcpyDeviceToDevice, ctx->stream));
  dst->max_row_len = src->max_row_len;
  dst->box_nx = src->box_nx;
  dst->box_ny = src->box_ny;
  dst->box_nz = src->box_nz;
  return launch_convert_f32(ctx, static_cast<const double*>(src->vals),
                            static_cast<float*>(dst->vals), src->nnz);
}

mfe_status mfe_spmv(mfe_ctx* ctx, const mfe_csr* A, const void* x, void* y)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, A));
  if (A->nrows > 0 && (!x || !y)) return fail(ctx, MFE_BAD_ARG, "null vector");
  MFE_TRY(set_device(ctx));
  return launch_spmv(ctx, A, x, y, nullptr, nullptr, nullptr);
}

// Where a kernel leaves the scalar of a call that returns it: pinned host
// memory, which the device writes directly (a dot of 29,791 entries from Python:
// 17.7 us against 27.5 with a device scalar and a copy).
static double* host_scalar(mfe_ctx* ctx) { return static_cast<double*>(host_scratch(ctx, sizeof(double))); }

static mfe_status take_scalar(mfe_ctx* ctx, const double* h, double* out)
{
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  *out = *h;
  return MFE_OK;
}

mfe_status mfe_matvec_and_dot(mfe_ctx* ctx, const mfe_csr* A, const void* x, void* y,
                              double* result)
{
  if (!ctx || !result) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, A));
  if (A->nrows > 0 && (!x || !y)) return fail(ctx, MFE_BAD_ARG, "null vector");
  MFE_TRY(set_device(ctx));
  if (A->nrows == 0) {
    *result = 0.0;
    return MFE_OK;
  }
  double* d = host_scalar(ctx);
  double* partials = static_cast<double*>(workspace(ctx, "api.partials", sizeof(double) * 8192));
  const bool fresh = ctx->ws.find("api.ticket") == ctx->ws.end();
  unsigned* ticket = static_cast<unsigned*>(workspace(ctx, "api.ticket", sizeof(unsigned)));
  if (!d || !partials || !ticket) return fail(ctx, MFE_OOM, "workspace allocation failed");
  if (fresh) MFE_CUDA_TRY(ctx, cudaMemsetAsync(ticket, 0, sizeof(unsigned), ctx->stream));
  DotSink sink;
  sink.partials = partials;
  sink.ticket = ticket;
  sink.out = d;
  MFE_TRY(launch_spmv(ctx, A, x, y, &sink, nullptr, nullptr));
  MFE_TRY(take_scalar(ctx, d, result));
  // the call blocks for the scalar anyway: a bounded wait of the product that
  // gave up is reported here, not at the next mfe_synchronize
  return take_spmv_error(ctx);
}

mfe_status mfe_dot(mfe_ctx* ctx, int64_t n, const double* x, const double* y, double* result)
{
  if (!ctx || !result || n < 0 || (n > 0 && (!x || !y))) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  if (n == 0) {
    *result = 0.0;
    return MFE_OK;
  }
  double* d = host_scalar(ctx);
  if (!d) return fail(ctx, MFE_OOM, "workspace allocation failed");
  MFE_TRY(launch_dot(ctx, n, x, y, d));
  return take_scalar(ctx, d, result);
}

mfe_status mfe_waxpby(mfe_ctx* ctx, int64_t n, double alpha, const double* x, double beta,
                      const double* y, double* w)
{
  if (!ctx || n < 0 || (n > 0 && (!x || !y || !w))) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  return launch_waxpby(ctx, n, alpha, x, beta, y, w);
}

mfe_status mfe_fused_waxpby(mfe_ctx* ctx, int64_t n, double alpha, const double* x, double beta,
                            const double* y, double* w, double alpha2, const double* x2,
                            double beta2, const double* y2, double* w2)
{
  if (!ctx || n < 0 || (n > 0 && (!x || !y || !w || !x2 || !y2 || !w2)))
    return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  return launch_fused_waxpby(ctx, n, alpha, x, beta, y, w, alpha2, x2, beta2, y2, w2);
}

mfe_status mfe_stencil64_from_csr(mfe_ctx* ctx, const mfe_csr* A_in, mfe_stencil64* S)
{
  if (!ctx || !S) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(check_csr(ctx, A_in));
  if (A_in->dtype != MFE_F64) return fail(ctx, MFE_BAD_ARG, "the FP64 stencil needs the FP64 matrix");
  MFE_TRY(set_device(ctx));
  mfe_csr A = *A_in;
  if (!csr_is_box(&A)) {
    int bx, by, bz;
    MFE_TRY(detect_box(ctx, &A, &bx, &by, &bz));
    A.box_nx = bx;
    A.box_ny = by;
    A.box_nz = bz;
  }
  bool ok = false;
  memset(S, 0, sizeof(*S));
  if (csr_is_box(&A)) MFE_TRY(stencil64_prepare(ctx, &A, S->w, &S->dd, &ok));
  if (!ok) {
    memset(S, 0, sizeof(*S));
    return fail(ctx, MFE_NOT_SUPPORTED, "A is not a verified miniFE box operator");
  }
  S->box_nx = A.box_nx;
  S->box_ny = A.box_ny;
  S->box_nz = A.box_nz;
  return MFE_OK;
}

mfe_status mfe_spmv_stencil64(mfe_ctx* ctx, const mfe_stencil64* S, const double* x, double* y)
{
  if (!ctx || !S || !x || !y || !box_ok(S->box_nx, S->box_ny, S->box_nz) || S->box_nx < 4 ||
      S->box_ny < 4 || S->box_nz < 4)
    return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  mfe_csr A;
  memset(&A, 0, sizeof(A));
  A.box_nx = S->box_nx;
  A.box_ny = S->box_ny;
  A.box_nz = S->box_nz;
  A.dtype = MFE_F64;
  return launch_spmv_st64(ctx, &A, S->w, S->dd, x, y, nullptr);
}

mfe_status mfe_gather(mfe_ctx* ctx, int64_t n, const int32_t* idx, const double* x, double* out)
{
  if (!ctx || n < 0 || (n > 0 && (!idx || !x || !out))) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  return launch_gather(ctx, n, idx, x, out);
}

mfe_status mfe_dot_f32(mfe_ctx* ctx, int64_t n, const float* x, const float* y, double* result)
{
  if (!ctx || !result || n < 0 || (n > 0 && (!x || !y))) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  if (n == 0) {
    *result = 0.0;
    return MFE_OK;
  }
  double* d = host_scalar(ctx);
  if (!d) return fail(ctx, MFE_OOM, "workspace allocation failed");
  MFE_TRY(launch_dot_f32(ctx, n, x, y, d));
  return take_scalar(ctx, d, result);
}

mfe_status mfe_multi_set_tuning(mfe_ctx* ctx, const mfe_multi_tuning* t)
{
  if (!ctx || !t) return MFE_BAD_ARG;
  if (t->z_chunk != 0 && (t->z_chunk < 4 || t->z_chunk > 1024))
    return fail(ctx, MFE_BAD_ARG, "z_chunk must be 0 or lie in [4, 1024]");
  ctx->multi_zchunk = t->z_chunk;
  return MFE_OK;
}

mfe_status mfe_inject_wait_timeout(mfe_ctx* ctx, int64_t wait_ns)
{
  if (!ctx) return MFE_BAD_ARG;
  if (wait_ns < 1000000 || wait_ns > 2000000000)
    return fail(ctx, MFE_BAD_ARG, "wait_ns must lie in [1 ms, 2 s]");
  ctx->inject_wait_ns = (uint64_t)wait_ns;
  return MFE_OK;
}

mfe_status mfe_inject_loop_fault(mfe_ctx* ctx, int64_t wait_ns)
{
  if (!ctx) return MFE_BAD_ARG;
  if (wait_ns != 0 && (wait_ns < 1000000 || wait_ns > 2000000000))
    return fail(ctx, MFE_BAD_ARG, "wait_ns must be 0 or lie in [1 ms, 2 s]");
  ctx->inject_loop_ns = wait_ns;
  return MFE_OK;
}

void mfe_cg_opts_default(mfe_cg_opts* o)
{
  if (!o) return;
  memset(o, 0, sizeof(*o));
  o->max_iter = 200;
  o->tol_mode = MFE_TOL_ABSOLUTE;
  o->tol = 2.220446049250313e-16;
  o->precision = MFE_PREC_F64;
}

static bool cg_opts_valid(const mfe_cg_opts& o)
{
  return o.max_iter >= 0 && o.tol >= 0.0 &&
         (o.precision == MFE_PREC_F64 || o.precision == MFE_PREC_MIXED) &&
         (o.precond == 0 || o.precond == 1) && (o.f64_operator == 0 || o.f64_operator == 1);
}

mfe_status mfe_cg_solve(mfe_ctx* ctx, const mfe_csr* A, const double* b, double* x,
                        const mfe_cg_opts* opts, mfe_cg_result* result)
{
  if (!ctx || !result) return MFE_BAD_ARG;
  memset(result, 0, sizeof(*result));
  MFE_TRY(check_csr(ctx, A));
  if (A->dtype != MFE_F64) return fail(ctx, MFE_BAD_ARG, "cg_solve needs the FP64 matrix");
  if (A->nrows > 0 && (!b || !x)) return fail(ctx, MFE_BAD_ARG, "null vector");
  mfe_cg_opts o;
  if (opts) o = *opts;
  else mfe_cg_opts_default(&o);
  if (!cg_opts_valid(o)) return fail(ctx, MFE_BAD_ARG, "bad CG options");
  MFE_TRY(set_device(ctx));
  if (A->nrows == 0) return MFE_OK;
  mfe_status st = cg_solve_impl(ctx, A, b, x, &o, result);
  result->status = st;
  return st;
}

namespace {

// Host threads the layout check may use: the CPUs this process may run on.
int host_threads()
{
  cpu_set_t set;
  CPU_ZERO(&set);
  int n = 0;
  if (sched_getaffinity(0, sizeof(set), &set) == 0) n = CPU_COUNT(&set);
  if (n <= 0) n = (int)std::thread::hardware_concurrency();
  return std::max(1, std::min(n, 64));
}

// Whether a host CSR is the closed-form 27-point box layout that
// generate_matrix_structure gives every miniFE matrix (rows in node order,
// ascending in-box neighbour columns): dimensions from row 0 (node (0,0,0):
// columns 0, 1, Nx, Nx + 1, NxNy, ...), then every row offset and column
// compared with the closed form, rows split over the host threads.
bool host_box_layout(int64_t n, int64_t nnz, const int32_t* ro, const int32_t* cols, int* bx,
                     int* by, int* bz)
{
  if (n < 8 || nnz < 8 || ro[0] != 0 || ro[1] != 8 || cols[0] != 0 || cols[1] != 1) return false;
  const int64_t Nx = cols[2], NxNy = cols[4];
  if (Nx < 2 || NxNy < 2 * Nx || NxNy % Nx != 0 || n % NxNy != 0) return false;
  const int64_t Ny = NxNy / Nx, Nz = n / NxNy;
  if (Nz < 2 || box_nnz((int)Nx - 1, (int)Ny - 1, (int)Nz - 1) != nnz) return false;
  if ((int64_t)ro[n] != nnz) return false;
  std::atomic<bool> ok{true};
  // rows are checked line by line (fixed iy, iz); on a line with 1 <= iy <=
  // Ny - 2 and 1 <= iz <= Nz - 2 the rows 1 .. Nx - 2 hold all 27 columns,
  // r + off[k] for fixed offsets, and their offsets step by 27
  int64_t off[27];
  {
    int k = 0;
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) off[k++] = dz * NxNy + dy * Nx + dx;
  }
  auto general_row = [&](int64_t r, int ix, int iy, int iz) {
    int64_t k = row_offset(ix, iy, iz, (int)Nx, (int)Ny, (int)Nz);
    bool good = ro[r] == k;
    for (int dz = -1; dz <= 1; ++dz) {
      if (iz + dz < 0 || iz + dz >= Nz) continue;
      for (int dy = -1; dy <= 1; ++dy) {
        if (iy + dy < 0 || iy + dy >= Ny) continue;
        const int64_t base = r + dz * NxNy + dy * Nx;
        for (int dx = -1; dx <= 1; ++dx) {
          if (ix + dx < 0 || ix + dx >= Nx) continue;
          good &= cols[k++] == base + dx;
        }
      }
    }
    return good;
  };
  const int64_t nlines = Ny * Nz;
  const int nt = (int)std::min<int64_t>(host_threads(), std::max<int64_t>(1, n / 65536));
  auto work = [&](int t) {
    const int64_t l0 = nlines * t / nt, l1 = nlines * (t + 1) / nt;
    for (int64_t l = l0; l < l1; ++l) {
      if (!ok.load(std::memory_order_relaxed)) return;
      const int iy = (int)(l % Ny), iz = (int)(l / Ny);
      const int64_t r0 = l * Nx;
      bool good = general_row(r0, 0, iy, iz) && general_row(r0 + Nx - 1, (int)Nx - 1, iy, iz);
      if (iy >= 1 && iy <= Ny - 2 && iz >= 1 && iz <= Nz - 2) {
        const int64_t k0 = row_offset(1, iy, iz, (int)Nx, (int)Ny, (int)Nz);
        for (int ix = 1; ix <= Nx - 2 && good; ++ix) {
          const int64_t r = r0 + ix, k = k0 + 27 * (int64_t)(ix - 1);
          bool g = ro[r] == k;
          const int32_t* c = cols + k;
          for (int q = 0; q < 27; ++q) g &= (int64_t)c[q] == r + off[q];
          good = g;
        }
      } else {
        for (int ix = 1; ix <= Nx - 2 && good; ++ix) good = general_row(r0 + ix, ix, iy, iz);
      }
      if (!good) {
        ok.store(false, std::memory_order_relaxed);
        return;
      }
    }
  };
  std::vector<std::thread> pool;
  for (int t = 1; t < nt; ++t) pool.emplace_back(work, t);
  work(0);
  for (auto& th : pool) th.join();
  if (!ok.load()) return false;
  *bx = (int)Nx - 1;
  *by = (int)Ny - 1;
  *bz = (int)Nz - 1;
  return true;
}

}  // namespace

namespace {

// Row 0 of a box CSR (node (0,0,0): columns 0, 1, Nx, Nx + 1, NxNy, ...)
// gives the box's dimensions; the sizes must agree with them.  The rest of
// the layout is checked by host_box_layout.
bool host_box_dims(int64_t n, int64_t nnz, const int32_t* ro, const int32_t* cols, int* bx, int* by,
                   int* bz)
{
  if (n < 8 || nnz < 8 || ro[0] != 0 || ro[1] != 8 || cols[0] != 0 || cols[1] != 1) return false;
  const int64_t Nx = cols[2], NxNy = cols[4];
  if (Nx < 2 || NxNy < 2 * Nx || NxNy % Nx != 0 || n % NxNy != 0) return false;
  const int64_t Ny = NxNy / Nx, Nz = n / NxNy;
  if (Nz < 2 || Nx > INT32_MAX || Ny > INT32_MAX || Nz > INT32_MAX) return false;
  if (box_nnz((int)Nx - 1, (int)Ny - 1, (int)Nz - 1) != nnz || (int64_t)ro[n] != nnz) return false;
  *bx = (int)Nx - 1;
  *by = (int)Ny - 1;
  *bz = (int)Nz - 1;
  return true;
}

mfe_status cuda_try(mfe_ctx* ctx, cudaError_t e, const char* where)
{
  return e == cudaSuccess ? MFE_OK : cuda_fail(ctx, e, where);
}

mfe_status side_stream(mfe_ctx* ctx)
{
  if (!ctx->side_stream)
    MFE_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&ctx->side_stream, cudaStreamNonBlocking));
  if (!ctx->ev_side) MFE_CUDA_TRY(ctx, cudaEventCreateWithFlags(&ctx->ev_side, cudaEventDisableTiming));
  if (!ctx->side_pinned)
    MFE_CUDA_TRY(ctx, cudaMallocHost(&ctx->side_pinned, sizeof(double) * kSt64TableLen + 64));
  return MFE_OK;
}

// What the speculative start waits for before a result counts: the host
// layout check (its own thread) and, on the side stream, the values copy and
// the device check of every entry.
struct SpecWait {
  mfe_ctx* ctx;
  std::thread layout;
  std::atomic<int> box{-1};  // 1: the box layout of the expected dimensions
  const unsigned* bad;       // pinned: the device check's result
  bool done = false, ok = false;
};

bool spec_settle(SpecWait* w)
{
  if (w->done) return w->ok;
  w->done = true;
  if (w->layout.joinable()) w->layout.join();
  bool good = cudaEventSynchronize(w->ctx->ev_side) == cudaSuccess &&
              cudaStreamWaitEvent(w->ctx->stream, w->ctx->ev_side, 0) == cudaSuccess;
  w->ok = good && w->box.load() == 1 && *w->bad == 0;
  return w->ok;
}

bool spec_confirm(void* arg) { return spec_settle(static_cast<SpecWait*>(arg)); }

}  // namespace

mfe_status mfe_cg_solve_host(mfe_ctx* ctx, int64_t nrows, int64_t nnz, const int32_t* ro,
                             const int32_t* cols, const double* vals, const double* b, double* x,
                             const mfe_cg_opts* opts, mfe_cg_result* result)
{
  if (!ctx || !result || nrows < 0 || nnz < 0 || nnz >= ((int64_t)1 << 31) ||
      (nrows > 0 && (!ro || !b || !x || (nnz > 0 && (!cols || !vals)))))
    return fail(ctx, MFE_BAD_ARG, "bad arguments");
  mfe_cg_opts o;
  if (opts) o = *opts;
  else mfe_cg_opts_default(&o);
  if (!cg_opts_valid(o)) return fail(ctx, MFE_BAD_ARG, "bad CG options");
  MFE_TRY(set_device(ctx));
  mfe_csr A;
  memset(&A, 0, sizeof(A));
  A.nrows = nrows;
  A.ncols = nrows;
  A.nnz = nnz;
  A.dtype = MFE_F64;
  A.vals = workspace(ctx, "host.vals", sizeof(double) * (size_t)(nnz + 4));
  double* db = static_cast<double*>(workspace(ctx, "host.b", sizeof(double) * (size_t)std::max<int64_t>(nrows, 1)));
  double* dx = static_cast<double*>(workspace(ctx, "host.x", sizeof(double) * (size_t)std::max<int64_t>(nrows, 1)));
  if (!A.vals || !db || !dx) return fail(ctx, MFE_OOM, "device allocation for host operands failed");
  cudaStream_t s = ctx->stream;
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(db, b, sizeof(double) * (size_t)nrows, cudaMemcpyHostToDevice, s));
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(dx, x, sizeof(double) * (size_t)nrows, cudaMemcpyHostToDevice, s));
  // The FP64 solver without preconditioner reads a box matrix's structure in
  // closed form only (box SpMV, stencil check and stencil SpMV), so a CSR
  // whose layout the host has verified is solved without copying its
  // 4 B-per-nonzero column indices and row offsets.
  const bool f64_plain = o.precision == MFE_PREC_F64 && o.precond == 0 &&
                         getenv("MFE_SPMV_GENERIC") == nullptr;
  int qx = 0, qy = 0, qz = 0;
  const bool dims = f64_plain && host_box_dims(nrows, nnz, ro, cols, &qx, &qy, &qz);
  // device arrays for the structure: filled only when the layout is not the box's
  auto structure_bufs = [&](bool box) {
    A.row_offsets = static_cast<int32_t*>(workspace(ctx, "host.ro", sizeof(int32_t) * (size_t)(nrows + 1)));
    A.cols = static_cast<int32_t*>(workspace(ctx, box ? "host.ro" : "host.cols",
                                             box ? sizeof(int32_t) * (size_t)(nrows + 1)
                                                 : sizeof(int32_t) * (size_t)(nnz + 4)));
    return A.row_offsets && A.cols;
  };
  int layout = -1;           // host layout check: 1 box, 0 not, -1 not run
  bool vals_copied = false;  // the values are on their way (ctx->stream waits for them)

  // Speculative start (FP64 stencil operator, x0 = 0): the CG runs while the
  // values are copied and checked on the side stream and the host threads
  // check the layout; the solve's result counts only once all have passed.
  double* htab = nullptr;
  double w8[8], dd = 0.0;
  if (dims && o.f64_operator == 0 && side_stream(ctx) == MFE_OK &&
      (htab = static_cast<double*>(ctx->side_pinned)) != nullptr &&
      stencil64_host_classes(qx + 1, qy + 1, qz + 1, vals, htab, w8, &dd)) {
    cudaStream_t s2 = ctx->side_stream;
    double* dtab = static_cast<double*>(workspace(ctx, "host.st64table", sizeof(double) * kSt64TableLen + 16));
    if (!dtab || !structure_bufs(true)) return fail(ctx, MFE_OOM, "device allocation for host operands failed");
    unsigned* dbad = reinterpret_cast<unsigned*>(dtab + kSt64TableLen);
    unsigned* hbad = reinterpret_cast<unsigned*>(htab + kSt64TableLen);
    *hbad = 1u;
    SpecWait w;
    w.ctx = ctx;
    w.bad = hbad;
    // the side stream starts after the work already queued on ctx->stream
    MFE_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_side, s));
    MFE_CUDA_TRY(ctx, cudaStreamWaitEvent(s2, ctx->ev_side, 0));
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(A.vals, vals, sizeof(double) * (size_t)nnz, cudaMemcpyHostToDevice, s2));
    vals_copied = true;
    mfe_status st = MFE_OK;
    do {
      if ((st = cuda_try(ctx, cudaMemcpyAsync(dtab, htab, sizeof(double) * kSt64TableLen,
                                              cudaMemcpyHostToDevice, s2), "table copy")) != MFE_OK) break;
      if ((st = stencil64_verify_on(ctx, s2, qx + 1, qy + 1, qz + 1, static_cast<const double*>(A.vals),
                                    dtab, dbad)) != MFE_OK) break;
      if ((st = cuda_try(ctx, cudaMemcpyAsync(hbad, dbad, sizeof(unsigned), cudaMemcpyDeviceToHost, s2),
                         "check result copy")) != MFE_OK) break;
      if ((st = cuda_try(ctx, cudaEventRecord(ctx->ev_side, s2), "event")) != MFE_OK) break;
      auto check_layout = [&w, nrows, nnz, ro, cols, qx, qy, qz]() {
        int bx = 0, by = 0, bz = 0;
        const bool ok = host_box_layout(nrows, nnz, ro, cols, &bx, &by, &bz);
        w.box.store(ok && bx == qx && by == qy && bz == qz ? 1 : 0);
      };
      try {
        w.layout = std::thread(check_layout);
      } catch (...) {
        check_layout();  // no thread to spare: check before the solve
      }
      A.box_nx = qx;
      A.box_ny = qy;
      A.box_nz = qz;
      A.max_row_len = 27;
      CgSpec spec;
      for (int c = 0; c < 8; ++c) spec.w8[c] = w8[c];
      spec.dd = dd;
      spec.confirm = spec_confirm;
      spec.arg = &w;
      memset(result, 0, sizeof(*result));
      st = cg_solve_spec(ctx, &A, db, dx, &o, result, &spec);
    } while (false);
    // nothing of this call stays in flight: the host thread ends and the
    // side stream has read the caller's values before anything returns
    spec_settle(&w);
    cudaStreamSynchronize(s2);
    layout = w.box.load();
    if (st != kSpecFailed) {
      if (st != MFE_OK && st != MFE_BREAKDOWN && st != MFE_MAXITER) return st;
      result->status = st;
      MFE_CUDA_TRY(ctx, cudaMemcpyAsync(x, dx, sizeof(double) * (size_t)nrows, cudaMemcpyDeviceToHost, s));
      MFE_CUDA_TRY(ctx, cudaStreamSynchronize(s));
      return st;
    }
    // the speculation did not hold: the ordinary solve from the caller's x0
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(dx, x, sizeof(double) * (size_t)nrows, cudaMemcpyHostToDevice, s));
  }

  if (!vals_copied)
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(A.vals, vals, sizeof(double) * (size_t)nnz, cudaMemcpyHostToDevice, s));
  // while the copy engine moves the values the host threads check the layout
  int bx = 0, by = 0, bz = 0;
  if (layout < 0) layout = dims && host_box_layout(nrows, nnz, ro, cols, &bx, &by, &bz) ? 1 : 0;
  else bx = qx, by = qy, bz = qz;
  const bool box = dims && layout == 1;
  if (!structure_bufs(box)) return fail(ctx, MFE_OOM, "device allocation for host operands failed");
  A.box_nx = A.box_ny = A.box_nz = 0;
  A.max_row_len = 0;
  if (box) {
    A.box_nx = bx;
    A.box_ny = by;
    A.box_nz = bz;
    A.max_row_len = 27;
  } else {
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(A.row_offsets, ro, sizeof(int32_t) * (size_t)(nrows + 1),
                                      cudaMemcpyHostToDevice, s));
    MFE_CUDA_TRY(ctx, cudaMemcpyAsync(A.cols, cols, sizeof(int32_t) * (size_t)nnz, cudaMemcpyHostToDevice, s));
  }
  mfe_status st = mfe_cg_solve(ctx, &A, db, dx, &o, result);
  if (st != MFE_OK && st != MFE_BREAKDOWN && st != MFE_MAXITER) return st;
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(x, dx, sizeof(double) * (size_t)nrows, cudaMemcpyDeviceToHost, s));
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(s));
  return st;
}

mfe_status mfe_cg_history(mfe_ctx* ctx, double* out, int32_t cap, int32_t* count)
{
  if (!ctx || !count) return MFE_BAD_ARG;
  const int32_t n = (int32_t)ctx->history.size();
  *count = n;
  if (out) memcpy(out, ctx->history.data(), sizeof(double) * (size_t)std::min(n, std::max(cap, 0)));
  return MFE_OK;
}

mfe_status mfe_verify_solution(mfe_ctx* ctx, int nx, int ny, int nz, const double* x,
                               double tolerance, int whole_domain, double* max_err, int* passed)
{
  if (!ctx || !x || !max_err) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  if (!box_ok(nx, ny, nz)) return fail(ctx, MFE_BAD_ARG, "bad box");
  MFE_TRY(set_device(ctx));
  MFE_TRY(launch_verify(ctx, nx, ny, nz, x, whole_domain, max_err));
  if (passed) *passed = *max_err <= tolerance ? 1 : 0;
  return MFE_OK;
}

mfe_status mfe_element_gradient(mfe_ctx* ctx, int nx, int ny, int nz, const double* u,
                                const double* lambda, double* g)
{
  if (!ctx || !u || !lambda || !g) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  if (!box_ok(nx, ny, nz)) return fail(ctx, MFE_BAD_ARG, "bad box");
  MFE_TRY(set_device(ctx));
  return launch_element_gradient(ctx, nx, ny, nz, u, lambda, g);
}

mfe_status mfe_adjoint_grad(mfe_ctx* ctx, int nx, int ny, int nz, const double* kappa,
                            const double* u_target, const mfe_cg_opts* opts, double* u_out,
                            double* grad, double* loss, mfe_cg_result* fwd, mfe_cg_result* adj)
{
  if (!ctx) return MFE_BAD_ARG;
  if (!u_target || !grad) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  if (!box_ok(nx, ny, nz)) return fail(ctx, MFE_BAD_ARG, "bad box");
  mfe_cg_opts o;
  if (opts) o = *opts;
  else mfe_cg_opts_default(&o);
  if (!cg_opts_valid(o)) return fail(ctx, MFE_BAD_ARG, "bad CG options");
  MFE_TRY(set_device(ctx));
  return adjoint_grad(ctx, nx, ny, nz, kappa, u_target, &o, u_out, grad, loss, fwd, adj);
}

mfe_status mfe_box_zero_boundary(mfe_ctx* ctx, int nx, int ny, int nz, double* v)
{
  if (!ctx || !v) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  if (!box_ok(nx, ny, nz)) return fail(ctx, MFE_BAD_ARG, "bad box");
  MFE_TRY(set_device(ctx));
  return launch_zero_boundary(ctx, nx, ny, nz, v);
}

mfe_status mfe_spmm(mfe_ctx* ctx, const mfe_csr* A, int32_t nrhs, const void* X, void* Y)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, A));
  if (nrhs < 1 || (A->nrows > 0 && (!X || !Y))) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  return launch_spmm(ctx, A, nrhs, X, Y);
}

mfe_status mfe_cg_solve_multi(mfe_ctx* ctx, const mfe_csr* A, int32_t nrhs, const double* B,
                              double* X, const mfe_cg_opts* opts, mfe_cg_result* results)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, A));
  if (!opts || !results || (A->nrows > 0 && (!B || !X))) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  if (A->nrows == 0) return fail(ctx, MFE_BAD_ARG, "empty matrix");
  MFE_TRY(set_device(ctx));
  return cg_multi(ctx, A, nrhs, B, X, opts, results);
}

mfe_status mfe_batch_solve_boxes(mfe_ctx* ctx, int32_t nbox, const int32_t* dims,
                                 const mfe_cg_opts* opts, double* x_out, mfe_cg_result* results)
{
  if (!ctx) return MFE_BAD_ARG;
  if (!dims || !opts || !x_out || !results) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  for (int32_t i = 0; i < nbox; ++i)
    if (!box_ok(dims[3 * i], dims[3 * i + 1], dims[3 * i + 2]))
      return fail(ctx, MFE_BAD_ARG, "bad box in the batch");
  MFE_TRY(set_device(ctx));
  return batch_solve_boxes(ctx, nbox, dims, opts, x_out, results);
}

static mfe_status check_ell(mfe_ctx* ctx, const mfe_ell* E, bool need_rows)
{
  if (!E) return fail(ctx, MFE_BAD_ARG, "null matrix");
  if (E->ncols_per_row < 1 || E->ncols_per_row > 1024 || E->nrows < 0 ||
      E->nrows * (int64_t)E->ncols_per_row >= ((int64_t)1 << 31))
    return fail(ctx, MFE_BAD_ARG, "ELL sizes out of range for 32-bit indices");
  if ((need_rows || E->nrows > 0) && (!E->cols || !E->vals)) return fail(ctx, MFE_BAD_ARG, "null ELL array");
  return MFE_OK;
}

mfe_status mfe_csr_to_ell(mfe_ctx* ctx, const mfe_csr* A, mfe_ell* E)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_csr(ctx, A));
  if (!E || E->ncols_per_row < 1 || E->ncols_per_row > 1024 ||
      A->nrows * (int64_t)E->ncols_per_row >= ((int64_t)1 << 31))
    return fail(ctx, MFE_BAD_ARG, "bad ELL target");
  if (A->nrows > 0 && (!E->cols || !E->vals)) return fail(ctx, MFE_BAD_ARG, "null ELL array");
  MFE_TRY(set_device(ctx));
  return launch_csr_to_ell(ctx, A, E);
}

mfe_status mfe_spmv_ell(mfe_ctx* ctx, const mfe_ell* E, const void* x, void* y)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_ell(ctx, E, false));
  if (E->dtype != MFE_F64 && E->dtype != MFE_F32) return fail(ctx, MFE_BAD_ARG, "bad dtype");
  if (E->nrows > 0 && (!x || !y)) return fail(ctx, MFE_BAD_ARG, "null vector");
  MFE_TRY(set_device(ctx));
  if (E->nrows == 0) return MFE_OK;
  return launch_spmv_ell(ctx, E, x, y, nullptr, nullptr, nullptr);
}

mfe_status mfe_cg_solve_ell(mfe_ctx* ctx, const mfe_ell* E, const double* b, double* x,
                            const mfe_cg_opts* opts, mfe_cg_result* result)
{
  if (!ctx || !result) return MFE_BAD_ARG;
  MFE_TRY(check_ell(ctx, E, false));
  if (E->dtype != MFE_F64) return fail(ctx, MFE_BAD_ARG, "cg_solve needs the FP64 matrix");
  MFE_TRY(set_device(ctx));
  if (E->nrows == 0) return MFE_OK;
  mfe_csr V;
  MFE_TRY(ell_view(ctx, E, &V));
  mfe_cg_opts o;
  if (opts) o = *opts;
  else mfe_cg_opts_default(&o);
  if (!cg_opts_valid(o) || o.precision != MFE_PREC_F64 || o.precond != 0)
    return mfe_cg_solve(ctx, &V, b, x, opts, result);  // validates, or the other solvers
  if (!b || !x) return fail(ctx, MFE_BAD_ARG, "null vector");
  // the iterations run on a sliced copy (one coalesced line per entry of 32 rows)
  const int64_t ne = sell_entries(E->nrows, E->ncols_per_row);
  mfe_sell S;
  memset(&S, 0, sizeof(S));
  S.cols = static_cast<int32_t*>(workspace(ctx, "ell.sell.cols", sizeof(int32_t) * (size_t)ne));
  S.vals = static_cast<double*>(workspace(ctx, "ell.sell.vals", sizeof(double) * (size_t)ne));
  if (!S.cols || !S.vals) return fail(ctx, MFE_OOM, "sliced ELL workspace allocation failed");
  MFE_TRY(launch_ell_to_sell(ctx, E, &S));
  memset(result, 0, sizeof(*result));
  const mfe_status st = cg_solve_sell(ctx, &V, &S, b, x, &o, result, E);
  result->status = st;
  return st;
}

static mfe_status check_sell(mfe_ctx* ctx, const mfe_sell* S)
{
  if (!S) return fail(ctx, MFE_BAD_ARG, "null matrix");
  if (S->ncols_per_row < 1 || S->ncols_per_row > 1024 || S->nrows < 0 ||
      sell_entries(S->nrows, S->ncols_per_row) >= ((int64_t)1 << 31))
    return fail(ctx, MFE_BAD_ARG, "sliced ELL sizes out of range for 32-bit indices");
  if (S->nrows > 0 && (!S->cols || !S->vals)) return fail(ctx, MFE_BAD_ARG, "null sliced ELL array");
  return MFE_OK;
}

mfe_status mfe_ell_to_sell(mfe_ctx* ctx, const mfe_ell* E, mfe_sell* S)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_ell(ctx, E, false));
  if (E->dtype != MFE_F64) return fail(ctx, MFE_BAD_ARG, "the sliced ELL copy is FP64");
  if (!S || (E->nrows > 0 && (!S->cols || !S->vals))) return fail(ctx, MFE_BAD_ARG, "null sliced ELL array");
  MFE_TRY(set_device(ctx));
  if (E->nrows == 0) {
    S->nrows = 0;
    S->ncols_per_row = E->ncols_per_row;
    return MFE_OK;
  }
  return launch_ell_to_sell(ctx, E, S);
}

mfe_status mfe_spmv_sell(mfe_ctx* ctx, const mfe_sell* S, const double* x, double* y)
{
  if (!ctx) return MFE_BAD_ARG;
  MFE_TRY(check_sell(ctx, S));
  if (S->nrows > 0 && (!x || !y)) return fail(ctx, MFE_BAD_ARG, "null vector");
  MFE_TRY(set_device(ctx));
  if (S->nrows == 0) return MFE_OK;
  return launch_spmv_sell(ctx, S, x, y, nullptr, nullptr);
}

mfe_status mfe_batch_create(mfe_ctx* ctx, int32_t nbox, const int32_t* dims, mfe_batch** out)
{
  if (!ctx) return MFE_BAD_ARG;
  if (!dims || !out) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  *out = nullptr;
  for (int32_t i = 0; i < nbox; ++i)
    if (!box_ok(dims[3 * i], dims[3 * i + 1], dims[3 * i + 2]))
      return fail(ctx, MFE_BAD_ARG, "bad box in the batch");
  MFE_TRY(set_device(ctx));
  return batch_create(ctx, nbox, dims, out);
}

mfe_status mfe_batch_set_tuning(mfe_ctx* ctx, mfe_batch* batch, const mfe_batch_tuning* t)
{
  if (!ctx) return MFE_BAD_ARG;
  if (!batch || !t) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  return batch_set_tuning(ctx, batch, t);
}

mfe_status mfe_batch_info(const mfe_batch* batch, int64_t* rows, int64_t* nnz,
                          double* assembly_seconds, mfe_batch_tuning* tuning)
{
  if (!batch) return MFE_BAD_ARG;
  batch_info(batch, rows, nnz, assembly_seconds, tuning);
  return MFE_OK;
}

mfe_status mfe_batch_solve(mfe_ctx* ctx, mfe_batch* batch, const mfe_cg_opts* opts,
                           double* x_out, mfe_cg_result* results)
{
  if (!ctx) return MFE_BAD_ARG;
  if (!batch || !opts || !results) return fail(ctx, MFE_BAD_ARG, "bad arguments");
  MFE_TRY(set_device(ctx));
  return batch_solve(ctx, batch, opts, x_out, results);
}

void mfe_batch_destroy(mfe_batch* batch) { batch_destroy(batch); }

}  // extern "C"
