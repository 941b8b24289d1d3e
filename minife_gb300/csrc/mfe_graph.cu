// The solvers' device-side loops: one CUDA graph with a conditional while node.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "mfe_internal.h"

namespace mfe {

namespace {

// a conditional node of `g` after deps; *inner is the graph it runs
cudaError_t add_conditional(cudaGraph_t g, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                            const cudaGraphNode_t* deps, size_t ndeps, cudaGraphNode_t* node, cudaGraph_t* inner)
{
  // cudaGraphNodeParams has no default constructor (it holds a union)
  alignas(cudaGraphNodeParams) unsigned char buf[sizeof(cudaGraphNodeParams)];
  memset(buf, 0, sizeof(buf));
  cudaGraphNodeParams* p = reinterpret_cast<cudaGraphNodeParams*>(buf);
  p->type = cudaGraphNodeTypeConditional;
  p->conditional.handle = h;
  p->conditional.type = type;
  p->conditional.size = 1;
  const cudaError_t e = cudaGraphAddNode(node, g, deps, nullptr, ndeps, p);
  if (e == cudaSuccess) *inner = p->conditional.phGraph_out[0];
  return e;
}

// `launch` captured on s into g after the nodes of deps, which become the
// capture's last nodes
struct Deps {
  cudaGraphNode_t node[4];
  size_t n = 0;
};
template <typename F>
cudaError_t capture(cudaStream_t s, cudaGraph_t g, Deps& deps, mfe_status* st, F&& launch)
{
  cudaError_t e = cudaStreamBeginCaptureToGraph(s, g, deps.n ? deps.node : nullptr, nullptr, deps.n,
                                                cudaStreamCaptureModeRelaxed);
  if (e != cudaSuccess) return e;
  *st = launch();
  cudaStreamCaptureStatus cs;
  const cudaGraphNode_t* last = nullptr;
  size_t n = 0;
  e = cudaStreamGetCaptureInfo(s, &cs, nullptr, nullptr, &last, nullptr, &n);
  if (e == cudaSuccess && (n < 1 || n > 4)) e = cudaErrorUnknown;
  if (e == cudaSuccess) {
    for (size_t i = 0; i < n; ++i) deps.node[i] = last[i];
    deps.n = n;
  }
  cudaGraph_t same;
  const cudaError_t e2 = cudaStreamEndCapture(s, &same);
  return e == cudaSuccess ? e2 : e;
}

}  // namespace

// The iterations that CG takes for a digit of the residual: about a quarter of the
// box's longest side.
int loop_copies(const mfe_cg_opts* o, int side, int most, int worth)
{
  const double digits = o->tol_mode == MFE_TOL_RELATIVE ? -std::log10(std::max(o->tol, 1e-17)) : 16.0;
  const double iterations = std::min<double>(o->max_iter, 0.25 * side * std::max(digits, 0.0));
  if (iterations < worth) return 1;
  const double per_update = 1.0 + 0.25 * side * -0.5 * std::log10(mixed_delta2(o));
  const double between = o->refine_k > 0 ? std::min<double>(o->refine_k, per_update) : per_update;
  int copies = most;
  while (copies > 1 && copies > between) copies /= 2;
  return copies;
}

mfe_status run_graph_loop(mfe_ctx* ctx, const GraphLoop& L, const char* where)
{
  // captured on the context's own stream (the legacy default stream cannot
  // be); launched on ctx->stream
  const cudaStream_t run_stream = ctx->stream, s = ctx->own_stream;
  cudaGraph_t g = nullptr, loop = nullptr, upd = nullptr;
  cudaGraphExec_t ex = nullptr;
  cudaGraphConditionalHandle h = 0, hu = 0;
  cudaGraphNode_t node;
  mfe_status st = MFE_OK;
  ctx->stream = s;
  cudaError_t e = cudaGraphCreate(&g, 0);
  if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
  Deps first;
  if (e == cudaSuccess) e = capture(s, g, first, &st, [&] { return L.begin(h); });
  if (e == cudaSuccess && st == MFE_OK)
    e = add_conditional(g, h, cudaGraphCondTypeWhile, first.node, first.n, &node, &loop);
  Deps deps;
  if (e == cudaSuccess && st == MFE_OK && L.update) e = cudaGraphConditionalHandleCreate(&hu, loop, 0, 0);
  for (int i = 0; i < L.copies && e == cudaSuccess && st == MFE_OK; ++i)
    e = capture(s, loop, deps, &st, [&] { return L.body(h, hu); });
  if (e == cudaSuccess && st == MFE_OK && L.update) {
    e = add_conditional(loop, hu, cudaGraphCondTypeIf, deps.node, deps.n, &node, &upd);
    Deps none;
    if (e == cudaSuccess) e = capture(s, upd, none, &st, [&] { return L.update(h); });
  }
  ctx->stream = run_stream;
  if (e == cudaSuccess && st == MFE_OK) e = cudaGraphInstantiate(&ex, g, 0);
  if (e == cudaSuccess && st == MFE_OK) e = cudaGraphLaunch(ex, ctx->stream);
  if (ex) cudaGraphExecDestroy(ex);
  if (g) cudaGraphDestroy(g);
  if (st != MFE_OK) return st;
  if (e != cudaSuccess) {
    cudaGetLastError();
    return cuda_fail(ctx, e, where);
  }
  return MFE_OK;
}

}  // namespace mfe
