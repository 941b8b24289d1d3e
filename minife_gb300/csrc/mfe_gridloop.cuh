// A solver's iteration loop as one cooperative kernel: barriers and sums over all
// its blocks, the rows that a block keeps, its launch.  Every wait is bounded.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <mutex>
#include <vector>

#include "mfe_common.cuh"
#include "mfe_internal.h"

namespace mfe {

// What the blocks of a loop meet by: how many have arrived at its barriers so far,
// and how long one waits for the others.
struct GridSync {
  unsigned* arrived;
  uint64_t wait_ns;
};

// The calling thread's block arrives at a barrier of all blocks and waits;
// false after the time limit.
__device__ __forceinline__ bool arrive_and_wait(const GridSync& sync, unsigned target)
{
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(sync.arrived) : "memory");
  auto there = [&] {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(sync.arrived) : "memory");
    return (int)(v - target) >= 0;
  };
  if (there()) return true;
  const uint64_t t0 = global_ns();
  for (unsigned i = 1; !there(); ++i)
    if ((i & 255u) == 0 && global_ns() - t0 > sync.wait_ns) return false;
  return true;
}

// All blocks; false (in every thread of the block) after the time limit.
__device__ __forceinline__ bool grid_barrier(const GridSync& sync, unsigned target)
{
  __shared__ bool s_ok;
  __syncthreads();
  if (threadIdx.x == 0) s_ok = arrive_and_wait(sync, target);
  __syncthreads();
  return s_ok;
}

// The sum of v over all threads of all blocks, given to then(total) in thread 0
// of every block before a block barrier.  The FP64 pipe takes one warp's
// addition in 17 clocks, so a reduction by shuffles in every warp would cost
// more than the rest: one warp adds the block's values from shared memory, and
// after the grid barrier the blocks' sums in block order.  s_v: a double per
// thread; beside(): what thread 32 does meanwhile.
template <int NT, typename Then, typename Beside>
__device__ __forceinline__ bool grid_sum(double v, double* s_v, double* slots, const GridSync& sync, unsigned target,
                                         Then&& then, Beside&& beside)
{
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
      ok = arrive_and_wait(sync, target);
    }
    __syncwarp();
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (unsigned i = threadIdx.x, j = 0; i < gridDim.x; i += 32, ++j) t[j & 3] += __ldcg(slots + i);
    const double total = warp_sum((t[0] + t[1]) + (t[2] + t[3]));
    if (threadIdx.x == 0) {
      s_ok = ok;
      then(total);
    }
  } else if (threadIdx.x == 32) {
    beside();
  }
  __syncthreads();
  return s_ok;
}

template <int NT, typename Then>
__device__ __forceinline__ bool grid_sum(double v, double* s_v, double* slots, const GridSync& sync, unsigned target,
                                         Then&& then)
{
  return grid_sum<NT>(v, s_v, slots, sync, target, then, [] {});
}

// A block's share of the vectors: a range that begins at a multiple of A (a
// power of two).
template <int A>
__device__ __forceinline__ int64_t share(int64_t n, unsigned b, unsigned nb)
{
  return b == nb ? n : (n * b / nb) & ~(int64_t)(A - 1);
}

// A loop's state back to memory, but for its error word: another block may have set
// that after its last wait.
template <typename State>
__device__ __forceinline__ void store_state(State* to, const State& from)
{
  static_assert(sizeof(State) % sizeof(unsigned) == 0, "words");
  const unsigned* f = reinterpret_cast<const unsigned*>(&from);
  unsigned* t = reinterpret_cast<unsigned*>(to);
  for (size_t i = 0; i < sizeof(State) / sizeof(unsigned); ++i)
    if (i != offsetof(State, err) / sizeof(unsigned)) t[i] = f[i];
}

// Shared memory for a block's static part and the system's, out of 227 KB per
// block and 228 KB per SM.
constexpr size_t kReserved = 8 * 1024, kRoom = 227 * 1024 - kReserved;

// Blocks of at least `rows` entries, one per SM, on half of the SMs up to `half`
// entries: there the shares cost nothing, and two loops run side by side.
inline int loop_blocks(const mfe_ctx* ctx, int64_t n, int rows, int64_t half)
{
  return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, (int64_t)rows),
                                                     n <= half ? (ctx->sm_count + 1) / 2 : ctx->sm_count));
}

// How many of its vectors (n elements of elem bytes over g blocks) a block can
// hold in `room` bytes, at most `most`; the bytes they take.
inline size_t plan_held(int64_t n, int g, size_t elem, size_t room, int most, int* span, int* held)
{
  *span = (int)((ceil_div(n, (int64_t)g) + 7) & ~(int64_t)3);
  *held = (int)std::min<size_t>(room / (elem * *span), most);
  return elem * *span * *held;
}

// The loop's count of arrivals set to zero on the stream.  A pending
// mfe_inject_loop_fault sets it one short instead, so that no block ever sees all
// of them arrive and each gives up after the injected time.
inline mfe_status start_sync(mfe_ctx* ctx, unsigned* arrived, GridSync* sync)
{
  const bool fault = ctx->inject_loop_ns > 0;
  sync->arrived = arrived;
  sync->wait_ns = fault ? (uint64_t)ctx->inject_loop_ns : kWaitLimitNs;
  MFE_CUDA_TRY(ctx, cudaMemsetAsync(arrived, fault ? 0xff : 0, sizeof(unsigned), ctx->stream));
  if (fault) ctx->inject_loop_ns = -1;
  return MFE_OK;
}

// A loop's blocks wait for one another, so two loops must never each hold a part
// of the device that the other needs.  A block may fill an SM, so loops (of any
// context and stream) run side by side while they have no more blocks together than
// the device has SMs: then a block that has not started always finds an SM without
// any.  A launch waits on the device for the oldest of the running ones until that
// holds.  (Whatever else runs on an SM ends by itself.)
// Measured, us per solve with 1, 2, 4 and 8 threads solving (1e-9): FP64 stencil 8^3
// 340, 180, 92, 74 (one loop after another 345, 181, 176, 171; as graphs 610, 333,
// 181, 156); 16^3 519, 292, 225, 189 (515, 373, 374, 371; 1040, 563, 295, 263); mixed
// 24^3 939, 505, 392, 366 (982, 736, 690, 677; 1451, 1369, 1080, 910).  Loops that fill
// the device go one after another: 30^3 916, 848, 784, 772, where graphs take 2303,
// 1154, 621, 555 (with more than two threads the graphs' gaps fill up; 24^3 to 52^3
// are so); 64^3 3641, 3579, 3513, 3533 (7519, 5110, 4011, 3990).
struct LoopOrder {
  struct Loop {
    cudaEvent_t end;
    int blocks;
  };
  std::mutex mu;
  std::vector<Loop> running;  // in the order of their launches
  std::vector<cudaEvent_t> spare;
};
inline LoopOrder& loop_order(int device)
{
  static LoopOrder order[64];
  return order[device & 63];
}

// launch() on ctx->stream beside the loops that run, as blocks allow
template <typename Launch>
mfe_status launch_in_order(mfe_ctx* ctx, int blocks, Launch&& launch)
{
  // a capture launches nothing (and the solve's first read of its state ends it)
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  MFE_CUDA_TRY(ctx, cudaStreamIsCapturing(ctx->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) return launch();
  blocks = std::min(blocks, ctx->sm_count);
  LoopOrder& order = loop_order(ctx->device);
  std::lock_guard<std::mutex> lock(order.mu);
  // (asking for an event must not end a capture that another thread has begun)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  MFE_CUDA_TRY(ctx, cudaThreadExchangeStreamCaptureMode(&mode));
  int held = 0;
  for (size_t i = 0; i < order.running.size();) {
    if (cudaEventQuery(order.running[i].end) == cudaSuccess) {
      order.spare.push_back(order.running[i].end);
      order.running.erase(order.running.begin() + i);
    } else {
      held += order.running[i++].blocks;
    }
  }
  cudaGetLastError();  // (cudaErrorNotReady)
  cudaError_t e = cudaSuccess;
  cudaEvent_t end = nullptr;
  if (order.spare.empty()) {
    e = cudaEventCreateWithFlags(&end, cudaEventDisableTiming);
  } else {
    end = order.spare.back();
    order.spare.pop_back();
  }
  const cudaError_t e2 = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e == cudaSuccess) e = e2;
  for (size_t i = 0; e == cudaSuccess && i < order.running.size() && held + blocks > ctx->sm_count; ++i) {
    e = cudaStreamWaitEvent(ctx->stream, order.running[i].end, 0);
    held -= order.running[i].blocks;
  }
  mfe_status st = e == cudaSuccess ? launch() : cuda_fail(ctx, e, "the order of the solvers' loops");
  if (st == MFE_OK) {
    e = cudaEventRecord(end, ctx->stream);
    if (e != cudaSuccess) {
      cudaStreamSynchronize(ctx->stream);  // nothing may start beside it unseen
      st = cuda_fail(ctx, e, "the order of the solvers' loops");
    }
  }
  if (st == MFE_OK) order.running.push_back({end, blocks});
  else if (end) order.spare.push_back(end);
  return st;
}

// The attribute set and the occupancy asked for, once per kernel and device; a
// launch of blocks that would not all be resident is refused (MFE_NOT_SUPPORTED:
// fewer blocks fit an SM, or fewer SMs are there for this process than the device
// has).
template <size_t kMost>
inline mfe_status coop_launch(mfe_ctx* ctx, const void* kern, int g, int threads, int per_sm, size_t smem,
                       std::atomic<int>* ready, void** args)
{
  if (ctx->inject_loop_ns == 0) {
    ctx->inject_loop_ns = -1;
    return fail(ctx, MFE_NOT_SUPPORTED, "a solver's loop kernel was refused (injected)");
  }
  std::atomic<int>& have = ready[ctx->device & 63];
  if (have.load(std::memory_order_acquire) == 0) {
    int blocks = 0;
    MFE_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
    MFE_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, threads, kMost));
    if (blocks < per_sm) return fail(ctx, MFE_NOT_SUPPORTED, "a solver's loop kernel does not fit the device");
    have.store(blocks, std::memory_order_release);
  }
  return launch_in_order(ctx, g, [&]() -> mfe_status {
    const cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(g), dim3(threads), args, smem, ctx->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
      cudaGetLastError();
      return fail(ctx, MFE_NOT_SUPPORTED, "a solver's loop kernel does not fit the device");
    }
    MFE_CUDA_TRY(ctx, e);
    return MFE_OK;
  });
}

}  // namespace mfe
