// CSR matrix-vector products on sm_103a.
//
// GB300 has a reduced FP64 pipe (about 2 FP64 FMA per clock per SM), which
// puts an FP64 CSR SpMV close to the FP64 issue limit as well as the HBM
// limit.  The main kernel (k_spmv_any) therefore sums a row in one lane or two
// (no shuffle-add trees, which would cost 5 extra FP64 adds per lane), while the
// values and column indices of 32 rows arrive in a warp's own shared memory by
// two 1-D bulk async copies (TMA, cp.async.bulk) tracked by an mbarrier, so the
// HBM reads stay fully coalesced; x is gathered through the read-only path
// (27-point rows touch three x-planes, which stay L1/L2 resident).  The
// reference's row-major ELLMatrix has its own kernel of this kind, whose groups
// start aligned.
// Epilogues: plain y = A x; y = A x with x.y (matvec_and_dot); and the CG
// residual r = b - A x with r.r.  Dots accumulate in FP64 and reduce
// deterministically (fixed grid, last block sums the block partials in order).
// Matrices whose rows are stated to be longer than 32 entries, or are on
// average, use a warp-per-row kernel.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "mfe_cgstate.cuh"
#include "mfe_common.cuh"
#include "mfe_internal.h"

namespace mfe {

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

enum SpmvMode { SPMV_PLAIN = 0, SPMV_DOT = 1, SPMV_RESID = 2 };

template <typename T>
struct SpmvParams {
  int64_t n;
  int64_t nnz;
  const int32_t* __restrict__ ro;
  const int32_t* __restrict__ cols;
  const T* __restrict__ vals;
  const T* __restrict__ x;
  T* __restrict__ y;
  const double* __restrict__ b;  // SPMV_RESID: y = b - A x
  double* partials;
  unsigned* ticket;
  double* dot_out;  // used when cg == nullptr
  CgState* cg;      // CG bookkeeping in the last block (nullable)
  unsigned* err;
  // fault injection (mfe_inject_wait_timeout), warp-staged kernels: nonzero =
  // no copy is issued and the bounded waits give up after this many ns
  uint64_t withhold_ns;
};

// Row sum with one FMA per nonzero.  Rows of up to LMAX entries run the same
// fully unrolled, predicated code (no divergence between the 27-entry
// interior rows and the 8/12/18-entry boundary rows of a warp), and two
// interleaved partial sums (even / odd entries) halve the dependent-FMA
// chain, which the FP64 pipe's long latency otherwise exposes; one extra add
// joins them.  Longer rows continue in a plain loop.
//
// All LMAX column/value/x loads are issued unconditionally before the first
// FMA (indices past the row end are clamped to its last entry, so every load
// stays inside the row), letting the 27 x-gathers overlap; the FMAs past the
// row end are discarded by a select, so the sum is exactly that of the row's
// own entries.
// Read-only-path gathers written as volatile asm: the compiler treats
// __ldg results as rematerialisable and sinks each gather next to its FMA,
// which serialises the gathers' latency; volatile loads stay where they are
// issued, so all of a row's gathers are in flight together.
__device__ __forceinline__ double ld_gather(const double* p)
{
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_gather(const float* p)
{
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

template <typename T, int LMAX>
__device__ __forceinline__ T row_dot(const T* __restrict__ rv, const int32_t* __restrict__ rc,
                                     int len, const T* __restrict__ x)
{
  if (len <= 0) return T(0);
  int32_t c[LMAX];
  T xv[LMAX], v[LMAX];
#pragma unroll
  for (int k = 0; k < LMAX; ++k) c[k] = rc[min(k, len - 1)];
#pragma unroll
  for (int k = 0; k < LMAX; ++k) xv[k] = ld_gather(&x[c[k]]);
#pragma unroll
  for (int k = 0; k < LMAX; ++k) v[k] = rv[min(k, len - 1)];
  T s0 = T(0), s1 = T(0);
#pragma unroll
  for (int k = 0; k < LMAX; k += 2) {
    const T t0 = fma(v[k], xv[k], s0);
    s0 = (k < len) ? t0 : s0;
    if (k + 1 < LMAX) {
      const T t1 = fma(v[k + 1], xv[k + 1], s1);
      s1 = (k + 1 < len) ? t1 : s1;
    }
  }
  for (int k = LMAX; k < len; ++k) s0 = fma(rv[k], __ldg(&x[rc[k]]), s0);
  return s0 + s1;
}

template <int MODE>
__device__ __forceinline__ void spmv_epilogue(double total, CgState* cg, double* dot_out)
{
  if (cg == nullptr) {
    if (MODE != SPMV_PLAIN) *dot_out = total;
    return;
  }
  if (MODE == SPMV_DOT) {
    // cg_solve.hpp:179-200: p.Ap and the breakdown pre-test
    cg->pAp = total;
    if (total < cg->brkdown_tol) cg->check_pending = 1;
  } else if (MODE == SPMV_RESID) {
    // cg_solve.hpp:124-144: r = b - A x, rtrans, normr, loop condition
    cg_resid_init(cg, total);
  }
}

// Warp-staged products: a warp per group of 32 rows, whose nonzeros are
// contiguous in both layouts below (CSR: ro[32g] .. ro[32g+32]; the
// reference's ELLMatrix: 32 g K .. 32 (g+1) K, short rows padded).  Lane 0
// stages a group's values and columns with two 1-D bulk copies (TMA) into the
// warp's own shared memory, with its own mbarrier (no block barrier in the
// loop), and every lane sums rows from there.  The 256^3 FP64 CSR product took
// 1.14 ms this way, two stages per warp, against 2.09 ms with 128-row tiles
// behind block barriers.
constexpr int kStgWarps = 2;    // warps per block
constexpr int kStgMaxLen = 32;  // longer rows: the warp-per-row kernel

// Stage capacity (elements) for a group of 32 rows of at most max_len
// entries: ELL groups start aligned and hold exactly 32 K; CSR groups carry
// up to 3 elements of alignment slack at each end.  A multiple of 4, so the
// column part of a stage starts 16-byte aligned.
__host__ __device__ constexpr int stg_cap(int max_len, bool ell)
{
  return ell ? 32 * max_len : ((32 * max_len + 8) + 3) & ~3;
}

// CSR rows.  A stage starts on the 16-byte boundaries at or below its
// group's first nonzero, and the ragged end of the arrays arrives by plain
// loads.  The stage is one per warp, of `cap` entries (the host's guess from the
// mean row length): twenty-four warps per SM, a part of them computing while the
// others' next groups arrive.  A group that does not fit the stage, or holds a row
// over kAnyLongest, is taken in parts of 16, 8, ... 1 rows with 2, 4, ... 32 lanes
// a row, through the stage as long as a part fits it, so the longest row need not
// be known.  `most`: what kCheckRows rows may take up when it is stated (INT_MAX
// else); more is an error in the caller's max_row_len, and recorded.
//
// What bounds it in FP64: the FP64 pipe, whose instructions take 17 clocks an SM whatever
// the number of lanes at work.  Hence the rows in pairs (row_pair): 1.48 M rows
// of 4 to 27 entries, 15.5 on average, take 18 FMAs a group instead of 27.
// Measured there, us per call: a pass for the longest row, two stages and 27
// FMAs 121; without the pass 107; in pairs 103; one stage, 16 / 20 / 24 warps per
// SM 86 / 79 / 76 (50 are the bytes at the HBM rate).  Rows of 27 entries (no
// pairs): 135 / 110; of 5: 126 / 69; of 20 to 40: 700 / 141.  Cutting a
// group's entries into 32 equal runs, a lane per run, took twice the
// instructions, 147 us.  FP32 rows (no pairs) against 128-row tiles behind block
// barriers, 1.48 M rows of 27 / of 4 to 27: longest row stated 68, 65 before and
// 63, 60 now; not stated (a pass for it before) 94, 90 and 63, 59.
// Rows whose lengths come in regions (half of them 4 to 7, half 27 to 32, so that
// every group of the second half is larger than the stage), FP64 / FP32: with the
// longest row known and a stage for it 133 / 73; such groups a row at a time over
// the warp 342 / 371; in parts 97 / 72.  Rows of 8 and 56 in turn 737 / 262 (a warp
// per row), 714 / 663 (a row at a time), 235 / 125; one row of 200 among 31 of 10 930
// / 465, 585 / 653, 241 / 97.  One row of 200,000 among rows of 20 takes 2990 / 1706
// (a warp per row), 1030 / 560.
constexpr int kAnyLongest = 54;
constexpr int kAnyWarps = 24;  // per SM, in blocks of W

// rows whose entries together are held against a stated longest row, and what they
// may take up with the rounding to 16 bytes
template <typename T>
constexpr int kCheckRows = sizeof(T) == 8 ? 32 : 128;
constexpr int stated_most(int rows, int max_len) { return (rows * max_len + 8 + 3) & ~3; }

// A group's 32 rows shared out in pairs: the lanes ranked by row length, the
// r-th shortest row's lane also takes the end of the r-th longest, so that both
// have half of the two rows' entries.  At most kPairSteps entries per lane.
constexpr int kPairSteps = 18;
struct RowPair {
  int other;   // the other row's lane
  int own;     // entries of the lane's own row that it takes
  int extra;   // and of the other's, from its entry `from` on
  int from;
};
__device__ __forceinline__ RowPair row_pair(int st, int en, uint8_t* lane_of_rank)
{
  const int lane = threadIdx.x & 31, len = en - st;
  unsigned same = 0xffffffffu;
  int rank = 0;
#pragma unroll
  for (int b = 5; b >= 0; --b) {  // len <= kAnyLongest < 64
    const bool one = (len >> b) & 1;
    const unsigned ones = __ballot_sync(0xffffffffu, one);
    if (one) rank += __popc(same & ~ones);
    same &= one ? ones : ~ones;
  }
  rank += __popc(same & ((1u << lane) - 1u));
  lane_of_rank[rank] = (uint8_t)lane;
  __syncwarp();
  RowPair q;
  q.other = lane_of_rank[31 - rank];
  const int olen = __shfl_sync(0xffffffffu, len, q.other), oen = __shfl_sync(0xffffffffu, en, q.other);
  const int give = (abs(len - olen)) / 2;
  q.own = len > olen ? len - give : len;
  q.extra = len < olen ? give : 0;
  q.from = oen - give;
  return q;
}

// the lane's row times x; gv, gc: the group's staged values and columns
__device__ __forceinline__ double pair_dot(const RowPair& q, int st, const double* gv, const int32_t* gc,
                                           const double* __restrict__ x)
{
  const int cnt = q.own + q.extra, jump = q.from - st - q.own;
  double s = 0.0, mine = 0.0;
#pragma unroll
  for (int k0 = 0; k0 < kPairSteps; k0 += kPairSteps / 2) {
    double v[kPairSteps / 2], xv[kPairSteps / 2];
#pragma unroll
    for (int k = 0; k < kPairSteps / 2; ++k) {
      const int i = min(k0 + k, max(cnt - 1, 0)), at = st + i + (i < q.own ? 0 : jump);
      xv[k] = cnt > 0 ? ld_gather(&x[gc[at]]) : 0.0;
      v[k] = gv[at];
    }
#pragma unroll
    for (int k = 0; k < kPairSteps / 2; ++k) {
      if (k0 + k == q.own) {
        mine = s;
        s = 0.0;
      }
      const double t = fma(v[k], xv[k], s);
      s = k0 + k < cnt ? t : s;
    }
  }
  if (q.own == kPairSteps) {
    mine = s;
    s = 0.0;
  }
  const double help = __shfl_sync(0xffffffffu, s, q.other);
  return mine + help;
}

// entries k, k + L, ... below end of a row times x; gv, gc: the values and columns;
// any: an entry of the warp's rows (loaded in place of one past a row's end)
template <typename T>
__device__ __forceinline__ T strided_dot(const T* gv, const int32_t* gc, int k, int end, int L, int any,
                                         const T* __restrict__ x)
{
  // gathers in flight (nine: rows of 8 and 56 in turn 254 us, and the registers cost the
  // other groups 0.7 %)
  constexpr int kBatch = 4;
  T s = T(0);
  for (; __any_sync(0xffffffffu, k < end); k += kBatch * L) {
    T v[kBatch], xv[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int at = k + i * L < end ? k + i * L : any;
      xv[i] = ld_gather(&x[gc[at]]);
      v[i] = gv[at];
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const T t = fma(v[i], xv[i], s);
      s = k + i * L < end ? t : s;
    }
  }
  return s;
}

template <typename T, int MODE, int W>
__global__ void __launch_bounds__(W * 32, kAnyWarps / W) k_spmv_any(SpmvParams<T> P, int cap, int most)
{
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar[W];
  __shared__ uint8_t lanes[W][32];
  __shared__ double red[32];
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  constexpr int VA = 16 / sizeof(T);
  const size_t vbytes = (size_t)cap * sizeof(T);
  unsigned char* const stage = smem + (size_t)w * (vbytes + (size_t)cap * sizeof(int32_t));
  T* const dv = reinterpret_cast<T*>(stage);
  int32_t* const dc = reinterpret_cast<int32_t*>(stage + vbytes);
  const int64_t ngroups = (P.n + 31) / 32;
  const int64_t nw = (int64_t)gridDim.x * W;
  const int64_t g0 = (int64_t)blockIdx.x * W + w;
  if (lane == 0) {
    mbar_init(&bar[w], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // up to 3 elements of slack at each end of a group (16-byte boundaries)
  auto staged = [&](int64_t a, int64_t e) { return e - a + 8 <= cap; };
  // the ends of [a, e) on 16-byte boundaries, within the arrays
  auto last = [&](int64_t from, int64_t e, int v) {
    return max(from, min((e + v - 1) & ~(int64_t)(v - 1), P.nnz & ~(int64_t)(v - 1)));
  };
  // lane 0, when the longest row is stated: do the kCheckRows<T> rows around group
  // g, nonzeros [a, e), keep to it?
  auto check = [&](int64_t g, int64_t a, int64_t e) {
    if constexpr (kCheckRows<T> != 32) {
      const int64_t r0 = g * 32 / kCheckRows<T> * kCheckRows<T>;
      a = __ldg(&P.ro[r0]);
      e = __ldg(&P.ro[min(P.n, r0 + kCheckRows<T>)]);
    }
    const int64_t av = a & ~(int64_t)(VA - 1), ac = a & ~(int64_t)3;
    if (max(last(av, e, VA), e) - av > most || max(last(ac, e, 4), e) - ac > most)
      atomicOr(P.err, ERR_TILE_OVERFLOW);
  };
  // lane 0: nonzeros [a, e) of one group into the stage
  auto issue = [&](int64_t a, int64_t e) {
    if (!staged(a, e)) {
      mbar_arrive_expect_tx(&bar[w], 0);
      return;
    }
    const int64_t av = a & ~(int64_t)(VA - 1), ac = a & ~(int64_t)3, bv = last(av, e, VA), bc = last(ac, e, 4);
    // ragged tail past the last 16-byte boundary of the arrays: plain loads
    for (int64_t k = bv; k < e; ++k) dv[k - av] = P.vals[k];
    for (int64_t k = bc; k < e; ++k) dc[k - ac] = P.cols[k];
    fence_proxy_async_smem();
    const unsigned bytes_v = (unsigned)((bv - av) * sizeof(T));
    const unsigned bytes_c = (unsigned)((bc - ac) * sizeof(int32_t));
    mbar_arrive_expect_tx(&bar[w], bytes_v + bytes_c);
    if (bytes_v) bulk_g2s(dv, P.vals + av, bytes_v, &bar[w]);
    if (bytes_c) bulk_g2s(dc, P.cols + ac, bytes_c, &bar[w]);
  };
  auto bounds = [&](int64_t g, int64_t& a, int64_t& e) {
    a = __ldg(&P.ro[g * 32]);
    e = __ldg(&P.ro[min(P.n, g * 32 + 32)]);
  };

  if (lane == 0 && P.withhold_ns == 0 && g0 < ngroups) {
    int64_t a, e;
    bounds(g0, a, e);
    issue(a, e);
  }
  const uint64_t wait_ns = P.withhold_ns ? P.withhold_ns : kWaitLimitNs;
  double dacc = 0.0;
  bool ok = true;
  unsigned phase = 0;  // copies that have landed
  auto landed = [&] {
    const bool there = __all_sync(0xffffffffu, mbar_wait_bounded(&bar[w], phase & 1u, wait_ns));
    if (there) ++phase;
    return there;
  };
  for (int64_t g = g0; g < ngroups; g += nw) {
    const int64_t r = g * 32 + lane;
    const int64_t gn = g + nw;  // the group the stage takes next
    int64_t a, e, na = 0, ne = 0;
    bounds(g, a, e);
    const int m = (int)(e - a);
    int st = m, en = m;  // the lane's row, from a
    if (r < P.n) {
      st = (int)(__ldg(&P.ro[r]) - a);
      en = (int)(__ldg(&P.ro[r + 1]) - a);
    }
    if (lane == 0) {
      if (most != INT_MAX) check(g, a, e);
      if (gn < ngroups) bounds(gn, na, ne);
    }
    ok = landed();
    if (!ok) break;
    T sum = T(0);
    const bool whole = staged(a, e);
    const int longest = __reduce_max_sync(0xffffffffu, en - st);
    if (__builtin_expect(whole && longest <= kAnyLongest, 1)) {
      const T* gv = dv + (a & (VA - 1));
      const int32_t* gc = dc + (a & 3);
      if constexpr (sizeof(T) == 8) {
        const RowPair q = row_pair(st, en, lanes[w]);
        if (__reduce_max_sync(0xffffffffu, q.own + q.extra) <= kPairSteps) sum = pair_dot(q, st, gv, gc, P.x);
        else sum = row_dot<T, 27>(gv + st, gc + st, en - st, P.x);
      } else {
        sum = row_dot<T, 27>(gv + st, gc + st, en - st, P.x);
      }
    } else {
      // R rows at a time, L lanes a row: as few lanes as leave 27 entries to each
      // and let the R rows fit the stage
      int L = 2;
      for (; L < 32; L *= 2) {
        const int R = 32 / L;
        const int lo = __shfl_sync(0xffffffffu, st, lane & ~(R - 1)), hi = __shfl_sync(0xffffffffu, en, lane | (R - 1));
        if (__all_sync(0xffffffffu, en - st <= 27 * L && (whole || staged(lo, hi)))) break;
      }
      const int R = 32 / L;
      for (int j = 0; j < L; ++j) {
        const int lo = __shfl_sync(0xffffffffu, st, j * R), hi = __shfl_sync(0xffffffffu, en, j * R + R - 1);
        const int of = j * R + lane / L;
        const int rs = __shfl_sync(0xffffffffu, st, of) + (lane & (L - 1)), re = __shfl_sync(0xffffffffu, en, of);
        T v;
        if (whole) {
          v = strided_dot(dv + (a & (VA - 1)), dc + (a & 3), rs, re, L, lo, P.x);
        } else if (staged(lo, hi)) {
          __syncwarp();  // every lane is done reading the stage
          if (lane == 0) issue(a + lo, a + hi);
          ok = landed();
          if (!ok) break;
          v = strided_dot(dv + ((a + lo) & (VA - 1)) - lo, dc + ((a + lo) & 3) - lo, rs, re, L, lo, P.x);
        } else {
          // one row, longer than the stage
          v = T(0);
          for (int k = rs; k < re; k += 32) v = fma(P.vals[a + k], __ldg(&P.x[P.cols[a + k]]), v);
        }
        for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const T mine = __shfl_sync(0xffffffffu, v, (lane & (R - 1)) * L);
        if (lane / R == j) sum = mine;
      }
      if (!ok) break;
    }
    if (r < P.n) {
      if (MODE == SPMV_RESID) {
        const double rr = P.b[r] - (double)sum;
        P.y[r] = (T)rr;
        dacc = fma(rr, rr, dacc);
      } else {
        P.y[r] = sum;
        if (MODE == SPMV_DOT) dacc = fma((double)sum, (double)__ldg(&P.x[r]), dacc);
      }
    }
    __syncwarp();  // every lane is done reading the stage
    if (lane == 0 && gn < ngroups) issue(na, ne);
  }
  if (!ok) {
    if (lane == 0) {
      atomicOr(P.err, ERR_WAIT_TIMEOUT);
      // drain: give the copy a bounded chance to land before the block exits (an
      // injected fault issued none)
      if (P.withhold_ns == 0) mbar_wait_bounded(&bar[w], phase & 1u);
    }
    __syncwarp();
  }
  // every warp reaches the block reduction, also after a timeout
  if (MODE != SPMV_PLAIN) {
    const double bt = block_sum(dacc, red);
    double total;
    if (grid_reduce_last(bt, P.partials, P.ticket, red, &total) && threadIdx.x == 0)
      spmv_epilogue<MODE>(total, P.cg, P.dot_out);
  }
}

// The reference's row-major ELL, K entries per row (K <= kStgMaxLen): group
// g's entries start at 32 g K, 16-byte aligned in both arrays, and row lane
// sits at lane K of its stage.  The stage size is computed from K here (not
// read from the parameter block), which lets the compiler fold each lane's
// stage addresses and keep a row's loads in flight together: 1.04 ms for the
// 256^3 product against 1.13 ms with the size read from P.  MODE: plain or
// the CG's initial residual.
// FP32 rows also name the five blocks per SM in the launch bounds (122
// registers: 0.579 against 0.595 ms at 256^3); FP64 rows name none (96
// registers; five blocks: 104 registers and 1.058 against 1.040 ms)
template <typename T>
constexpr int ell_min_blocks()
{
  return sizeof(T) == 4 ? 5 : 0;
}

// NS: stages per warp.  FP64 rows in numbers take one, which lets twice as many
// warps share an SM (ten blocks of two at K = 27): 1.48 M rows 99.7 / 93.8 us,
// 3.44 M 215 / 189, 8.12 M 515 / 428; 0.75 M 54.3 / 54.2, 0.53 M 41.7 / 43.4.
// FP32 rows two (1.48 M 52.3 / 62.9).  (One stage and seven to ten blocks per SM
// in the launch bounds, 64 registers for 56: 1.48 M 99.6-102.8.)
constexpr int64_t kEllOneStage = 1000000;

template <typename T, int MODE, int NS>
__global__ void __launch_bounds__(kStgWarps * 32, ell_min_blocks<T>()) k_spmv_ell(SpmvParams<T> P, int K)
{
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar[kStgWarps][NS];
  __shared__ double red[32];
  constexpr int VA = 16 / sizeof(T);
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  const size_t sbytes = (size_t)32 * K * (sizeof(T) + sizeof(int32_t));
  const size_t vbytes = (size_t)32 * K * sizeof(T);
  unsigned char* wbase = smem + (size_t)w * NS * sbytes;
  const int64_t ngroups = (P.n + 31) / 32;
  const int64_t nw = (int64_t)gridDim.x * kStgWarps;
  const int64_t g0 = (int64_t)blockIdx.x * kStgWarps + w;
  if (lane == 0) {
    for (int s = 0; s < NS; ++s) mbar_init(&bar[w][s], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // lane 0: group g into stage s; the ragged end past the last 16-byte
  // boundary of the matrix (last group only) by plain loads
  auto issue = [&](int64_t g, int s) {
    const int64_t a = g * 32 * K;
    const int64_t e = min(P.n, g * 32 + 32) * K;
    const int64_t bv = max(a, e & ~(int64_t)(VA - 1));
    const int64_t bc = max(a, e & ~(int64_t)3);
    T* dv = reinterpret_cast<T*>(wbase + (size_t)s * sbytes);
    int32_t* dc = reinterpret_cast<int32_t*>(wbase + (size_t)s * sbytes + vbytes);
    for (int64_t k = bv; k < e; ++k) dv[k - a] = P.vals[k];
    for (int64_t k = bc; k < e; ++k) dc[k - a] = P.cols[k];
    fence_proxy_async_smem();
    const unsigned bytes_v = (unsigned)((bv - a) * sizeof(T));
    const unsigned bytes_c = (unsigned)((bc - a) * sizeof(int32_t));
    mbar_arrive_expect_tx(&bar[w][s], bytes_v + bytes_c);
    if (bytes_v) bulk_g2s(dv, P.vals + a, bytes_v, &bar[w][s]);
    if (bytes_c) bulk_g2s(dc, P.cols + a, bytes_c, &bar[w][s]);
  };
  if (lane == 0 && P.withhold_ns == 0)
    for (int s = 0; s < NS; ++s) {
      const int64_t g = g0 + (int64_t)s * nw;
      if (g < ngroups) issue(g, s);
    }
  const uint64_t wait_ns = P.withhold_ns ? P.withhold_ns : kWaitLimitNs;
  double dacc = 0.0;
  bool ok = true;
  int it = 0;
  for (int64_t g = g0; g < ngroups; g += nw, ++it) {
    const int s = it % NS;
    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bar[w][s], (unsigned)((it / NS) & 1), wait_ns));
    if (!ok) break;
    const int64_t r = g * 32 + lane;
    if (r < P.n) {
      const T* rv = reinterpret_cast<const T*>(wbase + (size_t)s * sbytes) + (size_t)lane * K;
      const int32_t* rc =
          reinterpret_cast<const int32_t*>(wbase + (size_t)s * sbytes + vbytes) + (size_t)lane * K;
      const T sum = row_dot<T, 27>(rv, rc, K, P.x);
      if (MODE == SPMV_RESID) {
        const double rr = P.b[r] - (double)sum;
        P.y[r] = (T)rr;
        dacc = fma(rr, rr, dacc);
      } else {
        P.y[r] = sum;
      }
    }
    __syncwarp();  // every lane is done reading stage s
    const int64_t gn = g + (int64_t)NS * nw;
    if (lane == 0 && gn < ngroups) issue(gn, s);
  }
  if (!ok) {
    if (lane == 0) {
      atomicOr(P.err, ERR_WAIT_TIMEOUT);
      for (int j = it; j < it + NS; ++j)
        if (P.withhold_ns == 0 && g0 + (int64_t)j * nw < ngroups)
          mbar_wait_bounded(&bar[w][j % NS], (unsigned)((j / NS) & 1));
    }
    __syncwarp();
  }
  if (MODE == SPMV_RESID) {
    const double bt = block_sum(dacc, red);
    double total;
    if (grid_reduce_last(bt, P.partials, P.ticket, red, &total) && threadIdx.x == 0)
      spmv_epilogue<MODE>(total, P.cg, P.dot_out);
  }
}

// Warp-per-row fallback for long rows (shuffle-reduced).
template <typename T, int MODE>
__global__ void __launch_bounds__(256) k_spmv_warp(SpmvParams<T> P)
{
  __shared__ double red[32];
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  double dacc = 0.0;
  for (int64_t r = warp; r < P.n; r += nwarps) {
    const int32_t a = P.ro[r], e = P.ro[r + 1];
    T sum = T(0);
    for (int32_t k = a + lane; k < e; k += 32) sum = fma(P.vals[k], __ldg(&P.x[P.cols[k]]), sum);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) {
      if (MODE == SPMV_RESID) {
        const double rr = P.b[r] - (double)sum;
        P.y[r] = (T)rr;
        dacc = fma(rr, rr, dacc);
      } else {
        P.y[r] = sum;
        if (MODE == SPMV_DOT) dacc = fma((double)sum, (double)P.x[r], dacc);
      }
    }
  }
  if (MODE != SPMV_PLAIN) {
    const double bt = block_sum(dacc, red);
    double total;
    if (grid_reduce_last(bt, P.partials, P.ticket, red, &total) && threadIdx.x == 0)
      spmv_epilogue<MODE>(total, P.cg, P.dot_out);
  }
}

__global__ void k_max_row_len(int64_t n, const int32_t* __restrict__ ro, int* out)
{
  int m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, ro[i + 1] - ro[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// ---------------------------------------------------------------------------
// multi-RHS: Y = A X, X and Y row-major with nrhs columns; one thread per
// (row, rhs) pair walks the row, so A is read once per product through L1.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    k_spmm(int64_t n, int nrhs, const int32_t* __restrict__ ro, const int32_t* __restrict__ cols,
           const T* __restrict__ vals, const T* __restrict__ X, T* __restrict__ Y)
{
  const int64_t total = n * nrhs;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / nrhs;
    const int j = (int)(t - r * nrhs);
    const int32_t a = ro[r], e = ro[r + 1];
    T sum = T(0);
    for (int32_t k = a; k < e; ++k) sum = fma(vals[k], __ldg(&X[(int64_t)cols[k] * nrhs + j]), sum);
    Y[t] = sum;
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// ---- warp-staged kernels ----
mfe_status take_wait_injection(mfe_ctx* ctx, uint64_t* withhold_ns)
{
  *withhold_ns = 0;
  if (!ctx->inject_wait_ns) return MFE_OK;
  // one-shot, and only for a launch that runs now (not one being captured
  // into a graph, which would replay it)
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  MFE_CUDA_TRY(ctx, cudaStreamIsCapturing(ctx->stream, &cs));
  if (cs == cudaStreamCaptureStatusNone) {
    *withhold_ns = ctx->inject_wait_ns;
    ctx->inject_wait_ns = 0;
  }
  return MFE_OK;
}

template <typename T, int NS>
static size_t ell_smem(int K)
{
  return (size_t)kStgWarps * NS * stg_cap(K, true) * (sizeof(T) + sizeof(int32_t));
}

template <typename T, int NS>
static int ell_grid(mfe_ctx* ctx, int64_t nrows, int K)
{
  const size_t smem = ell_smem<T, NS>(K);
  const int per_sm = std::max(1, std::min(16, (int)((227 * 1024) / (smem + 1024))));
  return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(ceil_div(nrows, (int64_t)32), (int64_t)kStgWarps),
                                                     (int64_t)ctx->sm_count * per_sm));
}

// shared-memory opt-in for the longest rows, once per device and kernel (a
// function attribute: set before any stream capture launches the kernel)
static mfe_status staged_configure(mfe_ctx* ctx, const void* kernel, size_t smem, bool* configured)
{
  const int dev = ctx->device;
  if (dev >= 0 && dev < 64 && configured[dev]) return MFE_OK;
  MFE_CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (dev >= 0 && dev < 64) configured[dev] = true;
  return MFE_OK;
}

// k_spmv_any for n rows with nnz entries, at most max_len each (<= 0: not known):
// the stage holds 1.25 times the mean and two entries more per row, 32 at most
// (rows of independent lengths hardly ever fill it: 720 of 752 entries at most
// over 46,000 groups of rows of 4 to 27)
static int any_cap(int64_t n, int64_t nnz, int max_len)
{
  const int most = max_len > 0 ? std::min(max_len, kStgMaxLen) : kStgMaxLen;
  return stg_cap(std::max(1, std::min(most, (int)(1.25 * (double)nnz / (double)std::max<int64_t>(n, 1)) + 2)), false);
}

// Warps per block.  A block's warps take neighbouring groups, whose rows mostly
// read the same part of x: FP32 rows of columns within 3,000 of the diagonal, whose
// large stages leave little L1, 600,000 rows of 27 to 32 / 20 to 32 / 27 entries,
// blocks of two 119, 113, 110 us, of eight 93, 85, 87 (with columns within 30 even).
// FP64 rows and short ones keep two (1.48 M FP64 rows of 4 to 27: 75.6 and 77.6), and so
// do matrices of fewer than four groups a warp, whose last ones are then unevenly
// spread over the SMs (rows of 27, columns near the diagonal: 30^3 2.96 and 3.01 us,
// 52^3 5.50 and 6.14, 70^3 9.20 and 9.40, 100^3 38.2 and 38.2; the last groups of all warps
// dealt out over the blocks 52^3 5.76, 70^3 9.71, and FP64 rows slower by 1 %).
template <typename T>
static int any_warps(const mfe_ctx* ctx, int64_t nrows, int cap)
{
  // (a stage of more than 25 entries a row: a mean row of 19 or more)
  return sizeof(T) == 4 && cap > 25 * 32 && nrows >= (int64_t)4 * 32 * kAnyWarps * ctx->sm_count ? 8 : 2;
}

template <typename T>
static size_t any_smem(int cap, int warps)
{
  return (size_t)warps * cap * (sizeof(T) + sizeof(int32_t));
}

template <typename T>
static int any_grid(mfe_ctx* ctx, int64_t nrows, int cap)
{
  const int W = any_warps<T>(ctx, nrows, cap);
  const int per_sm = std::max(1, std::min(kAnyWarps / W, (int)((228 * 1024) / (any_smem<T>(cap, W) + 1024 + 256 * W))));
  return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(ceil_div(nrows, (int64_t)32), (int64_t)W),
                                                     (int64_t)ctx->sm_count * per_sm));
}

template <typename T, int MODE, int W>
static mfe_status launch_any_w(mfe_ctx* ctx, SpmvParams<T>& P, int cap, int most)
{
  static bool configured[64] = {};
  MFE_TRY(staged_configure(ctx, (const void*)k_spmv_any<T, MODE, W>, any_smem<T>(stg_cap(kStgMaxLen, false), W),
                           configured));
  k_spmv_any<T, MODE, W><<<any_grid<T>(ctx, P.n, cap), W * 32, any_smem<T>(cap, W), ctx->stream>>>(P, cap, most);
  return check_launch(ctx, "k_spmv_any");
}

template <typename T, int MODE>
static mfe_status launch_any(mfe_ctx* ctx, SpmvParams<T>& P, int max_len)
{
  const int cap = any_cap(P.n, P.nnz, max_len);
  const int most = max_len > 0 ? stated_most(kCheckRows<T>, max_len) : INT_MAX;
  MFE_TRY(take_wait_injection(ctx, &P.withhold_ns));
  if constexpr (sizeof(T) == 4) {
    if (any_warps<T>(ctx, P.n, cap) == 8) return launch_any_w<T, MODE, 8>(ctx, P, cap, most);
  }
  return launch_any_w<T, MODE, 2>(ctx, P, cap, most);
}

int spmv_grid(mfe_ctx* ctx, const mfe_csr* A)
{
  const int max_len = A->max_row_len > 0 ? A->max_row_len : kStgMaxLen;
  if (max_len > kStgMaxLen)  // the warp-per-row kernel
    return (int)std::max<int64_t>(
        1, std::min<int64_t>(ceil_div(A->nrows * 32, 256), (int64_t)ctx->sm_count * 8));
  const int cap = any_cap(A->nrows, A->nnz, A->max_row_len);
  return A->dtype == MFE_F64 ? any_grid<double>(ctx, A->nrows, cap) : any_grid<float>(ctx, A->nrows, cap);
}

mfe_status ensure_max_row_len(mfe_ctx* ctx, const mfe_csr* A, int* max_len)
{
  if (A->max_row_len > 0) {
    *max_len = A->max_row_len;
    return MFE_OK;
  }
  int* d = static_cast<int*>(workspace(ctx, "spmv.maxlen", sizeof(int)));
  if (!d) return fail(ctx, MFE_OOM, "workspace allocation failed");
  MFE_CUDA_TRY(ctx, cudaMemsetAsync(d, 0, sizeof(int), ctx->stream));
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(ceil_div(A->nrows, 256),
                                                                (int64_t)ctx->sm_count * 8));
  k_max_row_len<<<(unsigned)blocks, 256, 0, ctx->stream>>>(A->nrows, A->row_offsets, d);
  MFE_TRY(check_launch(ctx, "k_max_row_len"));
  int* h = static_cast<int*>(host_scratch(ctx, sizeof(int)));
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(h, d, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  *max_len = *h;
  return MFE_OK;
}

template <typename T, int MODE>
static mfe_status launch_t(mfe_ctx* ctx, const mfe_csr* A, const T* x, T* y, const DotSink* sink,
                           const double* b, CgState* cg, int max_len)
{
  SpmvParams<T> P;
  P.n = A->nrows;
  P.nnz = A->nnz;
  P.ro = A->row_offsets;
  P.cols = A->cols;
  P.vals = static_cast<const T*>(A->vals);
  P.x = x;
  P.y = y;
  P.b = b;
  P.partials = sink ? sink->partials : nullptr;
  P.ticket = sink ? sink->ticket : nullptr;
  P.dot_out = sink ? sink->out : nullptr;
  P.cg = cg;
  P.withhold_ns = 0;
  P.err = static_cast<unsigned*>(workspace(ctx, "spmv.err", sizeof(unsigned)));
  if (!P.err) return fail(ctx, MFE_OOM, "workspace allocation failed");
  if (cg) P.err = &cg->err;
  if (A->nrows == 0) return MFE_OK;
  if (max_len <= kStgMaxLen && aligned16(A->vals) && aligned16(A->cols))
    return launch_any<T, MODE>(ctx, P, max_len);
  const int grid = (int)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(A->nrows * 32, 256), (int64_t)ctx->sm_count * 8));
  k_spmv_warp<T, MODE><<<grid, 256, 0, ctx->stream>>>(P);
  return check_launch(ctx, "k_spmv_warp");
}

mfe_status launch_spmv(mfe_ctx* ctx, const mfe_csr* A, const void* x, void* y,
                       const DotSink* sink, const double* resid_b, void* cg_state)
{
  // bulk async copies need 16-byte aligned sources
  if (csr_is_box(A) && aligned16(A->vals) && aligned16(x) &&
      getenv("MFE_SPMV_GENERIC") == nullptr)
    return launch_spmv_box(ctx, A, x, y, sink, resid_b, cg_state);
  // the longest row where it is stated, else the mean, decides the kernel
  int max_len = A->max_row_len;
  if (max_len <= 0 && A->nnz > (int64_t)kStgMaxLen * A->nrows) max_len = kStgMaxLen + 1;
  CgState* cg = static_cast<CgState*>(cg_state);
  if (A->dtype == MFE_F64) {
    const double* xd = static_cast<const double*>(x);
    double* yd = static_cast<double*>(y);
    if (resid_b) return launch_t<double, SPMV_RESID>(ctx, A, xd, yd, sink, resid_b, cg, max_len);
    if (sink) return launch_t<double, SPMV_DOT>(ctx, A, xd, yd, sink, nullptr, cg, max_len);
    return launch_t<double, SPMV_PLAIN>(ctx, A, xd, yd, nullptr, nullptr, cg, max_len);
  }
  if (A->dtype == MFE_F32) {
    const float* xf = static_cast<const float*>(x);
    float* yf = static_cast<float*>(y);
    if (resid_b) return fail(ctx, MFE_NOT_SUPPORTED, "FP32 residual SpMV is not provided");
    if (sink) return launch_t<float, SPMV_DOT>(ctx, A, xf, yf, sink, nullptr, cg, max_len);
    return launch_t<float, SPMV_PLAIN>(ctx, A, xf, yf, nullptr, nullptr, cg, max_len);
  }
  return fail(ctx, MFE_BAD_ARG, "unknown matrix dtype");
}

template <typename T, int MODE, int NS>
static mfe_status launch_ell_ns(mfe_ctx* ctx, const mfe_ell* E, const T* x, T* y, const DotSink* sink,
                                const double* b, CgState* cg)
{
  static bool configured[64] = {};
  MFE_TRY(staged_configure(ctx, (const void*)k_spmv_ell<T, MODE, NS>, ell_smem<T, NS>(kStgMaxLen),
                           configured));
  SpmvParams<T> P;
  memset(&P, 0, sizeof(P));
  P.n = E->nrows;
  P.nnz = E->nrows * (int64_t)E->ncols_per_row;
  P.cols = E->cols;
  P.vals = static_cast<const T*>(E->vals);
  P.x = x;
  P.y = y;
  P.b = b;
  P.partials = sink ? sink->partials : nullptr;
  P.ticket = sink ? sink->ticket : nullptr;
  P.dot_out = sink ? sink->out : nullptr;
  P.cg = cg;
  P.err = static_cast<unsigned*>(workspace(ctx, "spmv.err", sizeof(unsigned)));
  if (!P.err) return fail(ctx, MFE_OOM, "workspace allocation failed");
  if (cg) P.err = &cg->err;
  MFE_TRY(take_wait_injection(ctx, &P.withhold_ns));
  const int K = E->ncols_per_row;
  k_spmv_ell<T, MODE, NS><<<ell_grid<T, NS>(ctx, P.n, K), kStgWarps * 32, ell_smem<T, NS>(K),
                        ctx->stream>>>(P, K);
  return check_launch(ctx, "k_spmv_ell");
}

template <typename T, int MODE>
static mfe_status launch_ell_t(mfe_ctx* ctx, const mfe_ell* E, const T* x, T* y, const DotSink* sink,
                               const double* b, CgState* cg)
{
  if (sizeof(T) == 8 && E->nrows >= kEllOneStage) return launch_ell_ns<T, MODE, 1>(ctx, E, x, y, sink, b, cg);
  return launch_ell_ns<T, MODE, 2>(ctx, E, x, y, sink, b, cg);
}

mfe_status launch_spmv_ell(mfe_ctx* ctx, const mfe_ell* E, const void* x, void* y,
                           const DotSink* sink, const double* resid_b, void* cg_state)
{
  if (E->nrows == 0) return MFE_OK;
  // products with x.y (no caller on the ELL) also take the CSR view
  const bool dot_only = sink != nullptr && resid_b == nullptr;
  if (E->ncols_per_row > kStgMaxLen || !aligned16(E->vals) || !aligned16(E->cols) || dot_only) {
    mfe_csr V;
    MFE_TRY(ell_view(ctx, E, &V));
    return launch_spmv(ctx, &V, x, y, sink, resid_b, cg_state);
  }
  CgState* cg = static_cast<CgState*>(cg_state);
  if (E->dtype == MFE_F64) {
    const double* xd = static_cast<const double*>(x);
    double* yd = static_cast<double*>(y);
    if (resid_b) return launch_ell_t<double, SPMV_RESID>(ctx, E, xd, yd, sink, resid_b, cg);
    return launch_ell_t<double, SPMV_PLAIN>(ctx, E, xd, yd, nullptr, nullptr, cg);
  }
  if (E->dtype == MFE_F32) {
    const float* xf = static_cast<const float*>(x);
    float* yf = static_cast<float*>(y);
    if (resid_b) return fail(ctx, MFE_NOT_SUPPORTED, "FP32 residual SpMV is not provided");
    return launch_ell_t<float, SPMV_PLAIN>(ctx, E, xf, yf, nullptr, nullptr, cg);
  }
  return fail(ctx, MFE_BAD_ARG, "unknown matrix dtype");
}

mfe_status launch_spmm(mfe_ctx* ctx, const mfe_csr* A, int nrhs, const void* X, void* Y)
{
  if (A->nrows == 0) return MFE_OK;
  if (spmm_box_eligible(A, nrhs, X, Y) && getenv("MFE_SPMV_GENERIC") == nullptr)
    return launch_spmm_box(ctx, A, nrhs, X, Y);
  const int64_t total = A->nrows * (int64_t)nrhs;
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(ceil_div(total, 256),
                                                                (int64_t)ctx->sm_count * 16));
  if (A->dtype == MFE_F64)
    k_spmm<double><<<(unsigned)blocks, 256, 0, ctx->stream>>>(
        A->nrows, nrhs, A->row_offsets, A->cols, static_cast<const double*>(A->vals),
        static_cast<const double*>(X), static_cast<double*>(Y));
  else
    k_spmm<float><<<(unsigned)blocks, 256, 0, ctx->stream>>>(
        A->nrows, nrhs, A->row_offsets, A->cols, static_cast<const float*>(A->vals),
        static_cast<const float*>(X), static_cast<float*>(Y));
  return check_launch(ctx, "k_spmm");
}

mfe_status take_spmv_error(mfe_ctx* ctx)
{
  auto it = ctx->ws.find("spmv.err");
  if (it == ctx->ws.end() || !it->second.ptr) return MFE_OK;
  unsigned h = 0;
  MFE_CUDA_TRY(ctx, cudaMemcpyAsync(&h, it->second.ptr, sizeof(unsigned), cudaMemcpyDeviceToHost,
                                    ctx->stream));
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  if (!h) return MFE_OK;
  MFE_CUDA_TRY(ctx, cudaMemsetAsync(it->second.ptr, 0, sizeof(unsigned), ctx->stream));
  MFE_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return fail(ctx, MFE_TIMEOUT,
              (h & 1u) ? "a matrix-vector kernel gave up a bounded wait"
                       : "a matrix-vector kernel met a tile larger than its stage");
}

}  // namespace mfe
