// The FP64 CG's product with the verified stencil operator, in fixed point on
// the integer pipe.
//
// The operator is mfe_stencil64.cu's: a Dirichlet row is dd * p, any other row
// (p~ = p with the Dirichlet nodes zeroed)
//   per plane z and position: a = p~, sx = the two x neighbours' sum, sy = the
//   two y neighbours', sxy = the four diagonal neighbours';
//   P1(z) = w4 a + w5 sx + w6 sy + w7 sxy   (the |dz| = 1 part)
//   Q(z)  = w0 a + w1 sx + w2 sy + w3 sxy   (the dz = 0 part)
//   y(z)  = P1(z-1) + Q(z) + P1(z+1)
// In FP64 that is 13.5 operations per row with p.Ap, and GB300's FP64 pipe
// takes 1.9 of them per clock and SM: 0.508 ms at 256^3 in the solve, against
// 0.041 ms for the bytes.  Its integer pipe does 60 multiply-adds of 32 x 32 +
// 64 bits per clock and SM, so the sums are formed there, closer to exact in norm
// than in FP64:
//
//   * Every p~ of a plane is split once, as it is staged in shared memory,
//     into its exponent e and a signed 60-bit integer v (2^7 times the
//     mantissa): p~ = v 2^(e - 1082).
//   * A thread owns four adjacent positions of the plane.  Per plane it takes
//     the largest exponent E of the 3 x 6 window its rows read, shifts the 18
//     integers to it (a floor at 2^-60 of the window's largest entry) and
//     adds them exactly in 64 bits.
//   * The weights are 62-bit integers W = w 2^k with sum |W| over the 27
//     entries at most 2^62, as signed halves wh 2^32 + wl.  A product W S
//     keeps wh sh and the two cross terms, three 32 x 32 + 64 bit
//     multiply-adds; the dropped wl sl is at most 1/4 unit of V below.
//   * V = the sum / 2^64, rounded, lies below 2^58: P1 and Q of a plane each
//     end in one 64-bit V at exponent E.  A row adds its V after shifting them
//     to the largest of their planes' E, converts once (round to nearest) and
//     moves the exponent.
//
// The result is within 2^-53 sum |w| max |p~| of exact, the maximum over the
// thread's windows in three planes, plus one rounding: in units of V, 2^-56 of that
// at most, 1/4 for the entries' floors, 0.85 for the weights' rounding, 4 x 1/4 dropped
// and 1/2 rounded in each of three plane parts, 2 where exponents are aligned.
// Measured along CGs of a 64 x 48 x 40 box (iterations 1 to 200; the arithmetic
// restated on the host against 113 bits), relative 2-norm, and the worst row's part
// of its own sum |w||p|: N(0, 1) right-hand sides 6e-17 to 8e-17 and 2e-16 to 4e-16
// (rows in FP64 1.4e-16 to 3.0e-16 and 4e-16 to 5e-16); miniFE's own, whose p falls by
// orders of magnitude next to the face at 1, 5e-17 to 7e-17 and, in one row in a
// hundred of the first iterations, up to 5e-14 (8e-17 to 3e-16 and 3e-16).
// So the product is closer than FP64 in norm, and row by row too where p has no such
// fronts; a row whose entries all lie 2^k below the window's largest loses k bits
// (a thread whose positions run over a line's end has both ends in its window).
// That is enough for the CG, whose
// scalars mix all of p and which stops on the CSR residual only; a product
// offered to a caller promises more, so that one (mfe_spmv_stencil64) and the
// Jacobi PCG's stay on the FP64 kernel.  Rows whose window holds an infinity, a
// NaN or entries so large or small that the result could leave the normal
// range are formed in FP64 (row_fp64).
//
// A CTA owns up to 4 NT consecutive positions of the xy plane and marches
// along z; the (plane tile, z) steps are shared out over the grid (fx_setup).  Per
// plane, with one barrier: the next plane's window (the tile and one line and
// one position on either side) is loaded coalesced while the current one is
// computed, then split into the other half of a two-plane buffer, and the
// rows of the last plane are written out coalesced from shared memory, where
// Dirichlet rows become dd * p and p.Ap takes its one FP64 FMA per row.  The
// split integers lie modulo 4 (element i at (i & 3) kS4 + i / 4), so that the
// 18 loads of neighbouring threads fall on neighbouring 16-byte words although
// each thread owns four adjacent positions.  p.Ap is summed in FP64 per thread,
// then per block and over the grid in block order (deterministic for a fixed
// grid).
//
// Measured at 256^3 in the solve: 0.218 ms against 0.508 ms; the solve of an
// N(0, 1) right-hand side to 2e-11 takes 0.40 ms per iteration instead of
// 0.70.  What bounds it: the integer pipe and, at 16 warps per SM, latency.  A row
// costs about 200 instructions; IMAD.WIDE and the ALU's instructions share one
// rate of 64 per clock and SM (microbenchmark: alternating LOP3 and IMAD.WIDE
// issue 2.0 per clock and SM together, as either alone).  At 200^3 the ALU pipe
// is busy 47 % of the time, the FP64 pipe (conversions, p.Ap) 44 %, the rest goes to the
// per-plane barrier and shared-memory queueing.  Tried and slower: exponents per
// row instead of per thread (0.34 ms without the dot against 0.19), the p and x
// updates fused into the staging pass (0.36 ms and more: its FP64 work then
// queues before the integer work of the same warps), the same with dedicated
// staging warps (0.37 ms), and x += alpha p of the iteration before carried by
// the rows written out (0.30 ms, of which the update kernel gives back 0.04).
#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "mfe_common.cuh"
#include "mfe_internal.h"

namespace mfe {

constexpr int kKP = 4;  // adjacent positions per thread

struct FxParams {
  int Nx, Ny, Nz, NxNy, ntile;
  int TP;             // positions per tile (at most 4 per thread, a multiple of 4)
  int L;              // staged elements per plane
  int nseg;           // runs a tile's planes are cut into (0: even shares of all steps)
  int line;           // staged elements from line y to line y + 1
  int wh[8], wl[8];   // weights 2^k w = wh 2^32 + wl, class 4|dz| + 2|dy| + |dx|
  int k, one;         // one: 1, as a number the compiler cannot see
  int e_lo, e_hi;     // window exponents whose rows stay in fixed point
  double w[8];        // the weights, and the Dirichlet diagonal
  double dd;
  const double* p;
  double* __restrict__ Ap;
};

__device__ __forceinline__ long long shr64(long long v, int s)
{
  long long r;  // shifts past 63 leave the sign
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}

__device__ __forceinline__ long long madw(int a, int b, long long c)
{
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// s = h 2^32 + l with signed halves
struct Half {
  int h, l;
};
__device__ __forceinline__ Half halves(long long s)
{
  const int l = (int)(unsigned)s;
  return {(int)(s >> 32) + (int)((unsigned)l >> 31), l};
}

// a staged entry: p~ = v 2^(e - 1082)
struct __align__(16) Split {
  long long v;
  int e, pad;
};

// stride of the quarters of n staged elements: 2 mod 8, so that the four start
// on different banks
__host__ __device__ constexpr int quarter_stride(int n) { return (n / 4 + 5) / 8 * 8 + 2; }

// p: read-only for the kernel, or (LOOP) written by it between two sweeps
template <bool LOOP>
__device__ __forceinline__ double fx_load(const double* a)
{
  return LOOP ? __ldcg(a) : __ldg(a);
}

// one interior row in FP64 (the separable sums, Dirichlet neighbours zeroed)
static __device__ __noinline__ double row_fp64(const FxParams& P, int ix, int iy, int z)
{
  double acc = 0.0;
  for (int dz = -1; dz <= 1; ++dz) {
    if (z + dz < 1 || z + dz > P.Nz - 2) continue;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int jx = ix + dx, jy = iy + dy;
        if (jx < 1 || jx > P.Nx - 2 || jy < 1 || jy > P.Ny - 2) continue;
        s[2 * (dy != 0) + (dx != 0)] += __ldcg(P.p + (int64_t)(z + dz) * P.NxNy + (int64_t)jy * P.Nx + jx);
      }
    const double* w = P.w + (dz ? 4 : 0);
    for (int c = 0; c < 4; ++c) acc = fma(w[c], s[c], acc);
  }
  return acc;
}

// NT threads (4 NT positions per tile at most), CM staged elements per thread
// and plane (P.L <= CM NT).  SEG: the window as three line segments instead
// of one run of positions.
template <int NT, int CM, bool SEG>
struct FxShape {
  static constexpr int kYq = NT + 4;                   // stride of a quarter of a plane of Ap
  static constexpr int kS4 = quarter_stride(CM * NT);  // stride of a quarter of a plane of p~
  static constexpr int kBuf = 4 * kS4;
  static constexpr size_t kSmem = 2 * ((size_t)kBuf * sizeof(Split) + (size_t)kKP * kYq * sizeof(double));
};

// Ap of block b's share (of nb blocks) of the (tile, z) steps, and the rows'
// terms of p.Ap added to dacc.  LOOP: within a kernel that writes p between two
// sweeps (mfe_cg_loop.cu), so p is read through L2.  Begins and ends without a
// barrier of its own: the caller orders two sweeps of a block by one.
template <int NT, int CM, bool SEG, bool LOOP>
__device__ __forceinline__ void fx_sweep(const FxParams& P, int b, int nb, unsigned char* smem, double (&dacc)[kKP])
{
  using Sh = FxShape<NT, CM, SEG>;
  constexpr int kYq = Sh::kYq, kS4 = Sh::kS4, kBuf = Sh::kBuf;
  Split* const sx = reinterpret_cast<Split*>(smem);              // 2 planes of p~
  double* const sy = reinterpret_cast<double*>(sx + 2 * kBuf);   // 2 planes of Ap
  const int tid = threadIdx.x;
  // the block's steps: one run of one tile, or an even share of all of them
  int64_t q0, q1;
  if (P.nseg > 0) {
    const int tile = b / P.nseg, seg = b - tile * P.nseg;
    q0 = (int64_t)tile * P.Nz + (int64_t)P.Nz * seg / P.nseg;
    q1 = (int64_t)tile * P.Nz + (int64_t)P.Nz * (seg + 1) / P.nseg;
  } else {
    const int64_t T = (int64_t)P.ntile * P.Nz;
    q0 = T * b / nb;
    q1 = T * (b + 1) / nb;
  }
  // the thread's window: entry t of line j at win[j][t & 3] (one further for t >= 4)
  const Split* win[3][4];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int o = j * P.line + t;
      win[j][t] = sx + (o & 3) * kS4 + (o >> 2) + tid;
    }
  Split* const put = sx + (tid & 3) * kS4 + (tid >> 2);  // staged element tid + m NT at put[m NT / 4]

  for (int64_t q = q0; q < q1;) {
    const int tile = (int)(q / P.Nz), za = (int)(q - (int64_t)tile * P.Nz);
    const int zb = (int)min((int64_t)P.Nz, za + (q1 - q));
    const int c0 = tile * P.TP, c1 = min(P.NxNy, c0 + P.TP);
    // staged element i: position c0 - 1 - Nx + i, or of line segment i /
    // line; bit m of inner: element tid + m NT is an interior node
    unsigned inner = 0;
    int pos[SEG ? CM : 1];
    pos[0] = c0 - 1 - P.Nx + tid;
#pragma unroll
    for (int m = 0; m < CM; ++m) {
      const int i = tid + m * NT;
      const int j = SEG ? i / P.line : 0;
      const int p = c0 - 1 + (j - 1) * P.Nx + (i - j * P.line);
      if (SEG) pos[m] = 0;
      if (i < P.L && p >= 0 && p < P.NxNy) {
        const int iy = p / P.Nx, ix = p - iy * P.Nx;
        if (SEG) pos[m] = p;
        if (ix >= 1 && ix <= P.Nx - 2 && iy >= 1 && iy <= P.Ny - 2) inner |= 1u << m;
      }
    }
    // bit r of drow: the row written out at c0 + tid + r NT is a Dirichlet
    // row; of orow: it is a row of the tile
    unsigned drow = 0, orow = 0;
#pragma unroll
    for (int r = 0; r < kKP; ++r) {
      const int p = c0 + tid + r * NT;
      const int iy = p / P.Nx, ix = p - iy * P.Nx;
      if (p < c1) orow |= 1u << r;
      if (ix == 0 || ix == P.Nx - 1 || iy == 0 || iy == P.Ny - 1) drow |= 1u << r;
    }

    double raw[CM];  // the thread's elements of the plane staged next
    auto fetch = [&](int z) {
      const unsigned in = z >= 1 && z <= P.Nz - 2 ? inner : 0u;
      const double* src = P.p + (int64_t)z * P.NxNy + (SEG ? 0 : pos[0]);
#pragma unroll
      for (int m = 0; m < CM; ++m) raw[m] = (in >> m) & 1u ? fx_load<LOOP>(src + (SEG ? pos[SEG ? m : 0] : m * NT)) : 0.0;
    };
    // the fetched elements split into half buf of the staged planes
    auto split = [&](auto buf) {
#pragma unroll
      for (int m = 0; m < CM; ++m) {
        const unsigned hi = (unsigned)__double2hiint(raw[m]), lo = (unsigned)__double2loint(raw[m]);
        int e = (int)((hi >> 20) & 0x7ffu);
        unsigned mh = hi & 0xfffffu;
        if (e) mh |= 0x100000u;
        else if (mh | lo) e = 1;  // subnormal
        const long long sg = (long long)((int)hi >> 31);
        const long long mag = (long long)(((unsigned long long)mh << 32 | lo) << 7);
        Split s;
        s.v = (mag ^ sg) - sg;
        s.e = e;
        s.pad = 0;
        *reinterpret_cast<int4*>(put + decltype(buf)::value * kBuf + m * (NT / 4)) = *reinterpret_cast<int4*>(&s);
      }
    };

    // S 2^Es: P1(z-1) + Q(z) of the row being formed; V1A / V1B at EA / EB:
    // P1 of the last two planes in turn
    long long S[kKP], V1A[kKP], V1B[kKP];
    int Es = 0, EA = 0, EB = 0;
#pragma unroll
    for (int r = 0; r < kKP; ++r) S[r] = V1A[r] = V1B[r] = 0;

    // the rows of plane zo, formed into half buf of sy, go out, with p.Ap
    auto write_out = [&](auto buf, int zo, const double* pc) {
      double* yo = P.Ap + (int64_t)zo * P.NxNy + c0 + tid;
      const double* so = sy + decltype(buf)::value * (kKP * kYq) + (tid & 3) * kYq + (tid >> 2);
      const unsigned dir = zo == 0 || zo == P.Nz - 1 ? ~0u : drow, wr = zo >= za ? orow : 0u;
#pragma unroll
      for (int r = 0; r < kKP; ++r) {
        if (((wr & ~dir) >> r) & 1u) {
          const double yv = so[r * (NT / 4)];
          dacc[r] = fma(yv, pc[r], dacc[r]);
          yo[r * NT] = yv;
        }
      }
      if (wr & dir) {
#pragma unroll 1
        for (int r = 0; r < kKP; ++r) {
          if (((wr & dir) >> r) & 1u) {
            const double c = fx_load<LOOP>(P.p + (int64_t)zo * P.NxNy + c0 + tid + r * NT), yv = P.dd * c;
            dacc[0] = fma(yv, c, dacc[0]);
            yo[r * NT] = yv;
          }
        }
      }
    };
    // p at the rows written out
    auto centres = [&](int zo, double* pc) {
      const double* po = P.p + (int64_t)zo * P.NxNy + c0 + tid;
      const unsigned wr = zo >= za ? orow : 0u;
#pragma unroll
      for (int r = 0; r < kKP; ++r) pc[r] = (wr >> r) & 1u ? fx_load<LOOP>(po + r * NT) : 0.0;
    };

    // Plane zp is staged in half `buf`: the rows of plane zp - 1 follow from
    // it, those of plane zp - 2 go out, and plane zp + 1 is staged in the other
    // half.  The loads of the last two are issued first, so that they arrive
    // during the integer work.  Threads without rows of the tile and planes of
    // Dirichlet nodes (staged as zeros) run the same code.
    auto step = [&](auto buf, int zp, const long long* V1p, int Ep, long long* V1n, int& En) {
      constexpr int BF = decltype(buf)::value;
      using Other = std::integral_constant<int, BF ^ 1>;
      __syncthreads();
      double pc[kKP];
      fetch(zp + 1);
      centres(zp - 2, pc);
      Split w[18];
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int t = 0; t < 6; ++t) {
          const int4 u = *reinterpret_cast<const int4*>(win[j][t & 3] + BF * kBuf + (t >> 2));
          w[6 * j + t].v = (long long)((unsigned long long)(unsigned)u.x | (unsigned long long)(unsigned)u.y << 32);
          w[6 * j + t].e = u.z;
        }
      int E = 0;
#pragma unroll
      for (int t = 0; t < 18; t += 2) E = max(E, max(w[t].e, w[t + 1].e));
      const int E3 = max(Es, E), E2 = max(Ep, E);
      const int sh = (E3 - 1018 - P.k) << 20;
      long long v[18];
#pragma unroll
      for (int t = 0; t < 18; ++t) v[t] = shr64(w[t].v, E - w[t].e);
      long long ey[6];  // lines y - 1 and y + 1 added
#pragma unroll
      for (int t = 0; t < 6; ++t) ey[t] = v[t] + v[12 + t];
      double* const so = sy + (BF ^ 1) * (kKP * kYq) + tid;
      double d[kKP];
      int up[kKP];
#pragma unroll
      for (int r = 0; r < kKP; ++r) {
        const Half s[4] = {halves(v[7 + r]), halves(v[6 + r] + v[8 + r]), halves(ey[r + 1]),
                           halves(ey[r] + ey[r + 2])};
        long long h1 = 0, m1 = 1ll << 31, hq = 0, mq = 1ll << 31;  // m >> 32 rounds
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          h1 = madw(P.wh[4 + c], s[c].h, h1);
          m1 = madw(P.wh[4 + c], s[c].l, m1);
          m1 = madw(P.wl[4 + c], s[c].h, m1);
          hq = madw(P.wh[c], s[c].h, hq);
          mq = madw(P.wh[c], s[c].l, mq);
          mq = madw(P.wl[c], s[c].h, mq);
        }
        V1n[r] = madw((int)(m1 >> 32), P.one, h1);  // h1 + (m1 >> 32) on the multiplier
        const long long Q = madw((int)(mq >> 32), P.one, hq);
        const long long V = shr64(S[r], E3 - Es) + shr64(V1n[r], E3 - E);
        d[r] = (double)V;
        up[r] = V != 0 ? sh : 0;  // the exponent's move (a zero stays one)
        S[r] = shr64(V1p[r], E2 - Ep) + shr64(Q, E2 - E);
      }
      write_out(buf, zp - 2, pc);
      split(Other{});
      // (the conversions have had the two calls above to finish)
#pragma unroll
      for (int r = 0; r < kKP; ++r) so[r * kYq] = __hiloint2double(__double2hiint(d[r]) + up[r], __double2loint(d[r]));
      if (E3 != 0 && (unsigned)(E3 - P.e_lo) > (unsigned)(P.e_hi - P.e_lo) && zp - 1 >= za) {
#pragma unroll 1
        for (int r = 0; r < kKP; ++r) {
          const int pp = c0 + kKP * tid + r, iy = pp / P.Nx, ix = pp - iy * P.Nx;
          if (pp < c1) so[r * kYq] = row_fp64(P, ix, iy, zp - 1);
        }
      }
      En = E;
      Es = E2;
    };
    using B0 = std::integral_constant<int, 0>;
    using B1 = std::integral_constant<int, 1>;

    fetch(za - 1);    // first plane of the window
    __syncthreads();  // the previous run's shared memory is no longer read
    split(B0{});
    int zp = za - 1;
    for (; zp + 1 <= zb; zp += 2) {
      step(B0{}, zp, V1B, EB, V1A, EA);
      step(B1{}, zp + 1, V1A, EA, V1B, EB);
    }
    double pc[kKP];
    if (zp <= zb) {
      step(B0{}, zp, V1B, EB, V1A, EA);
      __syncthreads();
      centres(zb - 1, pc);
      write_out(B1{}, zb - 1, pc);
    } else {
      __syncthreads();
      centres(zb - 1, pc);
      write_out(B0{}, zb - 1, pc);
    }
    q += zb - za;
  }
}

// The weights in fixed point: k with sum |w| 2^k over the 27 entries in
// (2^61, 2^62], and the range of window exponents whose results are sure to
// be normal numbers (0 < |V| <= 2^58 at 2^(E - 1018 - k)).
inline void fx_weights(FxParams& P, const double* w8)
{
  const int mult[8] = {1, 2, 2, 4, 2, 4, 4, 8};  // entries of each class
  double big = 0.0, sum = 0.0;
  for (int c = 0; c < 8; ++c) big = std::max(big, std::fabs(w8[c]));
  int ex, es;
  std::frexp(big, &ex);
  for (int c = 0; c < 8; ++c) sum += mult[c] * std::fabs(std::ldexp(w8[c], -ex));
  std::frexp(sum, &es);
  P.k = 62 - es - ex;
  for (int c = 0; c < 8; ++c) {
    P.w[c] = w8[c];
    const int64_t W = std::llrint(std::ldexp(w8[c], P.k));
    P.wl[c] = (int)(uint32_t)(uint64_t)W;
    P.wh[c] = (int)((W - P.wl[c]) >> 32);
  }
  P.one = 1;
  P.e_lo = std::max(1, P.k - 4);
  P.e_hi = std::min(2046, 1983 + P.k);
  if (P.e_lo > P.e_hi) P.e_lo = P.e_hi = 1 << 20;  // no such window: every row in FP64
}

// tiles of one size, a multiple of 4 and at most 4 NT; their window as one run
// of positions, or (three) as three line segments
inline void fx_tiles(FxParams& P, int NT, bool three)
{
  P.ntile = (int)ceil_div(P.NxNy, (int64_t)kKP * NT);
  P.TP = (int)((ceil_div(P.NxNy, (int64_t)P.ntile) + 3) & ~3);
  P.line = three ? P.TP + 2 : P.Nx;
  P.L = three ? 3 * P.line : P.TP + 2 + 2 * P.Nx;
}

// Which shape of the sweep: tiles of 2048 positions with one CTA per SM, or of
// 1024 with two; and how the (tile, z) steps are shared out: evenly over the
// CTAs, or as equal runs of one tile's planes each.  A run stages two planes
// more than it has steps, and an even share may end one tile and begin the
// next, which costs two planes again, so the choice is the one whose busiest
// CTA stages the fewest planes, and two CTAs per SM where they tie (one computes
// while the other waits at its plane's barrier, which gains more than the
// larger tile's smaller overlap).  Measured per iteration: even shares only
// against this rule, 97 x 64 x 83 elements 36.8 / 33.0 us, 128^3 77.6 / 72.1;
// one CTA against two at a tie, 150 x 160 x 170 125.5 / 119.2, 200^3 220.6 /
// 212.3, 240^3 350 / 333, 256^3 417 / 405.  The window is one run of positions
// while it fits six elements per thread, else three line segments (node lines
// over 511 long).
enum FxKind { FX_512 = 0, FX_256X2 = 1, FX_SEG = 2 };

inline FxKind fx_setup(const mfe_ctx* ctx, const mfe_csr* A, const double* w8, double dd, const double* p,
                       double* Ap, FxParams& P, int* grid)
{
  P.Nx = A->box_nx + 1;
  P.Ny = A->box_ny + 1;
  P.Nz = A->box_nz + 1;
  P.NxNy = P.Nx * P.Ny;
  fx_weights(P, w8);
  P.dd = dd;
  P.p = p;
  P.Ap = Ap;
  // planes of the busiest of `slots` CTAs
  auto share = [&](int slots) {
    const int64_t T = (int64_t)P.ntile * P.Nz;
    const int g = (int)std::min<int64_t>(T, slots);
    const int64_t even = ceil_div(T, g) + (T % g || (T / g) % P.Nz ? 4 : 2);
    const int nseg = std::min(P.Nz, slots / P.ntile);
    const int64_t runs = nseg > 0 ? ceil_div(P.Nz, nseg) + 2 : even + 1;
    P.nseg = runs < even ? nseg : 0;
    *grid = P.nseg ? P.ntile * nseg : g;
    return std::min(runs, even);
  };
  fx_tiles(P, 512, false);
  const int64_t p512 = share(ctx->sm_count);
  fx_tiles(P, 256, false);
  if (P.L <= 6 * 256 && share(2 * ctx->sm_count) <= p512) return FX_256X2;
  fx_tiles(P, 512, false);
  share(ctx->sm_count);
  if (P.L <= 6 * 512) return FX_512;
  fx_tiles(P, 256, true);
  share(ctx->sm_count);
  return FX_SEG;
}

}  // namespace mfe
