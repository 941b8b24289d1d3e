// Hex8 element math on the device, in the reference's floating-point
// operation order (ref/fem/Hex8.hpp).  The translation unit that includes
// this header is compiled with -fmad=false, so every multiply and add is
// rounded separately exactly as in the reference's g++ build, and division is
// IEEE round-to-nearest; element matrices and source vectors are therefore
// bit-identical to the reference's.
#pragma once

#include <cstdint>

#include "mfe_intmul.cuh"

namespace mfe {

// 2x2x2 Gauss points from gauss_pts(2) (ref/fem/gauss_pts.hpp:41,50-53): the
// truncated constant 0.577350269, weights 1.0.
constexpr double kGaussPt = 0.577350269;

// Reference-element shape-function gradients at the 8 Gauss points
// (compute_gradient_values, ref/fem/Hex8_ElemData.hpp:37-61), laid out
// [gp][node][dim]; gp = ig*4 + jg*2 + kg with pt = (gpts[ig], gpts[jg],
// gpts[kg]).  Filled once by the host (same expression order as
// Hex8::gradients, Hex8.hpp:68-113; products of constants, no adds to fuse).
struct Hex8Tables {
  double grad[8][8][3];
  double psi[8][8];  // shape_fns at each Gauss point (Hex8.hpp:44-65)
  // |grad[gp][i][d]| depends on the node's two other sides only:
  // mag[gp][d][a + 2 b] for sides a, b along the other two dimensions in order;
  // and the same taken apart for integer multiplication
  double mag[8][3][4];
  IntMul imag[8][3][4];
  IntMul ipsi[8][8];  // psi taken apart
};

// node i's side (0 or 1) along dimension d
__host__ __device__ constexpr int hex8_side(int i, int d)
{
  return d == 0 ? (i == 1 || i == 2 || i == 5 || i == 6) : d == 1 ? (i == 2 || i == 3 || i == 6 || i == 7) : i >= 4;
}

// diffusionMatrix_symm (Hex8.hpp:260-361) with conductivity k, and
// sourceVector (Hex8.hpp:364-410).  em: 36 upper-triangle entries, row-major;
// ev: 8 entries.  Both loops walk the Gauss points in the same order and
// compute the same Jacobian, so they share it.  jf(gp, J) provides the
// Jacobian at Gauss point gp (from per-axis tables, jacobian_column()).
// The sums lie in shared memory, entry i at em[i * S] and ev[i * S] (a column
// per thread): 88 registers less, so that three blocks of 128 threads share an
// SM and one warp's integer work runs beside another's FP64 work.
// Per Gauss point that leaves 214 operations for the FP64 pipe (438 with the
// multiplications) and about 4,000 integer instructions.  Measured, k_element
// over 256^3 elements (16 launches): 111 ms with all of it in FP64; 72 ms with
// the 108 products and 36 scalings of the matrix entries as integers (and 36
// gradient products for 72); 66 ms with the gradient and source products too;
// 61 ms with the sums in shared memory, 0.79 of the FP64 pipe's rate on what is
// left there (four blocks of 128 registers: 62 ms).
template <int S, typename JF>
__device__ __forceinline__ void element_matrix_vector_j(const Hex8Tables& T, JF jf, double k, double* em,
                                                        double* ev)
{
#pragma unroll
  for (int i = 0; i < 36; ++i) em[i * S] = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) ev[i * S] = 0.0;

#pragma unroll 1
  for (int gp = 0; gp < 8; ++gp) {
    double J[9];
    jf(gp, J);
    const double J00 = J[0], J01 = J[1], J02 = J[2], J10 = J[3], J11 = J[4], J12 = J[5],
                 J20 = J[6], J21 = J[7], J22 = J[8];
    const double term0 = J22 * J11 - J21 * J12;
    const double term1 = J22 * J01 - J21 * J02;
    const double term2 = J12 * J01 - J11 * J02;
    const double detJ = J00 * term0 - J10 * term1 + J20 * term2;
    const double inv_detJ = 1.0 / detJ;
    double iJ[9];
    iJ[0] = term0 * inv_detJ;
    iJ[1] = -term1 * inv_detJ;
    iJ[2] = term2 * inv_detJ;
    iJ[3] = -(J22 * J10 - J20 * J12) * inv_detJ;
    iJ[4] = (J22 * J00 - J20 * J02) * inv_detJ;
    iJ[5] = -(J12 * J00 - J10 * J02) * inv_detJ;
    iJ[6] = (J21 * J10 - J20 * J11) * inv_detJ;
    iJ[7] = -(J21 * J00 - J20 * J01) * inv_detJ;
    iJ[8] = (J11 * J00 - J10 * J01) * inv_detJ;

    // weights are 1.0: wi_wj_wk = 1*1*1 (Hex8.hpp:293-299)
    const double k_detJ_w = k * detJ * 1.0;
    // The multiplications run on the integer pipe (mfe_intmul.cuh), the
    // additions on the FP64 pipe.  detJ and k_detJ_w lie in [2^-200, 2^200] and
    // the entries of iJ are zero or in [2^-300, 2^300] on any box worth the name,
    // and then so are the gradients within [2^-340, 2^340]; the sums of their
    // products are zero or at least 2^-735, and every product is a normal
    // number.  Anything else takes the FP64 form (wide).
    bool wide = !intmul_range<200>(k_detJ_w) || !intmul_range<200>(detJ);
#pragma unroll
    for (int j = 0; j < 9; ++j) wide = wide || !(iJ[j] == 0.0 || intmul_range<300>(iJ[j]));
    // The gradients (Hex8.hpp:301-310): node i's is a sum of three products
    // +-|g| * iJ, and |g| takes four values per dimension, so 36 products do
    // for the 72 (a product's sign does not change its rounding).
    double dxyz[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double q[3][4];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double f = iJ[3 * c + d];
        const uint32_t fh = (uint32_t)__double2hiint(f), fl = (uint32_t)__double2loint(f);
        const IntMul F = intmul_split(fh, fl);
        const bool zero = (fh << 1) == 0u;  // (the product then is f)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          uint32_t h, l;
          intmul(T.imag[gp][d][t], F, h, l);
          q[d][t] = __hiloint2double((int)(zero ? fh : h), (int)(zero ? fl : l));
        }
      }
      if (wide) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
          for (int t = 0; t < 4; ++t) q[d][t] = T.mag[gp][d][t] * iJ[3 * c + d];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int sx = hex8_side(i, 0), sy = hex8_side(i, 1), sz = hex8_side(i, 2);
        const double p0 = sx ? q[0][sy + 2 * sz] : -q[0][sy + 2 * sz];
        const double p1 = sy ? q[1][sx + 2 * sz] : -q[1][sx + 2 * sz];
        const double p2 = sz ? q[2][sx + 2 * sy] : -q[2][sx + 2 * sy];
        dxyz[c][i] = p0 + p1 + p2;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 8; ++i) wide = wide || !intmul_range<340>(dxyz[c][i]);
    // em += k_detJ_w * ((dx dx) + (dy dy) + (dz dz)) per pair of nodes
    // (Hex8.hpp:312-340)
    if (!wide) {
      IntMul D[3][8];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 8; ++i) D[c][i] = intmul_split(dxyz[c][i]);
      const IntMul K = intmul_split(k_detJ_w);
      const uint32_t ksign = (uint32_t)__double2hiint(k_detJ_w) & 0x80000000u;
      int off = 0;
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int n = m; n < 8; ++n) {
          const double s = intmul(D[0][m], D[0][n]) + intmul(D[1][m], D[1][n]) + intmul(D[2][m], D[2][n]);
          const uint32_t sh = (uint32_t)__double2hiint(s), sl = (uint32_t)__double2loint(s);
          uint32_t ph, pl;
          intmul(intmul_split(sh, sl), K, ph, pl);
          if ((sh << 1) == 0u) {  // a sum of zero (none is subnormal)
            ph = sh ^ ksign;
            pl = 0u;
          }
          em[off * S] += __hiloint2double((int)ph, (int)pl);
          ++off;
        }
    } else {
      int off = 0;
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int n = m; n < 8; ++n) {
          em[off * S] += k_detJ_w * ((dxyz[0][m] * dxyz[0][n]) + (dxyz[1][m] * dxyz[1][n]) + (dxyz[2][m] * dxyz[2][n]));
          ++off;
        }
    }
    // sourceVector: term = Q*detJ*wi*wj*wk with Q = 1 (Hex8.hpp:402)
    const double term = 1.0 * detJ * 1.0 * 1.0 * 1.0;
    if (!wide) {
      const IntMul D = intmul_split(term);
#pragma unroll
      for (int i = 0; i < 8; ++i) ev[i * S] += intmul(T.ipsi[gp][i], D);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) ev[i * S] += T.psi[gp][i] * term;
    }
  }
}

// The Jacobian's column for physical axis x (entries J[a][0], a = 0..2) sums
// grad[gp][i][a] * x_i over the element's 8 nodes, whose x is x0 or x1: it
// depends on the element's x pair only, and likewise for y and z.  Computed
// with the reference's operations in its order (Hex8.hpp:198-236) (node order, from 0), the column
// of an element index along an axis is therefore exact for every element of
// that index.  axis: 0 x, 1 y, 2 z; (c0, c1) the index's coordinate pair.
__device__ __forceinline__ void jacobian_column(const Hex8Tables& T, int axis, double c0, double c1,
                                                int gp, double col[3])
{
  double s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const bool hi = axis == 0 ? (i == 1 || i == 2 || i == 5 || i == 6)
                              : (axis == 1 ? (i == 2 || i == 3 || i == 6 || i == 7) : (i >= 4));
    const double v = hi ? c1 : c0;
    s0 += T.grad[gp][i][0] * v;
    s1 += T.grad[gp][i][1] * v;
    s2 += T.grad[gp][i][2] * v;
  }
  col[0] = s0;
  col[1] = s1;
  col[2] = s2;
}

// Index of (a, b) in the 36-entry upper triangle (a, b in 0..7).
__host__ __device__ constexpr int sym_index(int a, int b)
{
  return a <= b ? a * 8 - (a * (a - 1)) / 2 + (b - a) : b * 8 - (b * (b - 1)) / 2 + (a - b);
}

// Local node index (exodus order, Hex8_box_utils.hpp:49-56) of the corner
// at offset (ox, oy, oz) in {0,1}^3 from the element's node 0.
__host__ __device__ constexpr int local_node(int ox, int oy, int oz)
{
  return oz * 4 + (oy ? (ox ? 2 : 3) : (ox ? 1 : 0));
}

}  // namespace mfe
