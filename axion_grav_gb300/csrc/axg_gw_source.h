// axg_gw_source.h -- the FP64 Green's-function sources at one site
// (grav_waves.f90:323-356 data1_to_arr_dphi and :209-232): the central
// differences d_i phi = (phi(x + e_i) - phi(x - e_i)) / d, d = 2 dx, then
// S_ij = 2 ((d_i phi)_re (d_j phi)_re + (d_i phi)_im (d_j phi)_im) for
// (i, j) = (1,1),(2,1),(2,2),(3,1),(3,2),(3,3), in the reference's operation
// order.  The division by d is a multiplication by 1/d when d is a power of
// two (the same single rounding), and the factor 2 is exact.
#ifndef AXG_GW_SOURCE_H
#define AXG_GW_SOURCE_H

#include "axg_detmath.h"
#include "axg_internal.h"
#include "axg_soft64.h"

// xr[k], xi[k]: the raw differences (or their sums over a coarse cell) of
// direction k; divided by d, then the six products.  Hardware operations.
static __device__ __noinline__ void gw_sources_from_diff_hw(const double xr[3], const double xi[3], double d,
                                                            double inv_d, int d_pow2, double S[6]) {
  double dr[3], di[3];
  for (int k = 0; k < 3; ++k) {
    dr[k] = d_pow2 ? AXD_MUL(xr[k], inv_d) : AXD_DIV(xr[k], d);
    di[k] = d_pow2 ? AXD_MUL(xi[k], inv_d) : AXD_DIV(xi[k], d);
  }
  int c = 0;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j <= i; ++j, ++c) S[c] = AXD_MUL(AXD_ADD(AXD_MUL(dr[i], dr[j]), AXD_MUL(di[i], di[j])), 2.0);
}

// x / d.  d a power of two: an exponent change.  Else the quotient by the
// correctly rounded reciprocal and two fused corrections, which is the
// correctly rounded quotient unless d's significand is all ones (P.
// Markstein, IBM J. Res. Dev. 34 (1990) 111): an integer product and four
// fused operations for the FP64 pipe's ~14 of a division.
__device__ __forceinline__ double gw_div_d(double x, double d, const axs_const &inv_d, int d_pow2, uint32_t &ok) {
  if (d_pow2) return axg_mul_pow2(x, inv_d.v);
  double q = axs_mulc(x, &inv_d, &ok);
  q = AXD_FMA(AXD_FMA(-d, q, x), inv_d.v, q);
  return AXD_FMA(AXD_FMA(-d, q, x), inv_d.v, q);
}

// copies, so that the arrays of the usual path stay in registers
__device__ __forceinline__ void gw_sources_redo(const double xr[3], const double xi[3], double d, double inv_d,
                                                int d_pow2, double S[6]) {
  const double a[3] = {xr[0], xr[1], xr[2]}, b[3] = {xi[0], xi[1], xi[2]};
  double T[6];
  gw_sources_from_diff_hw(a, b, d, inv_d, d_pow2, T);
#pragma unroll
  for (int k = 0; k < 6; ++k) S[k] = T[k];
}

// The same with the products on the integer pipes (axg_soft64.h), for kernels
// that the FP64 pipe bounds; a site with an operand outside their window (a
// zero difference, say) is done above.  The float-float row pass keeps the
// hardware products (gw_sources_fp64<false>): its butterflies fill the issue
// slots, and 256^3 rows took 1.39 ms with integer products against 1.29.
__device__ __forceinline__ void gw_sources_from_diff(const double xr[3], const double xi[3], double d, double inv_d,
                                                     int d_pow2, double S[6]) {
  const axs_const ic = axs_const_of(inv_d), dc = axs_const_of(d);
  uint32_t ok = d_pow2 || (ic.ok && dc.ok && !(dc.hi == 0x1fffffu && dc.lo == 0xffffffffu)) ? 0xffffffffu : 0u;
  ok &= axs_window2(xr[0], xi[0]) & axs_window2(xr[1], xi[1]) & axs_window2(xr[2], xi[2]);
  if (!(ok & AXS_WINDOW)) {
    gw_sources_redo(xr, xi, d, inv_d, d_pow2, S);
    return;
  }
  double dr[3], di[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    dr[k] = gw_div_d(xr[k], d, ic, d_pow2, ok);
    di[k] = gw_div_d(xi[k], d, ic, d_pow2, ok);
  }
  int c = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j, ++c)
      S[c] = axg_mul_pow2(AXD_ADD(axs_mul(dr[i], dr[j], &ok), axs_mul(di[i], di[j], &ok)), 2.0);  // == r1 + r1
  if (!(ok & AXS_WINDOW)) gw_sources_redo(xr, xi, d, inv_d, d_pow2, S);
}

// pa[k], pb[k]: phi at x + e_k and x - e_k, k = x, y, z
template <bool SOFT>
__device__ __forceinline__ void gw_sources_fp64(const double2 pa[3], const double2 pb[3], double d, double inv_d,
                                                int d_pow2, double S[6]) {
  double xr[3], xi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    xr[k] = AXD_SUB(pa[k].x, pb[k].x);
    xi[k] = AXD_SUB(pa[k].y, pb[k].y);
  }
  if constexpr (SOFT) {
    gw_sources_from_diff(xr, xi, d, inv_d, d_pow2, S);
  } else {
    double dr[3], di[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dr[k] = d_pow2 ? axg_mul_pow2(xr[k], inv_d) : AXD_DIV(xr[k], d);
      di[k] = d_pow2 ? axg_mul_pow2(xi[k], inv_d) : AXD_DIV(xi[k], d);
    }
    int c = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j, ++c)
        S[c] = axg_mul_pow2(AXD_ADD(AXD_MUL(dr[i], dr[j]), AXD_MUL(di[i], di[j])), 2.0);
  }
}

#endif  // AXG_GW_SOURCE_H
