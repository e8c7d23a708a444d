// axg_gw_site.h -- per-wave-vector arithmetic of the gravitational-wave
// spectra: the polarisation tensor, the Green phase, the float-float
// accumulator update and the TT basis.  Shared by the kernels that read a
// finished spectrum and those that consume it inside its last transform pass.
#pragma once
#include <cstdint>

#include "axg_internal.h"

// get_comwav_grav (grav_waves.f90:157-191): p = (qz c - i s, qz s + i c, -r)
// for the unit vector q of k, (c, s) its azimuth; e+_ij = p_i p_j, halved on
// the diagonal, in the component order (1,1),(2,1),(2,2),(3,1),(3,2),(3,3).
// Divisions are reciprocal multiplies (one rounding more than the reference).
template <typename R>
__device__ __forceinline__ bool gw_polarisation(R kx, R ky, R kz, R qq, R pr[6], R pi[6]) {
  if (!(qq > 0)) return false;
  const R iq = R(1) / qq;
  const R qx = kx * iq, qy = ky * iq, qz = kz * iq;
  const R r = sqrt(qx * qx + qy * qy);
  R c = 1, sn = 0;
  if (r > 0) {
    const R ir = R(1) / r;
    c = qx * ir;
    sn = qy * ir;
  }
  const R ar[3] = {qz * c, qz * sn, -r}, ai[3] = {-sn, c, 0};
  int comp = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j, ++comp) {
      R er = ar[i] * ar[j] - ai[i] * ai[j], ei = ar[i] * ai[j] + ai[i] * ar[j];
      if (i == j) {
        er *= R(0.5);
        ei *= R(0.5);
      }
      pr[comp] = er;
      pi[comp] = ei;
    }
  return true;
}

// (hi, lo) += x: TwoSum of hi and x, the error folded into lo, then
// renormalised (Fast2Sum); hi + lo carries about 48 significant bits
__device__ __forceinline__ void ff_add(float &hi, float &lo, float x) {
  const float s = hi + x;
  const float bb = s - hi;
  const float err = (hi - (s - bb)) + (x - bb);
  const float l = lo + err;
  hi = s + l;
  lo = l - (hi - s);
}

// cos and sin of |k| dk tau from k^2 (an exact float, > 0), ik = 1/|k| and the
// phase of |k| = 1 in quarter turns, Th + Tl: |k| = k^2 ik refined to float-float,
// the product's integer part taken off exactly, and the Taylor polynomials of
// sin and cos of (pi/2) f on |f| <= 1/2 (next terms 2e-9 and 1e-10).
__device__ __forceinline__ void gw_cos_sin(float k2, float ik, float Th, float Tl, float *cq, float *sq) {
  const float k = k2 * ik, kl = 0.5f * ik * fmaf(-k, k, k2);
  const float ph = k * Th, pl = fmaf(k, Th, -ph) + fmaf(k, Tl, kl * Th);
  const float m = rintf(ph), f = (ph - m) + pl, g = f * f;
  const float s = fmaf(f, 1.5707963267948966f,
                       f * fmaf(g, fmaf(g, fmaf(g, fmaf(g, 1.6044118478735982e-4f, -4.6817541353186881e-3f),
                                                7.9692626246167046e-2f),
                                        -0.64596409750624625f),
                                -4.3711390001898e-08f));  // pi/2 less its float
  const float c = fmaf(g, fmaf(g, fmaf(g, fmaf(g, fmaf(g, -2.5202042373060605e-5f, 9.1926027483942659e-4f),
                                               -2.0863480763352961e-2f),
                                       0.25366950790104802f),
                               -1.2337005501361698f),
                       1.f);
  const int q = (int)m;
  const float a = q & 1 ? c : s, b = q & 1 ? s : c;
  *sq = q & 2 ? -a : a;
  *cq = (q + 1) & 2 ? -b : b;
}
// 1 / sqrt(x), x > 0: the hardware's approximation and one Newton step
__device__ __forceinline__ float gw_rsqrt(float x) {
  const float r = rsqrtf(x);
  return fmaf(0.5f * r, fmaf(-x * r, r, 1.f), r);
}

// The float-float accumulators of one entry, updated from FP32 X+, X- and the
// weights w_c, w_s.  REF: a12 += w_s X+ + w_c X-, a21 = a12 - w_c (last X-), so
// that the a21 of before is not read.
struct F32Acc {
  float4 a11, a21, a12, a22;
  __device__ __forceinline__ void load(const float4 *__restrict__ acc, int64_t astride, int64_t s, int ref_compat) {
    a11 = acc[s];
    a12 = acc[2 * astride + s];
    a22 = acc[3 * astride + s];
    if (!ref_compat) a21 = acc[astride + s];
  }
  __device__ __forceinline__ void update(float wc, float ws, const float xp[2], const float xm[2], const float lm[2],
                                         int ref_compat) {
    ff_add(a11.x, a11.y, wc * xp[0]);
    ff_add(a11.z, a11.w, wc * xp[1]);
    ff_add(a22.x, a22.y, ws * xm[0]);
    ff_add(a22.z, a22.w, ws * xm[1]);
    if (ref_compat) {
      ff_add(a12.x, a12.y, fmaf(wc, xm[0], ws * xp[0]));
      ff_add(a12.z, a12.w, fmaf(wc, xm[1], ws * xp[1]));
      a21 = a12;
      ff_add(a21.x, a21.y, -wc * lm[0]);
      ff_add(a21.z, a21.w, -wc * lm[1]);
    } else {
      ff_add(a21.x, a21.y, ws * xp[0]);
      ff_add(a21.z, a21.w, ws * xp[1]);
      ff_add(a12.x, a12.y, wc * xm[0]);
      ff_add(a12.z, a12.w, wc * xm[1]);
    }
  }
  __device__ __forceinline__ void store(float4 *__restrict__ acc, int64_t astride, int64_t s) const {
    acc[s] = a11;
    acc[astride + s] = a21;
    acc[2 * astride + s] = a12;
    acc[3 * astride + s] = a22;
  }
};

// The TT part of a symmetric tensor spectrum U (components 11, 21, 22, 31, 32,
// 33) in the basis (m, l) normal to k: m = (-s, c, 0) with (c, s) the azimuth
// of k, l = k x m / |k|.  |Lambda U|^2 = |U_mm - U_ll|^2 / 2 + 2 |U_ml|^2 with
// U_mm - U_ll = sum a_c U_c and |k| U_ml = sum b_c U_c; a and b are rational
// in the integers k:
//   a_11 = s^2 - q^2 c^2,  a_21 = -2 s c (1 + q^2),  a_22 = c^2 - q^2 s^2,
//   a_31 = 2 kz kx / k^2,  a_32 = 2 kz ky / k^2,     a_33 = -(a_11 + a_22),
//   b_11 = kz s c,  b_21 = kz (s^2 - c^2),  b_22 = -b_11,  b_31 = -ky,  b_32 = kx
// with c^2 = kx^2 / p^2, s^2 = ky^2 / p^2, s c = kx ky / p^2, q = kz / k.
// a_33 that way, the trace drops out of the differences U_11 - U_33 and
// U_22 - U_33 exactly.  20 multiply-adds a tensor where P U P - P tr(P U) / 2,
// P = 1 - k k, and its squared norm took ~200 operations.
template <typename R>
struct TTBasis {
  R a11, a21, a22, a31, a32, b11, b21, b31, b32, ik2;
};
template <typename R>
__device__ __forceinline__ TTBasis<R> tt_basis(int kx, int ky, int kz, int k2) {
  const int p2 = kx * kx + ky * ky;
  const R ik2 = R(1) / (R)k2, ip2 = p2 ? R(1) / (R)p2 : R(0);
  const R cc = p2 ? (R)(kx * kx) * ip2 : R(1), ss = (R)(ky * ky) * ip2, sc = (R)(kx * ky) * ip2;
  const R qq = (R)(kz * kz) * ik2;
  TTBasis<R> t;
  t.a11 = ss - qq * cc;
  t.a21 = R(-2) * sc * (R(1) + qq);
  t.a22 = cc - qq * ss;
  t.a31 = (R)(2 * kz * kx) * ik2;
  t.a32 = (R)(2 * kz * ky) * ik2;
  t.b11 = (R)kz * sc;
  t.b21 = (R)kz * (ss - cc);
  t.b31 = (R)-ky;
  t.b32 = (R)kx;
  t.ik2 = ik2;
  return t;
}
