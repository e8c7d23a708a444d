// axg_spectrum.cu -- masked field spectrum with window deconvolution
// (spectrum.f90:23-171, 242-567, 736-954) on the GPU.
//
//   init (once): mode-coupling table mat_spec(0:500, num_cov) by the
//        reference's 200-point quadrature (spectrum.f90:74-98, 117-171);
//   conv spectrum: k_spec_degrade box-averages phidot over deg^3 and zeroes
//        coarse cells that hold a masked cell (flag bit 4 of the last
//        classification, the device-resident form of the reference's mask
//        files), cuFFT Z2Z backward, k_spec_bin bins |F dx^3|^2 dk^3;
//   window matrix: the reference sums |W(k)|^2 interp_ij(|k|) over all k for
//        each of the num_cov = nb(nb+1)/2 bin pairs (O(num_cov N^3),
//        spectrum.f90:385-428).  Here |W|^2 and the mode count are first
//        histogrammed by integer |k|^2 (k_spec_w2_hist), an exact regrouping,
//        and k_spec_mat sums prefix sums of the histogram against the cells
//        of the interpolation table (O(num_cov * 500)), or k_spec_mat_direct
//        the histogram itself where that is shorter;
//   packed Cholesky inverse (dpptrf/dpptri) and dspmv on the host (nb x nb).
#include <cmath>
#include <vector>

#include "axg_binning.h"
#include "axg_detmath.h"
#include "axg_internal.h"

namespace {

constexpr double kRefPi = 3.14159265359;
constexpr double kRefTwoPi = 2 * kRefPi;
constexpr int kNumLargeq = 500;
constexpr int kNumInt = 200;

template <typename V>
__global__ void k_spec_degrade(const V *__restrict__ phid, const int8_t *__restrict__ flags, int n, int deg,
                               double inv_deg3, int window, double dv_spa, double2 *__restrict__ out) {
  // inv_deg3 = 1 / deg^3
  const int m = n / deg;
  const int64_t m3 = (int64_t)m * m * m, n2 = (int64_t)n * n;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < m3; c += stride) {
    const int ix = (int)(c % m), iy = (int)((c / m) % m), iz = (int)(c / ((int64_t)m * m));
    double sr = 0.0, si = 0.0;
    bool masked = false;
    for (int z0 = iz * deg; z0 < (iz + 1) * deg; ++z0)
      for (int y0 = iy * deg; y0 < (iy + 1) * deg; ++y0)
        for (int x0 = ix * deg; x0 < (ix + 1) * deg; ++x0) {
          const int64_t f = z0 * n2 + (int64_t)y0 * n + x0;
          if (flags && (flags[f] & 4)) masked = true;
          if (!window) {
            const V v = phid[f];
            sr = sr + (double)v.x;
            si = si + (double)v.y;
          }
        }
    if (window)
      out[c] = make_double2(masked ? 0.0 : dv_spa, 0.0);
    else
      // deg^3 is a power of two: multiplying by its reciprocal is the same
      // single rounding as the reference's division
      out[c] = masked ? make_double2(0.0, 0.0) : make_double2(sr * inv_deg3, si * inv_deg3);
  }
}

// |F|^2 per k-site into the bins of |k|^2, F in FP64 (cuFFT) or float-float;
// the sums are scaled on the host
__device__ __forceinline__ double norm2(double2 w) { return w.x * w.x + w.y * w.y; }
__device__ __forceinline__ F2 norm2(float4 w) {
  const F2 r = {w.x, w.y}, i = {w.z, w.w};
  return f2_dot2(r, r, i, i, 1.f);
}
// times s (FP64: 1), and in FP64 for sites that fail squares_fit
__device__ __forceinline__ double norm2(double2 w, float) { return norm2(w); }
__device__ __forceinline__ F2 norm2(float4 w, float s) {
  return norm2(make_float4(s * w.x, s * w.y, s * w.z, s * w.w));
}
__device__ __forceinline__ double norm2_wide(double2 w, float) { return norm2(w); }
__device__ __forceinline__ double norm2_wide(float4 w, float s) {
  return norm2(make_double2(((double)w.x + (double)w.y) * (double)s, ((double)w.z + (double)w.w) * (double)s));
}
// the sample of a block: the first sites of rows 0, 1, ... of the plane kz = 0
__device__ __forceinline__ SquareScale field_scale(const double2 *, int) { return SquareScale(); }
__device__ __forceinline__ SquareScale field_scale(const float4 *__restrict__ F, int m) {
  const float4 w = F[min((int)(threadIdx.x >> 5), m - 1) * m + min((int)(threadIdx.x & 31), m - 1)];
  return SquareScale(fmaxf(fabsf(w.x), fabsf(w.z)));
}
template <typename V>
__global__ void __launch_bounds__(256) k_spec_bin(const V *__restrict__ F, int m, int rows,
                                                  const int16_t *__restrict__ tab, int nb, int copies,
                                                  double *__restrict__ conv, double *__restrict__ count) {
  BlockBins bins(bins_mem(), nb, copies);
  const SquareScale scale = field_scale(F, m);
  BinRun<decltype(norm2(F[0]))> run;
  walk_spectrum(m, m, rows, [&](int ix, int iy, int iz) {
    const int kx = kint(ix, m), ky = kint(iy, m), kz = kint(iz, m);
    const int b = tab[kx * kx + ky * ky + kz * kz];
    if (b < 0) return;
    const V f = F[((int64_t)iz * m + iy) * m + ix];
    const auto v = norm2(f, scale.s);
    if (squares_fit(v)) run.add(bins, b, v, 1u);
    else bins.add(b, norm2_wide(f, scale.s), 1u);
  });
  run.flush(bins);
  bins.finish(conv, count, scale.inv);
}

// the real window of compute_matrix_deconv over its dx^3: 1 on unmasked coarse
// cells (the pair sums take dx^6 on the host)
__global__ void k_spec_window(const int8_t *__restrict__ flags, int n, int deg, double *__restrict__ out) {
  const int m = n / deg;
  const int64_t m3 = (int64_t)m * m * m, n2 = (int64_t)n * n;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < m3; c += stride) {
    const int ix = (int)(c % m), iy = (int)((c / m) % m), iz = (int)(c / ((int64_t)m * m));
    bool masked = false;
    if (flags)
      for (int z0 = iz * deg; z0 < (iz + 1) * deg && !masked; ++z0)
        for (int y0 = iy * deg; y0 < (iy + 1) * deg && !masked; ++y0)
          for (int x0 = ix * deg; x0 < (ix + 1) * deg; ++x0)
            if (flags[z0 * n2 + (int64_t)y0 * n + x0] & 4) {
              masked = true;
              break;
            }
    out[c] = masked ? 0.0 : 1.0;
  }
}

// |W|^2 per integer |k|^2 from the half spectrum of the real window
// (|W(-k)| = |W(k)|: interior kx planes count twice).  W is the transform of
// ones and zeros: at most m^3, and below 2^-48 of that it is its own rounding,
// so float-float squares have the range for it.
template <typename V>
__global__ void k_spec_w2_hist(const V *__restrict__ W, int m, int rows, double *__restrict__ h) {
  const int mh = m / 2 + 1;
  walk_spectrum(m, mh, rows, [&](int ix, int iy, int iz) {
    const int kx = kint(ix, m), ky = kint(iy, m), kz = kint(iz, m);
    auto v = norm2(W[((int64_t)iz * m + iy) * mh + ix]);
    if (ix != 0 && 2 * ix != m) v = run_sum(v, v);
    atomicAdd(&h[kx * kx + ky * ky + kz * kz], run_value(v));
  });
}

// The window matrix of bin pair ij (spectrum.f90:385-428) is the sum over all
// k of |W(k)|^2 u_ij(|k|), divided by the sum of u_ij alone, with u_ij linear
// between the 501 nodes of its table.  Regrouped by |k|^2 and then by table
// cell: with the prefix sums of |W|^2 and of |W|^2 |k|, a cell [q_a, q_a + dq)
// adds
//   tab_a (S0 - D) + tab_(a+1) D,  S0 = sum h,  D = (sum h q - S0 q_a) / dq
// from two prefix differences.  The sums are double-double (T. J. Dekker,
// Numer. Math. 18 (1971) 224): S0 q_a cancels sum h q to a few thousandths.
// 1275 pairs x 500 cells instead of 1275 pairs x every |k|^2, ~14 FP64
// operations each on a pipe at 1/64 of the FP32 rate: 870 -> 154 us at 256^3
// with the scans, 3.4 ms -> 270 us at 512^3.  The sums of u_ij alone (h = the
// number of modes) belong to the lattice and are formed once.
struct DD {
  double h, l;
};
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  const double s = AXD_ADD(a.h, b.h), v = AXD_SUB(s, a.h);
  double e = AXD_ADD(AXD_SUB(a.h, AXD_SUB(s, v)), AXD_SUB(b.h, v));
  e = AXD_ADD(e, AXD_ADD(a.l, b.l));
  const double h = AXD_ADD(s, e);
  return {h, AXD_SUB(e, AXD_SUB(h, s))};
}
__device__ __forceinline__ DD dd_sub(DD a, DD b) { return dd_add(a, DD{-b.h, -b.l}); }
__device__ __forceinline__ DD dd_prod(double a, double b) {
  const double p = AXD_MUL(a, b);
  return {p, AXD_FMA(a, b, -p)};
}
struct Sums {
  DD h, hq;
};
__device__ __forceinline__ Sums sums_add(Sums a, Sums b) { return {dd_add(a.h, b.h), dd_add(a.hq, b.hq)}; }
__device__ __forceinline__ Sums sums_shfl(Sums a, int lane) {
  auto f = [lane](double x) { return __shfl_sync(0xffffffffu, x, lane); };
  return {{f(a.h.h), f(a.h.l)}, {f(a.hq.h), f(a.hq.l)}};
}
// inclusive scan over the lanes of a warp
__device__ __forceinline__ Sums warp_scan(Sums x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Sums y = sums_shfl(x, lane >= o ? lane - o : 0);
    if (lane >= o) x = sums_add(y, x);
  }
  return x;
}
constexpr int kScan = 128;  // |k|^2 values per CTA of the scan, a chunk

// q = |k| = sqrt(iq2) dwav; pre[iq2 + 1]: the sums of iq2's chunk up to and
// with iq2; tot[chunk]: the chunk's
__global__ void __launch_bounds__(kScan) k_spec_scan(const double *__restrict__ h, int64_t count, double dwav,
                                                     Sums *__restrict__ pre, Sums *__restrict__ tot) {
  const int64_t i = (int64_t)blockIdx.x * kScan + threadIdx.x;
  Sums x{};
  if (i < count) {
    x.h = {h[i], 0.0};
    x.hq = dd_prod(h[i], AXD_MUL(sqrt((double)i), dwav));
  }
  x = warp_scan(x);
  __shared__ Sums warp[kScan / 32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 31) warp[w] = x;
  __syncthreads();
  Sums before{};
  for (int k = 0; k < w; ++k) before = sums_add(before, warp[k]);
  if (w > 0) x = sums_add(before, x);
  if (i < count) pre[i + 1] = x;
  if (threadIdx.x == kScan - 1) tot[blockIdx.x] = x;
}

// the chunks' totals into the sums before each chunk: one warp, each lane a
// run of chunks (more warps would only queue for one SM's FP64 pipe)
__global__ void k_spec_scan_chunks(Sums *__restrict__ tot, int chunks) {
  const int lane = threadIdx.x, per = (chunks + 31) / 32, c0 = min(lane * per, chunks), c1 = min(c0 + per, chunks);
  Sums run{};
  for (int c = c0; c < c1; ++c) run = sums_add(run, tot[c]);
  Sums before = sums_shfl(warp_scan(run), lane > 0 ? lane - 1 : 0);
  if (lane == 0) before = Sums{};
  for (int c = c0; c < c1; ++c) {
    const Sums own = tot[c];
    tot[c] = before;
    before = sums_add(before, own);
  }
}

__global__ void __launch_bounds__(kScan) k_spec_scan_add(Sums *__restrict__ pre, const Sums *__restrict__ before,
                                                         int64_t count) {
  const int64_t i = (int64_t)blockIdx.x * kScan + threadIdx.x;
  if (i < count) pre[i + 1] = sums_add(before[blockIdx.x], pre[i + 1]);
  if (i == 0) pre[0] = Sums{};
}

// pre[k]: the sums over |k|^2 < k.  One CTA per bin pair, thread a the first
// |k|^2 of table cell a (a = 500: the end) and the sums up to it.
constexpr int kMatThreads = 512;
static_assert(kMatThreads > kNumLargeq, "a thread per node of the table");
__global__ void __launch_bounds__(kMatThreads) k_spec_mat(const Sums *__restrict__ pre,
                                                          const double *__restrict__ mat_spec,
                                                          const double *__restrict__ largeq0,
                                                          const double *__restrict__ dq_spec,
                                                          const long long *__restrict__ range, double dwav,
                                                          double *__restrict__ out) {
  const int ij = blockIdx.x, a = threadIdx.x, lane = a & 31;
  const long long lo = range[2 * ij], hi = range[2 * ij + 1];
  const double *tab = mat_spec + (int64_t)ij * (kNumLargeq + 1);
  const double lq0 = largeq0[ij], dq = dq_spec[ij], idq = 1.0 / dq, iw = 1.0 / dwav;
  auto first = [&](int c) -> long long {  // within [lo, hi + 1]
    if (c == 0 || hi < lo) return lo;
    if (c >= kNumLargeq) return hi + 1;
    const double e = (lq0 + dq * c) * iw;
    const long long k = (long long)ceil(e * e);
    return k < lo ? lo : (k > hi + 1 ? hi + 1 : k);
  };
  const long long k0 = first(a);
  const Sums p0 = pre[k0];
  long long k1 = __shfl_down_sync(0xffffffffu, k0, 1);
  Sums p1 = sums_shfl(p0, lane < 31 ? lane + 1 : 31);
  if (lane == 31) {
    k1 = first(a + 1);
    p1 = pre[k1];
  }
  double v = 0.0;
  if (a < kNumLargeq && k1 > k0) {
    const double qa = lq0 + dq * a;
    const DD s0 = dd_sub(p1.h, p0.h);
    DD sq = dd_prod(s0.h, qa);
    sq.l = AXD_FMA(s0.l, qa, sq.l);
    const double D = dd_sub(dd_sub(p1.hq, p0.hq), sq).h * idq;
    v = tab[a] * (s0.h - D) + tab[a + 1] * D;
  }
  __shared__ double sum[kMatThreads / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) sum[a >> 5] = v;
  __syncthreads();
  if (a == 0) {
    for (int w = 1; w < kMatThreads / 32; ++w) v += sum[w];
    out[ij] = v;
  }
}

// modes per integer |k|^2
__global__ void k_spec_modes(int m, double *__restrict__ cnt) {
  const int mh = m / 2 + 1;
  const int64_t nhalf = (int64_t)m * m * mh;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nhalf; s += stride) {
    const int ix = (int)(s % mh), iy = (int)((s / mh) % m), iz = (int)(s / ((int64_t)mh * m));
    const int kx = kint(ix, m), ky = kint(iy, m), kz = kint(iz, m);
    atomicAdd(&cnt[kx * kx + ky * ky + kz * kz], (ix == 0 || 2 * ix == m) ? 1.0 : 2.0);
  }
}

// spectrum.f90:117-171, every operation rounded once in the reference's order
__device__ double integrate_p_check(int num, double li, double si, double lj, double sj, double q) {
  const double qli = AXD_ADD(q, li);
  const double maxp = lj < qli ? lj : qli;
  const double a = AXD_SUB(q, li), b = AXD_SUB(si, q);
  double minp = a > b ? a : b;
  minp = minp > sj ? minp : sj;
  const double dp = AXD_DIV(AXD_SUB(maxp, minp), (double)num);
  double x = 0.0;
  if (dp > 0) {
    const double qq = AXD_MUL(q, q), l2 = AXD_MUL(li, li), s2 = AXD_MUL(si, si);
    for (int ip = 1; ip <= num; ++ip) {
      const double p = AXD_ADD(AXD_MUL(dp, ip - 0.5), minp);
      double maxmu = 1.0, minmu = -1.0;
      if (q != 0.0) {
        const double pp = AXD_MUL(p, p);
        maxmu = AXD_DIV(AXD_DIV(AXD_MUL(AXD_SUB(AXD_SUB(l2, pp), qq), 0.5), p), q);
        minmu = AXD_DIV(AXD_DIV(AXD_MUL(AXD_SUB(AXD_SUB(s2, pp), qq), 0.5), p), q);
        maxmu = maxmu < 1.0 ? maxmu : 1.0;
        minmu = minmu > -1.0 ? minmu : -1.0;
      }
      x = AXD_ADD(x, AXD_MUL(AXD_MUL(AXD_MUL(p, p), dp), AXD_SUB(maxmu, minmu)));
    }
  }
  return AXD_MUL(x, kRefTwoPi);
}

// mat_spec(0:500, ij) (spectrum.f90:74-98): the 200-point quadrature of every
// table node, a node per thread.  On one host thread it was most of a
// context's first spectrum: 530 ms for 50 bins.
__global__ void k_spec_table(int num_cov, const double *__restrict__ wav, const double *__restrict__ largeq0,
                             const double *__restrict__ dq_spec, double *__restrict__ mat_spec) {
  const int ij = blockIdx.x + 1;
  int i = (int)lround(sqrt(2.0 * ij));
  const int j = ij - i * (i - 1) / 2;
  for (int iq = threadIdx.x; iq <= kNumLargeq; iq += blockDim.x)
    mat_spec[(int64_t)(ij - 1) * (kNumLargeq + 1) + iq] =
        integrate_p_check(kNumInt, wav[i], wav[i - 1], wav[j], wav[j - 1],
                          AXD_ADD(largeq0[ij - 1], AXD_MUL(dq_spec[ij - 1], (double)iq)));
}

// reference LAPACK dpptrf + dpptri ('U'), packed upper
int pp_inverse(int n, double *ap) {
  int jj = 0;
  for (int j = 1; j <= n; ++j) {
    int jc = jj + 1;
    jj = jj + j;
    if (j > 1) {
      double *x = ap + (jc - 1);
      int kk = 1;
      for (int jx = 1; jx <= j - 1; ++jx) {
        double temp = x[jx - 1];
        int k = kk;
        for (int i = 1; i <= jx - 1; ++i) {
          temp = temp - ap[k - 1] * x[i - 1];
          ++k;
        }
        temp = temp / ap[kk + jx - 2];
        x[jx - 1] = temp;
        kk = kk + jx;
      }
    }
    double dot = 0.0;
    for (int i = 0; i < j - 1; ++i) dot = dot + ap[jc - 1 + i] * ap[jc - 1 + i];
    double ajj = ap[jj - 1] - dot;
    if (ajj <= 0.0) {
      ap[jj - 1] = ajj;
      return j;
    }
    ap[jj - 1] = std::sqrt(ajj);
  }
  int jc = 1;
  for (int j = 1; j <= n; ++j) {
    ap[jc + j - 2] = 1.0 / ap[jc + j - 2];
    double ajj = -ap[jc + j - 2];
    double *x = ap + (jc - 1);
    int kk = 1;
    for (int jx = 1; jx <= j - 1; ++jx) {
      if (x[jx - 1] != 0.0) {
        double temp = x[jx - 1];
        int k = kk;
        for (int i = 1; i <= jx - 1; ++i) {
          x[i - 1] = x[i - 1] + temp * ap[k - 1];
          ++k;
        }
        x[jx - 1] = x[jx - 1] * ap[kk + jx - 2];
      }
      kk = kk + jx;
    }
    for (int i = 0; i < j - 1; ++i) x[i] = ajj * x[i];
    jc = jc + j;
  }
  jj = 0;
  for (int j = 1; j <= n; ++j) {
    int jc2 = jj + 1;
    jj = jj + j;
    if (j > 1) {
      const double *xv = ap + (jc2 - 1);
      int kk = 0;
      for (int jx = 0; jx < j - 1; ++jx) {
        if (xv[jx] != 0.0) {
          double temp = 1.0 * xv[jx];
          int k = kk;
          for (int i = 0; i <= jx; ++i) {
            ap[k] = ap[k] + xv[i] * temp;
            ++k;
          }
        }
        kk += jx + 1;
      }
    }
    double ajj = ap[jj - 1];
    for (int i = 0; i < j; ++i) ap[jc2 - 1 + i] = ajj * ap[jc2 - 1 + i];
  }
  return 0;
}

// estimate_covmat (spectrum.f90:593-641): Gaussian modes with the measured
// spectrum (Philox stream 16 + iter), sigma per bin of nint(q/dq + 0.5)
__global__ void k_mc_fill(double2 *F, int m, const int16_t *__restrict__ tab, const double *sigma, uint64_t seed,
                          uint32_t iter) {
  const int64_t m3 = (int64_t)m * m * m;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < m3; s += stride) {
    const int kx = kint(s % m, m), ky = kint((s / m) % m, m), kz = kint(s / ((int64_t)m * m), m);
    const int b = tab[kx * kx + ky * ky + kz * kz];
    if (b >= 0) {
      const axd_u32x4 r = axd_draw(seed, 16u + iter, 0u, (uint64_t)s);
      const double u1 = axd_u01_open0(r.v[0], r.v[1]), u2 = axd_u01(r.v[2], r.v[3]);
      const double rad = sqrt(-2.0 * log(u1));
      double sn, cs;
      sincos(6.283185307179586 * u2, &sn, &cs);
      const double sg = sigma[b];
      F[s] = make_double2(rad * cs * sg, rad * sn * sg);
    } else {
      F[s] = make_double2(0.0, 0.0);
    }
  }
}

// masking (spectrum.f90:648): zero coarse cells holding a masked fine cell
__global__ void k_mc_mask(double2 *F, const int8_t *__restrict__ flags, int n, int deg) {
  const int m = n / deg;
  const int64_t m3 = (int64_t)m * m * m, n2 = (int64_t)n * n;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < m3; c += stride) {
    const int ix = (int)(c % m), iy = (int)((c / m) % m), iz = (int)(c / ((int64_t)m * m));
    bool masked = false;
    for (int z0 = iz * deg; z0 < (iz + 1) * deg && !masked; ++z0)
      for (int y0 = iy * deg; y0 < (iy + 1) * deg && !masked; ++y0)
        for (int x0 = ix * deg; x0 < (ix + 1) * deg; ++x0)
          if (flags[z0 * n2 + (int64_t)y0 * n + x0] & 4) {
            masked = true;
            break;
          }
    if (masked) F[c] = make_double2(0.0, 0.0);
  }
}

// The pair sums from the histogram itself, for few |k|^2 (window_sums): a thread
// per |k|^2 of the pair's range, |k| from a table of q[k] = sqrt(k) dwav.
__global__ void k_spec_q(int64_t iq2max, double dwav, double *__restrict__ q) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k <= iq2max; k += (int64_t)gridDim.x * blockDim.x)
    q[k] = sqrt((double)k) * dwav;
}
__global__ void __launch_bounds__(256) k_spec_mat_direct(const double *__restrict__ h, const double *__restrict__ q,
                                                         const double *__restrict__ mat_spec,
                                                         const double *__restrict__ largeq0,
                                                         const double *__restrict__ dq_spec,
                                                         const long long *__restrict__ range,
                                                         double *__restrict__ out) {
  const int ij = blockIdx.x;
  const int lo = (int)range[2 * ij], hi = (int)range[2 * ij + 1];
  const double *tab = mat_spec + (int64_t)ij * (kNumLargeq + 1);
  const double lq0 = largeq0[ij], idq = 1.0 / dq_spec[ij];
  double v = 0.0;
  for (int k = lo + (int)threadIdx.x; k <= hi; k += 256) {
    const double c = h[k];
    if (c == 0.0) continue;
    const double d = (q[k] - lq0) * idq;
    const int a = (int)floor(d);
    if (a < 0 || a >= kNumLargeq) continue;
    const double t0 = tab[a];
    v += c * (t0 + (d - a) * (tab[a + 1] - t0));
  }
  __shared__ double sum[8];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sum[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) v += sum[w];
    out[ij] = v;
  }
}

int grid_for(int64_t count) {
  int64_t b = (count + 255) / 256;
  if (b > 152 * 16) b = 152 * 16;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace

namespace {
// scratch of window_sums for |k|^2 <= iq2max, in Sums
size_t window_sums_scratch(int64_t iq2max) { return (size_t)(iq2max + 2) + (size_t)((iq2max + kScan) / kScan); }

constexpr int64_t kDirectSums = 3 * 52 * 52;  // |k|^2 below this: m < 104

// out[ij] = sum over |k|^2 of h u_ij(|k|) for every bin pair
int window_sums(axg_ctx *ctx, const double *h, int64_t iq2max, double dwav, Sums *scratch, double *out) {
  const int nb = ctx->p.num_bin, num_cov = nb * (nb + 1) / 2;
  const int chunks = (int)((iq2max + kScan) / kScan);
  Sums *pre = scratch, *tot = scratch + iq2max + 2;
  // The prefix sums' cost is the 501 nodes of each pair's table, 91 us for 50
  // bins at any m and 30 for the scans; the direct sums' the |k|^2 of its range:
  // 34 us at m = 48, 47 at 64, 68 at 80, 73 at 84 and growing by 6 every 4.
  if (iq2max < kDirectSums) {
    double *q = reinterpret_cast<double *>(pre);
    AXG_LAUNCH(ctx, "spec_q", k_spec_q, grid_for(iq2max + 1), 256, 0, iq2max, dwav, q);
    AXG_LAUNCH(ctx, "spec_mat_direct", k_spec_mat_direct, num_cov, 256, 0, h, q, ctx->spec_mat, ctx->spec_largeq0,
               ctx->spec_dq, ctx->spec_range, out);
    return AXG_OK;
  }
  AXG_LAUNCH(ctx, "spec_scan", k_spec_scan, chunks, kScan, 0, h, iq2max + 1, dwav, pre, tot);
  AXG_LAUNCH(ctx, "spec_scan_chunks", k_spec_scan_chunks, 1, 32, 0, tot, chunks);
  AXG_LAUNCH(ctx, "spec_scan_add", k_spec_scan_add, chunks, kScan, 0, pre, tot, iq2max + 1);
  AXG_LAUNCH(ctx, "spec_mat", k_spec_mat, num_cov, kMatThreads, 0, pre, ctx->spec_mat, ctx->spec_largeq0, ctx->spec_dq,
             ctx->spec_range, dwav, out);
  return AXG_OK;
}
}  // namespace

// init_spectrum (spectrum.f90:23-103): bin pairs on the host, tables on the device
int axg_spec_init(axg_ctx *ctx) {
  if (ctx->spec_ready) return AXG_OK;
  // an attempt that fails leaves nothing behind, so that the next one starts again
  auto undo = axg_on_exit([&] {
    if (ctx->spec_ready) return;
    for (void **q : {(void **)&ctx->spec_mat, (void **)&ctx->spec_largeq0, (void **)&ctx->spec_dq,
                     (void **)&ctx->spec_range, (void **)&ctx->spec_modes, (void **)&ctx->spec_buf})
      axg_free(ctx, q);
    if (ctx->plan_spec_ok) cufftDestroy(ctx->plan_spec);
    if (ctx->plan_window_ok) cufftDestroy(ctx->plan_window);
    ctx->plan_spec_ok = ctx->plan_window_ok = false;
  });
  const int nb = ctx->p.num_bin;
  const int num_cov = nb * (nb + 1) / 2;
  const int deg = 1 << ctx->p.degrade_spec;
  const int m = (int)(ctx->n / deg);
  const double dspa_spec = ctx->p.dspa * deg;
  std::vector<double> &wav = ctx->h_wav;
  wav.assign(nb + 1, 0.0);
  const double qmax = kRefPi / dspa_spec;
  const double dq = qmax / nb;
  for (int iq = 1; iq <= nb; ++iq) wav[iq] = wav[iq - 1] + dq;
  const double dwav = kRefTwoPi / dspa_spec / m;
  const int64_t iq2max = 3LL * (m / 2) * (m / 2);
  std::vector<double> l0(num_cov), hdq(num_cov);
  std::vector<long long> hr(2 * (size_t)num_cov);  // the |k|^2 inside each pair's table
  for (int ij = 1; ij <= num_cov; ++ij) {
    int i = (int)std::lround(std::sqrt(2.0 * ij));
    int j = ij - i * (i - 1) / 2;
    double lj = wav[j], sj = wav[j - 1], li = wav[i], si = wav[i - 1];
    double maxq = li + lj;
    double minq = (si > sj ? si : sj) - (li < lj ? li : lj);
    if (minq < 0) minq = 0.0;
    double d = maxq - minq;
    d = d / kNumLargeq;
    hdq[ij - 1] = d;
    l0[ij - 1] = minq;
    double e = (minq + d * kNumLargeq) / dwav;
    long long imax2 = (long long)std::ceil(e * e) - 1;
    e = minq / dwav;
    long long imin2 = (long long)std::ceil(e * e);
    hr[2 * (ij - 1)] = std::max(imin2, 0LL);
    hr[2 * (ij - 1) + 1] = std::min(imax2, (long long)iq2max);
  }
  AXG_TRY(axg_alloc(ctx, (void **)&ctx->spec_mat, (size_t)num_cov * (kNumLargeq + 1) * 8, "mat_spec"));
  AXG_TRY(axg_alloc(ctx, (void **)&ctx->spec_largeq0, (size_t)num_cov * 8, "largeq"));
  AXG_TRY(axg_alloc(ctx, (void **)&ctx->spec_dq, (size_t)num_cov * 8, "dq_spec"));
  AXG_TRY(axg_alloc(ctx, (void **)&ctx->spec_range, (size_t)num_cov * 16, "pair ranges"));
  AXG_TRY(axg_alloc(ctx, (void **)&ctx->spec_modes, (size_t)num_cov * 8, "pair mode sums"));
  double *d_wav = nullptr;  // bin edges, then the modes per |k|^2 and the scratch of their sums
  auto cleanup = axg_on_exit([&] {
    cudaStreamSynchronize(ctx->stream);
    axg_free(ctx, (void **)&d_wav);
  });
  const size_t edges = (wav.size() + 1) & ~(size_t)1, modes = ((size_t)iq2max + 2) & ~(size_t)1;
  AXG_TRY(axg_alloc(ctx, (void **)&d_wav, (edges + modes) * 8 + window_sums_scratch(iq2max) * sizeof(Sums),
                    "spectrum tables"));
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(d_wav, wav.data(), wav.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->spec_largeq0, l0.data(), (size_t)num_cov * 8, cudaMemcpyHostToDevice, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->spec_dq, hdq.data(), (size_t)num_cov * 8, cudaMemcpyHostToDevice, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->spec_range, hr.data(), hr.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  AXG_LAUNCH(ctx, "spec_table", k_spec_table, num_cov, 128, 0, num_cov, d_wav, ctx->spec_largeq0, ctx->spec_dq,
             ctx->spec_mat);
  double *cnt = d_wav + edges;
  AXG_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, modes * 8, ctx->stream));
  AXG_LAUNCH(ctx, "spec_modes", k_spec_modes, grid_for((int64_t)m * m * (m / 2 + 1)), 256, 0, m, cnt);
  AXG_TRY(window_sums(ctx, cnt, iq2max, dwav, (Sums *)(cnt + modes), ctx->spec_modes));
  ctx->ns_spec = m;
  // m^3 complex; the window pass uses it as m^3 reals followed by the D2Z
  // half spectrum m^2 (m/2 + 1), which needs 16 m^2 bytes more
  AXG_TRY(axg_alloc(ctx, (void **)&ctx->spec_buf, (size_t)m * m * m * 16 + (size_t)m * m * 16 + 256,
                    "spectrum buffer"));
  AXG_CUFFT_TRY(ctx, cufftPlan3d(&ctx->plan_spec, m, m, m, CUFFT_Z2Z));
  ctx->plan_spec_ok = true;
  AXG_CUFFT_TRY(ctx, cufftSetStream(ctx->plan_spec, ctx->stream));
  AXG_CUFFT_TRY(ctx, cufftPlan3d(&ctx->plan_window, m, m, m, CUFFT_D2Z));
  ctx->plan_window_ok = true;
  AXG_CUFFT_TRY(ctx, cufftSetStream(ctx->plan_window, ctx->stream));
  ctx->spec_ready = true;
  return AXG_OK;
}

int axg_spec_estimation(axg_ctx *ctx, double tau, double *wave, double *power, double *conv,
                        double *count) {
  AXG_TRY(axg_spec_init(ctx));
  if (!ctx->flags_valid) {
    int64_t c[3];
    AXG_TRY(axg_def_classify(ctx, (ctx->p.flags & 7) | AXG_F_SPEC_EST, c));
  }
  const int nb = ctx->p.num_bin;
  const int num_cov = nb * (nb + 1) / 2;
  const int deg = 1 << ctx->p.degrade_spec;
  const int n = (int)ctx->n, m = n / deg;
  const int64_t m3 = (int64_t)m * m * m;
  const double dspa_spec = ctx->p.dspa * deg;
  const double dwav = kRefTwoPi / dspa_spec / m;
  const double dv_spa = dspa_spec * dspa_spec * dspa_spec;
  const double dv_wav = std::pow(dwav / kRefTwoPi, 3);
  const bool fp32 = ctx->p.precision == AXG_PREC_FP32_MIXED;
  const int64_t iq2max = 3LL * (m / 2) * (m / 2);
  // scratch: histogram, pair sums, bin sums, and what window_sums needs
  double *scratch = nullptr;
  const size_t nscr = (((size_t)(iq2max + 1 + num_cov + 2 * nb)) + 1) & ~(size_t)1;
  AXG_TRY(axg_alloc(ctx, (void **)&scratch, nscr * 8 + window_sums_scratch(iq2max) * sizeof(Sums), "spectrum scratch"));
  int rc = AXG_OK;
  do {
    double *h = scratch, *mat0 = h + iq2max + 1, *d_conv = mat0 + num_cov, *d_cnt = d_conv + nb;
    AXG_CUDA_TRY(ctx, cudaMemsetAsync(scratch, 0, nscr * 8, ctx->stream));
    // ---- compute_matrix_deconv (spectrum.f90:344-444) ----
    // the window is real: D2Z half spectrum (|W|^2 is the same for either sign)
    double *wreal = (double *)ctx->spec_buf;
    double2 *whalf = (double2 *)(((uintptr_t)(wreal + m3) + 255) & ~(uintptr_t)255);
    // (our own transforms of an undegraded field read the flags in their row pass)
    const bool ff = axg_ff_use(m), direct = ff && deg == 1;
    const int wrows = walk_rows_single(m, m / 2 + 1), wgrid = walk_grid(m, m / 2 + 1, wrows);
    if (direct) {
      AXG_TRY(axg_ff_d2z_window(ctx, ctx->flags, whalf, m));
    } else {
      AXG_LAUNCH(ctx, "spec_window", k_spec_window, grid_for(m3), 256, 0, ctx->flags, n, deg, wreal);
      if (ff) AXG_TRY(axg_ff_d2z(ctx, wreal, whalf, m, 1, true));
      else AXG_CUFFT_TRY(ctx, cufftExecD2Z(ctx->plan_window, wreal, (cufftDoubleComplex *)whalf));
    }
    if (ff) AXG_LAUNCH(ctx, "spec_w2_hist", k_spec_w2_hist<float4>, wgrid, 256, 0, (const float4 *)whalf, m, wrows, h);
    else AXG_LAUNCH(ctx, "spec_w2_hist", k_spec_w2_hist<double2>, wgrid, 256, 0, whalf, m, wrows, h);
    AXG_TRY(window_sums(ctx, h, iq2max, dwav, (Sums *)(scratch + nscr), mat0));
    // ---- compute_conv_spec (spectrum.f90:466-567) ----
    if (direct) {
      AXG_TRY(axg_ff_z2z_masked(ctx, ctx->phid, fp32, ctx->flags, (double2 *)ctx->spec_buf, m, 1));
    } else {
      if (fp32)
        AXG_LAUNCH(ctx, "spec_degrade", k_spec_degrade<float2>, grid_for(m3), 256, 0, (const float2 *)ctx->phid,
                   ctx->flags, n, deg, 1.0 / ((double)deg * deg * deg), 0, dv_spa, ctx->spec_buf);
      else
        AXG_LAUNCH(ctx, "spec_degrade", k_spec_degrade<double2>, grid_for(m3), 256, 0, (const double2 *)ctx->phid,
                   ctx->flags, n, deg, 1.0 / ((double)deg * deg * deg), 0, dv_spa, ctx->spec_buf);
      if (ff)
        AXG_TRY(axg_ff_z2z(ctx, (double2 *)ctx->spec_buf, m, 1, true));
      else
        AXG_CUFFT_TRY(ctx, cufftExecZ2Z(ctx->plan_spec, (cufftDoubleComplex *)ctx->spec_buf,
                                        (cufftDoubleComplex *)ctx->spec_buf, CUFFT_INVERSE));
    }
    const double dq = ctx->h_wav[1] - ctx->h_wav[0];
    const int16_t *tab = nullptr;
    AXG_TRY(axg_bin_table(ctx, AXG_BIN_SPECTRUM, m, dwav, dq, nb, 0, nullptr, &tab));
    const int brows = walk_rows(m, m), bgrid = walk_grid(m, m, brows);
    if (ff)
      AXG_LAUNCH(ctx, "spec_bin", k_spec_bin<float4>, bgrid, 256, bin_smem(nb),
                 (const float4 *)ctx->spec_buf, m, brows, tab, nb, bin_copies(nb), d_conv, d_cnt);
    else
      AXG_LAUNCH(ctx, "spec_bin", k_spec_bin<double2>, bgrid, 256, bin_smem(nb),
                 (const double2 *)ctx->spec_buf, m, brows, tab, nb, bin_copies(nb), d_conv, d_cnt);
    std::vector<double> hm(2 * num_cov), hb(2 * nb);
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(hm.data(), mat0, (size_t)num_cov * 8, cudaMemcpyDeviceToHost, ctx->stream));
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(hm.data() + num_cov, ctx->spec_modes, (size_t)num_cov * 8, cudaMemcpyDeviceToHost,
                                      ctx->stream));
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(hb.data(), d_conv, hb.size() * 8, cudaMemcpyDeviceToHost, ctx->stream));
    AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    std::vector<double> mat(num_cov);
    for (int ij = 0; ij < num_cov; ++ij)
      mat[ij] = hm[ij] / hm[num_cov + ij] * (dv_spa * dv_spa) * dv_wav * dv_wav;
    if (pp_inverse(nb, mat.data()) != 0) {
      rc = axg_set_error(ctx, AXG_ERR_NUMERIC, "deconvolution matrix not positive definite");
      break;
    }
    // ---- spectrum_estimation (spectrum.f90:267-285) ----
    const double t2 = tau * tau * (dv_spa * dv_spa * dv_wav);  // |F dv_spa|^2 dv_wav tau^2
    std::vector<double> cv(nb), ct(nb), pw(nb, 0.0);
    for (int i = 1; i <= nb; ++i) {
      cv[i - 1] = hb[i - 1] * t2;
      ct[i - 1] = hb[nb + i - 1];
      for (int j = 1; j <= i; ++j) {
        int ij = i * (i - 1) / 2 + j;
        mat[ij - 1] = mat[ij - 1] / hb[nb + i - 1] / hb[nb + j - 1];
      }
    }
    // dspmv ('U')
    int kk = 1;
    for (int j = 1; j <= nb; ++j) {
      double temp1 = cv[j - 1], temp2 = 0.0;
      int k = kk;
      for (int i = 1; i <= j - 1; ++i) {
        pw[i - 1] = pw[i - 1] + temp1 * mat[k - 1];
        temp2 = temp2 + mat[k - 1] * cv[i - 1];
        ++k;
      }
      pw[j - 1] = pw[j - 1] + temp1 * mat[kk + j - 2] + 1.0 * temp2;
      kk = kk + j;
    }
    ctx->last_power = pw;
    ctx->last_mat_div = mat;
    ctx->last_cov.clear();
    for (int i = 0; i < nb; ++i) {
      if (wave) wave[i] = (ctx->h_wav[i + 1] + ctx->h_wav[i]) / 2;
      power[i] = pw[i];
      if (conv) conv[i] = cv[i] / ct[i];
      if (count) count[i] = ct[i];
    }
  } while (0);
  cudaStreamSynchronize(ctx->stream);
  axg_free(ctx, (void **)&scratch);
  return rc;
}

extern "C" {
int axg_spectrum_estimation(axg_ctx *ctx, double tau, double *wave, double *power, double *conv,
                            double *count) {
  if (!ctx || !power) return AXG_ERR_ARG;
  return axg_spec_estimation(ctx, tau, wave, power, conv, count);
}

// compute_crho (spectrum.f90:316-342) without the covariance term
int axg_compute_crho(axg_ctx *ctx, double *rho) {
  if (!ctx || !rho) return AXG_ERR_ARG;
  if (ctx->last_power.empty()) return axg_set_error(ctx, AXG_ERR_STATE, "no spectrum estimated yet");
  const int nb = ctx->p.num_bin;
  double r = 0.0;
  for (int i = 1; i <= nb; ++i) {
    const double q = (ctx->h_wav[i] + ctx->h_wav[i - 1]) / 2;
    const double dq = ctx->h_wav[i] - ctx->h_wav[i - 1];
    const double q2dq = q * q * dq / kRefTwoPi / kRefPi;
    r = r + ctx->last_power[i - 1] * q2dq;
  }
  *rho = r;
  return AXG_OK;
}
}

// estimate_covmat (spectrum.f90:569-734) on the last spectrum estimate
int axg_spec_covariance(axg_ctx *ctx, int min_mc, int max_mc, double tol, double *cov_out, int *iterations) {
  if (ctx->last_power.empty() || ctx->last_mat_div.empty())
    return axg_set_error(ctx, AXG_ERR_STATE, "no spectrum estimated yet");
  if (!ctx->flags_valid) return axg_set_error(ctx, AXG_ERR_STATE, "mask of the last classification is stale");
  const int nb = ctx->p.num_bin;
  const int num_cov = nb * (nb + 1) / 2;
  const int deg = 1 << ctx->p.degrade_spec;
  const int n = (int)ctx->n, m = n / deg;
  const int64_t m3 = (int64_t)m * m * m;
  const double dspa_spec = ctx->p.dspa * deg;
  const double dwav = kRefTwoPi / dspa_spec / m;
  const double dq = ctx->h_wav[1] - ctx->h_wav[0];
  std::vector<double> sigma(nb), cov(num_cov, 0.0), tmp((size_t)num_cov * max_mc, 0.0), pw0(nb), pw(nb);
  for (int i = 0; i < nb; ++i) {
    const double pwr = ctx->last_power[i];
    sigma[i] = std::sqrt(pwr > 0 ? pwr / 2 : 0.0) / (double)m3;
  }
  double *scr = nullptr;
  auto cleanup = axg_on_exit([&] {
    cudaStreamSynchronize(ctx->stream);
    axg_free(ctx, (void **)&scr);
  });
  AXG_TRY(axg_alloc(ctx, (void **)&scr, sizeof(double) * (size_t)(3 * nb), "covariance scratch"));
  int rc = AXG_OK, iter;
  double *d_sigma = scr, *d_pow = scr + nb, *d_cnt = scr + 2 * nb;
  const int16_t *tab = nullptr;
  AXG_TRY(axg_bin_table(ctx, AXG_BIN_SPECTRUM, m, dwav, dq, nb, 0, nullptr, &tab));
  const bool ff = axg_ff_use(m);  // float-float transforms (FP64 accuracy on the FP32 pipes)
  for (iter = 1; iter <= max_mc && rc == AXG_OK; ++iter) {
    if (iter == 1) AXG_CUDA_TRY(ctx, cudaMemcpyAsync(d_sigma, sigma.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, ctx->stream));
    AXG_CUDA_TRY(ctx, cudaMemsetAsync(d_pow, 0, sizeof(double) * 2 * nb, ctx->stream));
    AXG_LAUNCH(ctx, "mc_fill", k_mc_fill, grid_for(m3), 256, 0, ctx->spec_buf, m, tab, d_sigma, (uint64_t)ctx->p.seed,
               (uint32_t)iter);
    if (ff)
      AXG_TRY(axg_ff_z2z(ctx, (double2 *)ctx->spec_buf, m, 0));
    else
      AXG_CUFFT_TRY(ctx, cufftExecZ2Z(ctx->plan_spec, (cufftDoubleComplex *)ctx->spec_buf,
                                      (cufftDoubleComplex *)ctx->spec_buf, CUFFT_FORWARD));
    AXG_LAUNCH(ctx, "mc_mask", k_mc_mask, grid_for(m3), 256, 0, ctx->spec_buf, ctx->flags, n, deg);
    if (ff)
      AXG_TRY(axg_ff_z2z(ctx, (double2 *)ctx->spec_buf, m, 1, true));
    else
      AXG_CUFFT_TRY(ctx, cufftExecZ2Z(ctx->plan_spec, (cufftDoubleComplex *)ctx->spec_buf,
                                      (cufftDoubleComplex *)ctx->spec_buf, CUFFT_INVERSE));
    const int brows = walk_rows(m, m), bgrid = walk_grid(m, m, brows);
    if (ff)
      AXG_LAUNCH(ctx, "mc_bin", k_spec_bin<float4>, bgrid, 256, bin_smem(nb),
                 (const float4 *)ctx->spec_buf, m, brows, tab, nb, bin_copies(nb), d_pow, d_cnt);
    else
      AXG_LAUNCH(ctx, "mc_bin", k_spec_bin<double2>, bgrid, 256, bin_smem(nb),
                 (const double2 *)ctx->spec_buf, m, brows, tab, nb, bin_copies(nb), d_pow, d_cnt);
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(pw0.data(), d_pow, sizeof(double) * nb, cudaMemcpyDeviceToHost, ctx->stream));
    AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    // pow = mat_deconv pow0 - power (dspmv, beta = 1)
    const std::vector<double> &M = ctx->last_mat_div;
    for (int i = 0; i < nb; ++i) pw[i] = -ctx->last_power[i];
    int kk = 1;
    for (int j = 1; j <= nb; ++j) {
      double temp1 = pw0[j - 1], temp2 = 0.0;
      int k = kk;
      for (int i = 1; i <= j - 1; ++i) {
        pw[i - 1] = pw[i - 1] + temp1 * M[k - 1];
        temp2 = temp2 + M[k - 1] * pw0[i - 1];
        ++k;
      }
      pw[j - 1] = pw[j - 1] + temp1 * M[kk + j - 2] + temp2;
      kk = kk + j;
    }
    for (int i = 1; i <= nb; ++i)
      for (int j = 1; j <= i; ++j) {
        const int ij = i * (i - 1) / 2 + j;
        const double u = pw[i - 1] * pw[j - 1];
        tmp[(size_t)(iter - 1) * num_cov + ij - 1] = cov[ij - 1];
        for (int k = 1; k <= iter - 1; ++k) tmp[(size_t)(k - 1) * num_cov + ij - 1] += u;
        cov[ij - 1] = cov[ij - 1] + u;
      }
    if (iter < min_mc) continue;
    // jackknife convergence on the diagonal (spectrum.f90:696-718)
    double diff = 0.0;
    for (int i = 1; i <= nb; ++i) {
      const int ij = i * (i + 1) / 2;
      double u = 0.0, v = 0.0;
      for (int k = 1; k <= iter; ++k) {
        const double x = tmp[(size_t)(k - 1) * num_cov + ij - 1] / (iter - 1);
        u = u + x;
        v = v + x * x;
      }
      u = u / iter;
      v = v / iter;
      v = std::sqrt(v - u * u);
      const double x = cov[ij - 1] / iter;
      const double r = v / x;
      diff = diff > r ? diff : r;
    }
    if (diff < tol) break;
  }
  if (rc != AXG_OK) return rc;
  if (iter > max_mc) iter = max_mc + 1;
  for (int ij = 0; ij < num_cov; ++ij) cov[ij] = cov[ij] / iter;
  ctx->last_cov = cov;
  if (cov_out) std::copy(cov.begin(), cov.end(), cov_out);
  if (iterations) *iterations = iter;
  return AXG_OK;
}

extern "C" {
int axg_spectrum_covariance(axg_ctx *ctx, int min_mc, int max_mc, double tol, double *cov, int *iterations) {
  if (!ctx || min_mc < 2 || max_mc < min_mc || !(tol > 0)) return AXG_ERR_ARG;
  return axg_spec_covariance(ctx, min_mc, max_mc, tol, cov, iterations);
}

// compute_crho (spectrum.f90:316-342) with the covariance term of the last MC run
int axg_compute_crho_cov(axg_ctx *ctx, double *rho, double *drho) {
  if (!ctx || !rho || !drho) return AXG_ERR_ARG;
  if (ctx->last_power.empty() || ctx->last_cov.empty())
    return axg_set_error(ctx, AXG_ERR_STATE, "needs axg_spectrum_estimation and axg_spectrum_covariance first");
  const int nb = ctx->p.num_bin;
  const std::vector<double> &w = ctx->h_wav;
  double r = 0.0, d = 0.0;
  for (int i = 1; i <= nb; ++i) {
    double dd = 0.0;
    for (int j = 1; j <= i; ++j) {
      const int ij = i * (i - 1) / 2 + j;
      const double q = (w[j] + w[j - 1]) / 2, dq = w[j] - w[j - 1];
      double q2dq = q * q * dq / kRefPi / kRefPi;
      if (j == i) q2dq = q2dq / 2;
      dd = dd + ctx->last_cov[ij - 1] * q2dq;
    }
    const double q = (w[i] + w[i - 1]) / 2, dq = w[i] - w[i - 1];
    const double q2dq = q * q * dq / kRefTwoPi / kRefPi;
    d = d + dd * q2dq;
    r = r + ctx->last_power[i - 1] * q2dq;
  }
  *rho = r;
  *drho = std::sqrt(d);
  return AXG_OK;
}

// get_epsilon (spectrum.f90:1002-1036) for one pair of output times
int axg_epsilon(int32_t nb, const double *wav, const double *p1, const double *p2, const double *c1,
                const double *c2, double tau1, double tau2, double *eps, double *deps) {
  if (nb < 1 || !wav || !p1 || !p2 || !c1 || !c2 || !eps || !deps) return AXG_ERR_ARG;
  const double tau = (tau2 + tau1) / 2;
  const double f = tau / 2 / kRefTwoPi;
  double num = 0.0, den = 0.0;
  for (int i = 1; i <= nb; ++i) {
    const double d = p2[i - 1] - p1[i - 1];
    const double q = (wav[i - 1] + wav[i]) / 2;
    num = num + d * q * q;
    den = den + d * q;
  }
  const double e = num / den * f;
  double de = 0.0;
  for (int i = 1; i <= nb; ++i) {
    const double d1 = (wav[i - 1] + wav[i]) / 2;
    for (int j = 1; j <= i; ++j) {
      const int ij = i * (i - 1) / 2 + j;
      const double d2 = (wav[j - 1] + wav[j]) / 2;
      double d = (1 - e / d1 / f) * (1 - e / d2 / f) * (c2[ij - 1] + c1[ij - 1]) * d1 * d1 * d2 * d2;
      if (j != i) d = d * 2;
      de = de + d;
    }
  }
  *eps = e;
  *deps = std::sqrt(de / den / den) * f;
  return AXG_OK;
}
}
