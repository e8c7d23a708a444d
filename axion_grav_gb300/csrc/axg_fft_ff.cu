// axg_fft_ff.cu -- 3-D FFTs at FP64 accuracy in float-float arithmetic, and
// the FP32 transform of the Green's-function sources.
//
// GB300 issues FP64 at 1/64 of its FP32 rate, and an FP64 FFT is bound by
// it: cuFFT's 512^3 D2Z takes about 15.5 ms, while moving its bytes takes
// about 1 ms.  Here every value is a float-float pair (axg_ff.h) and the
// butterflies run on the FP32 pipes; complex twiddle products are two f2_dot2
// terms.  The input doubles are split into float-float on load and the
// output is hi + lo in double (or stays float-float for a consumer that
// reads it so), so the transform agrees with an FP64 FFT to about 1e-13 of
// the spectrum's largest value.
//
// Layout and convention are cuFFT's: batched D2Z, in [batch][n][n][n] reals,
// out [batch][n][n][n/2+1] complex, forward (exp(-2 pi i k x / n)),
// unnormalised; and in-place Z2Z of one [n][n][n] volume in either
// direction (the complex row pass replaces the real one).  Three passes,
// each one read and one write of the spectrum (the output buffer holds the
// float-float intermediate):
//   rows    : per x-row, the n reals as n/2 complex points z[m] = x[2m] +
//             i x[2m+1], an n/2-point FFT, and the split of Z into the n/2+1
//             outputs X[k] = E[k] + W_n^k O[k];
//   y, z    : n-point FFTs along y and along z, a few adjacent kx columns per
//             CTA so every row of the tile is one 64-byte segment.
// The complex-float transforms (FP32-mixed Green sources and u_ij fields)
// store their half spectra with padded kx rows (axg_f32_spec_pitch); their y
// pass moves its tiles by TMA (k_cols_tma), and the z pass hands its outputs to
// what reads them, the TT power's shell sums or the Green accumulation, instead
// of storing them (k_z_sink).
// Each line is a Stockham radix-8 FFT in registers (f_stockham): a 512-point
// line takes two shared-memory exchanges, the first pass reads its inputs
// from global memory and the column passes' last pass writes there.
// Twiddles W_n^k come from a float-float table made on the host in FP64.
// Powers of two from 16 to 512.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "axg_binning.h"
#include "axg_ff.h"
#include "axg_gw_site.h"
#include "axg_gw_source.h"
#include "axg_internal.h"
#include "axg_soft64.h"
#include "axg_tma.h"

namespace {

// complex float-float in a float4: (re.h, re.l, im.h, im.l)
__device__ __forceinline__ F2 re(float4 v) { return {v.x, v.y}; }
__device__ __forceinline__ F2 im(float4 v) { return {v.z, v.w}; }
__device__ __forceinline__ float4 cx(F2 r, F2 i) { return make_float4(r.h, r.l, i.h, i.l); }

// Complex arithmetic of the two value types the transforms run in: complex
// float (float2) and complex float-float (float4).
__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 c_mul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 c_conj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 c_half(float2 a) { return make_float2(0.5f * a.x, 0.5f * a.y); }
__device__ __forceinline__ float2 c_div_2i(float2 d) { return make_float2(0.5f * d.y, -0.5f * d.x); }  // d / 2i

__device__ __forceinline__ float4 c_add(float4 a, float4 b) { return cx(f2_add(re(a), re(b)), f2_add(im(a), im(b))); }
__device__ __forceinline__ float4 c_sub(float4 a, float4 b) { return cx(f2_sub(re(a), re(b)), f2_sub(im(a), im(b))); }
__device__ __forceinline__ float4 c_mul(float4 a, float4 b) {
  return cx(f2_dot2(re(a), re(b), im(a), im(b), -1.f), f2_dot2(re(a), im(b), im(a), re(b), 1.f));
}
__device__ __forceinline__ float4 c_conj(float4 a) { return make_float4(a.x, a.y, -a.z, -a.w); }
__device__ __forceinline__ float4 c_neg(float4 a) { return make_float4(-a.x, -a.y, -a.z, -a.w); }
__device__ __forceinline__ float4 c_half(float4 a) { return cx(f2_half(re(a)), f2_half(im(a))); }  // exact
__device__ __forceinline__ float4 c_div_2i(float4 d) { return cx(f2_half(im(d)), f2_neg(f2_half(re(d)))); }

// a W_4 = a (-i), inverse a (+i): exact
template <bool INV>
__device__ __forceinline__ float2 c_w4(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template <bool INV>
__device__ __forceinline__ float4 c_w4(float4 a) {
  return INV ? make_float4(-a.z, -a.w, a.x, a.y) : make_float4(a.z, a.w, -a.x, -a.y);
}

// a W_8 = a (1 -+ i) / sqrt 2 and a W_8^3 = a (-1 -+ i) / sqrt 2 (the upper
// sign forward); 1 / sqrt 2 as a float and as a float-float pair
constexpr float kRs2 = 0.70710678118654752440f;
constexpr float kRs2Hi = 0.70710676908493041992f, kRs2Lo = 1.2101617485882343e-08f;
template <bool INV>
__device__ __forceinline__ float2 c_w8(float2 a) {
  return INV ? make_float2((a.x - a.y) * kRs2, (a.x + a.y) * kRs2) : make_float2((a.x + a.y) * kRs2, (a.y - a.x) * kRs2);
}
template <bool INV>
__device__ __forceinline__ float2 c_w8_3(float2 a) {
  return INV ? make_float2((-a.x - a.y) * kRs2, (a.x - a.y) * kRs2)
             : make_float2((a.y - a.x) * kRs2, (-a.x - a.y) * kRs2);
}
template <bool INV>
__device__ __forceinline__ float4 c_w8(float4 a) {
  const F2 r = re(a), i = im(a), s = {kRs2Hi, kRs2Lo};
  return INV ? cx(f2_mul(f2_sub(r, i), s), f2_mul(f2_add(r, i), s)) : cx(f2_mul(f2_add(r, i), s), f2_mul(f2_sub(i, r), s));
}
template <bool INV>
__device__ __forceinline__ float4 c_w8_3(float4 a) {
  const F2 r = re(a), i = im(a), s = {kRs2Hi, kRs2Lo};
  return INV ? cx(f2_neg(f2_mul(f2_add(r, i), s)), f2_mul(f2_sub(r, i), s))
             : cx(f2_mul(f2_sub(i, r), s), f2_neg(f2_mul(f2_add(r, i), s)));
}

template <typename T>
__device__ __forceinline__ T c_zero() {
  T z;
  if constexpr (sizeof(T) == 8) z = make_float2(0.f, 0.f);
  else z = make_float4(0.f, 0.f, 0.f, 0.f);
  return z;
}

// a complex float-float from two doubles (re, im), split on the integer pipes
// (zeros, common in masked fields, past the FP64 conversions): by conversions, 8
// FP64-pipe operations, the complex row pass was bound by the FP64 pipe, 254 us
// at 256^3
__device__ __forceinline__ F2 f2_split(double x) {
  if ((__double_as_longlong(x) << 1) == 0) return F2{0.f, 0.f};
  F2 v;
  return axs_split(x, &v.h, &v.l) ? v : f2_from(x);
}
__device__ __forceinline__ float4 c_from(double2 x) { return cx(f2_split(x.x), f2_split(x.y)); }

// In-register DFTs of 2, 4 and 8 points, natural order in and out; INV uses
// exp(+2 pi i / R).  The 8-point one is two 4-point DFTs of the even and odd
// inputs joined with W_8^k.
template <bool INV, typename T>
__device__ __forceinline__ void c_dft4(T &x0, T &x1, T &x2, T &x3) {
  const T a = c_add(x0, x2), b = c_sub(x0, x2), c = c_add(x1, x3), d = c_w4<INV>(c_sub(x1, x3));
  x0 = c_add(a, c);
  x1 = c_add(b, d);
  x2 = c_sub(a, c);
  x3 = c_sub(b, d);
}
template <int R, bool INV, typename T>
__device__ __forceinline__ void c_dft(T *v) {
  if constexpr (R == 2) {
    const T t = v[0];
    v[0] = c_add(t, v[1]);
    v[1] = c_sub(t, v[1]);
  } else if constexpr (R == 4) {
    c_dft4<INV>(v[0], v[1], v[2], v[3]);
  } else {
    T e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    c_dft4<INV>(e0, e1, e2, e3);
    c_dft4<INV>(o0, o1, o2, o3);
    o1 = c_w8<INV>(o1);
    o2 = c_w4<INV>(o2);
    o3 = c_w8_3<INV>(o3);
    v[0] = c_add(e0, o0);
    v[4] = c_sub(e0, o0);
    v[1] = c_add(e1, o1);
    v[5] = c_sub(e1, o1);
    v[2] = c_add(e2, o2);
    v[6] = c_sub(e2, o2);
    v[3] = c_add(e3, o3);
    v[7] = c_sub(e3, o3);
  }
}

// Stockham autosort FFT of L points, L / 8 threads per line, 8 values per
// thread in registers.  Pass (R, NS), NS the product of the earlier radices:
// iteration jj < L / R reads x[jj + r L / R], multiplies input r by
// W_(NS R)^(r (jj mod NS)), takes the R-point DFT and writes output r to
// (jj / NS) NS R + jj mod NS + r NS.  Radix 8 while 8 divides what is left,
// then one radix-4 or radix-2 pass; a thread runs 8 / R iterations per pass.
// Input and output are in natural order.  Between passes the values go
// through shared memory, element i of the line at line[pad(i) * ls]
// (pad(i) = i + i / 8 keeps the radix-8 strides off a single bank); the last
// pass hands its outputs to `store`.  tw[k] = W_(L ts)^k, k < L ts.
__device__ __forceinline__ int fpad(int i) { return i + (i >> 3); }

// Unpadded lines of 8-byte (complex float) elements, element i at fswz(i):
// the low four bits, the element's bank pair within 128 bytes, XORed with
// bits 3..6.  Aligned runs of 16 elements (a half warp's 8-byte request) keep
// 16 distinct bank pairs, and so do the passes' stride-8 and stride-64
// writes.  With 8-byte elements the i + i / 8 padding made every consecutive
// read and write two-way conflicted; with 16-byte elements (float-float,
// 8 lanes per request) it is conflict-free and stays.
__device__ __forceinline__ int fswz(int i) { return i ^ ((i >> 3) & 15); }
template <bool SW>
__device__ __forceinline__ int fidx(int i) {
  if constexpr (SW) return fswz(i);
  else return fpad(i);
}

template <int L, int NS, bool INV, bool REC = false, bool SW = false, typename T, typename Store>
__device__ __forceinline__ void f_stockham(T v[8], int j, T *line, int ls, const T *tw, int ts, Store store) {
  constexpr int REM = L / NS, R = REM >= 8 ? 8 : REM, NI = 8 / R, TH = L / 8;
#pragma unroll
  for (int q = 0; q < NI; ++q) {
    const int jj = j + q * TH;
    if constexpr (NS > 1) {
      const int k = jj & (NS - 1);
      if constexpr (REC) {
        // one table read; the powers by complex multiplication (REC is for
        // the FP32 transforms).  SW: tw is the per-pass table of
        // load_twc, tw[NS + k] = W_(NS R)^k, read at consecutive k.
        T w1 = SW ? tw[NS + k] : tw[k * (L / (NS * R)) * ts];
        if (INV) w1 = c_conj(w1);
        T w = w1;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          v[q * R + r] = c_mul(v[q * R + r], w);
          w = c_mul(w, w1);
        }
      } else {
#pragma unroll
        for (int r = 1; r < R; ++r) {
          T w = tw[r * k * (L / (NS * R)) * ts];
          if (INV) w = c_conj(w);
          v[q * R + r] = c_mul(v[q * R + r], w);
        }
      }
    }
    c_dft<R, INV>(&v[q * R]);
  }
  if constexpr (NS * R == L) {
#pragma unroll
    for (int q = 0; q < NI; ++q) {
      const int jj = j + q * TH;
#pragma unroll
      for (int r = 0; r < R; ++r) store(jj + r * NS, v[q * R + r]);  // last pass: NS = L / R, jj < NS
    }
  } else {
#pragma unroll
    for (int q = 0; q < NI; ++q) {
      const int jj = j + q * TH, d = (jj / NS) * NS * R + (jj & (NS - 1));
#pragma unroll
      for (int r = 0; r < R; ++r) line[fidx<SW>(d + r * NS) * ls] = v[q * R + r];
    }
    __syncthreads();
    constexpr int NS2 = NS * R, R2 = L / NS2 >= 8 ? 8 : L / NS2;
#pragma unroll
    for (int q = 0; q < 8 / R2; ++q)
#pragma unroll
      for (int r = 0; r < R2; ++r) v[q * R2 + r] = line[fidx<SW>(j + q * TH + r * (L / R2)) * ls];
    __syncthreads();
    f_stockham<L, NS2, INV, REC, SW>(v, j, line, ls, tw, ts, store);
  }
}

// the twiddle table W_L^k, k < L, in shared memory from the first L / 2
// entries of the float-float table (W^(k + L/2) = -W^k)
__device__ __forceinline__ void load_tw(float4 *tw, const float4 *__restrict__ twff, int half) {
  for (int k = threadIdx.x; k < half; k += blockDim.x) {
    const float4 w = twff[k];
    tw[k] = w;
    tw[k + half] = c_neg(w);
  }
}
// The split of an M-point FFT Z of packed reals into X[k], k <= M:
// X[k] = E[k] + W_N^k O[k], E = (Z[k] + conj Z[M-k]) / 2,
// O = (Z[k] - conj Z[M-k]) / 2i (W_N^M = -1).
template <int M, typename T>
__device__ __forceinline__ T real_split(const T *line, int k, const T *tw) {
  const T zk = line[fpad(k % M)], zc = c_conj(line[fpad((M - k) % M)]);
  const T E = c_half(c_add(zk, zc)), O = c_div_2i(c_sub(zk, zc));
  return k == M ? c_sub(E, O) : c_add(E, k == 0 ? O : c_mul(tw[k], O));
}

// The twiddles of the FP32 row transforms in shared memory, from the
// float-float W_N^k table (N = 2M, high parts): tws[k] = W_N^k for k <= M / 2
// (the split) and twc[NS + k] = W_(NS R)^k, k < NS, for each pass NS > 1 of
// the M-point transform (NS a power of 8, R = min(8, M / NS); the ranges
// [NS, 2 NS) are disjoint).
template <int M>
__device__ __forceinline__ void load_tw_rows(float2 *tws, float2 *twc, const float4 *__restrict__ twff) {
  for (int e = threadIdx.x; e < M + M / 2 + 1; e += blockDim.x) {
    if (e <= M / 2) {
      const float4 w = twff[e];
      tws[e] = make_float2(w.x, w.z);
      continue;
    }
    const int c = e - (M / 2 + 1);
    int ns = 1;
    while (ns * 8 <= c) ns *= 8;
    const int k = c - ns;
    if (ns == 1 || k >= ns) continue;  // unused entries
    const int R = M / ns >= 8 ? 8 : M / ns;
    const float4 w = twff[k * (2 * M / (ns * R))];
    twc[c] = make_float2(w.x, w.z);
  }
}

// The split of the FP32 row transforms, two outputs per read pair: with
// E = (Z[k] + conj Z[M-k]) / 2, O = (Z[k] - conj Z[M-k]) / 2i and
// P = W_N^k O, X[k] = E + P and X[M - k] = conj(E - P) (E and O of M - k are
// the conjugates of those of k, W_N^(M-k) = -conj W_N^k); k = 0 gives X[0]
// and X[M], and its thread adds X[M/2].  Line b at s + b rowline_pitch<M>(),
// element i at fswz(i); task t of line b for t < M / 2, consecutive t on
// consecutive threads.
//
// Line pitch: M elements where a half warp's 16 threads lie in one line
// (M >= 128); shorter lines are M + M / 8 apart, so that the two or more
// lines of a half warp start on different banks.
template <int M>
constexpr int rowline_pitch() {
  return M >= 128 ? M : M + M / 8;
}
//
// The row kernels run 12 lines of M / 8 threads, i.e. 3 M / 2 threads:
// thread x takes t = x mod (M / 2) in lines x / (M / 2) + 3 i, so its two
// read addresses within a line and its twiddle serve all of its lines.
template <int M, int NL, typename Out>
__device__ __forceinline__ void split_pairs(const float2 *s, const float2 *tws, Out out) {
  constexpr int H = M / 2, LP = rowline_pitch<M>(), BS = 3;  // blockDim.x = BS H
  static_assert(NL % BS == 0, "split_pairs: lines in groups of three");
  const int t = threadIdx.x % H, b0 = threadIdx.x / H;
  const int ik = fswz(t), im = fswz((M - t) & (M - 1));
  const float2 w = tws[t];
#pragma unroll
  for (int i = 0; i < NL / BS; ++i) {
    const int b = b0 + BS * i;
    const float2 *line = s + b * LP;
    const float2 zk = line[ik], zm = c_conj(line[im]);
    const float2 E = c_half(c_add(zk, zm)), O = c_div_2i(c_sub(zk, zm));
    const float2 P = c_mul(w, O);
    out(b, t, c_add(E, P));
    out(b, M - t, c_conj(c_sub(E, P)));
    if (t == 0) {
      const float2 zh = line[fswz(H)], zhc = c_conj(zh);
      out(b, H, c_add(c_half(c_add(zh, zhc)), c_mul(tws[H], c_div_2i(c_sub(zh, zhc)))));
    }
  }
}

constexpr int kFfRows = 8;   // rows per CTA of the float-float real row pass
constexpr int kFfCRows = 4;  // rows per CTA of the float-float complex row pass
constexpr int kFfCols = 4;   // kx columns per CTA of the float-float column passes (64 bytes)

// What a row pass transforms: element pair m (real rows) or element x (complex
// rows) of row r.  Doubles from memory, the window of the field spectrum
// (dv on cells whose flag bit 4 is clear), or the field masked by the flags,
// formed here so that neither is stored first.
struct LoadReals {
  const double *in;
  __device__ __forceinline__ float4 pair(int64_t r, int n, int m) const {
    return c_from(reinterpret_cast<const double2 *>(in + r * n)[m]);
  }
};
struct LoadWindow {
  const int8_t *flags;
  __device__ __forceinline__ float4 pair(int64_t r, int n, int m) const {
    const char2 f = reinterpret_cast<const char2 *>(flags + r * n)[m];
    return make_float4(f.x & 4 ? 0.f : 1.f, 0.f, f.y & 4 ? 0.f : 1.f, 0.f);
  }
};
struct LoadComplex {
  const double2 *in;
  __device__ __forceinline__ float4 at(int64_t r, int n, int x) const { return c_from(in[r * n + x]); }
};
template <typename V>
struct LoadMasked {
  const V *in;
  const int8_t *flags;
  __device__ __forceinline__ float4 at(int64_t r, int n, int x) const {
    const int64_t i = r * n + x;
    const V v = in[i];
    if (flags[i] & 4) return make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (sizeof(v.x) == 4) return make_float4(v.x, 0.f, v.y, 0.f);
    else return c_from(v);
  }
};

// Row pass: kFfRows rows of N = 2M reals -> M + 1 complex each (float-float).
template <int M, typename Load>
__global__ void __launch_bounds__(kFfRows * M / 8) k_ff_rows(const Load in, float4 *__restrict__ out, int64_t rows,
                                                             const float4 *__restrict__ twff) {
  constexpr int N = 2 * M, NH = M + 1, TH = M / 8, LP = M + M / 8;
  __shared__ float4 s[kFfRows * LP];
  __shared__ float4 tw[N];  // W_N^k, k < N
  load_tw(tw, twff, M);
  const int64_t r0 = (int64_t)blockIdx.x * kFfRows;
  const int ln = threadIdx.x / TH, j = threadIdx.x % TH;
  const bool ok = r0 + ln < rows;
  float4 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = ok ? in.pair(r0 + ln, N, j + r * TH) : c_zero<float4>();
  __syncthreads();  // twiddles
  float4 *line = s + ln * LP;
  f_stockham<M, 1, false>(v, j, line, 1, tw, 2, [&](int i, float4 z) { line[fpad(i)] = z; });  // W_M = W_N^2
  __syncthreads();
  for (int idx = threadIdx.x; idx < kFfRows * NH; idx += blockDim.x) {
    const int b = idx / NH, k = idx % NH;
    if (r0 + b < rows) out[(r0 + b) * NH + k] = real_split<M>(s + b * LP, k, tw);
  }
}

// Complex row pass: kFfCRows contiguous rows of L complex values -> L
// float-float points each; the output may take the input's place (each CTA
// reads all of its rows before it writes).
template <int L, bool INV, typename Load>
__global__ void __launch_bounds__(kFfCRows * L / 8) k_ff_rows_c2c(const Load in, float4 *data, int64_t rows,
                                                                  const float4 *__restrict__ twff) {
  constexpr int TH = L / 8, LP = L + L / 8;
  __shared__ float4 s[kFfCRows * LP];
  __shared__ float4 tw[L];
  load_tw(tw, twff, L / 2);
  const int64_t r0 = (int64_t)blockIdx.x * kFfCRows;
  const int ln = threadIdx.x / TH, j = threadIdx.x % TH;
  const bool ok = r0 + ln < rows;
  float4 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = ok ? in.at(r0 + ln, L, j + r * TH) : c_zero<float4>();
  __syncthreads();
  float4 *out = data + (r0 + ln) * L;
  f_stockham<L, 1, INV>(v, j, s + ln * LP, 1, tw, 1, [&](int i, float4 z) {
    if (ok) out[i] = z;
  });
}

// Column pass: L-point FFTs along an axis of the half spectrum for NC
// adjacent kx.  Line (o, kx): element j at (o / ninner) shi + (o % ninner)
// slo + j sj + kx.  Thread (j, c) of column c loads its first-pass inputs
// from global memory and the last pass stores there; with `last` (float-
// float only) the result goes out as double2 in place.
template <typename T, int L, int NC>
constexpr size_t cols_smem() {
  return ((size_t)(L + L / 8) * NC + L) * sizeof(T);
}

template <typename T, int L, int NC, bool INV>
__global__ void __launch_bounds__(NC * L / 8) k_cols(T *__restrict__ data, int nh, int ninner, int64_t shi,
                                                     int64_t slo, int64_t sj, const float4 *__restrict__ twff,
                                                     int last) {
  constexpr int TH = L / 8, LP = L + L / 8;
  extern __shared__ __align__(16) unsigned char cols_sm[];
  T *s = reinterpret_cast<T *>(cols_sm);
  T *tw = s + LP * NC;  // W_L^k, k < L
  load_tw(tw, twff, L / 2);
  const int nkb = (nh + NC - 1) / NC;
  const int o = blockIdx.x / nkb, kx0 = (blockIdx.x % nkb) * NC;
  const int64_t base = (int64_t)(o / ninner) * shi + (int64_t)(o % ninner) * slo + kx0;
  const int c = threadIdx.x % NC, j = threadIdx.x / NC;
  const bool ok = kx0 + c < nh;
  T v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = ok ? data[base + (int64_t)(j + r * TH) * sj + c] : c_zero<T>();
  __syncthreads();  // twiddles
  f_stockham<L, 1, INV>(v, j, s + c, NC, tw, 1, [&](int i, T z) {
    if (!ok) return;
    const int64_t a = base + (int64_t)i * sj + c;
    if constexpr (sizeof(T) == 16) {
      if (last) {
        reinterpret_cast<double2 *>(data)[a] = make_double2(f2_to(re(z)), f2_to(im(z)));
        return;
      }
    }
    data[a] = z;
  });
}

// launch k_cols<T, L, NC, INV> (its shared memory may exceed the 48 KB default)
template <typename T, int L, int NC, bool INV>
int launch_cols(axg_ctx *ctx, const char *name, int64_t blocks, T *data, int nh, int ninner, int64_t shi, int64_t slo,
                int64_t sj, const float4 *tw, int last) {
  static bool attr = false;
  constexpr size_t sm = cols_smem<T, L, NC>();
  if (!attr && sm > 48 * 1024) {
    AXG_CUDA_TRY(ctx, cudaFuncSetAttribute(k_cols<T, L, NC, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    attr = true;
  }
  AXG_LAUNCH(ctx, name, (k_cols<T, L, NC, INV>), (unsigned)blocks, NC * L / 8, sm, data, nh, ninner, shi, slo, sj, tw,
             last);
  return AXG_OK;
}

template <int L, bool INV, typename Load>
int z2z_t(axg_ctx *ctx, const Load &in, double2 *data, const float4 *tw, bool keep_ff) {
  constexpr int n = L;
  const int64_t rows = (int64_t)n * n, plane = (int64_t)n * n, vol = plane * n;
  float4 *f = reinterpret_cast<float4 *>(data);
  AXG_LAUNCH(ctx, "fft_ff_rows_c2c", (k_ff_rows_c2c<L, INV, Load>), (unsigned)((rows + kFfCRows - 1) / kFfCRows),
             kFfCRows * L / 8, 0, in, f, rows, tw);
  const int nkb = n / kFfCols;
  AXG_TRY((launch_cols<float4, L, kFfCols, INV>(ctx, "fft_ff_y", (int64_t)n * nkb, f, n, n, vol, plane, (int64_t)n,
                                                 tw, 0)));
  AXG_TRY((launch_cols<float4, L, kFfCols, INV>(ctx, "fft_ff_z", (int64_t)n * nkb, f, n, n, vol, (int64_t)n, plane,
                                                 tw, keep_ff ? 0 : 1)));
  return AXG_OK;
}

// the y and z passes of a batched float-float D2Z whose row pass is done
template <int L>
int d2z_cols_t(axg_ctx *ctx, float4 *f, int batch, const float4 *tw, bool keep_ff) {
  constexpr int n = L, nh = L / 2 + 1;
  const int nkb = (nh + kFfCols - 1) / kFfCols;
  const int64_t plane = (int64_t)n * nh, vol = plane * n;
  // y: lines (field, z); z: lines (field, y)
  AXG_TRY((launch_cols<float4, L, kFfCols, false>(ctx, "fft_ff_y", (int64_t)batch * n * nkb, f, nh, n, vol, plane,
                                                   (int64_t)nh, tw, 0)));
  AXG_TRY((launch_cols<float4, L, kFfCols, false>(ctx, "fft_ff_z", (int64_t)batch * n * nkb, f, nh, n, vol,
                                                   (int64_t)nh, plane, tw, keep_ff ? 0 : 1)));
  return AXG_OK;
}

template <int L, typename Load>
int d2z_t(axg_ctx *ctx, const Load &in, double2 *out, int batch, const float4 *tw, bool keep_ff) {
  constexpr int n = L;
  const int64_t rows = (int64_t)batch * n * n;
  float4 *f = reinterpret_cast<float4 *>(out);
  AXG_LAUNCH(ctx, "fft_ff_rows", (k_ff_rows<L / 2, Load>), (unsigned)((rows + kFfRows - 1) / kFfRows),
             kFfRows * L / 16, 0, in, f, rows, tw);
  return d2z_cols_t<L>(ctx, f, batch, tw, keep_ff);
}

// FP64-plain Green step: the six FP64 sources (gw_sources_fp64, the
// reference's operations) formed inside the float-float row pass, so they
// never reach HBM.  One CTA per x-row (y, z): six lines, one per source, of
// M = N / 2 packed points z[m] = S(2m) + i S(2m + 1).  The FP64 pipe does
// the sources' arithmetic only; their float-float split runs on the integer
// pipes (f2_from_bits).  Output as k_ff_rows for batch 6.
// One thread per packed point m in the source phase (M threads, one round).
template <int M>
__global__ void __launch_bounds__(M) k_ff_gws_rows(const double2 *__restrict__ phi, double d, double inv_d,
                                                           int d_pow2, float4 *__restrict__ out,
                                                           const float4 *__restrict__ twff) {
  constexpr int N = 2 * M, NH = M + 1, TH = M / 8, LP = M + M / 8;
  __shared__ float4 s[8 * LP];
  __shared__ float4 tw[N];  // W_N^k, k < N
  load_tw(tw, twff, M);
  const int64_t row = blockIdx.x, nhalf = (int64_t)N * N * NH;
  const int y = (int)(row % N), z = (int)(row / N);
  const double2 *prow = phi + row * N;
  const double2 *pym = phi + ((int64_t)z * N + (y == 0 ? N - 1 : y - 1)) * N;
  const double2 *pyp = phi + ((int64_t)z * N + (y + 1 == N ? 0 : y + 1)) * N;
  const double2 *pzm = phi + ((int64_t)(z == 0 ? N - 1 : z - 1) * N + y) * N;
  const double2 *pzp = phi + ((int64_t)(z + 1 == N ? 0 : z + 1) * N + y) * N;
  for (int m = threadIdx.x; m < M; m += blockDim.x) {
    const int x0 = 2 * m;
    const double2 p0 = prow[x0], p1 = prow[x0 + 1];
    const double2 xm = prow[x0 == 0 ? N - 1 : x0 - 1], xp = prow[x0 + 2 == N ? 0 : x0 + 2];
    double S0[6], S1[6];
    {
      const double2 pa[3] = {p1, pyp[x0], pzp[x0]}, pb[3] = {xm, pym[x0], pzm[x0]};
      gw_sources_fp64<false>(pa, pb, d, inv_d, d_pow2, S0);
    }
    {
      const double2 pa[3] = {xp, pyp[x0 + 1], pzp[x0 + 1]}, pb[3] = {p0, pym[x0 + 1], pzm[x0 + 1]};
      gw_sources_fp64<false>(pa, pb, d, inv_d, d_pow2, S1);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c * LP + fpad(m)] = cx(f2_from_bits(S0[c]), f2_from_bits(S1[c]));
    s[6 * LP + fpad(m)] = s[7 * LP + fpad(m)] = c_zero<float4>();
  }
  __syncthreads();
  {
    // M threads = 8 lines of M / 8: lines 6 and 7 are scratch, transformed
    // so that every thread reaches the same barriers, and never read
    const int ln = threadIdx.x / TH, j = threadIdx.x % TH;
    float4 *line = s + ln * LP;
    float4 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = line[fpad(j + r * TH)];
    __syncthreads();
    f_stockham<M, 1, false>(v, j, line, 1, tw, 2, [&](int i, float4 x) { line[fpad(i)] = x; });  // W_M = W_N^2
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 6 * NH; idx += blockDim.x) {
    const int b = idx / NH, k = idx % NH;
    out[b * nhalf + row * NH + k] = real_split<M>(s + b * LP, k, tw);
  }
}

template <int L>
int ff_gws_d2z_t(axg_ctx *ctx, const double2 *phi, double d, double inv_d, int d_pow2, double2 *out,
                 const float4 *tw, bool keep_ff) {
  constexpr int n = L, M = L / 2;
  float4 *f = reinterpret_cast<float4 *>(out);
  AXG_LAUNCH(ctx, "gw_source_rows_fp64", k_ff_gws_rows<M>, (unsigned)((int64_t)n * n), M, 0, phi, d, inv_d, d_pow2,
             f, tw);
  return d2z_cols_t<L>(ctx, f, 6, tw, keep_ff);
}

// ---------------------------------------------------------------------------
// FP32 transform of the six Green's-function sources, the source computation
// fused into the row pass.  The FP32-mixed Green step needs the forward
// transforms of S_ij = (2 / d^2) (dr_i dr_j + di_i di_j), d_i the raw
// central differences of phi: the row kernel forms S_ij for its rows from
// phi (the stencil rows come through L1 / L2) and runs the real-to-half x
// transform of all six at once, so the real sources never reach HBM; the y
// and z passes are the TMA passes.  Output as cuFFT's R2C, rows padded:
// [6][n][n][pitch] complex float.  Twiddles are the high parts of the
// float-float table, i.e. W_n^k rounded to float.

constexpr int kSrcRows = 2;  // x-rows per CTA of the source row pass (6 x 2 lines)

// Opts a kernel into `smem` bytes of dynamic shared memory above the 48 KB
// default on the current device (a host-side call, repeated per launch so
// that every device a context runs on gets it)
template <typename K>
int allow_smem(axg_ctx *ctx, K kern, size_t smem) {
  if (smem > 48 * 1024)
    AXG_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return AXG_OK;
}

// Dynamic shared memory of the FP32 row kernels: nl lines, then the split
// and per-pass twiddles
template <int M>
constexpr size_t rows_f32_smem(int nl) {
  return ((size_t)nl * rowline_pitch<M>() + (M / 2 + 1) + M) * sizeof(float2);
}

// Row pass with the sources, for rows (y, z) = row0 .. row0 + kSrcRows - 1
// of the N = 2M lattice.  Line c kSrcRows + r holds source c of row r
// packed as M complex points z[m] = S(2m) + i S(2m + 1); an M-point FFT per
// line (M / 8 threads each), then the split into X[k], k <= M.
template <int M>
__global__ void __launch_bounds__(6 * kSrcRows * M / 8) k_gws_rows(const float2 *__restrict__ phi, float scale,
                                                                   float2 *__restrict__ out, int sp,
                                                                   const float4 *__restrict__ twff) {
  constexpr int N = 2 * M, NL = 6 * kSrcRows, TH = M / 8, LP = rowline_pitch<M>();
  extern __shared__ __align__(16) unsigned char rows_sm[];
  float2 *s = reinterpret_cast<float2 *>(rows_sm);
  float2 *tws = s + NL * LP, *twc = tws + (M / 2 + 1);
  load_tw_rows<M>(tws, twc, twff);
  const int64_t row0 = (int64_t)blockIdx.x * kSrcRows, nspec = (int64_t)N * N * sp;
  // Sources: thread m < M forms both rows' six sources at x = 2m, 2m + 1.
  // The rows are y0 and y0 + 1 of one z plane (y0 even), so their
  // y-neighbours are the rows y0 - 1 .. y0 + 2, two of them the rows
  // themselves: 12 loads for the pair instead of 14.
  static_assert(kSrcRows == 2, "the source phase pairs rows y0 and y0 + 1");
  const int y0 = (int)(row0 % N), z = (int)(row0 / N);
  const int64_t zr = (int64_t)z * N, zmr = (int64_t)(z == 0 ? N - 1 : z - 1) * N,
                zpr = (int64_t)(z + 1 == N ? 0 : z + 1) * N;
  const float2 *r0 = phi + (zr + y0) * N, *r1 = r0 + N;
  const float2 *rym = phi + (zr + (y0 == 0 ? N - 1 : y0 - 1)) * N;
  const float2 *ryp = phi + (zr + (y0 + 2 == N ? 0 : y0 + 2)) * N;
  const float2 *rzm0 = phi + (zmr + y0) * N, *rzm1 = rzm0 + N;
  const float2 *rzp0 = phi + (zpr + y0) * N, *rzp1 = rzp0 + N;
  for (int m = threadIdx.x; m < M; m += blockDim.x) {
    const int x0 = 2 * m, xl = x0 == 0 ? N - 1 : x0 - 1, xr = x0 + 2 == N ? 0 : x0 + 2;
    auto ld4 = [&](const float2 *row) { return *reinterpret_cast<const float4 *>(row + x0); };
    const float4 a_m = ld4(rym), a_0 = ld4(r0), a_1 = ld4(r1), a_p = ld4(ryp);
    const float4 zm0 = ld4(rzm0), zm1 = ld4(rzm1), zp0 = ld4(rzp0), zp1 = ld4(rzp1);
    const float2 xm0 = r0[xl], xp0 = r0[xr], xm1 = r1[xl], xp1 = r1[xr];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float4 c01 = r ? a_1 : a_0, pym = r ? a_0 : a_m, pyp = r ? a_p : a_1;  // phi(x0), phi(x0 + 1)
      const float4 pzm = r ? zm1 : zm0, pzp = r ? zp1 : zp0;
      const float2 xm = r ? xm1 : xm0, xp = r ? xp1 : xp0;
      float S[2][6];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        float dr[3], di[3];
        dr[0] = t == 0 ? c01.z - xm.x : xp.x - c01.x;
        di[0] = t == 0 ? c01.w - xm.y : xp.y - c01.y;
        dr[1] = t == 0 ? pyp.x - pym.x : pyp.z - pym.z;
        di[1] = t == 0 ? pyp.y - pym.y : pyp.w - pym.w;
        dr[2] = t == 0 ? pzp.x - pzm.x : pzp.z - pzm.z;
        di[2] = t == 0 ? pzp.y - pzm.y : pzp.w - pzm.w;
        int c = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j <= i; ++j, ++c) S[t][c] = scale * (dr[i] * dr[j] + di[i] * di[j]);
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) s[(c * kSrcRows + r) * LP + fswz(m)] = make_float2(S[0][c], S[1][c]);
    }
  }
  __syncthreads();
  {
    const int ln = threadIdx.x / TH, j = threadIdx.x % TH;
    float2 *line = s + ln * LP;
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = line[fswz(j + r * TH)];
    __syncthreads();
    f_stockham<M, 1, false, true, true>(v, j, line, 1, twc, 1, [&](int i, float2 x) { line[fswz(i)] = x; });
  }
  __syncthreads();
  split_pairs<M, NL>(s, tws, [&](int b, int k, float2 x) {
    out[(b / kSrcRows) * nspec + (row0 + b % kSrcRows) * sp + k] = x;
  });
}

// The u_ij spectrum's twelve real fields, tau u_c and u_c + tau u'_c (c =
// 11, 21, 22, 31, 32, 33; FP32-mixed subtracts the Kahan compensation from
// u first), formed inside the row pass as the Green sources are: one CTA per
// x-row, twelve lines.  Output [12][n][n][n/2+1] complex float.
template <int M>
__global__ void __launch_bounds__(12 * M / 8) k_uij_rows(const float *__restrict__ u, const float *__restrict__ ud,
                                                         const float *__restrict__ cu, int64_t n3, float tau,
                                                         float2 *__restrict__ out, int sp,
                                                         const float4 *__restrict__ twff) {
  constexpr int N = 2 * M, TH = M / 8, LP = rowline_pitch<M>();
  extern __shared__ __align__(16) unsigned char rows_sm[];
  float2 *s = reinterpret_cast<float2 *>(rows_sm);
  float2 *tws = s + 12 * LP, *twc = tws + (M / 2 + 1);
  load_tw_rows<M>(tws, twc, twff);
  const int64_t row = blockIdx.x, nspec = (int64_t)N * N * sp;
  for (int idx = threadIdx.x; idx < 6 * M; idx += blockDim.x) {
    const int c = idx / M, m = idx % M;
    const int64_t x = c * n3 + row * N + 2 * m;
    float2 uv = *reinterpret_cast<const float2 *>(u + x);
    if (cu) {
      const float2 cv = *reinterpret_cast<const float2 *>(cu + x);
      uv.x -= cv.x;
      uv.y -= cv.y;
    }
    const float2 dv = *reinterpret_cast<const float2 *>(ud + x);
    s[c * LP + fswz(m)] = make_float2(tau * uv.x, tau * uv.y);
    s[(6 + c) * LP + fswz(m)] = make_float2(uv.x + tau * dv.x, uv.y + tau * dv.y);
  }
  __syncthreads();
  {
    const int ln = threadIdx.x / TH, j = threadIdx.x % TH;
    float2 *line = s + ln * LP;
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = line[fswz(j + r * TH)];
    __syncthreads();
    f_stockham<M, 1, false, true, true>(v, j, line, 1, twc, 1, [&](int i, float2 x) { line[fswz(i)] = x; });
  }
  __syncthreads();
  split_pairs<M, 12>(s, tws, [&](int b, int k, float2 x) { out[b * nspec + row * sp + k] = x; });
}

// The same twelve fields in FP64 (tau u_c and u_c + tau u'_c), split into
// float-float on the integer pipes, in the float-float row pass.  Two CTAs
// per x-row, six fields each; M threads, lines 6 and 7 scratch as in
// k_ff_gws_rows.
template <int M>
__global__ void __launch_bounds__(M) k_ff_uij_rows(const double *__restrict__ u, const double *__restrict__ ud,
                                                   int64_t n3, double tau, float4 *__restrict__ out,
                                                   const float4 *__restrict__ twff) {
  constexpr int N = 2 * M, NH = M + 1, TH = M / 8, LP = M + M / 8;
  __shared__ float4 s[8 * LP];
  __shared__ float4 tw[N];  // W_N^k, k < N
  load_tw(tw, twff, M);
  const int half = (int)(blockIdx.x & 1);
  const int64_t row = blockIdx.x >> 1, nhalf = (int64_t)N * N * NH;
  for (int m = threadIdx.x; m < M; m += blockDim.x) {
    const int64_t x = row * N + 2 * m;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const double2 uv = *reinterpret_cast<const double2 *>(u + c * n3 + x);
      double2 w;
      if (half == 0) {
        w = make_double2(tau * uv.x, tau * uv.y);
      } else {
        const double2 dv = *reinterpret_cast<const double2 *>(ud + c * n3 + x);
        w = make_double2(uv.x + tau * dv.x, uv.y + tau * dv.y);
      }
      s[c * LP + fpad(m)] = cx(f2_from_bits(w.x), f2_from_bits(w.y));
    }
    s[6 * LP + fpad(m)] = s[7 * LP + fpad(m)] = c_zero<float4>();
  }
  __syncthreads();
  {
    const int ln = threadIdx.x / TH, j = threadIdx.x % TH;
    float4 *line = s + ln * LP;
    float4 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = line[fpad(j + r * TH)];
    __syncthreads();
    f_stockham<M, 1, false>(v, j, line, 1, tw, 2, [&](int i, float4 x) { line[fpad(i)] = x; });  // W_M = W_N^2
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 6 * NH; idx += blockDim.x) {
    const int b = idx / NH, k = idx % NH;
    out[(half * 6 + b) * nhalf + row * NH + k] = real_split<M>(s + b * LP, k, tw);
  }
}

constexpr int kFzCols = 8;  // kx columns per tile of the TMA passes: 64-byte boxes

// The z pass of the complex-float half spectra with its consumer: the
// transforms of a kx column's tensor components are contracted as they come
// out, in the registers that hold them, and never stored.
//
// A persistent CTA takes items of kFzCols kx columns x L z-points at one ky;
// the tiles of an item's fields follow each other through a ring of
// shared-memory stages filled by cp.async.bulk.tensor, and so do chunks of what
// the sink updates in memory.  The exchanges alternate between two line
// buffers, so that each needs one barrier; the first one also frees the stage.
// 128 registers a thread (16 warps an SM) hold the sums of a thread's eight
// outputs.
//
// 512^3: u_ij z pass and shell sums 3.04 + 0.83 -> 2.70 ms (the lines alone 1.6,
// the tiles' arrival 1.1); Green z pass and accumulation 1.34 + 2.31 -> 2.21 ms
// (10.9 GB, 0.73 of the copy peak); 128^3 40 + 44 -> 48 and 23 + 39 -> 41 us.
// With the accumulators read and written by the threads instead of through the
// ring the Green form took 3.92 ms, its 16 warps waiting on them, and with
// polarisations and TT coefficients over |k| (division, square root and 8 more
// registers an output) the u_ij form 3.79.
template <int L>
constexpr int zs_stages() {
  return L >= 512 ? 4 : 3;
}
template <int L>
constexpr int zs_blocks() {  // CTAs per SM: 512 threads, at most 16
  return L < 32 ? 16 : 4096 / (kFzCols * L);
}
template <int L>
constexpr size_t zs_smem() {  // without the sink's
  return (size_t)(zs_stages<L>() * L * kFzCols + 2 * (L + L / 8) * kFzCols + L) * sizeof(float2) + 8 * zs_stages<L>() +
         128 + 16;
}
// the last pass of an L-point line: its stride (L / its radix), and the z index
// of thread j's output in slot s less j
template <int L>
constexpr int z_last_ns() {
  int ns = 1;
  while (L / ns > 8) ns *= 8;
  return ns;
}
template <int L>
__host__ __device__ constexpr int z_off(int s) {
  constexpr int NS = z_last_ns<L>(), R = L / NS;
  return (s / R) * (L / 8) + (s % R) * NS;
}
// ... its wave number, from j as a float: outputs r >= R / 2 are the negative ones
template <int L>
__device__ __forceinline__ float z_wave(float jf, int s) {
  constexpr int R = L / z_last_ns<L>();
  return jf + (float)(z_off<L>(s) - (s % R >= R / 2 ? L : 0));
}

// j as a float the compiler knows nothing of: what depends on it is formed where
// it is used, not ahead of the loop over an item's fields (where the values of
// all eight outputs and six components spilled 300 bytes a thread)
__device__ __forceinline__ float fresh(int j) {
  asm volatile("" : "+r"(j));
  return (float)j;
}

// Twiddles of the passes NS = 8, 64 of an L-point line: W_(NS R)^(r k) at
// (r - 1) NS + k after those of the pass before, consecutive k on consecutive
// banks.
template <int L>
__device__ __forceinline__ void load_tw_z(float2 *tw, const float4 *__restrict__ twff) {
  int at = 0;
  for (int ns = 8; ns < L; ns *= 8) {
    const int R = L / ns >= 8 ? 8 : L / ns;
    for (int e = threadIdx.x; e < (R - 1) * ns; e += blockDim.x) {
      const int r = 1 + e / ns, k = e % ns, i = r * k * (L / (ns * R));  // < L
      const float4 w = twff[i & (L / 2 - 1)];
      tw[at + e] = i < L / 2 ? make_float2(w.x, w.z) : make_float2(-w.x, -w.z);
    }
    at += (R - 1) * ns;
  }
}

// fpad(i + s) - fpad(i) for the passes' offsets s: multiples of 8, or i + s % 8 < 8
constexpr int z_pad(int s) { return (s + s / 8) * kFzCols; }

// one exchange and the passes NS >= 8 after it: outputs of the pass before in v,
// element i + r NS0 of the line in v[r]; the outputs stay in v.  sync: the
// barrier of this exchange; buf: the buffers, swapped at each exchange.
template <int L, int NS, typename Sync>
__device__ __forceinline__ void z_passes(float2 v[8], int j, float2 *&b0, float2 *&b1, const float2 *tw, Sync sync) {
  constexpr int NS0 = NS / 8, R = L / NS >= 8 ? 8 : L / NS, NI = 8 / R, TH = L / 8;
  {
    const int d = (j / NS0) * NS + (j & (NS0 - 1));
    float2 *w = b0 + fpad(d) * kFzCols;
#pragma unroll
    for (int r = 0; r < 8; ++r) w[NS0 == 1 ? r * kFzCols : z_pad(r * NS0)] = v[r];
  }
  sync();
  {
    const float2 *p = b0 + fpad(j) * kFzCols;
#pragma unroll
    for (int q = 0; q < NI; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r) v[q * R + r] = p[z_pad(q * TH + r * (L / R))];
  }
  float2 *const t = b0;
  b0 = b1;
  b1 = t;
#pragma unroll
  for (int q = 0; q < NI; ++q) {
    const int k = (j + q * TH) & (NS - 1);
#pragma unroll
    for (int r = 1; r < R; ++r) v[q * R + r] = c_mul(v[q * R + r], tw[(r - 1) * NS + k]);
    c_dft<R, false>(&v[q * R]);
  }
  if constexpr (NS * R < L) z_passes<L, NS * 8>(v, j, b0, b1, tw + (R - 1) * NS, [] { __syncthreads(); });
}

// y pass of the complex-float half spectra (Z: z pass): persistent CTAs walk
// tiles of kFzCols kx columns x L points (one z plane of one field; one ky)
// through the ring of stages; a tile is transformed into its own stage and leaves by a bulk
// tensor store.  A wait that runs out raises AXG_KERR_MBAR_TIMEOUT.  512^3, six
// spectra: 1.30 ms by one CTA per 4 columns from the threads' loads (32-byte
// rows), 1.09 so (0.90 of the copy peak).
template <int L, bool Z>
__global__ void __launch_bounds__(kFzCols *L / 8, zs_blocks<L>())
    k_cols_tma(const __grid_constant__ CUtensorMap tm, int nkb, int ntiles_all, const float4 *__restrict__ twff, int *err) {
  using namespace axg_tma;
  constexpr int TH = L / 8, LP = L + L / 8, TILE = L * kFzCols, BOX = L < 256 ? L : 256, S = zs_stages<L>();
  extern __shared__ unsigned char zt_raw[];
  unsigned char *sm =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(zt_raw) + 127) & ~uintptr_t(127));
  float2 *tile = reinterpret_cast<float2 *>(sm);
  float2 *xb = tile + S * TILE;
  float2 *tw = xb + 2 * LP * kFzCols;
  uint64_t *bars = reinterpret_cast<uint64_t *>(tw + L);
  load_tw_z<L>(tw, twff);
  const uint32_t bar0 = smem_u32(bars);
  if (threadIdx.x == 0) {
    for (int q = 0; q < S; ++q) mbar_init(bar0 + 8 * q, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const int ntiles = (ntiles_all - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  int next = 0;  // thread 0: the CTA's next tile to load
  auto at = [&](int t, int &kb, int &z, int &f) {
    const int i = blockIdx.x + t * (int)gridDim.x, o = i / nkb;
    kb = i - o * nkb;
    f = o / L;
    z = o & (L - 1);
  };
  auto load_to = [&](int limit) {
    for (; next < limit && next < ntiles; ++next) {
      int kb, z, f;
      at(next, kb, z, f);
      const uint32_t dst = smem_u32(tile + next % S * TILE), bar = bar0 + 8 * (next % S);
      mbar_expect_tx(bar, TILE * sizeof(float2));
#pragma unroll
      for (int h = 0; h < L / BOX; ++h)
        tma_load_4d(dst + h * BOX * kFzCols * (int)sizeof(float2), &tm, kb * kFzCols, Z ? z : h * BOX,
                    Z ? h * BOX : z, f, bar);
    }
  };
  if (threadIdx.x == 0) load_to(S);
  const int c = threadIdx.x % kFzCols, j = threadIdx.x / kFzCols;
  float2 *b0 = xb + c, *b1 = b0 + LP * kFzCols;
  int t = 0, bad = 0;
  for (; t < ntiles; ++t) {
    const int late = !mbar_wait_bounded(bar0 + 8 * (t % S), (t / S) & 1);
    float2 *tl = tile + t % S * TILE;
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = tl[(j + r * TH) * kFzCols + c];
    c_dft<8, false>(v);
    z_passes<L, 8>(v, j, b0, b1, tw, [&] {
      bad = __syncthreads_or(late);  // every thread has read the stage
      if (threadIdx.x == 0 && !bad && t > 0 && next < ntiles) {
        bulk_wait_read0();  // the store of the tile before has, too
        load_to(t + S);
      }
    });
    if (bad) break;
#pragma unroll
    for (int s = 0; s < 8; ++s) tl[(j + z_off<L>(s)) * kFzCols + c] = v[s];
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      int kb, z, f;
      at(t, kb, z, f);
      const uint32_t src = smem_u32(tl);
#pragma unroll
      for (int h = 0; h < L / BOX; ++h)
        tma_store_4d(&tm, src + h * BOX * kFzCols * (int)sizeof(float2), kb * kFzCols, Z ? z : h * BOX,
                     Z ? h * BOX : z, f);
      bulk_commit();
    }
  }
  if (threadIdx.x == 0) {
    if (bad) {
      atomicCAS(err, 0, AXG_KERR_MBAR_TIMEOUT);
      for (int q = t + 1; q < next; ++q) mbar_wait_bounded(bar0 + 8 * (q % S), (q / S) & 1, 100000000LL);
    }
    bulk_wait0();
  }
}

// A sink: kFields tiles an item, field(f) the spectrum of tile f, then kChunks
// chunks of rows that it updates; begin, take (tile f's outputs in v, slot s
// at z = j + z_off(s)), chunk and end of an item; finish.
template <int L, typename Sink>
__global__ void __launch_bounds__(kFzCols *L / 8, zs_blocks<L>())
    k_z_sink(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tc, int nkb, int nitems,
             const float4 *__restrict__ twff, const typename Sink::Args args, int *err) {
  using namespace axg_tma;
  constexpr int TH = L / 8, LP = L + L / 8, TILE = L * kFzCols, BOX = L < 256 ? L : 256, S = zs_stages<L>(),
                NF = Sink::kFields, NT = NF + Sink::kChunks;
  constexpr uint32_t BYTES = TILE * sizeof(float2);
  extern __shared__ unsigned char zt_raw[];
  unsigned char *sm =
      reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(zt_raw) + 127) & ~uintptr_t(127));
  float2 *tile = reinterpret_cast<float2 *>(sm);  // [S][L][kFzCols], dense as the TMA box
  float2 *xb = tile + S * TILE;                    // two sets of exchange lines
  float2 *tw = xb + 2 * LP * kFzCols;
  uint64_t *bars = reinterpret_cast<uint64_t *>(tw + L);
  load_tw_z<L>(tw, twff);
  const uint32_t bar0 = smem_u32(bars);
  if (threadIdx.x == 0) {
    for (int q = 0; q < S; ++q) mbar_init(bar0 + 8 * q, 1);
    fence_barrier_init();
  }
  Sink sink(args, reinterpret_cast<double *>(bars + S));
  __syncthreads();
  const int ntiles = (nitems - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * NT;
  int next = 0;                      // thread 0: the CTA's next tile to load
  auto load_to = [&](int limit) {
    for (; next < limit && next < ntiles; ++next) {
      const int item = blockIdx.x + (next / NT) * (int)gridDim.x, o = item / nkb, kb = item % nkb, f = next % NT;
      const uint32_t dst = smem_u32(tile + next % S * TILE), bar = bar0 + 8 * (next % S);
      if (f < NF) {
        mbar_expect_tx(bar, BYTES);
#pragma unroll
        for (int h = 0; h < L / BOX; ++h)
          tma_load_4d(dst + h * BOX * kFzCols * (int)sizeof(float2), &tm, kb * kFzCols, o, h * BOX, Sink::field(f),
                      bar);
      } else {
        sink.load_chunk(&tc, dst, bar, kb, o, f - NF);
      }
    }
  };
  if (threadIdx.x == 0) load_to(S);
  const int c = threadIdx.x % kFzCols, j = threadIdx.x / kFzCols;
  float2 *b0 = xb + c, *b1 = b0 + LP * kFzCols;
  int t = 0, bad = 0;
  for (int item = blockIdx.x; item < nitems && !bad; item += gridDim.x) {
    const int ky = item / nkb, kb = item % nkb;
    sink.begin(kb * kFzCols + c, ky);
#pragma unroll 1
    for (int f = 0; f < NF; ++f, ++t) {
      const int late = !mbar_wait_bounded(bar0 + 8 * (t % S), (t / S) & 1);
      const float2 *tl = tile + t % S * TILE + j * kFzCols + c;
      float2 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = tl[r * TH * kFzCols];
      c_dft<8, false>(v);
      z_passes<L, 8>(v, j, b0, b1, tw, [&] {
        bad = __syncthreads_or(late);  // every thread has read the stage
        if (threadIdx.x == 0 && !bad) {
          if (Sink::kChunks && next < ntiles) bulk_wait_read0();  // the last chunk's store has, too
          load_to(t + 1 + S);
        }
      });
      if (bad) break;
      sink.take(f, v, j);
    }
    if constexpr (Sink::kChunks > 0) {
#pragma unroll
      for (int f = 0; f < Sink::kChunks; ++f) {
        if (bad) break;
        const int late = !mbar_wait_bounded(bar0 + 8 * (t % S), (t / S) & 1);
        float2 *tl = tile + t % S * TILE;
        if (!late) sink.chunk(f, reinterpret_cast<float4 *>(tl), j, c);
        fence_proxy_async();
        bad = __syncthreads_or(late);
        if (bad) break;
        if (threadIdx.x == 0) {
          if (next < ntiles) bulk_wait_read0();  // the store before this one has read its stage
          load_to(t + S);
          sink.store_chunk(&tc, smem_u32(tl), kb, ky, f);
          bulk_commit();
        }
        ++t;
      }
    }
    if (!bad) sink.end(j, c, b0, b1);
  }
  if (threadIdx.x == 0) {
    if (bad) {
      atomicCAS(err, 0, AXG_KERR_MBAR_TIMEOUT);
      for (int q = t + 1; q < next; ++q) mbar_wait_bounded(bar0 + 8 * (q % S), (q / S) & 1, 100000000LL);
    }
    bulk_wait0();
  }
  sink.finish();
}

// TT power of u_ij into shell sums: tt_basis times k^2, whose coefficients are
// polynomials in kz, U_mm - U_ll in A and |k| U_ml in B.  The trace drops out
// through the differences to component 33, so that one and 11 come first.
template <int L>
struct UijSink {
  static constexpr int kFields = 12, kChunks = 0;  // 33, 11, 22, 21, 31, 32 of w', then of w
  struct Args {
    const int16_t *tab;
    int nb, copies;
    float dwav2;
    double *numer, *denom;
  };
  __device__ __forceinline__ static int field(int f) {
    const int g = f % 6;
    return (f < 6 ? 6 : 0) + (g == 0 ? 5 : g == 1 ? 0 : g == 2 ? 2 : g == 3 ? 1 : g - 1);
  }
  __device__ __forceinline__ void load_chunk(const CUtensorMap *, uint32_t, uint32_t, int, int, int) {}
  __device__ __forceinline__ void store_chunk(const CUtensorMap *, uint32_t, int, int, int) {}
  const Args &a;
  BlockBins bins;
  BinRun<F2> run;
  int ix;
  float kx, ky, sc, df;  // s c and s^2 - c^2 of the azimuth
  float e[8];
  float2 A[8], B[8];
  __device__ UijSink(const Args &args, double *mem) : a(args), bins(mem, args.nb, args.copies) {}
  __device__ __forceinline__ void begin(int hx, int hy) {
    ix = hx;
    kx = (float)(hx < L / 2 ? hx : hx - L);
    ky = (float)(hy < L / 2 ? hy : hy - L);
    const float p2 = kx * kx + ky * ky, ip2 = p2 > 0.f ? 1.f / p2 : 0.f;
    sc = kx * ky * ip2;
    df = p2 > 0.f ? (ky * ky - kx * kx) * ip2 : -1.f;
  }
  __device__ __forceinline__ void take(int f, const float2 v[8], int j) {
    const int g = f < 6 ? f : f - 6;
    const float jf = fresh(j);
    if (g == 0) {
#pragma unroll
      for (int s = 0; s < 8; ++s) A[s] = v[s];
    } else if (g == 1) {
#pragma unroll
      for (int s = 0; s < 8; ++s) B[s] = v[s];
    } else if (g == 2) {
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        // k^2 (s^2 - q^2 c^2) = ky^2 + kz^2 (s^2 - c^2), and 22 with kx, -
        const float kz = z_wave<L>(jf, s), kd = kz * kz * df;
        const float a11 = fmaf(ky, ky, kd), a22 = fmaf(kx, kx, -kd), b11 = kz * sc;
        const float2 x33 = A[s], x11 = B[s];
        A[s].x = a11 * (x11.x - x33.x) + a22 * (v[s].x - x33.x);
        A[s].y = a11 * (x11.y - x33.y) + a22 * (v[s].y - x33.y);
        B[s].x = b11 * (x11.x - v[s].x);
        B[s].y = b11 * (x11.y - v[s].y);
      }
    } else if (g == 3) {
      const float m2 = -2.f * kx * ky, m4 = -4.f * sc;  // -2 s c (k^2 + kz^2)
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float kz = z_wave<L>(jf, s);
        add(s, fmaf(kz * kz, m4, m2), kz * df, v[s]);
      }
    } else {
      const float ka = 2.f * (g == 4 ? kx : ky), kb = g == 4 ? -ky : kx;
#pragma unroll
      for (int s = 0; s < 8; ++s) add(s, z_wave<L>(jf, s) * ka, kb, v[s]);
      if (g == 5) {
        const float p2 = kx * kx + ky * ky;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const float kz = z_wave<L>(jf, s), k2 = fmaf(kz, kz, p2), ik = gw_rsqrt(k2), i2 = ik * ik;
          const float px = A[s].x * i2, py = A[s].y * i2, cx = B[s].x * ik, cy = B[s].y * ik;
          const float p = 0.5f * (px * px + py * py) + 2.f * (cx * cx + cy * cy);
          e[s] = f < 6 ? p : fmaf(k2 * a.dwav2, p, e[s]);
        }
      }
    }
  }
  __device__ __forceinline__ void add(int s, float ca, float cb, float2 v) {
    A[s].x = fmaf(ca, v.x, A[s].x);
    A[s].y = fmaf(ca, v.y, A[s].y);
    B[s].x = fmaf(cb, v.x, B[s].x);
    B[s].y = fmaf(cb, v.y, B[s].y);
  }
  // The item's powers to the bins: through an exchange buffer, so that a thread
  // sums runs of |kz| (kz and -kz share their bin) before it adds to the shared
  // bins; added as they lie, 8 values in 8 bins, they took 0.6 ms at 512^3.
  __device__ __forceinline__ void end(int j, int c, float2 *&b0, float2 *&b1) {
    constexpr int TH = L / 8, PER = L / 2 / TH;
    float *x = reinterpret_cast<float *>(b0 - c) + c;
    auto at = [](int z) { return (z + z / 4) * kFzCols; };
#pragma unroll
    for (int s = 0; s < 8; ++s) x[at(j + z_off<L>(s))] = e[s];
    __syncthreads();
    if (ix <= L / 2) {
      const unsigned wgt = (ix == 0 || ix == L / 2) ? 1u : 2u;  // Hermitian partner of the half spectrum
      const int p2 = (int)(kx * kx + ky * ky);
      auto put = [&](int z, float p, float q, unsigned w) {  // p + q, floats whose sums need not be
        const int b = a.tab[p2 + z * z];
        if (b < 0) return;
        if (fmaxf(p, q) < 0x1p118f) {
          const F2 v = f2_add(F2{p, 0.f}, F2{q, 0.f});
          run.add(bins, b, F2{(float)wgt * v.h, (float)wgt * v.l}, wgt * w);
        } else {
          bins.add(b, (double)wgt * ((double)p + (double)q), wgt * w);
        }
      };
      if (j == 0) put(0, x[0], 0.f, 1u);
#pragma unroll
      for (int i = 1; i <= PER; ++i) {
        const int z = j * PER + i;
        if (z < L / 2) put(z, x[at(z)], x[at(L - z)], 2u);
        else put(z, x[at(z)], 0.f, 1u);
      }
      run.flush(bins);
    }
    float2 *const t = b0;
    b0 = b1;
    b1 = t;
  }
  __device__ __forceinline__ void finish() { bins.finish(a.numer, a.denom); }
};

// The Green accumulation.  With e+ times k^2, the contractions split into sums
// whose coefficients are polynomials in kz:
//   Sa = sum k^2 Re(e) Re(S), Se = sum k^2 Re(e) Im(S),
//   Sb = sum |k| Im(e) Im(S), Sg = sum |k| Im(e) Re(S)   (S conjugated),
// X+ = (Sa - Sb', Se + Sg'), X- = (Sa + Sb', Se - Sg') over k^2.  The sums carry
// k^2 <= 2e5, so a source spectrum may reach 1e33.  A chunk is the accumulators
// of one output slot of every thread.
template <int L>
struct GreenSink {
  static constexpr int kFields = 6, kChunks = 8;
  static constexpr int NH = L / 2 + 1, TH = L / 8, SP = axg_f32_spec_pitch(L);
  struct Args {
    float2 *srcF;
    int ref_compat;
    float Th, Tl, dw, dwl;
  };
  __device__ __forceinline__ static int field(int f) { return f; }
  const Args &a;
  int ix, iy;
  float kx, ky, cs, df;  // c s and c^2 - s^2 of the azimuth
  float2 R[8], I[8];     // (Sa, Se), (Sb, Sg)
  float2 last[8];        // the source 33
  __device__ GreenSink(const Args &args, double *) : a(args) {}
  // the chunk in a stage: [4][TH][kFzCols] float4
  __device__ __forceinline__ void load_chunk(const CUtensorMap *tc, uint32_t dst, uint32_t bar, int kb, int o, int f) {
    constexpr uint32_t ONE = TH * kFzCols * sizeof(float4);
    axg_tma::mbar_expect_tx(bar, (a.ref_compat ? 3 : 4) * ONE);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q != 1 || !a.ref_compat) axg_tma::tma_load_4d(dst + q * ONE, tc, kb * kFzCols * 2, o, z_off<L>(f), q, bar);
  }
  __device__ __forceinline__ void store_chunk(const CUtensorMap *tc, uint32_t src, int kb, int o, int f) {
    constexpr uint32_t ONE = TH * kFzCols * sizeof(float4);
#pragma unroll
    for (int q = 0; q < 4; ++q) axg_tma::tma_store_4d(tc, src + q * ONE, kb * kFzCols * 2, o, z_off<L>(f), q);
  }
  __device__ __forceinline__ void begin(int hx, int hy) {
    ix = hx;
    iy = hy;
    kx = (float)(hx < L / 2 ? hx : hx - L);
    ky = (float)(hy < L / 2 ? hy : hy - L);
    const float p2 = kx * kx + ky * ky, ip2 = p2 > 0.f ? 1.f / p2 : 0.f;
    cs = kx * ky * ip2;
    df = p2 > 0.f ? (kx * kx - ky * ky) * ip2 : 1.f;
#pragma unroll
    for (int s = 0; s < 8; ++s) R[s] = I[s] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(int s, float pr, float pi, float2 v) {
    R[s].x = fmaf(pr, v.x, R[s].x);
    R[s].y = fmaf(-pr, v.y, R[s].y);
    I[s].x = fmaf(-pi, v.y, I[s].x);
    I[s].y = fmaf(pi, v.x, I[s].y);
  }
  __device__ __forceinline__ void take(int f, const float2 v[8], int j) {
    const float jf = fresh(j);
    // e+_ij = p_i p_j, halved on the diagonal, |k| p = (kz c - i |k| s, kz s + i |k| c, -p)
    if (f == 0 || f == 2) {
      const float h = (f == 0 ? 0.5f : -0.5f) * df, k = f == 0 ? ky : kx, g = -0.5f * k * k, t = f == 0 ? -cs : cs;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float kz = z_wave<L>(jf, s);
        add(s, fmaf(kz * kz, h, g), kz * t, v[s]);
      }
    } else if (f == 1) {
      const float h = 2.f * cs, g = kx * ky;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float kz = z_wave<L>(jf, s);
        add(s, fmaf(kz * kz, h, g), kz * df, v[s]);
      }
    } else if (f < 5) {
      const float k = f == 3 ? -kx : -ky, t = f == 3 ? ky : -kx;  // p s = ky, p c = kx
#pragma unroll
      for (int s = 0; s < 8; ++s) add(s, z_wave<L>(jf, s) * k, t, v[s]);
    } else {
#pragma unroll
      for (int s = 0; s < 8; ++s) last[s] = v[s];
    }
    // the rows whose mirrors are entries of their own keep their transforms
    constexpr int ny = L / 2 / z_last_ns<L>();  // the slot of z = n/2, thread j = 0
    if (ix > 0 && ix < L / 2 && (iy == L / 2 || j == 0)) {
      float2 *o = a.srcF + ((int64_t)(f * L + j) * L + iy) * SP + ix;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (iy == L / 2 || s == ny) o[(int64_t)z_off<L>(s) * L * SP] = v[s];
    }
  }
  __device__ __forceinline__ void chunk(int s, float4 *tl, int j, int c) {
    float4 *t = tl + j * kFzCols + c;
    constexpr int ONE = TH * kFzCols;
    const float kz = z_wave<L>(fresh(j), s), p2 = kx * kx + ky * ky, k2 = fmaf(kz, kz, p2);
    F32Acc ac;
    ac.load(t, ONE, 0, a.ref_compat);
    if (k2 > 0.f) {
      const float ik = gw_rsqrt(k2), i2 = ik * ik;
      // e33 = p^2 / 2: its part of X-, and its parts of Sa and Se
      const float h = 0.5f * p2, lr = h * last[s].x, li = h * -last[s].y;
      const float Ra = (R[s].x + lr) * i2, Re = (R[s].y + li) * i2, Ib = I[s].x * ik, Ig = I[s].y * ik;
      const float x[2] = {Ra - Ib, Re + Ig}, m[2] = {Ra + Ib, Re - Ig}, l[2] = {lr * i2, li * i2};
      float sq, cq;
      gw_cos_sin(k2, ik, a.Th, a.Tl, &cq, &sq);
      ac.update(fmaf(a.dwl, cq, a.dw * cq), fmaf(a.dwl, sq, a.dw * sq), x, m, l, a.ref_compat);
    } else if (a.ref_compat) {
      ac.a21 = ac.a12;
    }
    ac.store(t, ONE, 0);
  }
  __device__ __forceinline__ void end(int, int, float2 *&, float2 *&) {}
  __device__ __forceinline__ void finish() {}
};

// a persistent TMA pass: as many CTAs as fit, at most `items`
template <int L, typename K, typename... A>
int launch_persistent(axg_ctx *ctx, const char *name, K kern, int items, size_t smem, const A &...args) {
  AXG_TRY(allow_smem(ctx, kern, smem));
  AXG_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  constexpr int threads = kFzCols * L / 8;
  int per_sm = 0, sms = 0;
  AXG_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
  if (per_sm < 1) return axg_set_error(ctx, AXG_ERR_CUDA, "transform kernel does not fit on an SM");
  AXG_CUDA_TRY(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  AXG_LAUNCH(ctx, name, kern, (unsigned)std::min(items, sms * per_sm), threads, smem, args...);
  return AXG_OK;
}

// The tensor maps of `batch` half spectra, (re, im) float pairs, by tiles along
// y and along z
template <int L>
int spec_tmaps(axg_ctx *ctx, float2 *F, int batch, CUtensorMap *my, CUtensorMap *mz) {
  constexpr int n = L, sp = axg_f32_spec_pitch(L), BOX = L < 256 ? L : 256;
  const cuuint64_t dims[4] = {(cuuint64_t)sp, (cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)batch};
  const cuuint64_t str[3] = {(cuuint64_t)sp * 8, (cuuint64_t)n * sp * 8, (cuuint64_t)n * n * sp * 8};
  const cuuint32_t ybox[4] = {kFzCols, BOX, 1, 1}, zbox[4] = {kFzCols, 1, BOX, 1};
  AXG_TRY(axg_encode_tmap(ctx, my, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, F, dims, str, ybox));
  return axg_encode_tmap(ctx, mz, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, F, dims, str, zbox);
}

// the y pass in complex float of a sink's half spectra and their z pass into it
template <int L, typename Sink>
int f_cols_sink(axg_ctx *ctx, const char *name, float2 *F, const float4 *tw, const typename Sink::Args &args,
                size_t sink_smem) {
  constexpr int n = L, nh = L / 2 + 1, batch = Sink::kFields, nkb = (nh + kFzCols - 1) / kFzCols;
  CUtensorMap my, mz;
  AXG_TRY(spec_tmaps<L>(ctx, F, batch, &my, &mz));
  CUtensorMap mc = mz;
  if (Sink::kChunks) {
    const cuuint64_t adims[4] = {(cuuint64_t)2 * nh, (cuuint64_t)n, (cuuint64_t)n, 4};
    const cuuint64_t astr[3] = {(cuuint64_t)nh * 16, (cuuint64_t)n * nh * 16, (cuuint64_t)ctx->acc_stride * 16};
    const cuuint32_t abox[4] = {2 * kFzCols, 1, L / 8, 1};
    AXG_TRY(axg_encode_tmap(ctx, &mc, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, ctx->acc, adims, astr, abox));
  }
  AXG_TRY((launch_persistent<L>(ctx, "fft_f32_y", k_cols_tma<L, false>, batch * n * nkb, zs_smem<L>(), my, nkb,
                                batch * n * nkb, tw, ctx->d_err)));
  return launch_persistent<L>(ctx, name, k_z_sink<L, Sink>, n * nkb, zs_smem<L>() + sink_smem, mz, mc, nkb, n * nkb,
                              tw, args, ctx->d_err);
}

template <int L>
int uij_power_t(axg_ctx *ctx, const float *u, const float *ud, const float *cu, float tau, float2 *F, double dwav,
                const int16_t *tab, int nb, double *numer, double *denom, const float4 *tw) {
  constexpr int n = L, M = L / 2;
  const int sp = axg_f32_spec_pitch(n);
  constexpr size_t smem = rows_f32_smem<M>(12);
  AXG_TRY(allow_smem(ctx, k_uij_rows<M>, smem));
  AXG_LAUNCH(ctx, "uij_rows_fp32", k_uij_rows<M>, (unsigned)((int64_t)n * n), 12 * M / 8, smem, u, ud, cu,
             (int64_t)n * n * n, tau, F, sp, tw);
  const typename UijSink<L>::Args args = {tab, nb, bin_copies(nb), (float)(dwav * dwav), numer, denom};
  return f_cols_sink<L, UijSink<L>>(ctx, "uij_z_bin_fp32", F, tw, args, bin_smem(nb));
}

template <int L>
int ff_uij_d2z_t(axg_ctx *ctx, const double *u, const double *ud, double tau, double2 *out, const float4 *tw) {
  constexpr int n = L, M = L / 2;
  float4 *f = reinterpret_cast<float4 *>(out);
  AXG_LAUNCH(ctx, "uij_rows_fp64", k_ff_uij_rows<M>, (unsigned)(2 * (int64_t)n * n), M, 0, u, ud,
             (int64_t)n * n * n, tau, f, tw);
  return d2z_cols_t<L>(ctx, f, 12, tw, false);
}

// Up to 64^3 a step is its kernels' latencies: an item's chain of fourteen tiles
// in the sink takes 9 us there, storing the transforms and accumulating from
// them 5 (Green step at 64^3 33 and 27 us); at 128^3 41 + 3 and 62.
constexpr int kGreenUnfused = 64;

template <int L>
int gws_accumulate_t(axg_ctx *ctx, const float2 *phi, float2 *srcF, float scale, double phase1, float dw,
                     float dwl, int ref_compat, const float4 *tw) {
  constexpr int n = L, M = L / 2;
  const int64_t rows = (int64_t)n * n;
  constexpr size_t smem = rows_f32_smem<M>(6 * kSrcRows);
  AXG_TRY(allow_smem(ctx, k_gws_rows<M>, smem));
  AXG_LAUNCH(ctx, "gw_source_rows_fp32", k_gws_rows<M>, (unsigned)(rows / kSrcRows), 6 * kSrcRows * M / 8, smem,
             phi, scale, srcF, axg_f32_spec_pitch(n), tw);
  if constexpr (L <= kGreenUnfused) {
    constexpr int items = 6 * n * ((n / 2 + kFzCols) / kFzCols), nkb = (n / 2 + kFzCols) / kFzCols;
    CUtensorMap my, mz;
    AXG_TRY(spec_tmaps<L>(ctx, srcF, 6, &my, &mz));
    AXG_TRY((launch_persistent<L>(ctx, "fft_f32_y", k_cols_tma<L, false>, items, zs_smem<L>(), my, nkb, items, tw,
                                  ctx->d_err)));
    return launch_persistent<L>(ctx, "fft_f32_z", k_cols_tma<L, true>, items, zs_smem<L>(), mz, nkb, items, tw,
                                ctx->d_err);
  } else {
    const float th = (float)phase1;
    const typename GreenSink<L>::Args args = {srcF, ref_compat, th, (float)(phase1 - (double)th), dw, dwl};
    return f_cols_sink<L, GreenSink<L>>(ctx, "gw_z_accumulate_fp32", srcF, tw, args, 0);
  }
}

}  // namespace

// 16..512: the sizes the tests and the benchmark run; larger N keep cuFFT
bool axg_ff_fft_supported(int n) { return n >= 16 && n <= 512 && (n & (n - 1)) == 0; }

bool axg_ff_use(int n) {
  const char *env = std::getenv("AXG_FFT_FF");
  return axg_ff_fft_supported(n) && !(env && env[0] == '0');
}

namespace {
int ensure_twiddles(axg_ctx *ctx, int n) {
  if (ctx->ff_tw_n != n) {
    axg_free(ctx, (void **)&ctx->ff_tw);
    ctx->ff_tw_n = 0;
    // W_n^k = exp(-2 pi i k / n), k < n / 2, split into float-float on the host
    std::vector<float> h((size_t)n / 2 * 4);
    const double two_pi = 6.283185307179586476925286766559;
    for (int k = 0; k < n / 2; ++k) {
      const double c = std::cos(two_pi * k / n), s = -std::sin(two_pi * k / n);
      const float ch = (float)c, sh = (float)s;
      h[4 * k + 0] = ch;
      h[4 * k + 1] = (float)(c - (double)ch);
      h[4 * k + 2] = sh;
      h[4 * k + 3] = (float)(s - (double)sh);
    }
    AXG_TRY(axg_alloc(ctx, (void **)&ctx->ff_tw, h.size() * sizeof(float), "FFT twiddles"));
    AXG_CUDA_TRY(ctx, cudaMemcpy(ctx->ff_tw, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
    ctx->ff_tw_n = n;
  }
  return AXG_OK;
}
}  // namespace

namespace {
template <typename Load>
int z2z_n(axg_ctx *ctx, const Load &in, double2 *data, int n, int inverse, bool keep_ff) {
  if (!axg_ff_fft_supported(n)) return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  AXG_TRY(ensure_twiddles(ctx, n));
  const float4 *tw = reinterpret_cast<const float4 *>(ctx->ff_tw);
#define AXG_FF_Z2Z(L)                                                              \
  case L:                                                                          \
    return inverse ? z2z_t<L, true, Load>(ctx, in, data, tw, keep_ff) : z2z_t<L, false, Load>(ctx, in, data, tw, keep_ff);
  switch (n) {
    AXG_FF_Z2Z(16)
    AXG_FF_Z2Z(32)
    AXG_FF_Z2Z(64)
    AXG_FF_Z2Z(128)
    AXG_FF_Z2Z(256)
    AXG_FF_Z2Z(512)
    default: return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  }
#undef AXG_FF_Z2Z
}

template <typename Load>
int d2z_n(axg_ctx *ctx, const Load &in, double2 *out, int n, int batch, bool keep_ff) {
  if (!axg_ff_fft_supported(n)) return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  AXG_TRY(ensure_twiddles(ctx, n));
  const float4 *tw = reinterpret_cast<const float4 *>(ctx->ff_tw);
  switch (n) {
    case 16: return d2z_t<16>(ctx, in, out, batch, tw, keep_ff);
    case 32: return d2z_t<32>(ctx, in, out, batch, tw, keep_ff);
    case 64: return d2z_t<64>(ctx, in, out, batch, tw, keep_ff);
    case 128: return d2z_t<128>(ctx, in, out, batch, tw, keep_ff);
    case 256: return d2z_t<256>(ctx, in, out, batch, tw, keep_ff);
    case 512: return d2z_t<512>(ctx, in, out, batch, tw, keep_ff);
    default: return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  }
}
}  // namespace

int axg_ff_z2z(axg_ctx *ctx, double2 *data, int n, int inverse, bool keep_ff) {
  return z2z_n(ctx, LoadComplex{data}, data, n, inverse, keep_ff);
}

int axg_ff_z2z_masked(axg_ctx *ctx, const void *field, bool fp32, const int8_t *flags, double2 *out, int n,
                      int inverse) {
  if (fp32) return z2z_n(ctx, LoadMasked<float2>{(const float2 *)field, flags}, out, n, inverse, true);
  return z2z_n(ctx, LoadMasked<double2>{(const double2 *)field, flags}, out, n, inverse, true);
}

int axg_ff_d2z(axg_ctx *ctx, const double *in, double2 *out, int n, int batch, bool keep_ff) {
  return d2z_n(ctx, LoadReals{in}, out, n, batch, keep_ff);
}

int axg_ff_d2z_window(axg_ctx *ctx, const int8_t *flags, double2 *out, int n) {
  return d2z_n(ctx, LoadWindow{flags}, out, n, 1, true);
}

bool axg_gw_fused_f32(int n) { return axg_ff_fft_supported(n) && n > kGreenUnfused; }

int axg_gw_source_accumulate_f32(axg_ctx *ctx, const float2 *phi, float2 *srcF, int n, float scale, double phase1,
                                 float dw, float dwl, int ref_compat) {
  if (!axg_ff_fft_supported(n)) return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "FP32 source transform size");
  AXG_TRY(ensure_twiddles(ctx, n));
  const float4 *tw = reinterpret_cast<const float4 *>(ctx->ff_tw);
  switch (n) {
    case 16: return gws_accumulate_t<16>(ctx, phi, srcF, scale, phase1, dw, dwl, ref_compat, tw);
    case 32: return gws_accumulate_t<32>(ctx, phi, srcF, scale, phase1, dw, dwl, ref_compat, tw);
    case 64: return gws_accumulate_t<64>(ctx, phi, srcF, scale, phase1, dw, dwl, ref_compat, tw);
    case 128: return gws_accumulate_t<128>(ctx, phi, srcF, scale, phase1, dw, dwl, ref_compat, tw);
    case 256: return gws_accumulate_t<256>(ctx, phi, srcF, scale, phase1, dw, dwl, ref_compat, tw);
    case 512: return gws_accumulate_t<512>(ctx, phi, srcF, scale, phase1, dw, dwl, ref_compat, tw);
    default: return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "FP32 source transform size");
  }
}

int axg_gw_source_d2z_ff(axg_ctx *ctx, const double2 *phi, double d, double inv_d, int d_pow2, double2 *out, int n,
                         bool keep_ff) {
  if (!axg_ff_fft_supported(n)) return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  AXG_TRY(ensure_twiddles(ctx, n));
  const float4 *tw = reinterpret_cast<const float4 *>(ctx->ff_tw);
  switch (n) {
    case 16: return ff_gws_d2z_t<16>(ctx, phi, d, inv_d, d_pow2, out, tw, keep_ff);
    case 32: return ff_gws_d2z_t<32>(ctx, phi, d, inv_d, d_pow2, out, tw, keep_ff);
    case 64: return ff_gws_d2z_t<64>(ctx, phi, d, inv_d, d_pow2, out, tw, keep_ff);
    case 128: return ff_gws_d2z_t<128>(ctx, phi, d, inv_d, d_pow2, out, tw, keep_ff);
    case 256: return ff_gws_d2z_t<256>(ctx, phi, d, inv_d, d_pow2, out, tw, keep_ff);
    case 512: return ff_gws_d2z_t<512>(ctx, phi, d, inv_d, d_pow2, out, tw, keep_ff);
    default: return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  }
}

int axg_uij_power_f32(axg_ctx *ctx, const float *u, const float *ud, const float *cu, float tau, float2 *F, int n,
                      double dwav, const int16_t *tab, int nb, double *numer, double *denom) {
  if (!axg_ff_fft_supported(n)) return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "FP32 u_ij transform size");
  AXG_TRY(ensure_twiddles(ctx, n));
  const float4 *tw = reinterpret_cast<const float4 *>(ctx->ff_tw);
  switch (n) {
    case 16: return uij_power_t<16>(ctx, u, ud, cu, tau, F, dwav, tab, nb, numer, denom, tw);
    case 32: return uij_power_t<32>(ctx, u, ud, cu, tau, F, dwav, tab, nb, numer, denom, tw);
    case 64: return uij_power_t<64>(ctx, u, ud, cu, tau, F, dwav, tab, nb, numer, denom, tw);
    case 128: return uij_power_t<128>(ctx, u, ud, cu, tau, F, dwav, tab, nb, numer, denom, tw);
    case 256: return uij_power_t<256>(ctx, u, ud, cu, tau, F, dwav, tab, nb, numer, denom, tw);
    case 512: return uij_power_t<512>(ctx, u, ud, cu, tau, F, dwav, tab, nb, numer, denom, tw);
    default: return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "FP32 u_ij transform size");
  }
}

int axg_uij_d2z_ff(axg_ctx *ctx, const double *u, const double *ud, double tau, double2 *out, int n) {
  if (!axg_ff_fft_supported(n)) return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  AXG_TRY(ensure_twiddles(ctx, n));
  const float4 *tw = reinterpret_cast<const float4 *>(ctx->ff_tw);
  switch (n) {
    case 16: return ff_uij_d2z_t<16>(ctx, u, ud, tau, out, tw);
    case 32: return ff_uij_d2z_t<32>(ctx, u, ud, tau, out, tw);
    case 64: return ff_uij_d2z_t<64>(ctx, u, ud, tau, out, tw);
    case 128: return ff_uij_d2z_t<128>(ctx, u, ud, tau, out, tw);
    case 256: return ff_uij_d2z_t<256>(ctx, u, ud, tau, out, tw);
    case 512: return ff_uij_d2z_t<512>(ctx, u, ud, tau, out, tw);
    default: return axg_set_error(ctx, AXG_ERR_UNSUPPORTED, "float-float FFT size");
  }
}
