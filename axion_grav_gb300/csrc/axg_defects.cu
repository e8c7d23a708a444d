// axg_defects.cu -- defect identification on the GPU (defects_3d.f90).
//
// This translation unit is compiled with -fmad=false: every floating-point
// expression below rounds each operation separately, exactly as IEEE host C
// does without contraction, and the FP64 atan2 / sin / cos are the
// deterministic versions of axg_detmath.h.  Cell flags, counts, plaquette
// windings and every per-cell fit (position, direction, length, velocity,
// wall area) are therefore bit-identical to a host evaluation of the same
// formulas.  FP32 phases serve only as a filter that decides the
// cells whose outcome cannot change within their error bound; all other
// cells go through the FP64 path.
//
// Passes (all O(N^3) passes are HBM-streaming, the fits are sparse):
//   1. classify  : FP32 phases of a tile of phi in shared memory, 8 corner
//                  phases, sort, largest circular gap -> int8 flags and
//                  counts (defects_3d.f90:67-103, 309-349).
//                  Filtered: the FP32 phases are within 1e-6 of the FP64
//                  ones, and sorting moves no value by more than that, so a
//                  cell whose every decision (wall gap against wrap gap,
//                  largest gap against pi and 7 pi / 4) clears a 2e-5
//                  margin has the FP64 flags; any other cell is redone from
//                  phi with the deterministic FP64 atan2, as on the host.
//   2. winding   : three plaquettes per site, filtered the same way (a
//                  corner difference within the margin of +-pi is redone in
//                  FP64)
//   3. compaction: string and wall cells listed in cell order
//   4. fits      : string cells by groups of eight lanes -- the search
//                  of position_string (1001 random starts, screened in FP32,
//                  + Nelder-Mead, defects_3d.f90:435-603; the chi2 in
//                  float-float on the FP32 pipes, axg_ffchi2.h), string_length
//                  (1027-1056), velocity_string (605-692), position_wall
//                  (1058-1233)
//   5. sums      : add_string_length / add_wall_area without grouping
#include <cmath>

#include "axg_detmath.h"
#include "axg_ffchi2.h"
#include "axg_internal.h"

namespace {

constexpr double kRefPi = 3.14159265359;
constexpr double kRefTwoPi = 2 * kRefPi;
constexpr double kStringPhdiff = kRefPi;
constexpr double kRemovalPhdiff = 7 * kRefPi / 4;
constexpr int kMaxIter = 1000;
constexpr int kNumSimp = 4;

// The FP64 value of site s.  comp: the Kahan compensation of an FP32-mixed
// phi (else null); the value is then (double)v - (double)c, the snapshot
// axg_download returns, so the FP64 decisions are those of the host's
// classification of the downloaded field.
template <typename V>
__device__ __forceinline__ void load_c(const V *a, const V *comp, int64_t s, double &re, double &im) {
  const V v = a[s];
  re = (double)v.x;
  im = (double)v.y;
  if (comp) {
    const V c = comp[s];
    re = re - (double)c.x;
    im = im - (double)c.y;
  }
}

// FP32 phase of a site, within 1e-6 of the FP64 one, or `unknown` (then every
// cell touching the site is decided in FP64).  n / d, the smaller over the
// larger component, goes through Hastings' eight-term arctangent (Abramowitz
// and Stegun 4.4.49: 2e-8 on [0, 1]); the fast quotient, the rounding of the
// ratio and of the quadrant sums stay below 4e-7, and 2.4e-7 more for an FP64
// field's truncation to float.
// About 20 instructions against some 40 of atan2f, whose care for special
// operands the range test replaces: outside [2^-100, 2^120] of the larger
// component, and for zeros, infinities and NaN (in either component: d is then
// NaN), the phase is unknown.
__device__ __forceinline__ float max_nan(float a, float b) {  // fmaxf drops a NaN
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float phase_fast(float re, float im, float unknown) {
  const float ar = fabsf(re), ai = fabsf(im), d = max_nan(ar, ai), q = __fdividef(fminf(ar, ai), d), t = q * q;
  float p = fmaf(t, 0.0028662257f, -0.0161657367f);
  p = fmaf(t, p, 0.0429096138f);
  p = fmaf(t, p, -0.0752896400f);
  p = fmaf(t, p, 0.1065626393f);
  p = fmaf(t, p, -0.1420889944f);
  p = fmaf(t, p, 0.1999355085f);
  p = fmaf(t, p, -0.3333314528f);
  p = fmaf(t * p, q, q);
  if (ai > ar) p = 1.5707963267948966f - p;
  if (re < 0.0f) p = 3.1415926535897932f - p;
  return d > 7.8886091e-31f && d < 1.3292280e36f ? copysignf(p, im) : unknown;
}
__device__ __forceinline__ float phase_of(float2 v, float unknown) { return phase_fast(v.x, v.y, unknown); }
// A double truncated to float on the integer pipes (the conversion and FP64
// comparisons run on the FP64 pipe): within 2^-23 of its size, a value below
// FP32's normal range as zero of its sign (phase_fast's range test then knows
// whether the other component is large enough for that), above it infinite.
__device__ __forceinline__ float f32_truncated(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x), m = h & 0x7fffffffu;
  uint32_t f = (m << 3 | l >> 29) - (896u << 23);
  if (m < (897u << 20)) f = 0u;
  if (m >= (1151u << 20)) f = m > 0x7ff00000u ? 0x7fc00000u : 0x7f800000u;
  return __uint_as_float(f | (h & 0x80000000u));
}
__device__ __forceinline__ float phase_of(double2 v, float unknown) {
  return phase_fast(f32_truncated(v.x), f32_truncated(v.y), unknown);
}

__device__ __forceinline__ void cswap(double &a, double &b) {
  const double lo = a < b ? a : b;
  const double hi = a < b ? b : a;
  a = lo;
  b = hi;
}

// Batcher-style 19-comparator sorting network for 8 values (ascending).
__device__ __forceinline__ void sort8(double v[8]) {
  cswap(v[0], v[1]); cswap(v[2], v[3]); cswap(v[4], v[5]); cswap(v[6], v[7]);
  cswap(v[0], v[2]); cswap(v[1], v[3]); cswap(v[4], v[6]); cswap(v[5], v[7]);
  cswap(v[1], v[2]); cswap(v[5], v[6]); cswap(v[0], v[4]); cswap(v[3], v[7]);
  cswap(v[1], v[5]); cswap(v[2], v[6]);
  cswap(v[1], v[4]); cswap(v[3], v[6]);
  cswap(v[2], v[4]); cswap(v[3], v[5]);
  cswap(v[3], v[4]);
}

__device__ __forceinline__ int64_t corner(int n, int ix, int iy, int iz, int c) {
  const int dx = c & 1, dy = (c >> 1) & 1, dz = (c >> 2) & 1;
  const int x = ix + dx == n ? 0 : ix + dx, y = iy + dy == n ? 0 : iy + dy,
            z = iz + dz == n ? 0 : iz + dz;
  return ((int64_t)z * n + y) * n + x;
}

// id_with_phase (defects_3d.f90:309-349) on sorted phases
__device__ __forceinline__ int8_t classify_sorted(const double pht[8], int which) {
  int8_t flag = 0;
  const double t = pht[0] - pht[7] + kRefTwoPi;
  double tmax = pht[1] - pht[0];
#pragma unroll
  for (int k = 1; k < 7; ++k) {
    const double g = pht[k + 1] - pht[k];
    tmax = g > tmax ? g : tmax;
  }
  if ((which & AXG_F_ID_WALLS) && tmax > t) {
    flag += 2;
  } else {
    tmax = t > tmax ? t : tmax;
  }
  if ((which & AXG_F_ID_STRINGS) && tmax < kStringPhdiff) flag += 1;
  if ((which & AXG_F_SPEC_EST) && tmax < kRemovalPhdiff) flag += 4;
  return flag;
}

// Adds the block's three tallies (10 bits each of the threads' packed
// counts) to dst: 3 global atomics per block.
__device__ __forceinline__ void block_tally3(unsigned packed, unsigned long long *dst) {
  __shared__ unsigned sh[3];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  if (tid < 3) sh[tid] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const unsigned c = __reduce_add_sync(0xffffffffu, (packed >> (10 * k)) & 0x3ffu);
    if ((tid & 31) == 0 && c) atomicAdd(&sh[k], c);
  }
  __syncthreads();
  if (tid < 3 && sh[tid]) atomicAdd(&dst[tid], (unsigned long long)sh[tid]);
}

// >> 4 (2 x 1e-6 phase error + FP32 rounding of a gap).  The phase error
// budget of 1e-6 covers phase_fast and, for an FP32-mixed field, the
// Kahan compensation the FP32 phase leaves out (|c| <= ulp(phi) / 2, so
// <= 1.2e-7 rad).
constexpr float kMargin = 2e-5f;

__device__ __forceinline__ void cswapf(float &a, float &b) {
  const float lo = fminf(a, b), hi = fmaxf(a, b);
  a = lo;
  b = hi;
}
// four values in ascending order (5 comparators)
__device__ __forceinline__ void sort4f(float v[4]) {
  cswapf(v[0], v[1]); cswapf(v[2], v[3]);
  cswapf(v[0], v[2]); cswapf(v[1], v[3]);
  cswapf(v[1], v[2]);
}
// two sorted fours into eight (Batcher's odd-even merge, 9 comparators)
__device__ __forceinline__ void merge44f(const float a[4], const float b[4], float v[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = a[i];
    v[4 + i] = b[i];
  }
  cswapf(v[0], v[4]); cswapf(v[1], v[5]); cswapf(v[2], v[6]); cswapf(v[3], v[7]);
  cswapf(v[2], v[4]); cswapf(v[3], v[5]);
  cswapf(v[1], v[2]); cswapf(v[3], v[4]); cswapf(v[5], v[6]);
}

// id_with_phase on FP32 phases; false when a decision lies inside the margin
__device__ __forceinline__ bool classify_sorted_f(const float p[8], int which, int &flag) {
  flag = 0;
  const float t = p[0] - p[7] + (float)kRefTwoPi;
  float tmax = p[1] - p[0];
#pragma unroll
  for (int k = 1; k < 7; ++k) tmax = fmaxf(tmax, p[k + 1] - p[k]);
  bool sure = true;
  if (which & AXG_F_ID_WALLS) {
    sure = fabsf(tmax - t) >= kMargin;
    if (tmax > t) flag += 2;
    else tmax = fmaxf(t, tmax);
  } else {
    tmax = fmaxf(t, tmax);
  }
  if (which & AXG_F_ID_STRINGS) {
    sure = sure && fabsf(tmax - (float)kStringPhdiff) >= kMargin;
    if (tmax < (float)kStringPhdiff) flag += 1;
  }
  if (which & AXG_F_SPEC_EST) {
    sure = sure && fabsf(tmax - (float)kRemovalPhdiff) >= kMargin;
    if (tmax < (float)kRemovalPhdiff) flag += 4;
  }
  return sure;
}

template <typename V>
__device__ __forceinline__ double phase64(const V *phi, const V *comp, int64_t s) {
  double re, im;
  load_c(phi, comp, s, re, im);
  return axd_atan2(im, re);
}

// The deterministic FP64 phase of every site, for the fits: each fitted cell
// reads its eight corners here instead of forming them (a string or wall
// cell's corners are shared with its neighbours, and the fits ran them as
// divergent FP64 chains at the start of every cell).
template <typename V>
__global__ void k_phase64_all(const V *__restrict__ phi, const V *__restrict__ cphi, int64_t n3,
                              double *__restrict__ ph) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n3; s += stride)
    ph[s] = phase64(phi, cphi, s);
}

// The cell passes.  A CTA owns 32 x kCellY columns of cells and walks zc
// planes: each plane of (32 + 1) x (kCellY + 1) phases is formed from phi in
// shared memory (the next two planes' phi are in flight), a thread reads the
// four corners of its cell in that plane and keeps those of the plane below.
// One read of phi and one write of the result; phases are never stored.
// cell(x, y, z, lower, upper): corner dy 2 + dx of the cell's lower and upper
// plane, returns the cell's packed counts, or a negative value when FP32
// cannot decide it.  Those cells are queued and decided at the end by
// exact(x, y, z, corners) from their FP64 phases, 32 cells at a time with a
// thread per corner phase (done where they turn up, one lane of a warp at a
// time, they took half of a 64^3 pass, and their FP64 chains held registers
// throughout the march; with a thread per cell a single queued cell took 14 us).
//
// Before, the phases went through HBM (12 + 4 B a site) and each cell loaded
// its eight corners with 64-bit index divisions, ~390 instructions a cell; now
// it is ~155, and the issue slots bound the passes (76 and 85 % busy under
// ncu).  512^3 FP32: classification 1.69 -> 0.66 ms, winding 1.94 -> 0.57;
// 128^3: 66 -> 23 and 54 -> 17 us.  3 to 6 CTAs per SM measured 0.67-0.76 ms.
constexpr int kCellX = 32, kCellY = 8, kCellZ = 32;  // at most kCellZ planes: the queue holds every cell of the CTA
template <typename V, typename Cell, typename Exact>
__device__ __forceinline__ unsigned cell_march(const V *__restrict__ phi, const V *__restrict__ cphi, int n, int zc,
                                               float unknown, Cell cell, Exact exact) {
  constexpr int W = kCellX + 1, H = kCellY + 1, NT = kCellX * kCellY;
  __shared__ float ph[2][H * W];
  __shared__ uint16_t queue[NT * kCellZ];
  __shared__ double exact_ph[NT];
  __shared__ int queued;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kCellX + tx;
  const int x0 = blockIdx.x * kCellX, y0 = blockIdx.y * kCellY, z0 = blockIdx.z * zc;
  const int nz = min(zc, n - z0);
  auto wrap = [n](int i) { return i >= n ? i - n : i; };
  // a thread's own site and, for the first W + H - 1 threads, one of the
  // right column and lower row; past the lattice's edge both repeat site 0
  const int x = x0 + tx, y = y0 + ty;
  const bool live = x < n && y < n, halo = tid < W + H - 1;
  const int hx = tid < W ? tid : W - 1, hy = tid < W ? H - 1 : tid - W;
  const int own = wrap(min(y, n)) * n + wrap(min(x, n)), rim = wrap(min(y0 + hy, n)) * n + wrap(min(x0 + hx, n));
  const int64_t n2 = (int64_t)n * n;
  // planes z0 .. z0 + nz; the last one is plane 0 when the walk ends at n
  const V *pa = phi + z0 * n2 + own, *pb = phi + z0 * n2 + rim;
  const int64_t last = z0 + nz == n ? -(int64_t)(n - 1) * n2 : n2;  // from plane z0 + nz - 1 to the last
  V a = pa[0], b = a, a1, b1;
  if (halo) b = pb[0];
  auto advance = [&](int k) {  // a1, b1: plane z0 + k
    const int64_t step = k == nz ? last : n2;
    pa += step;
    pb += step;
    a1 = *pa;
    if (halo) b1 = *pb;
  };
  b1 = b;
  advance(1);
  if (tid == 0) queued = 0;
  float lo[4];
  unsigned counts = 0;
  const int slot = ty * W + tx, hslot = hy * W + hx;
#pragma unroll 2
  for (int k = 0; k <= nz; ++k) {
    float *s = ph[k & 1];
    s[slot] = phase_of(a, unknown);
    if (halo) s[hslot] = phase_of(b, unknown);
    a = a1;
    b = b1;
    if (k + 2 <= nz) advance(k + 2);
    __syncthreads();
    const float *c = s + slot;
    const float hi[4] = {c[0], c[1], c[W], c[W + 1]};
    if (k > 0 && live) {
      const int r = cell(x, y, z0 + k - 1, lo, hi);
      if (r >= 0) {
        counts += (unsigned)r;
      } else {
        queue[atomicAdd(&queued, 1)] = (uint16_t)((k - 1) * NT + tid);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) lo[i] = hi[i];
  }
  __syncthreads();
  for (int q0 = 0; q0 < queued; q0 += NT / 8) {
    auto site = [&](int q, int &cx, int &cy, int &cz) {
      const int e = queue[q];
      cx = x0 + e % kCellX;
      cy = y0 + e / kCellX % kCellY;
      cz = z0 + e / NT;
    };
    int cx, cy, cz;
    if (q0 + tid / 8 < queued) {
      site(q0 + tid / 8, cx, cy, cz);
      exact_ph[tid] = phase64(phi, cphi, corner(n, cx, cy, cz, tid & 7));
    }
    __syncthreads();
    if (tid < NT / 8 && q0 + tid < queued) {
      site(q0 + tid, cx, cy, cz);
      double d[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) d[c] = exact_ph[8 * tid + c];
      counts += exact(cx, cy, cz, d);
    }
    __syncthreads();
  }
  static_assert(NT >= W + H - 1, "one halo site per thread");
  static_assert(NT * kCellZ <= 65536, "queue entries of 16 bits");
  return counts;
}

// WHICH: the flags asked for, or -1 for those of `flags_wanted`
template <typename V, int WHICH>
__global__ void __launch_bounds__(kCellX *kCellY, 5) k_classify(const V *__restrict__ phi,
                                                                const V *__restrict__ cphi, int n, int zc,
                                                                int flags_wanted,
                                                                int8_t *__restrict__ flags,
                                                                unsigned long long *__restrict__ counts) {
  const int which = WHICH >= 0 ? WHICH : flags_wanted;
  constexpr float kUnknown = 1e30f;  // sorts last
  float sorted[4];                   // the lower plane's corners in order, from the cell below
  const int64_t n2 = (int64_t)n * n;
  int8_t *dst = flags + ((int64_t)blockIdx.z * zc * n + blockIdx.y * kCellY + threadIdx.y) * n + blockIdx.x * kCellX +
                threadIdx.x;
  auto pack = [](int flag) { return (flag & 1) | (flag & 2) << 9 | (flag & 4) << 18; };
  const int zfirst = blockIdx.z * zc;
  auto cell = [&](int, int, int z, const float lo[4], const float hi[4]) {
    if (z == zfirst) {
#pragma unroll
      for (int i = 0; i < 4; ++i) sorted[i] = lo[i];
      sort4f(sorted);
    }
    float up[4] = {hi[0], hi[1], hi[2], hi[3]}, v[8];
    sort4f(up);
    merge44f(sorted, up, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) sorted[i] = up[i];
    int f;
    const bool sure = classify_sorted_f(v, which, f) && v[7] < 4.0f;
    *dst = (int8_t)f;
    dst += n2;
    return sure ? pack(f) : -1;
  };
  auto exact = [&](int x, int y, int z, double d[8]) {  // the FP64 classification of the host
    sort8(d);
    const int f = classify_sorted(d, which);
    flags[((int64_t)z * n + y) * n + x] = (int8_t)f;
    return (unsigned)pack(f);
  };
  block_tally3(cell_march(phi, cphi, n, zc, kUnknown, cell, exact), counts);
}

__device__ __forceinline__ double wrapd(double d) {
  const double pi = AXD_PI_HI, tp = 2 * AXD_PI_HI;
  if (d > pi) return d - tp;
  if (d <= -pi) return d + tp;
  return d;
}
__device__ __forceinline__ bool pierced(double a, double b, double c, double d) {
  double w = wrapd(b - a);
  w = w + wrapd(c - b);
  w = w + wrapd(d - c);
  w = w + wrapd(a - d);
  return w > AXD_PI_HI || w < -AXD_PI_HI;
}

// Plaquette winding.  The raw phase differences around a plaquette sum to
// zero, so the wrapped ones sum to -2 pi times the sum of the links' wrap
// numbers rint(d / 2 pi), and the plaquette is pierced when those do not
// cancel.  A link's number is the FP64 one unless |d| lies within kMargin of
// pi; then, or with a phase unknown, the site's plaquettes are redone in FP64.
template <typename V>
__global__ void __launch_bounds__(kCellX *kCellY, 5) k_winding(const V *__restrict__ phi,
                                                               const V *__restrict__ cphi, int n, int zc,
                                                               unsigned long long *__restrict__ counts) {
  constexpr float kInv = 0.15915494309189534f, kBig = 12582912.0f;  // 1 / 2 pi; 1.5 2^23: adding it rounds to an integer
  constexpr float kSure = 0.5f - kMargin * kInv;
  float kx[2] = {0.f, 0.f}, ky[2] = {0.f, 0.f};  // the lower plane's links: x at y, y + 1; y at x, x + 1
  float far = 0.f;                               // the largest |d / 2 pi - rint| among them
  const int zfirst = blockIdx.z * zc;
  auto pack = [](unsigned hit) { return (int)((hit & 1u) | (hit & 2u) << 9 | (hit & 4u) << 18); };
  auto link = [&](float a, float b, float &m) {
    const float t = (b - a) * kInv, k = (t + kBig) - kBig;
    m = fmaxf(m, fabsf(t - k));
    return k;
  };
  auto plane = [&](const float p[4], float lx[2], float ly[2]) {
    float m = 0.f;
    lx[0] = link(p[0], p[1], m);
    lx[1] = link(p[2], p[3], m);
    ly[0] = link(p[0], p[2], m);
    ly[1] = link(p[1], p[3], m);
    return m;
  };
  auto cell = [&](int, int, int z, const float lo[4], const float hi[4]) {
    if (z == zfirst) far = plane(lo, kx, ky);
    float ux[2], uy[2];
    const float up = plane(hi, ux, uy);
    float m = fmaxf(far, up);
    const float kz = link(lo[0], hi[0], m), kzx = link(lo[1], hi[1], m), kzy = link(lo[2], hi[2], m);
    const float wx = (ky[0] + kzy) - (uy[0] + kz), wy = (kz + ux[0]) - (kzx + kx[0]), wz = (kx[0] + ky[1]) - (kx[1] + ky[0]);
    const unsigned hit = (wx != 0.f ? 1u : 0u) | (wy != 0.f ? 2u : 0u) | (wz != 0.f ? 4u : 0u);
    const float s = (wx + wy) + wz;  // NaN where a phase is
    const bool sure = m <= kSure && s == s;
    far = up;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      kx[i] = ux[i];
      ky[i] = uy[i];
    }
    return sure ? pack(hit) : -1;
  };
  auto exact = [&](int, int, int, const double p[8]) {  // corner c = dx + 2 dy + 4 dz
    return (unsigned)pack((pierced(p[0], p[2], p[6], p[4]) ? 1u : 0u) | (pierced(p[0], p[4], p[5], p[1]) ? 2u : 0u) |
                          (pierced(p[0], p[1], p[3], p[2]) ? 4u : 0u));
  };
  block_tally3(cell_march(phi, cphi, n, zc, __int_as_float(0x7fc00000), cell, exact), counts);
}

// ---------------- compaction in cell order ----------------
constexpr int kChunk = 2048;  // cells per block
constexpr int kCThreads = 256;  // 8 consecutive cells per thread

__global__ void k_block_count(const int8_t *__restrict__ flags, int64_t n3, int *__restrict__ cs,
                              int *__restrict__ cw) {
  const int64_t b0 = (int64_t)blockIdx.x * kChunk + threadIdx.x * 8;
  int ns = 0, nw = 0;
  for (int k = 0; k < 8; ++k) {
    const int64_t s = b0 + k;
    if (s < n3) {
      const int8_t f = flags[s];
      ns += (f & 1) != 0;
      nw += (f & 2) != 0;
    }
  }
  __shared__ int sh[2][kCThreads];
  sh[0][threadIdx.x] = ns;
  sh[1][threadIdx.x] = nw;
  __syncthreads();
  for (int o = kCThreads / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + o];
      sh[1][threadIdx.x] += sh[1][threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    cs[blockIdx.x] = sh[0][0];
    cw[blockIdx.x] = sh[1][0];
  }
}

// exclusive scan of nb block counts (single block, sequential over chunks)
__global__ void k_scan_blocks(int *__restrict__ cs, int *__restrict__ cw, int nb) {
  __shared__ long long carry[2];
  __shared__ int sh[2][1024];
  if (threadIdx.x == 0) carry[0] = carry[1] = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + threadIdx.x;
    const int a = i < nb ? cs[i] : 0, b = i < nb ? cw[i] : 0;
    sh[0][threadIdx.x] = a;
    sh[1][threadIdx.x] = b;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      int x0 = 0, x1 = 0;
      if ((int)threadIdx.x >= o) {
        x0 = sh[0][threadIdx.x - o];
        x1 = sh[1][threadIdx.x - o];
      }
      __syncthreads();
      sh[0][threadIdx.x] += x0;
      sh[1][threadIdx.x] += x1;
      __syncthreads();
    }
    if (i < nb) {
      cs[i] = (int)(carry[0] + sh[0][threadIdx.x] - a);
      cw[i] = (int)(carry[1] + sh[1][threadIdx.x] - b);
    }
    __syncthreads();
    if (threadIdx.x == 1023) {
      carry[0] += sh[0][1023];
      carry[1] += sh[1][1023];
    }
    __syncthreads();
  }
}

__global__ void k_compact(const int8_t *__restrict__ flags, int64_t n3, const int *__restrict__ offs,
                          const int *__restrict__ offw, int64_t *__restrict__ scell,
                          int64_t *__restrict__ wcell) {
  const int64_t b0 = (int64_t)blockIdx.x * kChunk + threadIdx.x * 8;
  int ns = 0, nw = 0;
  int8_t f[8];
  for (int k = 0; k < 8; ++k) {
    const int64_t s = b0 + k;
    f[k] = s < n3 ? flags[s] : 0;
    ns += (f[k] & 1) != 0;
    nw += (f[k] & 2) != 0;
  }
  __shared__ int sh[2][kCThreads];
  sh[0][threadIdx.x] = ns;
  sh[1][threadIdx.x] = nw;
  __syncthreads();
  for (int o = 1; o < kCThreads; o <<= 1) {
    int x0 = 0, x1 = 0;
    if ((int)threadIdx.x >= o) {
      x0 = sh[0][threadIdx.x - o];
      x1 = sh[1][threadIdx.x - o];
    }
    __syncthreads();
    sh[0][threadIdx.x] += x0;
    sh[1][threadIdx.x] += x1;
    __syncthreads();
  }
  int ps = offs[blockIdx.x] + sh[0][threadIdx.x] - ns;
  int pw = offw[blockIdx.x] + sh[1][threadIdx.x] - nw;
  for (int k = 0; k < 8; ++k) {
    if (f[k] & 1) scell[ps++] = b0 + k;
    if (f[k] & 2) wcell[pw++] = b0 + k;
  }
}

// ---------------- per-cell fits ----------------
// defects_3d.f90:1027-1056
__device__ double string_length(const double pos[3], const double dir[3]) {
  const double atmax = 0.867, atmax0 = 0.86602540378378444;
  double tp = atmax, tn = -atmax;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j <= 1; ++j) {
      double w = j - 0.5;
      w = w - pos[i];
      if (fabs(w) > atmax * fabs(dir[i])) continue;
      const double t = w / dir[i];
      if (t > 0) {
        if (t < tp) tp = t;
      } else {
        if (t > tn) tn = t;
      }
    }
  if (tp < atmax0 && tn > -atmax0) return tp - tn;
  return 0.0;
}

// ---- string fits (defects_3d.f90:435-603) ----
//
// The fit of one string cell is a random search over 1001 starts, which keeps
// the kNumSimp + 1 best, followed by a Nelder-Mead simplex of up to 1000
// iterations (tol 0.05 on chi2).  In evolved fields about two thirds of the
// string cells never reach the tolerance and run all 1000 iterations, one or
// two chi2 after another: a cell is a serial chain of about 2000 chi2, each of
// 8 atan2 (one per corner) and 2 sin / cos.  With one lane per cell the chain
// took 57 ms whatever the lattice, lanes of a warp diverged over the search
// stages (12 of 32 active at 128^3), and every lane issued the FP64 work of
// its own simplex.
//
// Here eight lanes fit one cell, lane `sub` = corner `sub`.  A chi2 is one
// atan2 per lane; the terms go through shared memory and are added in the
// reference's corner order.  Lane sub also holds coordinate sub & 3 of every
// vertex (mu, phi, radius, angle), so the simplex arithmetic is one FP64
// operation where a lane with a whole vertex issued four.  chi2 values are
// kept as ordered integers (dkey): their comparisons stay off the FP64 pipe,
// which GB300 issues at 1/64 of the FP32 rate.  Three kernels, so that the
// lanes of a warp always run the same kind of work:
//   k_string_start   the random search, eight starts screened at a time;
//   k_string_simplex the simplex; groups take cells from a counter;
//   k_string_result  one thread per cell: length, velocity and output row.
// The whole search is bit-identical to the sequential one of the CPU
// restatement.  String fits, ms: 104.5 -> 36.8 at 128^3 (1.3e5 cells, FP32),
// 58.1 -> 12 at 64^3, 55 -> 5.2 at 32^3.  At 128^3 the issue slots bound it
// (ncu at 64^3: 68 % issue active, FP64 pipe 37 %; about 800 instructions per
// warp and chi2), on small lattices the chain of a cell.
constexpr int kGrp = 8;                 // lanes per cell
constexpr int kFitThreads = 128;        // 16 cells per CTA
constexpr int kIdle = 2;                // groups of a warp without work that end the eight-lane simplex
constexpr int kRounds = 4;              // random starts screened per lane before the next evaluations
constexpr int kFitStride = 5 * 4 + 5;   // doubles per cell of the simplex scratch: p[vertex][coordinate], chi2[vertex]
constexpr int64_t kFitChunk = 1 << 21;  // cells per pass of the three kernels (420 MB of scratch at most)
constexpr int64_t kFitChunkMin = 1 << 9;  // ... at least, where memory is short

// a double as an integer of the same order; -0 becomes +0.  An involution.
__device__ __forceinline__ long long dkey(double v) {
  const long long b = __double_as_longlong(v);
  return b == (long long)0x8000000000000000ULL ? 0 : b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double dkey_value(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}

// bounds of parameter k (mu, phi, radius, angle)
__device__ __forceinline__ double string_max(int k) {
  return k == 0 ? 1.0 : (k == 2 ? sqrt(3.0) / 2 : kRefPi);
}
__device__ __forceinline__ double string_min(int k) { return k == 0 ? -1.0 : (k == 2 ? 0.0 : -kRefPi); }

// Coordinate k of start point i of the random search (defects_3d.f90:
// 463-470): two uniforms per Philox draw, mapped onto the parameter box.
__device__ __forceinline__ double string_start(uint64_t seed, uint64_t cell, int i, int k) {
  const axd_u32x4 r = axd_draw(seed, 3u, (uint32_t)((i * 4 + k) >> 1), cell);
  const double x = (k & 1) ? axd_u01(r.v[2], r.v[3]) : axd_u01(r.v[0], r.v[1]);
  return string_max(k) * x + string_min(k) * (1 - x);
}

// A lower bound of the chi2 of start i from an FP32 evaluation, or -inf where
// the FP32 value cannot be bounded (a corner too close to the string axis for
// its angle to be resolved, or a phase difference within the error of the
// +-pi wrap).  The start is formed in FP32 too, from the top 32 bits of its
// uniforms: x and 1 - x each to 2^-25 relative and 2^-32 absolute, so mu to
// 2e-7, the angles to 7e-7, the radius to 1e-7, and sqrt(1 - mu^2) =
// 2 sqrt(x (1 - x)) to 4e-7 (x within 2^-20 of 0 or 1 is not screened).
// Error budget, all generous:
//   du, dv: those, __sincosf (absolute error 2^-21 on [-pi, pi]), products
//           and sums of terms below 2.4 in magnitude come to 3.1e-6:
//           |error| <= kDuv = 5e-6;
//   angle : the polynomial arctangent (Hastings' five terms, Abramowitz and
//           Stegun 4.4.47: 1.16e-5 on [0, 1]; ratio and quadrant sums in
//           FP32 below 6e-7) within kAng, plus the rotation of (du, dv) by an
//           error of kDuv at radius r: e = kAng + 2 kDuv / (r - 2 kDuv).
//           With atan2f the screens took 1.8 times the instructions, and a
//           bound 3e-4 tighter in chi2 saves no evaluation;
//   phase : FP32 rounding of ph, of the difference and of the wrap
//           constants, within kPh = 2e-6;
//   chi2  : a = <d^2> moves by at most (2 pi + E) E, b^2 = <d>^2 by at most
//           (2 pi + E + 2e-6)(E + 2e-6), FP32 summation by below 2e-5;
// and the total is doubled, plus 1e-4 (which also covers the 1e-14 between
// the FP64 chi2 and the float-float chi2 the search uses).
__device__ __forceinline__ float chi2_start_lower(const float phf[8], uint64_t seed, uint64_t cell, int i) {
  constexpr float kDuv = 5e-6f, kAng = 1.3e-5f, kPh = 2e-6f;
  constexpr float kPiF = (float)kRefPi, kTwoPiF = (float)kRefTwoPi;
  const axd_u32x4 r0 = axd_draw(seed, 3u, (uint32_t)(2 * i), cell), r1 = axd_draw(seed, 3u, (uint32_t)(2 * i + 1), cell);
  const uint32_t xm = r0.v[0];
  if (xm < 4096u || xm > 0xffffefffu) return -INFINITY;
  constexpr float k32 = 2.3283064365386963e-10f;  // 2^-32
  const float x0 = (float)xm * k32, y0 = (float)~xm * k32;
  const float mu = x0 - y0, sm = 2 * sqrtf(x0 * y0);
  const float ph = kTwoPiF * ((float)r0.v[2] * k32) - kPiF;
  const float rad = 0.86602540378443864676f * ((float)r1.v[0] * k32);
  const float ang = kTwoPiF * ((float)r1.v[2] * k32) - kPiF;
  float s4, c4, sp, cp;
  __sincosf(ang, &s4, &c4);
  __sincosf(ph, &sp, &cp);
  const float u0 = rad * c4, v0 = rad * s4;
  float a = 0.0f, b = 0.0f, rmin = INFINITY, wmin = INFINITY;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float x = (c & 1) - 0.5f, y = ((c >> 1) & 1) - 0.5f, z = (c >> 2) - 0.5f;
    const float du = -u0 + mu * (x * cp + y * sp) - z * sm;
    const float dv = -v0 - x * sp + y * cp;
    rmin = fminf(rmin, du * du + dv * dv);
    const float au = fabsf(du), av = fabsf(dv);
    const float q = __fdividef(fminf(au, av), fmaxf(au, av)), q2 = q * q;
    float at = fmaf(q2, 0.0208351f, -0.0851330f);
    at = fmaf(q2, at, 0.1801410f);
    at = fmaf(q2, at, -0.3302995f);
    at = q * fmaf(q2, at, 0.9998660f);
    if (av > au) at = 1.5707963267948966f - at;
    if (du < 0.0f) at = 3.1415926535897932f - at;
    float d = phf[c] - copysignf(at, dv);
    wmin = fminf(wmin, fabsf(fabsf(d) - kPiF));
    if (d >= kPiF)
      d = d - kTwoPiF;
    else if (d < -kPiF)
      d = d + kTwoPiF;
    a = a + d * d;
    b = b + d;
  }
  // one E for all corners, from the smallest radius
  const float r = sqrtf(rmin);
  if (!(r > 8 * kDuv)) return -INFINITY;
  const float E = kAng + kPh + 2 * kDuv / (r - 2 * kDuv);
  if (!(wmin > E + kPh)) return -INFINITY;
  a = a / 8;
  b = b / 8;
  const float tp = (float)kRefTwoPi;
  const float bound = 2 * ((tp + E) * E + (tp + E + 2e-6f) * (E + 2e-6f) + 2e-5f) + 1e-4f;
  return (a - b * b) - bound;
}

// sin (even lanes) or cos (odd lanes) of the reduced argument by the series of
// axd_ff_sincos: the coefficients of the lane's series, float-float for the
// first five terms and FP32 for the others, kept in registers.
struct LaneSeries {
  axd_ff k[5];
  float f[4];
  bool cosine;
  __device__ explicit LaneSeries(bool c) : cosine(c) {
    // (-1)^k / (2k+1)! and (-1)^k / (2k)!, as in axd_ff_sincos
    const float ks[9][2] = {{1.0f, 0.0f},
                            {-0.1666666716337204f, 4.967053879312289e-09f},
                            {0.008333333767950535f, -4.34617203337595e-10f},
                            {-0.00019841270113829523f, 2.725596874933456e-12f},
                            {2.7557318844628753e-06f, 3.793571224297229e-14f},
                            {-2.5052107943679403e-08f, 0.0f},
                            {1.6059044372074283e-10f, 0.0f},
                            {-7.647163609812713e-13f, 0.0f},
                            {2.8114573589663704e-15f, 0.0f}};
    const float kc[9][2] = {{1.0f, 0.0f},
                            {-0.5f, 0.0f},
                            {0.0416666679084301f, -1.2417634698280722e-09f},
                            {-0.0013888889225199819f, 3.3631094437103215e-11f},
                            {2.4801587642286904e-05f, -3.40699609366682e-13f},
                            {-2.755731998149713e-07f, 0.0f},
                            {2.0876755879584152e-09f, 0.0f},
                            {-1.147074536050896e-11f, 0.0f},
                            {4.7794772561329454e-14f, 0.0f}};
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      if (i < 5) k[i] = c ? axd_ff_mk(kc[i][0], kc[i][1]) : axd_ff_mk(ks[i][0], ks[i][1]);
      else f[i - 5] = c ? kc[i][0] : ks[i][0];
    }
  }
  // the series at r (r2 = r r), the operations of axd_ff_sincos
  __device__ __forceinline__ axd_ff operator()(axd_ff r, axd_ff r2) const {
    float q = f[3];
#pragma unroll
    for (int i = 2; i >= 0; --i) q = AXF_FMA(q, r2.h, f[i]);
    axd_ff p = axd_ff_mk(q, 0.0f);
#pragma unroll
    for (int i = 4; i >= 0; --i) p = axd_ff_add(axd_ff_mul(p, r2), k[i]);
    return axd_ff_mul(p, cosine ? axd_ff_mk(1.0f, 0.0f) : r);  // times (1, 0) is exact
  }
};

// axd_chi2_string_ff by the eight lanes of a group, every lane returning it.
// pc: the phase of corner `sub`; P: coordinate sub & 3 of the point.  All 32
// lanes of the warp call it together (lanes without a point pass any finite
// P).  Lanes 0-3 of the group reduce the angle, 4-7 phi, even lanes run the
// sine series and odd lanes the cosine; each lane forms its corner's d and d^2; even lanes then add the eight d^2 and odd lanes
// the eight d, in corner order, from shared memory (buf: the warp's 4 x 9
// float4, the ninth keeping the groups on different banks).
__device__ __forceinline__ double chi2_group(axd_ff pc, double P, int lane, float4 *buf, const LaneSeries &series) {
  constexpr unsigned kAll = 0xffffffffu;
  const axd_ff refpi = axd_ff_mk(3.1415927410125732f, -8.742257051608249e-08f);
  const axd_ff tworefpi = axd_ff_mk(6.2831854820251465f, -1.7484514103216497e-07f);
  const int sub = lane & 7, base = lane & ~7;
  auto from = [&](axd_ff v, int l) {
    return axd_ff_mk(__shfl_sync(kAll, v.h, base + l), __shfl_sync(kAll, v.l, base + l));
  };
  const axd_ff p = axd_ff_from(P);
  const axd_ff mu = from(p, 0), rad = from(p, 2), arg = from(p, sub < 4 ? 3 : 1);
  axd_ff sc;  // sin (even lanes) or cos (odd lanes) of arg, as axd_ff_sincos
  {
    const float P1 = 1.5707963705062866f, P2 = -4.371138828673793e-08f, P3 = -1.7151245100058819e-15f;
    const float kf = AXF_RINT(AXF_MUL(arg.h, 0.6366197723675814f));
    axd_ff r = axd_ff_add(arg, axd_ff_mk(-AXF_MUL(kf, P1), 0.0f));
    r = axd_ff_add(r, axd_ff_mk(-AXF_MUL(kf, P2), 0.0f));
    r = axd_ff_add(r, axd_ff_mk(-AXF_MUL(kf, P3), 0.0f));
    const int q = (int)kf & 3;
    const axd_ff own = series(r, axd_ff_mul(r, r));
    // arg = q pi/2 + r: for odd q the sine is the neighbour lane's cosine series and the other way round
    const axd_ff other = axd_ff_mk(__shfl_xor_sync(kAll, own.h, 1), __shfl_xor_sync(kAll, own.l, 1));
    sc = (q & 1) ? other : own;
    if ((sub & 1) ? (q == 1 || q == 2) : (q == 2 || q == 3)) sc = axd_ff_neg(sc);
  }
  const axd_ff s4 = from(sc, 0), c4 = from(sc, 1), sp = from(sc, 4), cp = from(sc, 5);
  const axd_ff u0 = axd_ff_mul(rad, c4), v0 = axd_ff_mul(rad, s4);
  const axd_ff sm = axd_ff_sqrt(axd_ff_sub(axd_ff_mk(1.0f, 0.0f), axd_ff_mul(mu, mu)));
  const axd_ff hcp = axd_ff_mulf(cp, 0.5f), hsp = axd_ff_mulf(sp, 0.5f), hsm = axd_ff_mulf(sm, 0.5f);
  const int ix = sub & 1, iy = (sub >> 1) & 1, iz = sub >> 2;
  const axd_ff xc = ix ? hcp : axd_ff_neg(hcp), ys = iy ? hsp : axd_ff_neg(hsp);
  const axd_ff xs = ix ? hsp : axd_ff_neg(hsp), yc = iy ? hcp : axd_ff_neg(hcp);
  const axd_ff zs = iz ? hsm : axd_ff_neg(hsm);
  const axd_ff du = axd_ff_sub(axd_ff_add(axd_ff_neg(u0), axd_ff_mul(mu, axd_ff_add(xc, ys))), zs);
  const axd_ff dv = axd_ff_add(axd_ff_sub(axd_ff_neg(v0), xs), yc);
  axd_ff d = axd_ff_sub(pc, axd_ff_atan2(dv, du));
  if (axd_ff_ge(d, refpi))
    d = axd_ff_sub(d, tworefpi);
  else if (axd_ff_gt(axd_ff_neg(refpi), d))
    d = axd_ff_add(d, tworefpi);
  const axd_ff d2 = axd_ff_mul(d, d);
  float4 *gb = buf + (lane >> 3) * (kGrp + 1);
  gb[sub] = make_float4(d2.h, d2.l, d.h, d.l);
  __syncwarp();
  const float2 *q = reinterpret_cast<const float2 *>(gb) + (sub & 1);
  axd_ff acc = axd_ff_mk(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 t = q[2 * i];
    acc = axd_ff_add(acc, axd_ff_mk(t.x, t.y));
  }
  __syncwarp();
  acc = axd_ff_mulf(acc, 0.125f);
  const axd_ff a = from(acc, 0), b = from(acc, 1);
  return axd_ff_to(axd_ff_sub(a, axd_ff_mul(b, b)));
}

// the corner phases of cell s: lane sub's corner
__device__ __forceinline__ double corner_phase(const double *__restrict__ ph64, int n, int64_t s, int sub) {
  const int ix = (int)(s % n), iy = (int)((s / n) % n), iz = (int)(s / ((int64_t)n * n));
  return ph64[corner(n, ix, iy, iz, sub)];
}

// The random search of one cell per group (defects_3d.f90:460-500).  It keeps
// kNumSimp + 1 starts in the order drawn; once that set is full, a start
// changes it only if its chi2 is at most the value in the last slot.  That
// value can rise (the first two starts are kept unsorted, defects_3d.f90:
// 471-476, and a larger early value moves up the list), but never above the
// largest value kept at any earlier time.  Each lane forms the FP32 lower
// bounds of kRounds starts; those not above the largest kept value are
// evaluated in draw order, each looked at again against the value kept by
// then.  A screened-out start has a chi2 above any threshold the sequential
// search could have compared it with.  About 30 of the 1001 are evaluated;
// rounds of 32 starts let the warp's four groups evaluate theirs together.  out: p[vertex][coordinate], chi2[vertex] per cell.
__global__ void __launch_bounds__(kFitThreads) k_string_start(const double *__restrict__ ph64, int n, uint64_t seed,
                                                              const int64_t *__restrict__ cells, int64_t ncell,
                                                              double *__restrict__ out) {
  __shared__ float4 sbuf[kFitThreads / 32][4 * (kGrp + 1)];
  const int lane = threadIdx.x & 31, sub = lane & 7, base = lane & ~7, k = sub & 3;
  float4 *buf = sbuf[threadIdx.x >> 5];
  const LaneSeries series(sub & 1);
  const int64_t c = (int64_t)blockIdx.x * (kFitThreads / kGrp) + threadIdx.x / kGrp;
  const bool live = c < ncell;
  const int64_t s = cells[live ? c : ncell - 1];
  const double pd = corner_phase(ph64, n, s, sub);
  const axd_ff pc = axd_ff_from(pd);
  float phf[8];
  {
    const float f = (float)pd;
#pragma unroll
    for (int i = 0; i < 8; ++i) phf[i] = __shfl_sync(0xffffffffu, f, base + i);
  }
  // a corner phase that is no number makes every chi2 one: no comparison of
  // the search holds, the first five starts stay and the simplex does not run
  const bool bad = (__ballot_sync(0xffffffffu, isnan(pd)) >> base) & 0xff;
  double p[kNumSimp + 1];
  long long ch[kNumSimp + 1];
  // the starts that fill the set, in the order of defects_3d.f90:471-490
#pragma unroll
  for (int i = 0; i <= kNumSimp; ++i) {
    const double t = string_start(seed, (uint64_t)s, i, k);
    const long long x = dkey(chi2_group(pc, t, lane, buf, series));
    bool go = true;
    if (i >= 2) {
#pragma unroll
      for (int q = i; q >= 1; --q) {
        const bool move = go && !bad && x <= ch[q - 1];
        if (move) {
          ch[q] = ch[q - 1];
          p[q] = p[q - 1];
        } else if (go) {
          ch[q] = x;
          p[q] = t;
          go = false;
        }
      }
      if (go) {
        ch[0] = x;
        p[0] = t;
      }
    } else {
      ch[i] = x;
      p[i] = t;
    }
  }
  for (int i0 = kNumSimp + 1; i0 <= kMaxIter; i0 += kRounds * kGrp) {
    float lb[kRounds];
#pragma unroll 1
    for (int r = 0; r < kRounds; ++r) {
      const int i = i0 + r * kGrp + sub;
      const float v = i <= kMaxIter ? chi2_start_lower(phf, seed, (uint64_t)s, i) : INFINITY;
#pragma unroll
      for (int q = 0; q < kRounds; ++q)
        if (q == r) lb[q] = v;
    }
    unsigned todo = 0xffffffffu;  // starts i0 + bit not yet passed over, in draw order
    for (;;) {
      long long top = ch[0];
#pragma unroll
      for (int q = 1; q <= kNumSimp; ++q) top = ch[q] > top ? ch[q] : top;
      // (double)lb > top, as floats: lb exceeds top exactly when it exceeds top rounded down
      const float thr = __double2float_rd(dkey_value(top));
      unsigned m = 0;
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
        m |= ((__ballot_sync(0xffffffffu, live && !bad && !(lb[r] > thr)) >> base) & 0xffu) << (kGrp * r);
      m &= todo;
      if (!__any_sync(0xffffffffu, m != 0)) break;
      const int j = m ? __ffs(m) - 1 : 0;
      todo = m ? (0xfffffffeu << j) : 0;
      const double t = string_start(seed, (uint64_t)s, i0 + j, k);
      const long long x = dkey(chi2_group(pc, t, lane, buf, series));
      if (m && x <= ch[kNumSimp]) {
        bool go = true;
#pragma unroll
        for (int q = kNumSimp; q >= 1; --q) {
          const bool move = go && x <= ch[q - 1];
          if (move) {
            ch[q] = ch[q - 1];
            p[q] = p[q - 1];
          } else if (go) {
            ch[q] = x;
            p[q] = t;
            go = false;
          }
        }
        if (go) {
          ch[0] = x;
          p[0] = t;
        }
      }
    }
  }
  if (live && sub < 4) {
    double *o = out + c * kFitStride;
#pragma unroll
    for (int q = 0; q <= kNumSimp; ++q) {
      o[4 * q + k] = p[q];
      if (sub == 0) o[20 + q] = dkey_value(ch[q]);
    }
  }
}

// Orders the simplex by chi2 as the reference's bubble sort does (strict
// comparisons, so equal values keep their order).  sorted: vertices 0..3 are
// in order already and only the last one has to find its place.
__device__ __forceinline__ void simplex_sort(double p[kNumSimp + 1], long long ch[kNumSimp + 1], bool sorted) {
  auto order = [&](int m) {  // swap vertices m and m + 1 when out of order
    const bool sw = ch[m] > ch[m + 1];
    const double a = p[m];
    p[m] = sw ? p[m + 1] : a;
    p[m + 1] = sw ? a : p[m + 1];
    const long long q = ch[m];
    ch[m] = sw ? ch[m + 1] : q;
    ch[m + 1] = sw ? q : ch[m + 1];
  };
  if (!sorted) {
#pragma unroll
    for (int i0 = kNumSimp - 1; i0 >= 1; --i0)
#pragma unroll
      for (int m = 0; m < i0; ++m) order(m);
  }
#pragma unroll
  for (int m = kNumSimp - 1; m >= 0; --m) order(m);
}

enum : int {
  kNmStart = 0,
  kNmReflect,
  kNmSecondPrep,
  kNmSecond,
  kShrink1,  // kShrink1 .. kShrink1 + kNumSimp - 1: shrink vertices 1..kNumSimp
  kNmSort = kShrink1 + kNumSimp,
  kFinished
};

// The Nelder-Mead simplex (defects_3d.f90:501-603), one cell per group, as a
// state machine that advances to its next chi2: every pass of the loop
// evaluates one chi2 per group, together for the warp's four groups, and a
// group whose cell is done takes the next from *next (zero at launch).  The
// grid is sized to the resident CTAs.  sim: as k_string_start leaves it; the
// best vertex and its chi2 come back in its first row.
__global__ void __launch_bounds__(kFitThreads, 6) k_string_simplex(const double *__restrict__ ph64, int n,
                                                                const int64_t *__restrict__ cells, int64_t ncell,
                                                                double *__restrict__ sim,
                                                                unsigned long long *__restrict__ next,
                                                                int2 *__restrict__ rest, unsigned *__restrict__ nrest) {
  __shared__ float4 sbuf[kFitThreads / 32][4 * (kGrp + 1)];
  const int lane = threadIdx.x & 31, sub = lane & 7, base = lane & ~7, k = sub & 3;
  const unsigned gmask = 0xffu << base;
  float4 *buf = sbuf[threadIdx.x >> 5];
  const LaneSeries series(sub & 1);
  const long long kmax = dkey(string_max(k)), kmin = dkey(string_min(k));
  const long long chi2max = dkey(8 * kRefPi * kRefPi), tol = dkey(0.05);
  double p[kNumSimp + 1] = {}, sum = 0.0, t = 0.0, s2 = 0.0, P = 0.0;
  long long ch[kNumSimp + 1] = {}, x = 0;  // x: chi2 of the reflected point
  axd_ff pc = axd_ff_mk(0.0f, 0.0f);
  int64_t c = 0;
  int stage = kFinished, it = 0;
  bool expand = false, done = false, sorted = false;  // sorted: vertices 0..3 are in order
  unsigned idle = 0;                                  // lanes whose group is done
  auto outside = [&](double v) {  // any coordinate out of the box
    const long long q = dkey(v);
    return (__ballot_sync(gmask, q > kmax || q < kmin)) != 0;
  };
  // the expansion / contraction decision with the second point's chi2
  auto second = [&](long long xs) {
    if (expand) {
      const bool first = x <= xs;
      ch[kNumSimp] = first ? x : xs;
      p[kNumSimp] = first ? t : s2;
      stage = kNmSort;
    } else if (xs <= ch[kNumSimp]) {
      ch[kNumSimp] = xs;
      p[kNumSimp] = s2;
      stage = kNmSort;
    } else {
      stage = kShrink1;
    }
  };
  auto fetch = [&]() {
    unsigned long long q = 0;
    if (sub == 0) q = atomicAdd(next, 1ull);
    c = (int64_t)__shfl_sync(gmask, q, base);
    if (c >= ncell) {
      done = true;
      return;
    }
    const double pd = corner_phase(ph64, n, cells[c], sub);
    pc = axd_ff_from(pd);
    const double *o = sim + c * kFitStride;
#pragma unroll
    for (int q2 = 0; q2 <= kNumSimp; ++q2) {
      p[q2] = o[4 * q2 + k];
      ch[q2] = dkey(o[20 + q2]);
    }
    it = 0;
    sorted = false;  // the random search leaves its first two starts as drawn
    // a chi2 that is no number compares false with the tolerance
    stage = isnan(o[20]) ? kFinished : kNmStart;
  };
  // an iteration's start with the queue empty and kIdle groups of the warp
  // done: the rest of this cell goes to k_string_simplex_warp
  auto hand_over = [&]() {
    if (__popc(idle) < kIdle * kGrp) return false;
    double *o = sim + c * kFitStride;
#pragma unroll
    for (int q2 = 0; q2 <= kNumSimp; ++q2) {
      if (sub < 4) o[4 * q2 + k] = p[q2];
      if (sub == 0) o[20 + q2] = dkey_value(ch[q2]);
    }
    if (sub == 0) rest[atomicAdd(nrest, 1u)] = make_int2((int)c, it);
    done = true;
    return true;
  };
  fetch();
  for (;;) {
    idle = __ballot_sync(0xffffffffu, done);
    while (!done) {  // to the next chi2, or the next cell
      if (stage == kNmSort) {
        simplex_sort(p, ch, sorted);
        sorted = true;
        stage = kNmStart;
      }
      if (stage == kNmStart) {
        if (ch[0] > tol && it < kMaxIter) {
          if (hand_over()) continue;
          ++it;
          sum = ((0.0 + p[0]) + p[1]) + p[2] + p[3];
        } else {
          stage = kFinished;
        }
      }
      if (stage == kNmStart || stage == kNmSecondPrep) {
        // with the centroid c = sum / 4: the reflected point 2 c - p, the
        // expansion 3 c - 4 p or the contraction 1.5 c - 0.5 p.  Scaling by
        // a power of two is exact, so a sum rounds as a multiple of c does.
        static_assert(kNumSimp == 4, "the centroid scaling is 1 / kNumSimp");
        const bool reflect = stage == kNmStart;
        if (!reflect) expand = x < ch[kNumSimp];
        const double alpha = reflect ? 0.5 : (expand ? 0.75 : 0.375), beta = reflect ? 1.0 : (expand ? 4.0 : 0.5);
        const double v = alpha * sum - axg_mul_pow2(p[kNumSimp], beta);
        const bool out = outside(v);
        if (reflect) {
          t = v;
          stage = out ? kNmSecondPrep : kNmReflect;
          x = out ? chi2max : x;
        } else {
          s2 = v;
          stage = kNmSecond;
          if (out) second(chi2max);
        }
        if (!out) {
          P = v;
          break;
        }
      }
      if (stage >= kShrink1 && stage < kNmSort) {  // shrink towards the best vertex
        const int j = stage - kShrink1 + 1;
#pragma unroll
        for (int q = 1; q <= kNumSimp; ++q)
          if (q == j) {
            p[q] = axg_mul_pow2(p[q] + p[0], 0.5);
            P = p[q];
          }
        sorted = false;
        break;
      }
      if (stage == kFinished) {
        double *o = sim + c * kFitStride;
        if (sub < 4) o[k] = p[0];
        if (sub == 0) o[20] = dkey_value(ch[0]);
        fetch();
      }
    }
    __syncwarp();
    if (__all_sync(0xffffffffu, done)) break;
    const long long v = dkey(chi2_group(pc, P, lane, buf, series));
    if (stage == kNmReflect) {
      x = v;
      stage = kNmSecondPrep;
    } else if (stage == kNmSecond) {
      second(v);
    } else if (!done) {
      const int j = stage - kShrink1 + 1;
#pragma unroll
      for (int q = 1; q <= kNumSimp; ++q)
        if (q == j) ch[q] = v;
      stage = j < kNumSimp ? stage + 1 : kNmSort;
    }
  }
}

// position, direction, goodness of fit and length from the best vertex
__device__ void string_result(const double p[4], double chi2, double pos[3], double dir[3], double *gof, double *sl) {
  const double mu = p[0], phi = p[1];
  double s4, c4, sp, cp;
  axd_sincos(p[3], &s4, &c4);
  const double u0 = p[2] * c4, v0 = p[2] * s4;
  axd_sincos(phi, &sp, &cp);
  const double sq = sqrt(1.0 - mu * mu);
  dir[0] = sq * cp;
  dir[1] = sq * sp;
  dir[2] = mu;
  pos[0] = u0 * mu * cp - v0 * sp;
  pos[1] = u0 * mu * sp + v0 * cp;
  pos[2] = -(u0 * sqrt(1 - mu * mu));
  *gof = exp(-chi2 / 2);
  *sl = string_length(pos, dir);
}

// reference BLAS dspr ('U')
__device__ void dspr_u(int n, double alpha, const double *x, double *ap) {
  int kk = 0;
  for (int j = 0; j < n; ++j) {
    if (x[j] != 0.0) {
      const double temp = alpha * x[j];
      int k = kk;
      for (int i = 0; i <= j; ++i) {
        ap[k] = ap[k] + x[i] * temp;
        ++k;
      }
    }
    kk += j + 1;
  }
}

// reference LAPACK dpptrf + dpptri ('U') on a packed 4x4
__device__ void pp_inverse4(double *ap) {
  const int n = 4;
  int jj = 0;
  for (int j = 1; j <= n; ++j) {
    const int jc = jj + 1;
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
    const double ajj = ap[jj - 1] - dot;
    if (ajj <= 0.0) {
      ap[jj - 1] = ajj;
      return;
    }
    ap[jj - 1] = sqrt(ajj);
  }
  int jc = 1;
  for (int j = 1; j <= n; ++j) {
    ap[jc + j - 2] = 1.0 / ap[jc + j - 2];
    const double ajj = -ap[jc + j - 2];
    double *x = ap + (jc - 1);
    int kk = 1;
    for (int jx = 1; jx <= j - 1; ++jx) {
      if (x[jx - 1] != 0.0) {
        const double temp = x[jx - 1];
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
    const int jc2 = jj + 1;
    jj = jj + j;
    if (j > 1) dspr_u(j - 1, 1.0, ap + (jc2 - 1), ap);
    const double ajj = ap[jj - 1];
    for (int i = 0; i < j; ++i) ap[jc2 - 1 + i] = ajj * ap[jc2 - 1 + i];
  }
}

// defects_3d.f90:605-692 (VEL=0)
template <typename V>
__device__ void velocity_string(const V *phi, const V *cphi, const V *phid, int n, double dspa, int ix, int iy,
                                int iz, const double pos[3], double vel[3]) {
  double wr[4] = {0, 0, 0, 0}, wi[4] = {0, 0, 0, 0}, dr[4] = {0, 0, 0, 0}, di[4] = {0, 0, 0, 0};
  double mat[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0}, mat0[10];
  double d[4];
  d[0] = 1.0;
  for (int k = 0; k <= 1; ++k) {
    const int zz = iz + k == n ? 0 : iz + k;
    d[3] = k - pos[2] - 0.5;
    for (int j = 0; j <= 1; ++j) {
      const int yy = iy + j == n ? 0 : iy + j;
      d[2] = j - pos[1] - 0.5;
      for (int i = 0; i <= 1; ++i) {
        const int xx = ix + i == n ? 0 : ix + i;
        d[1] = i - pos[0] - 0.5;
        const int64_t s = ((int64_t)zz * n + yy) * n + xx;
        double pr, pi_, qr, qi;
        load_c(phi, cphi, s, pr, pi_);
        load_c(phid, (const V *)nullptr, s, qr, qi);
        for (int l = 0; l < 4; ++l) {
          wr[l] = wr[l] + d[l] * pr;
          wi[l] = wi[l] + d[l] * pi_;
          dr[l] = dr[l] + d[l] * qr;
          di[l] = di[l] + d[l] * qi;
        }
        dspr_u(4, 1.0, d, mat);
      }
    }
  }
  for (int l = 0; l < 4; ++l) {
    wr[l] /= 8;
    wi[l] /= 8;
    dr[l] /= 8;
    di[l] /= 8;
  }
  for (int l = 0; l < 10; ++l) {
    mat[l] /= 8;
    mat0[l] = mat[l];
  }
  pp_inverse4(mat0);
  double w0r[4] = {0, 0, 0, 0}, w0i[4] = {0, 0, 0, 0}, d0r[4] = {0, 0, 0, 0}, d0i[4] = {0, 0, 0, 0};
  for (int ii = 1; ii <= 4; ++ii)
    for (int jj = 1; jj <= 4; ++jj) {
      int kk = ii > jj ? ii : jj;
      kk = kk * (kk - 1) / 2 + (ii < jj ? ii : jj);
      const double m = mat0[kk - 1];
      w0r[ii - 1] = w0r[ii - 1] + m * wr[jj - 1];
      w0i[ii - 1] = w0i[ii - 1] + m * wi[jj - 1];
      d0r[ii - 1] = d0r[ii - 1] + m * dr[jj - 1];
      d0i[ii - 1] = d0i[ii - 1] + m * di[jj - 1];
    }
  const double x = d0r[0], y = d0i[0];
  double a = 0, b = 0, c = 0;
  for (int l = 1; l < 4; ++l) {
    a = a + w0r[l] * w0r[l];
    b = b + w0r[l] * w0i[l];
    c = c + w0i[l] * w0i[l];
  }
  const double det = a * c - b * b;
  for (int l = 1; l < 4; ++l) {
    const double v = (x * c - y * b) * w0r[l] + (-(x * b) + y * a) * w0i[l];
    vel[l - 1] = -v / det * dspa;
  }
}

// defects_3d.f90:1058-1233
// The 20 x 20 grid of wall directions of position_wall (defects_3d.f90:
// 1135-1160): d0 = (sqrt(1 - mu^2) cos phi, sqrt(1 - mu^2) sin phi, mu) for
// mu = ((2 imu - 20) - 1) / 20, phi = pi ((2 iphi - 1) - 20) / 20, in the
// reference's operations; the same for every cell, so k_wall_fit forms it
// once per CTA in shared memory.
struct WallGrid {
  double d0[400][4];  // d0 and phi
  float f[400][3];    // d0 rounded to FP32, for the screen of position_wall
};

__device__ void wall_grid_fill(WallGrid &g) {
  for (int idx = threadIdx.x; idx < 400; idx += blockDim.x) {
    const int imu = idx / 20 + 1, iphi = idx % 20 + 1;
    const double mu = ((double)(-20 + 2 * imu) - 1.0) / 20;
    const double phi = kRefPi * ((2 * iphi - 1.0) - 20) / 20;
    double sp, cp;
    axd_sincos(phi, &sp, &cp);
    const double sq = sqrt(1 - mu * mu);
    g.d0[idx][0] = sq * cp;
    g.d0[idx][1] = sq * sp;
    g.d0[idx][2] = mu;
    g.d0[idx][3] = phi;
    for (int k = 0; k < 3; ++k) g.f[idx][k] = (float)g.d0[idx][k];
  }
}

// The direction search of position_wall screened in FP32.  Per direction
// the reference forms d_i = pp_i . d0, W = sum d_i, S = sum d_i^2 and
// chi2 = S - m w^2 with w = max(W, 0) / m.  With the points' mean c and
// q_i = pp_i - c that is
//   chi2 = sum (q_i . d0)^2 + m min(c . d0, 0)^2,
// a sum of squares without cancellation, so its FP32 value is good to a few
// ulp of chi2 itself.  q_i and c are formed in FP64 and rounded; with
// |q_i| < 1.8, |d0| = 1 and m <= 12 a projection is off by less than 7e-7
// (2^-24 for each factor and operation), so the sum of squares by less than
// 2 sqrt(12 chi2) 7e-7 + 6e-12, the second term by 2e-6 sqrt(chi2), and the
// FP32 summation by 1.5e-6 chi2; kWallErr covers their sum.  A direction whose
// FP32 value exceeds the smallest one by more than both errors cannot hold
// the FP64 minimum, so evaluating only the others in FP64, in the reference's
// loop order and with its strict-less update, selects the same direction and
// w.  (Screened as S - max(W, 0)^2 / m, whose error is 1e-4 of S, cells with
// close crossing points kept tens of directions, and a warp evaluated ~85 of
// them in FP64 one after another.)
__device__ __forceinline__ float wall_err(float f) { return 1e-5f * sqrtf(f) + 2e-6f * f + 1e-10f; }

__device__ void position_wall(const double ph[8], const WallGrid &grid, double pos[3], double dir[3], double *gof,
                              double *wa) {
  double pp[12][3], th[12], uv[12][2], sn[8], cs[8];
  for (int i = 0; i < 8; ++i) axd_sincos(ph[i], &sn[i], &cs[i]);
  int m = 0;
  for (int iz = 0; iz <= 1; ++iz)
    for (int iy = 0; iy <= 1; ++iy) {
      const double u = sn[(iz * 2 + iy) * 2 + 0], v = sn[(iz * 2 + iy) * 2 + 1];
      if (u * v < 0.0) {
        pp[m][0] = (u + v) / (u - v) / 2;
        pp[m][1] = iy - 0.5;
        pp[m][2] = iz - 0.5;
        ++m;
      }
    }
  for (int iy = 0; iy <= 1; ++iy)
    for (int ix = 0; ix <= 1; ++ix) {
      const double u = sn[(0 * 2 + iy) * 2 + ix], v = sn[(1 * 2 + iy) * 2 + ix];
      if (u * v < 0.0) {
        pp[m][0] = ix - 0.5;
        pp[m][1] = iy - 0.5;
        pp[m][2] = (u + v) / (u - v) / 2;
        ++m;
      }
    }
  for (int iz = 0; iz <= 1; ++iz)
    for (int ix = 0; ix <= 1; ++ix) {
      const double u = sn[(iz * 2 + 0) * 2 + ix], v = sn[(iz * 2 + 1) * 2 + ix];
      if (u * v < 0.0) {
        pp[m][0] = ix - 0.5;
        pp[m][1] = (u + v) / (u - v) / 2;
        pp[m][2] = iz - 0.5;
        ++m;
      }
    }
  if (m < 3) {
    for (int k = 0; k < 3; ++k) pos[k] = dir[k] = 0.0;
    *gof = 0.0;
    *wa = 0.0;
    return;
  }
  // the centred points in FP32 registers; those past m are zero and add
  // nothing (indexed by a loop over m they lived in local memory, and the 800
  // screens of a cell waited on its loads)
  double cen[3];
  for (int k = 0; k < 3; ++k) {
    cen[k] = 0.0;
    for (int i = 0; i < m; ++i) cen[k] = cen[k] + pp[i][k];
    cen[k] = cen[k] / m;
  }
  const float c0 = (float)cen[0], c1 = (float)cen[1], c2 = (float)cen[2];
  float q[12][3];
#pragma unroll
  for (int i = 0; i < 12; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) q[i][k] = i < m ? (float)(pp[i][k] - cen[k]) : 0.0f;
  auto screen = [&](int idx) {
    const float g0 = grid.f[idx][0], g1 = grid.f[idx][1], g2 = grid.f[idx][2];
    const float w = fminf(fmaf(c2, g2, fmaf(c1, g1, c0 * g0)), 0.0f);
    float f = 0.0f;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const float d = fmaf(q[i][2], g2, fmaf(q[i][1], g1, q[i][0] * g0));
      f = fmaf(d, d, f);
    }
    return fmaf((float)m * w, w, f);
  };
  float fmin = INFINITY;
  for (int idx = 0; idx < 400; ++idx) fmin = fminf(fmin, screen(idx));
  const float fcut = fmin + wall_err(fmin);
  auto kept = [&](int idx) {
    const float f = screen(idx);
    return f - wall_err(f) <= fcut;
  };
  // the directions to evaluate, in the reference's loop order: listed first
  // and then evaluated one per lane at a time, so that the FP64 work of the
  // warp's cells runs together (evaluated where the screen found them, each
  // of a warp's candidates issued it alone)
  constexpr int kCand = 8;
  uint16_t cand[kCand];
  int ncand = 0;
  for (int idx = 0; idx < 400; ++idx)
    if (kept(idx)) {
      if (ncand < kCand) cand[ncand] = (uint16_t)idx;
      ++ncand;
    }
  double chi2min = 6.0, mut = 0.0, phit = 0.0, wt = 0.0;
  auto evaluate = [&](int idx) {
    const double *d0 = grid.d0[idx];
    double w = 0.0, chi2 = 0.0;
    for (int i = 0; i < m; ++i) {
      double d = pp[i][0] * d0[0] + pp[i][1] * d0[1];
      d = d + pp[i][2] * d0[2];
      w = w + d;
      chi2 = chi2 + d * d;
    }
    if (w < 0.0)
      w = 0.0;
    else
      w = w / m;
    chi2 = chi2 - m * w * w;
    if (chi2 < chi2min) {
      chi2min = chi2;
      mut = d0[2];
      phit = d0[3];
      wt = w;
    }
  };
  for (int c = 0; c < ncand && c < kCand; ++c) evaluate(cand[c]);
  if (ncand > kCand)  // a flat minimum: the rest as found
    for (int idx = cand[kCand - 1] + 1; idx < 400; ++idx)
      if (kept(idx)) evaluate(idx);
  double spt, cpt;
  axd_sincos(phit, &spt, &cpt);
  const double sqt = sqrt(1 - mut * mut);
  double d0[3] = {sqt * cpt, sqt * spt, mut};
  int num = 0;
  for (int iz = 0; iz <= 1; ++iz)
    for (int iy = 0; iy <= 1; ++iy)
      for (int ix = 0; ix <= 1; ++ix) {
        const double disp[3] = {ix - 0.5, iy - 0.5, iz - 0.5};
        double d = disp[0] * d0[0] + disp[1] * d0[1];
        d = d + disp[2] * d0[2];
        d = d - wt;
        if (d * cs[(iz * 2 + iy) * 2 + ix] > 0.0) ++num;
      }
  if (num <= 4) {
    for (int k = 0; k < 3; ++k) d0[k] = -d0[k];
    wt = -wt;
  }
  for (int k = 0; k < 3; ++k) {
    dir[k] = d0[k];
    pos[k] = wt * d0[k];
  }
  *gof = exp(-chi2min / 2);
  const double dir1[3] = {mut * cpt, mut * spt, -sqrt(1 - mut * mut)};
  const double dir2[3] = {-spt, cpt, 0.0};
  for (int i = 0; i < m; ++i) {
    for (int k = 0; k < 3; ++k) pp[i][k] = pp[i][k] - pos[k];
    double u = dir1[0] * pp[i][0] + dir1[1] * pp[i][1];
    u = u + dir1[2] * pp[i][2];
    double v = dir2[0] * pp[i][0] + dir2[1] * pp[i][1];
    v = v + dir2[2] * pp[i][2];
    th[i] = axd_atan2(v, u);
    uv[i][0] = u;
    uv[i][1] = v;
  }
  for (int i = m - 1; i >= 1; --i)
    for (int j = 1; j <= i; ++j)
      if (th[j - 1] > th[j]) {
        const double w = th[j - 1];
        th[j - 1] = th[j];
        th[j] = w;
        const double a = uv[j - 1][0], b = uv[j - 1][1];
        uv[j - 1][0] = uv[j][0];
        uv[j - 1][1] = uv[j][1];
        uv[j][0] = a;
        uv[j][1] = b;
      }
  double area = 0.0;
  double w = th[m - 1] - kRefTwoPi;
  double u = sqrt(uv[m - 1][0] * uv[m - 1][0] + uv[m - 1][1] * uv[m - 1][1]);
  for (int i = 0; i < m; ++i) {
    const double v = sqrt(uv[i][0] * uv[i][0] + uv[i][1] * uv[i][1]);
    w = th[i] - w;
    area = area + 0.5 * u * v * axd_sin(w);
    u = v;
    w = th[i];
  }
  *wa = area;
}

// The simplex with a warp per cell, for the cells left when the queue of
// k_string_simplex runs dry and for lattices with few of them: then the serial
// chain of chi2 sets the time.  The four groups evaluate an iteration's
// reflected, expanded and contracted points at once (the two that the
// sequential search would not have asked for are dropped), and the four
// vertices of a shrink, so an iteration is one chi2 long instead of two to
// six.  list: (cell, iterations done), or null for cells 0 .. *count - 1.
__global__ void __launch_bounds__(kFitThreads, 6) k_string_simplex_warp(const double *__restrict__ ph64, int n,
                                                                     const int64_t *__restrict__ cells,
                                                                     const int2 *__restrict__ list,
                                                                     const unsigned *__restrict__ count, int64_t ncell,
                                                                     double *__restrict__ sim,
                                                                     unsigned long long *__restrict__ next) {
  __shared__ float4 sbuf[kFitThreads / 32][4 * (kGrp + 1)];
  const int lane = threadIdx.x & 31, sub = lane & 7, k = sub & 3, g = lane >> 3;
  float4 *buf = sbuf[threadIdx.x >> 5];
  const LaneSeries series(sub & 1);
  const long long kmax = dkey(string_max(k)), kmin = dkey(string_min(k));
  const long long chi2max = dkey(8 * kRefPi * kRefPi), tol = dkey(0.05);
  if (list) ncell = *count;
  for (;;) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(next, 1ull);
    q = __shfl_sync(0xffffffffu, q, 0);
    if ((int64_t)q >= ncell) return;
    const int64_t c = list ? list[q].x : (int64_t)q;
    int it = list ? list[q].y : 0;
    const axd_ff pc = axd_ff_from(corner_phase(ph64, n, cells[c], sub));
    double *o = sim + c * kFitStride;
    double p[kNumSimp + 1];
    long long ch[kNumSimp + 1];
#pragma unroll
    for (int v = 0; v <= kNumSimp; ++v) {
      p[v] = o[4 * v + k];
      ch[v] = dkey(o[20 + v]);
    }
    if (isnan(o[20])) continue;  // a chi2 that is no number compares false with the tolerance
    bool sorted = false;
    for (; ch[0] > tol && it < kMaxIter; ++it) {
      const double sum = ((0.0 + p[0]) + p[1]) + p[2] + p[3];
      // group 0: reflected, 1: expanded, 2: contracted (3: contracted, unused);
      // the scalings of k_string_simplex
      const double alpha = g == 0 ? 0.5 : (g == 1 ? 0.75 : 0.375), beta = g == 0 ? 1.0 : (g == 1 ? 4.0 : 0.5);
      const double pt = alpha * sum - axg_mul_pow2(p[kNumSimp], beta);
      const long long q = dkey(pt);
      const unsigned out = __ballot_sync(0xffffffffu, q > kmax || q < kmin);
      long long v = dkey(chi2_group(pc, pt, lane, buf, series));
      if ((out >> (lane & ~7)) & 0xff) v = chi2max;
      const long long x = __shfl_sync(0xffffffffu, v, 0), xe = __shfl_sync(0xffffffffu, v, 8),
                      xc = __shfl_sync(0xffffffffu, v, 16);
      const double t = __shfl_sync(0xffffffffu, pt, k), te = __shfl_sync(0xffffffffu, pt, 8 + k),
                   tc = __shfl_sync(0xffffffffu, pt, 16 + k);
      if (x < ch[kNumSimp]) {
        const bool first = x <= xe;
        ch[kNumSimp] = first ? x : xe;
        p[kNumSimp] = first ? t : te;
      } else if (xc <= ch[kNumSimp]) {
        ch[kNumSimp] = xc;
        p[kNumSimp] = tc;
      } else {  // shrink towards the best vertex, group g vertex g + 1
#pragma unroll
        for (int v2 = 1; v2 <= kNumSimp; ++v2) p[v2] = axg_mul_pow2(p[v2] + p[0], 0.5);
        const double own = g == 0 ? p[1] : (g == 1 ? p[2] : (g == 2 ? p[3] : p[4]));
        const long long w = dkey(chi2_group(pc, own, lane, buf, series));
#pragma unroll
        for (int v2 = 1; v2 <= kNumSimp; ++v2) ch[v2] = __shfl_sync(0xffffffffu, w, 8 * (v2 - 1));
        sorted = false;
      }
      simplex_sort(p, ch, sorted);
      sorted = true;
    }
    if (lane < 4) o[k] = p[0];
    if (lane == 0) o[20] = dkey_value(ch[0]);
  }
}

// Length, velocity and output row of the fitted string cells, one thread per
// cell (a group of eight lanes per cell would issue their long FP64 chains for
// one cell at a time).
template <typename V>
__global__ void __launch_bounds__(128) k_string_result(const V *__restrict__ phi, const V *__restrict__ cphi,
                                                       const V *__restrict__ phid, int n, double dspa,
                                                       const int64_t *__restrict__ cells, int64_t ncell,
                                                       const double *__restrict__ sim, double *__restrict__ out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ncell) return;
  const int64_t s = cells[k];
  const int ix = (int)(s % n), iy = (int)((s / n) % n), iz = (int)(s / ((int64_t)n * n));
  double pos[3], dir[3], vel[3], gof, l;
  string_result(sim + k * kFitStride, sim[k * kFitStride + 20], pos, dir, &gof, &l);
  velocity_string(phi, cphi, phid, n, dspa, ix, iy, iz, pos, vel);
  double *r = out + 13 * k;
  r[0] = pos[0] + ix + 0.5;
  r[1] = pos[1] + iy + 0.5;
  r[2] = pos[2] + iz + 0.5;
  r[3] = dir[0];
  r[4] = dir[1];
  r[5] = dir[2];
  r[6] = vel[0];
  r[7] = vel[1];
  r[8] = vel[2];
  r[9] = gof;
  r[10] = l;
  r[11] = (double)s;
  r[12] = -1.0;
}

__global__ void __launch_bounds__(128) k_wall_fit(const double *__restrict__ ph64, int n,
                                                  const int64_t *__restrict__ cells,
                                                  int64_t ncell, double *__restrict__ out) {
  __shared__ WallGrid grid;
  wall_grid_fill(grid);
  __syncthreads();
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ncell) return;
  const int64_t s = cells[k];
  const int ix = (int)(s % n), iy = (int)((s / n) % n), iz = (int)(s / ((int64_t)n * n));
  double pc[8];
  for (int c = 0; c < 8; ++c) pc[c] = ph64[corner(n, ix, iy, iz, c)];
  double pos[3], dir[3], gof, a;
  position_wall(pc, grid, pos, dir, &gof, &a);
  double *r = out + 10 * k;
  r[0] = pos[0] + ix + 0.5;
  r[1] = pos[1] + iy + 0.5;
  r[2] = pos[2] + iz + 0.5;
  r[3] = dir[0];
  r[4] = dir[1];
  r[5] = dir[2];
  r[6] = gof;
  r[7] = a;
  r[8] = (double)s;
  r[9] = -1.0;
}

// add_string_length / add_wall_area sums in a fixed order: kSumBlocks CTAs
// each add a strided share (k_defect_sums; one CTA took 1.36 ms for the 5e5
// rows of a 128^3 lattice, latency of 256 threads' strided loads), then one CTA
// adds their six sums (k_defect_sums_total).
constexpr int kSumBlocks = 304;

// the block's sum of a[0..5], result in thread 0
__device__ __forceinline__ void block_sum6(double a[6]) {
  __shared__ double sh[6][256];
  for (int q = 0; q < 6; ++q) sh[q][threadIdx.x] = a[q];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
      for (int q = 0; q < 6; ++q) sh[q][threadIdx.x] = sh[q][threadIdx.x] + sh[q][threadIdx.x + o];
    __syncthreads();
  }
  for (int q = 0; q < 6; ++q) a[q] = sh[q][0];
}

__global__ void __launch_bounds__(256) k_defect_sums(const double *__restrict__ strs, int64_t ns,
                                                     const double *__restrict__ walls, int64_t nw,
                                                     double *__restrict__ part) {
  double a[6] = {0, 0, 0, 0, 0, 0};  // sl, sqrt(v2), v2, gamma, count of v2<1; wa
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = first; k < ns; k += step) {
    const double *r = strs + 13 * k;
    a[0] = a[0] + r[10];
    double v2 = r[6] * r[6] + r[7] * r[7];
    v2 = v2 + r[8] * r[8];
    if (v2 < 1.0) {
      a[1] = a[1] + sqrt(v2);
      a[2] = a[2] + v2;
      a[3] = a[3] + 1 / sqrt(1 - v2);
      a[4] = a[4] + 1.0;
    }
  }
  for (int64_t k = first; k < nw; k += step) a[5] = a[5] + walls[10 * k + 7];
  block_sum6(a);
  if (threadIdx.x < 6) part[6 * blockIdx.x + threadIdx.x] = a[threadIdx.x];
}

__global__ void __launch_bounds__(256) k_defect_sums_total(const double *__restrict__ part, int nb,
                                                           double *__restrict__ out) {
  double a[6] = {0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    for (int q = 0; q < 6; ++q) a[q] = a[q] + part[6 * b + q];
  block_sum6(a);
  if (threadIdx.x == 0)
    for (int q = 0; q < 6; ++q) out[q] = a[q];
}

// ---------------- grouping (defects_3d.f90:1235-1652, 1735-2143) ----------------
// Connected components of the fitted positions under the periodic distance
// threshold: the partition the reference's grouping produces on one rank and
// one thread.  Hash grid of G^3 cells (cell side >= threshold) + lock-free
// union-find linking the larger root under the smaller, so the final label
// of every point is the smallest list index of its component.
constexpr int kUfMaxRetries = 1 << 20;

__device__ double lat_dist_periodic(int n, const double *a, const double *b) {
  double s = 0.0;
  for (int k = 0; k < 3; ++k) {
    const double dp = fabs(a[k] - b[k]);
    const double e = (double)n - dp;
    const double m = dp < e ? dp : e;
    s = s + m * m;
  }
  return sqrt(s);
}

__device__ int uf_find(volatile int *par, int x) {
  while (true) {
    const int p = par[x];
    if (p == x) return x;
    const int gp = par[p];
    if (gp != p) par[x] = gp;  // path halving: a valid ancestor, benign race
    x = p;
  }
}

__device__ void uf_union(int *par, int a, int b, int *err) {
  for (int it = 0; it < kUfMaxRetries; ++it) {
    a = uf_find(par, a);
    b = uf_find(par, b);
    if (a == b) return;
    if (a > b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicCAS(&par[b], b, a);
    if (old == b) return;
    b = old;
  }
  atomicExch(err, AXG_KERR_BOUNDS);
}

__device__ __forceinline__ int cell_of(double x, int n, int G) {
  double w = x - floor(x / n) * n;  // into [0, n)
  int c = (int)(w * G / n);
  return c < 0 ? 0 : (c >= G ? G - 1 : c);
}

__global__ void k_grp_init(int *par, int np) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < np) par[i] = i;
}

__global__ void k_grp_count(const double *rows, int width, int np, int n, int G, int *cell, int *count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const double *r = rows + (int64_t)width * i;
  const int c = (cell_of(r[2], n, G) * G + cell_of(r[1], n, G)) * G + cell_of(r[0], n, G);
  cell[i] = c;
  atomicAdd(&count[c], 1);
}

__global__ void k_scan_int(int *a, int m) {
  __shared__ long long carry;
  __shared__ int sh[1024];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < m; base += 1024) {
    const int i = base + threadIdx.x;
    const int v = i < m ? a[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const int x = (int)threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += x;
      __syncthreads();
    }
    if (i < m) a[i] = (int)(carry + sh[threadIdx.x] - v);
    __syncthreads();
    if (threadIdx.x == 1023) carry += sh[1023];
    __syncthreads();
  }
}

__global__ void k_grp_scatter(const int *cell, int np, const int *start, int *fill, int *sorted) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const int c = cell[i];
  sorted[start[c] + atomicAdd(&fill[c], 1)] = i;
}

__global__ void k_grp_link(const double *rows, int width, int np, int n, int G, double th, const int *cell,
                           const int *start, const int *count, const int *sorted, int *par, int *err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const double *ri = rows + (int64_t)width * i;
  const int c = cell[i];
  const int cx = c % G, cy = (c / G) % G, cz = c / (G * G);
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int nc = ((cz + dz + G) % G * G + (cy + dy + G) % G) * G + (cx + dx + G) % G;
        for (int q = start[nc]; q < start[nc] + count[nc]; ++q) {
          const int j = sorted[q];
          if (j <= i) continue;
          if (lat_dist_periodic(n, ri, rows + (int64_t)width * j) <= th) uf_union(par, i, j, err);
        }
      }
}

__global__ void k_grp_link_all(const double *rows, int width, int np, int n, double th, int *par, int *err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const double *ri = rows + (int64_t)width * i;
  for (int j = i + 1; j < np; ++j)
    if (lat_dist_periodic(n, ri, rows + (int64_t)width * j) <= th) uf_union(par, i, j, err);
}

__global__ void k_grp_label(double *rows, int width, int gcol, int vcol, int np, int *par, double *tot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const int g = uf_find(par, i);
  rows[(int64_t)width * i + gcol] = (double)g;
  atomicAdd(&tot[g], rows[(int64_t)width * i + vcol]);
}

__global__ void k_grp_out(const int *par, const double *tot, int np, double t2, double t3, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np || par[i] != i) return;
  atomicAdd(&out[0], tot[i]);
  if (tot[i] > t2) atomicAdd(&out[1], tot[i]);
  if (tot[i] > t3) atomicAdd(&out[2], tot[i]);
  atomicAdd(&out[3], 1.0);
}

int grid_for(int64_t count, int per = 256) {
  int64_t b = (count + per - 1) / per;
  if (b > 152 * 32) b = 152 * 32;
  return (int)(b < 1 ? 1 : b);
}

// planes a CTA of the cell passes walks: 32 (one extra plane of phases in 32),
// fewer on small lattices so that about four CTAs per SM remain
dim3 cell_grid(int n, int *zc) {
  const unsigned gx = (unsigned)((n + kCellX - 1) / kCellX), gy = (unsigned)((n + kCellY - 1) / kCellY);
  int c = kCellZ;
  while (c > 2 && (int64_t)gx * gy * ((n + c - 1) / c) < 4 * 152) c /= 2;
  *zc = c;
  return dim3(gx, gy, (unsigned)((n + c - 1) / c));
}

// grouping_strings / grouping_walls + the grouped branch of add_string_length
// / add_wall_area: out = (all, groups above t2, groups above t3, #groups)
int group_and_sum(axg_ctx *ctx, double *rows, int width, int gcol, int vcol, int64_t np64, double th, double t2,
                  double t3, double out[4]) {
  const int np = (int)np64;
  const int n = (int)ctx->n;
  int G = (int)std::floor(n / th);
  if (G > 64) G = 64;
  const bool grid = G >= 3;
  const int ncell = grid ? G * G * G : 1;
  int *ib = nullptr;
  double *db = nullptr;
  int rc = AXG_OK;
  auto cleanup = axg_on_exit([&] {
    cudaStreamSynchronize(ctx->stream);
    axg_free(ctx, (void **)&ib);
    axg_free(ctx, (void **)&db);
  });
  AXG_TRY(axg_alloc(ctx, (void **)&ib, sizeof(int) * ((size_t)4 * np + 3 * (size_t)ncell + 4), "grouping"));
  do {
    if ((rc = axg_alloc(ctx, (void **)&db, sizeof(double) * ((size_t)np + 4), "group totals"))) break;
    int *par = ib, *cell = ib + np, *sorted = ib + 2 * np, *count = ib + 3 * (size_t)np,
        *start = count + ncell, *fill = start + ncell;
    double *tot = db, *dout = db + np;
    AXG_CUDA_TRY(ctx, cudaMemsetAsync(ib + 3 * (size_t)np, 0, sizeof(int) * 3 * (size_t)ncell, ctx->stream));
    AXG_CUDA_TRY(ctx, cudaMemsetAsync(db, 0, sizeof(double) * ((size_t)np + 4), ctx->stream));
    const int blocks = (np + 255) / 256;
    AXG_LAUNCH(ctx, "group_init", k_grp_init, blocks, 256, 0, par, np);
    if (grid) {
      AXG_LAUNCH(ctx, "group_count", k_grp_count, blocks, 256, 0, rows, width, np, n, G, cell, count);
      AXG_CUDA_TRY(ctx, cudaMemcpyAsync(start, count, sizeof(int) * ncell, cudaMemcpyDeviceToDevice, ctx->stream));
      AXG_LAUNCH(ctx, "group_scan", k_scan_int, 1, 1024, 0, start, ncell);
      AXG_LAUNCH(ctx, "group_scatter", k_grp_scatter, blocks, 256, 0, cell, np, start, fill, sorted);
      AXG_LAUNCH(ctx, "group_link", k_grp_link, blocks, 256, 0, rows, width, np, n, G, th, cell, start, count, sorted,
                 par, ctx->d_err);
    } else {
      AXG_LAUNCH(ctx, "group_link_all", k_grp_link_all, blocks, 256, 0, rows, width, np, n, th, par, ctx->d_err);
    }
    AXG_LAUNCH(ctx, "group_label", k_grp_label, blocks, 256, 0, rows, width, gcol, vcol, np, par, tot);
    AXG_LAUNCH(ctx, "group_out", k_grp_out, blocks, 256, 0, par, tot, np, t2, t3, dout);
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(out, dout, sizeof(double) * 4, cudaMemcpyDeviceToHost, ctx->stream));
    AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    rc = axg_evo_check_error(ctx);
  } while (0);
  return rc;
}

// grouping threshold max(2, (width^2 hor)^(1/3)) (defects_3d.f90:1245-1246)
double group_threshold(double wid, double hor) {
  const double th = std::pow(wid * wid * hor, 1.0 / 3.0);
  return th > 2.0 ? th : 2.0;
}

}  // namespace

int axg_def_classify(axg_ctx *ctx, int which, int64_t counts[3]) {
  if (!ctx->flags) AXG_TRY(axg_alloc(ctx, (void **)&ctx->flags, (size_t)ctx->n3, "defect flags"));
  AXG_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_cnt, 0, 3 * sizeof(unsigned long long), ctx->stream));
  const int n = (int)ctx->n;
  int zc;
  const dim3 grid = cell_grid(n, &zc), block(kCellX, kCellY);
  const bool f32 = ctx->p.precision == AXG_PREC_FP32_MIXED;
  const auto *c32 = (const float2 *)ctx->cphi;
  if (f32 && which == 7)
    AXG_LAUNCH(ctx, "defect_classify", (k_classify<float2, 7>), grid, block, 0, (const float2 *)ctx->phi[ctx->cur], c32,
               n, zc, which, ctx->flags, ctx->d_cnt);
  else if (f32)
    AXG_LAUNCH(ctx, "defect_classify", (k_classify<float2, -1>), grid, block, 0, (const float2 *)ctx->phi[ctx->cur], c32,
               n, zc, which, ctx->flags, ctx->d_cnt);
  else if (which == 7)
    AXG_LAUNCH(ctx, "defect_classify", (k_classify<double2, 7>), grid, block, 0, (const double2 *)ctx->phi[ctx->cur],
               (const double2 *)nullptr, n, zc, which, ctx->flags, ctx->d_cnt);
  else
    AXG_LAUNCH(ctx, "defect_classify", (k_classify<double2, -1>), grid, block, 0, (const double2 *)ctx->phi[ctx->cur],
               (const double2 *)nullptr, n, zc, which, ctx->flags, ctx->d_cnt);
  unsigned long long h[3];
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(h, ctx->d_cnt, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  for (int k = 0; k < 3; ++k) counts[k] = (int64_t)h[k];
  ctx->flags_valid = true;
  ctx->last_ns = counts[0];
  ctx->last_nw = counts[1];
  ctx->last_nm = counts[2];
  return AXG_OK;
}

int axg_def_winding(axg_ctx *ctx, int64_t counts[3]) {
  AXG_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_cnt + 3, 0, 3 * sizeof(unsigned long long), ctx->stream));
  const int n = (int)ctx->n;
  int zc;
  const dim3 grid = cell_grid(n, &zc), block(kCellX, kCellY);
  if (ctx->p.precision == AXG_PREC_FP32_MIXED)
    AXG_LAUNCH(ctx, "string_winding", k_winding<float2>, grid, block, 0, (const float2 *)ctx->phi[ctx->cur],
               (const float2 *)ctx->cphi, n, zc, ctx->d_cnt + 3);
  else
    AXG_LAUNCH(ctx, "string_winding", k_winding<double2>, grid, block, 0, (const double2 *)ctx->phi[ctx->cur],
               (const double2 *)nullptr, n, zc, ctx->d_cnt + 3);
  unsigned long long h[3];
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(h, ctx->d_cnt + 3, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  for (int k = 0; k < 3; ++k) counts[k] = (int64_t)h[k];
  return AXG_OK;
}

int axg_def_id_defects(axg_ctx *ctx, double tau, double sl[3], double wa[3], double svel[3],
                       int64_t counts[3]) {
  const int which = ctx->p.flags & (AXG_F_ID_STRINGS | AXG_F_ID_WALLS | AXG_F_SPEC_EST);
  AXG_TRY(axg_def_classify(ctx, which, counts));
  const int64_t ns = counts[0], nw = counts[1];
  const int nb = (int)((ctx->n3 + kChunk - 1) / kChunk);
  int *bc = nullptr;
  int64_t *cells = nullptr;
  double *sim = nullptr;  // simplex scratch of the string fits
  int rc = AXG_OK;
  AXG_TRY(axg_alloc(ctx, (void **)&bc, (size_t)nb * 2 * sizeof(int), "block counts"));
  do {
    if ((rc = axg_alloc(ctx, (void **)&cells, (size_t)(ns + nw + 1) * 8, "defect cells"))) break;
    if (ns > ctx->cap_strings) {
      axg_free(ctx, (void **)&ctx->d_strings);
      ctx->cap_strings = ctx->last_ns = 0;  // until there is a list again
      if ((rc = axg_alloc(ctx, (void **)&ctx->d_strings, (size_t)ns * 13 * 8, "string list"))) break;
      ctx->cap_strings = ns;
    }
    if (nw > ctx->cap_walls) {
      axg_free(ctx, (void **)&ctx->d_walls);
      ctx->cap_walls = ctx->last_nw = 0;
      if ((rc = axg_alloc(ctx, (void **)&ctx->d_walls, (size_t)nw * 10 * 8, "wall list"))) break;
      ctx->cap_walls = nw;
    }
    AXG_LAUNCH(ctx, "defect_block_count", k_block_count, nb, kCThreads, 0, ctx->flags, ctx->n3, bc,
               bc + nb);
    AXG_LAUNCH(ctx, "defect_scan", k_scan_blocks, 1, 1024, 0, bc, bc + nb, nb);
    AXG_LAUNCH(ctx, "defect_compact", k_compact, nb, kCThreads, 0, ctx->flags, ctx->n3, bc, bc + nb,
               cells, cells + ns);
    const int n = (int)ctx->n;
    const bool f32 = ctx->p.precision == AXG_PREC_FP32_MIXED;
    if (ns + nw > 0) {
      if (!ctx->phase64) AXG_TRY(axg_alloc(ctx, (void **)&ctx->phase64, (size_t)ctx->n3 * 8, "FP64 phases"));
      if (f32)
        AXG_LAUNCH(ctx, "fit_phases_fp64", k_phase64_all<float2>, grid_for(ctx->n3), 256, 0,
                   (const float2 *)ctx->phi[ctx->cur], (const float2 *)ctx->cphi, ctx->n3, ctx->phase64);
      else
        AXG_LAUNCH(ctx, "fit_phases_fp64", k_phase64_all<double2>, grid_for(ctx->n3), 256, 0,
                   (const double2 *)ctx->phi[ctx->cur], (const double2 *)nullptr, ctx->n3, ctx->phase64);
    }
    if (ns > 0) {
      // simplex: resident CTAs only, groups take cells from a counter (d_cnt[8])
      int per_sm = 0, sms = 0;
      AXG_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_string_simplex, kFitThreads, 0));
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
      const int64_t resident = (int64_t)std::max(per_sm, 1) * std::max(sms, 1);
      unsigned long long *next = ctx->d_cnt + 8;
      constexpr int per_cta = kFitThreads / kGrp;
      // scratch: simplexes, the cells handed over to k_string_simplex_warp (at most the resident groups), their count
      const int64_t rcap = resident * per_cta;
      // (a lattice that leaves little memory is fitted in smaller rounds)
      int64_t chunk = std::min(ns, kFitChunk);
      while ((rc = axg_alloc(ctx, (void **)&sim, (size_t)(chunk * kFitStride + rcap + 1) * 8, "string fits")) ==
                 AXG_ERR_NOMEM &&
             chunk > kFitChunkMin)
        chunk = (chunk + 1) / 2;
      if (rc) break;
      int2 *rest = (int2 *)(sim + chunk * kFitStride);
      unsigned *nrest = (unsigned *)(rest + rcap);
      // few cells: a warp each from the start.  An iteration then costs the
      // issue slots of two but a third of the time (64^3, 1.5e4 cells: 9.3
      // against 11.5 ms through k_string_simplex; 128^3, 1.3e5: 30 ms through it)
      const int64_t few = 5 * (kFitThreads / 32) * resident;
      for (int64_t c0 = 0; c0 < ns; c0 += chunk) {
        const int64_t nc = std::min(chunk, ns - c0);
        AXG_LAUNCH(ctx, "string_start", k_string_start, (unsigned)((nc + per_cta - 1) / per_cta), kFitThreads, 0,
                   ctx->phase64, n, (uint64_t)ctx->p.seed, cells + c0, nc, sim);
        AXG_CUDA_TRY(ctx, cudaMemsetAsync(next, 0, sizeof(unsigned long long), ctx->stream));
        if (nc > few) {
          AXG_CUDA_TRY(ctx, cudaMemsetAsync(nrest, 0, sizeof(unsigned), ctx->stream));
          AXG_LAUNCH(ctx, "string_simplex", k_string_simplex,
                     (unsigned)std::min<int64_t>(resident, (nc + per_cta - 1) / per_cta), kFitThreads, 0, ctx->phase64,
                     n, cells + c0, nc, sim, next, rest, nrest);
          AXG_CUDA_TRY(ctx, cudaMemsetAsync(next, 0, sizeof(unsigned long long), ctx->stream));
        }
        AXG_LAUNCH(ctx, "string_simplex_warp", k_string_simplex_warp,
                   (unsigned)std::min<int64_t>(resident, nc > few ? resident : (nc + 3) / 4), kFitThreads, 0,
                   ctx->phase64, n, cells + c0, nc > few ? rest : nullptr, nrest, nc, sim, next);
        if (f32)
          AXG_LAUNCH(ctx, "string_result", k_string_result<float2>, (unsigned)((nc + 127) / 128), 128, 0,
                     (const float2 *)ctx->phi[ctx->cur], (const float2 *)ctx->cphi, (const float2 *)ctx->phid, n,
                     ctx->p.dspa, cells + c0, nc, sim, ctx->d_strings + 13 * c0);
        else
          AXG_LAUNCH(ctx, "string_result", k_string_result<double2>, (unsigned)((nc + 127) / 128), 128, 0,
                     (const double2 *)ctx->phi[ctx->cur], (const double2 *)nullptr, (const double2 *)ctx->phid, n,
                     ctx->p.dspa, cells + c0, nc, sim, ctx->d_strings + 13 * c0);
      }
    }
    if (nw > 0) {
      AXG_LAUNCH(ctx, "wall_fit", k_wall_fit, (unsigned)((nw + 127) / 128), 128, 0, ctx->phase64, n, cells + ns,
                 nw, ctx->d_walls);
    }
    static_assert(6 + 6 * kSumBlocks <= 4096, "the reduction buffer holds the sums and their parts");
    const int nsum = (int)std::min<int64_t>(kSumBlocks, (std::max(ns, nw) + 255) / 256 + 1);
    AXG_LAUNCH(ctx, "defect_sums", k_defect_sums, nsum, 256, 0, ctx->d_strings, ns, ctx->d_walls, nw, ctx->d_red + 6);
    AXG_LAUNCH(ctx, "defect_sums_total", k_defect_sums_total, 1, 256, 0, ctx->d_red + 6, nsum, ctx->d_red);
    double h[6];
    if (cudaMemcpyAsync(h, ctx->d_red, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
      rc = axg_set_error(ctx, AXG_ERR_CUDA, "defect sums");
      break;
    }
    sl[0] = sl[1] = sl[2] = h[0];
    if (h[4] > 0) {
      svel[0] = h[1] / h[4];
      svel[1] = h[2] / h[4];
      svel[2] = h[3] / h[4];
    } else {
      svel[0] = svel[1] = svel[2] = 0.0;
    }
    wa[0] = wa[1] = wa[2] = h[5];
    const double kPi = 3.14159265359, hor = tau / ctx->p.dspa;
    if ((ctx->p.flags & AXG_F_GROUP_STRINGS) && ns > 0) {
      double g[4];
      const double th = group_threshold(ctx->p.width_cr / ctx->p.dspa / tau, hor);
      if ((rc = group_and_sum(ctx, ctx->d_strings, 13, 12, 10, ns, th, 2 * hor, 2 * kPi * hor, g))) break;
      sl[0] = g[0];
      sl[1] = g[1];
      sl[2] = g[2];
    }
    if ((ctx->p.flags & AXG_F_GROUP_WALLS) && nw > 0) {
      double g[4];
      const double th = group_threshold(ctx->p.thickness_cr / ctx->p.dspa / tau, hor);
      if ((rc = group_and_sum(ctx, ctx->d_walls, 10, 9, 7, nw, th, kPi * hor * hor, 4 * kPi * hor * hor, g))) break;
      wa[0] = g[0];
      wa[1] = g[1];
      wa[2] = g[2];
    }
    ctx->last_ns = ns;
    ctx->last_nw = nw;
  } while (0);
  cudaStreamSynchronize(ctx->stream);
  axg_free(ctx, (void **)&bc);
  axg_free(ctx, (void **)&cells);
  axg_free(ctx, (void **)&sim);
  return rc;
}

extern "C" {

int axg_classify_cells(axg_ctx *ctx, int which, int64_t counts[3]) {
  if (!ctx || !counts) return AXG_ERR_ARG;
  return axg_def_classify(ctx, which & 7, counts);
}

int axg_download_defect_flags(axg_ctx *ctx, int8_t *flags) {
  if (!ctx || !flags) return AXG_ERR_ARG;
  if (!ctx->flags || !ctx->flags_valid)
    return axg_set_error(ctx, AXG_ERR_STATE, "no classification since the last state change");
  AXG_CUDA_TRY(ctx, cudaMemcpyAsync(flags, ctx->flags, (size_t)ctx->n3, cudaMemcpyDeviceToHost, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return AXG_OK;
}

int axg_string_winding(axg_ctx *ctx, int64_t counts[3]) {
  if (!ctx || !counts) return AXG_ERR_ARG;
  return axg_def_winding(ctx, counts);
}

int axg_id_defects(axg_ctx *ctx, int64_t idx, double tau, double sl[3], double wa[3], double svel[3],
                   int64_t counts[3]) {
  (void)idx;
  if (!ctx || !sl || !wa || !svel || !counts) return AXG_ERR_ARG;
  return axg_def_id_defects(ctx, tau, sl, wa, svel, counts);
}

int axg_download_defect_lists(axg_ctx *ctx, double *strings, int64_t max_strings, double *walls,
                              int64_t max_walls) {
  if (!ctx) return AXG_ERR_ARG;
  const int64_t ns = std::min(max_strings, ctx->last_ns), nw = std::min(max_walls, ctx->last_nw);
  if (strings && ns > 0 && ctx->d_strings)
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(strings, ctx->d_strings, (size_t)ns * 13 * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (walls && nw > 0 && ctx->d_walls)
    AXG_CUDA_TRY(ctx, cudaMemcpyAsync(walls, ctx->d_walls, (size_t)nw * 10 * 8, cudaMemcpyDeviceToHost, ctx->stream));
  AXG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return AXG_OK;
}

}  // extern "C"
