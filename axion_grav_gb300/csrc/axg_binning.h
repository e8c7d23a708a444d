// axg_binning.h -- shell binning shared by the spectra.
//
// Every shell bin the spectra use (nint(q/dq + 0.5) linear bins of
// grav_waves.f90:279 and spectrum.f90:538, the log bins) is a function of
// the integer |k|^2 alone, q = sqrt(|k|^2) dk.  axg_bin_table evaluates the
// same FP64 expressions once per |k|^2 on the host and keeps the table on the
// device, so a binning kernel does one 2-byte load per k instead of an FP64
// square root, division and rounding.  Kernels add into shared-memory bins
// through BinRun: each lane sums a short run of consecutive k-sites privately
// and adds to the shared bin only when its bin changes.
#pragma once
#include <cstdint>

#include "axg_internal.h"

enum axg_bin_kind {
  AXG_BIN_GW = 0,        // q > 0, linear or log bins (grav_waves.f90:279, log edges)
  AXG_BIN_SPECTRUM = 1,  // linear bins, bin 1 includes k = 0 (spectrum.f90:538)
};

// Device table of bins (-1: outside) indexed by |k|^2 in [0, 3 (m/2)^2] for an
// m^3 lattice; edges (nb + 1 values) only for log bins.  Cached in the context.
int axg_bin_table(axg_ctx *ctx, int kind, int m, double dwav, double dq, int nb, int logmode,
                  const double *edges, const int16_t **d_tab);

// The walk of walk_spectrum below: `rows` consecutive ky a thread, its threads
// counted in 32 bits (32-bit divisions), so at most 2^31 of them.
inline int64_t walk_threads(int n, int nx, int rows) { return (int64_t)nx * n * ((n + rows - 1) / rows); }
// long runs, but at least ~8 threads for each resident one
inline int walk_rows(int n, int nx) {
  int rows = 32;
  while (rows > 2 && walk_threads(n, nx, rows) < 4 * 152 * 2048) rows /= 2;
  return rows;
}
// no runs (kernels that add every entry by itself): a row a thread, more only
// where the threads would not count in 32 bits (1025 x 2048 x 2048 is 2^32)
inline int walk_rows_single(int n, int nx) {
  int rows = 1;
  while (walk_threads(n, nx, rows) > (1LL << 31)) rows *= 2;
  return rows;
}
inline int walk_grid(int n, int nx, int rows) {
  const int64_t b = (walk_threads(n, nx, rows) + 255) / 256;
  return (int)(b > 152 * 8 ? 152 * 8 : b);
}

#ifdef __CUDACC__
#include "axg_ff.h"

// the integer wave vector of index j
__device__ __forceinline__ int kint(int j, int n) { return (j + n / 2) % n - n / 2; }

// The block's bins in shared memory (bin_smem bytes at mem): sums in `copies` copies, spread
// over a warp's lanes, and counts.  A shared double is added to by a
// compare-and-swap loop, and neighbouring lanes, whose |k| is nearly the same,
// leave a bin together: with one copy the 256^3 field spectrum was binned in
// 296 us, waiting on that, with 32 in 118 (512^3: 2.12 ms -> 0.83).
struct BlockBins {
  double *v;
  unsigned *w;
  int nb, copies;
  __device__ BlockBins(double *mem, int nb_, int copies_) : v(mem), nb(nb_), copies(copies_) {
    w = reinterpret_cast<unsigned *>(v + nb * copies);
    for (int i = threadIdx.x; i < nb * copies; i += blockDim.x) v[i] = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) w[i] = 0u;
    __syncthreads();
  }
  __device__ __forceinline__ void add(int b, double val, unsigned wt) {
    atomicAdd(&v[b * copies + (threadIdx.x & (copies - 1))], val);
    atomicAdd(&w[b], wt);
  }
  // the block's totals, times a power of two, into the global sums and counts
  __device__ void finish(double *__restrict__ sum, double *__restrict__ count, double scale = 1.0) {
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x)
      if (w[b]) {
        double t = 0.0;
        for (int c = 0; c < copies; ++c) t += v[b * copies + c];
        atomicAdd(&sum[b], t * scale);
        atomicAdd(&count[b], (double)w[b]);
      }
  }
};
// the start of a kernel's dynamic shared memory
__device__ __forceinline__ double *bins_mem() {
  extern __shared__ double axg_bins_sm[];
  return axg_bins_sm;
}
inline int bin_copies(int nb) {
  int c = 32;
  while (c > 1 && nb * c > 2048) c /= 2;
  return c;
}
inline size_t bin_smem(int nb) { return (size_t)nb * bin_copies(nb) * sizeof(double) + (size_t)nb * sizeof(unsigned); }

// Per-thread run accumulation.  A thread keeps its kx and walks rows of
// consecutive ky, so that a warp's loads are coalesced and |k| changes by less
// than one per step; it sums privately and adds to the shared bin only when
// its bin changes.  (Walking four sites along kx instead, a warp's loads were
// 32 to 64 bytes apart and every other site changed the bin.)  Val: double, or
// float-float, summed on the FP32 pipes and converted when the run ends (the
// FP64 pipe, at 1/64 of their rate, bounded a pass that converted every site).
__device__ __forceinline__ double run_sum(double a, double b) { return a + b; }
__device__ __forceinline__ F2 run_sum(F2 a, F2 b) { return f2_add(a, b); }
__device__ __forceinline__ double run_value(double a) { return a; }
__device__ __forceinline__ double run_value(F2 a) { return f2_to(a); }
// Squares of float-float values have FP32's exponents.  A sum of a site's
// squares within [2^-96, 2^116] is good to 2^-46 of itself (no error term falls
// below 2^-149) and a run of 2^9 of them stays finite; a site outside (or zero)
// is squared in FP64 and added to the block's bins by itself: 256^3 k_spec_bin
// 100 us, with every site outside 240; k_gw_bin_green 106 and 445.
__device__ __forceinline__ bool squares_fit(F2 v) {
  const unsigned lo = (127u - 96u) << 23, hi = (127u + 116u) << 23;
  return __float_as_uint(v.h) - lo <= hi - lo;
}
__device__ __forceinline__ bool squares_fit(double) { return true; }
// So that few sites are outside, the values are multiplied by a power of two
// that puts the largest of a sample, one `m` a thread of the block, at 2^34:
// sites from 2^-82 to 2^24 of it are inside, which spans the FP64 noise of a
// smooth field's spectrum.  Without it a band-limited 128^3 lattice's Green bins
// took 98 us a call instead of 60, most sites being such noise.  The sample only
// decides how fast a site is summed; finish() takes the factor out again.
struct SquareScale {
  float s = 1.f;     // 2^k
  double inv = 1.0;  // 2^-2k
  __device__ SquareScale() {}
  __device__ explicit SquareScale(float m) {
    __shared__ unsigned top;
    if (threadIdx.x == 0) top = 0u;
    __syncthreads();
    const unsigned u = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((threadIdx.x & 31) == 0 && u) atomicMax(&top, u);
    __syncthreads();
    const int e = (int)(top >> 23);
    const int k = e == 0 || e == 255 ? 0 : min(127 + 34 - e, 100);  // zeros, infinities, NaN: as they are
    s = __int_as_float((127 + k) << 23);
    inv = __hiloint2double((1023 - 2 * k) << 20, 0);
  }
};
template <typename Val>
struct BinRun {
  int bin = -1;
  Val v{};
  unsigned w = 0;  // count (or Hermitian weight sum, <= 2 per site)
  __device__ __forceinline__ void add(BlockBins &bins, int b, Val val, unsigned wt) {
    if (b != bin) {
      flush(bins);
      bin = b;
      v = val;
      w = wt;
    } else {
      v = run_sum(v, val);
      w += wt;
    }
  }
  __device__ __forceinline__ void flush(BlockBins &bins) {
    if (bin >= 0) bins.add(bin, run_value(v), w);
    bin = -1;
  }
};

// The walk: f(hx, hy, hz) for every entry of an n x n x nx spectrum (nx kx
// values a row), `rows` consecutive hy per thread.
template <typename F>
__device__ __forceinline__ void walk_spectrum(int n, int nx, int rows, F f) {
  const unsigned groups = (unsigned)((n + rows - 1) / rows), total = (unsigned)nx * groups * (unsigned)n;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const unsigned r = t / (unsigned)nx, hx = t - r * (unsigned)nx, hz = r / groups, g = r - hz * groups;
    const int y1 = min((int)(g + 1) * rows, n);
    for (int hy = (int)g * rows; hy < y1; ++hy) f((int)hx, hy, (int)hz);
  }
}
#endif
