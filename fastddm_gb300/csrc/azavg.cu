// Azimuthal average: weighted per-bin mean and unbiased weighted standard
// deviation of every row of a stack of half-plane maps.
//
// Bound: the FP64 pipe (64 cycles per warp instruction).  Each thread owns one (bin, row) and adds up the
// bin's pixels in increasing pixel order, evaluating term = (x * w) / sum_w and err += (w * (x - mean)^2) / bias
// with explicitly rounded FP64 operations (no FMA contraction).  That is the
// operation order of the reference's per-pixel loops
// (src/python/azimuthalaverage.py:435-444, :457-476), so the sums are
// reproducible and independent of scheduling.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include "fddm_b200.h"
#include "fddm_internal.h"

namespace {

// x / b correctly rounded, for one b and many x.  The FP64 pipe takes 64 cycles per warp instruction
// on this part and the library division about ten of them; with the reciprocal of b to twice the
// precision (rh + rl), a quotient within one unit in the last place takes two (q0), and Markstein's
// theorem (P. Markstein, IBM J. Res. Dev. 34, 1990) makes the third and fourth, the exact remainder
// and its correction by rh, the correctly rounded x / b.  Exponents near the ends of the range, zeros,
// infinities and NaN take the library division.
struct Divisor {
  double b, rh, rl;
  bool plain;  // b is such a number
};
__device__ __forceinline__ bool far_exponent(double x) {  // outside 2^-400 .. 2^400
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7FFu;
  return e - 623u > 800u;
}
__device__ __forceinline__ Divisor divisor(double b) {
  Divisor d;
  d.b = b;
  d.rh = __drcp_rn(b);
  d.rl = __dmul_rn(__fma_rn(-b, d.rh, 1.0), d.rh);
  d.plain = far_exponent(b);
  return d;
}
__device__ __forceinline__ double near_quotient(double x, const Divisor& d) {  // of exponents in the range
  const double q = __fma_rn(x, d.rh, __dmul_rn(x, d.rl));
  return __fma_rn(__fma_rn(-q, d.b, x), d.rh, q);
}
__device__ __forceinline__ double divide(double x, const Divisor& d) {
  return d.plain || far_exponent(x) ? __ddiv_rn(x, d.b) : near_quotient(x, d);
}

// term(0) / b + term(1) / b + ... over the pixels pix[i0..i1), added one by one in that order.  The
// terms of kGroup pixels are read and divided together, the next group's loads in flight meanwhile: what
// is left in sequence is one addition a pixel.
constexpr int kGroup = 2;
template <class Term>
__device__ __forceinline__ double sum_terms(const double* __restrict__ d, const int32_t* __restrict__ pix,
                                            const double* __restrict__ w, int i0, int i1, double b, Term term) {
  const Divisor by = divisor(b);
  double acc = 0.0;
  double x[kGroup], u[kGroup];
  const int whole = i0 + (i1 - i0) / kGroup * kGroup;
  auto load = [&](int i) {
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      const int p = pix[i + j];
      x[j] = d[p];
      u[j] = w[p];
    }
  };
  if (i0 < whole) load(i0);
  for (int i = i0; i < whole; i += kGroup) {
    double t[kGroup], q[kGroup];
    bool far = by.plain;
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      t[j] = term(x[j], u[j]);
      far |= far_exponent(t[j]);
      q[j] = near_quotient(t[j], by);
    }
    if (i + kGroup < whole) load(i + kGroup);
    if (far) {
#pragma unroll
      for (int j = 0; j < kGroup; ++j) q[j] = divide(t[j], by);
    }
#pragma unroll
    for (int j = 0; j < kGroup; ++j) acc = __dadd_rn(acc, q[j]);
  }
  for (int i = whole; i < i1; ++i) {
    const int p = pix[i];
    acc = __dadd_rn(acc, divide(term(d[p], w[p]), by));
  }
  return acc;
}

// One warp: kRows rows of 32 / kRows consecutive bins.  The lanes of a bin read the same pixel list and
// weights (a warp of 32 bins spends as many cycles on reading lists as on arithmetic) and neighbouring
// bins share sectors of the map; small blocks spread the long lists over the SMs.  202 rows of
// 1024 x 513, 512 bins, lists of up to 2270 pixels: 3.2 ms with 8 rows (3.4 with 4, 3.3 with 32, 3.8 with
// 1), 6.5 ms in blocks of 128 bins and one row read one pixel at a time; 14 operations a pixel on
// the FP64 pipe are 2.5 ms.
constexpr int kRows = 8;
__global__ void __launch_bounds__(32) k_azavg(const double* __restrict__ data, int64_t nrows, int64_t npix,
                                              const int32_t* __restrict__ off, const int32_t* __restrict__ pix,
                                              int nbins, const double* __restrict__ w,
                                              const double* __restrict__ sumw, const double* __restrict__ bias,
                                              double* __restrict__ avg, double* __restrict__ err) {
  const int b = blockIdx.x * (32 / kRows) + threadIdx.x / kRows;
  const int64_t row = (int64_t)blockIdx.y * kRows + threadIdx.x % kRows;
  if (b >= nbins || row >= nrows) return;
  const double* d = data + row * npix;
  const size_t o = (size_t)b * nrows + row;
  const double sw = sumw[b];
  if (sw == 0.0) {
    avg[o] = __longlong_as_double(0x7ff8000000000000ll);
    if (err) err[o] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const int i0 = off[b], i1 = off[b + 1];
  const double mean = sum_terms(d, pix, w, i0, i1, sw, [](double x, double u) { return __dmul_rn(x, u); });
  avg[o] = mean;
  if (err) {
    const double e = sum_terms(d, pix, w, i0, i1, bias[b], [=](double x, double u) {
      const double dv = __dsub_rn(x, mean);
      return __dmul_rn(u, __dmul_rn(dv, dv));
    });
    err[o] = __dsqrt_rn(e);
  }
}

// Fast variant: one warp per (bin, row).  The lanes stride over the bin's
// pixels with FP64 fused multiply-adds, the warp combines its lanes in a fixed
// butterfly order (so results are reproducible from run to run), and the mean
// divides the weighted sum once: (sum x w) / sum_w instead of the reference's
// sum of (x w) / sum_w.  Same quantities, rounded differently (relative
// differences of order 1e-15 against the bit-exact kernel above).
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(256) k_azavg_warp(const double* __restrict__ data, int64_t nrows, int64_t npix,
                                                    const int32_t* __restrict__ off, const int32_t* __restrict__ pix,
                                                    int nbins, const double* __restrict__ w,
                                                    const double* __restrict__ sumw, const double* __restrict__ bias,
                                                    double* __restrict__ avg, double* __restrict__ err) {
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t row = blockIdx.y;
  if (b >= nbins) return;  // whole warps leave together
  const double* d = data + row * npix;
  const size_t o = (size_t)b * nrows + row;
  const double sw = sumw[b];
  if (sw == 0.0) {
    if (lane == 0) {
      avg[o] = __longlong_as_double(0x7ff8000000000000ll);
      if (err) err[o] = __longlong_as_double(0x7ff8000000000000ll);
    }
    return;
  }
  const int i0 = off[b], i1 = off[b + 1];
  double acc = 0.0;
  for (int i = i0 + lane; i < i1; i += 32) {
    const int p = pix[i];
    acc = fma(d[p], w[p], acc);
  }
  const double mean = warp_sum_d(acc) / sw;
  if (lane == 0) avg[o] = mean;
  if (err) {
    double e = 0.0;
    for (int i = i0 + lane; i < i1; i += 32) {
      const int p = pix[i];
      const double dv = d[p] - mean;
      e = fma(w[p] * dv, dv, e);
    }
    e = warp_sum_d(e);
    if (lane == 0) err[o] = sqrt(e / bias[b]);
  }
}

// Set-up on the device: the bin of every pixel, the lists of the bins' pixels in increasing order (a stable
// counting sort over chunks of pixels) and the per-bin sums, added in pixel order as the host's.
// Bound: launches and the chains of additions (a bin's sum waits for one FP64 addition a pixel).
// 525,312 pixels, 512 bins: 1.4 ms with the uploads, most of it the copies; numpy's search, sort and
// sums with the uploads 19 ms.
constexpr int kMinChunk = 1024;
constexpr int kMaxBins = 16384;

// Pixels of a chunk: 1024, or as many more as keep the table of chunks x bins within the pixels' own size (4 bytes
// each) or 16 MB.  With 1024 throughout, 4096 x 2049 pixels and 16,384 bins took 537 MB of scratch.
int64_t chunk_pixels(uint64_t npix, uint64_t nbins) {
  const uint64_t most = npix > (1u << 22) ? npix : (1u << 22);
  uint64_t chunk = kMinChunk;
  while ((npix + chunk - 1) / chunk * nbins > most) chunk *= 2;
  return (int64_t)chunk;
}

// bin (edges[bin - 1] < dist <= edges[bin]) or -1 for a pixel that takes no part, counted per chunk
__global__ void __launch_bounds__(256) k_bin_keys(const double* __restrict__ dist, const double* __restrict__ w,
                                                  const uint8_t* __restrict__ mask, int npix, int64_t chunk,
                                                  const double* __restrict__ edges, int nbins, double x_min,
                                                  int32_t* __restrict__ key, int32_t* __restrict__ count) {
  int32_t* mine = count + (size_t)blockIdx.x * nbins;
  for (int64_t j = threadIdx.x; j < chunk; j += blockDim.x) {
    const int64_t p = blockIdx.x * chunk + j;
    if (p >= npix) return;
    const double x = dist[p];
    int lo = 0, hi = nbins;  // first edge not below x; NaN is above every edge
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (edges[mid] < x || x != x) lo = mid + 1;
      else hi = mid;
    }
    const bool in = lo < nbins && !(x < x_min) && w[p] != 0.0 && (!mask || mask[p]);
    key[p] = in ? lo : -1;
    if (in) atomicAdd(mine + lo, 1);
  }
}

// count[chunk][bin] -> pixels of the bin in earlier chunks; total[bin]
__global__ void __launch_bounds__(32) k_bin_scan(int32_t* __restrict__ count, int nchunks, int nbins,
                                                 int32_t* __restrict__ total) {
  const int b = blockIdx.x * 32 + threadIdx.x;
  if (b >= nbins) return;
  int run = 0;
#pragma unroll 16
  for (int c = 0; c < nchunks; ++c) {
    const size_t i = (size_t)c * nbins + b;
    const int n = count[i];
    count[i] = run;
    run += n;
  }
  total[b] = run;
}

// off[0..nbins]: exclusive sums of the totals held in off[1..nbins]; one warp
__global__ void __launch_bounds__(32) k_bin_offsets(int32_t* __restrict__ off, int nbins) {
  const int lane = threadIdx.x;
  int base = 0;
  if (lane == 0) off[0] = 0;
  for (int b0 = 0; b0 < nbins; b0 += 32) {
    int v = b0 + lane < nbins ? off[1 + b0 + lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (b0 + lane < nbins) off[1 + b0 + lane] = base + v;
    base += __shfl_sync(0xffffffffu, v, 31);
  }
}

// one warp a chunk, 32 pixels at a time: equal keys of a step rank by lane
__global__ void __launch_bounds__(128) k_bin_scatter(const int32_t* __restrict__ key, int npix, int nchunks,
                                                     int64_t chunk, int32_t* __restrict__ next, const int32_t* __restrict__ off,
                                                     int nbins, int32_t* __restrict__ pix) {
  const int lane = threadIdx.x & 31;
  const int64_t c = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= nchunks) return;  // whole warps leave together
  int32_t* mine = next + (size_t)c * nbins;
  const int64_t end = min((c + 1) * chunk, (int64_t)npix);
  for (int64_t p0 = c * chunk; p0 < end; p0 += 32) {
    const int64_t p = p0 + lane;
    const int k = p < npix ? key[p] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, k);
    const int rank = __popc(same & ((1u << lane) - 1u));
    const int at = k >= 0 ? mine[k] : 0;
    __syncwarp();
    if (k >= 0) {
      pix[off[k] + at + rank] = (int32_t)p;
      if (rank == 0) mine[k] = at + __popc(same);
    }
    __syncwarp();
  }
}

// One warp a bin.  The terms of 32 pixels are read and computed by the lanes and added one after the
// other in pixel order (every lane holds the sum): sum of w, of w2, of dist * w / sum_w.
__device__ __forceinline__ double add_in_order(double acc, double t, int n) {
  for (int j = 0; j < n; ++j) acc = __dadd_rn(acc, __shfl_sync(0xffffffffu, t, j));
  return acc;
}
__global__ void __launch_bounds__(32) k_bin_sums(const double* __restrict__ dist, const double* __restrict__ w,
                                                 const double* __restrict__ w2, const int32_t* __restrict__ off,
                                                 const int32_t* __restrict__ pix, double* __restrict__ sumw,
                                                 double* __restrict__ bias, double* __restrict__ mean) {
  const int b = blockIdx.x, lane = threadIdx.x;
  const int i0 = off[b], i1 = off[b + 1];
  double sw = 0.0, sw2 = 0.0;
  for (int i = i0; i < i1; i += 32) {
    const int n = min(32, i1 - i);
    const int p = lane < n ? pix[i + lane] : 0;
    sw = add_in_order(sw, lane < n ? w[p] : 0.0, n);
    if (w2) sw2 = add_in_order(sw2, lane < n ? w2[p] : 0.0, n);
  }
  if (!w2) sw2 = sw;
  double k = 0.0;
  for (int i = i0; i < i1; i += 32) {
    const int n = min(32, i1 - i);
    const int p = lane < n ? pix[i + lane] : 0;
    k = add_in_order(k, lane < n ? __ddiv_rn(__dmul_rn(dist[p], w[p]), sw) : 0.0, n);
  }
  if (lane) return;
  sumw[b] = sw;
  mean[b] = k;
  if (bias) bias[b] = sw > 0.0 ? __dsub_rn(sw, __ddiv_rn(sw2, sw)) : 0.0;
}

int check_args(const double* d_data, const int32_t* d_bin_offsets, const double* d_weight, const double* d_sumw,
               const double* d_bias, const double* d_avg, const double* d_err, uint64_t nrows, uint64_t npix,
               uint64_t nbins) {
  if (!d_data || !d_bin_offsets || !d_weight || !d_sumw || !d_avg || (d_err && !d_bias))
    return fddm::fail_with(FDDM_ERR_INVALID, "null pointer argument");
  if (nrows > 65535 || nbins > (1u << 30) || npix > (1ull << 31))
    return fddm::fail_with(FDDM_ERR_UNSUPPORTED, "azimuthal average: more than 65535 rows or 2^31 pixels");
  return FDDM_OK;
}

}  // namespace

extern "C" int fddm_b200_azimuthal_average_fast(const double* d_data, uint64_t nrows, uint64_t npix,
                                                const int32_t* d_bin_offsets, const int32_t* d_bin_pixels,
                                                uint64_t nbins, const double* d_weight, const double* d_sumw,
                                                const double* d_bias, double* d_avg, double* d_err, void* stream) {
  fddm::set_last_error("");
  const int rc = check_args(d_data, d_bin_offsets, d_weight, d_sumw, d_bias, d_avg, d_err, nrows, npix, nbins);
  if (rc != FDDM_OK) return rc;
  if (nbins == 0 || nrows == 0) return FDDM_OK;
  dim3 grid((unsigned)((nbins + 7) / 8), (unsigned)nrows);
  k_azavg_warp<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_data, (int64_t)nrows, (int64_t)npix,
                                                                   d_bin_offsets, d_bin_pixels, (int)nbins, d_weight,
                                                                   d_sumw, d_bias, d_avg, d_err);
  const cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return fddm::fail_with(FDDM_ERR_CUDA, cudaGetErrorString(ce));
  fddm::count_launches(1);
  return FDDM_OK;
}

extern "C" int fddm_b200_azimuthal_average(const double* d_data, uint64_t nrows, uint64_t npix,
                                           const int32_t* d_bin_offsets, const int32_t* d_bin_pixels,
                                           uint64_t nbins, const double* d_weight, const double* d_sumw,
                                           const double* d_bias, double* d_avg, double* d_err, void* stream) {
  fddm::set_last_error("");
  const int rc = check_args(d_data, d_bin_offsets, d_weight, d_sumw, d_bias, d_avg, d_err, nrows, npix, nbins);
  if (rc != FDDM_OK) return rc;
  if (nbins == 0 || nrows == 0) return FDDM_OK;
  dim3 grid((unsigned)((nbins + 32 / kRows - 1) / (32 / kRows)), (unsigned)((nrows + kRows - 1) / kRows));
  k_azavg<<<grid, 32, 0, static_cast<cudaStream_t>(stream)>>>(d_data, (int64_t)nrows, (int64_t)npix, d_bin_offsets,
                                                              d_bin_pixels, (int)nbins, d_weight, d_sumw, d_bias,
                                                              d_avg, d_err);
  const cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return fddm::fail_with(FDDM_ERR_CUDA, cudaGetErrorString(ce));
  fddm::count_launches(1);
  return FDDM_OK;
}

extern "C" int fddm_b200_azimuthal_bins_workspace(uint64_t npix, uint64_t nbins, size_t* bytes) {
  fddm::set_last_error("");
  if (!bytes) return fddm::fail_with(FDDM_ERR_INVALID, "null pointer argument");
  if (npix == 0 || nbins == 0 || npix >= (1ull << 31) - kMinChunk || nbins > (uint64_t)kMaxBins)
    return fddm::fail_with(FDDM_ERR_UNSUPPORTED, "azimuthal bins: no pixels or bins, 2^31 pixels or more than 16384 bins");
  const uint64_t chunk = (uint64_t)chunk_pixels(npix, nbins);
  *bytes = (npix + (npix + chunk - 1) / chunk * nbins) * sizeof(int32_t);
  return FDDM_OK;
}

extern "C" int fddm_b200_azimuthal_bins(const double* d_dist, const double* d_weight, const double* d_weight2,
                                        const uint8_t* d_mask, uint64_t npix, const double* d_edges, uint64_t nbins,
                                        double x_min, void* d_workspace, size_t workspace_bytes,
                                        int32_t* d_bin_offsets, int32_t* d_bin_pixels, double* d_sumw, double* d_bias,
                                        double* d_mean, void* stream) {
  size_t need = 0;
  const int rc = fddm_b200_azimuthal_bins_workspace(npix, nbins, &need);
  if (rc != FDDM_OK) return rc;
  if (!d_dist || !d_weight || !d_edges || !d_workspace || !d_bin_offsets || !d_bin_pixels || !d_sumw || !d_mean)
    return fddm::fail_with(FDDM_ERR_INVALID, "null pointer argument");
  if (workspace_bytes < need) return fddm::fail_with(FDDM_ERR_NOMEM, "azimuthal bins: workspace too small");
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t chunk = chunk_pixels(npix, nbins);
  const int n = (int)npix, nb = (int)nbins, nchunks = (int)((npix + chunk - 1) / chunk);
  int32_t* key = static_cast<int32_t*>(d_workspace);
  int32_t* count = key + npix;
  cudaError_t ce = cudaMemsetAsync(count, 0, (size_t)nchunks * nbins * sizeof(int32_t), st);
  if (ce != cudaSuccess) return fddm::fail_with(FDDM_ERR_CUDA, cudaGetErrorString(ce));
  k_bin_keys<<<nchunks, 256, 0, st>>>(d_dist, d_weight, d_mask, n, chunk, d_edges, nb, x_min, key, count);
  k_bin_scan<<<(nb + 31) / 32, 32, 0, st>>>(count, nchunks, nb, d_bin_offsets + 1);
  k_bin_offsets<<<1, 32, 0, st>>>(d_bin_offsets, nb);
  k_bin_scatter<<<(nchunks + 3) / 4, 128, 0, st>>>(key, n, nchunks, chunk, count, d_bin_offsets, nb, d_bin_pixels);
  k_bin_sums<<<nb, 32, 0, st>>>(d_dist, d_weight, d_weight2, d_bin_offsets, d_bin_pixels, d_sumw, d_bias, d_mean);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) return fddm::fail_with(FDDM_ERR_CUDA, cudaGetErrorString(ce));
  fddm::count_launches(5);
  return FDDM_OK;
}
