// Row and column passes of the float-float tier for power-of-two FFT sizes, every size known at
// compile time (n = 2^LG, LG = 5 .. 12): the same transforms as k_rows / k_cols (ddm_impl.cuh).
//
// Bound: FP32 instruction issue.  Against the general kernels:
//   * shared-memory and twiddle addresses are constant distances from the butterfly's first
//     element (as in fx.cuh), no per-pass plan in registers;
//   * the row pass's first pass takes the pixels straight from the staged rows, without a
//     float-float copy of the rows in between; 8- and 16-bit pixels without a window are exact
//     in one float and so are their sums of up to eight, so its additions are single FADDs
//     instead of TwoSums;
//   * the halving of the packed rows' unpack goes into the column pass's scale.
// 12 frames of 1024 x 1024 uint8: rows 103 -> 81 us (6.92 -> 5.24 million warp instructions a frame),
// columns 134 -> 116 us (7.65 -> 6.69 million).
#pragma once
#include "ddm_impl.cuh"

namespace fddm {

// Radices: radix 8, then one or two radix-4 passes where LG is not a multiple of three (with the
// radix-4 passes first the median error of windowed stacks was 4 % larger).
__host__ __device__ constexpr int p2_passes(int LG) { return (LG + 2) / 3; }
__host__ __device__ constexpr int p2_radix(int LG, int s) { return s < p2_passes(LG) - (3 - LG % 3) % 3 ? 8 : 4; }
__host__ __device__ constexpr int p2_block(int LG, int s) {
  int m = 1 << LG;
  for (int i = 0; i < s; ++i) m /= p2_radix(LG, i);
  return m;
}
// position of coefficient k after the forward transform
__host__ __device__ constexpr int p2_perm(int LG, int k) {
  int pos = 0, m = 1 << LG;
  for (int s = 0; s < p2_passes(LG); ++s) {
    m /= p2_radix(LG, s);
    pos += (k % p2_radix(LG, s)) * m;
    k /= p2_radix(LG, s);
  }
  return pos;
}

// Slot of element i of transform f: the low three bits are exclusive-ored with the row number (as
// swz), with f, so that one element of several transforms lies in different banks, and with the
// lowest digit of the first pass (bit B0), so that consecutive coefficients do too.
template <int LG> struct p2_layout {
  static constexpr int n = 1 << LG;
  static constexpr int B0 = LG - (p2_radix(LG, 0) == 8 ? 3 : 2);
  static __host__ __device__ constexpr int low(int i) {
    return i ^ ((i >> 3) & 7) ^ (B0 >= 3 ? ((i >> B0) & 1) << 2 : 0);
  }
  static __device__ __forceinline__ int slot(int f, int i) { return f * n + (low(i) ^ (f & 7)); }
  // slot of element i + r * S from the slot of element i, where i has zeros at the bits of r * S
  template <int S> static __device__ __forceinline__ int step(int s, int r) {
    const int c = low(r * S);
    return (s ^ (c & 7)) + (c & ~7);
  }
};

// Twiddles of a thread's first butterfly in pass s: loaded before the barrier in front of the
// pass, so that the wait for the other warps covers their latency.
template <int LG, int s>
__device__ __forceinline__ void p2_twiddles(const FftPlan& p, int tid, cx<ff>* w) {
  constexpr int R = p2_radix(LG, s), S = p2_block(LG, s) / R;
  if constexpr (S > 1) {
    const cx<ff>* tw = reinterpret_cast<const cx<ff>*>(p.ptw[s]) + tid % S;
#pragma unroll
    for (int m = 1; m < R; ++m) w[m] = tw[(m - 1) * S];
  }
}

// Forward passes s, s + 1 .. last over nfft transforms, a barrier after each; w holds pass s's
// twiddles of this thread's first butterfly.
template <int LG, int s>
__device__ __forceinline__ void p2_passes_from(cx<ff>* __restrict__ buf, int nfft, const FftPlan& p, cx<ff>* w, int tid,
                                               int nthr) {
  if constexpr (s < p2_passes(LG)) {
    constexpr int n = 1 << LG, R = p2_radix(LG, s), M = p2_block(LG, s), S = M / R, bpf = n / R;
    using L = p2_layout<LG>;
    const cx<ff>* tw = reinterpret_cast<const cx<ff>*>(p.ptw[s]);
    for (int beta = tid; beta < nfft * bpf; beta += nthr) {
      const int f = beta / bpf, loc = beta % bpf, j = loc % S;
      const int sb = L::slot(f, (loc / S) * M + j);
      cx<ff> v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = buf[L::template step<S>(sb, r)];
      dft<ff, R, false>(v);
      if constexpr (S > 1) {
        if (nthr % S != 0 && beta != tid) {  // the same column otherwise
#pragma unroll
          for (int m = 1; m < R; ++m) w[m] = tw[j + (m - 1) * S];
        }
#pragma unroll
        for (int m = 1; m < R; ++m) v[m] = twmul<ff>::mul(v[m], w[m]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) buf[L::template step<S>(sb, r)] = v[r];
    }
    if constexpr (s + 1 < p2_passes(LG)) p2_twiddles<LG, s + 1>(p, tid, w);
    __syncthreads();
    p2_passes_from<LG, s + 1>(buf, nfft, p, w, tid, nthr);
  }
}

// ---------------------------------------------------------------------------
// Exact first pass: inputs whose low words are zero and whose sums of up to R are exact floats
// ---------------------------------------------------------------------------
struct cf {
  float r, i;
};
__device__ __forceinline__ cf operator+(cf a, cf b) { return {__fadd_rn(a.r, b.r), __fadd_rn(a.i, b.i)}; }
__device__ __forceinline__ cf operator-(cf a, cf b) { return {__fsub_rn(a.r, b.r), __fsub_rn(a.i, b.i)}; }
__device__ __forceinline__ cx<ff> wide(cf a) { return {{a.r, 0.0f}, {a.i, 0.0f}}; }
// exact float times float-float, not renormalised
__device__ __forceinline__ ff mul_exact(float a, ff b) {
  const float p = __fmul_rn(a, b.h);
  return {p, __fmaf_rn(a, b.l, __fmaf_rn(a, b.h, -p))};
}
// a + b, a an exact float
__device__ __forceinline__ ff add_exact(float a, ff b) {
  const ff s = two_sum(a, b.h);
  return {s.h, __fadd_rn(s.l, b.l)};
}
// a w, a exact: the dot products of ff_dot2_nn without a's low words
__device__ __forceinline__ ff dot2_exact(float a, ff b, float c, ff d) {  // a b + c d
  const float p1 = __fmul_rn(a, b.h), e1 = __fmaf_rn(a, b.h, -p1);
  const float p2 = __fmul_rn(c, d.h), e2 = __fmaf_rn(c, d.h, -p2);
  const ff s = two_sum(p1, p2);
  float lo = __fadd_rn(__fadd_rn(e1, e2), s.l);
  lo = __fmaf_rn(a, b.l, lo);
  lo = __fmaf_rn(c, d.l, lo);
  return {s.h, lo};
}
__device__ __forceinline__ cx<ff> twmul_exact(cf a, cx<ff> w) {
  return {dot2_exact(a.r, w.r, -a.i, w.i), dot2_exact(a.r, w.i, a.i, w.r)};
}

// DFT of exact inputs: outputs that stay exact in e[] (flag bit in the return mask), others in v[]
template <int R> __device__ __forceinline__ void dft_exact(const cf* x, cf* e, cx<ff>* v) {
  if constexpr (R == 4) {
    const cf t0 = x[0] + x[2], t1 = x[0] - x[2], t2 = x[1] + x[3], d = x[1] - x[3];
    e[0] = t0 + t2;
    e[1] = {__fadd_rn(t1.r, d.i), __fsub_rn(t1.i, d.r)};
    e[2] = t0 - t2;
    e[3] = {__fsub_rn(t1.r, d.i), __fadd_rn(t1.i, d.r)};
  } else {
    cf a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = x[k] + x[k + 4];
    cx<ff> unused[1];
    cf ea[4];
    dft_exact<4>(a, ea, unused);
#pragma unroll
    for (int k = 0; k < 4; ++k) e[2 * k] = ea[k];
    // odd outputs: b_r w8^r through a radix-4 transform
    const ff h = {kSqrtHalfH, kSqrtHalfL};
    const cf b0 = x[0] - x[4], b1 = x[1] - x[5], b2 = x[2] - x[6], b3 = x[3] - x[7];
    const cx<ff> c1 = {mul_exact(__fadd_rn(b1.r, b1.i), h), mul_exact(__fsub_rn(b1.i, b1.r), h)};
    const cx<ff> c3 = {mul_exact(__fsub_rn(b3.i, b3.r), h), mul_exact(-__fadd_rn(b3.r, b3.i), h)};
    const cf t0 = {__fadd_rn(b0.r, b2.i), __fsub_rn(b0.i, b2.r)};  // b0 - i b2
    const cf t1 = {__fsub_rn(b0.r, b2.i), __fadd_rn(b0.i, b2.r)};  // b0 + i b2
    const cx<ff> t2 = badd(c1, c3), d = bsub(c1, c3);
    v[1] = {add_exact(t0.r, t2.r), add_exact(t0.i, t2.i)};
    v[5] = {add_exact(t0.r, ff_neg(t2.r)), add_exact(t0.i, ff_neg(t2.i))};
    v[3] = {add_exact(t1.r, d.i), add_exact(t1.i, ff_neg(d.r))};  // t1 - i d
    v[7] = {add_exact(t1.r, ff_neg(d.i)), add_exact(t1.i, d.r)};
  }
}

// ---------------------------------------------------------------------------
// Row pass
// dynamic smem: pairs * n * cx<ff> + 2 * raw_stage_bytes + n ints
// ---------------------------------------------------------------------------
template <class IN, int LG>
__global__ void __launch_bounds__(256) k_rows_p2(const __grid_constant__ SpatialArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int n = 1 << LG, R0 = p2_radix(LG, 0), S0 = n / R0;
  constexpr bool small_int = sizeof(IN) <= 2;
  using L = p2_layout<LG>;
  cx<ff>* buf = reinterpret_cast<cx<ff>*>(smem_raw);
  const int W = a.W, H = a.H, nkx = n / 2 + 1;
  const int npairs = (H + 1) >> 1;
  const int ngroups = (npairs + a.pairs_per_block - 1) / a.pairs_per_block;
  const int nitems = ngroups * a.tc;
  const ff* win = reinterpret_cast<const ff*>(a.window_s);
  const int tid = threadIdx.x, nthr = blockDim.x;
  const bool async_raw = a.raw_stage_bytes > 0;
  unsigned char* raw[2] = {smem_raw + (size_t)a.pairs_per_block * n * sizeof(cx<ff>), nullptr};
  raw[1] = raw[0] + a.raw_stage_bytes;
  int* perm = reinterpret_cast<int*>(raw[1] + a.raw_stage_bytes);
  for (int i = tid; i < n; i += nthr) perm[i] = p2_perm(LG, i);
  const cx<ff>* tw0 = reinterpret_cast<const cx<ff>*>(a.px.ptw[0]);
  int b = 0;
  if (async_raw && (int)blockIdx.x < nitems) rows_issue_raw<ff, IN>(a, blockIdx.x, raw[0], ngroups, tid, nthr);

  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int g = item % ngroups, tl = item / ngroups;
    const int pair0 = g * a.pairs_per_block;
    const int np = min(a.pairs_per_block, npairs - pair0);
    const size_t t = (size_t)a.t0 + tl;
    if (async_raw) {
      cp_async_wait_all();
      __syncthreads();
      const int next = item + gridDim.x;
      if (next < nitems) rows_issue_raw<ff, IN>(a, next, raw[b ^ 1], ngroups, tid, nthr);
    } else {
      __syncthreads();
    }
    const int y0 = 2 * pair0;
    // first pass from the rows (staged, or in place), zero beyond the frame
    const IN* src = async_raw ? reinterpret_cast<const IN*>(raw[b])
                              : reinterpret_cast<const IN*>(a.img) + (t * H + y0) * (size_t)W;
    for (int beta = tid; beta < np * S0; beta += nthr) {
      const int p = beta / S0, j = beta % S0;
      const IN* ra = src + (size_t)(2 * p) * W;
      const bool two = y0 + 2 * p + 1 < H;
      const int sb = L::slot(p, j);
      cx<ff> v[R0];
      if (small_int && !win) {
        cf x[R0], e[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const int c = j + r * S0;
          x[r] = {c < W ? (float)ra[c] : 0.0f, c < W && two ? (float)ra[W + c] : 0.0f};
        }
        dft_exact<R0>(x, e, v);
        v[0] = wide(e[0]);
#pragma unroll
        for (int m = 1; m < R0; ++m) {
          const cx<ff> w = tw0[(m - 1) * S0 + j];
          v[m] = R0 == 4 || m % 2 == 0 ? twmul_exact(e[m], w) : twmul<ff>::mul(v[m], w);
        }
      } else {
        const ff* wa = win + (size_t)(y0 + 2 * p) * W;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const int c = j + r * S0;
          v[r] = czero<ff>();
          if (c < W) {
            v[r].r = pix<ff, IN>::get(ra, c);
            if (two) v[r].i = pix<ff, IN>::get(ra + W, c);
            if (win) {
              v[r].r = ff_mul(v[r].r, wa[c]);
              if (two) v[r].i = ff_mul(v[r].i, wa[W + c]);
            }
          }
        }
        dft<ff, R0, false>(v);
#pragma unroll
        for (int m = 1; m < R0; ++m) v[m] = twmul<ff>::mul(v[m], tw0[(m - 1) * S0 + j]);
      }
#pragma unroll
      for (int r = 0; r < R0; ++r) buf[L::template step<S0>(sb, r)] = v[r];
    }
    cx<ff> w[8];
    p2_twiddles<LG, 1>(a.px, tid, w);
    __syncthreads();
    p2_passes_from<LG, 1>(buf, np, a.px, w, tid, nthr);

    // twice the spectra of the two real rows of each pair (the column pass's scale halves them)
    const unsigned rnp = np == a.pairs_per_block ? a.rpairs : div_reciprocal_dev(np);
    cx<ff>* R = reinterpret_cast<cx<ff>*>(a.rbuf) + (size_t)tl * nkx * a.Hpad;
    for (int e = tid; e < np * nkx; e += nthr) {
      const int k = div_by(e, rnp);
      const int p = e - k * np;
      const cx<ff> zk = buf[L::slot(p, perm[k])];
      const cx<ff> zn = buf[L::slot(p, perm[(n - k) & (n - 1)])];
      cx<ff>* dst = R + (size_t)k * a.Hpad + 2 * (pair0 + p);
      dst[0] = {ff_add(zk.r, zn.r), ff_sub(zk.i, zn.i)};
      dst[1] = {ff_add(zk.i, zn.i), ff_sub(zn.r, zk.r)};
    }
    b ^= 1;
  }
}

// ---------------------------------------------------------------------------
// Column pass
// dynamic smem: 2 * cols * frames * n * cx<ff> + n ints
// ---------------------------------------------------------------------------
template <int LG>
__device__ __forceinline__ void cols_p2_issue(const SpatialArgs& a, int item, cx<ff>* buf, int ncg, unsigned rCK,
                                              int tid, int nthr) {
  constexpr int n = 1 << LG;
  const int H = a.H, nkx = a.nkx;
  const int CK = a.cols_per_block, TG = a.frames_per_block;
  const int kc0 = (item % ncg) * CK, tl0 = (item / ncg) * TG;
  const int nk = min(CK, nkx - kc0), ntg = min(TG, a.tc - tl0);
  const cx<ff>* R = reinterpret_cast<const cx<ff>*>(a.rbuf);
  for (int e = tid; e < CK * TG * n; e += nthr) {
    const int c = e >> LG, y = e & (n - 1);
    const int tl = div_by(c, rCK);
    const int kc = c - tl * CK;
    cx<ff>* dst = &buf[p2_layout<LG>::slot(c, y)];
    if (kc < nk && tl < ntg && y < H) cp_async<sizeof(cx<ff>)>(dst, &R[((size_t)(tl0 + tl) * nkx + kc0 + kc) * a.Hpad + y]);
    else *dst = czero<ff>();
  }
  cp_async_commit();
}

template <int LG>
__global__ void __launch_bounds__(512) k_cols_p2(const __grid_constant__ SpatialArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int n = 1 << LG, half = n / 2;
  using L = p2_layout<LG>;
  const int nkx = a.nkx, CK = a.cols_per_block, TG = a.frames_per_block, NB = CK * TG;
  const int ncg = (nkx + CK - 1) / CK;
  const int nitems = ncg * ((a.tc + TG - 1) / TG);
  cx<ff>* bufs[2] = {reinterpret_cast<cx<ff>*>(smem_raw), reinterpret_cast<cx<ff>*>(smem_raw) + NB * n};
  const unsigned rTG = a.rframes, rCK = a.rcols;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const ff norm = {a.norm_h, a.norm_l};
  // a power-of-two scale (nx ny a power of four) is exact
  const bool norm_p2 = a.norm_l == 0.0f && (__float_as_uint(a.norm_h) & 0x007FFFFFu) == 0u;
  cx<ff>* F = reinterpret_cast<cx<ff>*>(a.spec);
  int* perm = reinterpret_cast<int*>(bufs[1] + NB * n);
  for (int i = tid; i < n; i += nthr) perm[i] = p2_perm(LG, i);
  int b = 0;
  if ((int)blockIdx.x < nitems) cols_p2_issue<LG>(a, blockIdx.x, bufs[0], ncg, rCK, tid, nthr);

  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    cx<ff> w[8];
    p2_twiddles<LG, 0>(a.py, tid, w);
    cp_async_wait_all();
    __syncthreads();
    const int next = item + gridDim.x;
    if (next < nitems) cols_p2_issue<LG>(a, next, bufs[b ^ 1], ncg, rCK, tid, nthr);
    cx<ff>* buf = bufs[b];
    const int kc0 = (item % ncg) * CK, tl0 = (item / ncg) * TG;
    const int nk = min(CK, nkx - kc0), ntg = min(TG, a.tc - tl0);
    p2_passes_from<LG, 0>(buf, NB, a.py, w, tid, nthr);
    // scale by 1/sqrt(nx ny), y-fftshift, F[q][t]
    for (int e = tid; e < NB * n; e += nthr) {
      const int rest = div_by(e, rTG), tl = e - rest * TG;
      const int ky = div_by(rest, rCK), kc = rest - ky * CK;
      if (tl < ntg && kc < nk) {
        const cx<ff> z = buf[L::slot(tl * CK + kc, perm[ky])];
        const cx<ff> v = norm_p2 ? cx<ff>{ff_scale2(z.r, a.norm_h), ff_scale2(z.i, a.norm_h)} : cscale(z, norm);
        const size_t q = (size_t)((ky + half) & (n - 1)) * nkx + kc0 + kc;
        F[q * a.Tpad + a.t0 + tl0 + tl] = v;
      }
    }
    b ^= 1;
  }
}

}  // namespace fddm
