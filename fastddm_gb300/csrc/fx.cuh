// Block fixed-point arithmetic for the transforms of the float-float tier.
//
// A value is (h + l) units: h a 32-bit integer, l a float of order one.  The unit is common
// to a whole transform and chosen from the energy of its input, so that no sum of a pass
// can leave the 32 bits (by Cauchy-Schwarz a partial sum of K inputs is at most sqrt(K)
// times the 2-norm of the input), and l carries 24 more bits below the unit.
//
// Why: a float-float addition is 8 instructions (an exact TwoSum of the high words and the
// sum of the low ones); here the high words add exactly as integers, so an addition is one
// IADD and one FADD, which GB300 issues at full rate on different pipes.  A twiddle product
// takes four 32 x 32 -> 64-bit products (the exact high part; a quarter of the issue rate)
// and float corrections.  A radix-8 butterfly with its seven twiddles measured 407 cycles
// per warp and sub-partition against 793 in float-float.
//
// Accuracy: with the 2-norm bound the inputs' root mean square sits 2^23 units or higher for
// up to 16,000 samples, and every rounding is about 2^-25 units, so the error is 2^-48 of
// the root mean square per pass, as in float-float.  Spectra concentrated in few
// coefficients, where the structure function cancels, gain: their error stays relative to
// the root mean square, float-float's grows with the largest coefficient.
//
// Scaling: a twiddle product is v w / 2 (an int32 holds 2^31 w), so a forward pass of radix R
// raises the bound by sqrt(R) / 2; the host follows the bound through the plan (fx_constants)
// and picks the unit so that it stays below 2^31.  Inverse passes double their input first
// and do not scale: the sum of the powers bounds every value there.
#pragma once
#include "dft_consts.cuh"
#include "fddm_internal.h"
#include "fx_consts.cuh"
#include "scalar.cuh"
#include "fft.cuh"

namespace fddm {

struct fx {
  int h;
  float l;
};

// integer sums wrap in unsigned arithmetic (transforms of non-finite data may overflow;
// their results are replaced)
__device__ __forceinline__ int iadd(int a, int b) { return (int)((unsigned)a + (unsigned)b); }
__device__ __forceinline__ int isub(int a, int b) { return (int)((unsigned)a - (unsigned)b); }
__device__ __forceinline__ fx fx_add(fx a, fx b) { return {iadd(a.h, b.h), __fadd_rn(a.l, b.l)}; }
__device__ __forceinline__ fx fx_sub(fx a, fx b) { return {isub(a.h, b.h), __fsub_rn(a.l, b.l)}; }
__device__ __forceinline__ fx fx_neg(fx a) { return {isub(0, a.h), -a.l}; }
__device__ __forceinline__ cx<fx> fx_add(cx<fx> a, cx<fx> b) { return {fx_add(a.r, b.r), fx_add(a.i, b.i)}; }
__device__ __forceinline__ cx<fx> fx_sub(cx<fx> a, cx<fx> b) { return {fx_sub(a.r, b.r), fx_sub(a.i, b.i)}; }
__device__ __forceinline__ cx<fx> fx_zero() { return {{0, 0.0f}, {0, 0.0f}}; }

__device__ __forceinline__ long long mul_wide(int a, int b) { return (long long)a * (long long)b; }

constexpr long long kRound32 = 1ll << 31, kRound31 = 1ll << 30;

// p / 2^32 for p that already holds the rounding offset kRound32: the rounded integer, and the
// remainder in [-1/2, 1/2) times 2^32
struct fx_parts {
  int h;
  float rem;
};
__device__ __forceinline__ float fx_rem(unsigned lo) { return __int2float_rn((int)(lo ^ 0x80000000u)); }
__device__ __forceinline__ fx_parts fx_high32(long long p) { return {(int)(p >> 32), fx_rem((unsigned)p)}; }
// p / 2^31 for p that already holds kRound31
__device__ __forceinline__ fx_parts fx_high31(long long p) {
  const unsigned lo = (unsigned)p, hi = (unsigned)(p >> 32);
  return {(int)__funnelshift_l(lo, hi, 1), fx_rem(lo << 1)};
}
// the remainder joins the other low-order terms last, in the one rounding at full size
__device__ __forceinline__ fx fx_join(fx_parts p, float low) {
  return {p.h, __fmaf_rn(p.rem, 2.3283064365386963e-10f, low)};
}

// Twiddle table of one pass (kind 3 of the pass tables): for row m and column j the integers
// round(2^31 w) with their remainders over 2^32, (R - 1) * stride of them, then w / 2 as floats,
// as many.
struct __align__(16) fxw {
  int wr, wi;
  float dr, di;
};
struct __align__(8) fxc {
  float r, i;
};

// v w / 2
__device__ __forceinline__ cx<fx> fx_twmul(cx<fx> v, fxw w, fxc c) {
  const long long pr = mul_wide(v.i.h, -w.wi) + (mul_wide(v.r.h, w.wr) + kRound32);
  const long long pi = mul_wide(v.i.h, w.wr) + (mul_wide(v.r.h, w.wi) + kRound32);
  const float fr = __int2float_rn(v.r.h), fi = __int2float_rn(v.i.h);
  float r = __fmul_rn(fr, w.dr), i = __fmul_rn(fr, w.di);
  r = __fmaf_rn(-fi, w.di, r);
  i = __fmaf_rn(fi, w.dr, i);
  r = __fmaf_rn(v.r.l, c.r, r);
  i = __fmaf_rn(v.r.l, c.i, i);
  r = __fmaf_rn(-v.i.l, c.i, r);
  i = __fmaf_rn(v.i.l, c.r, i);
  return {fx_join(fx_high32(pr), r), fx_join(fx_high32(pi), i)};
}

// 2 a with the integer part of the low word moved to the integer (|a| < 2^30, |a.l| < 2^20):
// sums of an inverse pass let l grow to several units, which would coarsen its rounding
__device__ __forceinline__ fx fx_twice(fx a) {
  const float q = __fmaf_rn(a.l, 2.0f, 12582912.0f);  // 2 l rounds to an integer in the low mantissa bits
  const int n = isub((int)__float_as_uint(q), 0x4B400000);
  return {iadd(iadd(a.h, a.h), n), __fmaf_rn(a.l, 2.0f, -__fsub_rn(q, 12582912.0f))};
}

// v conj(w)
__device__ __forceinline__ cx<fx> fx_twmul_inv(cx<fx> v, fxw w, fxc c) {
  w.wi = -w.wi;
  w.di = -w.di;
  c.i = -c.i;
  return fx_twmul({fx_twice(v.r), fx_twice(v.i)}, w, c);
}

// v / 2, the first output of a twiddled forward pass.  A half goes down; or (NEAR) to the side that draws the low
// word to zero: always down, the low words of a long series' lowest frequencies grow to tens of units from pass
// to pass, and their roundings with them (20,000 frames of 32 x 32, 48 movies: 2-norm error of D 6.3e-15 down,
// 5.0e-15 near, 5.2e-15 in float-float).  The shorter series' error is below float-float's either way (4000
// frames: 3.7e-15 and 3.2e-15 against 5.6e-15), and near took 0.4 to 1 % of their time.
template <bool NEAR> __device__ __forceinline__ fx fx_half(fx a) {
  const int h = (NEAR ? iadd(a.h, 1 + ((int)__float_as_uint(a.l) >> 31)) : a.h) >> 1;
  return {h, __fmaf_rn(a.l, 0.5f, __int2float_rn(isub(a.h, iadd(h, h))) * 0.5f)};
}
template <bool NEAR> __device__ __forceinline__ cx<fx> fx_half(cx<fx> a) { return {fx_half<NEAR>(a.r), fx_half<NEAR>(a.i)}; }

// a sqrt(1/2)
__device__ __forceinline__ fx fx_sqrt_half(fx a) {
  const float low = __fmaf_rn(a.l, kSqrtHalfH, __fmul_rn(__int2float_rn(a.h), -5.576365324361232e-12f));
  return fx_join(fx_high31(mul_wide(a.h, 1518500250) + kRound31), low);
}

// ---------------------------------------------------------------------------
// In-register DFTs of size R (INV: conjugate), as in fft.cuh
// ---------------------------------------------------------------------------
template <bool INV>
__device__ __forceinline__ void fx_dft4(cx<fx>& x0, cx<fx>& x1, cx<fx>& x2, cx<fx>& x3) {
  const cx<fx> t0 = fx_add(x0, x2), t1 = fx_sub(x0, x2), t2 = fx_add(x1, x3), d = fx_sub(x1, x3);
  x0 = fx_add(t0, t2);
  x2 = fx_sub(t0, t2);
  const cx<fx> m = {fx_add(t1.r, d.i), fx_sub(t1.i, d.r)};  // t1 - i d
  const cx<fx> p = {fx_sub(t1.r, d.i), fx_add(t1.i, d.r)};  // t1 + i d
  x1 = INV ? p : m;
  x3 = INV ? m : p;
}

template <bool INV>
__device__ __forceinline__ void fx_dft8_tail(cx<fx>* v, cx<fx> a0, cx<fx> a1, cx<fx> a2, cx<fx> a3, cx<fx> b0,
                                             cx<fx> b1, cx<fx> b2, cx<fx> b3) {
  if (!INV) {
    b1 = {fx_sqrt_half(fx_add(b1.r, b1.i)), fx_sqrt_half(fx_sub(b1.i, b1.r))};
    b3 = {fx_sqrt_half(fx_sub(b3.i, b3.r)), fx_sqrt_half(fx_neg(fx_add(b3.r, b3.i)))};
    b2 = {b2.i, fx_neg(b2.r)};
  } else {
    b1 = {fx_sqrt_half(fx_sub(b1.r, b1.i)), fx_sqrt_half(fx_add(b1.r, b1.i))};
    b3 = {fx_sqrt_half(fx_neg(fx_add(b3.r, b3.i))), fx_sqrt_half(fx_sub(b3.r, b3.i))};
    b2 = {fx_neg(b2.i), b2.r};
  }
  fx_dft4<INV>(a0, a1, a2, a3);
  fx_dft4<INV>(b0, b1, b2, b3);
  v[0] = a0; v[2] = a1; v[4] = a2; v[6] = a3;
  v[1] = b0; v[3] = b1; v[5] = b2; v[7] = b3;
}

// Odd radix by conjugate pairs; the cosine and sine sums accumulate in 64 bits and round once.
template <int R, bool INV> __device__ __forceinline__ void fx_dft_odd(cx<fx>* v) {
  constexpr int H = (R - 1) / 2;
  constexpr int OFF = odd_off<fx, R>::v;
  cx<fx> a[H], b[H];
#pragma unroll
  for (int r = 1; r <= H; ++r) {
    a[r - 1] = fx_add(v[r], v[R - r]);
    b[r - 1] = fx_sub(v[r], v[R - r]);
  }
  const cx<fx> x0 = v[0];
#pragma unroll
  for (int r = 0; r < H; ++r) v[0] = fx_add(v[0], a[r]);
#pragma unroll
  for (int m = 1; m <= H; ++m) {
    long long cr = kRound31, ci = kRound31, sr = kRound31, si = kRound31;
    float clr = x0.r.l, cli = x0.i.l, slr = 0.0f, sli = 0.0f;
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      const int idx = OFF + (r * m) % R;
      const int C = kFxCosI[idx], S = kFxSinI[idx];
      const float c = kCosH[idx], s = kSinH[idx], dc = kFxCosR[idx], ds = kFxSinR[idx];
      const cx<fx> x = a[r - 1], y = b[r - 1];
      cr += mul_wide(x.r.h, C);
      ci += mul_wide(x.i.h, C);
      sr += mul_wide(y.r.h, S);
      si += mul_wide(y.i.h, S);
      clr = __fmaf_rn(__int2float_rn(x.r.h), dc, __fmaf_rn(x.r.l, c, clr));
      cli = __fmaf_rn(__int2float_rn(x.i.h), dc, __fmaf_rn(x.i.l, c, cli));
      slr = __fmaf_rn(__int2float_rn(y.r.h), ds, __fmaf_rn(y.r.l, s, slr));
      sli = __fmaf_rn(__int2float_rn(y.i.h), ds, __fmaf_rn(y.i.l, s, sli));
    }
    const fx pr = fx_join(fx_high31(cr), clr), pi = fx_join(fx_high31(ci), cli);
    const cx<fx> re = {{iadd(x0.r.h, pr.h), pr.l}, {iadd(x0.i.h, pi.h), pi.l}};
    const cx<fx> im = {fx_join(fx_high31(sr), slr), fx_join(fx_high31(si), sli)};
    const cx<fx> lo = {fx_add(re.r, im.i), fx_sub(re.i, im.r)};  // re - i im
    const cx<fx> hi = {fx_sub(re.r, im.i), fx_add(re.i, im.r)};  // re + i im
    v[m] = INV ? hi : lo;
    v[R - m] = INV ? lo : hi;
  }
}

template <int R, bool INV> __device__ __forceinline__ void fx_dft(cx<fx>* v) {
  if constexpr (R == 2) {
    const cx<fx> a = fx_add(v[0], v[1]);
    v[1] = fx_sub(v[0], v[1]);
    v[0] = a;
  } else if constexpr (R == 4) {
    fx_dft4<INV>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    fx_dft8_tail<INV>(v, fx_add(v[0], v[4]), fx_add(v[1], v[5]), fx_add(v[2], v[6]), fx_add(v[3], v[7]),
                      fx_sub(v[0], v[4]), fx_sub(v[1], v[5]), fx_sub(v[2], v[6]), fx_sub(v[3], v[7]));
  } else {
    fx_dft_odd<R, INV>(v);
  }
}

// Forward DFT whose upper half of inputs is zero (R = 2, 4, 8)
template <int R> __device__ __forceinline__ void fx_dft_halfzero(cx<fx>* v) {
  if constexpr (R == 8) {
    fx_dft8_tail<false>(v, v[0], v[1], v[2], v[3], v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 4) {
    const cx<fx> x0 = v[0], x1 = v[1];
    v[0] = fx_add(x0, x1);
    v[2] = fx_sub(x0, x1);
    v[1] = {fx_add(x0.r, x1.i), fx_sub(x0.i, x1.r)};
    v[3] = {fx_sub(x0.r, x1.i), fx_add(x0.i, x1.r)};
  } else {
    v[1] = v[0];
  }
}

// ---------------------------------------------------------------------------
// In-place passes over `nfft` transforms of length n in swizzled shared memory (the
// counterparts of fft.cuh's; same positions, same digit-reversed order).  NEAR as in fx_half.
// ---------------------------------------------------------------------------
template <int R, bool INV, bool NEAR>
__device__ __forceinline__ void fx_pass(cx<fx>* __restrict__ buf, int nfft, int ld, int n, int M, unsigned rs,
                                        unsigned rb, const void* __restrict__ table, int tid, int nthr) {
  const int stride = M / R, bpf = n / R;
  const int total = nfft * bpf;
  const fxw* tw = reinterpret_cast<const fxw*>(table);
  const fxc* tc = reinterpret_cast<const fxc*>(tw + (R - 1) * stride);
  for (int beta = tid; beta < total; beta += nthr) {
    const int f = nfft > 1 ? div_by(beta, rb) : 0, loc = beta - f * bpf;
    const int blk = div_by(loc, rs), j = loc - blk * stride;
    const int base = f * ld + blk * M + j;
    cx<fx> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = buf[swz<fx>(base + r * stride)];
    if (stride > 1) {
      const fxw* w = tw + j;
      const fxc* c = tc + j;
      if (INV) {
#pragma unroll
        for (int m = 1; m < R; ++m) v[m] = fx_twmul_inv(v[m], w[(m - 1) * stride], c[(m - 1) * stride]);
        fx_dft<R, true>(v);
      } else {
        fx_dft<R, false>(v);
        v[0] = fx_half<NEAR>(v[0]);
#pragma unroll
        for (int m = 1; m < R; ++m) v[m] = fx_twmul(v[m], w[(m - 1) * stride], c[(m - 1) * stride]);
      }
    } else {
      fx_dft<R, INV>(v);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) buf[swz<fx>(base + r * stride)] = v[r];
  }
}

// Passes of power-of-two transforms with every size known at compile time (the temporal
// kernel's common lengths): element r of a butterfly sits at a constant distance from the first,
// up to the swizzle's low bits, and twiddles at constant distances from the column's first, so
// the address arithmetic of the general pass (about a quarter of its instructions) goes away.
template <int R, int M> struct fx_slots {
  static constexpr int S = M / R;
  // base has zeros where r * S has bits, and swz is linear over exclusive or
  static __device__ __forceinline__ int at(int sbase, int r) {
    const int c = (r * S) ^ (((r * S) >> 3) & 7);
    return (sbase ^ (c & 63)) + (c & ~63);
  }
};
template <int R, int M> __device__ __forceinline__ int fx_base(int beta) {
  constexpr int S = M / R;
  return swz<fx>((beta / S) * M + beta % S);  // S is a power of two
}

// Twiddled forward pass over two transforms of length n at once (the second at buf + n): a
// thread takes the same butterfly of both, so each twiddle is loaded once for two products.
template <int R, int M>
__device__ __forceinline__ void fx_pass_two(cx<fx>* __restrict__ buf, int n, const void* __restrict__ table, int tid,
                                            int nthr) {
  constexpr int S = M / R;
  const fxw* tw = reinterpret_cast<const fxw*>(table);
  const fxc* tc = reinterpret_cast<const fxc*>(tw + (R - 1) * S);
  for (int beta = tid; beta < n / R; beta += nthr) {
    const int sb = fx_base<R, M>(beta);
    const fxw* w = tw + beta % S;
    const fxc* c = tc + beta % S;
    cx<fx> v[R], u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = buf[fx_slots<R, M>::at(sb, r)];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = buf[n + fx_slots<R, M>::at(sb, r)];
    fx_dft<R, false>(v);
    fx_dft<R, false>(u);
    buf[sb] = fx_half<false>(v[0]);
    buf[n + sb] = fx_half<false>(u[0]);
#pragma unroll
    for (int m = 1; m < R; ++m) {
      const fxw wm = w[(m - 1) * S];
      const fxc cm = c[(m - 1) * S];
      buf[fx_slots<R, M>::at(sb, m)] = fx_twmul(v[m], wm, cm);
      buf[n + fx_slots<R, M>::at(sb, m)] = fx_twmul(u[m], wm, cm);
    }
  }
}

template <int R, int M>
__device__ __forceinline__ void fx_pass_inverse(cx<fx>* __restrict__ buf, int n, const void* __restrict__ table, int tid,
                                                int nthr) {
  constexpr int S = M / R;
  const fxw* tw = reinterpret_cast<const fxw*>(table);
  const fxc* tc = reinterpret_cast<const fxc*>(tw + (R - 1) * S);
  for (int beta = tid; beta < n / R; beta += nthr) {
    const int sb = fx_base<R, M>(beta);
    const fxw* w = tw + beta % S;
    const fxc* c = tc + beta % S;
    cx<fx> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = buf[fx_slots<R, M>::at(sb, r)];
#pragma unroll
    for (int m = 1; m < R; ++m) v[m] = fx_twmul_inv(v[m], w[(m - 1) * S], c[(m - 1) * S]);
    fx_dft<R, true>(v);
#pragma unroll
    for (int r = 0; r < R; ++r) buf[fx_slots<R, M>::at(sb, r)] = v[r];
  }
}

template <bool INV, bool NEAR = false>
__device__ __forceinline__ void fx_pass_dispatch(cx<fx>* buf, int nfft, int ld, const FftPlan& p, int s, int tid,
                                                 int nthr) {
  const int n = p.n, M = p.block[s];
  const unsigned rs = p.rstride[s], rb = p.rbpf[s];
  const void* t = p.ptw[s];
  switch (p.radix[s]) {
    case 2: fx_pass<2, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 4: fx_pass<4, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 8: fx_pass<8, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 3: fx_pass<3, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 5: fx_pass<5, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 7: fx_pass<7, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 11: fx_pass<11, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    case 13: fx_pass<13, INV, NEAR>(buf, nfft, ld, n, M, rs, rb, t, tid, nthr); break;
    default: break;
  }
}

// First forward pass of one zero-padded transform (zeros at indices >= limit, limit <= n/2,
// neither loaded nor written beforehand); radix 2, 4 or 8.
template <int R>
__device__ __forceinline__ void fx_first_pass_padded(cx<fx>* __restrict__ buf, const FftPlan& p, int limit, int tid,
                                                     int nthr) {
  const int stride = p.n / R;
  const fxw* tw = reinterpret_cast<const fxw*>(p.ptw[0]);
  const fxc* tc = reinterpret_cast<const fxc*>(tw + (R - 1) * stride);
  for (int j = tid; j < stride; j += nthr) {
    cx<fx> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int idx = j + r * stride;
      v[r] = r < R / 2 && idx < limit ? buf[swz<fx>(idx)] : fx_zero();
    }
    fx_dft_halfzero<R>(v);
    if (stride > 1) {
      if (R == 2) {  // x_t and x_t w_N^t: nothing is summed, so nothing is scaled
        v[1] = fx_twmul(fx_add(v[1], v[1]), tw[j], tc[j]);
      } else {
        v[0] = fx_half<false>(v[0]);
#pragma unroll
        for (int m = 1; m < R; ++m) v[m] = fx_twmul(v[m], tw[(m - 1) * stride + j], tc[(m - 1) * stride + j]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) buf[swz<fx>(j + r * stride)] = v[r];
  }
}

// Forward transform of a zero-padded input; the plan starts with radix 2, 4 or 8.
__device__ __forceinline__ void fx_forward_padded(cx<fx>* buf, const FftPlan& p, int limit, int tid, int nthr) {
  switch (p.radix[0]) {
    case 2: fx_first_pass_padded<2>(buf, p, limit, tid, nthr); break;
    case 4: fx_first_pass_padded<4>(buf, p, limit, tid, nthr); break;
    default: fx_first_pass_padded<8>(buf, p, limit, tid, nthr); break;
  }
  __syncthreads();
  for (int s = 1; s < p.npass; ++s) {
    fx_pass_dispatch<false>(buf, 1, p.n, p, s, tid, nthr);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Conversions and squares
// ---------------------------------------------------------------------------
// a s (s a power of two, |a s| < 2^31) as a fixed-point value.  The low word of a float-float
// number may reach half a unit in the last place of the high word, many units here: its
// integer part moves to h.
__device__ __forceinline__ fx fx_from_ff(ff a, float s) {
  const float t = __fmul_rn(a.h, s);
  const int h1 = __float2int_rn(t);
  const float v = __fmaf_rn(a.l, s, __fsub_rn(t, __int2float_rn(h1)));
  const float q = __fadd_rn(v, 12582912.0f);  // |v| < 2^8: v rounds to an integer in the low mantissa bits
  return {iadd(h1, isub((int)__float_as_uint(q), 0x4B400000)), __fsub_rn(v, __fsub_rn(q, 12582912.0f))};
}

// |z|^2 in square units without the squares of the low words, rounded to an integer
__device__ __forceinline__ long long fx_sqsum64(cx<fx> z) {
  const float c = __fmaf_rn(__int2float_rn(z.i.h), z.i.l, __fmul_rn(__int2float_rn(z.r.h), z.r.l));
  return mul_wide(z.r.h, z.r.h) + (mul_wide(z.i.h, z.i.h) + (long long)__float2int_rn(__fadd_rn(c, c)));
}

// a 2^u (mul = 2^u, mulf the same as a float; |a| 2^u < 2^31, |a.l| 2^u < 2^20), the integer part of
// the low word in h
__device__ __forceinline__ fx fx_times(fx a, int mul, float mulf) {
  const float q = __fmaf_rn(a.l, mulf, 12582912.0f);  // the low word rounds to an integer in the low mantissa bits
  const int n = isub((int)__float_as_uint(q), 0x4B400000);
  return {a.h * mul + n, __fmaf_rn(a.l, mulf, -__fsub_rn(q, 12582912.0f))};
}

// ---------------------------------------------------------------------------
// 64-bit values (units of 2^-32): the powers, and the first inverse pass over them, whose
// sums are exact
// ---------------------------------------------------------------------------
struct __align__(16) cx64 {
  long long r, i;
};
__device__ __forceinline__ cx64 add64(cx64 a, cx64 b) { return {a.r + b.r, a.i + b.i}; }
__device__ __forceinline__ cx64 sub64(cx64 a, cx64 b) { return {a.r - b.r, a.i - b.i}; }
__device__ __forceinline__ fx fx_from64(long long p) { return fx_join(fx_high32(p + kRound32), 0.0f); }
__device__ __forceinline__ cx<fx> fx_from64(cx64 a) { return {fx_from64(a.r), fx_from64(a.i)}; }

// a with the integer part of the low word in h
__device__ __forceinline__ fx fx_settle(fx a) {
  const float q = __fadd_rn(a.l, 12582912.0f);
  return {iadd(a.h, isub((int)__float_as_uint(q), 0x4B400000)), __fsub_rn(a.l, __fsub_rn(q, 12582912.0f))};
}

// |z|^2 2^up (0 <= up <= kMaxPowerShift; c = 2^(up - 5)); the low words' part is rounded to 2^-26.
// The low words of coefficients that sum many values reach tens of units: settled first.
__device__ __forceinline__ long long fx_power64(cx<fx> z, int up, float c) {
  z = {fx_settle(z.r), fx_settle(z.i)};
  const float c2 = 0.5f * c;  // l (2 h + l)
  const float low = __fmaf_rn(z.i.l, __fmaf_rn(__int2float_rn(z.i.h), c, __fmul_rn(z.i.l, c2)),
                              __fmul_rn(z.r.l, __fmaf_rn(__int2float_rn(z.r.h), c, __fmul_rn(z.r.l, c2))));
  const long long p = mul_wide(z.r.h, z.r.h) + mul_wide(z.i.h, z.i.h);
  return (long long)((unsigned long long)p << up) + mul_wide(__float2int_rn(low), 64);
}
constexpr int kMaxPowerShift = 8;

// x sqrt(1/2) to the last unit (|x| < 2^63): with x = h 2^32 + l, C = round(2^31 sqrt(1/2)) and
// K = 2^33 (2^31 sqrt(1/2) - C) rounded, 2 h C + (l C) / 2^31 + (h K) / 2^32
__device__ __forceinline__ long long sqrt_half64(long long x) {
  const int C = 1518500250, K = -102865788;
  const int h = (int)((x + kRound32) >> 32), l = (int)((unsigned)x);
  return 2 * mul_wide(h, C) + (mul_wide(l, C) >> 31) + (mul_wide(h, K) >> 32);
}

template <bool INV> __device__ __forceinline__ void dft4_64(cx64& x0, cx64& x1, cx64& x2, cx64& x3) {
  const cx64 t0 = add64(x0, x2), t1 = sub64(x0, x2), t2 = add64(x1, x3), d = sub64(x1, x3);
  x0 = add64(t0, t2);
  x2 = sub64(t0, t2);
  x1 = INV ? cx64{t1.r - d.i, t1.i + d.r} : cx64{t1.r + d.i, t1.i - d.r};
  x3 = INV ? cx64{t1.r + d.i, t1.i - d.r} : cx64{t1.r - d.i, t1.i + d.r};
}

// Inverse DFT of size R of 64-bit values, outputs in fixed point
template <int R> __device__ __forceinline__ void fx_first_inverse(const cx64* z, cx<fx>* v) {
  if constexpr (R == 2) {
    v[0] = fx_from64(add64(z[0], z[1]));
    v[1] = fx_from64(sub64(z[0], z[1]));
  } else if constexpr (R == 4) {
    cx64 a[4] = {z[0], z[1], z[2], z[3]};
    dft4_64<true>(a[0], a[1], a[2], a[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = fx_from64(a[k]);
  } else if constexpr (R == 8) {  // even outputs from the sums, odd ones from the rotated differences
    cx64 a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = add64(z[k], z[k + 4]);
    dft4_64<true>(a[0], a[1], a[2], a[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[2 * k] = fx_from64(a[k]);
    const cx64 b1 = sub64(z[1], z[5]), b2 = sub64(z[2], z[6]), b3 = sub64(z[3], z[7]);
    a[0] = sub64(z[0], z[4]);
    a[1] = {sqrt_half64(b1.r - b1.i), sqrt_half64(b1.r + b1.i)};
    a[2] = {-b2.i, b2.r};
    a[3] = {sqrt_half64(-(b3.r + b3.i)), sqrt_half64(b3.r - b3.i)};
    dft4_64<true>(a[0], a[1], a[2], a[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[2 * k + 1] = fx_from64(a[k]);
  } else {
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = fx_from64(z[k]);
    fx_dft<R, true>(v);
  }
}

// The inverse pass of stride 1 over the paired powers, in place
template <int R> __device__ __forceinline__ void fx_first_inverse_pass(cx<fx>* __restrict__ buf, int n, int tid, int nthr) {
  for (int b = tid; b < n / R; b += nthr) {
    cx64 z[R];
    cx<fx> v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) z[i] = *reinterpret_cast<const cx64*>(&buf[swz<fx>(b * R + i)]);
    fx_first_inverse<R>(z, v);
#pragma unroll
    for (int i = 0; i < R; ++i) buf[swz<fx>(b * R + i)] = v[i];
  }
}
__device__ __forceinline__ void fx_first_inverse_dispatch(cx<fx>* buf, int R, int n, int tid, int nthr) {
  switch (R) {
    case 2: fx_first_inverse_pass<2>(buf, n, tid, nthr); break;
    case 4: fx_first_inverse_pass<4>(buf, n, tid, nthr); break;
    case 8: fx_first_inverse_pass<8>(buf, n, tid, nthr); break;
    case 3: fx_first_inverse_pass<3>(buf, n, tid, nthr); break;
    case 5: fx_first_inverse_pass<5>(buf, n, tid, nthr); break;
    case 7: fx_first_inverse_pass<7>(buf, n, tid, nthr); break;
    case 11: fx_first_inverse_pass<11>(buf, n, tid, nthr); break;
    case 13: fx_first_inverse_pass<13>(buf, n, tid, nthr); break;
    default: break;
  }
}

}  // namespace fddm
