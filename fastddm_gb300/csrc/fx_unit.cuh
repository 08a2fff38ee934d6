// A mode's unit that is not a power of two: 2^-k 16 / j, j = 16 .. 31, which uses the half bit that a power of
// two leaves unused on average (the long-series and the diff kernel).
#pragma once
#include "tfx.cuh"

namespace fddm {

namespace {

// 16 / j and its square for j = 16 .. 31
__constant__ const double kUnit[16] = {1.0,       16.0 / 17, 16.0 / 18, 16.0 / 19, 16.0 / 20, 16.0 / 21,
                                       16.0 / 22, 16.0 / 23, 16.0 / 24, 16.0 / 25, 16.0 / 26, 16.0 / 27,
                                       16.0 / 28, 16.0 / 29, 16.0 / 30, 16.0 / 31};
__constant__ const double kUnit2[16] = {1.0, 256.0 / 289, 256.0 / 324, 256.0 / 361, 256.0 / 400, 256.0 / 441,
                                        256.0 / 484, 256.0 / 529, 256.0 / 576, 256.0 / 625, 256.0 / 676, 256.0 / 729,
                                        256.0 / 784, 256.0 / 841, 256.0 / 900, 256.0 / 961};

struct FxUnit {
  int k;
  float scale;         // units of one: 2^k j / 16
  double unit, unit2;  // 16 / j: a unit in 2^-k; its square
};
// The finest unit for a series of this energy (2-norm at most 2^beta units)
__device__ __forceinline__ FxUnit fx_unit(float energy, float beta) {
  const float lg = fx_log2_scale(energy, beta);
  FxUnit u;
  u.k = (int)floorf(lg);
  const int j = min(max((int)(16.0f * exp2f(lg - floorf(lg))), 16), 31);
  u.scale = __fmul_rn(pow2f(u.k), 0.0625f * (float)j);
  u.unit = kUnit[j - 16];
  u.unit2 = kUnit2[j - 16];
  return u;
}

// a s rounded to a fixed-point value as fx_from_ff, for s with five significant bits
__device__ __forceinline__ fx fx_from_ff_any(ff a, float s) {
  const float t = __fmul_rn(a.h, s), e = __fmaf_rn(a.h, s, -t);
  const int h1 = __float2int_rn(t);
  return fx_settle({h1, __fmaf_rn(a.l, s, __fadd_rn(__fsub_rn(t, __int2float_rn(h1)), e))});
}

}  // namespace

}  // namespace fddm
