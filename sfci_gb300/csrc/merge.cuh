// The cut on exact merged sums and the exact 128-bit accumulation, shared by the
// product's merge kernels (spmspv.cu, rows.cu).
#pragma once

#include <cmath>

#include "common.cuh"

namespace sfci {

// The post-merge cut |a| > cut as an integer test on the accumulated sum: sums
// whose magnitude is at most `below` (cut * 2^FX_FRAC * (1 - 2^-40), rounded
// down) cannot survive and are dropped without converting them; the rest are
// converted and compared exactly.  A negative cut keeps everything.
struct FxCut {
  u64 below_lo, below_hi;
  long long cutk;  // cut_key(cut)
  int all;
};
// the cut on a 128-bit sum (hi:lo) in units of 2^-FX_FRAC
__device__ __forceinline__ bool fx_survives_value(u64 lo, u64 hi, const FxCut& c, double& v) {
  if (!c.all) {
    u64 mlo = lo, mhi = hi;
    if ((long long)hi < 0) {
      mhi = ~hi + (lo == 0 ? 1ull : 0ull);
      mlo = 0ull - lo;
    }
    if (mhi < c.below_hi || (mhi == c.below_hi && mlo <= c.below_lo)) return false;
  }
  v = fx_to_double(lo, hi);
  return above_cut(v, c.cutk);
}
// the cut on a split accumulator (acc_hi * 2^FX_SPLIT + acc_lo)
__device__ __forceinline__ bool fx_survives(u64 acc_lo, u64 acc_hi, const FxCut& c, double& v) {
  u64 lo, hi;
  fx_value(acc_lo, acc_hi, lo, hi);
  return fx_survives_value(lo, hi, c, v);
}
inline FxCut fx_cut(double cut) {
  FxCut c{};
  c.cutk = cut_key(cut);
  c.all = cut < 0.0 ? 1 : 0;
  if (!c.all) {
    // cut * 2^FX_FRAC is exact in double; the 2^-40 margin covers the rounding
    // of the product below and of the final conversion
    const double y = std::ldexp(cut, FX_FRAC) * (1.0 - std::ldexp(1.0, -40));
    const unsigned __int128 t = y >= std::ldexp(1.0, 127) ? ~(unsigned __int128)0 >> 1 : (unsigned __int128)y;
    c.below_lo = (u64)t;
    c.below_hi = (u64)(t >> 64);
  }
  return c;
}

// add x exactly to a 128-bit fixed-point accumulator acc[0..1] (low, high):
// the carry of each low-word addition is known from its returned old value, so
// the total is the exact sum whatever the order of the additions
__device__ __forceinline__ void fx_atomic_add128(u64* acc, double x, unsigned& bad) {
  u64 l, h;
  fx128_of(x, l, h, bad);
  if ((l | h) == 0) return;
  const u64 old = atomicAdd((unsigned long long*)acc, (unsigned long long)l);
  const u64 hh = h + ((old + l < old) ? 1ull : 0ull);
  if (hh) atomicAdd((unsigned long long*)(acc + 1), (unsigned long long)hh);
}

}  // namespace sfci
