// Order-independent (bit-reproducible) histogram sums.
//
// A contribution v (double) enters a histogram entry as the 128-bit two's-complement integer
// floor(v * 2^60), kept as two 64-bit words (lo, hi) = value mod 2^64, value >> 64.  Integer
// additions commute, so an entry accumulated by atomics from any number of threads and blocks, in
// any order, over any number of launches, holds the same bits -- the same result alone and in a
// mix of concurrent requests.  Resolution 2^-60 (8.7e-19) absolute per contribution, range
// |sum| < 2^67 (1.5e20).  Non-finite contributions cannot be represented: they are counted in one
// extra word after the entries, and the readers turn every entry of such a histogram into NaN.
//
// Layout of a histogram of n entries: words [2 i] = lo, [2 i + 1] = hi of entry i, word [2 n] =
// count of non-finite contributions; (2 n + 1) * 8 bytes, zero-initialised by the caller.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include "wbgpu_common.cuh"

typedef unsigned long long wbg_u64;

// (lo, hi) of floor(v 2^60) for finite v (of |v| >= 2^67 the nearest end of the range), from the bits of v: the FP64 pipe issues 64 times slower than the
// integer one, and its v 2^-4 - floor(v 2^-4) would round the fraction of a negative v
WBG_D void fx_split(double v, wbg_u64& lo, wbg_u64& hi) {
  const wbg_u64 u = (wbg_u64)__double_as_longlong(v);
  const int e = (int)(u >> 52) & 0x7ff;
  const wbg_u64 m = (u & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull);
  const int s = (e ? e : 1) - 1015;  // |v| 2^60 = m 2^s
  bool frac = false;                 // a fraction was cut off |v| 2^60
  if (s >= 75) {  // |v| >= 2^67
    lo = 0;
    hi = (long long)u < 0 ? 0x8000000000000000ull : 0x7fffffffffffffffull;
    return;
  }
  if (s >= 64) {
    lo = 0;
    hi = m << (s - 64);
  } else if (s > 0) {
    lo = m << s;
    hi = m >> (64 - s);
  } else {
    hi = 0;
    lo = s > -64 ? m >> -s : 0;
    frac = s > -64 ? (lo << -s) != m : m != 0;
  }
  if ((long long)u < 0) {  // floor: minus the magnitude, one less where a fraction was cut off
    lo = ~lo;
    hi = ~hi;
    if (!frac && ++lo == 0) ++hi;
  }
}

// entry += (lo, hi): the carry of the low word is taken from the value the low word held right
// before this add, so the pair is exact once every add has completed, whatever the interleaving
WBG_D void fx_add(wbg_u64* entry, wbg_u64 lo, wbg_u64 hi) {
  if (lo == 0 && hi == 0) return;
  const wbg_u64 old = atomicAdd(entry, lo);
  const wbg_u64 carry = (old + lo < old) ? 1ull : 0ull;
  if (hi + carry != 0) atomicAdd(entry + 1, hi + carry);
}

// entry += v; a non-finite v is counted in *nonfinite instead
WBG_D void fx_add_double(wbg_u64* entry, double v, wbg_u64* nonfinite) {
  if (v == 0.0) return;
  if (!isfinite(v)) {
    atomicAdd(nonfinite, 1ull);
    return;
  }
  wbg_u64 lo, hi;
  fx_split(v, lo, hi);
  fx_add(entry, lo, hi);
}

// value of an entry as a double: the three parts hi 2^4, (lo >> 32) 2^-28 and (lo & 2^32-1) 2^-60
// are exact doubles (|hi| < 2^53), summed smallest first
WBG_HD double fx_value(wbg_u64 lo, wbg_u64 hi) {
  const double a = (double)(lo & 0xffffffffull) * 0x1p-60;
  const double b = (double)(lo >> 32) * 0x1p-28;
  return (double)(long long)hi * 0x1p4 + (b + a);
}

// a block's shared-memory histogram (n entries + the non-finite count) added to a global one
WBG_D void fx_flush(const wbg_u64* sh, int n, wbg_u64* global) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) fx_add(global + 2 * i, sh[2 * i], sh[2 * i + 1]);
  if (threadIdx.x == 0 && sh[2 * n]) atomicAdd(global + 2 * n, sh[2 * n]);
}

WBG_D void fx_zero(wbg_u64* sh, int n) {
  for (int i = threadIdx.x; i < 2 * n + 1; i += blockDim.x) sh[i] = 0ull;
}

WBG_HD size_t fx_words(size_t n) { return 2 * n + 1; }
