// Balanced digits of the split-precision slices (shared by the slicer kernels and the host-side test of the
// digit arithmetic): base 256 for up to six slices, base 128 for seven and eight (whose base-256 form would
// exceed the 53 bits of the operand).
//
// Base 256.  With the row exponent e (|a| < 2^(e-1)) and X = rint(a 2^(8S - 1 - e)), |X| <= 2^(8S-2) and
// X = sum_p d_p 256^p with d_p in [-128, 127] (|d| <= 64 for the top one).  Adding 128 in every digit turns them into
// the bytes of X + H, H = 128 (256^S - 1) / 255, so digit p is that byte with its top bit flipped.  The same count of
// slices and digit products holds four bits more at S = 5 than base 128, whose digits use half of the INT8 range.
//
// Base 128.
// With the row exponent e (|a| < 2^(e-1)) and X = rint(a 2^(7S - e)), |X| < 2^(7S-1) and
// X = sum_p d_p 128^p with d_p in [-64, 63] for p < S - 1 and the top digit in [-64, 64].
// Rounding to nearest and signed digits make both the representation error and the digit products
// left out of the kept diagonals zero-mean, so they do not add up along the contraction the way the
// errors of truncation toward zero do.  Adding H = 64 (128^S - 1) / 127 (64 in every digit) turns
// the balanced digits into the unsigned base-128 digits of X + H >= 0.
#pragma once

#include <stdint.h>

#ifndef __CUDA_ARCH__
#include <cmath>
#include <cstring>
#endif

#ifdef __CUDACC__
#define GB_DIGITS_FN __host__ __device__ __forceinline__
#else
#define GB_DIGITS_FN inline
#endif

namespace gb200 {

// H = 64 (128^S - 1) / 127, for 1 <= S <= 8
GB_DIGITS_FN uint64_t balanced_bias(int S) { return ((((uint64_t)1) << (7 * S)) - 1) / 127 * 64; }

// digit s (s = 0 the top one, weight 128^(S-1-s)) of X from U = X + balanced_bias(S) (computed
// modulo 2^64, so U >= 0 for every |X| < 2^(7S-1)), as a byte
GB_DIGITS_FN uint32_t balanced_digit_byte(uint64_t U, int S, int s) {
  const int p = S - 1 - s;
  const int d = (s == 0) ? (int)(U >> (7 * p)) - 64 : (int)((U >> (7 * p)) & 127u) - 64;
  return (uint32_t)d & 0xFFu;
}

// X + balanced_bias(S) for X = rint(x) (round to nearest, ties to even), |x| < 2^(7S-1).  For
// S <= 7 (|x| < 2^48) adding 1.5 * 2^52 leaves rint(x) in the low mantissa bits of the sum, so its
// bit pattern minus that of 1.5 * 2^52 is rint(x): one addition instead of a conversion.
GB_DIGITS_FN uint64_t balanced_input(double x, int S) {
  if (S <= 7) {
    const double t = x + 6755399441055744.0;
#ifdef __CUDA_ARCH__
    const uint64_t bits = (uint64_t)__double_as_longlong(t);
#else
    uint64_t bits;
    std::memcpy(&bits, &t, sizeof bits);
#endif
    return bits - 0x4338000000000000ull + balanced_bias(S);
  }
#ifdef __CUDA_ARCH__
  return (uint64_t)__double2ll_rn(x) + balanced_bias(S);
#else
  return (uint64_t)std::llrint(x) + balanced_bias(S);
#endif
}

// Digit s of four values at once: byte i of the word is balanced_digit_byte(U_i, S, s).  The four
// raw digits d in [0, 128] are packed first; d - 64 (mod 256) is d ^ 64 where bit 6 of d is set
// and d | 0xC0 where it is not, which three logic operations apply to all four bytes.
GB_DIGITS_FN uint32_t balanced_digit_word(uint64_t u0, uint64_t u1, uint64_t u2, uint64_t u3, int S, int s) {
  const int sh = 7 * (S - 1 - s);
  const uint32_t t0 = (uint32_t)(u0 >> sh), t1 = (uint32_t)(u1 >> sh), t2 = (uint32_t)(u2 >> sh),
                 t3 = (uint32_t)(u3 >> sh);
#ifdef __CUDA_ARCH__
  uint32_t w = __byte_perm(__byte_perm(t0, t1, 0x0040), __byte_perm(t2, t3, 0x0040), 0x5410);
#else
  uint32_t w = (t0 & 0xFFu) | ((t1 & 0xFFu) << 8) | ((t2 & 0xFFu) << 16) | ((t3 & 0xFFu) << 24);
#endif
  if (s > 0) w &= 0x7F7F7F7Fu;  // the top digit takes all bits above it (at most 128)
  return w ^ 0x40404040u ^ ((~w & 0x40404040u) << 1);
}

// X + H for X = rint(x), |x| <= 2^(8S-2), S <= 6: 1.5 * 2^52 leaves rint(x) in the low mantissa bits of the sum.
// Only the low 8 S bits of the result mean anything.  wide_negate gives the same of -X.
GB_DIGITS_FN uint64_t wide_bias(int S) { return ((((uint64_t)1) << (8 * S)) - 1) / 255 * 128; }
GB_DIGITS_FN uint64_t wide_input(double x, int S) {
  const double t = x + 6755399441055744.0;
#ifdef __CUDA_ARCH__
  const uint64_t bits = (uint64_t)__double_as_longlong(t);
#else
  uint64_t bits;
  std::memcpy(&bits, &t, sizeof bits);
#endif
  return bits - 0x4338000000000000ull + wide_bias(S);
}
GB_DIGITS_FN uint64_t wide_negate(uint64_t u, int S) { return 2 * wide_bias(S) - u; }

// Digit s (s = 0 the top one) of four values: byte i of the word is that of U_i.
GB_DIGITS_FN uint32_t wide_digit_word(uint64_t u0, uint64_t u1, uint64_t u2, uint64_t u3, int S, int s) {
  const int p = S - 1 - s;
#ifdef __CUDA_ARCH__
  const int sel = p & 3, pick = sel | ((4 + sel) << 4);
  const uint32_t t0 = (uint32_t)(p < 4 ? u0 : u0 >> 32), t1 = (uint32_t)(p < 4 ? u1 : u1 >> 32),
                 t2 = (uint32_t)(p < 4 ? u2 : u2 >> 32), t3 = (uint32_t)(p < 4 ? u3 : u3 >> 32);
  return __byte_perm(__byte_perm(t0, t1, pick), __byte_perm(t2, t3, pick), 0x5410) ^ 0x80808080u;
#else
  const uint32_t w = (uint32_t)((u0 >> (8 * p)) & 0xFFu) | (uint32_t)((u1 >> (8 * p)) & 0xFFu) << 8 |
                     (uint32_t)((u2 >> (8 * p)) & 0xFFu) << 16 | (uint32_t)((u3 >> (8 * p)) & 0xFFu) << 24;
  return w ^ 0x80808080u;
#endif
}

// two's complement negation of each byte (no carry between bytes)
GB_DIGITS_FN uint32_t negate_bytes(uint32_t w) { return (0x80808080u - (w & 0x7F7F7F7Fu)) ^ (~w & 0x80808080u); }

}  // namespace gb200
