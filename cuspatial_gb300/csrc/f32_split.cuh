// A float64 as the sum of two float32 parts, formed on the integer pipe: on
// GB300 a float64 subtraction and a conversion issue at about 1.9 lanes per
// SM per cycle each, integer and float32 instructions at 64 to 128.
// Plain C++ as well, so that the host tests can check it.
//
// For |v| in [2^-100, 2^100): v = hi + lo + e with hi the top 24 significant
// bits of v (cut toward zero), lo the next 23 (exact in float32) and
// 0 <= |e| < 2^-46 |v|, all of v's sign.
#pragma once

#include "f32_diff.cuh"

namespace cspt {

struct F32Pair {
  float hi, lo;
};

// Whether split_f32 covers v: exponent field in [923, 1123).  Zeros, tiny,
// huge and non-finite values are not covered.
CSPT_HD inline bool splits_f32(double v)
{
  uint32_t const h = static_cast<uint32_t>(bits_of(v) >> 32) & 0x7FFFFFFFu;
  return h - (923u << 20) < (200u << 20);
}

CSPT_HD inline F32Pair split_f32(double v)
{
  uint64_t const b    = bits_of(v);
  uint32_t const h    = static_cast<uint32_t>(b >> 32), l = static_cast<uint32_t>(b);
  uint32_t const sign = h & 0x80000000u;
  // exponent field e -> e - 896 (double to float bias), top 23 mantissa bits
  uint32_t const t = (((h << 3) | (l >> 29)) + 0x40000000u) & 0x7FFFFFFFu;
  F32Pair r;
  r.hi = float_of_bits(t | sign);
  // the next 23 bits as 1.l 2^(E-23) - 1.0 2^(E-23): the subtraction is exact
  uint32_t const eb = ((t & 0x7F800000u) - (23u << 23)) | sign;
  r.lo              = float_of_bits(eb | ((l >> 6) & 0x7FFFFFu)) - float_of_bits(eb);
  return r;
}

}  // namespace cspt
