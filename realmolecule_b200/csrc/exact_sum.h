// exact_sum.h -- sums of doubles that do not depend on the order of their terms.
//
// An accumulator is a fixed-point number of 66 limbs of 32 bits, the first of weight 2^-1074, which
// holds any double (Kulisch, "Computer Arithmetic and Validity", 2008: the long accumulator).  A limb is kept in
// a 64-bit word, so 2^31 terms fit before a carry has to move on, and a term is at most three integer
// additions, which commute: threads may add in any order.  The sum is exact; exact_round gives the double
// next to it (round to nearest, ties to even).  The last word collects what is not finite.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define RQ_HD __host__ __device__ __forceinline__
#else
#define RQ_HD inline
#endif

namespace rq {

constexpr int kExLimbs = 66, kExFlags = kExLimbs, kExWords = kExLimbs + 1;
constexpr int kExPosInf = 1, kExNegInf = 2, kExNaN = 4;  // bits of the last word

// The additions that v stands for: p[0 .. 2] to the words w, w + 1, w + 2 (w returned).  A value that is
// not finite returns kExFlags and the bit to set in p[0].
RQ_HD int exact_split(double v, long long (&p)[3]) {
  uint64_t bits;
  std::memcpy(&bits, &v, sizeof bits);
  const bool neg = bits >> 63;
  int e = (int)(bits >> 52) & 0x7ff;
  uint64_t m = bits & 0xfffffffffffffull;
  if (e == 0x7ff) {
    p[0] = m ? kExNaN : neg ? kExNegInf : kExPosInf;
    p[1] = p[2] = 0;
    return kExFlags;
  }
  if (e) m |= 1ull << 52;
  else e = 1;
  const int w = (e - 1) >> 5, s = (e - 1) & 31;
  const uint64_t lo = (m & 0xffffffffu) << s, hi = ((m >> 32) << s) + (lo >> 32);
  p[0] = (long long)(lo & 0xffffffffu);
  p[1] = (long long)(hi & 0xffffffffu);
  p[2] = (long long)(hi >> 32);
  if (neg) {
    p[0] = -p[0];
    p[1] = -p[1];
    p[2] = -p[2];
  }
  return w;
}

// The double next to the accumulator whose limbs outside [first, last] are 0: word(i) is limb i, flags the
// last word.
template <class Word>
RQ_HD double exact_round(Word word, int first, int last, long long flags) {
  if (flags) {
    if ((flags & kExNaN) || (flags & (kExPosInf | kExNegInf)) == (kExPosInf | kExNegInf)) return NAN;
    return (flags & kExPosInf) ? INFINITY : -INFINITY;
  }
  // two more limbs take the carry of the last (a word is below 2^63: 31 bits above its limb); what is left
  // above them is the sign, or beyond every double
  const int end = last + 2 < kExLimbs - 1 ? last + 2 : kExLimbs - 1;
  auto limb = [&](int i) { return i <= last ? word(i) : 0ll; };
  long long c = 0;
  for (int i = first; i <= end; ++i) c = (limb(i) + c) >> 32;
  const bool neg = c < 0;
  if (c > 0 || c < -1) return neg ? -INFINITY : INFINITY;
  // digits of the magnitude from the lowest: the highest that is not 0, the two below it, and whether anything
  // lies below those
  uint32_t hi = 0, mid = 0, low = 0, d1 = 0, d2 = 0;
  bool sticky = false, below = false, carry = true;
  int top = -1;
  c = 0;
  for (int i = first; i <= end; ++i) {
    const long long t = limb(i) + c;
    c = t >> 32;
    uint32_t d = (uint32_t)t;
    if (neg) {  // two's complement
      const uint32_t x = ~d + (carry ? 1u : 0u);
      carry = carry && d == 0;
      d = x;
    }
    if (d) {
      top = i; hi = d; mid = d1; low = d2;
      sticky = below;
    }
    below = below || d2 != 0;
    d2 = d1;
    d1 = d;
  }
  if (top < 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int z = __clz(hi);
#else
  const int z = __builtin_clz(hi);
#endif
  const uint64_t hm = ((uint64_t)hi << 32) | mid;
  uint64_t m = z ? (hm << z) | (low >> (32 - z)) : hm;
  if (sticky || (uint32_t)(low << z) != 0) m |= 1;  // below the 53 bits that are kept
  const double x = std::ldexp((double)m, 32 * top - 32 - z - 1074);
  return neg ? -x : x;
}

}  // namespace rq
