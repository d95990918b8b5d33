// How an activation is written as a sum of e5m2 terms (hq_mx_rows.cu).  Plain arithmetic, the same on the host
// (tests/test_mx_terms.py) and in the kernel.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define HQ_TERMS_FN __host__ __device__ __forceinline__
#else
#define HQ_TERMS_FN inline
#endif

namespace hq {

// Term i stands for t * 2^-shift(i) of the block's scale.  The first leaves at most 2^12 of 57,344 over, which 2^3 brings to 2^15;
// each one after that leaves at most 2^11 of 2^15, which 2^4 brings back.  e5m2's smallest step is 2^-16, so the sum of three
// terms holds multiples of 2^-23, of four 2^-27.
HQ_TERMS_FN constexpr int mx_terms_shift(int term) { return term == 0 ? 0 : 4 * term - 1; }

// Biased e8m0 exponent of the first term's scale, from the f32 bits of a block's largest magnitude: it comes to 28,672 .. 57,344
// (e5m2's largest value).  The last term's exponent may not fall below 0.
HQ_TERMS_FN int mx_terms_exponent(uint32_t max_bits, int terms) {
  if (max_bits == 0u) return 127;
  const int e = (int)((max_bits + 0x1FFFFFu) >> 23) - 15, low = mx_terms_shift(terms - 1);
  return e < low ? low : e;
}

}  // namespace hq
