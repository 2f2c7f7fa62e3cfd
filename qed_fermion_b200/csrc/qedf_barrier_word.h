// The word of the solver's grid barrier: arrivals counted over a whole solve in the low 56 bits,
// the error code that ends the solve in the top byte.  Blocks add 1 to the whole word per arrival,
// and the count never reaches the error: with an error in the upper half and 32 bits of count,
// 2^32 arrivals (3.6 million iterations of 592 blocks) read as one.  Waiting compares the low
// 32 bits, which may wrap: no block is a whole turn behind.
#pragma once

#ifdef __CUDACC__
#define QEDF_HD __host__ __device__
#else
#define QEDF_HD
#endif

namespace qedf {

constexpr int BAR_ERROR_SHIFT = 56;

// bits to set in the word for an error code (1 to 255)
QEDF_HD constexpr unsigned long long bar_error_bits(unsigned int code) {
  return (unsigned long long)code << BAR_ERROR_SHIFT;
}
// 0: no error
QEDF_HD constexpr unsigned int bar_error(unsigned long long word) { return (unsigned int)(word >> BAR_ERROR_SHIFT); }
// of a word without error: have `target` arrivals (modulo 2^32) happened
QEDF_HD constexpr bool bar_reached(unsigned long long word, unsigned int target) {
  return (int)((unsigned int)word - target) >= 0;
}

}  // namespace qedf
