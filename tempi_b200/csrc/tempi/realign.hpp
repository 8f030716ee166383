// Index arithmetic of the realign kernel (pack.cu k_realign), shared with the
// host so that it can be checked there at the sizes a GPU test rarely takes.
// Rows and packed buffers are 16 to 2^31 - 1 bytes: columns and packed offsets
// of a 16-byte word (-15 or more, its first byte may lie before the row) fit
// an int, but 16 bytes beyond one may not.  So ends are compared as n - 16,
// never as a sum, and multiples of 16 are formed without a sign.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define TEMPI_HD __host__ __device__ __forceinline__
#else
#define TEMPI_HD inline
#endif

namespace tempi {

constexpr int64_t kRealignMinRow = 16; // a packed word touches at most two rows

// 16-byte words that `bytes` packed bytes touch, the first `a0` bytes into one
TEMPI_HD uint32_t packed_words(uint32_t bytes, uint32_t a0) {
  return (a0 + bytes + 15) / 16;
}
// the offset of word t's first byte in the packed bytes
TEMPI_HD int packed_word(uint32_t t, uint32_t a0) { return int(16 * t - a0); }

// 16-byte words a row of n bytes can touch, whatever its alignment
TEMPI_HD uint32_t row_slots(uint32_t n) { return (n + 30) / 16; }
// The column of slot j's first byte in a row of n bytes that starts `lo` bytes
// into its first word; false when the slot lies past the row's end.
TEMPI_HD bool slot_in_row(uint32_t j, uint32_t lo, int n, int *column) {
  const uint32_t past = 16 * j; // from the first word's start
  *column = int(past - lo);
  return past < uint32_t(n) + lo;
}

// whether a word at `at` ends within the n bytes
TEMPI_HD bool ends_within(int at, int n) { return at <= n - 16; }

// whether the aligned word at `lo` holds one of the bytes [0, n), and the word
// after it (lo is -30 or more and less than n)
TEMPI_HD bool word_holds(int lo, int n) { return lo > -16 && lo < n; }
TEMPI_HD bool next_word_holds(int lo, int n) { return lo > -32 && lo < n - 16; }

} // namespace tempi
