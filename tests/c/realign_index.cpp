// The realign kernel's index arithmetic (tempi/realign.hpp) against the same
// decisions in 64 bits: every row length and packed size near the ends of the
// accepted range, every alignment, the words at both ends of the object.
// Built with -fsanitize=signed-integer-overflow, so an overflow fails too.
#include "realign.hpp"

#include <algorithm>
#include <cstdio>
#include <cstdlib>

using namespace tempi;

static void check(bool ok, const char *what, long long a, long long b, long long c) {
  if (!ok) {
    std::printf("%s at %lld %lld %lld\n", what, a, b, c);
    std::exit(1);
  }
}

int main() {
  const long long kMost = 2147483647LL;
  for (int k = 0; k < 128; ++k) {
    const long long n = k < 64 ? 16 + k : kMost - (k - 64);
    for (uint32_t a = 0; a < 16; ++a) {
      // the packed words of an object of n bytes
      const long long words = (a + n + 15) / 16;
      check(packed_words(uint32_t(n), a) == words, "packed_words", n, a, 0);
      for (long long t = 0; t < words; t += t == 3 && words > 16 ? words - 11 : 1) {
        const long long p = 16 * t - a;
        check(packed_word(uint32_t(t), a) == p, "packed_word", n, a, t);
        check(ends_within(int(p), int(n)) == (p + 16 <= n), "ends_within", n, a, t);
      }
      // the slots of a row of n bytes, and what each loads from a source of n
      const long long slots = (n + 30) / 16;
      check(row_slots(uint32_t(n)) == slots, "row_slots", n, a, 0);
      for (long long j = 0; j < slots; j += j == 3 && slots > 16 ? slots - 11 : 1) {
        const long long at = 16 * j - a;
        int column = 0;
        const bool in = slot_in_row(uint32_t(j), a, int(n), &column);
        check(in == (at < n), "slot_in_row", n, a, j);
        if (!in)
          continue;
        check(column == at, "column", n, a, j);
        check(ends_within(column, int(n)) == (at + 16 <= n), "ends_within", n, a, j);
        for (uint32_t m = 0; m < 16; ++m) {
          const long long lo = at - m;
          check(word_holds(column - int(m), int(n)) == (lo + 16 > 0 && lo < n), "word_holds",
                n, lo, m);
          check(next_word_holds(column - int(m), int(n)) == (lo + 32 > 0 && lo + 16 < n),
                "next_word_holds", n, lo, m);
        }
      }
    }
  }
  std::puts("OK");
  return 0;
}
