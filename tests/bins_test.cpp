// CPU test of the minimizer bins' word (spades-rs_b200/csrc/spk_bins.h), built
// and run by tests/test_bins.py.  A word with a small record field takes records
// until the field has wrapped several times: ranks and sums are exact up to the
// limit, and the limit is reported before the first rank is handed out again.
// Exit status 0 when every check passes.
#include <cstdint>
#include <cstdio>

#include "../spades-rs_b200/csrc/spk_bins.h"

template <int WINB>
static int fill(uint32_t windows) {
  using B = spk::BinWord<WINB>;
  const uint64_t field = 1ULL << (64 - WINB);  // ranks before the field wraps
  uint64_t word = 0, told = 0;
  for (uint64_t i = 0; i < 4 * field; i++) {
    const uint64_t before = word;
    word += B::record(windows);
    const uint32_t rank = B::rank(before);
    if (B::too_many(rank)) told++;
    if (i < field && rank != i) return std::printf("rank %u of record %llu\n", rank, (unsigned long long)i);
    if (i + 1 < field && (B::records(word) != i + 1 || B::windows(word) != (i + 1) * windows))
      return std::printf("sums after record %llu\n", (unsigned long long)i);
    // every record from half the field on comes after the report
    if (told != (i < field / 2 ? 0 : 1 + (i - field / 2) / field))
      return std::printf("record %llu: told %llu times\n", (unsigned long long)i, (unsigned long long)told);
  }
  return 0;
}

int main() {
  // (windows that fill a good part of their field without carrying out of it)
  if (fill<56>(3) || fill<60>(255) || fill<52>(113)) return 1;
  static_assert(spk::BinWord<36>::rank_limit == 1u << 27, "half of the record field");
  std::printf("bins ok\n");
  return 0;
}
