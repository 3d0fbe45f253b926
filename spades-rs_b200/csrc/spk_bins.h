// spk_bins.h -- the word of a minimizer bin (spk_superk.cuh): its super-k-mer
// records above the sum of their windows, so that one atomic adds a record to
// both and returns its rank.  No CUDA here, so the limits are tested on machines
// without a GPU (tests/bins_test.cpp).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define SPK_HD __host__ __device__
#else
#define SPK_HD
#endif

namespace spk {

// WINB: bits of the window sum.
template <int WINB>
struct BinWord {
  static constexpr uint64_t win_mask = (1ULL << WINB) - 1;
  // A rank the record field still holds with as much room again above it.  A
  // bin that passes it hands this rank out exactly once before the field can
  // wrap (ranks then start again and records would share places), so whoever
  // sees a record of this rank gives the partition up.
  static constexpr uint32_t rank_limit = 1u << (63 - WINB);
  SPK_HD static constexpr uint64_t record(uint32_t windows) { return (1ULL << WINB) | windows; }
  SPK_HD static constexpr uint64_t records(uint64_t word) { return word >> WINB; }
  SPK_HD static constexpr uint64_t windows(uint64_t word) { return word & win_mask; }
  // The rank of the record whose atomic found `before`.
  SPK_HD static constexpr uint32_t rank(uint64_t before) { return (uint32_t)(before >> WINB); }
  SPK_HD static constexpr bool too_many(uint32_t rank) { return rank == rank_limit; }
};

}  // namespace spk
