// spk_superk.cuh -- the default job's partition by minimizer and the count of
// its super-k-mers (included by spk_count.cu, which holds the span helpers).
//
// A read's k-mer windows are cut into super-k-mers: runs of consecutive windows
// whose smallest hashed canonical m-mer (the minimizer; Roberts et al. 2004, Li
// et al. 2013 for the partitioning) is the same.  All occurrences of a k-mer, on
// either strand, have the same minimizer, so a bin of minimizers holds every
// occurrence of its k-mers.  What moves to the bins is one 8-byte record per
// super-k-mer (where it starts in the packed reads, how many windows it has)
// instead of one 8- to 32-byte key per occurrence, twice: at k = 55 a record
// stands for 20 windows.
//
//   k_sk_reads   one warp per read: hashed canonical m-mers, sliding minimum,
//                a record per run to a stream, with its bin and its rank there
//                (one atomic per record, which also sums the bin's windows)
//   k_sk_bins_*  exact bin offsets, and the batches: runs of neighbouring bins
//                with about T windows, so that every batch fits one CTA's table
//   k_sk_place   the stream's records to their bins
//   k_sk_count   one CTA per batch: gathers the records' bases, drops repeated
//                super-k-mers and counts the k-mers of the others in shared
//                memory; then the k-mer list and the singletons
//   k_bloom_ops  the Bloom operations of list and singletons, by Bloom range
//
// Bins have exact sizes, so no read set overflows them; a batch with more
// distinct k-mers than slots is counted in parts (by hash bits), alone, and a
// bin too large for one CTA (SkLimits) sends the job to the spans, or where its
// k-mers repeat too often for those to the general path.
#pragma once

#include "spk_bins.h"

namespace spk {

constexpr uint32_t kSkChunk = 128;    // stream entries a warp reserves at a time
constexpr int kSkReadBlock = 256;
constexpr uint32_t kSkBinBlock = 256, kSkBinIpt = 4, kSkBinChunk = kSkBinBlock * kSkBinIpt;
constexpr uint32_t kSkMaxBins = 1u << 22;
typedef BinWord<36> SkBin;            // 2^36 windows; 2^28 records, of which half are used

// Length of the minimizers: 15 above 32 bases; 13 and 11 below, where a longer
// one leaves fewer windows per super-k-mer.
__host__ __device__ constexpr unsigned sk_m(unsigned k) { return k > 32 ? 15u : k >= 27 ? 13u : 11u; }
// k this partition takes: windows of at least 11 m-mers.  k = 64 and 96, which fill
// their top limb, keep the schedules they had (spans, and the table): nothing here
// needs the spare bits, but the two have not been timed this way.
__host__ constexpr bool sk_fits(unsigned k) { return k >= 21 && (k <= 32 || 2 * k < 64 * ((k + 31) / 32)); }

struct SkStream {
  uint4* rec;                 // x, y: record; z: bin; w: rank in the bin
  uint64_t cap;
  unsigned long long* fill;   // entries reserved (a record of no windows is a gap)
  unsigned long long* bins;   // per bin: its records and windows (SkBin)
  uint32_t nbins;
  int* err;
};
// A record: start (bases from the start of `words`) << 8 | windows (1..255).

__device__ __forceinline__ uint32_t sk_hash(uint32_t c) {
  uint32_t h = (c ^ 0x2545F491u) * 0x9E3779B1u;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 13;
  return h;
}
// (minimizers are small hashes: mixed again before they pick a bin)
__device__ __forceinline__ uint32_t sk_bin(uint32_t h, uint32_t nbins) {
  uint32_t g = h * 0x85EBCA6Bu;
  g ^= g >> 16;
  g *= 0x7FEB352Du;
  g ^= g >> 15;
  return __umulhi(g, nbins);
}

template <int V>
struct SkInt {
  static constexpr int value = V;
};
// One warp per read, 32 R m-mer positions at a time, R neighbouring ones per lane.
// The sliding minimum over the w = k - m + 1 m-mers of a window doubles its reach
// with log2(w) steps.  Bound by issue (about 350 instructions a read of 150 bases):
// with a lane's positions side by side, most of the first steps stay inside the
// lane and the others are one exchange per position (32 apart, each step took an
// exchange and a select per position, 440 instructions).
// rpw: reads a warp takes at a time (at most 32).
template <int R>
__global__ void __launch_bounds__(kSkReadBlock) k_sk_reads(ReadsView rd, unsigned k, unsigned m, uint32_t rpw,
                                                            SkStream S, unsigned long long* __restrict__ occ_out) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t w = k - m + 1, seg = 32 * R - w + 1;
  const unsigned msh = 32 - 2 * m;
  unsigned p2 = 1;  // largest power of two <= w
  while (2 * p2 <= w) p2 *= 2;
  const unsigned dr = (w - p2) % R, dq = (w - p2) / R;
  uint64_t occ = 0;
  uint64_t cur = 0;   // this warp's reserved stream entries
  uint32_t rem = 0;
  __shared__ uint2 s_runs[kSkReadBlock / 32][32 * R + 1];
  uint2* runs = s_runs[threadIdx.x >> 5];
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  // Stream places of the lanes with `act` set.
  auto place = [&](bool act) -> uint64_t {
    const unsigned mask = __ballot_sync(FULL, act);
    const uint32_t n = __popc(mask), t = __popc(mask & lanemask_lt());
    uint64_t at = cur + t;
    if (n > rem) {
      unsigned long long nb = 0;
      if (lane == 0) nb = atomicAdd(S.fill, (unsigned long long)kSkChunk);
      nb = __shfl_sync(FULL, nb, 0);
      if (t >= rem) at = nb + (t - rem);
      cur = nb + (n - rem);
      rem = kSkChunk - (n - rem);
    } else {
      cur += n;
      rem -= n;
    }
    return at;
  };
  auto put = [&](uint64_t at, uint64_t base, uint32_t nw, uint32_t bin, uint32_t rank) {
    if (at < S.cap) {
      const uint64_t r = base << 8 | nw;
      S.rec[at] = make_uint4((uint32_t)r, (uint32_t)(r >> 32), bin, rank);
    } else {
      atomicOr(S.err, (int)kErrRegion);
    }
  };
  for (uint64_t b = warp * rpw; b < rd.n_reads; b += nwarps * rpw) {
    uint32_t len = 0;
    uint64_t off = 0;
    if (lane < rpw && b + lane < rd.n_reads) {
      len = __ldg(rd.lengths + b + lane);
      off = __ldg(rd.offsets + b + lane);
      if (off + ((uint64_t)len + 3) / 4 > rd.data_len) {  // src/packed_reads.rs:600-602
        atomicOr(rd.err, 4);
        len = 0;
      }
    }
    for (uint32_t j = 0; j < rpw; j++) {
      const uint32_t L = __shfl_sync(FULL, len, j);
      if (L < k) continue;
      const uint64_t base0 = 4 * (rd.byte_base + __shfl_sync(FULL, off, j));
      const uint32_t nwin = L - k + 1;
      occ += nwin;
      for (uint32_t a = 0; a < nwin; a += seg) {
        const uint32_t nw = min(seg, nwin - a), nm = nw + w - 1;
        const uint64_t base = base0 + a, bit0 = 2 * base;
        const uint64_t* p = rd.words + (bit0 >> 6);
        const uint32_t s = (uint32_t)(bit0 & 63);
        const uint32_t need = s + 2 * (nm + m - 1);  // bits from p that the segment covers
        // the lane's R positions: the 32 bases from its first
        const uint32_t lb = s + 2 * R * lane, wi = lb >> 6;
        const uint64_t u = R * lane < nm ? bswap64(__ldg(p + wi)) : 0ULL;
        const uint64_t v = 64 * (wi + 1) < need ? bswap64(__ldg(p + wi + 1)) : 0ULL;
        const uint64_t x = shl2(u, v, lb & 63);
        uint32_t M[R], T[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint32_t f = __funnelshift_l((uint32_t)x, (uint32_t)(x >> 32), 2 * r) >> msh;
          uint32_t z = __brev(~(f << msh) & (~0u << msh));  // the complement, bits reversed: low 2m bits
          z = ((z >> 1) & 0x55555555u) | ((z & 0x55555555u) << 1);
          const uint32_t h = sk_hash(min(f, z));
          M[r] = R * lane + r < nm ? h : 0xFFFFFFFFu;
        }
        // M[r]: the minimum of the e m-mers from its position.  (What comes from
        // past lane 31 reaches no window of the segment.)
        auto reach = [&](auto at, unsigned q0) {  // ... and of as many `at` + R q0 positions on
          constexpr int A = decltype(at)::value;
#pragma unroll
          for (int r = 0; r < R; r++) {
            const unsigned q = q0 + (r + A) / R;
            T[r] = M[(r + A) % R];
            if ((r + A) / R || q0) T[r] = __shfl_down_sync(FULL, T[r], q);
          }
#pragma unroll
          for (int r = 0; r < R; r++) M[r] = min(M[r], T[r]);
        };
        if (w >= 2) reach(SkInt<1 % R>{}, 1 / R);
        if (w >= 4) reach(SkInt<2 % R>{}, 2 / R);
        if (w >= 8) reach(SkInt<4 % R>{}, 4 / R);
        if (w >= 16) reach(SkInt<8 % R>{}, 8 / R);
        if (w >= 32) reach(SkInt<16 % R>{}, 16 / R);
        if (w >= 64) reach(SkInt<32 % R>{}, 32 / R);
        switch (dr) {  // the last d = w - p2 positions: d = dr + R dq
          case 0: if (dq) reach(SkInt<0>{}, dq); break;
          case 1: reach(SkInt<1>{}, dq); break;
          case 2: reach(SkInt<2>{}, dq); break;
          case 3: reach(SkInt<(R > 3 ? 3 : 0)>{}, dq); break;
          case 4: reach(SkInt<(R > 4 ? 4 : 0)>{}, dq); break;
          case 5: reach(SkInt<(R > 5 ? 5 : 0)>{}, dq); break;
          case 6: reach(SkInt<(R > 6 ? 6 : 0)>{}, dq); break;
          default: reach(SkInt<(R > 7 ? 7 : 0)>{}, dq); break;
        }
        // runs of equal minima among the segment's nw windows: their first
        // windows and minima side by side in shared memory, then a lane per run
        const uint32_t left = __shfl_up_sync(FULL, M[R - 1], 1);
        uint32_t nruns = 0, at = 0, starts = 0;
#pragma unroll
        for (int r = 0; r < R; r++) {
          const bool start = R * lane + r < nw && (M[r] != (r ? M[r ? r - 1 : 0] : left) || (r == 0 && lane == 0));
          const unsigned mk = __ballot_sync(FULL, start);
          starts |= (start ? 1u : 0u) << r;
          nruns += __popc(mk);
          at += __popc(mk & lanemask_lt());
        }
#pragma unroll
        for (int r = 0; r < R; r++)
          if (starts >> r & 1) runs[at++] = make_uint2(R * lane + r, M[r]);
        if (lane == 0) runs[nruns] = make_uint2(nw, 0);
        __syncwarp();
        for (uint32_t t0 = 0; t0 < nruns; t0 += 32) {
          const uint32_t t = t0 + lane;
          uint32_t at0 = 0, left = 0, bin = 0;
          if (t < nruns) {
            const uint2 q = runs[t];
            at0 = q.x;
            left = runs[t + 1].x - at0;
            bin = sk_bin(q.y, S.nbins);
          }
          // (a run of more than w windows, a minimizer repeated in a tandem
          // repeat, becomes several records)
          do {
            const uint32_t c = min(left, w);
            uint32_t rank = 0;
            if (c) rank = SkBin::rank(atomicAdd(S.bins + bin, (unsigned long long)SkBin::record(c)));
            const uint64_t at = place(c > 0);
            if (c) put(at, base + at0, c, bin, rank);
            at0 += c;
            left -= c;
          } while (__any_sync(FULL, left > 0));
        }
        __syncwarp();
      }
    }
  }
  for (uint32_t t = lane; t < rem; t += 32)
    if (cur + t < S.cap) S.rec[cur + t] = make_uint4(0, 0, 0, 0);
  if (lane == 0 && occ) atomicAdd(occ_out, (unsigned long long)occ);
}

// Sums of each chunk of bins: records, windows.
__global__ void __launch_bounds__(kSkBinBlock) k_sk_bins_reduce(const unsigned long long* __restrict__ bins,
                                                                 uint32_t n, unsigned long long* __restrict__ sums) {
  __shared__ unsigned long long sr, sw;
  if (threadIdx.x == 0) sr = sw = 0;
  __syncthreads();
  uint64_t r = 0, w = 0;
  for (uint32_t j = 0; j < kSkBinIpt; j++) {
    const uint32_t i = blockIdx.x * kSkBinChunk + j * kSkBinBlock + threadIdx.x;
    const uint64_t v = i < n ? bins[i] : 0;
    r += SkBin::records(v);
    w += SkBin::windows(v);
  }
  warp_add_u64(&sr, r);
  warp_add_u64(&sw, w);
  __syncthreads();
  if (threadIdx.x == 0) {
    sums[2 * blockIdx.x] = sr;
    sums[2 * blockIdx.x + 1] = sw;
  }
}

// Each bin's first record (base) and each batch's (bstart[b], b = 0..nbat): a
// batch is the bins whose windows start in [b T, (b + 1) T) of the prefix sum.
__global__ void __launch_bounds__(kSkBinBlock) k_sk_bins_apply(const unsigned long long* __restrict__ bins,
                                                                uint32_t n,
                                                                const unsigned long long* __restrict__ sums,
                                                                uint32_t T, uint32_t nbat,
                                                                uint32_t* __restrict__ base,
                                                                uint32_t* __restrict__ bstart) {
  __shared__ unsigned long long pre[2];
  __shared__ unsigned long long wr[kSkBinBlock / 32], ww[kSkBinBlock / 32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) pre[0] = pre[1] = 0;
  __syncthreads();
  {
    uint64_t r = 0, w = 0;  // the chunks before this one
    for (uint32_t c = threadIdx.x; c < blockIdx.x; c += kSkBinBlock) {
      r += sums[2 * c];
      w += sums[2 * c + 1];
    }
    warp_add_u64(&pre[0], r);
    warp_add_u64(&pre[1], w);
  }
  const uint32_t i0 = blockIdx.x * kSkBinChunk + threadIdx.x * kSkBinIpt;
  uint64_t v[kSkBinIpt], r = 0, w = 0;
#pragma unroll
  for (uint32_t j = 0; j < kSkBinIpt; j++) {
    v[j] = i0 + j < n ? bins[i0 + j] : 0;
    r += SkBin::records(v[j]);
    w += SkBin::windows(v[j]);
  }
  uint64_t xr = r, xw = w;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint64_t yr = __shfl_up_sync(FULL, xr, d), yw = __shfl_up_sync(FULL, xw, d);
    if ((int)lane >= d) {
      xr += yr;
      xw += yw;
    }
  }
  if (lane == 31) {
    wr[warp] = xr;
    ww[warp] = xw;
  }
  __syncthreads();
  uint64_t pr = pre[0] + xr - r, pw = pre[1] + xw - w;
  for (unsigned q = 0; q < warp; q++) {
    pr += wr[q];
    pw += ww[q];
  }
  uint64_t prevw = (i0 > 0 && i0 <= n) ? SkBin::windows(bins[i0 - 1]) : 0;
#pragma unroll
  for (uint32_t j = 0; j < kSkBinIpt; j++) {
    const uint32_t i = i0 + j;
    if (i >= n) break;
    base[i] = (uint32_t)pr;
    const uint32_t b1 = (uint32_t)(pw / T);
    const uint32_t b0 = i ? (uint32_t)((pw - prevw) / T) + 1 : 0;
    for (uint32_t b = b0; b <= b1 && b <= nbat; b++) bstart[b] = (uint32_t)pr;
    prevw = SkBin::windows(v[j]);
    pr += SkBin::records(v[j]);
    pw += prevw;
    if (i == n - 1)
      for (uint32_t b = b1 + 1; b <= nbat; b++) bstart[b] = (uint32_t)pr;
  }
}

// The stream's records to their bins.  A bin of more records than its word counts
// (2^27 short reads of one sequence) sends the job to the spans, as a stream that
// overflowed does.
__global__ void __launch_bounds__(256) k_sk_place(SkStream S, const uint32_t* __restrict__ base,
                                                   uint64_t* __restrict__ out) {
  const uint64_t n = min((uint64_t)*S.fill, S.cap);
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint4 q = __ldcs(S.rec + i);
    const uint64_t r = (uint64_t)q.y << 32 | q.x;
    const uint64_t at = (r & 255) ? (uint64_t)__ldg(base + q.z) + q.w : S.cap;
    if (SkBin::too_many(q.w)) atomicOr(S.err, (int)kErrRegion);
    if (at < S.cap) out[at] = r;  // (beyond it only after the stream overflowed: the job runs again)
  }
}

// ---------------------------------------------------------------------------
// The count of a batch.
// ---------------------------------------------------------------------------
template <int NL>
struct SkShape {
  // Keys of several limbs stay in the staged records: their slots hold a hash
  // tag and where the k-mer was first seen, 8 bytes instead of 16 to 32.
  static constexpr bool ref = NL >= 2;
  // Small tables leave room for five CTAs an SM, whose barriers and gathers
  // overlap (k = 33, 3 Mb x 60x: 1.24 ms against 1.37 with 4,096 slots and three
  // CTAs; k = 55, 5 Mb x 100x: 4.4 either way); the longer records of k > 64 need
  // the larger ones (k = 127: 1.8 against 3.6 ms, where 2,048 slots stage too few).
  static constexpr int threads = NL <= 2 ? 256 : 384;
  static constexpr int ctas = NL <= 2 ? 5 : 3;
  static constexpr uint32_t log2s = NL <= 2 ? 11 : 12;
  static constexpr uint32_t S = 1u << log2s;  // slots
  // Windows per batch: about a third of the slots filled at the distinct share of
  // the benchmark's reads (0.14 of the occurrences at k = 21, 0.27 at 55, 0.38 at
  // 77, 0.52 at 127); fuller tables probe longer, emptier ones end in more batches
  // (k = 55, 5 Mb x 100x: 4.26, 4.28, 4.25, 4.26, 4.43 ms at 2,000, 2,400, 2,800,
  // 3,400, 4,000 in 2,048 slots; k = 33, 3 Mb x 60x: 1.53, 1.48, 1.45, 1.46, 1.50).
  static constexpr uint32_t T = NL == 1 ? 3500 : NL == 2 ? 2800 : NL == 3 ? 4100 : 2600;
};
// 32-bit words a record's bases take: at most w windows, w + k - 1 = 2k - m bases.
__host__ __device__ __forceinline__ uint32_t sk_words(unsigned k) { return (2 * k - sk_m(k) + 15) / 16; }
constexpr uint32_t kSkMaxRecs = 2048;  // a record's index takes 11 bits
// What one CTA may spend on one batch before the job is given up and counted by
// spans, which do not depend on minimizers.  A bin is never split, and a batch
// with many times a table's distinct k-mers is counted in as many parts, each
// staging all of its records: 20,000 reads around one minimizer (k = 55, 820,000
// distinct k-mers) took 3.1 s on one CTA, by spans 2.7 ms.
// A CTA counts about 150 windows a microsecond with its SM full.  The spans take
// 1 to 3 ms of a small job and 0.06 ns an occurrence of a large one, or 0.2 to 0.4
// where the k-mers repeat too and overflow their regions; the limit lets a CTA work
// for about as long (1.3 ms and 0.1 ns an occurrence), so that neither a set it
// would have finished sooner is given up (30 kb at 5,000x, k = 55: 11.8 ms against
// 33 by spans; 5% of poly-G reads, 150,000 records in one bin: 6.0 against 40) nor
// much is spent before one is.
struct SkLimits {
  uint32_t recs;  // records of a batch (at most 2^25: a reference holds 25 bits of record)
  uint32_t cost;  // windows counted, and two for every record staged
  uint32_t hot;   // a k-mer counted more often would overflow its span's region too
};
// slack: what a span's region holds beyond its mean share of the occurrences.
static SkLimits sk_limits(uint64_t occ, uint64_t slack) {
  const uint32_t cost = (uint32_t)std::min<uint64_t>(200000 + occ / 64, 1u << 26);
  return SkLimits{cost / 2, cost, (uint32_t)std::min<uint64_t>(slack, 0xFFFFFFFFu)};
}
// Records staged at a time, and the entries (a power of two) of their table.
struct SkStage {
  uint32_t rc, dd;
  size_t smem;
};
// Shared memory: keys, counts, used slots; then the staged records (bases,
// multiplicities, the records' table or the live records, window counts).  As many
// records are staged as leave room for the CTAs an SM is to hold.
template <int NL>
static SkStage sk_stage(unsigned k) {
  typedef SkShape<NL> P;
  const size_t budget = (size_t)(228 * 1024) / P::ctas - 1024 - 2560;  // of one CTA, less its static arrays
  const size_t table = (size_t)P::S * (8 + 4 + 2);
  auto bytes = [&](uint32_t rc, uint32_t dd) { return (size_t)rc * (4 * sk_words(k) + 4 + 1) + (size_t)dd * 4; };
  SkStage g{128, 256, 0};
  for (uint32_t rc = 128; rc <= kSkMaxRecs; rc += 64) {
    uint32_t dd = 256;
    while (dd < rc + rc / 4) dd *= 2;
    if (table + bytes(rc, dd) <= budget) g = SkStage{rc, dd, 0};
  }
  g.smem = table + bytes(g.rc, g.dd);
  return g;
}

// The slot hash (not the reference's: it never leaves the batch): a multilinear
// sum over the key's 32-bit words, mixed.
template <int NL>
__device__ __forceinline__ uint32_t sk_key_hash(const Seq<NL>& C) {
  uint32_t a = 0x9E3779B9u;
  const uint32_t A[8] = {0x2C1B3C6Du, 0x297A2D39u, 0x85EBCA6Bu, 0xC2B2AE35u,
                         0x27D4EB2Fu, 0x165667B1u, 0x7FEB352Du, 0x846CA68Bu};
#pragma unroll
  for (int j = 0; j < NL; j++) a += (uint32_t)C.v[j] * A[2 * j] + (uint32_t)(C.v[j] >> 32) * A[2 * j + 1];
  a ^= a >> 16;
  a *= 0x9E3779B1u;
  return a ^ a >> 15;
}

// One probe step of a one-limb key C at slot kp: 1 = C's slot, 2 = claimed for C
// now, 0 = another key's.  Empty slots are all ones, which no key is.
__device__ __forceinline__ int sk_step(uint64_t* kp, uint64_t C) {
  const uint64_t cur = *(volatile uint64_t*)kp;
  if (cur == C) return 1;
  if (cur != kEmpty) return 0;
  const uint64_t old = atomicCAS((unsigned long long*)kp, (unsigned long long)kEmpty, (unsigned long long)C);
  return old == kEmpty ? 2 : old == C ? 1 : 0;
}

// ---- windows as W2 = 2 NL 32-bit words, word 0 most significant ----
// The bits of a key sit at the top of its words; `low` = 64 NL - 2k bits below
// them are clear (mask1 and mask2 of the last two words).
template <int NL>
struct SkCut {
  uint32_t low, rot, mask1, mask2;
};
template <int NL>
__device__ __forceinline__ SkCut<NL> sk_cut(unsigned k) {
  const uint32_t low = 64 * NL - 2 * k, rot = low & 31;
  return SkCut<NL>{low, rot, low >= 32 ? 0u : ~0u << rot, low >= 32 ? ~0u << rot : ~0u};
}
// The window that starts at base o of the staged record whose words are sq[i * RC]
// (words past the record are masked off).
template <int NL>
__device__ __forceinline__ void sk_window(const uint32_t* sq, uint32_t RC, uint32_t o, const SkCut<NL>& c,
                                          uint32_t (&L)[2 * NL]) {
  sq += (o >> 4) * RC;
  const uint32_t sh = 2 * (o & 15);
  uint32_t u = sq[0];
#pragma unroll
  for (int i = 0; i < 2 * NL; i++) {
    const uint32_t v = sq[(i + 1) * RC];
    L[i] = __funnelshift_l(v, u, sh);
    u = v;
  }
  L[2 * NL - 1] &= c.mask1;
  L[2 * NL - 2] &= c.mask2;
}
// The same from the packed reads, base `b` (a reference to a record staged in an
// earlier round).
template <int NL>
__device__ __forceinline__ void sk_window_far(const uint64_t* __restrict__ words, uint64_t b, unsigned k,
                                              const SkCut<NL>& c, uint32_t (&L)[2 * NL]) {
  const uint64_t* p = words + (b >> 5);
  const unsigned s = 2 * (unsigned)(b & 31);
  uint64_t u = bswap64(__ldg(p));
#pragma unroll
  for (int i = 0; i < NL; i++) {
    const uint64_t v = 64u * (i + 1) < s + 2 * k ? bswap64(__ldg(p + i + 1)) : 0ULL;
    const uint64_t x = shl2(u, v, s);
    L[2 * i] = (uint32_t)(x >> 32);
    L[2 * i + 1] = (uint32_t)x;
    u = v;
  }
  L[2 * NL - 1] &= c.mask1;
  L[2 * NL - 2] &= c.mask2;
}
// The reverse complement, at the bottom of G.
template <int NL>
__device__ __forceinline__ void sk_revcomp(const uint32_t (&L)[2 * NL], const SkCut<NL>& c, uint32_t (&G)[2 * NL]) {
  constexpr int W2 = 2 * NL;
#pragma unroll
  for (int i = 0; i < W2; i++) {
    uint32_t z = ~L[W2 - 1 - i];
    if (i == 0) z &= c.mask1;
    if (i == 1) z &= c.mask2;
    z = __brev(z);
    G[i] = ((z >> 1) & 0x55555555u) | ((z & 0x55555555u) << 1);
  }
}
// Words from the top to the bottom (down) and back (up).
template <int NL>
__device__ __forceinline__ void sk_down(const uint32_t (&L)[2 * NL], const SkCut<NL>& c, uint32_t (&F)[2 * NL]) {
#pragma unroll
  for (int i = 2 * NL - 1; i >= 0; i--) {
    const uint32_t l1 = i >= 1 ? L[i >= 1 ? i - 1 : 0] : 0u, l2 = i >= 2 ? L[i >= 2 ? i - 2 : 0] : 0u;
    F[i] = c.low >= 32 ? __funnelshift_r(l1, l2, c.rot) : __funnelshift_r(L[i], l1, c.rot);
  }
}
template <int NL>
__device__ __forceinline__ void sk_up(const uint32_t (&F)[2 * NL], const SkCut<NL>& c, uint32_t (&L)[2 * NL]) {
  constexpr int W2 = 2 * NL;
#pragma unroll
  for (int i = 0; i < W2; i++) {
    const uint32_t f1 = i + 1 < W2 ? F[i + 1 < W2 ? i + 1 : 0] : 0u, f2 = i + 2 < W2 ? F[i + 2 < W2 ? i + 2 : 0] : 0u;
    L[i] = c.low >= 32 ? __funnelshift_l(f2, f1, c.rot) : __funnelshift_l(f1, F[i], c.rot);
  }
}
template <int NL>
__device__ __forceinline__ Seq<NL> sk_seq(const uint32_t (&F)[2 * NL]) {
  Seq<NL> V;
#pragma unroll
  for (int i = 0; i < NL; i++) V.v[i] = (uint64_t)F[2 * NL - 2 - 2 * i] << 32 | F[2 * NL - 1 - 2 * i];
  return V;
}

template <int NL>
__global__ void __launch_bounds__(SkShape<NL>::threads, SkShape<NL>::ctas)
    k_sk_count(const uint64_t* __restrict__ words, const uint64_t* __restrict__ recs,
               const uint32_t* __restrict__ bstart, uint32_t nbat, unsigned long long* __restrict__ next_batch,
               unsigned k, uint32_t RC, uint32_t DD, SkLimits lim, ListOut lo, int* __restrict__ err) {
  typedef SkShape<NL> P;
  constexpr uint32_t S = P::S;
  constexpr int TH = P::threads, kWarps = TH / 32, kRounds = (S + TH - 1) / TH;
  constexpr int W2 = 2 * NL;  // 32-bit words of a key
  extern __shared__ __align__(16) unsigned char sk_smem_[];
  constexpr bool REF = P::ref;
  uint64_t* keys = (uint64_t*)sk_smem_;
  uint32_t* cnt = (uint32_t*)(keys + S);
  uint16_t* used = (uint16_t*)(cnt + S);
  unsigned char* uni = (unsigned char*)(used + S);
  const uint32_t SW = sk_words(k);
  uint32_t* seq = (uint32_t*)uni;        // word i (16 bases, the first on top) of record t: seq[i * RC + t]
  uint32_t* mult = seq + (size_t)SW * RC;
  uint32_t* dd = mult + RC;
  uint32_t* lrec = dd;                   // live records: first window << 11 | record (over the records' table)
  uint8_t* nws = (uint8_t*)(dd + DD);
  __shared__ uint32_t lw[2][kRounds * kWarps];
  __shared__ uint32_t wsum[kWarps];
  __shared__ unsigned long long lbase[2];
  __shared__ unsigned s_hist[kHistBins];
  __shared__ uint32_t s_batch, s_used, s_live;
  __shared__ uint32_t s_spent, s_cost, s_staged;  // of the batch's parts before, of this one; its records staged
  __shared__ int s_full, s_stop;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lmin = lo.lmin < 2 ? 2u : lo.lmin;
  const SkCut<NL> cut = sk_cut<NL>(k);
  constexpr uint64_t kFree = REF ? 0ULL : kEmpty;  // an empty slot
  uint64_t occ2 = 0;
  // No more batches for any CTA once records are missing (the stream overflowed) or
  // a batch is given up: the job runs again another way.  The flag alone would not
  // do: threads of one CTA could see it or not.
  auto stop_all = [&](uint32_t why) {
    if (why) atomicOr(err, (int)why);
    atomicMax(next_batch, (unsigned long long)nbat);
  };
  if (threadIdx.x == 0 && (*(volatile int*)err & (int)kErrRegion)) stop_all(0);
  for (int i = threadIdx.x; i < kHistBins; i += TH) s_hist[i] = 0;
  for (uint32_t i = threadIdx.x; i < S; i += TH) keys[i] = kFree;
  for (uint32_t i = threadIdx.x; i < S; i += TH) cnt[i] = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_batch = (uint32_t)min((unsigned long long)nbat, atomicAdd(next_batch, 1ULL));
    __syncthreads();
    const uint32_t bt = s_batch;
    if (bt >= nbat) break;
    const uint32_t r0 = bstart[bt], r1 = bstart[bt + 1];
    if (r0 == r1) continue;
    if (r1 - r0 > lim.recs) {
      if (threadIdx.x == 0) stop_all(kErrHot);
      continue;
    }
    if (threadIdx.x == 0) {
      s_spent = s_cost = 0;
      s_stop = 0;
    }
    // The batch, or the part of it whose hash bits [0, depth) are `part`: a part
    // with too many distinct k-mers for the table is cut in two.
    uint32_t depth = 0, part = 0;
    for (;;) {
      if (threadIdx.x == 0) {
        s_used = 0;
        s_full = 0;
        s_spent += s_cost;
        s_cost = s_staged = 0;
      }
      for (uint32_t q0 = r0; q0 < r1; q0 += RC) {
        // ---- stage up to RC records: their bases, the first on top ----
        __syncthreads();
        if (*(volatile int*)&s_full) break;
        const uint32_t n = min(RC, r1 - q0);
        if (threadIdx.x == 0) s_live = 0;
        for (uint32_t i = threadIdx.x; i < DD; i += TH) dd[i] = 0xFFFFFFFFu;
        for (uint32_t t = threadIdx.x; t < n; t += TH) {
          const uint64_t rec = __ldcs(recs + q0 + t);
          const uint32_t nw = (uint32_t)(rec & 255);
          const uint64_t bit0 = 2 * (rec >> 8);
          const unsigned s = (unsigned)(bit0 & 63);
          const uint64_t* p = words + (bit0 >> 6);
          const uint32_t bits = 2 * (nw + k - 1);
          uint64_t u = bswap64(__ldg(p));
#pragma unroll
          for (uint32_t i = 0; i < 2 * NL; i++) {
            if (64 * i >= bits) break;
            const uint64_t v = 64 * (i + 1) < s + bits ? bswap64(__ldg(p + i + 1)) : 0ULL;
            uint64_t x = shl2(u, v, s);
            u = v;
            if (bits - 64 * i < 64) x &= ~(~0ULL >> (bits - 64 * i));  // nothing past the last base
            seq[2 * i * RC + t] = (uint32_t)(x >> 32);
            if (bits - 64 * i > 32) seq[(2 * i + 1) * RC + t] = (uint32_t)x;
          }
          nws[t] = (uint8_t)nw;
          mult[t] = 1;
        }
        __syncthreads();
        // ---- equal records become one with a multiplicity ----
        uint32_t dead = 0;  // bit j: this thread's j-th record repeats another
        for (uint32_t t = threadIdx.x, j = 0; t < n; t += TH, j++) {
          const uint32_t nw = nws[t], words32 = (nw + k + 14) / 16;
          uint32_t h = nw;
          for (uint32_t i = 0; i < words32; i++) h = (h ^ seq[i * RC + t]) * 0x9E3779B1u + (h >> 15);
          h ^= h >> 16;
          h *= 0x7FEB352Du;
          const uint32_t tag = h & ~(kSkMaxRecs - 1);
          uint32_t at = (h ^ (h >> 13)) & (DD - 1);
          for (;;) {
            const uint32_t old = atomicCAS(dd + at, 0xFFFFFFFFu, tag | t);
            if (old == 0xFFFFFFFFu) break;
            if ((old & ~(kSkMaxRecs - 1)) == tag) {
              const uint32_t o = old & (kSkMaxRecs - 1);
              bool eq = nws[o] == nw;
              for (uint32_t i = 0; eq && i < words32; i++) eq = seq[i * RC + o] == seq[i * RC + t];
              if (eq) {
                atomicAdd(mult + o, 1u);
                dead |= 1u << j;
                break;
              }
            }
            at = (at + 1) & (DD - 1);
          }
        }
        __syncthreads();  // (the records' table is done with: the live records take its place)
        // ---- the live records side by side, with the windows before each ----
        for (uint32_t t0 = 0, j = 0; t0 < n; t0 += TH, j++) {
          const uint32_t t = t0 + threadIdx.x;
          const bool live = t < n && !(dead >> j & 1);
          const uint32_t lv = live ? 1u << 20 | nws[t] : 0u;  // (at most 2,048 records, 231,424 windows)
          uint32_t x = lv;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, d);
            if ((int)lane >= d) x += y;
          }
          if (lane == 31) wsum[warp] = x;
          __syncthreads();
          const uint32_t before = s_live;
          uint32_t at = before + x - lv, total = before;
#pragma unroll
          for (int q = 0; q < kWarps; q++) {
            if (q < (int)warp) at += wsum[q];
            total += wsum[q];
          }
          if (live) lrec[at >> 20] = (at & 0xFFFFF) << 11 | t;
          __syncthreads();
          if (threadIdx.x == 0) s_live = total;
        }
        __syncthreads();
        const uint32_t nlive = s_live >> 20, nwin = s_live & 0xFFFFF;
        if (threadIdx.x == 0) {
          s_cost += nwin + 2 * n;
          s_staged += n;
          // (given up, here or by another CTA: a batch of several rounds looks)
          if (s_spent + s_cost > lim.cost || (q0 != r0 && (*(volatile int*)err & (int)kErrHot))) s_full = s_stop = 1;
        }
        // ---- count: each warp a share of the windows ----
        // Lanes without a k-mer to place take the next windows, a dozen at a
        // time at least; every turn is one probe step for the lanes that have
        // one, so a long probe sequence holds up its own lane only.
        {
          const uint32_t share = (nwin + kWarps - 1) / kWarps;
          uint32_t cur = warp * share;
          const uint32_t end = min(nwin, cur + share);
          uint32_t r = 0;  // the live record that holds window cur
          for (uint32_t b = kSkMaxRecs / 2; b; b >>= 1)
            if (r + b < nlive && (lrec[r + b] >> 11) <= cur) r += b;
          bool pend = false;
          Seq<NL> C;                       // the k-mer to place; REF: its window and
          uint32_t L[W2], G[W2];           // the reverse complement, a tag and the reference
          uint64_t mine = 0;
          uint32_t slot = 0, step = 0, mu = 0;
#pragma unroll
          for (int q = 0; q < NL; q++) C.v[q] = 0;
#pragma unroll
          for (int q = 0; q < W2; q++) L[q] = G[q] = 0;
          for (;;) {
            const unsigned idle = __ballot_sync(FULL, !pend);
            const uint32_t ni = __popc(idle);
            if (cur < end && ni >= 12) {
              // records that start among the next 32 windows
              const uint32_t q = r + 1 + lane;
              const uint32_t st = q < nlive ? (lrec[q] >> 11) - cur : 32u;
              const unsigned mk = __reduce_or_sync(FULL, st < 32 ? 1u << st : 0u);
              const uint32_t rank = __popc(idle & lanemask_lt()), taken = min(ni, end - cur);
              if (!pend && rank < taken) {
                const uint32_t e = lrec[r + __popc(mk & (unsigned)((2ULL << rank) - 1))];
                const uint32_t rt = e & (kSkMaxRecs - 1), o = cur + rank - (e >> 11);
                mu = mult[rt];
                sk_window<NL>(seq + rt, RC, o, cut, L);
                uint32_t F[W2];
                sk_revcomp<NL>(L, cut, F);
                uint32_t h;
                if constexpr (REF) {
                  sk_up<NL>(F, cut, G);
                  bool fwd = true;  // canonical: the smaller of the two, src/dna.rs:185-192
#pragma unroll
                  for (int i = W2 - 1; i >= 0; i--) fwd = L[i] < G[i] || (L[i] == G[i] && fwd);
                  uint32_t D[W2];
#pragma unroll
                  for (int i = 0; i < W2; i++) D[i] = fwd ? L[i] : G[i];
                  h = sk_key_hash<NL>(sk_seq<NL>(D));
                  const uint32_t tag = (h * 0x297A2D39u ^ D[1] * 0x85EBCA6Bu ^ D[2] * 0xC2B2AE35u) | 1u;
                  mine = (uint64_t)tag << 32 | ((q0 - r0 + rt) << 7 | o);
                } else {
                  sk_down<NL>(L, cut, G);
                  const Seq<NL> V = sk_seq<NL>(G), Rc = sk_seq<NL>(F);
                  C = seq_le<NL>(V, Rc) ? V : Rc;  // canonical, src/dna.rs:185-192
                  h = sk_key_hash<NL>(C);
                }
                slot = h >> (32 - P::log2s);
                step = 0;
                pend = depth == 0 || (h & ((1u << depth) - 1)) == part;
              }
              r += __popc(mk & (unsigned)((2ULL << taken) - 1));
              cur += taken;
            }
            if (!__any_sync(FULL, pend)) {
              if (cur >= end) break;
              continue;
            }
            int got = -1;
            if (pend) {
              if constexpr (REF) {
                // An empty slot is claimed by one CAS of tag and reference (the
                // bases it refers to do not change); a slot with the same tag is
                // compared base by base with both strands of the window.
                uint64_t v = *(volatile uint64_t*)(keys + slot);
                got = 0;
                if (v == kFree) {
                  v = atomicCAS((unsigned long long*)(keys + slot), (unsigned long long)kFree, (unsigned long long)mine);
                  if (v == kFree) got = 2;
                }
                if (got == 0 && (uint32_t)(v >> 32) == (uint32_t)(mine >> 32)) {
                  const uint32_t ir = ((uint32_t)v >> 7) - (q0 - r0), io = (uint32_t)v & 127;
                  uint32_t D[W2];
                  if (ir < n) sk_window<NL>(seq + ir, RC, io, cut, D);
                  else sk_window_far<NL>(words, (__ldg(recs + r0 + ((uint32_t)v >> 7)) >> 8) + io, k, cut, D);
                  bool eq = true, er = true;
#pragma unroll
                  for (int i = 0; i < W2; i++) {
                    eq &= D[i] == L[i];
                    er &= D[i] == G[i];
                  }
                  got = eq || er;
                }
              } else {
                got = sk_step(keys + slot, C.v[0]);
              }
            }
            const unsigned won = __ballot_sync(FULL, got == 2);
            if (won) {
              uint32_t u0 = 0;
              if (lane == 0) u0 = atomicAdd(&s_used, (uint32_t)__popc(won));
              u0 = __shfl_sync(FULL, u0, 0) + __popc(won & lanemask_lt());
              if (got == 2 && u0 < S) used[u0] = (uint16_t)slot;
              if (u0 >= S - S / 16) s_full = 1;
            }
            if (got == 1 || got == 2) {
              atomicAdd(cnt + slot, mu);
              pend = false;
            } else if (got == 0) {
              slot = (slot + ++step) & (S - 1);  // (triangular steps reach every slot)
              if (step >= S) s_full = 1;
              // (a full table's counts are dropped: no long probes for them)
              if ((step & 31) == 0 && *(volatile int*)&s_full) pend = false;
            }
          }
        }
      }
      __syncthreads();
      const uint32_t n = min(s_used, S);
      // (REF) the records still staged: those of the last round
      const uint32_t qlast = (r1 - r0 - 1) / RC * RC, nlast = r1 - r0 - qlast;
      if (s_full) {
        // too many distinct k-mers: this part again as two, unless the limit is
        // reached or far away from what is ahead.  The table filled after a share
        // of the records; if new k-mers kept coming, as many parts as that share
        // goes into the whole would follow (on the way to the first part: for
        // each of the parts ahead), each with all of the records.  They come ever
        // more slowly where reads repeat, so eight times the limit is allowed.
        uint32_t top = 0;
        for (uint32_t i = threadIdx.x; i < S; i += TH) keys[i] = kFree;
        for (uint32_t i = threadIdx.x; i < S; i += TH) {
          top = max(top, cnt[i]);
          cnt[i] = 0;
        }
        if (threadIdx.x == 0) {
          const float f = (float)(r1 - r0) / (float)s_staged;
          const float ahead = (float)s_cost * f * f * (part == 0 ? (float)(1u << depth) : 1.f);
          if (depth == 16 || ahead > 8.f * lim.cost) s_stop = 1;
          if (s_stop) stop_all(kErrHot);
        }
        depth++;
        __syncthreads();
        if (s_stop) {
          if (top > lim.hot) atomicOr(err, (int)kErrRepeat);
          break;
        }
        continue;
      }
      // ---- write the part out ----
      // Entries of each (round, warp) of the loop below: a ballot per round,
      // then one reservation for the list and one for the singletons.
      const uint32_t rounds = (n + TH - 1) / TH;
      for (uint32_t r = 0; r < rounds; r++) {
        const uint32_t i = r * TH + threadIdx.x;
        const uint32_t c = i < n ? cnt[used[i]] : 0u;
        const unsigned bl = __ballot_sync(FULL, c >= lmin), bs = __ballot_sync(FULL, c == 1);
        if (lane == 0) {
          lw[0][r * kWarps + warp] = __popc(bl);
          lw[1][r * kWarps + warp] = __popc(bs);
        }
        if (c >= 2) {
          atomicAdd(&s_hist[c < kHistBins - 1 ? c : kHistBins - 1], 1u);
          occ2 += c;
        }
      }
      __syncthreads();
      if (warp < 2) {
        const uint32_t m = rounds * kWarps;
        uint32_t carry = 0;
        for (uint32_t b = 0; b < m; b += 32) {
          const uint32_t v = b + lane < m ? lw[warp][b + lane] : 0u;
          uint32_t x = v;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, d);
            if ((int)lane >= d) x += y;
          }
          if (b + lane < m) lw[warp][b + lane] = carry + x - v;
          carry += __shfl_sync(FULL, x, 31);
        }
        if (lane == 0) lbase[warp] = carry ? atomicAdd(lo.fill + warp, (unsigned long long)carry) : 0ULL;
      }
      __syncthreads();
      for (uint32_t r = 0; r < rounds; r++) {
        const uint32_t i = r * TH + threadIdx.x;
        const uint32_t s = i < n ? used[i] : 0u;
        const uint32_t c = i < n ? cnt[s] : 0u;
        Seq<NL> C;
        if constexpr (REF) {
          // the key from where it was first seen (in the last staged records, or
          // in the reads)
          const uint32_t ref = c ? (uint32_t)keys[s] : qlast << 7, ir = (ref >> 7) - qlast, io = ref & 127;
          uint32_t L[W2], G[W2], F[W2];
          if (ir < nlast) sk_window<NL>(seq + ir, RC, io, cut, L);
          else sk_window_far<NL>(words, (__ldg(recs + r0 + (ref >> 7)) >> 8) + io, k, cut, L);
          sk_revcomp<NL>(L, cut, G);
          sk_down<NL>(L, cut, F);
          const Seq<NL> V = sk_seq<NL>(F), Rc = sk_seq<NL>(G);
          C = seq_le<NL>(V, Rc) ? V : Rc;
        } else {
          C.v[0] = keys[s];
        }
        const unsigned bl = __ballot_sync(FULL, c >= lmin), bs = __ballot_sync(FULL, c == 1);
        if (c >= lmin) {
          const uint64_t q = lbase[0] + lw[0][r * kWarps + warp] + __popc(bl & lanemask_lt());
          if (q < lo.cap) {
#pragma unroll
            for (int j = 0; j < NL; j++) lo.l[j][q] = C.v[j];
            lo.cnt[q] = c;
          }
        } else if (c == 1) {
          const uint64_t q = lbase[1] + lw[1][r * kWarps + warp] + __popc(bs & lanemask_lt());
          if (q < lo.scap) {
#pragma unroll
            for (int j = 0; j < NL; j++) lo.s[j][q] = C.v[j];
          }
        }
      }
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < n; i += TH) {
        const uint32_t s = used[i];
        keys[s] = kFree;
        cnt[s] = 0;
      }
      // the next part, of the same depth (a shallower one would overflow as the
      // parts around it did): the first bit counts most
      uint32_t b = depth;
      while (b > 0 && (part >> (b - 1) & 1)) part &= ~(1u << --b);
      if (b == 0) break;
      part |= 1u << (b - 1);
      __syncthreads();
    }
  }
  warp_add_u64(lo.occ2, occ2);
  __syncthreads();
  for (int i = threadIdx.x; i < kHistBins; i += TH)
    if (s_hist[i]) atomicAdd(lo.hist + i, (unsigned long long)s_hist[i]);
}

// ---------------------------------------------------------------------------
// The Bloom operations of the counted k-mers (three per distinct k-mer: its bit
// in the range, and whether it was counted twice or more), binned by range for
// k_bloom_apply.  Tiles of 4,096 k-mers, first of the list, then of the
// singletons: positions and ranks in their range's share of the tile in
// registers, one reservation per tile and range, then the tile in range order
// out of shared memory, in runs of a dozen operations.
//
// Bound by the ranking's shared-memory atomics and by issue (three hashes per
// k-mer).  As the write-out of each counted batch these operations came in runs
// of five, behind a dozen barriers per 1,800 k-mers.
// ---------------------------------------------------------------------------
constexpr int kOpsBlock = 512;
constexpr uint32_t kOpsPer = 8;                       // k-mers per thread and tile
constexpr uint32_t kOpsTile = kOpsBlock * kOpsPer;
static size_t ops_smem(uint32_t nranges) { return (size_t)3 * kOpsTile * 4 + (size_t)nranges * (8 + 4 + 4); }

template <int NL>
__global__ void __launch_bounds__(kOpsBlock, 3) k_bloom_ops(ListOut lo, unsigned k, FastMod fm, RangeView rv) {
  extern __shared__ __align__(16) unsigned char ops_smem_[];
  const uint32_t nr = rv.nranges;
  unsigned long long* gb = (unsigned long long*)ops_smem_;  // where a range's share goes, less its start
  uint32_t* sorted = (uint32_t*)(gb + nr);
  uint32_t* hist = sorted + 3 * kOpsTile;
  uint32_t* start = hist + nr;
  __shared__ uint32_t wsum[kOpsBlock / 32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t nl = min((uint64_t)lo.fill[0], lo.cap), ns = min((uint64_t)lo.fill[1], lo.scap);
  const uint64_t tl = (nl + kOpsTile - 1) / kOpsTile, ts = (ns + kOpsTile - 1) / kOpsTile;
  const uint32_t per = (nr + kOpsBlock - 1) / kOpsBlock;
  const uint32_t b0 = min(nr, threadIdx.x * per), b1 = min(nr, b0 + per);
  for (uint64_t tile = blockIdx.x; tile < tl + ts; tile += gridDim.x) {
    const bool list = tile < tl;
    const uint64_t i0 = (list ? tile : tile - tl) * kOpsTile, n = list ? nl : ns;
    for (uint32_t r = threadIdx.x; r < nr; r += kOpsBlock) hist[r] = 0;
    __syncthreads();
    uint32_t op[kOpsPer][3];
    uint16_t rk[kOpsPer][3];
#pragma unroll
    for (uint32_t u = 0; u < kOpsPer; u++) {
      const uint64_t i = i0 + u * kOpsBlock + threadIdx.x;
      if (i < n) {
        Seq<NL> C;
#pragma unroll
        for (int j = 0; j < NL; j++) C.v[j] = list ? lo.l[j][i] : lo.s[j][i];
        uint64_t raw[3], pos[3];
        bloom_positions<NL>(C, k, fm, raw, pos);
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const uint32_t r = (uint32_t)(pos[j] >> kLog2Range);
          op[u][j] = r << 20 | ((uint32_t)pos[j] & ((1u << kLog2Range) - 1)) << 1 | (list ? 1u : 0u);
          rk[u][j] = (uint16_t)atomicAdd(hist + r, 1u);
        }
      }
    }
    __syncthreads();
    uint32_t sum = 0;
    for (uint32_t r = b0; r < b1; r++) sum += hist[r];
    uint32_t x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, x, d);
      if ((int)lane >= d) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t before = x - sum, total = 0;
#pragma unroll
    for (unsigned w = 0; w < kOpsBlock / 32; w++) {
      if (w < warp) before += wsum[w];
      total += wsum[w];
    }
    for (uint32_t r = b0; r < b1; r++) {
      const uint32_t c = hist[r];
      start[r] = before;
      gb[r] = (c ? range_base(rv, r) + atomicAdd(rv.fill + (uint64_t)r * kFillStride, c) : 0ULL) - before;
      before += c;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kOpsPer; u++)
      if (i0 + u * kOpsBlock + threadIdx.x < n)
#pragma unroll
        for (int j = 0; j < 3; j++) sorted[start[op[u][j] >> 20] + rk[u][j]] = op[u][j];
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < total; q += kOpsBlock) {
      const uint32_t v = sorted[q], r = v >> 20;
      const uint64_t at = gb[r] + q;
      const uint64_t end = rv.uniform ? (uint64_t)(r + 1) * rv.uniform : rv.base[r + 1];
      if (at < end) rv.ops[at] = v & 0xFFFFFu;
      else atomicOr(rv.err, (int)kErrRange);
    }
    __syncthreads();
  }
}

}  // namespace spk
