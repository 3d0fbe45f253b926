// spk_sort.cu -- LSD radix sort of multi-limb keys (SoA) and an ordered
// stream compaction, both written for this library.
//
// Sort: 8-bit digits, one pass per digit of the significant bits.  Each pass
// is a tile histogram, one exclusive scan over (digit, tile) and a stable
// scatter.  Inside a tile, items are ranked per warp with __match_any_sync on
// the digit, then offset by the per-warp prefix of each digit, so equal
// digits keep their input order (stability across passes).
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "spk_internal.h"

namespace spk {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int RS_BLOCK = 256;
constexpr int RS_WARPS = RS_BLOCK / 32;
constexpr int RS_IPT = 8;
constexpr int RS_TILE = RS_BLOCK * RS_IPT;  // 2048 items

__global__ void __launch_bounds__(RS_BLOCK) k_rs_hist(const uint64_t* __restrict__ limb, uint64_t n,
                                                       unsigned sh, uint32_t* __restrict__ hist,
                                                       uint32_t ntiles) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * RS_TILE;
#pragma unroll
  for (int j = 0; j < RS_IPT; j++) {
    const uint64_t i = base + j * RS_BLOCK + threadIdx.x;
    if (i < n) atomicAdd(&h[(unsigned)(__ldg(limb + i) >> sh) & 255u], 1u);
  }
  __syncthreads();
  hist[(uint64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of n u32 values in place, one block of 1024 threads.  Used
// for short arrays (the per-chunk sums of scan_u32).
__global__ void __launch_bounds__(1024) k_scan_u32(uint32_t* __restrict__ a, uint64_t n) {
  __shared__ uint32_t ws[32];
  __shared__ uint32_t carry_s;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (uint64_t base = 0; base < n; base += 1024) {
    const uint64_t i = base + threadIdx.x;
    const uint32_t v = i < n ? a[i] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t t = __shfl_up_sync(FULLM, x, d);
      if ((int)lane >= d) x += t;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t y = ws[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t t = __shfl_up_sync(FULLM, y, d);
        if ((int)lane >= d) y += t;
      }
      ws[lane] = y;
    }
    __syncthreads();
    const uint32_t carry = carry_s;
    const uint32_t excl = carry + (warp ? ws[warp - 1] : 0u) + x - v;
    if (i < n) a[i] = excl;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = carry + ws[31];
    __syncthreads();
  }
}

// Multi-block exclusive scan: chunk sums, a scan of the sums, then a
// block-wide scan of every chunk with its offset.
constexpr int SC_BLOCK = 256, SC_IPT = 16, SC_CHUNK = SC_BLOCK * SC_IPT;

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t t = __shfl_up_sync(FULLM, x, d);
    if ((int)lane >= d) x += t;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  uint32_t pre = 0, tot = 0;
  for (unsigned w = 0; w < blockDim.x / 32; w++) {
    const uint32_t s = ws[w];
    if (w < warp) pre += s;
    tot += s;
  }
  __syncthreads();
  if (total) *total = tot;
  return pre + x - v;
}

__global__ void __launch_bounds__(SC_BLOCK) k_scan_reduce(const uint32_t* __restrict__ a, uint64_t n,
                                                           uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[SC_BLOCK / 32];
  const uint64_t base = (uint64_t)blockIdx.x * SC_CHUNK;
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < SC_IPT; j++) {
    const uint64_t i = base + j * SC_BLOCK + threadIdx.x;
    if (i < n) s += a[i];
  }
  uint32_t tot;
  block_excl_scan(s, ws, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SC_BLOCK) k_scan_apply(uint32_t* __restrict__ a, uint64_t n,
                                                          const uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[SC_BLOCK / 32];
  // Thread t owns the contiguous items [t*IPT, t*IPT + IPT) of the chunk.
  const uint64_t base = (uint64_t)blockIdx.x * SC_CHUNK + (uint64_t)threadIdx.x * SC_IPT;
  uint32_t v[SC_IPT];
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < SC_IPT; j++) {
    v[j] = base + j < n ? a[base + j] : 0u;
    s += v[j];
  }
  uint32_t run = sums[blockIdx.x] + block_excl_scan(s, ws, nullptr);
#pragma unroll
  for (int j = 0; j < SC_IPT; j++) {
    if (base + j < n) a[base + j] = run;
    run += v[j];
  }
}

// Short arrays by one block of 1024 threads, up to 16 items each: one launch of
// about 4 us where the three above take 9 with their gaps.
constexpr uint64_t SC_SMALL = 16384;
__global__ void __launch_bounds__(1024) k_scan_small(uint32_t* __restrict__ a, uint32_t n) {
  __shared__ uint32_t ws[32];
  const uint32_t ipt = (n + 1023) / 1024, base = threadIdx.x * ipt;
  uint32_t v[SC_SMALL / 1024], s = 0;
#pragma unroll
  for (uint32_t j = 0; j < SC_SMALL / 1024; j++) {
    v[j] = j < ipt && base + j < n ? a[base + j] : 0u;
    s += v[j];
  }
  uint32_t run = block_excl_scan(s, ws, nullptr);
#pragma unroll
  for (uint32_t j = 0; j < SC_SMALL / 1024; j++) {
    if (j < ipt && base + j < n) a[base + j] = run;
    run += v[j];
  }
}

int scan_u32(cudaStream_t st, uint32_t* a, uint64_t n, DevBuf& sums, uint32_t* launches) {
  if (n <= SC_SMALL) {
    k_scan_small<<<1, 1024, 0, st>>>(a, (uint32_t)n);
    SPK_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
    return SPK_OK;
  }
  const uint64_t nb = (n + SC_CHUNK - 1) / SC_CHUNK;
  int rc;
  if (sums.bytes < nb * 4 && (rc = sums.alloc(nb * 4, st))) return rc;
  k_scan_reduce<<<(unsigned)nb, SC_BLOCK, 0, st>>>(a, n, sums.as<uint32_t>());
  k_scan_u32<<<1, 1024, 0, st>>>(sums.as<uint32_t>(), nb);
  k_scan_apply<<<(unsigned)nb, SC_BLOCK, 0, st>>>(a, n, sums.as<uint32_t>());
  SPK_CUDA(cudaGetLastError());
  if (launches) *launches += 3;
  return SPK_OK;
}

template <int NL, bool HASV>
__global__ void __launch_bounds__(RS_BLOCK) k_rs_scatter(
    const uint64_t* __restrict__ s0, const uint64_t* __restrict__ s1, const uint64_t* __restrict__ s2,
    const uint64_t* __restrict__ s3, const uint32_t* __restrict__ sv, uint64_t* __restrict__ d0,
    uint64_t* __restrict__ d1, uint64_t* __restrict__ d2, uint64_t* __restrict__ d3,
    uint32_t* __restrict__ dv, uint64_t n, unsigned dlimb, unsigned sh,
    const uint32_t* __restrict__ offs, uint32_t ntiles) {
  __shared__ uint32_t wh[RS_WARPS][256];
  __shared__ uint32_t goff[256];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  const uint64_t base = (uint64_t)blockIdx.x * RS_TILE + warp * (32 * RS_IPT);

  uint64_t key[RS_IPT][NL];
  uint32_t val[RS_IPT], dig[RS_IPT], rank[RS_IPT];
#pragma unroll
  for (int r = 0; r < RS_IPT; r++) {
    const uint64_t i = base + r * 32 + lane;
    const bool ok = i < n;
#pragma unroll
    for (int j = 0; j < NL; j++) {
      const uint64_t* s = j == 0 ? s0 : j == 1 ? s1 : j == 2 ? s2 : s3;
      key[r][j] = ok ? __ldg(s + i) : 0;
    }
    val[r] = (HASV && ok) ? __ldg(sv + i) : 0u;
    uint64_t dl = 0;
#pragma unroll
    for (int j = 0; j < NL; j++)
      if ((unsigned)j == dlimb) dl = key[r][j];
    dig[r] = ok ? (unsigned)(dl >> sh) & 255u : 0xFFFFFFFFu;
  }
  for (int j = threadIdx.x; j < RS_WARPS * 256; j += RS_BLOCK) (&wh[0][0])[j] = 0;
  goff[threadIdx.x] = offs[(uint64_t)threadIdx.x * ntiles + blockIdx.x];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_IPT; r++) {
    const bool ok = dig[r] != 0xFFFFFFFFu;
    const unsigned vm = __ballot_sync(FULLM, ok);
    unsigned peers = 0;
    if (ok) {
      peers = __match_any_sync(vm, dig[r]);
      rank[r] = wh[warp][dig[r]] + __popc(peers & lt);
    }
    __syncwarp();
    if (ok && lane == (unsigned)(__ffs(peers) - 1)) wh[warp][dig[r]] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) {
      const uint32_t x = wh[w][threadIdx.x];
      wh[w][threadIdx.x] = run;
      run += x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_IPT; r++) {
    if (dig[r] == 0xFFFFFFFFu) continue;
    const uint64_t p = (uint64_t)goff[dig[r]] + wh[warp][dig[r]] + rank[r];
    d0[p] = key[r][0];
    if (NL > 1) d1[p] = key[r][NL > 1 ? 1 : 0];
    if (NL > 2) d2[p] = key[r][NL > 2 ? 2 : 0];
    if (NL > 3) d3[p] = key[r][NL > 3 ? 3 : 0];
    if (HASV) dv[p] = val[r];
  }
}

template <int NL>
static void launch_scatter(cudaStream_t st, uint64_t* src[4], uint32_t* sv, uint64_t* dst[4],
                           uint32_t* dv, uint64_t n, unsigned dlimb, unsigned sh,
                           const uint32_t* offs, uint32_t ntiles) {
  if (sv)
    k_rs_scatter<NL, true><<<ntiles, RS_BLOCK, 0, st>>>(src[0], src[1], src[2], src[3], sv, dst[0],
                                                      dst[1], dst[2], dst[3], dv, n, dlimb, sh,
                                                      offs, ntiles);
  else
    k_rs_scatter<NL, false><<<ntiles, RS_BLOCK, 0, st>>>(src[0], src[1], src[2], src[3], nullptr,
                                                       dst[0], dst[1], dst[2], dst[3], nullptr, n,
                                                       dlimb, sh, offs, ntiles);
}

int radix_sort_bufs(cudaStream_t st, int nl, uint64_t n, unsigned nbits, DevBuf* keys,
                    DevBuf* vals, uint32_t* launches) {
  if (n <= 1) return SPK_OK;
  if (n >= (1ULL << 32)) return fail(SPK_E_INVALID_ARG, "sort: more than 2^32 items");
  const uint32_t ntiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
  int rc;
  DevBuf tk[4], tv, hist, sums;
  for (int j = 0; j < nl; j++)
    if ((rc = tk[j].alloc(n * 8, st))) return rc;
  if (vals && (rc = tv.alloc(n * 4, st))) return rc;
  if ((rc = hist.alloc((uint64_t)256 * ntiles * 4, st))) return rc;
  uint64_t* a[4] = {nullptr, nullptr, nullptr, nullptr};
  uint64_t* b[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int j = 0; j < nl; j++) { a[j] = keys[j].as<uint64_t>(); b[j] = tk[j].as<uint64_t>(); }
  uint32_t* av = vals ? vals->as<uint32_t>() : nullptr;
  uint32_t* bv = vals ? tv.as<uint32_t>() : nullptr;
  const unsigned passes = (nbits + 7) / 8;
  for (unsigned p = 0; p < passes; p++) {
    const unsigned bit = 8 * p, dlimb = bit / 64, sh = bit % 64;
    k_rs_hist<<<ntiles, RS_BLOCK, 0, st>>>(a[dlimb], n, sh, hist.as<uint32_t>(), ntiles);
    if ((rc = scan_u32(st, hist.as<uint32_t>(), (uint64_t)256 * ntiles, sums, launches))) return rc;
    if (launches) *launches += 2;
    switch (nl) {
      case 1: launch_scatter<1>(st, a, av, b, bv, n, dlimb, sh, hist.as<uint32_t>(), ntiles); break;
      case 2: launch_scatter<2>(st, a, av, b, bv, n, dlimb, sh, hist.as<uint32_t>(), ntiles); break;
      case 3: launch_scatter<3>(st, a, av, b, bv, n, dlimb, sh, hist.as<uint32_t>(), ntiles); break;
      default: launch_scatter<4>(st, a, av, b, bv, n, dlimb, sh, hist.as<uint32_t>(), ntiles); break;
    }
    SPK_CUDA(cudaGetLastError());
    for (int j = 0; j < nl; j++) std::swap(a[j], b[j]);
    std::swap(av, bv);
  }
  if (passes & 1) {  // sorted data sits in the temporaries: hand them over
    for (int j = 0; j < nl; j++) std::swap(keys[j], tk[j]);
    if (vals) std::swap(*vals, tv);
  }
  return SPK_OK;
}

// ---------------------------------------------------------------------------
// Bucket sort: an MSD split into buckets of about 16 items, then each bucket
// sorted on its own.  The top 12 bits of the keys split the list into coarse
// bins; a bin of c items is cut into ceil(c / 16) buckets (fewer and larger
// ones beyond 2^20 buckets) by the 32 bits that follow, so bucket sizes stay
// even where GC content makes some prefixes ten times as common as others.
// Runs of neighbouring buckets of at most 32 items together are sorted by one
// warp in registers, one item per lane; buckets of up to BS_WARP items by one
// warp with up to four items per lane; larger ones by the CTA in shared
// memory; and a bucket of more than BS_LOCAL items (keys that share a long
// prefix) goes to the LSD radix sort above.  Equal keys do not occur (the lists
// hold distinct k-mers), so stability is not needed.
//
// The split costs one read and one scattered write of the list whatever the
// number of buckets (their write frontiers stay in L2), while a bucket's sort
// grows with the square of its log.  With 2^16 buckets of 120 items and
// bitonic stages in shared memory the local sort took 0.49 ms for the 5 M
// edges of 5 Mb x 100x (k = 55), in registers 0.24; equal cuts by the top 18
// bits took 1.34 ms for the 3.4 M k-mers of a genome of 35% GC, where the
// A/T-rich buckets went to the shared-memory sort.  Lists below 2^18 items
// took the LSD sort, 5 launches for each of its 8 to 32 passes (85 launches
// for a 10 kb sample at k = 31: 1.01 -> 0.78 ms for the job).
// ---------------------------------------------------------------------------
constexpr uint32_t BS_COARSE_BITS = 12, BS_COARSE = 1u << BS_COARSE_BITS;
constexpr uint32_t BS_PER = 16;                 // items per bucket aimed at
constexpr uint32_t BS_MAX_BUCKETS = 1u << 20;   // ... up to this many buckets (plus one per coarse bin)
constexpr uint32_t BS_LOCAL = 2048;
constexpr int BS_BLOCK = 256;
constexpr uint32_t BS_CHUNK = BS_BLOCK;  // buckets a CTA takes at a time (32 per warp)
constexpr uint32_t BS_MAX_BIG = 4096;
constexpr uint64_t BS_STAGE_WORDS = 1024;  // big-bucket list offset in the host staging block

struct Limbs {
  uint64_t* p[4];
};

// Device words of one sort, zeroed before it: coarse counts, the plan (the
// first bucket of every coarse bin, then their total), a ticket, the number
// of big buckets and their list, and the buckets' offsets.
struct BsWork {
  uint32_t *coarse, *plan, *ticket, *nbig, *big, *off;
};
static BsWork bs_work(uint32_t* w) {
  BsWork b{};
  b.coarse = w;
  b.plan = b.coarse + BS_COARSE;
  b.ticket = b.plan + BS_COARSE + 1;
  b.nbig = b.ticket + 1;
  b.big = b.nbig + 1;
  b.off = b.big + 3 * BS_MAX_BIG + 1;
  return b;
}
// Most buckets a list of n items is cut into.
static uint32_t bs_max_buckets(uint64_t n) {
  return (uint32_t)std::min<uint64_t>((n + BS_PER - 1) / BS_PER, BS_MAX_BUCKETS) + BS_COARSE;
}
static size_t bs_work_bytes(uint64_t n) { return (3 + 2 * BS_COARSE + 3 * BS_MAX_BIG + 1 + (size_t)bs_max_buckets(n)) * 4; }

// The top 44 of a key's nbits bits (shorter keys: followed by zeros).
template <int NL>
__device__ __forceinline__ uint64_t bs_top(const Limbs& L, uint64_t i, unsigned nbits) {
  if (nbits < 44) return L.p[0][i] << (44 - nbits);
  const unsigned limb = (nbits - 44) / 64, sh = (nbits - 44) % 64;
  uint64_t lo = 0, hi = 0;
#pragma unroll
  for (int j = 0; j < NL; j++) {
    if ((unsigned)j == limb) lo = L.p[j][i];
    if ((unsigned)j == limb + 1 && sh > 20) hi = L.p[j][i];
  }
  return ((lo >> sh) | ((hi << 1) << (63 - sh))) & ((1ULL << 44) - 1);
}
// The bucket of a key: its coarse bin's share cut evenly by the next 32 bits
// (a non-decreasing function of the key).
__device__ __forceinline__ uint32_t bs_bucket(uint64_t top, const uint32_t* __restrict__ plan) {
  const uint32_t c = (uint32_t)(top >> 32);
  const uint32_t p0 = __ldg(plan + c), p1 = __ldg(plan + c + 1);
  return p0 + __umulhi((uint32_t)top, p1 - p0);
}

// Coarse counts; the last CTA turns them into the plan.
// n_dev (nullable): the item count in device memory, at most n.
template <int NL>
__global__ void __launch_bounds__(BS_BLOCK) k_bs_coarse(Limbs L, uint64_t n, const unsigned long long* n_dev,
                                                         unsigned nbits, BsWork W) {
  __shared__ uint32_t h[BS_COARSE];
  __shared__ uint32_t ws[BS_BLOCK / 32];
  __shared__ bool last;
  if (n_dev) n = min(n, (uint64_t)*n_dev);
  for (uint32_t c = threadIdx.x; c < BS_COARSE; c += BS_BLOCK) h[c] = 0;
  __syncthreads();
  for (uint64_t i = blockIdx.x * (uint64_t)BS_BLOCK + threadIdx.x; i < n; i += (uint64_t)gridDim.x * BS_BLOCK)
    atomicAdd(&h[bs_top<NL>(L, i, nbits) >> 32], 1u);
  __syncthreads();
  for (uint32_t c = threadIdx.x; c < BS_COARSE; c += BS_BLOCK)
    if (h[c]) atomicAdd(W.coarse + c, h[c]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(W.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const uint32_t per = (uint32_t)max((uint64_t)BS_PER, (n + BS_MAX_BUCKETS - 1) / BS_MAX_BUCKETS);
  constexpr uint32_t IPT = BS_COARSE / BS_BLOCK;
  uint32_t v[IPT], s = 0;
#pragma unroll
  for (uint32_t j = 0; j < IPT; j++) {
    const uint32_t c = __ldcg(W.coarse + threadIdx.x * IPT + j);
    v[j] = c / per + (c % per != 0);
    s += v[j];
  }
  uint32_t tot, run = block_excl_scan(s, ws, &tot);
#pragma unroll
  for (uint32_t j = 0; j < IPT; j++) {
    W.plan[threadIdx.x * IPT + j] = run;
    run += v[j];
  }
  if (threadIdx.x == 0) W.plan[BS_COARSE] = tot;
}

template <int NL>
__global__ void __launch_bounds__(BS_BLOCK) k_bs_hist(Limbs L, uint64_t n, const unsigned long long* n_dev,
                                                       unsigned nbits, BsWork W) {
  if (n_dev) n = min(n, (uint64_t)*n_dev);
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    atomicAdd(W.off + bs_bucket(bs_top<NL>(L, i, nbits), W.plan), 1u);
}

// W.off: the buckets' first positions, advanced to their ends as items arrive.
template <int NL, bool HASV>
__global__ void __launch_bounds__(BS_BLOCK) k_bs_scatter(Limbs S, const uint32_t* __restrict__ sv, Limbs D,
                                                          uint32_t* __restrict__ dv, uint64_t n,
                                                          const unsigned long long* n_dev, unsigned nbits,
                                                          BsWork W) {
  if (n_dev) n = min(n, (uint64_t)*n_dev);
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t p = atomicAdd(W.off + bs_bucket(bs_top<NL>(S, i, nbits), W.plan), 1u);
#pragma unroll
    for (int j = 0; j < NL; j++) D.p[j][p] = S.p[j][i];
    if (HASV) dv[p] = sv[i];
  }
}

constexpr uint32_t BS_WARP = 128;  // largest bucket one warp sorts

// Items [o, o + m), m <= 32 R, of T sorted ascending into D by one warp in
// registers: item r * 32 + lane in register r, a bitonic network whose
// distances below 32 are lane exchanges and whose others swap registers.
// Missing items are all-ones keys, which no item exceeds.
template <int NL, bool HASV, int R>
__device__ __forceinline__ void warp_sort(const Limbs& T, const uint32_t* __restrict__ tv, const Limbs& D,
                                          uint32_t* __restrict__ dv, uint32_t o, uint32_t m) {
  const unsigned lane = threadIdx.x & 31;
  uint64_t key[R][NL];
  uint32_t val[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const uint32_t i = r * 32 + lane;
    const bool in = i < m;
#pragma unroll
    for (int j = 0; j < NL; j++) key[r][j] = in ? T.p[j][o + i] : ~0ULL;
    val[r] = (HASV && in) ? tv[o + i] : 0u;
  }
  auto gt = [](const uint64_t (&a)[NL], const uint64_t (&b)[NL]) {
    bool g = a[0] > b[0];
#pragma unroll
    for (int j = 1; j < NL; j++) g = a[j] > b[j] || (a[j] == b[j] && g);
    return g;
  };
#pragma unroll
  for (uint32_t kk = 2; kk <= 32 * R; kk <<= 1) {
#pragma unroll
    for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
        const int q = (int)(j / 32);
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (r & q) continue;
          const bool up = ((r * 32 + lane) & kk) == 0;
          if (gt(key[r], key[r | q]) == up) {
#pragma unroll
            for (int l = 0; l < NL; l++) {
              const uint64_t t = key[r][l];
              key[r][l] = key[r | q][l];
              key[r | q][l] = t;
            }
            const uint32_t t = val[r];
            val[r] = val[r | q];
            val[r | q] = t;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          uint64_t ok[NL];
#pragma unroll
          for (int l = 0; l < NL; l++) ok[l] = __shfl_xor_sync(FULLM, key[r][l], j);
          const uint32_t ov = HASV ? __shfl_xor_sync(FULLM, val[r], j) : 0u;
          const bool lower = (lane & j) == 0, up = ((r * 32 + lane) & kk) == 0;
          // the lower lane of a pair keeps the smaller item when the run goes up
          const bool mine_gt = gt(key[r], ok), theirs_gt = gt(ok, key[r]);
          if (lower == up ? mine_gt : theirs_gt) {
#pragma unroll
            for (int l = 0; l < NL; l++) key[r][l] = ok[l];
            val[r] = ov;
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const uint32_t i = r * 32 + lane;
    if (i >= m) continue;
#pragma unroll
    for (int j = 0; j < NL; j++) D.p[j][o + i] = key[r][j];
    if (HASV) dv[o + i] = val[r];
  }
}

// Sorts every bucket of at most BS_LOCAL items from T into D; off[b] is the
// end of bucket b (its start is off[b - 1]).  A CTA takes BS_CHUNK buckets at a
// time, 32 per warp; the buckets too large for a warp wait in s_mid for the
// whole CTA.  Larger ones than BS_LOCAL are copied to D unsorted and listed in
// big[3i..3i+2] = (bucket, offset, size) for the host, which sorts them from T.
// Bound by the exchanges (15 stages of 2 NL + 1 shuffles for 32 items).
template <int NL, bool HASV>
__global__ void __launch_bounds__(BS_BLOCK) k_bs_local(Limbs T, const uint32_t* __restrict__ tv, Limbs D,
                                                        uint32_t* __restrict__ dv, BsWork W) {
  extern __shared__ __align__(16) uint64_t bs_smem[];
  __shared__ uint32_t s_mid[BS_CHUNK];
  __shared__ uint32_t s_nmid;
  const uint32_t nb = W.plan[BS_COARSE];
  const uint32_t* __restrict__ off = W.off;
  const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t* sk = bs_smem;                                // NL arrays of BS_LOCAL limbs
  uint32_t* svl = (uint32_t*)(bs_smem + NL * BS_LOCAL);  // values
  for (uint32_t c0 = blockIdx.x * BS_CHUNK; c0 < nb; c0 += gridDim.x * BS_CHUNK) {
    if (threadIdx.x == 0) s_nmid = 0;
    __syncthreads();
    const uint32_t b0 = c0 + w * 32;
    if (b0 < nb) {
      const uint32_t nw = min(32u, nb - b0);
      const uint32_t end = off[b0 + min(lane, nw - 1)];
      uint32_t s = b0 ? off[b0 - 1] : 0u;
      uint32_t cur = 0;
      while (cur < nw) {
        // buckets cur..last hold at most 32 items together
        const unsigned fit = __ballot_sync(FULLM, lane >= cur && lane < nw && end - s <= 32);
        if (fit) {
          const uint32_t last = 31 - __clz(fit);
          const uint32_t e = __shfl_sync(FULLM, end, last);
          if (e > s) warp_sort<NL, HASV, 1>(T, tv, D, dv, s, e - s);
          s = e;
          cur = last + 1;
          continue;
        }
        const uint32_t e = __shfl_sync(FULLM, end, cur);
        const uint32_t m = e - s;
        if (m <= 64) {
          warp_sort<NL, HASV, 2>(T, tv, D, dv, s, m);
        } else if (m <= BS_WARP) {
          warp_sort<NL, HASV, 4>(T, tv, D, dv, s, m);
        } else if (lane == 0) {
          s_mid[atomicAdd(&s_nmid, 1u)] = b0 + cur;
        }
        s = e;
        cur++;
      }
    }
    __syncthreads();
    const uint32_t nmid = s_nmid;
    for (uint32_t q = 0; q < nmid; q++) {
      const uint32_t b = s_mid[q];
      const uint32_t o = b ? off[b - 1] : 0u, m = off[b] - o;
      if (m > BS_LOCAL) {
        if (threadIdx.x == 0) {
          const unsigned i = atomicAdd(W.nbig, 1u);
          if (i < BS_MAX_BIG) {
            W.big[3 * i] = b;
            W.big[3 * i + 1] = o;
            W.big[3 * i + 2] = m;
          }
        }
        // The bucket goes to its place unsorted, so that D holds the whole
        // list (in every bucket's range) before the host sorts this range.
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
#pragma unroll
          for (int j = 0; j < NL; j++) D.p[j][o + i] = T.p[j][o + i];
          if (HASV) dv[o + i] = tv[o + i];
        }
        continue;
      }
      uint32_t P = 1;
      while (P < m) P <<= 1;
      for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
        const bool in = i < m;
#pragma unroll
        for (int j = 0; j < NL; j++) sk[j * BS_LOCAL + i] = in ? T.p[j][o + i] : ~0ULL;
        if (HASV) svl[i] = in ? tv[o + i] : 0u;
      }
      __syncthreads();
      for (uint32_t kk = 2; kk <= P; kk <<= 1) {
        for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
          for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
            const uint32_t x = i ^ j;
            if (x <= i) continue;
            // a > b on the limbs, most significant first
            bool g = false, eq = true;
#pragma unroll
            for (int l = NL - 1; l >= 0; l--) {
              const uint64_t u = sk[l * BS_LOCAL + i], v = sk[l * BS_LOCAL + x];
              if (eq && u != v) {
                g = u > v;
                eq = false;
              }
            }
            const bool up = (i & kk) == 0;
            if (g == up && !eq) {
#pragma unroll
              for (int l = 0; l < NL; l++) {
                const uint64_t t = sk[l * BS_LOCAL + i];
                sk[l * BS_LOCAL + i] = sk[l * BS_LOCAL + x];
                sk[l * BS_LOCAL + x] = t;
              }
              if (HASV) {
                const uint32_t t = svl[i];
                svl[i] = svl[x];
                svl[x] = t;
              }
            }
          }
          __syncthreads();
        }
      }
      for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
#pragma unroll
        for (int j = 0; j < NL; j++) D.p[j][o + i] = sk[j * BS_LOCAL + i];
        if (HASV) dv[o + i] = svl[i];
      }
      __syncthreads();
    }
    __syncthreads();  // s_mid is reused
  }
}

// The buckets k_bs_local left unsorted, side by side: seg[3i..3i+2] = (offset
// in the concatenation C, offset in the list L, size).  Gathers L's segments
// into C (back = false) or writes C's back into L; one CTA per segment.
template <int NL, bool HASV>
__global__ void __launch_bounds__(BS_BLOCK) k_bs_segments(Limbs L, uint32_t* lv, Limbs C, uint32_t* cv,
                                                           const uint32_t* __restrict__ seg, bool back) {
  const uint32_t co = seg[3 * blockIdx.x], lo = seg[3 * blockIdx.x + 1], m = seg[3 * blockIdx.x + 2];
  for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
#pragma unroll
    for (int j = 0; j < NL; j++) {
      if (back) L.p[j][lo + i] = C.p[j][co + i];
      else C.p[j][co + i] = L.p[j][lo + i];
    }
    if (HASV) {
      if (back) lv[lo + i] = cv[co + i];
      else cv[co + i] = lv[lo + i];
    }
  }
}
template <int NL>
static void launch_segments(cudaStream_t st, bool hasv, Limbs L, uint32_t* lv, Limbs C, uint32_t* cv,
                            const uint32_t* seg, uint32_t nseg, bool back) {
  if (hasv) k_bs_segments<NL, true><<<nseg, BS_BLOCK, 0, st>>>(L, lv, C, cv, seg, back);
  else k_bs_segments<NL, false><<<nseg, BS_BLOCK, 0, st>>>(L, lv, C, cv, seg, back);
}

// K, v: the list; T, tv: its bucketed copy; D, dv: the sorted list (may be K, v).
template <int NL, bool HASV>
static int bs_launch(cudaStream_t st, Limbs K, uint32_t* v, Limbs T, uint32_t* tv, Limbs D, uint32_t* dv, uint64_t n,
                     const unsigned long long* n_dev, unsigned nbits, const BsWork& W, uint32_t* launches) {
  const int sms = current_sm_count();
  const uint32_t nb = bs_max_buckets(n);
  const unsigned g = (unsigned)std::max<uint64_t>(
      std::min<uint64_t>((n + BS_BLOCK - 1) / BS_BLOCK, (uint64_t)sms * 16), 1);
  // (a CTA of the coarse count flushes its 4,096 bins: a few CTAs per SM)
  const unsigned gc = (unsigned)std::max<uint64_t>(std::min<uint64_t>(n / 1024, (uint64_t)sms * 4), 1);
  k_bs_coarse<NL><<<gc, BS_BLOCK, 0, st>>>(K, n, n_dev, nbits, W);
  k_bs_hist<NL><<<g, BS_BLOCK, 0, st>>>(K, n, n_dev, nbits, W);
  DevBuf sums;
  int rc;
  if ((rc = scan_u32(st, W.off, nb, sums, launches))) return rc;
  k_bs_scatter<NL, HASV><<<g, BS_BLOCK, 0, st>>>(K, v, T, tv, n, n_dev, nbits, W);
  const size_t smem = BS_LOCAL * (NL * 8 + (HASV ? 4 : 0));
  if ((rc = raise_smem_limit((const void*)k_bs_local<NL, HASV>, smem))) return rc;
  const unsigned gl = (unsigned)std::min<uint32_t>((nb + BS_CHUNK - 1) / BS_CHUNK, (uint32_t)sms * 8);
  k_bs_local<NL, HASV><<<gl, BS_BLOCK, smem, st>>>(T, tv, D, dv, W);
  SPK_CUDA(cudaGetLastError());
  if (launches) *launches += 4;
  return SPK_OK;
}
static int bs_launch_nl(int nl, bool hasv, cudaStream_t st, Limbs K, uint32_t* v, Limbs T, uint32_t* tv,
                        Limbs D, uint32_t* dv, uint64_t n, const unsigned long long* n_dev, unsigned nbits, const BsWork& W,
                        uint32_t* launches) {
  switch (nl * 2 + (hasv ? 1 : 0)) {
    case 2: return bs_launch<1, false>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    case 3: return bs_launch<1, true>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    case 4: return bs_launch<2, false>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    case 5: return bs_launch<2, true>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    case 6: return bs_launch<3, false>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    case 7: return bs_launch<3, true>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    case 8: return bs_launch<4, false>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
    default: return bs_launch<4, true>(st, K, v, T, tv, D, dv, n, n_dev, nbits, W, launches);
  }
}

int sort_bufs(cudaStream_t st, int nl, uint64_t n, unsigned nbits, DevBuf* keys, DevBuf* vals,
              uint64_t* h_staging, uint32_t* launches) {
  if (n <= 1) return SPK_OK;
  if (!h_staging) return radix_sort_bufs(st, nl, n, nbits, keys, vals, launches);
  if (n >= (1ULL << 32)) return fail(SPK_E_INVALID_ARG, "sort: more than 2^32 items");
  int rc;
  DevBuf tk[4], tv, work;
  Limbs K{}, T{};
  for (int j = 0; j < nl; j++) {
    if ((rc = tk[j].alloc(n * 8, st))) return rc;
    K.p[j] = keys[j].as<uint64_t>();
    T.p[j] = tk[j].as<uint64_t>();
  }
  if (vals && (rc = tv.alloc(n * 4, st))) return rc;
  if ((rc = work.alloc(bs_work_bytes(n), st))) return rc;
  SPK_CUDA(cudaMemsetAsync(work.p, 0, bs_work_bytes(n), st));
  const BsWork W = bs_work(work.as<uint32_t>());
  uint32_t* v = vals ? vals->as<uint32_t>() : nullptr;
  uint32_t* tvp = vals ? tv.as<uint32_t>() : nullptr;
  if ((rc = bs_launch_nl(nl, vals != nullptr, st, K, v, T, tvp, K, v, n, nullptr, nbits, W, launches))) return rc;
  uint64_t* hs = h_staging + BS_STAGE_WORDS;
  SPK_CUDA(cudaMemcpyAsync(hs, W.nbig, 4, cudaMemcpyDeviceToHost, st));
  SPK_CUDA(cudaStreamSynchronize(st));
  const unsigned nbig_h = ((unsigned*)hs)[0];
  if (nbig_h > BS_MAX_BIG) {
    // Too many large buckets: sort the bucketed copy as a whole instead.
    for (int j = 0; j < nl; j++)
      SPK_CUDA(cudaMemcpyAsync(K.p[j], T.p[j], n * 8, cudaMemcpyDeviceToDevice, st));
    if (vals) SPK_CUDA(cudaMemcpyAsync(v, tvp, n * 4, cudaMemcpyDeviceToDevice, st));
    return radix_sort_bufs(st, nl, n, nbits, keys, vals, launches);
  }
  if (nbig_h == 0) return SPK_OK;
  SPK_CUDA(cudaMemcpyAsync(hs, W.big, (size_t)nbig_h * 12, cudaMemcpyDeviceToHost, st));
  SPK_CUDA(cudaStreamSynchronize(st));
  std::vector<uint32_t> bl((const uint32_t*)hs, (const uint32_t*)hs + 3 * nbig_h);
  for (unsigned q = 0; q < nbig_h; q++) {
    const uint64_t o = bl[3 * q + 1], m = bl[3 * q + 2];
    DevBuf bk[4], bvv;
    for (int j = 0; j < nl; j++) {
      if ((rc = bk[j].alloc(m * 8, st))) return rc;
      SPK_CUDA(cudaMemcpyAsync(bk[j].p, T.p[j] + o, m * 8, cudaMemcpyDeviceToDevice, st));
    }
    if (vals) {
      if ((rc = bvv.alloc(m * 4, st))) return rc;
      SPK_CUDA(cudaMemcpyAsync(bvv.p, tvp + o, m * 4, cudaMemcpyDeviceToDevice, st));
    }
    if ((rc = radix_sort_bufs(st, nl, m, nbits, bk, vals ? &bvv : nullptr, launches))) return rc;
    for (int j = 0; j < nl; j++)
      SPK_CUDA(cudaMemcpyAsync(K.p[j] + o, bk[j].p, m * 8, cudaMemcpyDeviceToDevice, st));
    if (vals) SPK_CUDA(cudaMemcpyAsync(v + o, bvv.p, m * 4, cudaMemcpyDeviceToDevice, st));
  }
  return SPK_OK;
}

// Bucket sort of a list whose length is known only on the device (*n_dev, at
// most n_cap): the same split and shared-memory sorts, enqueued without
// reading anything back.  Buckets over BS_LOCAL items stay in the bucketed
// copy and are listed on the device; sort_dev_finish sorts them once the
// host has the counts.  Temporaries: tmp_keys (nullable, NL limb arrays of
// n_cap items that the caller no longer needs) or new allocations.  exact: n_cap
// is the length, and the sorted list goes to new buffers of its size that a result
// keeps (keys and vals then hold those).
int sort_dev_enqueue(cudaStream_t st, int nl, uint64_t n_cap, const unsigned long long* n_dev,
                     unsigned nbits, DevBuf* keys, DevBuf* vals, DevBuf* tmp_keys, bool exact, DevSort& ds,
                     uint32_t* launches) {
  if (n_cap >= (1ULL << 32)) return fail(SPK_E_INVALID_ARG, "sort: more than 2^32 items");
  ds.nl = nl;
  ds.nbits = nbits;
  ds.n_cap = n_cap;
  ds.has_vals = vals != nullptr;
  int rc;
  Limbs K{}, T{};
  for (int j = 0; j < nl; j++) {
    if (tmp_keys) ds.tk[j] = std::move(tmp_keys[j]);
    else if ((rc = ds.tk[j].alloc(std::max<uint64_t>(n_cap, 1) * 8, st))) return rc;
    K.p[j] = keys[j].as<uint64_t>();
    T.p[j] = ds.tk[j].as<uint64_t>();
  }
  if (vals && (rc = ds.tv.alloc(std::max<uint64_t>(n_cap, 1) * 4, st))) return rc;
  if ((rc = ds.work.alloc(bs_work_bytes(n_cap), st))) return rc;
  SPK_CUDA(cudaMemsetAsync(ds.work.p, 0, bs_work_bytes(n_cap), st));
  uint32_t* v = vals ? vals->as<uint32_t>() : nullptr;
  uint32_t* tvp = vals ? ds.tv.as<uint32_t>() : nullptr;
  DevBuf dk[4], dvb;
  Limbs D = K;
  uint32_t* dv = v;
  if (exact) {
    for (int j = 0; j < nl; j++) {
      if ((rc = dk[j].alloc_keep(std::max<uint64_t>(n_cap, 2) * 8, st))) return rc;
      D.p[j] = dk[j].as<uint64_t>();
    }
    if (vals && (rc = dvb.alloc_keep(std::max<uint64_t>(n_cap, 4) * 4, st))) return rc;
    if (vals) dv = dvb.as<uint32_t>();
  }
  if ((rc = bs_launch_nl(nl, vals != nullptr, st, K, v, T, tvp, D, dv, n_cap, n_dev, nbits,
                         bs_work(ds.work.as<uint32_t>()), launches)))
    return rc;
  if (exact) {  // (the old buffers are freed after the sort, in stream order)
    for (int j = 0; j < nl; j++) keys[j] = std::move(dk[j]);
    if (vals) *vals = std::move(dvb);
  }
  ds.pending = true;
  return SPK_OK;
}

const unsigned* sort_dev_nbig(const DevSort& ds) {
  return bs_work(ds.work.as<uint32_t>()).nbig;
}

// Sorts the buckets sort_dev_enqueue left over (nbig_host of them, read
// back by the caller; n_host = the list length) and frees the temporaries.
int sort_dev_finish(cudaStream_t st, DevSort& ds, DevBuf* keys, DevBuf* vals, uint64_t n_host,
                    unsigned nbig_host, uint64_t* h_staging, uint32_t* launches) {
  if (!ds.pending) return SPK_OK;
  ds.pending = false;
  const int nl = ds.nl;
  int rc;
  uint32_t* v = vals ? vals->as<uint32_t>() : nullptr;
  uint32_t* tvp = vals ? ds.tv.as<uint32_t>() : nullptr;
  if (nbig_host > BS_MAX_BIG) {
    // Too many large buckets: sort the bucketed copy as a whole instead.
    for (int j = 0; j < nl; j++)
      SPK_CUDA(cudaMemcpyAsync(keys[j].p, ds.tk[j].p, n_host * 8, cudaMemcpyDeviceToDevice, st));
    if (vals) SPK_CUDA(cudaMemcpyAsync(v, tvp, n_host * 4, cudaMemcpyDeviceToDevice, st));
    rc = radix_sort_bufs(st, nl, n_host, ds.nbits, keys, vals, launches);
  } else if (nbig_host > 0) {
    // The large buckets side by side, in list order, sorted as one array on
    // their whole keys (their top bits keep the buckets apart), then put
    // back: one sort however many buckets there are.
    uint32_t* hs = (uint32_t*)(h_staging + BS_STAGE_WORDS);
    uint32_t* seg = bs_work(ds.work.as<uint32_t>()).big;
    SPK_CUDA(cudaMemcpyAsync(hs, seg, (size_t)nbig_host * 12, cudaMemcpyDeviceToHost, st));
    SPK_CUDA(cudaStreamSynchronize(st));
    std::vector<std::pair<uint32_t, uint32_t>> segs(nbig_host);  // (offset in the list, size)
    for (unsigned q = 0; q < nbig_host; q++) segs[q] = {hs[3 * q + 1], hs[3 * q + 2]};
    std::sort(segs.begin(), segs.end());
    uint64_t total = 0;
    for (unsigned q = 0; q < nbig_host; q++) {
      hs[3 * q] = (uint32_t)total;
      hs[3 * q + 1] = segs[q].first;
      hs[3 * q + 2] = segs[q].second;
      total += segs[q].second;
    }
    SPK_CUDA(cudaMemcpyAsync(seg, hs, (size_t)nbig_host * 12, cudaMemcpyHostToDevice, st));
    DevBuf ck[4], cvb;
    Limbs L{}, Cc{};
    for (int j = 0; j < nl; j++) {
      if ((rc = ck[j].alloc(total * 8, st))) return rc;
      L.p[j] = keys[j].as<uint64_t>();
      Cc.p[j] = ck[j].as<uint64_t>();
    }
    if (vals && (rc = cvb.alloc(total * 4, st))) return rc;
    uint32_t* cvp = vals ? cvb.as<uint32_t>() : nullptr;
    switch (nl) {
      case 1: launch_segments<1>(st, vals, L, v, Cc, cvp, seg, nbig_host, false); break;
      case 2: launch_segments<2>(st, vals, L, v, Cc, cvp, seg, nbig_host, false); break;
      case 3: launch_segments<3>(st, vals, L, v, Cc, cvp, seg, nbig_host, false); break;
      default: launch_segments<4>(st, vals, L, v, Cc, cvp, seg, nbig_host, false); break;
    }
    SPK_CUDA(cudaGetLastError());
    if ((rc = radix_sort_bufs(st, nl, total, ds.nbits, ck, vals ? &cvb : nullptr, launches))) return rc;
    for (int j = 0; j < nl; j++) Cc.p[j] = ck[j].as<uint64_t>();  // the sort may have swapped buffers
    cvp = vals ? cvb.as<uint32_t>() : nullptr;
    switch (nl) {
      case 1: launch_segments<1>(st, vals, L, v, Cc, cvp, seg, nbig_host, true); break;
      case 2: launch_segments<2>(st, vals, L, v, Cc, cvp, seg, nbig_host, true); break;
      case 3: launch_segments<3>(st, vals, L, v, Cc, cvp, seg, nbig_host, true); break;
      default: launch_segments<4>(st, vals, L, v, Cc, cvp, seg, nbig_host, true); break;
    }
    SPK_CUDA(cudaGetLastError());
    if (launches) *launches += 2;
  } else {
    rc = SPK_OK;
  }
  ds.release();
  return rc;
}

// ---------------------------------------------------------------------------
// Ordered compaction with conversion of sequence values to Kmer256 limbs.
// Item i of a sorted SoA list is kept when cin == nullptr or cin[i] >=
// min_count; kept items are written in list order as AoS Kmer256 limbs.
// ---------------------------------------------------------------------------
constexpr int OC_BLOCK = 256, OC_IPT = 16, OC_TILE = OC_BLOCK * OC_IPT;

__global__ void __launch_bounds__(OC_BLOCK) k_oc_count(const uint32_t* __restrict__ cin, uint64_t n,
                                                        uint32_t min_count,
                                                        uint32_t* __restrict__ bc) {
  __shared__ uint32_t s;
  if (threadIdx.x == 0) s = 0;
  __syncthreads();
  uint32_t c = 0;
  const uint64_t base = (uint64_t)blockIdx.x * OC_TILE;
  for (int j = 0; j < OC_IPT; j++) {
    const uint64_t i = base + j * OC_BLOCK + threadIdx.x;
    c += i < n && (cin == nullptr || cin[i] >= min_count);
  }
  atomicAdd(&s, c);
  __syncthreads();
  if (threadIdx.x == 0) bc[blockIdx.x] = s;
}

template <int NL>
__global__ void __launch_bounds__(OC_BLOCK) k_oc_write(const uint64_t* l0, const uint64_t* l1,
                                                        const uint64_t* l2, const uint64_t* l3,
                                                        const uint32_t* __restrict__ cin, uint64_t n,
                                                        unsigned k, uint32_t min_count,
                                                        const uint32_t* __restrict__ bc,
                                                        uint64_t* __restrict__ out,
                                                        uint32_t* __restrict__ cout, uint64_t out_cap) {
  __shared__ uint32_t ws[OC_BLOCK / 32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Thread t owns the contiguous items [t*IPT, t*IPT+IPT) of the tile.
  const uint64_t base = (uint64_t)blockIdx.x * OC_TILE + (uint64_t)threadIdx.x * OC_IPT;
  uint32_t keepmask = 0;
#pragma unroll
  for (int j = 0; j < OC_IPT; j++) {
    const uint64_t i = base + j;
    if (i < n && (cin == nullptr || cin[i] >= min_count)) keepmask |= 1u << j;
  }
  const uint32_t c = __popc(keepmask);
  uint32_t x = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t t = __shfl_up_sync(FULLM, x, d);
    if ((int)lane >= d) x += t;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  uint32_t wpre = 0;
  for (unsigned w = 0; w < warp; w++) wpre += ws[w];
  uint64_t p = (uint64_t)bc[blockIdx.x] + wpre + x - c;
#pragma unroll 1
  for (int j = 0; j < OC_IPT; j++) {
    if (!(keepmask & (1u << j))) continue;
    if (p >= out_cap) break;  // (a caller's count of the kept items that was short)
    const uint64_t i = base + j;
    Seq<NL> V;
    V.v[0] = l0[i];
    if (NL > 1) V.v[NL > 1 ? 1 : 0] = l1[i];
    if (NL > 2) V.v[NL > 2 ? 2 : 0] = l2[i];
    if (NL > 3) V.v[NL > 3 ? 3 : 0] = l3[i];
    uint64_t w[4];
    kmer256_limbs<NL>(V, k, w);
#pragma unroll
    for (int q = 0; q < NL; q++) out[p * NL + q] = w[q];
    if (cout) cout[p] = cin[i];
    p++;
  }
}

// The conversion of a whole list (no filter).
struct ListLimbs {
  const uint64_t* p[4];
};
template <int NL>
__global__ void __launch_bounds__(OC_BLOCK) k_oc_all(ListLimbs L, uint64_t n, unsigned k, uint64_t* __restrict__ out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    Seq<NL> V;
#pragma unroll
    for (int j = 0; j < NL; j++) V.v[j] = __ldcs(L.p[j] + i);
    uint64_t w[4];
    kmer256_limbs<NL>(V, k, w);
#pragma unroll
    for (int q = 0; q < NL; q++) out[i * NL + q] = w[q];
  }
}

// Returns the number of kept items in *m (host value; synchronises st when cin
// filters and the number is not known).
int ordered_convert(cudaStream_t st, int nl, uint64_t n, unsigned k, DevBuf* limbs,
                    const uint32_t* cin, uint32_t min_count, DevBuf* out, DevBuf* cout,
                    uint64_t* h_staging, uint64_t* m, uint64_t known_m) {
  int rc;
  if (!cin) {  // every item is kept: nothing to count
    *m = n;
    if ((rc = out->alloc_keep(std::max<uint64_t>(n, 1) * nl * 8, st))) return rc;
    if (n) {
      const ListLimbs L{{limbs[0].as<uint64_t>(), nl > 1 ? limbs[1].as<uint64_t>() : nullptr,
                         nl > 2 ? limbs[2].as<uint64_t>() : nullptr, nl > 3 ? limbs[3].as<uint64_t>() : nullptr}};
      const unsigned g = (unsigned)std::min<uint64_t>((n + OC_BLOCK - 1) / OC_BLOCK, (uint64_t)current_sm_count() * 16);
      uint64_t* o = out->as<uint64_t>();
      switch (nl) {
        case 1: k_oc_all<1><<<g, OC_BLOCK, 0, st>>>(L, n, k, o); break;
        case 2: k_oc_all<2><<<g, OC_BLOCK, 0, st>>>(L, n, k, o); break;
        case 3: k_oc_all<3><<<g, OC_BLOCK, 0, st>>>(L, n, k, o); break;
        default: k_oc_all<4><<<g, OC_BLOCK, 0, st>>>(L, n, k, o); break;
      }
      SPK_CUDA(cudaGetLastError());
    }
    return SPK_OK;
  }
  const uint32_t nt = (uint32_t)std::max<uint64_t>((n + OC_TILE - 1) / OC_TILE, 1);
  DevBuf bc;
  if ((rc = bc.alloc((uint64_t)(nt + 1) * 4, st))) return rc;
  SPK_CUDA(cudaMemsetAsync(bc.p, 0, (uint64_t)(nt + 1) * 4, st));
  if (n) {
    k_oc_count<<<nt, OC_BLOCK, 0, st>>>(cin, n, min_count, bc.as<uint32_t>());
  }
  DevBuf sums;
  if ((rc = scan_u32(st, bc.as<uint32_t>(), nt + 1, sums))) return rc;
  if (known_m != ~0ULL) {
    *m = known_m;
  } else {
    SPK_CUDA(cudaMemcpyAsync(h_staging, bc.as<uint32_t>() + nt, 4, cudaMemcpyDeviceToHost, st));
    SPK_CUDA(cudaStreamSynchronize(st));
    *m = (uint64_t)((uint32_t*)h_staging)[0];
  }
  if ((rc = out->alloc_keep(std::max<uint64_t>(*m, 1) * nl * 8, st))) return rc;
  if (cout && (rc = cout->alloc_keep(std::max<uint64_t>(*m, 1) * 4, st))) return rc;
  if (n && *m) {
    const uint64_t* p[4] = {nullptr, nullptr, nullptr, nullptr};
    for (int j = 0; j < nl; j++) p[j] = limbs[j].as<uint64_t>();
    uint64_t* o = out->as<uint64_t>();
    uint32_t* oc = cout ? cout->as<uint32_t>() : nullptr;
    switch (nl) {
      case 1: k_oc_write<1><<<nt, OC_BLOCK, 0, st>>>(p[0], p[1], p[2], p[3], cin, n, k, min_count, bc.as<uint32_t>(), o, oc, *m); break;
      case 2: k_oc_write<2><<<nt, OC_BLOCK, 0, st>>>(p[0], p[1], p[2], p[3], cin, n, k, min_count, bc.as<uint32_t>(), o, oc, *m); break;
      case 3: k_oc_write<3><<<nt, OC_BLOCK, 0, st>>>(p[0], p[1], p[2], p[3], cin, n, k, min_count, bc.as<uint32_t>(), o, oc, *m); break;
      default: k_oc_write<4><<<nt, OC_BLOCK, 0, st>>>(p[0], p[1], p[2], p[3], cin, n, k, min_count, bc.as<uint32_t>(), o, oc, *m); break;
    }
    SPK_CUDA(cudaGetLastError());
  }
  return SPK_OK;
}

}  // namespace spk
