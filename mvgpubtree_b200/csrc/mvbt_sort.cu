// Stable LSD radix sort of 32-bit keys with 32-bit payloads, hand-written for sm_100a: the sort
// stage of the sorted batch front-end (mvbt_sort.h). The payload of each key is the caller's word for
// it, or its position in the caller's array, generated by the first pass.
//
// A pass over one 8-bit digit is three kernels:
//   k_sort_hist     per tile of keys, the count of each digit (shared-memory counters), digit-major:
//                   counts[d * tiles + tile];
//   k_sort_rows     one block per digit: exclusive prefix over its tiles, and the digit's total;
//   k_sort_scatter  per tile: the warps rank their keys in input order (so the sort is stable) against
//                   per-warp digit counters in shared memory, with no block barrier inside the ranking;
//                   keys and payloads are reordered by digit in shared memory and written so that
//                   consecutive threads write consecutive positions of one digit's run.
// HBM-bound streaming: a pass reads the keys twice and reads and writes keys and payloads once. (A
// pass in one kernel, each tile adding up the digit counts of the tiles before it as they are
// published, was measured and not kept: the chain of look-backs took about 40 ns a tile whatever
// the tile held, 0.30-0.33 ms a pass of 2^25 keys.)
#include <cuda_runtime.h>

#include <cstdint>

#include "mvbt_sort.h"

namespace {

constexpr int kRadix       = 256;
constexpr int kThreads     = 256;
constexpr int kWarps       = kThreads / 32;
constexpr int kItemsLarge  = 16;  // keys per thread: tiles of 4096 keys ...
constexpr int kItemsSmall  = 8;   // ... or 2048, when there would be too few large tiles
constexpr int kScanThreads = 1024;
constexpr int kScanItems   = 4;
constexpr int kScanChunk   = kScanThreads * kScanItems;

// Large tiles write longer runs of each digit and leave fewer counts to scan; small ones spread a
// short sort over more SMs. Four passes, large / small tiles: 2^20 keys 84 / 74 us, 2.0M keys 115 /
// 99 us (large as 512 threads there), 2^22 keys 159 / 164 us, 2^25 keys 952 / 1043 us.
constexpr uint32_t kLargeFrom = 7u << 19;

inline uint32_t items_for(uint32_t n) { return n >= kLargeFrom ? kItemsLarge : kItemsSmall; }
inline uint32_t tiles_for(uint32_t n) {
  const uint64_t tile = (uint64_t)kThreads * items_for(n);
  return (uint32_t)((n + tile - 1) / tile);
}

template <int kItems>
__global__ void __launch_bounds__(kThreads) k_sort_hist(const uint32_t* __restrict__ keys, uint32_t n, int shift,
                                                        uint32_t tiles, uint32_t* __restrict__ counts) {
  constexpr uint32_t kTile = kThreads * kItems;
  __shared__ uint32_t h[kRadix];
  if (threadIdx.x < kRadix) h[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t first   = blockIdx.x * kTile;
  const uint32_t in_tile = n - first < kTile ? n - first : kTile;
  uint32_t k[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const uint32_t j = threadIdx.x + (uint32_t)r * kThreads;
    k[r]             = j < in_tile ? keys[first + j] : 0u;
  }
#pragma unroll
  for (int r = 0; r < kItems; ++r)
    if (threadIdx.x + (uint32_t)r * kThreads < in_tile) atomicAdd(&h[(k[r] >> shift) & 255u], 1u);
  __syncthreads();
  if (threadIdx.x < kRadix) counts[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// The lanes of the warp that hold a key (ok) of the same digit. Eight ballots, one per bit: on uniform
// digits (about 30 distinct ones in a warp) __match_any_sync took an SM about 64 cycles, and with it
// a pass over 2^25 keys took 0.40 ms.
__device__ __forceinline__ uint32_t same_digit(uint32_t d, bool ok) {
  uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const bool bit   = (d >> b) & 1u;
    const uint32_t m = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? m : ~m;
  }
  return peers;
}

// Stable scatter of one tile by the digit at `shift`. vin == nullptr: the payload is the key's
// input position (first pass). before: k_sort_rows' prefixes, totals: its digit totals.
template <int kItems>
__global__ void __launch_bounds__(kThreads, 3)
    k_sort_scatter(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
                   uint32_t* __restrict__ vout, uint32_t n, int shift, uint32_t tiles,
                   const uint32_t* __restrict__ before, const uint32_t* __restrict__ totals) {
  constexpr uint32_t kTile = kThreads * kItems;
  __shared__ uint2 s_pair[kTile];
  __shared__ uint16_t s_cnt[kWarps][kRadix];  // keys of each digit: per warp, then prefix over the warps
  __shared__ uint32_t s_start[kRadix];        // tile-local first position of each digit
  __shared__ uint32_t s_glob[kRadix];         // global position of a digit's key = s_glob + tile-local one
  __shared__ uint32_t s_warp[2][kRadix / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kWarps * kRadix / 2; i += kThreads) reinterpret_cast<uint32_t*>(s_cnt)[i] = 0;
  __syncthreads();
  const uint32_t tile    = blockIdx.x;
  const uint32_t base    = tile * kTile + (uint32_t)warp * (32 * kItems) + lane;  // may pass n, never 2^32
  const uint32_t in_tile = n - tile * kTile < kTile ? n - tile * kTile : kTile;
  const uint32_t mine    = (uint32_t)warp * (32 * kItems) + lane;  // tile-local position of the first key
  uint32_t k[kItems], v[kItems], rank[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) k[r] = mine + 32u * r < in_tile ? kin[base + 32u * r] : 0u;
#pragma unroll
  for (int r = 0; r < kItems; ++r)  // on their way while the keys are ranked
    v[r] = !vin ? base + 32u * r : (mine + 32u * r < in_tile ? vin[base + 32u * r] : 0u);
  const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const bool ok         = mine + 32u * r < in_tile;
    const uint32_t d      = (k[r] >> shift) & 255u;
    const uint32_t peers  = same_digit(d, ok);
    const uint32_t before = s_cnt[warp][d];
    __syncwarp();
    if (ok && (peers & lt_mask) == 0) s_cnt[warp][d] = (uint16_t)(before + __popc(peers));
    __syncwarp();
    rank[r] = before + __popc(peers & lt_mask);
  }
  __syncthreads();
  uint32_t count = 0, total = 0, row = 0;
  if (tid < kRadix) {  // the digit's first position in the tile, and in the output
    total = totals[tid];
    row   = before[(uint64_t)tid * tiles + tile];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = s_cnt[w][tid];
      s_cnt[w][tid]    = (uint16_t)count;
      count += c;
    }
    uint32_t inc = count, tot = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d), z = __shfl_up_sync(0xffffffffu, tot, d);
      if (lane >= d) inc += y, tot += z;
    }
    if (lane == 31) s_warp[0][warp] = inc, s_warp[1][warp] = tot;
    count = inc - count;
    total = tot - total;
  }
  __syncthreads();
  if (tid < kRadix) {
    for (int w = 0; w < warp; ++w) count += s_warp[0][w], total += s_warp[1][w];
    s_start[tid] = count;
    s_glob[tid]  = total + row - count;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    if (mine + 32u * r < in_tile) {
      const uint32_t d = (k[r] >> shift) & 255u;
      s_pair[rank[r] + s_start[d] + s_cnt[warp][d]] = make_uint2(k[r], v[r]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const uint32_t j = tid + (uint32_t)r * kThreads;
    if (j < in_tile) {
      const uint2 p     = s_pair[j];
      const uint32_t at = s_glob[(p.x >> shift) & 255u] + j;
      kout[at]          = p.x;
      vout[at]          = p.y;
    }
  }
}

// Exclusive scan of 1024 threads x kScanItems values held per thread; returns the block total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t (&v)[kScanItems], uint32_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t sum = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint32_t x = v[j];
    v[j]             = sum;
    sum += x;
  }
  uint32_t inc = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += y;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = s_warp[lane], wi = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, wi, d);
      if (lane >= d) wi += y;
    }
    s_warp[lane] = wi - w;  // exclusive prefix of warp totals
    if (lane == 31) s_warp[32] = wi;
  }
  __syncthreads();
  const uint32_t off = s_warp[warp] + inc - sum;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) v[j] += off;
  const uint32_t total = s_warp[32];
  __syncthreads();
  return total;
}

// Block d: the exclusive prefix of digit d's counts over the tiles, in place, and their total.
__global__ void __launch_bounds__(kScanThreads) k_sort_rows(uint32_t* __restrict__ counts, uint32_t tiles,
                                                            uint32_t* __restrict__ totals) {
  __shared__ uint32_t s_warp[33];
  uint32_t* row  = counts + (uint64_t)blockIdx.x * tiles;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < tiles; base += kScanChunk) {
    uint32_t v[kScanItems];
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
      const uint32_t i = base + threadIdx.x * kScanItems + j;
      v[j]             = i < tiles ? row[i] : 0u;
    }
    const uint32_t total = block_exclusive_scan(v, s_warp);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
      const uint32_t i = base + threadIdx.x * kScanItems + j;
      if (i < tiles) row[i] = v[j] + carry;
    }
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Whether sorted position i of n holds a pair that a load keeps: the last occurrence of its key.
__device__ __forceinline__ bool kept(const uint32_t* keys, uint32_t i, uint32_t n, uint32_t key) {
  return i < n && key != 0xFFFFFFFFu && !(i + 1 < n && keys[i + 1] == key);
}

// Kept pairs per tile of kKeepTile positions: counts[1 + tile].
constexpr uint32_t kKeepItems = 8, kKeepTile = kThreads * kKeepItems;
__global__ void __launch_bounds__(kThreads) k_keep_count(const uint32_t* __restrict__ keys, uint32_t n,
                                                         uint32_t* __restrict__ counts) {
  __shared__ uint32_t s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  const uint32_t first = blockIdx.x * kKeepTile + threadIdx.x;
  uint32_t c = 0;
#pragma unroll
  for (uint32_t r = 0; r < kKeepItems; ++r) {
    const uint32_t i = first + r * kThreads;
    if (i >= first && i < n && kept(keys, i, n, keys[i])) ++c;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, c);
  __syncthreads();
  if (threadIdx.x == 0) counts[1 + blockIdx.x] = s_sum;
}

// One block: counts[1 + tile] becomes the tile's first output position, counts[0] the total.
__global__ void __launch_bounds__(kScanThreads) k_keep_scan(uint32_t* __restrict__ counts, uint32_t tiles) {
  __shared__ uint32_t s_warp[33];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < tiles; base += kScanChunk) {
    uint32_t v[kScanItems];
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
      const uint32_t i = base + threadIdx.x * kScanItems + j;
      v[j]             = i < tiles ? counts[1 + i] : 0u;
    }
    const uint32_t total = block_exclusive_scan(v, s_warp);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
      const uint32_t i = base + threadIdx.x * kScanItems + j;
      if (i < tiles) counts[1 + i] = v[j] + carry;
    }
    carry += total;
  }
  if (threadIdx.x == 0) counts[0] = carry;
}

// The tile's kept pairs, compacted: a ballot per row of 256 positions.
__global__ void __launch_bounds__(kThreads) k_keep_move(const uint32_t* __restrict__ keys,
                                                        const uint32_t* __restrict__ values, uint32_t n,
                                                        uint32_t* __restrict__ k_out, uint32_t* __restrict__ v_out,
                                                        const uint32_t* __restrict__ counts) {
  __shared__ uint32_t s_cnt[kKeepItems * kWarps], s_at[kKeepItems * kWarps];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t first = blockIdx.x * kKeepTile + threadIdx.x;
  uint32_t k[kKeepItems], m[kKeepItems];
#pragma unroll
  for (uint32_t r = 0; r < kKeepItems; ++r) {
    const uint32_t i = first + r * kThreads;
    const bool ok    = i >= first && i < n;
    k[r]             = ok ? keys[i] : 0u;
    m[r]             = __ballot_sync(0xffffffffu, ok && kept(keys, i, n, k[r]));
    if (lane == 0) s_cnt[r * kWarps + warp] = __popc(m[r]);
  }
  __syncthreads();
  if (threadIdx.x < kKeepItems * kWarps) {  // exclusive scan of the rows' warps, in order
    uint32_t sum = 0;
    for (uint32_t j = 0; j < threadIdx.x; ++j) sum += s_cnt[j];
    s_at[threadIdx.x] = sum;
  }
  __syncthreads();
  const uint32_t base = counts[1 + blockIdx.x];
#pragma unroll
  for (uint32_t r = 0; r < kKeepItems; ++r) {
    if (!((m[r] >> lane) & 1u)) continue;
    const uint32_t at = base + s_at[r * kWarps + warp] + (uint32_t)__popc(m[r] & ((1u << lane) - 1u));
    k_out[at]         = k[r];
    v_out[at]         = values[first + r * kThreads];
  }
}

int launch_error() {
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

}  // namespace

namespace mvbt_sort {

uint64_t scratch_words(uint32_t n) { return (uint64_t)kRadix * tiles_for(n) + kRadix; }

uint64_t keep_words(uint32_t n) { return 1 + ((uint64_t)n + kKeepTile - 1) / kKeepTile; }

int keep_last(const uint32_t* keys, const uint32_t* values, uint32_t n, uint32_t* k_out, uint32_t* v_out,
              uint32_t* counts, cudaStream_t s) {
  const uint32_t tiles = (uint32_t)(((uint64_t)n + kKeepTile - 1) / kKeepTile);
  k_keep_count<<<tiles, kThreads, 0, s>>>(keys, n, counts);
  k_keep_scan<<<1, kScanThreads, 0, s>>>(counts, tiles);
  k_keep_move<<<tiles, kThreads, 0, s>>>(keys, values, n, k_out, v_out, counts);
  return launch_error() ? 2 : 0;
}

int sort_pairs(const uint32_t* keys, const uint32_t* payload, uint32_t n, int low_bit, uint32_t* k_out,
               uint32_t* v_out, uint32_t* k_tmp, uint32_t* v_tmp, uint32_t* scratch, cudaStream_t s) {
  if (n == 0) return 0;
  if (low_bit < 0 || low_bit > 24 || (low_bit & 7)) return 1;
  const uint32_t tiles = tiles_for(n);
  const int passes     = (32 - low_bit) / 8;
  uint32_t* counts     = scratch;
  uint32_t* totals     = scratch + (uint64_t)kRadix * tiles;
  const uint32_t* kin  = keys;
  const uint32_t* vin  = payload;
  const bool large     = items_for(n) == kItemsLarge;
  for (int p = 0; p < passes; ++p) {
    // the last pass lands in k_out / v_out; earlier ones alternate so that it does
    const bool to_out = ((passes - 1 - p) & 1) == 0;
    uint32_t* ko      = to_out ? k_out : k_tmp;
    uint32_t* vo      = to_out ? v_out : v_tmp;
    const int shift   = low_bit + 8 * p;
    if (large) k_sort_hist<kItemsLarge><<<tiles, kThreads, 0, s>>>(kin, n, shift, tiles, counts);
    else k_sort_hist<kItemsSmall><<<tiles, kThreads, 0, s>>>(kin, n, shift, tiles, counts);
    k_sort_rows<<<kRadix, kScanThreads, 0, s>>>(counts, tiles, totals);
    if (large) k_sort_scatter<kItemsLarge><<<tiles, kThreads, 0, s>>>(kin, vin, ko, vo, n, shift, tiles, counts, totals);
    else k_sort_scatter<kItemsSmall><<<tiles, kThreads, 0, s>>>(kin, vin, ko, vo, n, shift, tiles, counts, totals);
    if (launch_error()) return 2;
    kin = ko;
    vin = vo;
  }
  return 0;
}

}  // namespace mvbt_sort
