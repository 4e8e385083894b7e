// Device-side multiversion B-link tree for sm_100a.
//
// This header is the device half of the library. Its kernels (mvgpubtree_b200/csrc) and user
// kernels call the same tile-cooperative operations, the counterparts of the reference's
// device methods:
//   cooperative_find          <- gpu_blink_tree::cooperative_find (include/gpu_blink_tree.hpp:277-303)
//                                gpu_versioned_btree::cooperative_find(key, tile, alloc, ts, ...)
//                                (include/gpu_versioned_blink_tree.hpp:438-474)
//   cooperative_insert        <- cooperative_insert_blink (include/gpu_blink_tree.hpp:522-733) and
//                                cooperative_insert_versioned_in_place
//                                (include/gpu_versioned_blink_tree.hpp:824-1086)
//   cooperative_erase         <- cooperative_erase (include/gpu_blink_tree.hpp:357-390,
//                                include/gpu_versioned_blink_tree.hpp:393-436)
//   cooperative_range_query   <- cooperative_range_query (include/gpu_blink_tree.hpp:306-355) and
//                                concurrent_cooperative_range_query
//                                (include/gpu_versioned_blink_tree.hpp:504-559)
//   take_snapshot             <- take_snapshot(tile) (include/gpu_versioned_blink_tree.hpp:332-344)
//
// Node format (128 bytes, 128-byte aligned, 32 words):
//   pairs 0..12  {key, value}  leaf: key/value, interior: {separator, child index}; sorted by key,
//                              unused pairs are {0xFFFFFFFF, 0xFFFFFFFF}
//   pair 13      {low fence, mod}     low fence = smallest key the node may hold (fixed for the
//                                     node's life); mod = bit31 lock | bits 0..30 modification
//                                     count, bumped by the release that follows a change
//   pair 14      {high key, link}     high key = exclusive upper fence (0xFFFFFFFF on the
//                                     rightmost node of a level); link = bits 0..27 right-sibling
//                                     index (0x0FFFFFFF = none)
//   pair 15      {ts, older|level}    ts = epoch of this version; bits 28..31 level (0 = leaf),
//                                     bits 0..27 index of the next older version (none = 0x0FFFFFFF)
// A tile of W threads (W = 8 or 16) holds one node in registers: lane l owns pairs
// [l*16/W, (l+1)*16/W), so an 8-lane tile reads a node as eight 16-byte vector loads and a
// 16-lane tile as sixteen 8-byte loads -- one 128-byte line either way.
//
// A node is read as several vector loads that are not one atomic access, so a node read while a
// writer stores it can mix two versions, even inside one lane. Every visit therefore checks
// low <= key (a mixed parent can route one child too far right; the visit then restarts from the
// anchor) and key < high (too far left: follow the right link), and a reader that uses the data of
// a leaf validates it (see recheck_version / read_leaf_latest).
//
// Concurrency protocol (B-link, Lehman-Yao style):
//   * readers never lock; a reader whose key is >= a node's high key follows the right link;
//   * a writer locks one leaf (atomicOr on the lock bit of the mod word, bounded spin with
//     __nanosleep backoff; the release that follows a change clears the bit and bumps the count
//     in one exchange, so the mod word is a sequence lock for readers of the newest state),
//     moves right under lock coupling, and applies its change; a full node splits into itself
//     and a new right sibling (right written first, then left, each followed by a fence), then
//     the writer releases the node and inserts the separator into the parent recorded on its
//     way down (moving right there as needed); node 0 is a fixed anchor whose single entry points
//     at the top of the tree, and the tree grows by building a new top node and re-pointing the
//     anchor, so no node ever changes its level or role (a reader that sees a mix of two
//     versions of a node still follows a valid route);
//   * versioning (versioned trees): a writer in epoch E that first touches a node whose ts < E
//     copies it to a fresh node O and publishes the header {ts = E, older = O} once O is complete,
//     and nodes created by splits in epoch E point to the same O. A reader at snapshot S follows
//     `older` while ts > S, so the version it uses is immutable; a reader under writers validates
//     the leaf it uses with its mod word and header read again after it (recheck_version).
//   * every wait is bounded; on a limit the operation gives up, records an error bit in the
//     control block and returns (no trap, no unbounded loop).
#pragma once

#include <cstdint>

#if defined(MVBT_HOST_EMULATION)
// Host build of this header for the CPU emulation harness (tests/emu): each W-lane tile runs as W
// host threads and the CUDA primitives below map to GCC atomics. The sm_100a build never sees
// this branch.
#include <atomic>
#include <chrono>
#include <cstring>
#include <thread>
#define MVBT_DEV inline
#define MVBT_COLD static inline
#define MVBT_OUTLINE inline
#define MVBT_CALL inline
struct uint2 {
  uint32_t x, y;
};
inline uint2 make_uint2(uint32_t x, uint32_t y) { return uint2{x, y}; }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline void __threadfence() { std::atomic_thread_fence(std::memory_order_seq_cst); }
inline void __threadfence_block() { std::atomic_thread_fence(std::memory_order_seq_cst); }
inline void __nanosleep(unsigned) { std::this_thread::yield(); }
template <class T, class U>
inline T atomicOr(T* p, U v) { return __atomic_fetch_or(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U>
inline T atomicAnd(T* p, U v) { return __atomic_fetch_and(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U>
inline T atomicAdd(T* p, U v) { return __atomic_fetch_add(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U>
inline T atomicExch(T* p, U v) { return __atomic_exchange_n(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U, class V>
inline T atomicCAS(T* p, U expected, V desired) {
  T e = (T)expected;
  __atomic_compare_exchange_n(p, &e, (T)desired, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST);
  return e;
}
template <class T, class U>
inline T atomicMin(T* p, U v) {
  T cur = __atomic_load_n(p, __ATOMIC_RELAXED);
  while (cur > (T)v && !__atomic_compare_exchange_n(p, &cur, (T)v, false, __ATOMIC_SEQ_CST, __ATOMIC_RELAXED)) {}
  return cur;
}
template <class T, class U>
inline T atomicMax(T* p, U v) {
  T cur = __atomic_load_n(p, __ATOMIC_RELAXED);
  while (cur < (T)v && !__atomic_compare_exchange_n(p, &cur, (T)v, false, __ATOMIC_SEQ_CST, __ATOMIC_RELAXED)) {}
  return cur;
}
namespace mvbt {
namespace emu {
inline thread_local uint32_t sm = 0;  // emulated SM id of the calling lane
inline std::atomic<uint32_t> slow{1};      // global_ns runs this much slower than the host's clock
}
}  // namespace mvbt
#else
#include <cooperative_groups.h>
#ifndef MVBT_DEV
#define MVBT_DEV __device__ __forceinline__
#endif
// Rarely taken paths (chunk refills, the retire log). Inlined: an out-of-line call raises the
// register count of the persistent kernels past the three-blocks-per-SM limit.
#ifndef MVBT_COLD
#define MVBT_COLD __device__ __forceinline__
#endif
// The separator push of a split (taken by a minority of writes). Inlined by default, as the
// persistent kernels need; a translation unit whose kernels are not register-bound defines it as
// __device__ __noinline__ so that one copy of that code is shared by every call site and the hot
// loop of a write stays small in the instruction cache.
#ifndef MVBT_OUTLINE
#define MVBT_OUTLINE __device__ __forceinline__
#endif
// A called function: the rare path of a warp's writes, kept out of its loop's code and registers.
#define MVBT_CALL __device__ __noinline__
#endif

namespace mvbt {
#if !defined(MVBT_HOST_EMULATION)
namespace cg = cooperative_groups;
#endif

// ----------------------------------------------------------------------------------------------
// Constants
// ----------------------------------------------------------------------------------------------
constexpr int kNodeWords      = 32;
constexpr int kDataPairs      = 13;
constexpr int kSplitLeft      = 7;  // a full node plus one entry (14) splits 7 | 7
constexpr uint32_t kEmptyKey  = 0xFFFFFFFFu;
constexpr uint32_t kNotFound  = 0xFFFFFFFFu;
constexpr uint32_t kLatest    = 0xFFFFFFFFu;  // read the newest version
constexpr uint32_t kNone      = 0x0FFFFFFFu;  // "no node" in 28-bit index fields
constexpr uint32_t kIndexMask = 0x0FFFFFFFu;
// Mod word (node word 27): bit 31 lock; bits 0..28 modification count of a live node. A version
// copy is never locked or changed again, so its mod word records instead that it is retired and
// the epoch E it was made in (it is read only at snapshots below E); a node that reclamation
// freed carries kFreeBit until it is reused.
constexpr uint32_t kLockBit    = 0x80000000u;
constexpr uint32_t kRetiredBit = 0x40000000u;
constexpr uint32_t kFreeBit    = 0x20000000u;
constexpr uint32_t kCountMask  = 0x1FFFFFFFu;  // count (live node) or epoch (retired copy)
constexpr int kModWord         = 27;
constexpr uint32_t kRingChunk  = 0x80000000u;  // per-SM chunk base: positions in the free ring
constexpr uint32_t kRingEmpty  = 0xFFFFFFFFu;  // a free-ring slot not written yet (or read already)
constexpr uint32_t kReclaimClaim = 64;        // log positions a warp reclaims at once inside a launch
constexpr uint32_t kReclaimAll = 0xFFFFFFFFu;  // reclaim watermark: the current epoch
constexpr uint32_t kAnchor    = 0;  // fixed entry node: one entry {0 -> top}, level = top + 1
constexpr uint32_t kFirstLeaf = 1;  // the initial leaf (holds the tombstone {0, 0})
constexpr int kMaxLevels      = 16;
constexpr int kMaxSmSlots     = 256;
constexpr uint32_t kMaxSteps  = 1u << 16;  // node visits per operation before giving up
constexpr uint32_t kCoupledHops  = 4;       // right moves taken while holding a lock
constexpr uint32_t kChaseRestart = 16;      // unlocked right moves before restarting at the anchor

// Sticky error bits in control_block::error.
enum : uint32_t {
  kErrPoolExhausted = 1u,
  kErrSpinLimit     = 2u,
  kErrCorrupt       = 4u,
  kErrStepLimit     = 8u,
};

// Device-resident tree state (one per tree).
struct control_block {
  uint32_t epoch;       // current write epoch == id the next take_snapshot returns
  uint32_t error;       // sticky error bits
  uint32_t bump;        // first never-allocated node index
  uint32_t capacity;    // pool capacity in nodes
  uint32_t chunk;       // nodes per per-SM allocation chunk
  uint32_t spin_limit;  // lock / wait attempts before giving up
  uint32_t wait_ns;     // wall-clock limit of one bounded wait (ns)
  uint32_t reserved;
  unsigned long long stat_cow;    // copy-on-write versions created
  unsigned long long stat_split;  // node splits
  unsigned long long stat_max_hops;   // longest move-right walk under locks
  unsigned long long stat_max_steps;  // longest unlocked descent of a writer (node visits)
  unsigned long long stat_restarts;   // locked approaches abandoned for an unlocked re-approach
  uint32_t err_site[32];              // errors per raising site (diagnostics; 16 = the
                                      // offsets check of mvbt_batch_run_noalloc, 17 = a
                                      // bulk load that did not fit the pool, 18 / 19 = a free-ring
                                      // slot that stayed empty / unread)
  unsigned long long sm_pool[kMaxSmSlots];  // per-SM chunk cursor: (base << 32) | used
  // Reclamation of version copies (off when reclaim_cap == 0). The retire log holds the index of
  // every copy not yet reclaimed, in the order the copies were made (which is epoch order); the
  // free ring the nodes reclamation freed. Allocation refills a per-SM chunk from the free ring
  // before the bump pointer. Both run while kernels run: a copy reserves a log position
  // (retire_tail) and writes it; a reclaimer claims log positions below a limit it knows to be
  // safe (retire_head), frees the copies, reserves ring positions (free_tail), writes them and
  // then counts them in free_avail; an allocation takes free_avail first, then ring positions
  // (free_head), waits for each slot to be written and clears it again (kRingEmpty) as it reads it.
  unsigned long long retire_log;   // device address of uint32_t[reclaim_cap]
  unsigned long long free_ring;    // device address of uint32_t[ring_cap]
  unsigned long long retire_head, retire_tail;  // log positions (monotonic; slot = pos % cap)
  unsigned long long free_head, free_tail;      // ring positions (monotonic; slot = pos % cap)
  unsigned long long free_avail;                // ring entries written and not yet taken (signed)
  uint32_t reclaim_cap;     // retire log entries: a power of two >= pool capacity
  uint32_t rc_first_kept;   // first log entry (relative to retire_head) a pass had to keep
  uint32_t ring_cap;        // free ring slots: a power of two >= capacity + kMaxSmSlots * chunk
  uint32_t reserved2;
  unsigned long long stat_reclaimed;    // nodes freed (passes between kernels and reclamation in them)
  unsigned long long stat_log_dropped;  // copies not logged because the log was full (never freed)
  // Per-SM shares of counters, one 128-B line per SM slot ([slot][0] copies, [slot][1] splits,
  // [slot][2] freed nodes handed out again): the counting atomics of different SMs land on
  // different lines instead of all on one word. stat_cow / stat_split stay 0; a count is its
  // slots' sum (stat_total).
  unsigned long long sm_stats[kMaxSmSlots][16];
};


#if defined(MVBT_HOST_EMULATION)
#define MVBT_HD inline
#else
#define MVBT_HD __host__ __device__ __forceinline__
#endif

// Total of per-SM counter k (0 copies, 1 splits, 2 freed nodes reused) plus the unsharded field.
MVBT_HD unsigned long long stat_total(const control_block& c, int k) {
  unsigned long long s = k == 0 ? c.stat_cow : (k == 1 ? c.stat_split : 0ull);
  for (int i = 0; i < kMaxSmSlots; ++i) s += c.sm_stats[i][k];
  return s;
}

// Word t (0..63) of the initial tree. Node 0 is the anchor: an interior node whose only entry
// {0 -> 1} points at the top of the tree, level 1. Node 1 is a leaf holding the tombstone {0, 0}.
// Both have high key 0xFFFFFFFF, no sibling, ts 0 and no older version. The anchor's single
// entry is the only pointer that changes when the tree grows, and no node ever changes level, so
// a reader that sees a mix of two versions of any node still finds a valid route.
MVBT_HD uint32_t initial_tree_word(int t) {
  const int node = t >> 5, w = t & 31;
  if (w == 26 || w == 27) return 0u;                 // low fence 0, modification count 0
  if (w < 26) {
    if (w == 0) return 0u;                           // first key: 0
    if (w == 1) return node == 0 ? kFirstLeaf : 0u;  // anchor -> leaf 1; tombstone value 0
    return kEmptyKey;
  }
  if (w == 28) return kEmptyKey;                     // high key
  if (w == 29) return kNone;                         // link
  if (w == 30) return 0u;                            // ts
  return (node == 0 ? (1u << 28) : 0u) | kNone;      // level | no older version
}
constexpr int kInitialNodes = 2;

// retire_log / free_ring: device addresses of uint32_t[reclaim_cap] and uint32_t[ring_cap]
// (powers of two), or 0 with reclaim_cap 0 (reclamation off).
MVBT_HD void init_control(control_block& c, uint32_t capacity, uint32_t chunk, uint32_t spin_limit,
                          uint32_t wait_ns, unsigned long long retire_log = 0,
                          unsigned long long free_ring = 0, uint32_t reclaim_cap = 0,
                          uint32_t ring_cap = 0) {
  c.epoch         = 0;
  c.error         = 0;
  c.bump          = kInitialNodes;  // nodes 0 (anchor) and 1 (first leaf)
  c.capacity      = capacity;
  c.chunk         = chunk;
  c.spin_limit    = spin_limit;
  c.wait_ns       = wait_ns;
  c.reserved      = 0;
  c.stat_cow      = 0;
  c.stat_split    = 0;
  c.stat_max_hops  = 0;
  c.stat_restarts  = 0;
  c.stat_max_steps = 0;
  for (int i = 0; i < 32; ++i) c.err_site[i] = 0;
  // used == chunk: the first allocation on each SM refills its chunk from the bump pointer
  for (int i = 0; i < kMaxSmSlots; ++i) c.sm_pool[i] = chunk;
  for (int i = 0; i < kMaxSmSlots; ++i)
    for (int j = 0; j < 16; ++j) c.sm_stats[i][j] = 0;
  c.retire_log       = retire_log;
  c.free_ring        = free_ring;
  c.retire_head      = 0;
  c.retire_tail      = 0;
  c.free_head        = 0;
  c.free_tail        = 0;
  c.free_avail       = 0;
  c.reclaim_cap      = reclaim_cap;
  c.rc_first_kept    = 0xFFFFFFFFu;
  c.ring_cap         = ring_cap;
  c.reserved2        = 0;
  c.stat_reclaimed   = 0;
  c.stat_log_dropped = 0;
}

// ----------------------------------------------------------------------------------------------
// Low-level memory access
// ----------------------------------------------------------------------------------------------
template <int W>
struct node_regs {
  static constexpr int P = 16 / W;  // pairs per lane
  uint32_t k[P];
  uint32_t v[P];
};

#if defined(MVBT_HOST_EMULATION)
MVBT_DEV uint32_t sm_id() { return emu::sm; }
template <class Tile>
MVBT_DEV uint32_t tile_ordinal(const Tile&) { return emu::sm; }
MVBT_DEV unsigned long long global_ns() {
  return (unsigned long long)std::chrono::duration_cast<std::chrono::nanoseconds>(
             std::chrono::steady_clock::now().time_since_epoch())
      .count() / emu::slow.load(std::memory_order_relaxed);
}
MVBT_DEV uint32_t ld_relaxed_u32(const uint32_t* p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
MVBT_DEV uint32_t ld_acquire_u32(const uint32_t* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }
MVBT_DEV uint32_t ld_block_u32(const uint32_t* p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
MVBT_DEV void st_relaxed_u32(uint32_t* p, uint32_t v) { __atomic_store_n(p, v, __ATOMIC_RELAXED); }
MVBT_DEV unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  return __atomic_load_n(p, __ATOMIC_RELAXED);
}
template <int W>
MVBT_DEV void ld_lane(const uint32_t* p, node_regs<W>& n, bool) {
  for (int j = 0; j < 16 / W; ++j) {
    n.k[j] = __atomic_load_n(p + 2 * j, __ATOMIC_RELAXED);
    n.v[j] = __atomic_load_n(p + 2 * j + 1, __ATOMIC_RELAXED);
  }
}
template <int W>
MVBT_DEV void st_lane(uint32_t* p, const node_regs<W>& n) {
  for (int j = 0; j < 16 / W; ++j) {
    __atomic_store_n(p + 2 * j, n.k[j], __ATOMIC_RELAXED);
    __atomic_store_n(p + 2 * j + 1, n.v[j], __ATOMIC_RELAXED);
  }
}
template <bool kStrong>
MVBT_DEV void copy_16(uint32_t* dst, const uint32_t* src) {
  for (int j = 0; j < 4; ++j) dst[j] = __atomic_load_n(src + j, __ATOMIC_RELAXED);
}
MVBT_DEV void copy_wait() {}
MVBT_DEV void store_16(uint32_t* dst, const uint32_t (&w)[4]) {
  for (int j = 0; j < 4; ++j) __atomic_store_n(dst + j, w[j], __ATOMIC_RELAXED);
}
#else
// Ordinal of the calling tile among the tiles of the launch.
template <class Tile>
MVBT_DEV uint32_t tile_ordinal(const Tile& t) {
  return (blockIdx.x * blockDim.x + threadIdx.x) / t.num_threads();
}
MVBT_DEV uint32_t sm_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}

MVBT_DEV unsigned long long global_ns() {
  unsigned long long r;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(r));
  return r;
}

MVBT_DEV uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t r;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(r) : "l"(p) : "memory");
  return r;
}
MVBT_DEV unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long r;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(r) : "l"(p) : "memory");
  return r;
}
// An acquire load: what this thread does next comes after the writes that the read value stands for.
MVBT_DEV uint32_t ld_acquire_u32(const uint32_t* p) {
  uint32_t r;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(r) : "l"(p) : "memory");
  return r;
}
// A word of shared memory that other warps of the block change.
MVBT_DEV uint32_t ld_block_u32(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
MVBT_DEV void st_relaxed_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" : : "l"(p), "r"(v) : "memory");
}

// Loads this lane's share of a node. strong = L2-coherent relaxed loads (needed while writers
// may run in the same kernel); otherwise read-only cached loads.
template <int W>
MVBT_DEV void ld_lane(const uint32_t* p, node_regs<W>& n, bool strong) {
  if constexpr (W == 8) {
    if (strong) {
      asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(n.k[0]), "=r"(n.v[0]), "=r"(n.k[1]), "=r"(n.v[1])
                   : "l"(p)
                   : "memory");
    } else {
      asm("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
          : "=r"(n.k[0]), "=r"(n.v[0]), "=r"(n.k[1]), "=r"(n.v[1])
          : "l"(p));
    }
  } else {
    if (strong) {
      asm volatile("ld.relaxed.gpu.global.v2.u32 {%0,%1}, [%2];"
                   : "=r"(n.k[0]), "=r"(n.v[0])
                   : "l"(p)
                   : "memory");
    } else {
      asm("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(n.k[0]), "=r"(n.v[0]) : "l"(p));
    }
  }
}

template <int W>
MVBT_DEV void st_lane(uint32_t* p, const node_regs<W>& n) {
  if constexpr (W == 8) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};"
                 :
                 : "l"(p), "r"(n.k[0]), "r"(n.v[0]), "r"(n.k[1]), "r"(n.v[1])
                 : "memory");
  } else {
    asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1,%2};"
                 :
                 : "l"(p), "r"(n.k[0]), "r"(n.v[0])
                 : "memory");
  }
}

// Asynchronous copy of 16 bytes from global to shared memory (both 16-byte aligned), and the wait
// for this thread's copies. kStrong: read at L2 (writers may run in the same kernel).
template <bool kStrong>
MVBT_DEV void copy_16(uint32_t* dst, const uint32_t* src) {
  if constexpr (kStrong)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :
                 : "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;"
                 :
                 : "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
MVBT_DEV void copy_wait() { asm volatile("cp.async.wait_all;" : : : "memory"); }
MVBT_DEV void store_16(uint32_t* dst, const uint32_t (&w)[4]) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};"
               :
               : "l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
               : "memory");
}

#endif  // MVBT_HOST_EMULATION

// ----------------------------------------------------------------------------------------------
// Register-resident node helpers (all are tile-collective: every lane must call them)
// ----------------------------------------------------------------------------------------------
template <int W>
struct layout {
  static constexpr int P          = 16 / W;
  static constexpr int kFenceLane = 13 / P;  // lane owning pair 13 {low, mod}
  static constexpr int kFenceSlot = 13 % P;
  static constexpr int kLinkLane  = 14 / P;  // lane owning pair 14 {high, link}
  static constexpr int kLinkSlot  = 14 % P;
  static constexpr int kVerLane   = 15 / P;  // lane owning pair 15 {ts, older|level}
  static constexpr int kVerSlot   = 15 % P;
};

struct header {
  uint32_t high;
  uint32_t link;
  uint32_t ts;
  uint32_t ol;   // older | level << 28
  uint32_t low;  // low fence: every key of the node is >= low (fixed for the life of the node)
  uint32_t mod;  // modification count, published before every change of the node
  MVBT_DEV uint32_t level() const { return ol >> 28; }
  MVBT_DEV uint32_t older() const { return ol & kIndexMask; }
  MVBT_DEV uint32_t sibling() const { return link & kIndexMask; }
  MVBT_DEV bool is_leaf() const { return level() == 0; }
};

// Every lane loads the header words (26..31) of the node at p itself: read-only cached loads, for
// readers that run with no writer in flight. They read the 128-byte line the lane's own share
// comes from, so they cost two L1 accesses where get_header costs six shuffles.
#if defined(MVBT_HOST_EMULATION)
MVBT_DEV header ld_header_words(const uint32_t* p) {
  header h;
  h.low  = __atomic_load_n(p + 26, __ATOMIC_RELAXED);
  h.mod  = __atomic_load_n(p + 27, __ATOMIC_RELAXED);
  h.high = __atomic_load_n(p + 28, __ATOMIC_RELAXED);
  h.link = __atomic_load_n(p + 29, __ATOMIC_RELAXED);
  h.ts   = __atomic_load_n(p + 30, __ATOMIC_RELAXED);
  h.ol   = __atomic_load_n(p + 31, __ATOMIC_RELAXED);
  return h;
}
#else
MVBT_DEV header ld_header_words(const uint32_t* p) {
  header h;
  asm("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(h.low), "=r"(h.mod) : "l"(p + 26));
  asm("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
      : "=r"(h.high), "=r"(h.link), "=r"(h.ts), "=r"(h.ol)
      : "l"(p + 28));
  return h;
}
#endif

MVBT_DEV header make_header(uint32_t low, uint32_t mod, uint32_t high, uint32_t link, uint32_t ts,
                            uint32_t ol) {
  header h;
  h.low  = low;
  h.mod  = mod;
  h.high = high;
  h.link = link;
  h.ts   = ts;
  h.ol   = ol;
  return h;
}

template <int W, class Tile>
MVBT_DEV header get_header(const node_regs<W>& n, const Tile& t) {
  using L = layout<W>;
  header h;
  h.low  = t.shfl(n.k[L::kFenceSlot], L::kFenceLane);
  h.mod  = t.shfl(n.v[L::kFenceSlot], L::kFenceLane);
  h.high = t.shfl(n.k[L::kLinkSlot], L::kLinkLane);
  h.link = t.shfl(n.v[L::kLinkSlot], L::kLinkLane);
  h.ts   = t.shfl(n.k[L::kVerSlot], L::kVerLane);
  h.ol   = t.shfl(n.v[L::kVerSlot], L::kVerLane);
  return h;
}

template <int W, class Tile>
MVBT_DEV void set_header(node_regs<W>& n, const header& h, const Tile& t) {
  using L      = layout<W>;
  const int r  = t.thread_rank();
  if (r == L::kFenceLane) {
    n.k[L::kFenceSlot] = h.low;
    n.v[L::kFenceSlot] = h.mod;
  }
  if (r == L::kLinkLane) {
    n.k[L::kLinkSlot] = h.high;
    n.v[L::kLinkSlot] = h.link;
  }
  if (r == L::kVerLane) {
    n.k[L::kVerSlot] = h.ts;
    n.v[L::kVerSlot] = h.ol;
  }
}

// Pair index of slot j in this lane.
template <int W, class Tile>
MVBT_DEV int pair_index(const Tile& t, int j) {
  return t.thread_rank() * (16 / W) + j;
}

// Number of valid data pairs.
template <int W, class Tile>
MVBT_DEV int count_valid(const node_regs<W>& n, const Tile& t) {
  int c = 0;
#pragma unroll
  for (int j = 0; j < 16 / W; ++j) {
    bool valid = pair_index<W>(t, j) < kDataPairs && n.k[j] != kEmptyKey;
    c += __popc(t.ballot(valid));
  }
  return c;
}

// Number of valid data pairs whose key is < key (= insertion position).
template <int W, class Tile>
MVBT_DEV int count_less(const node_regs<W>& n, uint32_t key, const Tile& t) {
  int c = 0;
#pragma unroll
  for (int j = 0; j < 16 / W; ++j) {
    bool less = pair_index<W>(t, j) < kDataPairs && n.k[j] != kEmptyKey && n.k[j] < key;
    c += __popc(t.ballot(less));
  }
  return c;
}

// Interior search: child of the last pair whose separator is <= key. Returns kNone if no
// separator is <= key (only possible on a corrupt route).
template <int W, class Tile>
MVBT_DEV uint32_t child_for(const node_regs<W>& n, uint32_t key, const Tile& t) {
  constexpr int P = 16 / W;
  int cnt         = 0;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    bool le = pair_index<W>(t, j) < kDataPairs && n.k[j] != kEmptyKey && n.k[j] <= key;
    cnt += le ? 1 : 0;
  }
  uint32_t mask = t.ballot(cnt > 0);
  uint32_t cand = n.v[0];
  if constexpr (P == 2) cand = (cnt == 2) ? n.v[1] : n.v[0];
  int src        = mask ? (31 - __clz(mask)) : 0;
  uint32_t child = t.shfl(cand, src);
  return mask ? child : kNone;
}

// Leaf search: value stored for key, or kNotFound.
template <int W, class Tile>
MVBT_DEV uint32_t leaf_value(const node_regs<W>& n, uint32_t key, const Tile& t) {
  constexpr int P = 16 / W;
  bool hit        = false;
  uint32_t val    = kNotFound;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    if (pair_index<W>(t, j) < kDataPairs && n.k[j] == key) {
      hit = true;
      val = n.v[j];
    }
  }
  uint32_t mask = t.ballot(hit);
  uint32_t r    = t.shfl(val, mask ? (__ffs(mask) - 1) : 0);
  return (mask && key != kEmptyKey) ? r : kNotFound;
}

// Range-query step on one leaf: writes the pairs of n with lo <= key < hi ascending at
// out[count...] (those below cap; out nullable) and returns how many there are. Collective.
template <int W, class Tile>
MVBT_DEV uint32_t leaf_collect(const node_regs<W>& n, uint32_t lo, uint32_t hi, uint2* out, uint32_t cap,
                               uint32_t count, const Tile& t) {
  constexpr int P = 16 / W;
  int first = -1, inr = 0;
  bool in[P];
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int q = pair_index<W>(t, j);
    in[j]       = q < kDataPairs && n.k[j] != kEmptyKey && n.k[j] >= lo && n.k[j] < hi;
    const uint32_t m = t.ballot(in[j]);
    inr += __popc(m);
    if (m) {
      const int f = (__ffs(m) - 1) * P + j;
      first       = (first < 0 || f < first) ? f : first;
    }
  }
  if (out != nullptr) {
#pragma unroll
    for (int j = 0; j < P; ++j) {
      if (in[j]) {
        const uint32_t o = count + (uint32_t)(pair_index<W>(t, j) - first);
        if (o < cap) out[o] = make_uint2(n.k[j], n.v[j]);
      }
    }
  }
  return (uint32_t)inr;
}

// Fetches pair `src` (per-lane index, 0..15) of node n. Collective.
template <int W, class Tile>
MVBT_DEV void fetch_pair(const node_regs<W>& n, int src, uint32_t& k, uint32_t& v, const Tile& t) {
  constexpr int P = 16 / W;
  src             = src < 0 ? 0 : (src > 15 ? 15 : src);
  if constexpr (P == 1) {
    k = t.shfl(n.k[0], src);
    v = t.shfl(n.v[0], src);
  } else {
    int lane    = src >> 1;
    uint32_t k0 = t.shfl(n.k[0], lane), k1 = t.shfl(n.k[1], lane);
    uint32_t v0 = t.shfl(n.v[0], lane), v1 = t.shfl(n.v[1], lane);
    k           = (src & 1) ? k1 : k0;
    v           = (src & 1) ? v1 : v0;
  }
}

// Data pairs of the merged sequence "n's valid pairs with {key, val} inserted at pos":
// entry e < pos -> old e, e == pos -> new, e > pos -> old e - 1. Entries past `total` are empty.
// Output pair q of `out` takes merged entry q + first (q < take), else empty. Header pairs of
// `out` are copied from n.
template <int W, class Tile>
MVBT_DEV void build_from_merged(const node_regs<W>& n,
                                int pos,
                                uint32_t key,
                                uint32_t val,
                                int first,
                                int take,
                                node_regs<W>& out,
                                const Tile& t) {
  constexpr int P = 16 / W;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int q = pair_index<W>(t, j);
    const int e = q + first;
    int src     = (e < pos) ? e : e - 1;
    uint32_t fk, fv;
    fetch_pair<W>(n, src, fk, fv, t);
    if (q >= kDataPairs) {
      out.k[j] = n.k[j];
      out.v[j] = n.v[j];
    } else if (q >= take) {
      out.k[j] = kEmptyKey;
      out.v[j] = kEmptyKey;
    } else if (e == pos) {
      out.k[j] = key;
      out.v[j] = val;
    } else {
      out.k[j] = fk;
      out.v[j] = fv;
    }
  }
}

// Removes data pair pos (shifting the rest down).
template <int W, class Tile>
MVBT_DEV void remove_at(node_regs<W>& n, int pos, const Tile& t) {
  constexpr int P = 16 / W;
  node_regs<W> out;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int q = pair_index<W>(t, j);
    int src     = (q < pos) ? q : q + 1;
    uint32_t fk, fv;
    fetch_pair<W>(n, src, fk, fv, t);
    if (q >= kDataPairs) {
      out.k[j] = n.k[j];
      out.v[j] = n.v[j];
    } else if (src >= kDataPairs) {
      out.k[j] = kEmptyKey;
      out.v[j] = kEmptyKey;
    } else {
      out.k[j] = fk;
      out.v[j] = fv;
    }
  }
  n = out;
}

// Pair index of the data pair holding key, or -1.
template <int W, class Tile>
MVBT_DEV int find_pos(const node_regs<W>& n, uint32_t key, const Tile& t) {
  constexpr int P = 16 / W;
  int pos         = -1;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    uint32_t mask = t.ballot(pair_index<W>(t, j) < kDataPairs && n.k[j] == key);
    int p         = mask ? (__ffs(mask) - 1) * P + j : -1;
    pos           = (pos < 0) ? p : ((p >= 0 && p < pos) ? p : pos);
  }
  return key == kEmptyKey ? -1 : pos;
}

// ----------------------------------------------------------------------------------------------
// The tree view: a plain struct passed to kernels by value.
// ----------------------------------------------------------------------------------------------
// ---- allocation and retirement slow paths (free functions: no copy of the tree view) ----
// Whether the bounded wait that started at t0 (lane 0's clock) has run past `limit` ns, decided by
// lane 0 for the whole tile or warp. Every lane of a group that runs warp-synchronous operations
// inside a wait loop must leave the loop together: a lane that left alone would make the next
// shuffle or ballot of the others name a lane that no longer takes part.
template <class Group>
MVBT_DEV bool wait_expired(unsigned long long t0, unsigned long long limit, const Group& g) {
  uint32_t late = 0;
  if (g.thread_rank() == 0) late = global_ns() - t0 > limit ? 1u : 0u;
  return g.shfl(late, 0) != 0;
}

// Node `used` of the chunk that starts at `base`: consecutive nodes of the bump range, or the node
// stored at consecutive free-ring positions (kRingChunk set). A ring slot is read once: the reader
// waits (bounded) for its pusher to have written it and clears it (kRingEmpty) for the ring's next
// lap. Returns kNone (and records kErrSpinLimit) if the slot stays empty past the wait limit. The
// ring and the retire log start filled with kRingEmpty (all bits set).
MVBT_DEV uint32_t chunk_node(control_block* c, uint32_t base, uint32_t used) {
  if (!(base & kRingChunk)) return base + used;
  uint32_t* slot = reinterpret_cast<uint32_t*>(c->free_ring) +
                   (((unsigned long long)(base & ~kRingChunk) + used) & (c->ring_cap - 1u));
  uint32_t v                  = ld_relaxed_u32(slot);
  const unsigned long long t0 = v == kRingEmpty ? global_ns() : 0;
  while (v == kRingEmpty) {
    if (global_ns() - t0 > c->wait_ns) {
      atomicOr(&c->error, kErrSpinLimit);
      atomicAdd(&c->err_site[18], 1u);
      return kNone;
    }
    __nanosleep(64);
    v = ld_relaxed_u32(slot);
  }
  st_relaxed_u32(slot, kRingEmpty);
  atomicAdd(&c->sm_stats[sm_id() % kMaxSmSlots][2], 1ull);  // a freed node handed out again
  return v;
}
// Takes C free-ring entries for a chunk: one atomic on free_avail (undone if fewer are there),
// then one on the ring head for their positions. False: allocate from the bump pointer instead.
MVBT_DEV bool take_free_chunk(control_block* c, uint32_t C, uint32_t& base) {
  if ((long long)ld_relaxed_u64(&c->free_avail) < (long long)C) return false;
  const long long a = (long long)atomicAdd(&c->free_avail, (unsigned long long)(-(long long)C));
  if (a < (long long)C) {
    atomicAdd(&c->free_avail, (unsigned long long)C);
    return false;
  }
  const unsigned long long h = atomicAdd(&c->free_head, (unsigned long long)C);
  base                       = kRingChunk | (uint32_t)(h & (c->ring_cap - 1u));
  return true;
}
// Appends the nodes of the lanes with `freed` set to the free ring (warp-collective, every lane of
// `warp` calls it): one reservation per warp, the slots written (waiting, bounded, for a slot the
// ring's previous lap has not yet read), then one fence and the count published in free_avail.
// ring_cap >= capacity + kMaxSmSlots * chunk: the entries written and not yet read (free nodes,
// and the rest of per-SM chunks taken from the ring) never fill the ring, so a pusher meets a
// slot of the previous lap only while its reader is about to clear it -- or while it is the unread
// rest of the chunk of an SM that has stopped allocating, which flush_chunk returns in time.
// kCount: the nodes were freed just now (stat_reclaimed). Returns whether the push went past one of the
// positions, 16 to a lap, where the chunks are looked over (return_idle_chunks).
template <bool kCount = true, class Warp>
MVBT_DEV bool ring_push(control_block* c, bool freed, uint32_t node, const Warp& warp) {
  const uint32_t m = warp.ballot(freed);
  if (!m) return false;
  const uint32_t lane = warp.thread_rank();
  const int lead      = __ffs(m) - 1;
  unsigned long long base = 0;
  if ((int)lane == lead) base = atomicAdd(&c->free_tail, (unsigned long long)__popc(m));
  base = warp.shfl(base, lead);
  if (freed) {
    uint32_t* slot = reinterpret_cast<uint32_t*>(c->free_ring) +
                     ((base + __popc(m & ((1u << lane) - 1u))) & (c->ring_cap - 1u));
    const unsigned long long t0 = global_ns();
    while (ld_relaxed_u32(slot) != kRingEmpty) {
      if (global_ns() - t0 > c->wait_ns) {
        atomicOr(&c->error, kErrSpinLimit);
        atomicAdd(&c->err_site[19], 1u);
        break;
      }
      __nanosleep(64);
    }
    st_relaxed_u32(slot, node);
  }
  __threadfence();
  warp.sync();
  if ((int)lane == lead) {
    atomicAdd(&c->free_avail, (unsigned long long)__popc(m));
    if (kCount) atomicAdd(&c->stat_reclaimed, (unsigned long long)__popc(m));
  }
  const uint32_t pos = (uint32_t)base & (c->ring_cap - 1u), part = c->ring_cap / 16;
  return pos / part != (pos + (uint32_t)__popc(m)) / part;
}
// Returns the unread rest of SM slot `sm`'s chunk to the free ring if the chunk is a run of ring
// positions that lies `behind` or more positions behind the ring's tail (warp-collective). Without it
// an SM that took a chunk and then stopped allocating would keep its positions unread until the ring's
// tail comes round, and the pushers that meet them would wait out their limit.
// Returns what ring_push did.
template <class Warp>
MVBT_DEV bool flush_chunk(control_block* c, uint32_t sm, uint32_t behind, const Warp& warp) {
  unsigned long long* slot = &c->sm_pool[sm];
  const uint32_t C         = c->chunk;
  unsigned long long cur   = 0;
  uint32_t take            = 0;
  if (warp.thread_rank() == 0) {
    cur                 = ld_relaxed_u64(slot);
    const uint32_t base = (uint32_t)(cur >> 32), used = (uint32_t)cur;
    const uint32_t lag  = ((uint32_t)ld_relaxed_u64(&c->free_tail) - (base & ~kRingChunk)) & (c->ring_cap - 1u);
    // used up without taking the refill on: the next request refills it
    if ((base & kRingChunk) && used < C && lag >= behind &&
        atomicCAS(slot, cur, (cur & 0xFFFFFFFF00000000ull) | C) == cur)
      take = C - used;
  }
  take = warp.shfl(take, 0);
  if (take == 0) return false;
  cur = warp.shfl(cur, 0);
  const uint32_t base = (uint32_t)(cur >> 32), used = (uint32_t)cur;
  bool past           = false;
  for (uint32_t j = 0; j < take; j += 32) {  // read (and clear) before pushing: no pusher waits for this warp
    const uint32_t at = j + warp.thread_rank();
    uint32_t node     = kNone;
    if (at < take) {
      node = chunk_node(c, base, used + at);
      atomicAdd(&c->sm_stats[sm_id() % kMaxSmSlots][2], (unsigned long long)-1ll);  // not handed out after all
    }
    past |= ring_push<false>(c, node != kNone, node, warp);
  }
  return past;
}
// flush_chunk of all SM slots: warp w looks at slots [32 w, 32 w + 32), a lane at each.
template <class Warp>
MVBT_DEV bool flush_chunks(control_block* c, uint32_t w, uint32_t behind, const Warp& warp) {
  if (w >= (uint32_t)kMaxSmSlots / 32) return false;
  bool past = false;
  const unsigned long long cur = ld_relaxed_u64(&c->sm_pool[32 * w + warp.thread_rank()]);
  const uint32_t base = (uint32_t)(cur >> 32);
  const uint32_t lag  = ((uint32_t)ld_relaxed_u64(&c->free_tail) - (base & ~kRingChunk)) & (c->ring_cap - 1u);
  for (uint32_t m = warp.ballot((base & kRingChunk) && (uint32_t)cur < c->chunk && lag >= behind); m; m &= m - 1u)
    past |= flush_chunk(c, 32 * w + (uint32_t)__ffs(m) - 1u, behind, warp);
  return past;
}
// After a push that went past one of the ring's 16 marks: returns the unread rests of all chunks half a lap
// behind. Whichever SMs run or stand still, a chunk goes back 7/16 of a lap before the tail comes round to it.
template <class Warp>
MVBT_CALL void return_idle_chunks(control_block* c, Warp warp) {
  for (bool past = true; past;) {  // the rests that it pushes may pass the next mark
    past = false;
    for (uint32_t w = 0; w < (uint32_t)kMaxSmSlots / 32; ++w) past |= flush_chunks(c, w, c->ring_cap / 2, warp);
  }
}
// Records a version copy in the retire log. A copy the full log cannot take is never freed
// (counted in stat_log_dropped).
MVBT_COLD void retire_logged(control_block* c, uint32_t copy) {
  const uint32_t cap           = c->reclaim_cap;
  const unsigned long long pos = atomicAdd(&c->retire_tail, 1ull);
  if (pos - ld_relaxed_u64(&c->retire_head) < cap)
    reinterpret_cast<uint32_t*>(c->retire_log)[pos & (cap - 1u)] = copy;
  else
    atomicAdd(&c->stat_log_dropped, 1ull);
}

// Path memory of a tile that runs ops in ascending key order (the sorted batch front-end): lane l
// remembers the node it last passed at level l and that node's fences [low, high). The next op
// starts at the lowest remembered node whose fences cover its key instead of at the anchor, so a
// run of nearby keys shares the upper levels and often the leaf. Any node whose low fence is <= the
// key is a valid start (low fences never change; a split that lowered the high fence since the
// node was read is repaired by the right-link chase), and a remembered version is the one a
// snapshot read resolved to, so its children route that snapshot. Levels >= W are not kept.
template <int W>
struct finger {
  uint32_t idx  = kNone;
  uint32_t low  = 0;
  uint32_t high = 0;
  // Lowest remembered node covering key, or the anchor.
  template <class Tile>
  MVBT_DEV uint32_t start_for(uint32_t key, const Tile& t) const {
    const uint32_t m = t.ballot(idx != kNone && low <= key && key < high);
    return m ? t.shfl(idx, __ffs(m) - 1) : kAnchor;
  }
  template <class Tile>
  MVBT_DEV void record(uint32_t level, uint32_t node, uint32_t lo, uint32_t hi, const Tile& t) {
    if (t.thread_rank() == (int)level) {
      idx  = node;
      low  = lo;
      high = hi;
    }
  }
};

struct device_tree {
  uint32_t* pool;       // node words; node i starts at pool + 32 * i
  control_block* ctl;   // device control block
  uint32_t versioned;   // 1 = multiversion tree, 0 = plain B-link tree
  uint32_t capacity;    // pool size in nodes: every index read from memory is checked against it
  uint32_t reclaim = 0; // 1: version copies go to the retire log (the tree was made with reclaim)

  MVBT_DEV uint32_t* node_ptr(uint32_t idx) const { return pool + (size_t)idx * kNodeWords; }
  // An index is dereferenced only after this check; a bad one records kErrCorrupt instead.
  template <class Tile>
  MVBT_DEV bool valid(uint32_t idx, const Tile& t) const {
    if (idx < capacity) return true;
    if (t.thread_rank() == 0) set_error(kErrCorrupt, 1);
    return false;
  }

  template <int W, class Tile>
  MVBT_DEV void load(uint32_t idx, node_regs<W>& n, bool strong, const Tile& t) const {
    ld_lane<W>(node_ptr(idx) + t.thread_rank() * (32 / W), n, strong);
  }
  template <int W, class Tile>
  MVBT_DEV void store(uint32_t idx, const node_regs<W>& n, const Tile& t) const {
    st_lane<W>(node_ptr(idx) + t.thread_rank() * (32 / W), n);
  }
  // Stores only the lanes that own header pairs.
  template <int W, class Tile>
  MVBT_DEV void store_header(uint32_t idx, const node_regs<W>& n, const Tile& t) const {
    using L     = layout<W>;
    const int r = t.thread_rank();
    if (r == L::kFenceLane || r == L::kLinkLane || r == L::kVerLane)
      st_lane<W>(node_ptr(idx) + r * (32 / W), n);
  }

  // Records error bits and counts the site that raised them (control_block::err_site).
  // Orders every lane's earlier stores before any lane's later ones. A fence orders only the
  // calling thread's own accesses; the warp barrier after it carries that order across the lanes
  // of the tile, so a store that publishes a node (a link, a header) is never visible before the
  // stores of other lanes that wrote what it points to.
  template <class Tile>
  MVBT_DEV void publish_fence(const Tile& t) const {
    __threadfence();
    t.sync();
  }

  MVBT_DEV void set_error(uint32_t bits, uint32_t site = 0) const {
    atomicOr(&ctl->error, bits);
    atomicAdd(&ctl->err_site[site & 31], 1u);
  }
  MVBT_DEV uint32_t current_epoch() const { return ld_relaxed_u32(&ctl->epoch); }

  // ---- allocation: per-SM chunks, refilled from the free ring or the global bump pointer ----
  // Returns a node index, or a free-ring position tagged kRingChunk that alloc() resolves.
  MVBT_DEV uint32_t alloc_one() const {
    control_block* c              = ctl;
    unsigned long long* slot      = &c->sm_pool[sm_id() % kMaxSmSlots];
    const uint32_t C              = c->chunk;
    const uint32_t limit          = c->spin_limit;
    const unsigned long long t0 = global_ns();
    for (uint32_t tries = 0; tries < limit; ++tries) {
      if (tries && (ld_relaxed_u32(&c->error) & kErrPoolExhausted)) return kNone;
      unsigned long long old = atomicAdd(slot, 1ull);
      uint32_t base = (uint32_t)(old >> 32), used = (uint32_t)old;
      if (used < C) return base + used;
      if (used == C) {  // this thread refills the chunk
        uint32_t rb = 0;
        if (reclaim && take_free_chunk(c, C, rb)) {
          atomicExch(slot, ((unsigned long long)rb << 32) | 1ull);
          return rb;
        }
        uint32_t nb = atomicAdd(&c->bump, C);
        if ((unsigned long long)nb + C > c->capacity) {
          atomicOr(&c->error, kErrPoolExhausted);
          atomicAdd(&c->err_site[15], 1u);
          return kNone;
        }
        atomicExch(slot, ((unsigned long long)nb << 32) | 1ull);
        return nb;
      }
      // another thread is refilling: wait (bounded) for the chunk base to change
      for (uint32_t w = 0; w < limit; ++w) {
        __nanosleep(64);
        unsigned long long cur = ld_relaxed_u64(slot);
        if ((uint32_t)(cur >> 32) != base || (uint32_t)cur < C) break;
        if (ld_relaxed_u32(&c->error) & kErrPoolExhausted) return kNone;
        if (global_ns() - t0 > c->wait_ns) break;
      }
      if (global_ns() - t0 > c->wait_ns) break;
    }
    atomicOr(&c->error, kErrSpinLimit);
    atomicAdd(&c->err_site[0], 1u);
    return kNone;
  }
  template <class Tile>
  MVBT_DEV uint32_t alloc(const Tile& t) const {
    uint32_t idx = kNone;
    if (t.thread_rank() == 0) {
      idx = alloc_one();
      // a position in the free ring (a chunk of reclaimed nodes): the node stored there, read
      // once (reading clears the slot), by this lane alone
      if (idx != kNone && (idx & kRingChunk)) idx = chunk_node(ctl, idx, 0);
    }
    return t.shfl(idx, 0);
  }

  // ---- locks on the mod word ----
  template <class Tile>
  MVBT_DEV bool lock(uint32_t idx, const Tile& t) const {
    if (!valid(idx, t)) return false;
    uint32_t* word               = node_ptr(idx) + kModWord;
    uint32_t backoff             = 32;
    const uint32_t lim           = ctl->spin_limit;
    const unsigned long long t0  = global_ns();
    const unsigned long long lns = ctl->wait_ns;
    for (uint32_t i = 0; i < lim; ++i) {
      uint32_t old = 0;
      if (t.thread_rank() == 0) old = atomicOr(word, kLockBit);
      old = t.shfl(old, 0);
      if (!(old & kLockBit)) {
        __threadfence();
        t.sync();
        return true;
      }
      // wait until the lock looks free before the next atomic
      for (uint32_t w = 0; w < 64; ++w) {
        __nanosleep(backoff);
        uint32_t cur = 0;
        if (t.thread_rank() == 0) cur = ld_relaxed_u32(word);
        cur = t.shfl(cur, 0);
        if (!(cur & kLockBit)) break;
        backoff = backoff < 1024 ? backoff * 2 : 1024;
      }
      if (wait_expired(t0, lns, t)) break;
    }
    if (t.thread_rank() == 0) set_error(kErrSpinLimit, 2);
    return false;
  }
  // Releases a node this tile locked and left unchanged (the count stays).
  template <class Tile>
  MVBT_DEV void unlock(uint32_t idx, const Tile& t) const {
    __threadfence();
    t.sync();
    if (t.thread_rank() == 0) atomicAnd(node_ptr(idx) + kModWord, ~kLockBit);
  }
  // Releases a node this tile locked and changed: after every lane's stores are ordered (fence +
  // warp barrier), one exchange clears the lock bit and bumps the count. h.mod is the mod word
  // read under the lock; while the lock is held only failing lock attempts (atomicOr of a bit
  // that is already set) touch the word, so the exchange loses nothing.
  template <class Tile>
  MVBT_DEV void release(uint32_t idx, const header& h, const Tile& t) const {
    __threadfence();
    t.sync();
    if (t.thread_rank() == 0)
      atomicExch(node_ptr(idx) + kModWord, ((h.mod & kCountMask) + 1u) & kCountMask);
  }

  // ---- versioning ----
  // Makes the version visible to older snapshots immutable before node idx (locked, content n)
  // is changed in epoch E. On a versioned tree the first change in epoch E copies the node to a
  // fresh node O and publishes {ts = E, older = O} before any data changes, so a snapshot reader
  // that re-reads ts after reading the data sees that it must use O. Readers of the newest state
  // need nothing here: the lock bit and the count bumped by release() cover them.
  template <int W, class Tile>
  MVBT_DEV bool prepare_write(uint32_t idx, node_regs<W>& n, header& h, uint32_t E, const Tile& t) const {
    if (versioned && h.ts != E) {
      uint32_t copy = alloc(t);
      if (copy == kNone) return false;
      node_regs<W> c = n;
      header hc      = h;
      hc.mod         = kRetiredBit | (E & kCountMask);  // immutable; read only at snapshots < E
      set_header<W>(c, hc, t);
      store<W>(copy, c, t);
      publish_fence(t);  // the copy is complete before the header names it
      h.ts = E;
      h.ol = (h.ol & ~kIndexMask) | copy;
      set_header<W>(n, h, t);
      store_header<W>(idx, n, t);
      // No fence between the header and the data change: a snapshot reader that saw data of this
      // change before the header finds the mod word changed (the lock preceded every store here)
      // and reads the leaf again (recheck_version); the release's fence publishes both.
      if (t.thread_rank() == 0) retire(copy);
    }
    return true;
  }

  // ---- reclamation of version copies ----
  // Records a version copy in the retire log (reclamation on), else counts it.
  MVBT_DEV void retire(uint32_t copy) const {
    if (reclaim)
      retire_logged(ctl, copy);
    else
      atomicAdd(&ctl->sm_stats[sm_id() % kMaxSmSlots][0], 1ull);
  }
  // One retire-log entry at position pos. A copy made in epoch E is read only at snapshots below
  // E, so with no live snapshot below the watermark M it is unreachable once E <= M (compared in a
  // window of 2^28 epochs). Returns 1 if the entry's copy is now marked free (the caller appends
  // idx to the free ring), 2 if it must be kept, 0 if the entry holds nothing (consumed, or a copy
  // the full log dropped). A consumed or freed entry's slot is cleared. check_epoch = false: the
  // caller knows the position holds a reclaimable copy (reclaim_online).
  MVBT_DEV int reclaim_entry(unsigned long long pos, uint32_t M, uint32_t& idx, bool check_epoch = true) const {
    control_block* c = ctl;
    uint32_t* slot   = reinterpret_cast<uint32_t*>(c->retire_log) + (pos & (c->reclaim_cap - 1u));
    idx              = ld_relaxed_u32(slot);
    if (idx >= capacity) return 0;
    uint32_t* mod    = node_ptr(idx) + kModWord;
    const uint32_t m = ld_relaxed_u32(mod);
    if (!(m & kRetiredBit)) {
      st_relaxed_u32(slot, kNone);
      return 0;
    }
    if (check_epoch && ((M - m) & kCountMask) > (kCountMask >> 1)) return 2;  // made after the watermark
    st_relaxed_u32(mod, kFreeBit);
    st_relaxed_u32(slot, kNone);
    return 1;
  }
  // End of a reclaim pass between kernels (one thread, after every entry): moves the log head
  // past the consumed entries, up to the first copy the pass had to keep. retire_tail stays the
  // count of every copy made. Positions beyond head + capacity were never written (those copies
  // were dropped); they alias slots this pass cleared, so a later pass passes over them.
  MVBT_DEV void reclaim_publish() const {
    control_block* c              = ctl;
    const unsigned long long head = c->retire_head;
    unsigned long long n          = c->retire_tail - head;
    if (n > c->reclaim_cap) n = c->reclaim_cap;
    const uint32_t keep = c->rc_first_kept;
    c->retire_head      = head + (keep == 0xFFFFFFFFu ? n : keep);
    c->rc_first_kept    = 0xFFFFFFFFu;
  }
  // Reclamation while kernels run (warp-collective): claims up to kReclaimClaim retire-log positions
  // below `limit` -- positions the caller knows hold only copies that no live snapshot reads -- frees
  // their copies and appends them to the free ring. Returns the number of positions claimed.
  template <class Warp>
  MVBT_DEV uint32_t reclaim_online(unsigned long long limit, const Warp& warp) const {
    control_block* c       = ctl;
    unsigned long long h   = 0;
    uint32_t n             = 0;
    if (warp.thread_rank() == 0) {
      h = ld_relaxed_u64(&c->retire_head);
      const unsigned long long tail = ld_relaxed_u64(&c->retire_tail);
      if (limit > tail) limit = tail;  // never past the entries reserved so far
      if (h < limit) {
        n = (uint32_t)(limit - h < kReclaimClaim ? limit - h : kReclaimClaim);
        if (atomicCAS(&c->retire_head, h, h + n) != h) n = 0;  // another warp took them
      }
    }
    h = warp.shfl(h, 0);
    n = warp.shfl(n, 0);
    if (n == 0) return 0;
    __threadfence();  // the copies' last readers finished before `limit` was published
    bool past = false;
    for (uint32_t j = 0; j < n; j += 32) {
      const uint32_t at = j + warp.thread_rank();
      uint32_t idx      = kNone;
      const bool freed  = at < n && reclaim_entry(h + at, 0, idx, false) == 1;
      past |= ring_push(c, freed, idx, warp);
    }
    if (past) return_idle_chunks(c, warp);
    return n;
  }

  // Moves from node idx to the version visible at ts (snapshot readers only). Sets `copy` when it
  // followed at least one older pointer: such a version is never written again.
  template <int W, class Tile>
  MVBT_DEV bool to_version(uint32_t& idx, node_regs<W>& n, header& h, uint32_t ts, bool strong,
                           bool& copy, const Tile& t) const {
    uint32_t hops = 0;
    while (h.ts > ts) {
      uint32_t older = h.older();
      if (older == kNone || ++hops > kMaxSteps) {
        if (t.thread_rank() == 0) set_error(kErrCorrupt, 3);
        return false;
      }
      idx = older;
      if (!valid(idx, t)) return false;
      load<W>(idx, n, strong, t);
      h    = get_header<W>(n, t);
      copy = true;
    }
    return true;
  }

  // Reads leaf idx for a reader of the newest state while writers may run: a sequence lock on
  // the mod word (lock bit | count). A writer holds the lock bit while it changes a reachable
  // leaf and clears it with a bumped count in one exchange after its stores, so the data is
  // consistent when the mod word is unlocked in a read ordered before the data (fence) and
  // unchanged in a re-read ordered after it (fence). Lock and count share one word on purpose:
  // two words read separately could show the state before a writer's lock in one and after its
  // change in the other. Each lane reads the word itself, so its own fences order it around its
  // own share of the node; the read counts only if it held in every lane. Bounded: gives up
  // after the wait limit (kErrSpinLimit) and returns false.
  template <int W, class Tile>
  MVBT_DEV bool read_leaf_latest(uint32_t idx, node_regs<W>& n, const Tile& t) const {
    const uint32_t* p             = node_ptr(idx);
    const unsigned long long t0   = global_ns();
    const unsigned long long lim  = ctl->wait_ns;
    uint32_t backoff              = 32;
    for (;;) {
      const uint32_t mod0 = ld_relaxed_u32(p + kModWord);
      __threadfence();
      ld_lane<W>(p + t.thread_rank() * (32 / W), n, true);
      __threadfence();
      const uint32_t mod1 = ld_relaxed_u32(p + kModWord);
      const bool torn     = (mod0 & kLockBit) != 0 || mod0 != mod1;
      if (t.ballot(torn) == 0) return true;
      if (wait_expired(t0, lim, t)) break;
      __nanosleep(backoff);
      backoff = backoff < 1024 ? backoff * 2 : 1024;
    }
    if (t.thread_rank() == 0) set_error(kErrSpinLimit, 2);
    return false;
  }

  // A concurrent snapshot reader that is about to use the data of a leaf version it read with
  // ts <= snapshot re-reads the leaf's mod word and header after a fence (mod0 = the mod word of
  // the read itself). Returns the immutable copy to read instead if the header now shows a version
  // newer than the snapshot (a writer publishes {ts = E, older = copy} only after the copy is
  // complete). Otherwise sets retry if the mod word was locked or has changed: a writer locked the
  // leaf before any of its stores, so data of a change the header does not show yet can only have
  // been read while the word differs. Returns kNone with retry false if the data read is the
  // version at ts: no writer changed the leaf since before the read, or one did and released it
  // before the mod word was read, whose release fence also published its header (then ts2 > ts).
  template <class Tile>
  MVBT_DEV uint32_t recheck_version(uint32_t idx, uint32_t ts, uint32_t mod0, bool& retry,
                                    const Tile& t) const {
    __threadfence();
    t.sync();
    unsigned long long v = 0;
    uint32_t mod1        = 0;
    if (t.thread_rank() == 0) {
      mod1 = ld_relaxed_u32(node_ptr(idx) + kModWord);
      v    = ld_relaxed_u64(reinterpret_cast<const unsigned long long*>(node_ptr(idx) + 30));
    }
    v            = t.shfl(v, 0);
    mod1         = t.shfl(mod1, 0);
    uint32_t ts2 = (uint32_t)v, ol2 = (uint32_t)(v >> 32);
    retry        = false;
    if (ts2 > ts) return ol2 & kIndexMask;
    retry = (mod0 & kLockBit) != 0 || mod1 != mod0;
    return kNone;
  }

  // ------------------------------------------------------------------------------------------
  // Point lookup at snapshot ts (kLatest = newest). concurrent = writers may run meanwhile.
  // ------------------------------------------------------------------------------------------
  // f (nullable): path memory of a sorted run; every node the lookup passes on key's route is
  // recorded in it (the version a snapshot read resolved to).
  template <int W, class Tile>
  MVBT_DEV uint32_t cooperative_find(uint32_t key, const Tile& t, uint32_t ts = kLatest,
                                     bool concurrent = false, uint32_t start = kAnchor,
                                     finger<W>* f = nullptr) const {
    const bool snap   = versioned && ts != kLatest;
    const bool seqlk  = !snap && concurrent;  // newest state under writers: read leaves locked-free
    uint32_t idx      = start;  // the anchor, or a node on key's route found earlier
    bool via_older    = false;  // idx was reached through an older-version pointer
    bool leaf_next    = false;  // idx is a leaf (child of a level-1 node, or a leaf's sibling)
    node_regs<W> n;
    for (uint32_t step = 0; step < kMaxSteps; ++step) {
      if (!valid(idx, t)) return kNotFound;
      const bool stable = seqlk && leaf_next;
      if (stable) {
        if (!read_leaf_latest<W>(idx, n, t)) return kNotFound;
      } else {
        load<W>(idx, n, concurrent, t);
      }
      header h  = get_header<W>(n, t);
      bool copy = via_older;
      via_older = false;
      if (snap && !to_version<W>(idx, n, h, ts, concurrent, copy, t)) return kNotFound;
      if (key < h.low) {  // routed too far right by a torn read upstream: start over
        idx       = kAnchor;
        leaf_next = false;
        continue;
      }
      if (key >= h.high && h.sibling() != kNone) {
        idx       = h.sibling();
        leaf_next = h.is_leaf();
        continue;
      }
      if (h.is_leaf()) {
        if (snap && concurrent && !copy) {
          bool retry     = false;
          uint32_t older = recheck_version(idx, ts, h.mod, retry, t);
          if (older != kNone) {  // changed under us: use the immutable copy instead
            idx       = older;
            via_older = true;
            continue;
          }
          if (retry) {  // a writer is changing it: read it again (bounded by the step limit)
            __nanosleep(64);
            continue;
          }
        } else if (seqlk && !stable) {
          leaf_next = true;  // reached without knowing it was a leaf: read it again, consistently
          continue;
        }
        if (f) f->record(0, idx, h.low, h.high, t);
        return leaf_value<W>(n, key, t);
      }
      if (f) f->record(h.level(), idx, h.low, h.high, t);
      leaf_next = h.level() == 1;
      idx       = child_for<W>(n, key, t);
      if (idx == kNone) {
        idx       = kAnchor;
        leaf_next = false;
      }
    }
    if (t.thread_rank() == 0) set_error(kErrStepLimit, 4);
    return kNotFound;
  }

  // The point lookup of a tree no writer changes meanwhile (concurrent = false): the same route
  // and result as cooperative_find(key, t, ts), but every lane loads the header
  // words itself (ld_header_words) beside its share of the node instead of receiving them by
  // shuffle, and the versions a snapshot read passes over are read as headers alone.
  template <int W, class Tile>
  MVBT_DEV uint32_t find_quiescent(uint32_t key, const Tile& t, uint32_t ts = kLatest) const {
    const bool snap = versioned && ts != kLatest;
    uint32_t idx    = kAnchor;
    node_regs<W> n;
    for (uint32_t step = 0; step < kMaxSteps; ++step) {
      if (!valid(idx, t)) return kNotFound;
      const header h = ld_header_words(node_ptr(idx));
      load<W>(idx, n, false, t);  // issued with the header loads: one round trip per visit
      if (snap && h.ts > ts) {  // a newer version: move to the older one
        idx = h.older();
        if (idx == kNone) {
          if (t.thread_rank() == 0) set_error(kErrCorrupt, 3);
          return kNotFound;
        }
        continue;
      }
      if (key < h.low) {
        idx = kAnchor;
        continue;
      }
      if (key >= h.high && h.sibling() != kNone) {
        idx = h.sibling();
        continue;
      }
      if (h.is_leaf()) {
        return leaf_value<W>(n, key, t);
      }
      idx = child_for<W>(n, key, t);
      if (idx == kNone) idx = kAnchor;
    }
    if (t.thread_rank() == 0) set_error(kErrStepLimit, 4);
    return kNotFound;
  }

  // ------------------------------------------------------------------------------------------
  // Range query [lo, hi) at snapshot ts. Writes at most cap pairs {key, value} ascending at out
  // (nullable) and returns the full count.
  // ------------------------------------------------------------------------------------------
  // f (nullable): path memory of a sorted run (as in cooperative_find), recorded along lo's route.
  template <int W, class Tile>
  MVBT_DEV uint32_t cooperative_range_query(uint32_t lo, uint32_t hi, const Tile& t, uint32_t ts,
                                            uint2* out, uint32_t cap, bool concurrent = false,
                                            uint32_t start = kAnchor, finger<W>* f = nullptr) const {
    if (hi <= lo) return 0;
    const bool snap  = versioned && ts != kLatest;
    const bool seqlk = !snap && concurrent;  // newest state under writers (read_leaf_latest)
    uint32_t idx     = start;  // the anchor, or a node on lo's route found earlier
    bool via_older   = false;
    bool leaf_next   = false;
    node_regs<W> n;
    header h;
    // descend to the leaf that holds lo and settle on a consistent version of it
    for (uint32_t step = 0;; ++step) {
      if (step >= kMaxSteps) {
        if (t.thread_rank() == 0) set_error(kErrStepLimit, 5);
        return 0;
      }
      if (!valid(idx, t)) return 0;
      const bool stable = seqlk && leaf_next;
      if (stable) {
        if (!read_leaf_latest<W>(idx, n, t)) return 0;
      } else {
        load<W>(idx, n, concurrent, t);
      }
      h         = get_header<W>(n, t);
      bool copy = via_older;
      via_older = false;
      if (snap && !to_version<W>(idx, n, h, ts, concurrent, copy, t)) return 0;
      if (lo < h.low) {
        idx       = kAnchor;
        leaf_next = false;
        continue;
      }
      if (lo >= h.high && h.sibling() != kNone) {
        idx       = h.sibling();
        leaf_next = h.is_leaf();
        continue;
      }
      if (h.is_leaf()) {
        if (snap && concurrent && !copy) {
          bool retry     = false;
          uint32_t older = recheck_version(idx, ts, h.mod, retry, t);
          if (older != kNone) {
            idx       = older;
            via_older = true;
            continue;
          }
          if (retry) {
            __nanosleep(64);
            continue;
          }
        } else if (seqlk && !stable) {
          leaf_next = true;
          continue;
        }
        if (f) f->record(0, idx, h.low, h.high, t);
        break;
      }
      if (f) f->record(h.level(), idx, h.low, h.high, t);
      leaf_next = h.level() == 1;
      idx       = child_for<W>(n, lo, t);
      if (idx == kNone) {
        idx       = kAnchor;
        leaf_next = false;
      }
    }
    // scan leaves to the right (a sibling chain is never longer than the pool)
    uint32_t count = 0;
    for (uint32_t leaves = 0;; ++leaves) {
      count += leaf_collect<W>(n, lo, hi, out, cap, count, t);
      if (!(hi > h.high && h.sibling() != kNone)) break;
      if (leaves >= capacity) {
        if (t.thread_rank() == 0) set_error(kErrStepLimit, 6);
        break;
      }
      // next leaf: load, resolve the snapshot version, validate before its data is used
      idx           = h.sibling();
      bool settled  = false;
      for (uint32_t tries = 0; tries < kMaxSteps && !settled; ++tries) {
        if (!valid(idx, t)) return count;
        if (seqlk) {
          if (!read_leaf_latest<W>(idx, n, t)) return count;
        } else {
          load<W>(idx, n, concurrent, t);
        }
        h         = get_header<W>(n, t);
        bool copy = via_older;
        via_older = false;
        if (snap && !to_version<W>(idx, n, h, ts, concurrent, copy, t)) return count;
        if (snap && concurrent && !copy) {
          bool retry     = false;
          uint32_t older = recheck_version(idx, ts, h.mod, retry, t);
          if (older != kNone) {
            idx       = older;
            via_older = true;
            continue;
          }
          if (retry) {
            __nanosleep(64);
            continue;
          }
        }
        settled = true;
      }
      if (!settled) {
        if (t.thread_rank() == 0) set_error(kErrStepLimit, 7);
        return count;
      }
    }
    return count;
  }

  // The range query of a tree no writer changes meanwhile (concurrent = false): the same route
  // and result as cooperative_range_query(lo, hi, t, ts, out, cap), with every
  // lane loading the header words itself (as find_quiescent) on the descent and along the leaf
  // chain, and the versions a snapshot read passes over read as headers alone.
  template <int W, class Tile>
  MVBT_DEV uint32_t range_quiescent(uint32_t lo, uint32_t hi, const Tile& t, uint32_t ts, uint2* out,
                                    uint32_t cap) const {
    if (hi <= lo) return 0;
    const bool snap = versioned && ts != kLatest;
    uint32_t idx    = kAnchor;
    node_regs<W> n;
    header h;
    for (uint32_t step = 0;; ++step) {  // descend to the leaf that holds lo
      if (step >= kMaxSteps) {
        if (t.thread_rank() == 0) set_error(kErrStepLimit, 5);
        return 0;
      }
      if (!valid(idx, t)) return 0;
      h = ld_header_words(node_ptr(idx));
      load<W>(idx, n, false, t);  // issued with the header loads
      if (snap && h.ts > ts) {    // a newer version: move to the older one
        idx = h.older();
        if (idx == kNone) {
          if (t.thread_rank() == 0) set_error(kErrCorrupt, 3);
          return 0;
        }
        continue;
      }
      if (lo < h.low) {
        idx = kAnchor;
        continue;
      }
      if (lo >= h.high && h.sibling() != kNone) {
        idx = h.sibling();
        continue;
      }
      if (h.is_leaf()) {
        break;
      }
      idx = child_for<W>(n, lo, t);
      if (idx == kNone) idx = kAnchor;
    }
    uint32_t count = 0;
    for (uint32_t leaves = 0;; ++leaves) {  // scan leaves to the right
      count += leaf_collect<W>(n, lo, hi, out, cap, count, t);
      if (!(hi > h.high && h.sibling() != kNone)) break;
      if (leaves >= capacity) {
        if (t.thread_rank() == 0) set_error(kErrStepLimit, 6);
        break;
      }
      idx = h.sibling();
      for (uint32_t hops = 0;; ++hops) {  // the next leaf, at ts
        if (!valid(idx, t)) return count;
        h = ld_header_words(node_ptr(idx));
        load<W>(idx, n, false, t);
        if (!(snap && h.ts > ts)) break;
        idx = h.older();
        if (idx == kNone || hops >= kMaxSteps) {
          if (t.thread_rank() == 0) set_error(kErrCorrupt, 3);
          return count;
        }
      }
    }
    return count;
  }

  // ------------------------------------------------------------------------------------------
  // Writers
  // ------------------------------------------------------------------------------------------
  // Descends to the leaf for key (newest versions, strong loads), recording in `path` the
  // interior node visited at each level: lane l holds level l in path0 and level l + W in path1.
  // Returns the leaf its level-1 parent names without reading it: the writer reads it under its
  // lock (lock_covering with direct = true), one round trip instead of three.
  template <int W, class Tile>
  MVBT_DEV uint32_t descend_for_write(uint32_t key, uint32_t& path0, uint32_t& path1,
                                      uint32_t& top_level, const Tile& t) const {
    uint32_t idx = kAnchor;
    node_regs<W> n;
    top_level = 0;
    bool first = true;
    for (uint32_t step = 0; step < kMaxSteps; ++step) {
      if (!valid(idx, t)) return kNone;
      load<W>(idx, n, true, t);
      header h = get_header<W>(n, t);
      if (first) {
        top_level = h.level();
        first     = false;
      }
      if (key < h.low) {  // routed too far right by a torn read: start over from the anchor
        idx   = kAnchor;
        first = true;
        path0 = kNone;
        path1 = kNone;
        continue;
      }
      if (key >= h.high && h.sibling() != kNone) {
        idx = h.sibling();
        continue;
      }
      uint32_t lvl = h.level();
      if (lvl == 0) {
        if (step > 16 && t.thread_rank() == 0) atomicMax(&ctl->stat_max_steps, (unsigned long long)step);
        return idx;
      }
      if (lvl < (uint32_t)W) {
        if (t.thread_rank() == (int)lvl) path0 = idx;
      } else {
        if (t.thread_rank() == (int)(lvl - W)) path1 = idx;
      }
      const uint32_t child = child_for<W>(n, key, t);
      if (child == kNone) {
        idx = kAnchor;
        continue;
      }
      if (lvl == 1) {
        if (step > 16 && t.thread_rank() == 0) atomicMax(&ctl->stat_max_steps, (unsigned long long)step);
        return child;
      }
      idx = child;
    }
    if (t.thread_rank() == 0) set_error(kErrStepLimit, 8);
    return kNone;
  }

  // Unlocked approach to the node at `level` whose range covers key, starting from idx (a node
  // at `level` or above on key's route): walks down along key and right along links. A long
  // chase to the right means the start is stale (many splits since it was read), so the walk
  // restarts from the anchor, which reaches the key in about height steps. Returns the index
  // with n/h loaded, or kNone on failure.
  template <int W, class Tile>
  MVBT_DEV uint32_t seek(uint32_t idx, uint32_t level, uint32_t key, node_regs<W>& n, header& h,
                         const Tile& t) const {
    uint32_t chase = 0;
    for (uint32_t step = 0; step < kMaxSteps; ++step) {
      if (!valid(idx, t)) return kNone;
      load<W>(idx, n, true, t);
      h = get_header<W>(n, t);
      if (key < h.low) {
        idx   = kAnchor;
        chase = 0;
        continue;
      }
      if (key >= h.high && h.sibling() != kNone) {
        if (++chase > kChaseRestart) {
          idx   = kAnchor;
          chase = 0;
        } else {
          idx = h.sibling();
        }
        continue;
      }
      if (h.level() == level) return idx;
      if (h.level() < level) {
        if (t.thread_rank() == 0) set_error(kErrCorrupt, 9);
        return kNone;
      }
      idx   = child_for<W>(n, key, t);
      chase = 0;
      if (idx == kNone) idx = kAnchor;
    }
    if (t.thread_rank() == 0) set_error(kErrStepLimit, 12);
    return kNone;
  }

  // Locks the node at `level` that covers key, starting from idx (the node recorded on the way
  // down, or the anchor). Only a few lock-coupled hops to the right are taken while holding a
  // lock; a node further right is re-approached unlocked. direct: idx is a live node at `level`
  // named by its parent or recorded on the way down, locked before it is read (a stale or
  // misrouted one is released again unchanged and approached as above). Returns the locked index
  // with n/h loaded; kNone on failure.
  template <int W, class Tile>
  MVBT_DEV uint32_t lock_covering(uint32_t idx, uint32_t level, uint32_t key, node_regs<W>& n,
                                  header& h, const Tile& t, bool direct = false) const {
    for (uint32_t attempt = 0; attempt < kMaxSteps; ++attempt) {
      if (!direct || attempt > 0) {
        idx = seek<W>(idx, level, key, n, h, t);
        if (idx == kNone) return kNone;
      }
      if (!lock(idx, t)) return kNone;
      load<W>(idx, n, true, t);
      h = get_header<W>(n, t);
      if (h.level() != level || key < h.low) {  // the anchor grew, or the approach was misrouted
        unlock(idx, t);
        if (key < h.low || h.level() < level) idx = kAnchor;
        continue;
      }
      uint32_t hops = 0;
      while (key >= h.high && h.sibling() != kNone && hops < kCoupledHops) {
        uint32_t sib = h.sibling();
        if (!lock(sib, t)) {
          unlock(idx, t);
          return kNone;
        }
        unlock(idx, t);
        idx = sib;
        load<W>(idx, n, true, t);
        h = get_header<W>(n, t);
        ++hops;
        if (h.level() != level) {  // a right link always stays on its level
          unlock(idx, t);
          if (t.thread_rank() == 0) set_error(kErrCorrupt, 10);
          return kNone;
        }
      }
      if (hops > 2 && t.thread_rank() == 0) atomicMax(&ctl->stat_max_hops, (unsigned long long)hops);
      if (!(key >= h.high && h.sibling() != kNone)) return idx;
      unlock(idx, t);  // still far to the left: approach again without holding locks
      if (t.thread_rank() == 0) atomicAdd(&ctl->stat_restarts, 1ull);
    }
    if (t.thread_rank() == 0) set_error(kErrStepLimit, 11);
    return kNone;
  }

  // Splits locked node idx (content n, header h, already prepared for epoch E) while inserting
  // {key, val}: the left half stays in idx, the right half goes to a new node written first.
  // Outputs the separator and the new node for the parent; releases the lock on idx. New nodes
  // of epoch E point at the version of idx older snapshots read, so such a reader that reaches
  // one continues from a node that covers its key.
  template <int W, class Tile>
  MVBT_DEV bool split_insert(uint32_t idx, node_regs<W>& n, header& h, uint32_t key, uint32_t val,
                             uint32_t E, uint32_t& sep_key, uint32_t& sep_child, const Tile& t) const {
    const int pos     = count_less<W>(n, key, t);
    const uint32_t ts = versioned ? E : 0u;
    uint32_t r = alloc(t);
    if (r == kNone) {
      unlock(idx, t);
      return false;
    }
    node_regs<W> left, right;
    build_from_merged<W>(n, pos, key, val, 0, kSplitLeft, left, t);
    build_from_merged<W>(n, pos, key, val, kSplitLeft, kDataPairs + 1 - kSplitLeft, right, t);
    uint32_t rmin = t.shfl(right.k[0], 0);
    header hr = make_header(rmin, 0u, h.high, h.sibling(), ts,
                            (h.level() << 28) | (versioned ? h.older() : kNone));
    header hl = make_header(h.low, h.mod, rmin, r, h.ts, h.ol);
    set_header<W>(right, hr, t);
    set_header<W>(left, hl, t);
    store<W>(r, right, t);
    publish_fence(t);
    store<W>(idx, left, t);
    if (t.thread_rank() == 0) atomicAdd(&ctl->sm_stats[sm_id() % kMaxSmSlots][1], 1ull);
    release(idx, h, t);
    sep_key   = rmin;
    sep_child = r;
    return true;
  }

  // The split node was the top: build a new top {0 -> old top, sep -> new node} one level up and
  // point the (locked, prepared) anchor at it. Releases the anchor.
  template <int W, class Tile>
  MVBT_DEV bool grow(node_regs<W>& n, header& h, uint32_t sep_key, uint32_t sep_child, uint32_t E,
                     const Tile& t) const {
    const uint32_t old_top = t.shfl(n.v[0], 0);
    const uint32_t top     = alloc(t);
    if (top == kNone) {
      unlock(kAnchor, t);
      return false;
    }
    const uint32_t lvl   = h.level();  // level of the new top
    const uint32_t older = versioned ? h.older() : kNone;
    node_regs<W> x;
#pragma unroll
    for (int j = 0; j < 16 / W; ++j) {
      const int q = pair_index<W>(t, j);
      x.k[j]      = q == 0 ? 0u : (q == 1 ? sep_key : kEmptyKey);
      x.v[j]      = q == 0 ? old_top : (q == 1 ? sep_child : kEmptyKey);
    }
    header hx = make_header(0u, 0u, kEmptyKey, kNone, versioned ? E : 0u, (lvl << 28) | older);
    set_header<W>(x, hx, t);
    store<W>(top, x, t);
    publish_fence(t);
#pragma unroll
    for (int j = 0; j < 16 / W; ++j)
      if (pair_index<W>(t, j) == 0) n.v[j] = top;
    h.ol = ((lvl + 1) << 28) | (h.ol & kIndexMask);
    set_header<W>(n, h, t);
    store<W>(kAnchor, n, t);
    if (t.thread_rank() == 0) atomicAdd(&ctl->sm_stats[sm_id() % kMaxSmSlots][1], 1ull);
    release(kAnchor, h, t);
    return true;
  }

  // Insert or update key -> value in write epoch E. Returns true on success.
  template <int W, class Tile>
  MVBT_DEV bool cooperative_insert(uint32_t key, uint32_t value, const Tile& t, uint32_t E) const {
    if (key == kEmptyKey) return false;
    uint32_t path0 = kNone, path1 = kNone, top = 0;
    const uint32_t leaf = descend_for_write<W>(key, path0, path1, top, t);
    if (leaf == kNone) return false;
    return insert_at<W>(key, value, t, E, leaf, path0, path1, top);
  }

  // The insert after its descent: `leaf` and the path (path0 / path1 / top, as descend_for_write
  // records them) may have been found before other writers changed the tree; lock_covering moves
  // right as far as needed and a stale path entry only lengthens the approach to a parent.
  template <int W, class Tile>
  MVBT_DEV bool insert_at(uint32_t key, uint32_t value, const Tile& t, uint32_t E, uint32_t leaf,
                          uint32_t path0, uint32_t path1, uint32_t top) const {
    if (key == kEmptyKey) return false;
    {
      node_regs<W> n;
      header h;
      leaf = lock_covering<W>(leaf, 0, key, n, h, t, true);
      if (leaf == kNone) return false;
      // update in place if present
      int pos = find_pos<W>(n, key, t);
      if (pos >= 0) {
        if (!prepare_write<W>(leaf, n, h, E, t)) {
          unlock(leaf, t);
          return false;
        }
#pragma unroll
        for (int j = 0; j < 16 / W; ++j)
          if (pair_index<W>(t, j) == pos) n.v[j] = value;
        store<W>(leaf, n, t);
        release(leaf, h, t);
        return true;
      }
      if (!prepare_write<W>(leaf, n, h, E, t)) {
        unlock(leaf, t);
        return false;
      }
      int nvalid = count_valid<W>(n, t);
      if (nvalid < kDataPairs) {
        int ipos = count_less<W>(n, key, t);
        node_regs<W> out;
        build_from_merged<W>(n, ipos, key, value, 0, nvalid + 1, out, t);
        store<W>(leaf, out, t);
        release(leaf, h, t);
        return true;
      }
      // full leaf: split, then push separators up
      uint32_t sep_key = 0, sep_child = kNone;
      if (!split_insert<W>(leaf, n, h, key, value, E, sep_key, sep_child, t)) return false;
      return push_up<W>(sep_key, sep_child, E, path0, path1, top, t);
    }
  }

  // Inserts the separator {sep_key -> sep_child} of a leaf split into the level above, splitting
  // full interior nodes in turn and growing the tree at the anchor. path0 / path1 / top are the
  // parent hints as descend_for_write records them.
  template <int W, class Tile>
  MVBT_OUTLINE bool push_up(uint32_t sep_key, uint32_t sep_child, uint32_t E, uint32_t path0, uint32_t path1,
                        uint32_t top, const Tile& t) const {
    node_regs<W> n;
    header h;
    int nvalid;
    uint32_t level = 1;
    while (sep_child != kNone) {
      uint32_t start;
      if (level <= top) {
        start = (level < (uint32_t)W) ? t.shfl(path0, level) : t.shfl(path1, level - W);
        if (start == kNone) start = kAnchor;
      } else {
        start = kAnchor;
      }
      if (level >= (uint32_t)kMaxLevels) {
        if (t.thread_rank() == 0) set_error(kErrCorrupt, 13);
        return false;
      }
      uint32_t p = lock_covering<W>(start, level, sep_key, n, h, t, start != kAnchor);
      if (p == kNone) return false;
      if (!prepare_write<W>(p, n, h, E, t)) {
        unlock(p, t);
        return false;
      }
      if (p == kAnchor) return grow<W>(n, h, sep_key, sep_child, E, t);
      nvalid = count_valid<W>(n, t);
      if (nvalid < kDataPairs) {
        int ipos = count_less<W>(n, sep_key, t);
        node_regs<W> out;
        build_from_merged<W>(n, ipos, sep_key, sep_child, 0, nvalid + 1, out, t);
        store<W>(p, out, t);
        release(p, h, t);
        return true;
      }
      uint32_t k2 = sep_key, c2 = sep_child;
      if (!split_insert<W>(p, n, h, k2, c2, E, sep_key, sep_child, t)) return false;
      ++level;
    }
    return true;
  }

  // Erase key in write epoch E. Returns true if the key was present.
  template <int W, class Tile>
  MVBT_DEV bool cooperative_erase(uint32_t key, const Tile& t, uint32_t E) const {
    if (key == kEmptyKey) return false;
    uint32_t path0 = kNone, path1 = kNone, top = 0;
    const uint32_t leaf = descend_for_write<W>(key, path0, path1, top, t);
    if (leaf == kNone) return false;
    return erase_at<W>(key, t, E, leaf);
  }

  // The erase after its descent (the leaf may be stale: lock_covering moves right).
  template <int W, class Tile>
  MVBT_DEV bool erase_at(uint32_t key, const Tile& t, uint32_t E, uint32_t leaf) const {
    if (key == kEmptyKey) return false;
    node_regs<W> n;
    header h;
    leaf = lock_covering<W>(leaf, 0, key, n, h, t, true);
    if (leaf == kNone) return false;
    int pos = find_pos<W>(n, key, t);
    if (pos < 0) {
      unlock(leaf, t);
      return false;
    }
    if (!prepare_write<W>(leaf, n, h, E, t)) {
      unlock(leaf, t);
      return false;
    }
    remove_at<W>(n, pos, t);
    store<W>(leaf, n, t);
    release(leaf, h, t);
    return true;
  }

  // Snapshot: returns the id of the new snapshot (the pre-increment epoch).
  template <class Tile>
  MVBT_DEV uint32_t take_snapshot(const Tile& t) const {
    __threadfence();
    uint32_t s = 0;
    if (t.thread_rank() == 0) s = atomicAdd(&ctl->epoch, 1u);
    return t.shfl(s, 0);
  }
};

// ----------------------------------------------------------------------------------------------
// Lookups of a whole warp in a tree no writer changes meanwhile (concurrent = false)
// ----------------------------------------------------------------------------------------------
// Each lane holds one key. A step of the warp copies the node every lane has reached into shared
// memory -- eight lanes per node, each distinct neighbour once -- and each lane then searches its
// own node there. A tile per key (find_quiescent) spends the instructions of a whole tile on
// one key's node; here 32 keys share them, and keys that are near each other share the node
// reads too.
struct alignas(16) warp_stage {
  uint32_t node[32][kNodeWords];  // 16-byte pieces of node s at piece ^ (s & 7): the lanes' reads
                                  // of one word of different nodes spread over the banks
  uint32_t idx[32];               // the nodes to copy
  // Word w of staged node s, and its words 28..31.
  MVBT_DEV uint32_t word(uint32_t s, uint32_t w) const { return node[s][(((w >> 2) ^ (s & 7u)) << 2) | (w & 3u)]; }
  MVBT_DEV const uint32_t* last_words(uint32_t s) const { return &node[s][(7u ^ (s & 7u)) << 2]; }
};
#if defined(MVBT_HOST_EMULATION)
MVBT_DEV void ld_shared_4(const uint32_t* p, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  a = p[0], b = p[1], c = p[2], d = p[3];
}
#else
MVBT_DEV void ld_shared_4(const uint32_t* p, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  a = v.x, b = v.y, c = v.z, d = v.w;
}
#endif

// Path memory of a warp that runs keys in ascending order: the last key's node per level
// {index, low, high}, from which the next keys start.
struct warp_path {
  uint32_t at[kMaxLevels][3];
  template <class Warp>
  MVBT_DEV void clear(const Warp& warp) {
    const uint32_t lane = warp.thread_rank();
    if (lane < (uint32_t)kMaxLevels) record(lane, kNone, kEmptyKey, 0);  // covers nothing
    warp.sync();
  }
  MVBT_DEV void record(uint32_t level, uint32_t idx, uint32_t low, uint32_t high) {
    at[level][0] = idx;
    at[level][1] = low;
    at[level][2] = high;
  }
  // Lowest remembered node that covers all of [first, last], or the anchor. Every lane looks at a level.
  template <class Warp>
  MVBT_DEV uint32_t start(uint32_t first, uint32_t last, const Warp& warp) const {
    const uint32_t l  = warp.thread_rank() & (kMaxLevels - 1u);
    const uint32_t in = warp.ballot(at[l][1] <= first && last < at[l][2]);
    return in ? at[__ffs(in) - 1][0] : kAnchor;
  }
};

// Copies the nodes idx of the live lanes (m) into st, neighbouring lanes' equal ones once; returns
// the lane's slot. The caller keeps every lane's reads of the last nodes before this (warp.sync).
template <bool kStrong, class Warp>
MVBT_DEV uint32_t stage_nodes(const device_tree& T, uint32_t idx, bool live, uint32_t m, warp_stage& st,
                              const Warp& warp) {
  const uint32_t lane  = warp.thread_rank();
  const uint32_t prev  = warp.shfl(idx, lane ? (int)lane - 1 : 0);
  const bool lead      = live && (lane == 0 || !((m >> (lane - 1)) & 1u) || prev != idx);
  const uint32_t leads = warp.ballot(lead);
  const uint32_t slot  = (uint32_t)__popc(leads & ((2u << lane) - 1u)) - 1u;
  if (lead) st.idx[slot] = idx;
  warp.sync();
  const uint32_t nodes = (uint32_t)__popc(leads), piece = lane & 7u;
  for (uint32_t s = lane >> 3; s < nodes; s += 4)
    copy_16<kStrong>(&st.node[s][(piece ^ (s & 7u)) << 2], T.node_ptr(st.idx[s]) + piece * 4);
  copy_wait();
  warp.sync();
  return slot;
}

// Pairs of staged node s whose key is <= key: they are sorted, and unused ones hold the highest key.
MVBT_DEV uint32_t count_up_to(const warp_stage& st, uint32_t s, uint32_t key) {
  uint32_t c = st.word(s, 2 * 7) <= key ? 8u : 0u;
  if (st.word(s, 2 * (c + 3)) <= key) c += 4;
  if (c + 1 < (uint32_t)kDataPairs && st.word(s, 2 * (c + 1)) <= key) c += 2;
  if (c < (uint32_t)kDataPairs && st.word(s, 2 * c) <= key) c += 1;
  return c;
}

// The value of each live lane's key at snapshot ts (kLatest: newest), kNotFound elsewhere; the
// route and results of find_quiescent. start: a node on the key's route (the anchor, or path->start).
// path (nullable): the nodes that the highest live lane passes are recorded in it.
template <class Warp>
MVBT_DEV uint32_t find_warp(const device_tree& T, uint32_t key, bool live, uint32_t ts, uint32_t start,
                            warp_path* path, warp_stage& st, const Warp& warp) {
  const bool snap     = T.versioned && ts != kLatest;
  const uint32_t lane = warp.thread_rank();
  uint32_t found      = kNotFound;
  uint32_t idx        = start;
  live                = live && key != kEmptyKey;
  const uint32_t all  = warp.ballot(live);
  const bool last     = path && live && (all >> lane) == 1u;
  for (uint32_t step = 0; step < kMaxSteps; ++step) {
    if (live && idx >= T.capacity) {
      T.set_error(kErrCorrupt, 1);
      live = false;
    }
    const uint32_t m = warp.ballot(live);
    if (m == 0) return found;
    const uint32_t slot = stage_nodes<false>(T, idx, live, m, st, warp);
    if (live) {
      const uint32_t low = st.word(slot, 26);
      uint32_t high, link, nts, ol;
      ld_shared_4(st.last_words(slot), high, link, nts, ol);
      link &= kIndexMask;
      if (snap && nts > ts) {  // a newer version: move to the older one
        idx = ol & kIndexMask;
        if (idx == kNone) {
          T.set_error(kErrCorrupt, 3);
          live = false;
        }
      } else if (key < low) {
        idx = kAnchor;
      } else if (key >= high && link != kNone) {
        idx = link;
      } else {
        const uint32_t level = ol >> 28;
        if (last) path->record(level, idx, low, high);
        const uint32_t c  = count_up_to(st, slot, key);
        const uint32_t pk = c ? st.word(slot, 2 * c - 2) : kEmptyKey;
        const uint32_t pv = c ? st.word(slot, 2 * c - 1) : kAnchor;
        if (level == 0) {
          if (pk == key) found = pv;
          live = false;
        } else {
          idx = pv;
        }
      }
    }
    warp.sync();
  }
  if (live) T.set_error(kErrStepLimit, 4);
  return found;
}

// find_warp at snapshot ts (of each lane) while writers run in the same kernel: cooperative_find's
// route and checks. start: a node on the key's route, as read at the newest state.
template <class Warp>
MVBT_DEV uint32_t find_warp_live(const device_tree& T, uint32_t key, bool live, uint32_t ts, uint32_t start,
                                 warp_stage& st, const Warp& warp) {
  uint32_t found = kNotFound;
  uint32_t idx   = start;
  bool copy      = false;  // idx is an older version, which is never written again
  live           = live && key != kEmptyKey;
  for (uint32_t step = 0; step < kMaxSteps; ++step) {
    if (live && idx >= T.capacity) {
      T.set_error(kErrCorrupt, 1);
      live = false;
    }
    const uint32_t m = warp.ballot(live);
    if (m == 0) return found;
    const uint32_t slot = stage_nodes<true>(T, idx, live, m, st, warp);
    bool check          = false;  // the leaf of the snapshot, unless a writer is changing it
    uint32_t value      = kNotFound;
    if (live) {
      const uint32_t low = st.word(slot, 26);
      uint32_t high, link, nts, ol;
      ld_shared_4(st.last_words(slot), high, link, nts, ol);
      link &= kIndexMask;
      if (nts > ts) {
        idx  = ol & kIndexMask;
        copy = true;
        if (idx == kNone) {
          T.set_error(kErrCorrupt, 3);
          live = false;
        }
      } else if (key < low) {
        idx  = kAnchor;
        copy = false;
      } else if (key >= high && link != kNone) {
        idx  = link;
        copy = false;
      } else {
        const uint32_t c  = count_up_to(st, slot, key);
        const uint32_t pk = c ? st.word(slot, 2 * c - 2) : kEmptyKey;
        const uint32_t pv = c ? st.word(slot, 2 * c - 1) : kAnchor;
        if ((ol >> 28) == 0) {
          if (pk == key) value = pv;
          check = !copy;
          live  = check;
          found = value;
        } else {
          idx  = pv;
          copy = false;
        }
      }
    }
    if (warp.ballot(check)) {  // as recheck_version
      __threadfence();
      warp.sync();
      if (check) {
        const uint32_t* node = T.node_ptr(idx);
        const uint32_t mod0 = st.word(slot, kModWord), mod1 = ld_relaxed_u32(node + kModWord);
        const unsigned long long v = ld_relaxed_u64(reinterpret_cast<const unsigned long long*>(node + 30));
        if ((uint32_t)v > ts) {  // changed meanwhile: its immutable copy instead
          idx  = (uint32_t)(v >> 32) & kIndexMask;
          copy = true;
        } else if (!(mod0 & kLockBit) && mod1 == mod0) {
          live = false;
        } else {
          __nanosleep(64);  // a writer is changing it: read it again
        }
      }
    }
    warp.sync();
  }
  if (live) T.set_error(kErrStepLimit, 4);
  return found;
}

// Range queries [lo, hi) of the live lanes at snapshot ts: cooperative_range_query's route, pairs and
// full count (kLive: while writers run, at snapshots; otherwise range_quiescent's). Each lane writes
// at most cap pairs at out (nullable). The lanes walk their leaves in step: the warp stages one leaf
// per lane, each lane finds its pairs there, and eight lanes per query write them. start, path: as in
// find_warp.
template <bool kLive, class Warp>
MVBT_DEV uint32_t range_warp(const device_tree& T, uint32_t lo, uint32_t hi, bool live, uint32_t ts, uint2* out,
                             uint32_t cap, uint32_t start, warp_path* path, warp_stage& st, const Warp& warp) {
  const bool snap     = T.versioned && ts != kLatest;
  const uint32_t lane = warp.thread_rank();
  live                = live && hi > lo;
  uint32_t idx = start, count = 0, hops = 0, leaves = 0;
  bool copy = false, scan = false;  // idx is an older version; idx is the next leaf to the right
  const uint32_t all = warp.ballot(live);
  const bool last    = path && live && (all >> lane) == 1u;
  for (;;) {
    if (live && idx >= T.capacity) {
      T.set_error(kErrCorrupt, 1);
      live = false;
    }
    if (live && ++hops > kMaxSteps) {
      T.set_error(kErrStepLimit, scan ? 7 : 5);
      live = false;
    }
    const uint32_t m = warp.ballot(live);
    if (m == 0) return count;
    const uint32_t slot = stage_nodes<kLive>(T, idx, live, m, st, warp);
    bool use            = false;  // the staged node is the lane's next leaf at ts
    uint32_t high = 0, link = kNone;
    if (live) {
      const uint32_t low = st.word(slot, 26);
      uint32_t nts, ol;
      ld_shared_4(st.last_words(slot), high, link, nts, ol);
      link &= kIndexMask;
      if (snap && nts > ts) {
        idx  = ol & kIndexMask;
        copy = true;
        if (idx == kNone) {
          T.set_error(kErrCorrupt, 3);
          live = false;
        }
      } else if (scan) {
        use = true;
      } else if (lo < low) {
        idx  = kAnchor;
        copy = false;
      } else if (lo >= high && link != kNone) {
        idx  = link;
        copy = false;
      } else {
        const uint32_t level = ol >> 28;
        if (last) path->record(level, idx, low, high);
        use = level == 0;
        if (!use) {
          const uint32_t c = count_up_to(st, slot, lo);
          idx              = c ? st.word(slot, 2 * c - 1) : kAnchor;
          copy             = false;
        }
      }
    }
    if (kLive) {
      const bool check = use && !copy;
      if (warp.ballot(check)) {  // as recheck_version
        __threadfence();
        warp.sync();
        if (check) {
          const uint32_t* node = T.node_ptr(idx);
          const uint32_t mod0 = st.word(slot, kModWord), mod1 = ld_relaxed_u32(node + kModWord);
          const unsigned long long v = ld_relaxed_u64(reinterpret_cast<const unsigned long long*>(node + 30));
          if ((uint32_t)v > ts) {  // changed meanwhile: its immutable copy instead
            idx  = (uint32_t)(v >> 32) & kIndexMask;
            copy = true;
            use  = false;
          } else if ((mod0 & kLockBit) || mod1 != mod0) {
            use = false;  // a writer is changing it: read it again
            __nanosleep(64);
          }
        }
      }
    }
    const uint32_t uses = warp.ballot(use);
    uint32_t first = 0, pairs = 0, room = 0;
    if (use) {
      first = lo ? count_up_to(st, slot, lo - 1u) : 0u;
      pairs = count_up_to(st, slot, hi - 1u) - first;
      room  = out == nullptr || count >= cap ? 0u : (pairs < cap - count ? pairs : cap - count);
    }
    const uint32_t info = use ? slot | (first << 8) | (room << 16) : 0u;
    const unsigned long long to = (unsigned long long)(out + count);
    for (uint32_t q = 0; q < 32; q += 4) {  // four queries at a time
      if (((uses >> q) & 15u) == 0) continue;
      const int src             = (int)(q + (lane >> 3));
      const uint32_t what       = warp.shfl(info, src);
      const unsigned long long at = warp.shfl(to, src);
      const uint32_t s = what & 255u, a = (what >> 8) & 255u;
      for (uint32_t j = lane & 7u; j < what >> 16; j += 8) {
        const uint32_t* w = &st.node[s][((((a + j) >> 1) ^ (s & 7u)) << 2) | (((a + j) & 1u) << 1)];
        reinterpret_cast<uint2*>(at)[j] = make_uint2(w[0], w[1]);
      }
    }
    if (use) {
      count += pairs;
      hops = 0;
      if (hi > high && link != kNone) {
        idx  = link;
        scan = true;
        copy = false;
        if (++leaves > T.capacity) {  // a sibling chain is never longer than the pool
          T.set_error(kErrStepLimit, 6);
          live = false;
        }
      } else {
        live = false;
      }
    }
    warp.sync();
  }
}

// ----------------------------------------------------------------------------------------------
// Writes of a whole warp
// ----------------------------------------------------------------------------------------------
struct write_stage : warp_stage {
  uint32_t op[32][2];  // each lane's {key, value}; once tried, whether its leaf was full in place of the key
  uint32_t dst[32];    // where each staged node is stored (kNone: nowhere)
  uint32_t parent[32]; // the level-1 node that named each lane's leaf (kNone: not seen)
};

// The stages of a block's warps follow one another in shared memory, and their staged nodes start on 128-byte
// boundaries: with 16 bytes more per stage the batched kernel took 8.7-9.2 ms for 256 batches of 11.1M ops,
// against 8.0-8.4.
static_assert(sizeof(write_stage) % 128 == 0, "staged nodes start on 128-byte boundaries");

// The leaf that each live lane's key belongs to, unread: the child its level-1 node names (kNone:
// failed), and that node (st.parent), where a split of the leaf puts its separator. Routing at the newest
// state while writers run, as descend_for_write.
template <class Warp>
MVBT_DEV uint32_t leaf_warp(const device_tree& T, uint32_t key, bool live, uint32_t start, warp_path* path,
                            write_stage& st, const Warp& warp) {
  const uint32_t lane = warp.thread_rank();
  st.parent[lane]     = kNone;
  uint32_t leaf       = kNone;
  uint32_t idx        = start;
  const uint32_t all  = warp.ballot(live);
  const bool last     = path && live && (all >> lane) == 1u;
  for (uint32_t step = 0; step < kMaxSteps; ++step) {
    if (live && idx >= T.capacity) {
      T.set_error(kErrCorrupt, 1);
      live = false;
    }
    const uint32_t m = warp.ballot(live);
    if (m == 0) return leaf;
    const uint32_t slot = stage_nodes<true>(T, idx, live, m, st, warp);
    if (live) {
      const uint32_t low = st.word(slot, 26);
      uint32_t high, link, nts, ol;
      ld_shared_4(st.last_words(slot), high, link, nts, ol);
      link &= kIndexMask;
      const uint32_t level = ol >> 28;
      if (key < low) {
        idx = kAnchor;
      } else if (key >= high && link != kNone) {
        idx = link;
      } else if (level == 0) {  // reached through a sibling link or a misrouted read
        leaf = idx;
        live = false;
      } else {
        if (last) path->record(level, idx, low, high);
        const uint32_t c = count_up_to(st, slot, key);
        if (c && level == 1) st.parent[lane] = idx;
        idx = c ? st.word(slot, 2 * c - 1) : kAnchor;
        if (c && level == 1) {
          leaf = idx;
          live = false;
        }
      }
    }
    warp.sync();
  }
  if (live) T.set_error(kErrStepLimit, 8);
  return leaf;
}

// A fresh node for each lane with `need` set (kNone: the pool is full or the wait limit ran out): the
// warp's nodes with one atomic on the SM's chunk cursor instead of one per node.
template <class Warp>
MVBT_DEV uint32_t alloc_warp(const device_tree& T, bool need, const Warp& warp) {
  const uint32_t m = warp.ballot(need);
  if (m == 0) return kNone;
  control_block* c    = T.ctl;
  const uint32_t lane = warp.thread_rank();
  const uint32_t C    = c->chunk;
  const uint32_t k    = (uint32_t)__popc(m);
  const int lead      = __ffs(m) - 1;
  uint32_t idx        = kNone;
  if (C < 32) {  // a request could span chunks
    if (need) idx = T.alloc_one();
  } else {
    uint32_t base = 0, used = 0, next = kNone;  // nodes base + used .. below chunk C, then next, next + 1, ..
    bool got = false;
    if ((int)lane == lead) {
      unsigned long long* slot    = &c->sm_pool[sm_id() % kMaxSmSlots];
      const uint32_t limit        = c->spin_limit;
      const unsigned long long t0 = global_ns();
      for (uint32_t tries = 0; tries < limit; ++tries) {
        if (tries && (ld_relaxed_u32(&c->error) & kErrPoolExhausted)) break;
        const unsigned long long old = atomicAdd(slot, (unsigned long long)k);
        base = (uint32_t)(old >> 32), used = (uint32_t)old;
        if (used + k <= C) {
          got = true;
          break;
        }
        if (used <= C) {  // this request holds position C: it refills the chunk, as alloc_one does
          got = true;
          if (!(T.reclaim && take_free_chunk(c, C, next))) {
            next = atomicAdd(&c->bump, C);
            if ((unsigned long long)next + C > c->capacity) {
              next = kNone;
              atomicOr(&c->error, kErrPoolExhausted);
              atomicAdd(&c->err_site[15], 1u);
            }
          }
          if (next != kNone) atomicExch(slot, ((unsigned long long)next << 32) | (used + k - C));
          break;
        }
        for (uint32_t w = 0; w < limit; ++w) {  // another request refills it
          __nanosleep(64);
          const unsigned long long cur = ld_relaxed_u64(slot);
          if ((uint32_t)(cur >> 32) != base || (uint32_t)cur < C) break;
          if (ld_relaxed_u32(&c->error) & kErrPoolExhausted) break;
          if (global_ns() - t0 > c->wait_ns) break;
        }
        if (global_ns() - t0 > c->wait_ns) break;
      }
      if (!got && !(ld_relaxed_u32(&c->error) & kErrPoolExhausted)) {
        atomicOr(&c->error, kErrSpinLimit);
        atomicAdd(&c->err_site[0], 1u);
      }
    }
    base             = warp.shfl(base, lead);
    used             = warp.shfl(used, lead);
    next             = warp.shfl(next, lead);
    const bool given = warp.shfl(got ? 1u : 0u, lead) != 0;
    if (need && given) {
      const uint32_t at = used + (uint32_t)__popc(m & ((1u << lane) - 1u));
      if (at < C) idx = base + at;
      else if (next != kNone) idx = next + (at - C);
    }
  }
  if (idx != kNone && (idx & kRingChunk)) idx = chunk_node(c, idx, 0);  // a position in the free ring
  return idx;
}

// Records the lanes' version copies (`has` set), as device_tree::retire, with one reservation.
template <class Warp>
MVBT_DEV void retire_warp(const device_tree& T, bool has, uint32_t copy, const Warp& warp) {
  const uint32_t m = warp.ballot(has);
  if (m == 0) return;
  control_block* c    = T.ctl;
  const uint32_t lane = warp.thread_rank();
  const int lead      = __ffs(m) - 1;
  unsigned long long pos = 0;
  if ((int)lane == lead) {
    if (T.reclaim) pos = atomicAdd(&c->retire_tail, (unsigned long long)__popc(m));
    else atomicAdd(&c->sm_stats[sm_id() % kMaxSmSlots][0], (unsigned long long)__popc(m));
  }
  if (!T.reclaim) return;  // the same in every lane
  pos = warp.shfl(pos, lead) + (uint32_t)__popc(m & ((1u << lane) - 1u));
  if (has) {
    if (pos - ld_relaxed_u64(&c->retire_head) < c->reclaim_cap)
      reinterpret_cast<uint32_t*>(c->retire_log)[pos & (c->reclaim_cap - 1u)] = copy;
    else
      atomicAdd(&c->stat_log_dropped, 1ull);
  }
}

// Applies one op to staged leaf s of n pairs; false: an insert found it full. Called by one lane.
MVBT_DEV bool apply_staged(warp_stage& st, uint32_t s, uint32_t& n, uint32_t key, uint32_t value, bool erase) {
  auto at           = [&](uint32_t w) -> uint32_t& { return st.node[s][(((w >> 2) ^ (s & 7u)) << 2) | (w & 3u)]; };
  const uint32_t c  = count_up_to(st, s, key);
  const bool hit    = c && at(2 * c - 2) == key;
  if (erase) {
    if (!hit) return true;
    for (uint32_t p = c; p < n; ++p) at(2 * p - 2) = at(2 * p), at(2 * p - 1) = at(2 * p + 1);
    at(2 * n - 2) = kEmptyKey, at(2 * n - 1) = kEmptyKey;
    --n;
    return true;
  }
  if (hit) {
    at(2 * c - 1) = value;
    return true;
  }
  if (n == (uint32_t)kDataPairs) return false;
  for (uint32_t p = n; p > c; --p) at(2 * p) = at(2 * p - 2), at(2 * p + 1) = at(2 * p - 1);
  at(2 * c) = key, at(2 * c + 1) = value;
  ++n;
  return true;
}

// Calls f(src) by each tile for the lanes of m, a tile's share at a time: src is the lane (the same in
// every lane of the tile) and run says whether the tile has one. f runs with the tile converged.
template <int W, class Warp, class F>
MVBT_DEV void for_lanes(uint32_t m, const Warp& warp, const F& f) {
  for (uint32_t left = m; left;) {
    uint32_t own = left;
    for (uint32_t q = 0; q < warp.thread_rank() / (uint32_t)W; ++q) own &= own - 1u;
    f(own != 0, own ? __ffs(own) - 1 : 0);
    for (uint32_t q = 0; q < 32u / W; ++q) left &= left - 1u;
    warp.sync();
  }
}

// Splits staged leaf s, which is full, while inserting {key, value}: the left half stays in slot s, the right half
// is built in slot r for the node `right`. Contents as device_tree::split_insert's. Called by one lane.
MVBT_DEV void split_staged(const device_tree& T, write_stage& st, uint32_t s, uint32_t r, uint32_t key, uint32_t value,
                           uint32_t E, uint32_t right) {
  auto at = [&](uint32_t q, uint32_t w) -> uint32_t& { return st.node[q][(((w >> 2) ^ (q & 7u)) << 2) | (w & 3u)]; };
  constexpr uint32_t kLeft = (uint32_t)kSplitLeft, kRight = (uint32_t)kDataPairs + 1u - kLeft;
  const uint32_t c = count_up_to(st, s, key);  // the pair's place among the kDataPairs + 1
  for (uint32_t q = 0; q < (uint32_t)kDataPairs; ++q) {
    const uint32_t i = kLeft + q, from = i > c ? i - 1u : i;
    at(r, 2 * q)     = q >= kRight ? kEmptyKey : (i == c ? key : at(s, 2 * from));
    at(r, 2 * q + 1) = q >= kRight ? kEmptyKey : (i == c ? value : at(s, 2 * from + 1));
  }
  if (c < kLeft) {
    for (uint32_t p = kLeft - 1u; p > c; --p) at(s, 2 * p) = at(s, 2 * p - 2), at(s, 2 * p + 1) = at(s, 2 * p - 1);
    at(s, 2 * c) = key, at(s, 2 * c + 1) = value;
  }
  for (uint32_t p = kLeft; p < (uint32_t)kDataPairs; ++p) at(s, 2 * p) = kEmptyKey, at(s, 2 * p + 1) = kEmptyKey;
  const uint32_t low = at(r, 0);
  at(r, 26) = low, at(r, kModWord) = 0u, at(r, 28) = at(s, 28), at(r, 29) = at(s, 29) & kIndexMask;
  at(r, 30) = T.versioned ? E : 0u, at(r, 31) = T.versioned ? at(s, 31) & kIndexMask : kNone;
  at(s, 28) = low, at(s, 29) = right;
}

// One write by a tile, from the leaf where its warp found it, under its level-1 node `parent` (kNone: unknown).
template <int W, class Tile>
MVBT_CALL void write_tile(device_tree T, uint32_t key, uint32_t value, bool erase, uint32_t E, uint32_t leaf,
                          uint32_t parent, Tile tile) {
  if (erase) T.erase_at<W>(key, tile, E, leaf);
  else T.insert_at<W>(key, value, tile, E, leaf, parent, kNone, 1u);  // path0 holds level 1 in its lane 1
}
// A split's separator by a tile, into the level-1 node `node` (kNone: unknown) or where it leads.
template <int W, class Tile>
MVBT_CALL void push_tile(device_tree T, uint32_t key, uint32_t child, uint32_t E, uint32_t node, Tile tile) {
  T.push_up<W>(key, child, E, node, kNone, 1u, tile);
}

// Runs the live lanes' inserts (key -> value) and erases in write epoch E. The warp locks the leaves
// of all its keys with one atomic per leaf, stages them, copies the versions that need it, applies
// every key of a leaf to its staged copy and writes the leaves back, so two fences serve up to 32
// leaves where a tile per key (insert_at, erase_at) spends them on one. The steps on a leaf and their
// order are those of the tile path: lock, read, version copy complete before a header names it,
// leaf stored, release. No lane waits for a lock while the warp holds one: leaves found locked are
// tried again after the others are released.
// A leaf without room for a new key is split by the tile path (one key per leaf at a time), and the leaf's
// other keys go on from there.
// kSplit: a full leaf is split where it is staged, while there are slots for the right halves; these are stored
// before their left halves name them, and the separators are then written like keys, a level up: separators
// of one parent share its lock. What is left goes to the tile path: splits without a slot, and separators
// whose parent is full, stale or the anchor. For keys in order, whose leaves have parents in common: 4M new
// keys into a plain tree of 16M 2.44 -> 1.66 ms, once more 4.32 -> 2.81. Keys all over the tree split
// few leaves of a warp at once, under as many parents, and the other leaves wait for the additional round:
// 500K inserts beside 500K range queries 0.84 -> 0.86 ms, so these take the tile path.
// leaf: each live lane's leaf as leaf_warp found it (which also left its parent in st.parent), possibly stale
// (kNone: the op is given up). Two live lanes may hold one key only if either order will do.
template <int W, bool kSplit = false, class Warp, class Tile>
MVBT_DEV void write_warp(const device_tree& T, uint32_t key, uint32_t value, bool erase, bool live, uint32_t E,
                         uint32_t leaf, write_stage& st, const Warp& warp, const Tile& tile) {
  constexpr uint32_t kTiles = 32 / W;
  const uint32_t lane       = warp.thread_rank();
  const uint32_t piece      = lane & 7u;
  bool pend                 = live && key != kEmptyKey && leaf != kNone;
  const uint32_t erases     = warp.ballot(erase);
  uint32_t seps             = 0;  // lanes whose op has become the separator of the split it made
  uint32_t tries = 0, backoff = 32;
  unsigned long long t0     = 0;
  auto store = [&](uint32_t from, uint32_t to) {  // the staged nodes [from, to) to where st.dst says
    for (uint32_t s = from + (lane >> 3); s < to; s += 4) {
      const uint32_t dst = st.dst[s];
      if (dst == kNone) continue;
      uint32_t w[4];
      ld_shared_4(&st.node[s][(piece ^ (s & 7u)) << 2], w[0], w[1], w[2], w[3]);
      store_16(T.node_ptr(dst) + piece * 4, w);
    }
  };
  for (uint32_t step = 0; step < kMaxSteps;) {
    if (pend && leaf >= T.capacity) {
      T.set_error(kErrCorrupt, 1);
      pend = false;
    }
    const uint32_t all = warp.ballot(pend);
    if (all == 0) return;
    const bool up     = kSplit && (all & seps) != 0;  // a round for separators, in level 1, or one for keys
    const uint32_t pm = up ? all & seps : all;
    const bool mem    = (pm >> lane) & 1u;
    const bool del    = !up && erase;
    // one leader per run of lanes with the same node (kSplit: whatever lanes between them are done)
    const uint32_t below = pm & (kSplit ? (1u << lane) - 1u : lane ? 1u << (lane - 1u) : 0u);
    const uint32_t prev  = warp.shfl(leaf, kSplit ? (below ? 31 - __clz(below) : 0) : (lane ? (int)lane - 1 : 0));
    const bool lead      = mem && (below == 0 || prev != leaf);
    const uint32_t lm    = warp.ballot(lead);
    uint32_t* const mod  = T.node_ptr(mem ? leaf : 0u) + kModWord;
    bool locked          = false;
    if (lead) locked = !(atomicOr(mod, kLockBit) & kLockBit);
    const uint32_t okm = warp.ballot(locked);
    if (okm == 0) {  // all held elsewhere: as device_tree::lock, bounded by the clock and the attempts alone
      if (tries == 0) t0 = global_ns();
      if (++tries >= T.ctl->spin_limit || wait_expired(t0, T.ctl->wait_ns, warp)) {
        if (lead) T.set_error(kErrSpinLimit, 2);
        return;
      }
      // wait until one looks free before the next atomics
      for (uint32_t w = 0; w < 64; ++w) {
        __nanosleep(backoff);
        if (warp.ballot(lead && !(ld_relaxed_u32(mod) & kLockBit))) break;
        backoff = backoff < 1024 ? backoff * 2 : 1024;
      }
      continue;
    }
    ++step;
    tries   = 0;
    backoff = 32;
    __threadfence();
    warp.sync();
    const uint32_t upto = lm & ((2u << lane) - 1u);
    const uint32_t boss = upto ? 31u - (uint32_t)__clz(upto) : 0u;  // the lane's leader
    const bool have     = mem && ((okm >> boss) & 1u);
    const uint32_t slot = (uint32_t)__popc(okm & ((1u << boss) - 1u));
    const uint32_t nodes = (uint32_t)__popc(okm);
    if (locked) st.idx[slot] = leaf;
    st.op[lane][0] = key;
    st.op[lane][1] = value;
    warp.sync();
    for (uint32_t s = lane >> 3; s < nodes; s += 4)
      copy_16<true>(&st.node[s][(piece ^ (s & 7u)) << 2], T.node_ptr(st.idx[s]) + piece * 4);
    copy_wait();
    warp.sync();
    // what each lane finds: its node, a node further right, or a stale route
    bool cover = false, act = false, stale = false;
    uint32_t high = 0, link = 0, nts = 0, ol = 0;
    if (have) {
      ld_shared_4(st.last_words(slot), high, link, nts, ol);
      const uint32_t sib = link & kIndexMask;
      if ((ol >> 28) != (up ? 1u : 0u) || key < st.word(slot, 26)) {
        stale = true;
      } else if (key >= high && sib != kNone) {
        leaf = sib;  // next round
      } else {
        cover            = true;
        const uint32_t c = count_up_to(st, slot, key);
        act              = (c && st.word(slot, 2 * c - 2) == key) ||
              (!del && ((kSplit && !up) || st.word(slot, 2 * (kDataPairs - 1)) == kEmptyKey));
      }
    }
    const uint32_t coverm = warp.ballot(cover), actm = warp.ballot(act);
    const uint32_t after  = lm & ~((2u << lane) - 1u);  // leaders above this lane
    const uint32_t mine   = (after ? (1u << (__ffs(after) - 1)) - 1u : 0xFFFFFFFFu) & ~((1u << lane) - 1u) & pm;
    bool change           = locked && (actm & mine) != 0;  // (leaders) some op changes the node
    const bool need       = change && T.versioned && nts != E;
    const uint32_t copies = warp.ballot(need);
    uint32_t copy         = kNone;
    bool dropped          = false;  // no node for the version copy: the node's ops are given up
    if (copies) {
      copy = alloc_warp(T, need, warp);
      if (need && copy == kNone) {
        dropped = true;
        change  = false;
      }
      if (locked) st.dst[slot] = copy;
      warp.sync();
      for (uint32_t s = lane >> 3; s < nodes; s += 4) {
        const uint32_t dst = st.dst[s];
        if (dst == kNone) continue;
        uint32_t w[4];
        ld_shared_4(&st.node[s][(piece ^ (s & 7u)) << 2], w[0], w[1], w[2], w[3]);
        if (piece == kModWord / 4) w[kModWord % 4] = kRetiredBit | (E & kCountMask);  // read only at snapshots < E
        store_16(T.node_ptr(dst) + piece * 4, w);
      }
      __threadfence();  // the copies are complete before a header names them
      warp.sync();
      retire_warp(T, copy != kNone, copy, warp);
    }
    const uint32_t changem = warp.ballot(change), dropm = warp.ballot(dropped);
    uint32_t fulls = 0, n = 0;  // (leaders) the ops that found the node full; its pairs
    if (change) {
      if (copy != kNone) {
        auto at = [&](uint32_t w) -> uint32_t& { return st.node[slot][(((w >> 2) ^ (slot & 7u)) << 2) | (w & 3u)]; };
        at(30)  = E;
        at(31)  = (ol & ~kIndexMask) | copy;
      }
      n = count_up_to(st, slot, kEmptyKey - 1u);
      for (uint32_t todo = coverm & mine; todo; todo &= todo - 1u) {
        const uint32_t j = (uint32_t)__ffs(todo) - 1u;
        if (!apply_staged(st, slot, n, st.op[j][0], st.op[j][1], !up && ((erases >> j) & 1u))) fulls |= 1u << j;
      }
    }
    // (leaders) the lane whose op splits the leaf, and the slot of the right half
    uint32_t cut = 32, half = 0;
    const uint32_t want = !kSplit || up ? 0u : warp.ballot(fulls != 0);
    if (want) {
      half            = nodes + (uint32_t)__popc(want & ((1u << lane) - 1u));
      const bool room = fulls != 0 && half < 32;
      const uint32_t right = alloc_warp(T, room, warp);
      if (room) {
        cut           = (uint32_t)__ffs(fulls) - 1u;
        st.idx[half]  = right;
        st.dst[half]  = right;
        fulls &= fulls - 1u;
        if (right == kNone) {  // no node: the op is given up
          cut = 32;
        } else {
          split_staged(T, st, slot, half, st.op[cut][0], st.op[cut][1], E, right);
          const uint32_t low = st.word(half, 26);
          uint32_t nr        = (uint32_t)(kDataPairs + 1 - kSplitLeft);
          n                  = (uint32_t)kSplitLeft;
          for (uint32_t todo = fulls; todo; todo &= todo - 1u) {
            const uint32_t j  = (uint32_t)__ffs(todo) - 1u;
            const bool to_right = st.op[j][0] >= low;
            if (apply_staged(st, to_right ? half : slot, to_right ? nr : n, st.op[j][0], st.op[j][1], false)) fulls &= ~(1u << j);
          }
        }
      }
      const uint32_t made = warp.ballot(cut < 32);
      if (lane == 0 && made) atomicAdd(&T.ctl->sm_stats[sm_id() % kMaxSmSlots][1], (unsigned long long)__popc(made));
      const uint32_t end = nodes + (uint32_t)__popc(want);
      warp.sync();
      store(nodes, end < 32 ? end : 32u);
      __threadfence();  // the right halves are complete before their left ones name them
      warp.sync();
    }
    if (locked) st.dst[slot] = change ? st.idx[slot] : kNone;
    warp.sync();
    store(0, nodes);
    __threadfence();
    warp.sync();
    if (locked) {
      if (change) atomicExch(mod, ((st.word(slot, kModWord) & kCountMask) + 1u) & kCountMask);
      else atomicAnd(mod, ~kLockBit);
    }
    fulls = warp.shfl(fulls, (int)boss);
    if (kSplit) {
      cut  = warp.shfl(cut, (int)boss);
      half = warp.shfl(half, (int)boss);
    }
    bool full = false, rise = false;
    if (cover) {
      if ((changem >> boss) & 1u) {
        full = (fulls >> lane) & 1u;
        rise = kSplit && cut == lane;
      } else {
        full = !((dropm >> boss) & 1u) && !del;  // an erase that found nothing is done
      }
      pend = full || rise;
    }
    if (rise) {  // the op is in; its lane goes on with the split's separator
      key   = st.word(half, 26);
      value = st.idx[half];
      leaf  = st.parent[lane];
    }
    if (kSplit) seps |= warp.ballot(rise);
    // The tile path: stale routes, separators without a parent, and one op of each full node, which splits it.
    const bool lost      = stale || (rise && (leaf == kNone || leaf == kAnchor));
    const uint32_t fullm = warp.ballot(full);
    const bool first     = full && (fullm & ((1u << lane) - 1u) & ~((1u << boss) - 1u)) == 0;
    if (lost && (rise || up)) leaf = kNone;  // a separator's way from the anchor
    for (uint32_t left = warp.ballot(lost || first); left;) {
      uint32_t m = left;
      for (uint32_t q = 0; q < lane / W; ++q) m &= m - 1u;
      const bool run     = m != 0;  // the same in every lane of a tile
      const int src      = run ? __ffs(m) - 1 : 0;
      const uint32_t k   = warp.shfl(key, src), v = warp.shfl(value, src), to = warp.shfl(leaf, src);
      if (run) {
        if (kSplit && ((seps >> src) & 1u)) push_tile<W>(T, k, v, E, to, tile);
        else write_tile<W>(T, k, v, (erases >> src) & 1u, E, to, st.parent[src], tile);
      }
      for (uint32_t q = 0; q < kTiles; ++q) left &= left - 1u;
      warp.sync();
    }
    if (lost || first) pend = false;
    warp.sync();
  }
  if (pend) T.set_error(kErrStepLimit, 11);
}

// ----------------------------------------------------------------------------------------------
// The two concurrent calls
// ----------------------------------------------------------------------------------------------
// They hand out units of up to 32 ops, one unit per warp at a time: unit u of the
// `writes + reads` units is a write unit or a read unit (Bresenham split), so both kinds run side
// by side in every wave. Returns whether it is a write unit, and its number among its kind.
MVBT_DEV bool split_unit(uint64_t u, uint64_t writes, uint64_t reads, uint64_t& number) {
  const uint64_t total = writes + reads;
  const uint64_t a = (u * writes) / total, b = ((u + 1) * writes) / total;
  number           = b > a ? a : u - a;
  return b > a;
}

// Inserts beside range queries, by the warps first, first + stride, ..: writes run by the warp (write_warp);
// range queries at snapshot S by the warp (range_warp), those of a plain tree's newest state (S = kLatest) a
// tile per query from their leaves. slow: the tile of kSlow lanes that writes fall back to.
template <int W, int kSlow, class Warp, class Tile, class Slow>
MVBT_DEV void insert_range_units(const device_tree& T, const uint32_t* keys, const uint32_t* values, uint32_t n_ins,
                                 const uint32_t* lower, const uint32_t* upper, uint32_t n_rq, uint2* result,
                                 uint32_t avg_len, uint32_t* counts, uint32_t lanes, uint32_t S, uint64_t first,
                                 uint64_t stride, write_stage& st, const Warp& warp, const Tile& tile, const Slow& slow) {
  const uint32_t lane   = warp.thread_rank();
  const bool ver        = T.versioned != 0;
  const uint32_t E      = ver ? S + 1 : 0u;
  const uint64_t writes = ((uint64_t)n_ins + lanes - 1) / lanes, reads = ((uint64_t)n_rq + lanes - 1) / lanes;
  for (uint64_t u = first; u < writes + reads; u += stride) {
    uint64_t number;
    const bool write   = split_unit(u, writes, reads, number);
    const uint64_t i   = number * lanes + lane;
    const bool has     = lane < lanes && i < (write ? n_ins : n_rq);
    const uint32_t key = has ? (write ? keys[i] : lower[i]) : kEmptyKey;
    const uint32_t leaf = leaf_warp(T, key, has && key != kEmptyKey, kAnchor, nullptr, st, warp);
    if (write) {
      write_warp<kSlow>(T, key, has ? values[i] : 0u, false, has, E, leaf, st, warp, slow);
    } else {
      const uint32_t at = leaf == kNone ? kAnchor : leaf;
      if (ver) {
        uint2* out       = result ? result + i * (uint64_t)avg_len : nullptr;
        const uint32_t c = range_warp<true>(T, key, has ? upper[i] : 0u, has, S, out, avg_len, at, nullptr, st, warp);
        if (counts && has) counts[i] = c;
        continue;
      }
      for_lanes<W>(warp.ballot(has), warp, [&](bool run, int src) {
        const uint32_t lo = warp.shfl(key, src), from = warp.shfl(at, src);
        if (run) {
          const uint64_t r = number * lanes + src;
          uint2* out       = result ? result + r * (uint64_t)avg_len : nullptr;
          const uint32_t c = T.cooperative_range_query<W>(lo, upper[r], tile, S, out, avg_len, true, from);
          if (counts && tile.thread_rank() == 0) counts[r] = c;
        }
      });
    }
  }
}

// Erases beside finds likewise: finds at snapshot S by the warp (find_warp_live), finds of a plain tree's newest
// state a tile per key from their leaves.
template <int W, int kSlow, class Warp, class Tile, class Slow>
MVBT_DEV void find_erase_units(const device_tree& T, const uint32_t* fkeys, uint32_t* fres, uint32_t n_find,
                               const uint32_t* ekeys, uint32_t n_erase, uint32_t lanes, uint32_t S, uint64_t first,
                               uint64_t stride, write_stage& st, const Warp& warp, const Tile& tile, const Slow& slow) {
  const uint32_t lane   = warp.thread_rank();
  const bool ver        = T.versioned != 0;
  const uint32_t E      = ver ? S + 1 : 0u;
  const uint64_t writes = ((uint64_t)n_erase + lanes - 1) / lanes, reads = ((uint64_t)n_find + lanes - 1) / lanes;
  for (uint64_t u = first; u < writes + reads; u += stride) {
    uint64_t number;
    const bool write   = split_unit(u, writes, reads, number);
    const uint64_t i   = number * lanes + lane;
    const bool has     = lane < lanes && i < (write ? n_erase : n_find);
    const uint32_t key = has ? (write ? ekeys[i] : fkeys[i]) : kEmptyKey;
    const uint32_t leaf = leaf_warp(T, key, has && key != kEmptyKey, kAnchor, nullptr, st, warp);
    const uint32_t at   = leaf == kNone ? kAnchor : leaf;
    if (write) {
      write_warp<kSlow>(T, key, 0u, true, has, E, leaf, st, warp, slow);
    } else if (ver) {
      const uint32_t v = find_warp_live(T, key, has, S, at, st, warp);
      if (has) fres[i] = v;
    } else {
      for_lanes<W>(warp.ballot(has), warp, [&](bool run, int src) {
        const uint32_t k = warp.shfl(key, src), from = warp.shfl(at, src);
        if (run) {
          const uint32_t v = T.cooperative_find<W>(k, tile, S, true, from);
          if (tile.thread_rank() == 0) fres[number * lanes + src] = v;
        }
      });
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Mixed operation batches
//
// A batch is a list of ops {type, key, arg}: find (arg unused), insert (arg = value), erase, and
// range query (arg = exclusive upper bound, output slot at range_out + out_off[i] holding at most
// cap[i] pairs). One snapshot per batch: batch b reads at snapshot S0 + b and writes in epoch
// S0 + b + 1, so every result is that of the batch applied after all earlier batches. The
// reference issues each op kind of a batch as its own host launch
// (include/gpu_versioned_blink_tree.hpp:106-216); here a batch is one launch, or many batches
// are one persistent launch.
// ----------------------------------------------------------------------------------------------
enum : uint32_t { kOpFind = 0, kOpInsert = 1, kOpErase = 2, kOpRange = 3 };

struct batch_view {
  const uint32_t* type;
  const uint32_t* key;
  const uint32_t* arg;
  const uint64_t* out_off;  // range output offset, pairs
  const uint32_t* cap;      // range output capacity, pairs
  uint32_t* result;         // find value or range count (0 for writes)
  uint2* range_out;
};

MVBT_DEV bool is_write_op(uint32_t type) { return type == kOpInsert || type == kOpErase; }

// Schedule of the persistent batched launch. Within each batch the claim order puts writes first
// (perm maps a claim position to an op index). Writes of batch b may start once every write of
// the batches before b has finished, reads of batch b likewise (they read the state after those
// writes; writes of b and later batches go into newer versions, so the reads may lag behind).
// Two device queues hand out work: write ordinals (the critical path, small claims, served first)
// and read ordinals (larger claims, taken when no write is ready). done_batches counts the leading
// batches whose writes are all finished.
struct batch_sched {
  const uint64_t* batch_off;     // [nb + 1] claim positions of each batch
  const uint32_t* perm;          // claim position -> op index
  const uint32_t* n_writes;      // [nb] writes per batch
  const uint64_t* wpre;          // [nb + 1] first write ordinal of each batch
  const uint64_t* rpre;          // [nb + 1] first read ordinal of each batch
  uint32_t* writes_done;         // [nb] finished writes (zero at launch)
  uint32_t* done_batches;        // zero at launch
  unsigned long long* wcursor;   // next write ordinal (zero at launch)
  unsigned long long* rcursor;   // next read ordinal (zero at launch)
  const uint32_t* params;        // [0] num_batches, [1] snapshot of batch 0, [2] external watermark
  // Reclamation inside the launch (all null: off). A copy made in epoch E is read only at
  // snapshots below E; batch b writes in epoch S0 + b + 1 and reads at S0 + b. So once batches
  // 0..b have finished their writes and their reads, the copies batch b and earlier made (all at
  // retire-log positions below the log tail read when batch b's writes had finished) are read by
  // no snapshot of this launch; params[2] is the caller's watermark: the oldest snapshot it still
  // reads outside the launch (copies made in later epochs are kept; kReclaimAll: none held).
  uint32_t* reads_done            = nullptr;  // [nb] finished reads (zero at launch)
  uint32_t* full_done             = nullptr;  // leading batches with writes and reads all finished
  unsigned long long* tail_at     = nullptr;  // [nb] log tail once batch b's writes finished (~0: not yet)
  unsigned long long* rc_limit    = nullptr;  // log positions below it are reclaimable
  unsigned long long* series      = nullptr;  // [nb][4] when batch b's writes finished: epoch, bump,
                                              // free_avail, stat_reclaimed (memory over time)
};

constexpr uint32_t kWriteClaims  = 128; // claims a batch's writes are cut into at least, while lanes last
constexpr uint32_t kReadClaims   = 4;   // claims of reads per warp of the launch likewise
constexpr uint32_t kPollNs       = 400; // how often a block looks at done_batches while its warps wait
constexpr uint32_t kPatienceNs   = 50000; // how long reads wait for a chain that stands still (a link takes 20-35 us)
constexpr uint32_t kAdvanceEvery = 64;  // a look in 64 also advances the batch chain

// Largest b in [lo, nb) with pre[b] <= x (pre is non-decreasing), starting from the hint lo.
MVBT_DEV uint32_t batch_of_ordinal(const uint64_t* pre, uint32_t nb, uint64_t x, uint32_t lo) {
  if (lo >= nb) lo = 0;
  if (pre[lo] > x) lo = 0;
  if (lo + 1 < nb && pre[lo + 1] > x) return lo;
  uint32_t hi = nb;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Advances done_batches past every leading batch whose writes are all finished (lane 0 only). With
// reclamation on, the thread that advances past batch d records the retire-log tail (read after
// d's writes finished and before any write of d + 1 can start) and a memory sample.
MVBT_DEV void advance_done(const batch_sched& sc, uint32_t nb, control_block* ctl = nullptr) {
  uint32_t d = ld_relaxed_u32(sc.done_batches);
  while (d < nb) {
    if (ld_relaxed_u32(&sc.writes_done[d]) < sc.n_writes[d]) break;
    __threadfence();
    const unsigned long long tail = (sc.tail_at && ctl) ? ld_relaxed_u64(&ctl->retire_tail) : 0ull;
    uint32_t prev = atomicCAS(sc.done_batches, d, d + 1);
    if (prev == d && sc.tail_at && ctl) {
      if (sc.series) {
        unsigned long long* e = sc.series + 4ull * d;
        e[0] = ld_relaxed_u32(sc.params + 1) + d + 1u;
        e[1] = ld_relaxed_u32(&ctl->bump);
        // a chunk taker's reservation on free_avail is undone when fewer entries are there, so
        // the word can dip below zero for a moment: recorded as none free
        const unsigned long long fa = ld_relaxed_u64(&ctl->free_avail);
        e[2] = (long long)fa < 0 ? 0ull : fa;
        e[3] = ld_relaxed_u64(&ctl->stat_reclaimed);
      }
      atomicExch(&sc.tail_at[d], tail);
    }
    d = (prev == d) ? d + 1 : prev;
  }
}

// Reclamation on: advances full_done past every leading batch whose writes and reads are all
// finished and raises rc_limit to the log tail recorded for it (lane 0 only).
MVBT_DEV void advance_full(const batch_sched& sc, uint32_t nb) {
  uint32_t f       = ld_relaxed_u32(sc.full_done);
  const uint32_t d = ld_relaxed_u32(sc.done_batches);
  const uint32_t S0 = ld_relaxed_u32(sc.params + 1), ext = ld_relaxed_u32(sc.params + 2);
  while (f < d && f < nb) {
    const uint32_t reads = (uint32_t)(sc.batch_off[f + 1] - sc.batch_off[f]) - sc.n_writes[f];
    if (ld_relaxed_u32(&sc.reads_done[f]) < reads) break;
    __threadfence();
    const unsigned long long t = ld_relaxed_u64(&sc.tail_at[f]);
    if (t == ~0ull) break;  // its writes' advancer has not recorded the tail yet
    const uint32_t prev = atomicCAS(sc.full_done, f, f + 1);
    if (prev == f) {
      // batch f's copies were made in epoch S0 + f + 1: free only at or below the watermark
      if (ext == kReclaimAll || S0 + f + 1u <= ext) atomicMax(sc.rc_limit, t);
      ++f;
    } else {
      f = prev;
    }
  }
}

// Whether writes of the window that warps claim from (the batch after the finished ones, and the next) are left.
MVBT_DEV bool writes_to_claim(const batch_sched& sc, uint32_t nb) {
  const uint32_t d = ld_relaxed_u32(sc.done_batches);
  return ld_relaxed_u64(sc.wcursor) < sc.wpre[d + 2 < nb ? d + 2 : nb];
}

// What the warps of a block last saw of done_batches, and when one of them looked (ns, low 32 bits).
struct batch_gate {
  uint32_t done;
  uint32_t looked;
};

// Reads that a warp has claimed and holds back: in shared memory, the worker has no registers to spare.
struct held_reads {
  unsigned long long first;  // their claim
  uint32_t lanes;            // the lanes still to run (0: none held)
};

enum : uint32_t { kWaiting = 0, kReady = 1, kTimedOut = 2, kWritesLeft = 3 };

// Waits (bounded: as long as done_batches moves within the wait limit) until the writes of every batch before
// b have finished. reads: the caller waits with reads, and is told kWritesLeft if done_batches stands still
// for kPatienceNs while writes of the next two batches are left to claim, which it then has to take.
// Thousands of warps can wait at once for one word on one L2 slice. So one warp of a block at a time
// looks at it, every kPollNs, and the others read what it saw in shared memory: 592 blocks then
// read the word about once a nanosecond, where a read per warp and half microsecond queued for longer
// than the write phase that was waited for.
template <class Warp>
MVBT_DEV uint32_t wait_batch_ready(const device_tree& T, const batch_sched& sc, uint32_t nb, uint32_t b, bool reads,
                                   batch_gate& gate, const Warp& warp) {
  unsigned long long t0 = global_ns();  // of the start, or of the last move seen
  uint32_t seen         = 0;
  for (uint32_t w = 0;; ++w) {
    uint32_t state = kWaiting;
    if (warp.thread_rank() == 0) {
      uint32_t d = ld_block_u32(&gate.done);
      if (d < b) {
        const uint32_t now = (uint32_t)global_ns(), last = ld_block_u32(&gate.looked);
        if (now - last >= kPollNs && atomicCAS(&gate.looked, last, now) == last) {
          if (w % kAdvanceEvery == kAdvanceEvery - 1) advance_done(sc, nb, T.ctl);
          d = ld_acquire_u32(sc.done_batches);  // the writes counted in d come before it, and
          __threadfence_block();                // before the word that the other warps see
          atomicMax(&gate.done, d);
        }
      }
      const unsigned long long now = global_ns();
      if (d >= b) {
        state = kReady;
      } else if (d > seen) {
        seen = d;
        t0   = now;
      } else if (now - t0 > T.ctl->wait_ns) {
        state = kTimedOut;
      } else if (reads && now - t0 > kPatienceNs && w % 8 == 7 && writes_to_claim(sc, nb)) {
        state = kWritesLeft;
      }
    }
    state = warp.shfl(state, 0);
    if (state != kWaiting) {
      __threadfence();
      warp.sync();
      return state;
    }
    __nanosleep(kPollNs / 4);
  }
}

// One step of reclamation inside the launch (warp-collective): advances full_done, then frees up to
// kReclaimClaim copies below rc_limit. Returns true if it claimed any log position.
template <class Warp>
MVBT_DEV bool reclaim_step(const device_tree& T, const batch_sched& sc, uint32_t nb, const Warp& warp) {
  unsigned long long lim = 0;
  if (warp.thread_rank() == 0) {
    advance_full(sc, nb);
    lim = ld_relaxed_u64(sc.rc_limit);
  }
  lim = warp.shfl(lim, 0);
  return T.reclaim_online(lim, warp) > 0;
}
// At the end of a warp's work: one more reclamation step, then leave. The
// copies the last batches made become reclaimable only when their last reads finish, at the very
// end of the launch, when few warps are left; draining them there would stretch the launch, so
// they wait for the next launch, whose warps free them from its start while work runs.
template <class Warp>
MVBT_DEV void reclaim_drain(const device_tree& T, const batch_sched& sc, uint32_t nb, const Warp& warp) {
  if (warp.thread_rank() == 0) advance_done(sc, nb, T.ctl);
  reclaim_step(T, sc, nb, warp);
}

// Runs the ops of the lanes with `live` set (op index i, key, and its leaf as leaf_warp found it), all
// of one batch or at least of one snapshot S: writes and finds by the warp, range queries by its
// tiles. Results go to B.result.
template <int W, class Warp, class Tile>
MVBT_DEV void run_ops_warp(const device_tree& T, const batch_view& B, uint64_t i, uint32_t type, uint32_t key,
                           bool live, uint32_t S, uint32_t leaf, write_stage& st, const Warp& warp, const Tile& tile) {
  constexpr uint32_t kTiles = 32 / W;
  const uint32_t at  = leaf == kNone ? kAnchor : leaf;
  const bool write   = live && is_write_op(type);
  if (warp.ballot(write)) {
    const uint32_t value = write && type == kOpInsert ? B.arg[i] : 0u;
    write_warp<W>(T, key, value, type == kOpErase, write, S + 1, leaf, st, warp, tile);
  }
  const bool find = live && type == kOpFind;
  uint32_t r      = 0;
  if (warp.ballot(find)) {
    const uint32_t v = find_warp_live(T, key, find, S, at, st, warp);
    if (find) r = v;
  }
  const bool range = live && type == kOpRange;
  if (live && !range) B.result[i] = r;
  for (uint32_t left = warp.ballot(range); left;) {
    uint32_t m = left;
    for (uint32_t q = 0; q < warp.thread_rank() / W; ++q) m &= m - 1u;
    const bool run     = m != 0;  // the same in every lane of a tile
    const int src      = run ? __ffs(m) - 1 : 0;
    const uint64_t op  = warp.shfl(i, src);
    const uint32_t lo  = warp.shfl(key, src), from = warp.shfl(at, src);
    if (run) {
      uint2* out       = B.range_out ? B.range_out + B.out_off[op] : nullptr;
      const uint32_t c = T.cooperative_range_query<W>(lo, B.arg[op], tile, S, out, B.cap[op], true, from);
      if (tile.thread_rank() == 0) B.result[op] = c;
    }
    for (uint32_t q = 0; q < kTiles; ++q) left &= left - 1u;
    warp.sync();
  }
}

// One batch [begin, end) at snapshot S, `lanes` ops to a warp at a time, by the warps first, first + stride, ..
template <int W, class Warp, class Tile>
MVBT_DEV void mixed_ops(const device_tree& T, const batch_view& B, uint64_t begin, uint64_t end, uint32_t lanes, uint32_t S,
                        uint64_t first, uint64_t stride, write_stage& st, const Warp& warp, const Tile& tile) {
  const uint32_t lane = warp.thread_rank();
  for (uint64_t g = begin + first * lanes; g < end; g += stride * lanes) {
    const uint64_t i    = g + lane;
    const bool has      = lane < lanes && i < end;
    const uint32_t type = has ? B.type[i] : (uint32_t)kOpFind, key = has ? B.key[i] : kEmptyKey;
    const uint32_t leaf = leaf_warp(T, key, has && key != kEmptyKey, kAnchor, nullptr, st, warp);
    run_ops_warp<W>(T, B, i, type, key, has, S, leaf, st, warp, tile);
  }
}

// Ops a warp claims at once: a full warp's worth, less when there would be fewer than `share` claims (0 for a list
// without batches, such as rejected offsets leave).
MVBT_DEV uint32_t claim_size(uint64_t ops, uint64_t share, uint32_t least) {
  const uint64_t c = share ? ops / share : 0;
  return c >= 32 ? 32u : (c < least ? least : (uint32_t)c);
}

// Worker loop of one warp in the persistent batched launch. The warp claims consecutive claim
// positions, one per lane; all its lanes descend together (leaf_warp), then the lanes of each batch,
// in order, wait for it and run (run_ops_warp). warps: how many the launch has; gate: the block's; held: the
// warp's.
// No warp waits for good for a write that no warp has claimed: claims of writes wait for the writes before
// them, which were claimed before them. A claim of reads may reach far past the window below, and so may
// those of all warps at once; if writes of the window are left meanwhile (wait_batch_ready), the warp holds
// its reads, takes writes, and comes back to them when there are none to take.
template <int W, class Warp, class Tile>
MVBT_DEV void batched_worker(const device_tree& T, const batch_view& B, const batch_sched& sc, uint32_t warps,
                             batch_gate& gate, held_reads& held, write_stage& st, const Warp& warp, const Tile& tile) {
  constexpr uint32_t kTiles = 32 / W;
  const uint32_t lane = warp.thread_rank();
  const uint32_t nb   = ld_relaxed_u32(sc.params + 0);
  const uint32_t S0   = ld_relaxed_u32(sc.params + 1);
  const uint64_t TW = sc.wpre[nb], TR = sc.rpre[nb];
  const uint32_t wclaim = claim_size(TW, (uint64_t)nb * kWriteClaims, kTiles);
  const uint32_t rclaim = claim_size(TR, (uint64_t)warps * kReadClaims, kTiles);
  uint32_t wb = 0, rb = 0;  // batch hints for the two queues
  unsigned long long idle_since = 0;
  if (lane == 0) held.lanes = 0;
  for (uint32_t spin = 0;;) {
    warp.sync();
    uint32_t d = 0;
    unsigned long long g = 0, r = 0;
    if (lane == 0) {
      d = ld_relaxed_u32(sc.done_batches);
      g = ld_relaxed_u64(sc.wcursor);
      r = ld_relaxed_u64(sc.rcursor);
    }
    d = warp.shfl(d, 0);
    g = warp.shfl(g, 0);
    r = warp.shfl(r, 0);
    const uint32_t back = held.lanes;
    if (g >= TW && r >= TR && !back) {
      // all work is claimed: help reclaim what the finished batches no longer need, then leave
      if (sc.rc_limit) reclaim_drain(T, sc, nb, warp);
      break;
    }
    __threadfence();  // the batches counted in d are finished: see their writes
    warp.sync();
    // Writes first: they gate every later batch. Work is taken up to one batch past the finished
    // ones; the ops of a batch that is not ready do their descent, then wait.
    bool writes = false, reads = false;
    if (g < TW) {
      wb     = batch_of_ordinal(sc.wpre, nb, g, wb);
      writes = wb <= d + 1;
    }
    if (!writes && back) {
      reads = true;
    } else if (!writes && r < TR) {
      rb    = batch_of_ordinal(sc.rpre, nb, r, rb);
      reads = rb <= d + 1;
    }
    bool did = false;
    if (writes || reads) {
      const uint32_t claim     = writes ? wclaim : rclaim;
      const uint64_t total     = writes ? TW : TR;
      const uint64_t* pre      = writes ? sc.wpre : sc.rpre;
      const bool resume        = reads && back;
      unsigned long long first = 0;
      if (resume) {
        first = held.first;
      } else {
        if (lane == 0) first = atomicAdd(writes ? sc.wcursor : sc.rcursor, (unsigned long long)claim);
        first = warp.shfl(first, 0);
      }
      did = first < total;
      const unsigned long long x = first + lane;
      const bool has             = resume ? (back >> lane) & 1u : lane < claim && x < total;
      bool hold                  = false;
      uint32_t b = nb, type = kOpFind, key = kEmptyKey;
      uint64_t i = 0;
      if (has) {
        b    = batch_of_ordinal(pre, nb, x, writes ? wb : rb);
        i    = sc.perm[sc.batch_off[b] + (writes ? 0u : sc.n_writes[b]) + (x - pre[b])];
        type = B.type[i];
        key  = B.key[i];
      }
      const uint32_t leaf = leaf_warp(T, key, has && key != kEmptyKey, kAnchor, nullptr, st, warp);
      uint32_t ready      = d;
      for (uint32_t left = warp.ballot(has); left;) {
        const uint32_t now = warp.shfl(b, __ffs(left) - 1);  // the first batch left
        const uint32_t cur = warp.ballot(has && b == now);
        if (now > ready) {
          const uint32_t state = wait_batch_ready(T, sc, nb, now, reads, gate, warp);
          if (state == kWritesLeft) {
            if (lane == 0) held = held_reads{first, left};
            hold = true;
            break;
          }
          if (state == kTimedOut && lane == 0) T.set_error(kErrSpinLimit, 14);
          ready = now;
        }
        run_ops_warp<W>(T, B, i, type, key, has && b == now, S0 + now, leaf, st, warp, tile);
        // The warp whose writes complete a batch advances done_batches. No fence before the count: every
        // write path ends with the fence of its last release or unlock, which orders its stores before
        // it. Reads: their loads are complete before they are counted.
        if (!writes && sc.reads_done) __threadfence();
        warp.sync();
        if (lane == 0) {
          const uint32_t n = (uint32_t)__popc(cur);
          if (!writes) {
            if (sc.reads_done) atomicAdd(&sc.reads_done[now], n);
          } else if (atomicAdd(&sc.writes_done[now], n) + n >= sc.n_writes[now]) {
            advance_done(sc, nb, T.ctl);
          }
        }
        left &= ~cur;
      }
      if (lane == 0 && resume && !hold) held.lanes = 0;
      // Reclamation keeps pace with copying even when no warp is ever idle: a step after each claim of
      // reads, which nothing waits for, and after a claim of writes only if their batch has more of them
      // than reads (the next batch waits for them). A step takes 64 copies, two for each op of a full claim, so
      // either kind keeps up with the copies of its batch.
      if (did && sc.rc_limit) {
        const bool more = has && writes && 2ull * sc.n_writes[b] > sc.batch_off[b + 1] - sc.batch_off[b];
        if (warp.ballot(reads || more)) reclaim_step(T, sc, nb, warp);
      }
    }
    if (did) {
      spin       = 0;
      idle_since = 0;
      continue;
    }
    // nothing runnable yet: help advance done_batches, reclaim, then back off (bounded)
    if (lane == 0) advance_done(sc, nb, T.ctl);
    if (sc.rc_limit && reclaim_step(T, sc, nb, warp)) {
      spin       = 0;
      idle_since = 0;
      continue;
    }
    if (idle_since == 0) idle_since = global_ns();
    if (wait_expired(idle_since, T.ctl->wait_ns, warp)) {
      if (lane == 0) T.set_error(kErrSpinLimit, 14);
      break;
    }
    __nanosleep(spin < 8 ? 256 : 2048);
    ++spin;
  }
}

}  // namespace mvbt
