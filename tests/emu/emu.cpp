// CPU emulation harness for the device tree (test infrastructure).
//
// Compiles include/mvbt_device.cuh for the host (MVBT_HOST_EMULATION) and runs every W-lane tile
// as W host threads: shfl / ballot / sync go through a per-tile exchange buffer and a barrier,
// atomics are GCC atomics on the shared pool. Several tiles run at once, so the lock, split and
// versioning protocols are exercised concurrently on the CPU before any GPU run.
#undef _FORTIFY_SOURCE  // its longjmp takes a jump to another stack for an error
#define MVBT_HOST_EMULATION 1
#include <setjmp.h>
#include <ucontext.h>

#include <barrier>
#include <cstdint>
#include <cstring>
#include <functional>
#include <memory>
#include <thread>
#include <vector>

#include "mvbt.h"
#include "mvbt_device.cuh"

namespace {

// The lanes of an emulated warp (run_warps) are contexts of one host thread that switch where they
// wait, which costs a fraction of 32 host threads meeting in a barrier.
struct fibers {
  ucontext_t ctx[32];      // how a lane starts; it goes on by longjmp, which needs no system call
  jmp_buf home, at[32];
  bool started[32], done[32];
  std::vector<char> stack[32];
  std::function<void(int)> body;
  int lane = 0;
  void yield() {
    if (_setjmp(at[lane]) == 0) _longjmp(home, 1);
  }
  void enter(int l) {
    lane = l;
    if (_setjmp(home) != 0) return;
    if (started[l]) _longjmp(at[l], 1);
    started[l] = true;
    setcontext(&ctx[l]);
  }
  static void entry(unsigned lo, unsigned hi) {
    auto* f = reinterpret_cast<fibers*>((uintptr_t)lo | ((uintptr_t)hi << 32));
    f->body(f->lane);
    f->done[f->lane] = true;
    f->yield();
  }
  void run(std::function<void(int)> fn) {
    body = std::move(fn);
    const uintptr_t self = reinterpret_cast<uintptr_t>(this);
    for (int l = 0; l < 32; ++l) {
      started[l] = done[l] = false;
      stack[l].resize(256 << 10);
      getcontext(&ctx[l]);
      ctx[l].uc_stack.ss_sp   = stack[l].data();
      ctx[l].uc_stack.ss_size = stack[l].size();
      ctx[l].uc_link          = nullptr;  // a finished lane yields for good
      makecontext(&ctx[l], reinterpret_cast<void (*)()>(&entry), 2, (unsigned)self, (unsigned)(self >> 32));
    }
    for (volatile int left = 32; left > 0;)
      for (volatile int l = 0; l < 32; ++l)
        if (!done[l]) {
          enter(l);
          if (done[l]) left = left - 1;
        }
  }
};

struct tile_shared {
  std::barrier<> bar;
  uint64_t slot[32];
  fibers* fib = nullptr;  // the lanes are contexts of one thread
  std::barrier<>* meet = nullptr;  // the other warps, to be met at this tile's meet_at-th shuffle
  int meet_at = 0, shuffles = 0;
  int width, arrived = 0;
  unsigned generation = 0;
  explicit tile_shared(int w) : bar(w), width(w) {}
  void sync() {
    if (!fib) {
      bar.arrive_and_wait();
      return;
    }
    const unsigned mine = generation;
    if (++arrived == width) {
      arrived = 0;
      ++generation;
      return;
    }
    while (generation == mine) fib->yield();
  }
};

// Emulated cooperative-groups tile of W lanes.
struct emu_tile {
  int rank;
  int W;
  tile_shared* sh;
  int thread_rank() const { return rank; }
  void sync() const { sh->sync(); }
  template <class T>
  T shfl(T v, int src) const {
    sh->slot[rank] = (uint64_t)v;
    if (rank == 0 && sh->meet && ++sh->shuffles == sh->meet_at) sh->meet->arrive_and_wait();
    sync();
    T r = (T)sh->slot[((src % W) + W) % W];
    sync();
    return r;
  }
  unsigned ballot(int p) const {
    sh->slot[rank] = p ? 1u : 0u;
    sync();
    unsigned m = 0;
    for (int i = 0; i < W; ++i)
      if (sh->slot[i]) m |= 1u << i;
    sync();
    return m;
  }
};

struct emu_tree {
  std::vector<uint32_t> pool;
  std::vector<uint32_t> retire_log, free_ring;  // reclamation on
  mvbt::control_block ctl;
  uint32_t capacity;
  int versioned;
  mvbt::device_tree view() {
    mvbt::device_tree t;
    t.pool      = pool.data();
    t.ctl       = &ctl;
    t.versioned = (uint32_t)versioned;
    t.capacity  = capacity;
    t.reclaim   = retire_log.empty() ? 0u : 1u;
    return t;
  }
};

// Runs op(i, tile) for i in [0, n) over `tiles` concurrent tiles of W threads (grid-stride).
void run(uint64_t n, int tiles, int W, const std::function<void(uint64_t, const emu_tile&)>& op) {
  if (n == 0) return;
  if (tiles < 1) tiles = 1;
  std::vector<std::unique_ptr<tile_shared>> sh;
  for (int t = 0; t < tiles; ++t) sh.emplace_back(new tile_shared(W));
  std::vector<std::thread> th;
  for (int t = 0; t < tiles; ++t) {
    for (int l = 0; l < W; ++l) {
      th.emplace_back([&, t, l] {
        mvbt::emu::sm = (uint32_t)t;
        emu_tile tile{l, W, sh[t].get()};
        for (uint64_t i = (uint64_t)t; i < n; i += (uint64_t)tiles) op(i, tile);
      });
    }
  }
  for (auto& x : th) x.join();
}

// Runs fn(warp, tile) on `warps` emulated warps of 32 threads, each split into tiles of W lanes. meet_at > 0:
// no warp goes past its meet_at-th shuffle before all have come to theirs.
void run_warps(int warps, int W, const std::function<void(const emu_tile&, const emu_tile&)>& fn, int meet_at = 0) {
  if (warps < 1) warps = 1;
  const int tpw = 32 / W;
  std::vector<std::unique_ptr<tile_shared>> wsh, tsh;
  std::barrier<> meet(warps);
  for (int w = 0; w < warps; ++w) {
    wsh.emplace_back(new tile_shared(32));
    if (meet_at) wsh.back()->meet = &meet, wsh.back()->meet_at = meet_at;
    for (int j = 0; j < tpw; ++j) tsh.emplace_back(new tile_shared(W));
  }
  std::vector<std::thread> th;
  for (int w = 0; w < warps; ++w) {
    th.emplace_back([&, w] {
      mvbt::emu::sm = (uint32_t)w;
      auto f        = std::make_unique<fibers>();
      wsh[w]->fib   = f.get();
      for (int j = 0; j < tpw; ++j) tsh[w * tpw + j]->fib = f.get();
      f->run([&](int l) {
        emu_tile warp{l, 32, wsh[w].get()};
        emu_tile tile{l % W, W, tsh[w * tpw + l / W].get()};
        fn(warp, tile);
      });
    });
  }
  for (auto& x : th) x.join();
}

}  // namespace

extern "C" {

void* emu_create(int versioned, uint32_t capacity, uint32_t spin_limit, uint32_t chunk, int reclaim) {
  auto* t      = new emu_tree();
  t->capacity  = capacity;
  t->versioned = versioned;
  t->pool.assign((size_t)capacity * 32, 0xA5A5A5A5u);  // garbage, as fresh cudaMalloc memory
  for (int i = 0; i < 32 * mvbt::kInitialNodes; ++i) t->pool[i] = mvbt::initial_tree_word(i);
  chunk             = chunk ? chunk : 8;
  uint32_t log_cap  = 0, ring_cap = 0;
  if (reclaim) {  // the same power-of-two sizes as the library
    auto pow2 = [](uint64_t x) {
      uint64_t p = 1;
      while (p < x) p <<= 1;
      return (uint32_t)p;
    };
    log_cap  = pow2(capacity);
    ring_cap = pow2((uint64_t)capacity + (uint64_t)mvbt::kMaxSmSlots * chunk);
    t->retire_log.assign(log_cap, 0xFFFFFFFFu);  // both start empty, as mvbt_create fills them
    t->free_ring.assign(ring_cap, 0xFFFFFFFFu);
  }
  mvbt::init_control(t->ctl, capacity, chunk, spin_limit ? spin_limit : (1u << 20), 4000u * 1000u * 1000u,
                     reclaim ? (unsigned long long)t->retire_log.data() : 0ull,
                     reclaim ? (unsigned long long)t->free_ring.data() : 0ull, log_cap, ring_cap);
  return t;
}

// A reclaim pass, as mvbt_reclaim runs it (k_reclaim + k_reclaim_finish), single-threaded.
void emu_reclaim(void* h, uint32_t M) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  auto& c = t->ctl;
  if (M == mvbt::kReclaimAll) M = c.epoch;
  const unsigned long long head = c.retire_head;
  const unsigned long long n    = std::min<unsigned long long>(c.retire_tail - head, c.reclaim_cap);
  uint32_t* ring                = reinterpret_cast<uint32_t*>(c.free_ring);
  for (unsigned long long i = 0; i < n; ++i) {
    uint32_t idx = 0;
    const int r  = v.reclaim_entry(head + i, M, idx);
    if (r == 1) {  // the ring push of one lane: reserve, write, publish
      ring[c.free_tail++ & (c.ring_cap - 1u)] = idx;
      c.free_avail += 1;
      c.stat_reclaimed += 1;
    }
    if (r == 2) c.rc_first_kept = std::min<uint32_t>(c.rc_first_kept, (uint32_t)i);
  }
  v.reclaim_publish();
}

void emu_destroy(void* h) { delete static_cast<emu_tree*>(h); }

uint32_t emu_errors(void* h) { return static_cast<emu_tree*>(h)->ctl.error; }
uint32_t emu_bump(void* h) { return static_cast<emu_tree*>(h)->ctl.bump; }
void emu_stats(void* h, uint64_t* out) {
  auto& c = static_cast<emu_tree*>(h)->ctl;
  out[0] = mvbt::stat_total(c, 0);
  out[1] = mvbt::stat_total(c, 1);
  out[2] = c.stat_max_hops;
  out[3] = c.stat_max_steps;
  for (int i = 0; i < 16; ++i) out[4 + i] = c.err_site[i];
  out[20] = c.stat_restarts;
  out[21] = c.reclaim_cap ? c.retire_tail : mvbt::stat_total(c, 0);
  out[22] = c.stat_reclaimed;
  out[23] = c.reclaim_cap ? (uint64_t)std::max<long long>(0, (long long)c.free_avail) : 0;
  out[24] = mvbt::stat_total(c, 2);
  out[25] = c.stat_log_dropped;
}

// Locks (on != 0) or releases the first leaf from outside, as a writer that holds it for long would.
void emu_hold_first_leaf(void* h, int on) {
  uint32_t* mod = &static_cast<emu_tree*>(h)->pool[32 * mvbt::kFirstLeaf + mvbt::kModWord];
  if (on) __atomic_fetch_or(mod, mvbt::kLockBit, __ATOMIC_SEQ_CST);
  else __atomic_fetch_and(mod, ~mvbt::kLockBit, __ATOMIC_SEQ_CST);
}

// Lets the emulated clock run `by` times slower: a wait then looks about as often as on the GPU before its
// limit has passed.
void emu_slow_clock(uint32_t by) { mvbt::emu::slow.store(by ? by : 1u); }

uint32_t emu_snapshot(void* h) {
  auto* t = static_cast<emu_tree*>(h);
  return __atomic_fetch_add(&t->ctl.epoch, 1u, __ATOMIC_SEQ_CST);
}

#define EMU_DISPATCH(W, BODY)                    \
  if (W == 8) {                                  \
    constexpr int kW = 8;                        \
    BODY;                                        \
  } else {                                       \
    constexpr int kW = 16;                       \
    BODY;                                        \
  }

void emu_insert(void* h, const uint32_t* keys, const uint32_t* vals, uint64_t n, int tiles, int W) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  EMU_DISPATCH(W, run(n, tiles, kW, [&](uint64_t i, const emu_tile& tile) {
    uint32_t E = v.versioned ? v.current_epoch() : 0u;
    v.cooperative_insert<kW>(keys[i], vals[i], tile, E);
  }));
}

void emu_erase(void* h, const uint32_t* keys, uint64_t n, int tiles, int W) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  EMU_DISPATCH(W, run(n, tiles, kW, [&](uint64_t i, const emu_tile& tile) {
    uint32_t E = v.versioned ? v.current_epoch() : 0u;
    v.cooperative_erase<kW>(keys[i], tile, E);
  }));
}

// quiescent != 0: the lookup of a tree no writer changes meanwhile (find_quiescent).
void emu_find(void* h, const uint32_t* keys, uint32_t* out, uint64_t n, uint32_t ts, int tiles, int W,
              int quiescent) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  if (!v.versioned) ts = mvbt::kLatest;
  EMU_DISPATCH(W, run(n, tiles, kW, [&](uint64_t i, const emu_tile& tile) {
    uint32_t r = quiescent ? v.find_quiescent<kW>(keys[i], tile, ts) : v.cooperative_find<kW>(keys[i], tile, ts, true);
    if (tile.thread_rank() == 0) out[i] = r;
  }));
}

// Warp lookups (find_warp): `lanes` keys per warp at a time over `warps` warps; sorted != 0: each
// warp takes a contiguous run of groups and keeps the last key's path, as the sorted kernel does
// (low_bits: the key bits its order left out).
void emu_find_warp(void* h, const uint32_t* keys, const uint32_t* pos, uint32_t* out, uint64_t n, uint32_t ts,
                   int warps, uint32_t lanes, int sorted, uint32_t low_bits) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  if (!v.versioned) ts = mvbt::kLatest;
  const uint64_t groups = (n + lanes - 1) / lanes, per = (groups + warps - 1) / warps;
  std::vector<mvbt::warp_stage> stage(warps);
  std::vector<mvbt::warp_path> path(warps);
  run_warps(warps, 8, [&](const emu_tile& warp, const emu_tile&) {
    const uint64_t w = mvbt::emu::sm;
    uint64_t g       = sorted ? w * per : w;
    const uint64_t end = sorted ? std::min(g + per, groups) : groups;
    if (sorted) path[w].clear(warp);
    for (; g < end; g += sorted ? 1 : warps) {
      const uint64_t i = g * lanes + warp.thread_rank();
      const bool live  = (uint32_t)warp.thread_rank() < lanes && i < n;
      const uint32_t k = live ? keys[i] : 0u;
      uint32_t start = mvbt::kAnchor;
      if (sorted) {
        const uint32_t m = warp.ballot(live);
        start = path[w].start(warp.shfl(k, 0) & ~low_bits, warp.shfl(k, 31 - __clz(m)) | low_bits, warp);
      }
      const uint32_t r = mvbt::find_warp(v, k, live, ts, start, sorted ? &path[w] : nullptr, stage[w], warp);
      if (live) out[sorted ? pos[i] : i] = r;
    }
  });
}

// Range queries by warps (range_warp), 32 per warp at a time; live != 0: the form that runs beside writers
// (snapshots only), from the leaf that its descent at the newest state finds; sorted as above.
void emu_range_warp(void* h, const uint32_t* lo, const uint32_t* hi, const uint32_t* pos, uint32_t* pairs,
                    uint32_t* counts, uint32_t avg_len, uint64_t n, uint32_t ts, int warps, int live, int sorted) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  if (!v.versioned) ts = mvbt::kLatest;
  const uint64_t groups = (n + 31) / 32, per = (groups + warps - 1) / warps;
  std::vector<mvbt::write_stage> stage(warps);
  std::vector<mvbt::warp_path> path(warps);
  run_warps(warps, 8, [&](const emu_tile& warp, const emu_tile&) {
    const uint64_t w = mvbt::emu::sm;
    auto& st         = stage[w];
    uint64_t g       = sorted ? w * per : w;
    const uint64_t end = sorted ? std::min(g + per, groups) : groups;
    if (sorted) path[w].clear(warp);
    for (; g < end; g += sorted ? 1 : warps) {
      const uint64_t i = g * 32 + warp.thread_rank();
      const bool has   = i < n;
      const uint64_t p = !has ? 0 : (sorted ? pos[i] : i);
      const uint32_t a = has ? lo[i] : 0u, b = has ? hi[p] : 0u;
      uint2* o         = reinterpret_cast<uint2*>(pairs) + p * (uint64_t)avg_len;
      uint32_t start = mvbt::kAnchor, c;
      if (live) {
        const uint32_t leaf = mvbt::leaf_warp(v, a, has && a != mvbt::kEmptyKey, start, nullptr, st, warp);
        c = mvbt::range_warp<true>(v, a, b, has, ts, o, avg_len, leaf == mvbt::kNone ? mvbt::kAnchor : leaf, nullptr, st, warp);
      } else {
        if (sorted) {
          const uint32_t m = warp.ballot(has);
          start = path[w].start(warp.shfl(a, 0), warp.shfl(a, 31 - __clz(m)), warp);
        }
        c = mvbt::range_warp<false>(v, a, b, has, ts, o, avg_len, start, sorted ? &path[w] : nullptr, st, warp);
      }
      if (has) counts[p] = c;
    }
  });
}

// Warp writes (write_warp), 32 ops per warp at a time over `warps` warps: kind 1 insert, 2 erase.
// sorted != 0: the ops are in key order, each warp takes a contiguous run with its path memory, and of
// a repeated key the last op alone is run.
void emu_write_warp(void* h, const uint32_t* kind, const uint32_t* keys, const uint32_t* vals, uint64_t n, int warps,
                    int W, int sorted) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  const uint32_t E      = v.versioned ? v.current_epoch() : 0u;
  const uint64_t groups = (n + 31) / 32, per = (groups + warps - 1) / warps;
  std::vector<mvbt::write_stage> stage(warps);
  std::vector<mvbt::warp_path> path(warps);
  EMU_DISPATCH(W, run_warps(warps, kW, [&](const emu_tile& warp, const emu_tile& tile) {
    const uint64_t w = mvbt::emu::sm;
    auto& st         = stage[w];
    uint64_t g       = sorted ? w * per : w;
    const uint64_t end = sorted ? std::min(g + per, groups) : groups;
    if (sorted) path[w].clear(warp);
    for (; g < end; g += sorted ? 1 : warps) {
      const uint64_t i = g * 32 + warp.thread_rank();
      const bool has   = i < n;
      const uint32_t k = has ? keys[i] : 0u;
      const bool live  = has && !(sorted && i + 1 < n && keys[i + 1] == k);
      uint32_t start   = mvbt::kAnchor;
      if (sorted) {
        const uint32_t m = warp.ballot(has);
        start = path[w].start(warp.shfl(k, 0), warp.shfl(k, 31 - __clz(m)), warp);
      }
      const uint32_t leaf = mvbt::leaf_warp(v, k, live && k != mvbt::kEmptyKey, start, sorted ? &path[w] : nullptr, st, warp);
      const uint32_t val = has ? vals[i] : 0u;
      if (sorted) mvbt::write_warp<kW, true>(v, k, val, has && kind[i] == 2, live, E, leaf, st, warp, tile);
      else mvbt::write_warp<kW>(v, k, val, has && kind[i] == 2, live, E, leaf, st, warp, tile);
    }
  }));
}

// quiescent != 0: the range query of a tree no writer changes meanwhile (range_quiescent).
void emu_range(void* h, const uint32_t* lo, const uint32_t* hi, uint32_t* pairs, uint32_t* counts,
               uint32_t avg_len, uint64_t n, uint32_t ts, int tiles, int W, int quiescent) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  if (!v.versioned) ts = mvbt::kLatest;
  EMU_DISPATCH(W, run(n, tiles, kW, [&](uint64_t i, const emu_tile& tile) {
    uint2* o   = pairs ? reinterpret_cast<uint2*>(pairs) + i * (uint64_t)avg_len : nullptr;
    uint32_t c = quiescent ? v.range_quiescent<kW>(lo[i], hi[i], tile, ts, o, avg_len)
                           : v.cooperative_range_query<kW>(lo[i], hi[i], tile, ts, o, avg_len, true);
    if (counts && tile.thread_rank() == 0) counts[i] = c;
  }));
}

// One run mixing inserts and range queries in units of `lanes` ops; queries read snapshot S, inserts land in
// S + 1.
void emu_insert_range(void* h, const uint32_t* keys, const uint32_t* vals, uint64_t n_ins,
                      const uint32_t* lo, const uint32_t* hi, uint64_t n_rq, uint32_t* pairs,
                      uint32_t* counts, uint32_t avg_len, int tiles, int W, uint32_t lanes) {
  auto* t          = static_cast<emu_tree*>(h);
  auto v           = t->view();
  const uint32_t S = v.versioned ? emu_snapshot(h) : mvbt::kLatest;
  const int warps  = std::max(1, tiles * W / 32);
  std::vector<mvbt::write_stage> stage(warps);
  EMU_DISPATCH(W, run_warps(warps, kW, [&](const emu_tile& warp, const emu_tile& tile) {
    const uint32_t w = mvbt::emu::sm;
    mvbt::insert_range_units<kW, kW>(v, keys, vals, (uint32_t)n_ins, lo, hi, (uint32_t)n_rq, reinterpret_cast<uint2*>(pairs),
                                     avg_len, counts, lanes, S, w, (uint64_t)warps, stage[w], warp, tile, tile);
  }));
}

// Sorted runs (the sorted batch front-end): keys[0, n) ascending, pos[i] = the input position of
// keys[i]. kind: 0 find, 1 range beside writers, each of `tiles` tiles taking one contiguous share of the
// run with its path memory (mvbt::finger, one per lane, as registers are on the GPU); 2 insert (a
// repeated key: its last occurrence wins), 3 erase, 4 find and 5 range of a tree no writer changes
// meanwhile, by as many warps as the tiles make.
void emu_sorted_run(void* h, int kind, const uint32_t* keys, const uint32_t* pos, const uint32_t* arg,
                    uint32_t* out, uint32_t* pairs, uint32_t avg_len, uint64_t n, uint32_t ts, int tiles, int W) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  if (!v.versioned) ts = mvbt::kLatest;
  if (n == 0) return;
  if (tiles < 1) tiles = 1;
  if (kind >= 2) {
    const int warps = std::max(1, tiles * W / 32);
    if (kind == 4) return emu_find_warp(h, keys, pos, out, n, ts, warps, 32, 1, 0);
    if (kind == 5) {
      std::vector<uint32_t> none(pairs ? 0 : 2 * n * (uint64_t)avg_len), counts(out ? 0 : n);
      return emu_range_warp(h, keys, arg, pos, pairs ? pairs : none.data(), out ? out : counts.data(), avg_len, n, ts, warps, 0, 1);
    }
    std::vector<uint32_t> kinds(n, kind == 2 ? 1u : 2u), vals(n, 0u);
    if (kind == 2)
      for (uint64_t i = 0; i < n; ++i) vals[i] = arg[pos[i]];
    return emu_write_warp(h, kinds.data(), keys, vals.data(), n, warps, W, 1);
  }
  const uint64_t per = (n + tiles - 1) / tiles;
  EMU_DISPATCH(W, {
    std::vector<std::unique_ptr<tile_shared>> sh;
    for (int x = 0; x < tiles; ++x) sh.emplace_back(new tile_shared(kW));
    std::vector<std::thread> th;
    for (int x = 0; x < tiles; ++x) {
      for (int l = 0; l < kW; ++l) {
        th.emplace_back([&, x, l] {
          mvbt::emu::sm = (uint32_t)x;
          emu_tile tile{l, kW, sh[x].get()};
          mvbt::finger<kW> f;
          const uint64_t b = (uint64_t)x * per, e = std::min<uint64_t>(n, b + per);
          for (uint64_t i = b; i < e; ++i) {
            const uint32_t k = keys[i];
            if (kind == 0) {
              const uint32_t r = v.cooperative_find<kW>(k, tile, ts, true, f.start_for(k, tile), &f);
              if (tile.thread_rank() == 0) out[pos[i]] = r;
            } else {
              uint2* o = pairs ? reinterpret_cast<uint2*>(pairs) + pos[i] * (uint64_t)avg_len : nullptr;
              const uint32_t c = v.cooperative_range_query<kW>(k, arg[pos[i]], tile, ts, o, avg_len, true,
                                                               f.start_for(k, tile), &f);
              if (out && tile.thread_rank() == 0) out[pos[i]] = c;
            }
          }
        });
      }
    }
    for (auto& y : th) y.join();
  });
}

// One run mixing finds and erases likewise; finds read snapshot S (a plain tree's newest state).
void emu_find_erase(void* h, const uint32_t* fkeys, uint32_t* out, uint64_t n_find,
                    const uint32_t* ekeys, uint64_t n_erase, int tiles, int W, uint32_t lanes) {
  auto* t          = static_cast<emu_tree*>(h);
  auto v           = t->view();
  const uint32_t S = v.versioned ? emu_snapshot(h) : mvbt::kLatest;
  const int warps  = std::max(1, tiles * W / 32);
  std::vector<mvbt::write_stage> stage(warps);
  EMU_DISPATCH(W, run_warps(warps, kW, [&](const emu_tile& warp, const emu_tile& tile) {
    const uint32_t w = mvbt::emu::sm;
    mvbt::find_erase_units<kW, kW>(v, fkeys, out, (uint32_t)n_find, ekeys, (uint32_t)n_erase, lanes, S, w, (uint64_t)warps,
                                   stage[w], warp, tile, tile);
  }));
}

// Mixed batches. mode 0: the persistent worker loop (claim order writes-first per batch, batch b
// waits for the writes of batch b - 1); mode 1: one snapshot + one run per batch.
// reclaim = 1: reclamation inside the persistent run (mvbt_batch_plan_set_reclaim) with external
// watermark ext; series (nullable) receives 4 values per batch as mvbt_batch_plan_memory_series.
// together = 1: no warp of a persistent run claims before all have looked at the queues (three shuffles), as
// the warps of a block that start together nearly do.
void emu_batch_run(void* h, uint32_t nb, const uint64_t* off, const uint32_t* type, const uint32_t* key,
                   const uint32_t* arg, const uint64_t* out_off, const uint32_t* cap, uint32_t* result,
                   uint32_t* range_out, int mode, int tiles, int W, int reclaim, uint32_t ext,
                   uint64_t* series, int together) {
  auto* t = static_cast<emu_tree*>(h);
  auto v  = t->view();
  mvbt::batch_view B{type, key, arg, out_off, cap, result, reinterpret_cast<uint2*>(range_out)};
  const int warps = std::max(1, tiles * W / 32);
  std::vector<mvbt::write_stage> stage(warps);
  if (mode == 1) {  // as many ops to a warp as it takes to give each warp some, as the library does
    for (uint32_t b = 0; b < nb; ++b) {
      const uint32_t S = emu_snapshot(h);
      const uint32_t lanes = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(4, (off[b + 1] - off[b]) / (uint64_t)warps));
      EMU_DISPATCH(W, run_warps(warps, kW, [&](const emu_tile& warp, const emu_tile& tile) {
        const uint32_t w = mvbt::emu::sm;
        mvbt::mixed_ops<kW>(v, B, off[b], off[b + 1], lanes, S, w, (uint64_t)warps, stage[w], warp, tile);
      }));
    }
    return;
  }
  std::vector<uint32_t> perm(off[nb]), n_writes(nb, 0), writes_done(nb, 0);
  std::vector<uint64_t> wpre(nb + 1, 0), rpre(nb + 1, 0);
  for (uint32_t b = 0; b < nb; ++b) {  // claim order: writes | finds | ranges
    uint64_t pos = off[b];
    for (uint64_t i = off[b]; i < off[b + 1]; ++i)
      if (mvbt::is_write_op(type[i])) perm[pos++] = (uint32_t)i, ++n_writes[b];
    for (uint64_t i = off[b]; i < off[b + 1]; ++i)
      if (type[i] == mvbt::kOpFind) perm[pos++] = (uint32_t)i;
    for (uint64_t i = off[b]; i < off[b + 1]; ++i)
      if (type[i] == mvbt::kOpRange) perm[pos++] = (uint32_t)i;
    wpre[b + 1] = wpre[b] + n_writes[b];
    rpre[b + 1] = rpre[b] + (off[b + 1] - off[b]) - n_writes[b];
  }
  unsigned long long cursors[2] = {0, 0};
  uint32_t done                 = 0;
  uint32_t params[3]            = {nb, t->ctl.epoch, ext};
  mvbt::batch_sched sc{off, perm.data(), n_writes.data(), wpre.data(), rpre.data(), writes_done.data(),
                       &done, &cursors[0], &cursors[1], params};
  std::vector<uint32_t> reads_done(nb, 0);
  std::vector<unsigned long long> tail_at(nb, ~0ull), ser(4ull * nb, 0);
  uint32_t full_done           = 0;
  unsigned long long rc_limit  = 0;
  if (reclaim && t->ctl.reclaim_cap) {  // as k_batch_begin_reclaim
    const uint32_t S0 = params[1];
    rc_limit      = (ext == mvbt::kReclaimAll || S0 <= ext) ? t->ctl.retire_tail : t->ctl.retire_head;
    sc.reads_done = reads_done.data();
    sc.full_done  = &full_done;
    sc.tail_at    = tail_at.data();
    sc.rc_limit   = &rc_limit;
    sc.series     = ser.data();
  }
  if (sc.rc_limit)  // as k_count_ops
    run_warps(mvbt::kMaxSmSlots / 32, 8, [&](const emu_tile& warp, const emu_tile&) {
      mvbt::flush_chunks(&t->ctl, mvbt::emu::sm, t->ctl.ring_cap / 2, warp);
    });
  mvbt::batch_gate gate{0, 0};  // the warps as one block
  std::vector<mvbt::held_reads> held(warps);
  EMU_DISPATCH(W, run_warps(warps, kW, [&](const emu_tile& warp, const emu_tile& tile) {
    mvbt::batched_worker<kW>(v, B, sc, (uint32_t)warps, gate, held[mvbt::emu::sm], stage[mvbt::emu::sm], warp, tile);
  }, together ? 3 : 0));
  t->ctl.epoch = params[1] + nb;
  if (series && sc.series) std::memcpy(series, ser.data(), ser.size() * sizeof(uint64_t));
}

int emu_validate(void* h, uint32_t ts, mvbt_report* rep) {
  auto* t     = static_cast<emu_tree*>(h);
  uint64_t nn = std::min<uint64_t>(t->ctl.bump, t->capacity);
  return mvbt_validate_image(t->pool.data(), nn, t->versioned, ts, rep);
}

}  // extern "C"
