// xor_build.cu -- device construction of the 3-hash xor filter.
//
// Produces a table with the reference's header (n_keys, m_cells, mix_seed,
// seed schedule: spike/ribbon/xor_filter.hpp:185-192,256-470 and
// fourcore_xor_store.hpp:67-119) from the same key set, built on the GPU:
//
//  1. Key set.  Pair mode enumerates unordered pairs of the DISTINCT values
//     of i^6 mod 2^64 (1<=i<=N); many i share a value (every multiple of 2048
//     has i^6 = 0 mod 2^64), so this already removes most duplicate keys.
//     The keys are partitioned by mix64(key) into slices whose hash set stays
//     in L2, and each slice's duplicates are removed there (the reference
//     sorts + uniques).  The survivors are the unique keys.
//  2. Incidence: every cell is one 64-bit word, count << 42 | sum of the
//     indices of its keys, and each key adds (1 << 42) + index to its three
//     cells (binned by L2-sized cell slice when HBM allows).
//  3. Peel in rounds.  A cell with count 1 holds exactly one key, named by
//     its index; in round r every such key is claimed by the lowest of its
//     count-1 cells (so a key is claimed once), then removed from its other
//     two cells.  The 2-core is unique, so peeling succeeds for exactly the
//     seeds for which the reference's FIFO peel succeeds.
//  4. Fill in reverse round order, in place: the claimed cell of a round-r key
//     becomes fp(h) ^ cell(c1) ^ cell(c2).  Its other cells were never claimed
//     in rounds <= r (a count-1 cell cannot hold a second unpeeled key), so
//     they are final already and a round needs no ordering inside it.
// Cells then hold exactly the reference's cell relation (FN = 0, same FPR);
// which key owns which cell differs from the FIFO order, so bytes differ.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "s615_device.cuh"

namespace s615 {

namespace {

namespace cg = cooperative_groups;

constexpr u64 kEmpty = ~0ULL;

// Bytes the context's HBM budget still allows (one read of the shared count).
size_t budget_room(const s615_ctx* ctx) {
  const size_t u = ctx->used.load();
  return ctx->budget > u ? ctx->budget - u : 0;
}

int grid_for(s615_ctx* ctx, u64 n, int threads) {
  const u64 want = (n + threads - 1) / threads;
  const u64 cap = (u64)ctx->num_sms * 16;
  return (int)(want < cap ? (want ? want : 1) : cap);
}

// Blocks for n items at `per` items a block.  The kernels that read or update
// random cells take one small tile per block: the block scheduler then hands
// tiles out as SMs become free.  Scattered accesses are served per group of 2
// to 8 SMs at an equal rate per group, so a static split waits for the largest
// groups (random reads over 28 GB: 3.65e10/s split evenly, 4.71e10/s dealt out).
u32 blocks_for(u64 n, u64 per) {
  const u64 b = (n + per - 1) / per;
  return (u32)std::min<u64>(std::max<u64>(b, 1), 0x7FFFFFFFull);
}

// Positions of the flagged items in a list whose length is *count, K per
// thread, with ONE global atomic per block (a shared-memory scan of the warps'
// counts): the lists' counters are single addresses, and per-warp atomics on
// them serialise in their L2 slice (~1.7e8/s; the peel of N = 76,667 took 1,554
// ms with them, 711 ms per block).  Every thread of the block calls this (it
// synchronises the block); pos[k] is set where take[k] is.
template <int K>
__device__ __forceinline__ void block_positions(const bool (&take)[K], unsigned long long* count,
                                                u64 (&pos)[K]) {
  __shared__ u32 s_cnt[32];
  __shared__ unsigned long long s_base;
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  u32 b[K];
  u32 wtot = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    b[k] = __ballot_sync(0xFFFFFFFFu, take[k]);
    wtot += __popc(b[k]);
  }
  __syncthreads();   // the previous call's offsets have been read
  if (lane == 0) s_cnt[wid] = wtot;
  __syncthreads();
  if (threadIdx.x == 0) {
    u32 tot = 0;
    for (u32 w = 0; w < nw; ++w) {
      const u32 n = s_cnt[w];
      s_cnt[w] = tot;
      tot += n;
    }
    s_base = tot ? atomicAdd(count, (unsigned long long)tot) : 0ull;
  }
  __syncthreads();
  u64 at = s_base + s_cnt[wid];
  const u32 below = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    pos[k] = at + __popc(b[k] & below);
    at += __popc(b[k]);
  }
}

// ---- partition through shared memory ----------------------------------------
// Items (8 B each) are sorted by slice in two passes over the same source.
// k_part_count counts each block's items per slice in shared memory; a scan
// over (slice, block) gives every block its own output range per slice;
// k_part_scatter then takes tiles of kTile items, orders a tile by slice in
// shared memory and writes each slice's run with consecutive threads.  Writing
// items one by one was bound by the rate of scattered stores (2e10/s: 150 of
// the 219 ms of the N = 48,000 incidence); runs of 5 to 12 items divide the
// store requests accordingly.
constexpr u32 kMaxSlices = 4608;
constexpr u32 kItemChunks = 1024;   // order_items: chunk fields told apart
constexpr int kPartThreads = 512;
constexpr int kPartPer = 16;
constexpr u32 kTile = kPartThreads * kPartPer;   // items per tile: 64 KB staged

// Source of the key partition: the t-th raw key, t < n.  Pairs are numbered
// along rows a and nv - 1 - a laid end to end (nv + 1 pairs together), so a
// flat range of t has no short rows.
struct KeySource {
  const u64* vals;   // pair mode: distinct values; null: keys
  const u64* keys;
  u64 nv, n, row_recip;
  u32 shards, shard;
  u64 srecip;
  u32 S, s_lo, s_hi;   // slices in all, and those this pass takes
  __device__ __forceinline__ u64 key(u64 t) const {
    if (!vals) return keys[t];
    const u64 len = nv + 1;
    u64 p = mulhi64(t, row_recip), q = t - p * len;   // p is at most 1 short
    if (q >= len) { q -= len; ++p; }
    const u64 first = nv - p;
    const u64 a = q < first ? p : nv - 1 - p;
    const u64 b = q < first ? p + q : a + (q - first);
    return vals[a] + vals[b];
  }
  // The key's slice, or ~0 when this build or pass does not take it.
  __device__ __forceinline__ u32 slice(u64 k) const {
    if (shards > 1 && fast_mod(mix64(k + kShardSeed), shards, srecip) != shard) return ~0u;
    const u32 s = (u32)mulhi64(mix64(k), S);
    return s >= s_lo && s < s_hi ? s : ~0u;
  }
  static constexpr int kItems = 1;   // items per element
  __device__ __forceinline__ void get(u64 t, u64 (&item)[1], u32 (&sl)[1]) const {
    item[0] = key(t);
    sl[0] = slice(item[0]);
  }
};

template <class Src>
__global__ void __launch_bounds__(kPartThreads) k_part_count(Src src, u64 k0, u64 per, u64 k1, u32 S,
                                                             u32* __restrict__ bhist) {
  extern __shared__ u32 hist[];
  for (u32 i = threadIdx.x; i < S; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  const u64 lo = k0 + blockIdx.x * per, hi = min(k1, lo + per);
  for (u64 t = lo + threadIdx.x; t < hi; t += blockDim.x) {
    u64 item[Src::kItems];
    u32 sl[Src::kItems];
    src.get(t, item, sl);
#pragma unroll
    for (int j = 0; j < Src::kItems; ++j)
      if (sl[j] != ~0u && S615_CHECK(sl[j] < S, kChkList)) atomicAdd(&hist[sl[j]], 1u);
  }
  __syncthreads();
  for (u32 i = threadIdx.x; i < S; i += blockDim.x) bhist[(u64)blockIdx.x * S + i] = hist[i];
}

// One block per slice: the exclusive scan of its G block counts, and its total.
__global__ void k_part_scan(const u32* __restrict__ bhist, u32 G, u32 S,
                            unsigned long long* __restrict__ brel,
                            unsigned long long* __restrict__ total) {
  __shared__ unsigned long long s_w[32];
  const u32 sl = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long run = 0;
  for (u32 b0 = 0; b0 < G; b0 += blockDim.x) {
    const u32 b = b0 + threadIdx.x;
    const unsigned long long c = b < G ? bhist[(u64)b * S + sl] : 0ull;
    unsigned long long x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= (u32)o) x += y;
    }
    if (lane == 31) s_w[wid] = x;
    __syncthreads();
    unsigned long long before = run, all = run;
    for (u32 w = 0; w < blockDim.x / 32; ++w) {
      if (w < wid) before += s_w[w];
      all += s_w[w];
    }
    if (b < G) brel[(u64)b * S + sl] = before + x - c;
    run = all;
    __syncthreads();
  }
  if (threadIdx.x == 0) total[sl] = run;
}

// soff[s] = items of slices [s0, s) for s in [s0, s1]; one block.
__global__ void k_part_offsets(const unsigned long long* __restrict__ total, u32 s0, u32 s1,
                               unsigned long long* __restrict__ soff) {
  __shared__ unsigned long long s_w[32];
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long run = 0;
  for (u32 b0 = s0; b0 < s1; b0 += blockDim.x) {
    const u32 b = b0 + threadIdx.x;
    const unsigned long long c = b < s1 ? total[b] : 0ull;
    unsigned long long x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= (u32)o) x += y;
    }
    if (lane == 31) s_w[wid] = x;
    __syncthreads();
    unsigned long long before = run, all = run;
    for (u32 w = 0; w < blockDim.x / 32; ++w) {
      if (w < wid) before += s_w[w];
      all += s_w[w];
    }
    if (b < s1) soff[b] = before + x - c;
    run = all;
    __syncthreads();
  }
  if (threadIdx.x == 0) soff[s1] = run;
}

// Dynamic shared memory of k_part_scatter: the staged tile, each staged item's
// slice, and per slice its count, its start in the tile and its output cursor.
constexpr size_t part_smem(u32 S) {
  return (size_t)kTile * 8 + (size_t)S * 8 + (size_t)S * 4 * 2 + (size_t)kTile * 2;
}

template <class Src>
__global__ void __launch_bounds__(kPartThreads, 2) k_part_scatter(
    Src src, u64 k0, u64 per, u64 k1, u32 S, const unsigned long long* __restrict__ brel,
    const unsigned long long* __restrict__ soff, unsigned long long* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* stage = reinterpret_cast<unsigned long long*>(smem);
  unsigned long long* cur = stage + kTile;
  u32* cnt = reinterpret_cast<u32*>(cur + S);
  u32* off = cnt + S;
  u16* sid = reinterpret_cast<u16*>(off + S);
  __shared__ u32 s_w[kPartThreads / 32];
  constexpr int E = kPartPer / Src::kItems;   // elements per thread and tile
  constexpr int I = E * Src::kItems;          // items per thread and tile (<= kPartPer)
  const u32 tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (u32 i = tid; i < S; i += kPartThreads) {
    cur[i] = soff[i] + brel[(u64)blockIdx.x * S + i];
    cnt[i] = 0;
  }
  __syncthreads();
  const u64 lo = k0 + blockIdx.x * per, hi = min(k1, lo + per);
  for (u64 t0 = lo; t0 < hi; t0 += (u64)kPartThreads * E) {
    u64 item[I];
    u32 at[I];   // slice | rank in the tile's run << 13 (both below 2^13), ~0: none
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const u64 t = t0 + (u64)e * kPartThreads + tid;
      u64 it[Src::kItems];
      u32 sl[Src::kItems];
#pragma unroll
      for (int j = 0; j < Src::kItems; ++j) { it[j] = 0; sl[j] = ~0u; }
      if (t < hi) src.get(t, it, sl);
#pragma unroll
      for (int j = 0; j < Src::kItems; ++j) {
        const bool ok = sl[j] != ~0u && S615_CHECK(sl[j] < S, kChkList);
        item[e * Src::kItems + j] = it[j];
        at[e * Src::kItems + j] = ok ? sl[j] | (atomicAdd(&cnt[sl[j]], 1u) << 13) : ~0u;
      }
    }
    __syncthreads();
    // exclusive scan of the counts over the slices, ceil(S / threads) per thread
    const u32 each = (S + kPartThreads - 1) / kPartThreads;
    const u32 i0 = min(tid * each, S), i1 = min(i0 + each, S);
    u32 sum = 0;
    for (u32 i = i0; i < i1; ++i) sum += cnt[i];
    u32 x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= (u32)o) x += y;
    }
    if (lane == 31) s_w[wid] = x;
    __syncthreads();
    u32 before = 0, total = 0;
    for (u32 w = 0; w < kPartThreads / 32; ++w) {
      if (w < wid) before += s_w[w];
      total += s_w[w];
    }
    u32 run = before + x - sum;
    for (u32 i = i0; i < i1; ++i) { off[i] = run; run += cnt[i]; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < I; ++k)
      if (at[k] != ~0u) {
        const u32 sl = at[k] & 8191u, pos = off[sl] + (at[k] >> 13);
        stage[pos] = item[k];
        sid[pos] = (u16)sl;
      }
    __syncthreads();
    for (u32 pos = tid; pos < total; pos += kPartThreads) {
      const u32 sl = sid[pos];
      out[cur[sl] + (pos - off[sl])] = stage[pos];
    }
    __syncthreads();
    for (u32 i = i0; i < i1; ++i) { cur[i] += cnt[i]; cnt[i] = 0; }
    __syncthreads();
  }
}

// One slice's keys into a hash set that stays in L2: a key is appended to out
// when its insertion finds it new.  The other table is cleared meanwhile for
// the next slice.  Four keys a thread, their probes in flight together.  A
// full table (it has at least two slots a key) and the all-ones key set flags.
// Bound by the round trips of the probes: 34 ms for the 1.15e9 keys of N =
// 48,000 (46 ms with each key probed to its end in turn); a hash set of all keys
// in HBM, scanned afterwards, took 110 ms or more.
constexpr int kDedupPer = 4;
static_assert(kDedupPer == 4, "the probe loop's condition");
__global__ void k_dedupe(const u64* __restrict__ keys, u64 n, unsigned long long* table, u64 tmask,
                         ulonglong2* clear, u64* __restrict__ out, u64 cap,
                         unsigned long long* n_out, u32* flags) {
  const u64 nt = (u64)gridDim.x * blockDim.x;
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < (tmask + 1) / 2; i += nt)
    clear[i] = make_ulonglong2(kEmpty, kEmpty);
  const u64 span = (u64)blockDim.x * kDedupPer;
  for (u64 base = blockIdx.x * span; base < n; base += (u64)gridDim.x * span) {
    u64 key[kDedupPer], at[kDedupPer], old[kDedupPer];
    bool fresh[kDedupPer], live[kDedupPer];
#pragma unroll
    for (int k = 0; k < kDedupPer; ++k) {
      const u64 i = base + (u64)k * blockDim.x + threadIdx.x;
      live[k] = i < n;
      key[k] = live[k] ? keys[i] : 0;
      if (live[k] && key[k] == kEmpty) { flags[0] = 1; live[k] = false; }
      at[k] = mix64(key[k] ^ 0x5bd1e9955bd1e995ULL) & tmask;
    }
    // one probe of every unsettled key per step, so that a step is one round trip
    // to L2 for the thread's keys together
#pragma unroll
    for (int k = 0; k < kDedupPer; ++k) fresh[k] = false;
    for (u64 probe = 0; live[0] || live[1] || live[2] || live[3]; ++probe) {
      if (probe > tmask) { flags[1] = 1; break; }
#pragma unroll
      for (int k = 0; k < kDedupPer; ++k)
        if (live[k])
          old[k] = atomicCAS(table + ((at[k] + probe) & tmask), (unsigned long long)kEmpty,
                             (unsigned long long)key[k]);
#pragma unroll
      for (int k = 0; k < kDedupPer; ++k)
        if (live[k]) {
          fresh[k] = old[k] == kEmpty;
          live[k] = !fresh[k] && old[k] != key[k];
        }
    }
    u64 pos[kDedupPer];
    block_positions<kDedupPer>(fresh, n_out, pos);   // every thread of the block, every pass
#pragma unroll
    for (int k = 0; k < kDedupPer; ++k)
      if (fresh[k] && pos[k] < cap) out[pos[k]] = key[k];   // past cap: counted, not written
  }
}

// ---- cell words -------------------------------------------------------------
// During the build every cell is one 64-bit word: the number of unpeeled keys
// in the cell above bit 42 and the sum of their key indices below it.  An
// update of a cell is then one atomic add (the reference's incidence keeps an
// xor of hashes and a count: two arrays, two read-modify-writes per update),
// and a cell of count 1 names its key directly; the key's hash is
// recomputed from the key array.  Indices are below 2^34 and a count above
// 255 fails the build, so the sum never reaches bit 42.  After the peel the
// word array is filled in place with the final r-bit cells.
constexpr int kCntShift = 42;
constexpr u64 kSumMask = (1ull << kCntShift) - 1;
constexpr u64 kMaxKeys = 1ull << 34;
__device__ __forceinline__ u64 cnt_of(u64 w) { return w >> kCntShift; }
__device__ __forceinline__ u64 upd(u64 idx) { return (1ull << kCntShift) + idx; }

// Checked builds: the key and cell counts of the build in flight, set before
// the incidence, bound every key index a kernel decodes (from a loop or from a
// cell word's index sum) and the cells of the binned apply.  One build at a
// time per process in such a build.
#ifdef S615_CHECKED
static __device__ u64 g_check_nkeys, g_check_ncells;
#define S615_KEY_OK(idx) S615_CHECK((idx) < g_check_nkeys, kChkList)
#define S615_CELL_OK(c) S615_CHECK((c) < g_check_ncells, kChkList)
#else
#define S615_KEY_OK(idx) true
#define S615_CELL_OK(c) true
#endif

__device__ __forceinline__ u64 key_hash(const u64* keys, u64 idx, u64 seed) {
  if (!S615_KEY_OK(idx)) return 0;
  return mix64(keys[idx] + seed);
}

// Checked builds: all three cells of a key lie in [0, 3 * block).
__device__ __forceinline__ bool cells_ok(const u64* c, u64 block) {
  return S615_CHECK(c[0] < 3 * block && c[1] < 3 * block && c[2] < 3 * block, kChkList);
}

__global__ void k_incidence(const u64* __restrict__ keys, u64 n, u64 seed, u64 block, u64 recip,
                            unsigned long long* W) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    u64 c[3];
    cell_indices(key_hash(keys, i, seed), block, recip, c);
    if (!cells_ok(c, block)) continue;
#pragma unroll
    for (int t = 0; t < 3; ++t) atomicAdd(W + c[t], (unsigned long long)upd(i));
  }
}

// The largest count of any cell (a count above 255 fails the build).
__global__ void k_max_count(const unsigned long long* __restrict__ W, u64 m, unsigned* mx) {
  unsigned local = 0;
  for (u64 c = blockIdx.x * (u64)blockDim.x + threadIdx.x; c < m; c += (u64)gridDim.x * blockDim.x)
    { const u64 k = cnt_of(W[c]); local = max(local, k > 0xFFFFFFFFull ? 0xFFFFFFFFu : (unsigned)k); }
#pragma unroll
  for (int o = 16; o; o >>= 1) local = max(local, __shfl_xor_sync(0xFFFFFFFFu, local, o));
  if ((threadIdx.x & 31) == 0 && local) atomicMax(mx, local);
}

// ---- incidence through shared-memory radix bins ---------------------------
// The cells are cut into slices of 2^sbits cells (16 MB of cell words:
// L2-sized) and the three updates of every key are partitioned by slice (one
// 8-byte entry each: key index << 32 | slice-local cell offset); k_bin_apply
// walks them slice by slice with the whole grid, and its atomic adds land on a
// slice that is resident in L2.
struct UpdateSource {
  const u64* keys;
  u64 k0, seed, block, recip;
  u32 sbits;
  static constexpr int kItems = 3;
  __device__ __forceinline__ void get(u64 i, u64 (&item)[3], u32 (&sl)[3]) const {
    u64 c[3];
    cell_indices(key_hash(keys, i, seed), block, recip, c);
    const bool ok = cells_ok(c, block);
    const u64 lmask = (1ull << sbits) - 1;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      item[t] = ((i - k0) << 32) | (c[t] & lmask);
      sl[t] = ok ? (u32)(c[t] >> sbits) : ~0u;
    }
  }
};

// A cooperative grid walks the slices in order and splits each slice's
// entries over all its threads, with a grid-wide sync after every slice, so
// the whole GPU works on one slice (16 MB) at a time and its atomic adds hit
// in L2.  (Without the syncs, blocks drift apart over the walk and the slices
// in use outgrow L2.)
// kSync = false is the same walk without the syncs, for a device or setting
// where a cooperative launch is refused (the result is the same; only the L2
// hit rate suffers).
template <bool kSync>
__global__ void k_bin_apply(const unsigned long long* __restrict__ ent, u64 k0,
                            const unsigned long long* __restrict__ soff, u32 sbits, u32 S,
                            unsigned long long* W) {
  const u64 nt = (u64)gridDim.x * blockDim.x, tid = blockIdx.x * (u64)blockDim.x + threadIdx.x;
  for (u32 sl = 0; sl < S; ++sl) {
    unsigned long long* base = W + ((u64)sl << sbits);
    const u64 e1 = soff[sl + 1];
    for (u64 i = soff[sl] + tid; i < e1; i += nt) {
      const u64 e = ent[i];
      const u32 off = (u32)e, idx = (u32)(e >> 32);
      if (S615_KEY_OK(k0 + idx) && S615_CELL_OK(((u64)sl << sbits) + off))
        atomicAdd(base + off, (unsigned long long)upd(k0 + idx));
    }
    if constexpr (kSync) cg::this_grid().sync();
  }
}

// ---- peel ------------------------------------------------------------------
// Round r claims every key whose lowest count-1 cell is a count-1 cell (so a
// key is claimed once), then removes each claimed key from its two other
// cells; a claimed cell keeps its key's index with count 0.  Every count-1
// cell at the start of round r > 1 got its count 1 while round r-1 removed
// keys (a count-1 cell of round r-1 either claimed its key or lost it to a
// lower cell of the same key), so after a full scan in round 1 each round
// visits only the cells whose count went from 2 to 1 in the round before.
// Claimed cells are appended in round order (as offsets within their third
// of the table), and the fill walks that list backwards.  Without room for
// the lists every round scans all cells and tags its claims with the round.

// A list of cells, each entry a u32 offset within its third of the table and
// the third (0, 1, 2) in a byte: a cell index needs more than 32 bits once m
// passes 2^32, an offset within a third does not (block < 2^32 for every
// single table).
struct CellList {
  u32* off;
  u8* third;
  __host__ __device__ CellList at(u64 k) const { return CellList{off + k, third + k}; }
  __device__ __forceinline__ u64 cell(u64 k, u64 block) const { return third[k] * block + off[k]; }
};

// Write cell c at position `at` of the list, or set *over past its capacity.
__device__ __forceinline__ bool list_put(CellList list, u64 at, u64 cap, u64 c, u64 block, u32* over) {
  if (at >= cap) {
    *over = 1;
    return false;
  }
  const u32 t = c >= 2 * block ? 2u : c >= block ? 1u : 0u;
  list.off[at] = (u32)(c - t * block);
  list.third[at] = (u8)t;
  return true;
}

// The claimed cells of the peel, in round order.  With idx and hash set
// (HBM permitting: they reuse the incidence's entry buffers) the claim also
// records each claimed key's index and hash, so the apply and the fill read
// them in order instead of fetching the cell word and the key again.
struct ClaimList {
  CellList cells;
  u32* idx;                    // null: read from the cell word
  unsigned long long* hash;    // null: recomputed from the key array
  __host__ __device__ ClaimList at(u64 k) const {
    return ClaimList{cells.at(k), idx ? idx + k : nullptr, hash ? hash + k : nullptr};
  }
};

// Rounds of few candidates go out kRounds at a time, each reading its sizes from
// here: round j of a batch has candidates [0, ncand[j]) and claims the list's
// entries [end[j], end[j + 1]).  A round whose candidates overflowed their list,
// and those after it, do nothing.  With the host waiting for the sizes twice in
// every round, a round took at least 70 us: building N = 1,500 took 7.0 ms,
// 6,000 11.6 and 16,000 52.0; in batches of 8 it takes 4.5, 9.5 and 50.1.  A
// batch's grids are for its first round's candidates and half as many again
// (the kernels stride), so a round with none left costs an empty launch.
constexpr int kRounds = 8;
struct PeelState {
  unsigned long long norder;               // claimed cells so far
  unsigned long long ncand[kRounds + 1], end[kRounds + 1];
  u32 over[kRounds + 2];
};
// Candidates up to which rounds are batched: 2 million take 0.27 ms, so above
// it the two waits are less than a fifth of a round, and a batch that a large
// round shrinks in would launch grids far too wide.
constexpr u64 kBatchCand = 1ull << 21;

// Claims among the candidate cells [0, ncand), or among every cell when the
// candidate list is null: a count-1 cell claims its key unless a lower cell of
// the key has count 1 too.  A candidate costs a chain of scattered reads (its
// word, its key, the key's lower cells), so each thread follows kClaimPer
// chains at once.
constexpr int kClaimPer = 4;
__global__ void k_claim_list(CellList cand, u64 ncand, const unsigned long long* __restrict__ W,
                             const u64* __restrict__ keys, u64 seed, u64 block, u64 recip,
                             ClaimList out, unsigned long long* n_order, u64 order_cap, u32* over,
                             const PeelState* ps, int j) {
  if (ps) ncand = ps->over[j] ? 0 : ps->ncand[j];   // round j of a batch
  const u64 span = (u64)blockDim.x * kClaimPer;
  for (u64 base = blockIdx.x * span; base < ncand; base += (u64)gridDim.x * span) {
    bool claim[kClaimPer];
    u64 c[kClaimPer], w[kClaimPer], h[kClaimPer];
#pragma unroll
    for (int k = 0; k < kClaimPer; ++k) {
      const u64 i = base + (u64)k * blockDim.x + threadIdx.x;
      claim[k] = i < ncand;
      c[k] = claim[k] ? (cand.off ? cand.cell(i, block) : i) : 0;
      claim[k] = claim[k] && S615_CHECK(c[k] < 3 * block, kChkList);
    }
#pragma unroll
    for (int k = 0; k < kClaimPer; ++k) w[k] = claim[k] ? W[c[k]] : 0;
#pragma unroll
    for (int k = 0; k < kClaimPer; ++k) {
      claim[k] = claim[k] && cnt_of(w[k]) == 1;
      h[k] = claim[k] ? key_hash(keys, w[k] & kSumMask, seed) : 0;
    }
    u64 w0[kClaimPer], w1[kClaimPer];   // the words of the key's lower cells, 0: none
#pragma unroll
    for (int k = 0; k < kClaimPer; ++k) {
      w0[k] = w1[k] = 0;
      if (claim[k]) {
        u64 cs[3];
        cell_indices(h[k], block, recip, cs);
        claim[k] = cells_ok(cs, block);
        if (claim[k] && cs[0] < c[k]) w0[k] = W[cs[0]];
        if (claim[k] && cs[1] < c[k]) w1[k] = W[cs[1]];
      }
    }
#pragma unroll
    for (int k = 0; k < kClaimPer; ++k)
      claim[k] = claim[k] && cnt_of(w0[k]) != 1 && cnt_of(w1[k]) != 1;
    u64 pos[kClaimPer];
    block_positions<kClaimPer>(claim, n_order, pos);   // every thread of the block, every pass
#pragma unroll
    for (int k = 0; k < kClaimPer; ++k)
      if (claim[k] && list_put(out.cells, pos[k], order_cap, c[k], block, over) && out.hash) {
        out.idx[pos[k]] = (u32)(w[k] & kSumMask);
        out.hash[pos[k]] = h[k];
      }
  }
}

// Claimed keys a thread applies per pass of k_apply_list: their eight atomics
// are in flight together, and the block synchronises (in the append) once
// per pass instead of once per key.
constexpr int kApplyPer = 4;

__global__ void k_apply_list(ClaimList in, u64 L, unsigned long long* W,
                             const u64* __restrict__ keys, u64 seed, u64 block, u64 recip,
                             CellList next, unsigned long long* n_next, u64 next_cap, u32* over,
                             PeelState* ps, int j) {
  if (ps) {   // round j of a batch: what its claim appended
    const u64 from = ps->end[j], to = ps->norder;
    if (blockIdx.x == 0 && threadIdx.x == 0) ps->end[j + 1] = to;
    in = in.at(from);
    L = to - from;
  }
  const u64 span = (u64)blockDim.x * kApplyPer;
  for (u64 base = blockIdx.x * span; base < L; base += (u64)gridDim.x * span) {
    bool to[2 * kApplyPer];
    u64 nc[2 * kApplyPer];
    u64 old[2 * kApplyPer];
#pragma unroll
    for (int q = 0; q < kApplyPer; ++q) {
      to[2 * q] = to[2 * q + 1] = false;
      nc[2 * q] = nc[2 * q + 1] = 0;
      old[2 * q] = old[2 * q + 1] = 0;
      const u64 i = base + (u64)q * blockDim.x + threadIdx.x;   // coalesced over the block
      if (i < L && S615_CHECK(in.cells.cell(i, block) < 3 * block, kChkList)) {
        const u64 c = in.cells.cell(i, block);
        u64 idx, h;
        if (in.hash) {
          idx = in.idx[i];
          h = in.hash[i];
        } else {
          idx = W[c] & kSumMask;
          h = key_hash(keys, idx, seed);
        }
        // remove the key from its two other cells (results read below, so the
        // atomics of all kApplyPer keys are in flight together)
        u64 cs[3];
        cell_indices(h, block, recip, cs);
        if (cells_ok(cs, block) && S615_KEY_OK(idx)) {   // always true in the default build
          const int own = cs[0] == c ? 0 : cs[1] == c ? 1 : 2;
          nc[2 * q] = own == 0 ? cs[1] : cs[0];
          nc[2 * q + 1] = own == 2 ? cs[1] : cs[2];
          old[2 * q] = atomicAdd(W + nc[2 * q], (unsigned long long)(0 - upd(idx)));
          old[2 * q + 1] = atomicAdd(W + nc[2 * q + 1], (unsigned long long)(0 - upd(idx)));
          to[2 * q] = to[2 * q + 1] = true;   // pending: the count check follows
          // Without the recorded index the word keeps it, at count 0, for the
          // fill.  With it the word is left as it is (count 1): no unpeeled key
          // has this cell, so nothing but a scan of every cell would read it
          // again before the fill writes it (k_zero_claimed goes before such a
          // scan).  The store would be a third scattered update per key.
          if (!in.hash) W[c] = idx;
        }
      }
    }
    // a cell whose count went from 2 to 1 is a candidate of the next round
#pragma unroll
    for (int k = 0; k < 2 * kApplyPer; ++k) to[k] = to[k] && cnt_of(old[k]) == 2;
    // every thread of the block reaches the append (it synchronises the block)
    u64 pos[2 * kApplyPer];
    block_positions<2 * kApplyPer>(to, n_next, pos);
#pragma unroll
    for (int k = 0; k < 2 * kApplyPer; ++k)
      if (to[k]) list_put(next, pos[k], next_cap, nc[k], block, over);
  }
}

// Reverse fill of claimed cell c: fingerprint of its key xor its two other
// cells, which are final already (filled in a later round, or never claimed
// and 0).
__device__ __forceinline__ void fill_cell(unsigned long long* W, u64 h, u64 block, u64 recip,
                                          u64 mask, u64 c) {
  u64 cs[3];
  cell_indices(h, block, recip, cs);
  if (!cells_ok(cs, block) || !S615_CHECK(c < 3 * block, kChkList)) return;
  u64 v = h & mask;
#pragma unroll
  for (int t = 0; t < 3; ++t)
    if (cs[t] != c) v ^= W[cs[t]];
  W[c] = v & mask;
}

// Count 0 for the claimed cells, before a round that scans every cell.
__global__ void k_zero_claimed(CellList in, u64 L, unsigned long long* W, u64 block) {
  const u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x;
  if (i < L && S615_CHECK(in.cell(i, block) < 3 * block, kChkList)) W[in.cell(i, block)] = 0ull;
}

constexpr int kFillPer = 4;   // fills in flight per thread
__global__ void k_fill_list(ClaimList in, u64 L, unsigned long long* W,
                            const u64* __restrict__ keys, u64 seed, u64 block, u64 recip, u64 mask) {
  const u64 span = (u64)blockDim.x * kFillPer;
  for (u64 base = blockIdx.x * span; base < L; base += (u64)gridDim.x * span) {
    u64 c[kFillPer], h[kFillPer], v[kFillPer];
    bool on[kFillPer];
#pragma unroll
    for (int k = 0; k < kFillPer; ++k) {
      const u64 i = base + (u64)k * blockDim.x + threadIdx.x;
      on[k] = i < L;
      c[k] = on[k] ? in.cells.cell(i, block) : 0;
      on[k] = on[k] && S615_CHECK(c[k] < 3 * block, kChkList);
      h[k] = on[k] && in.hash ? (u64)in.hash[i] : 0;
    }
    if (!in.hash) {
#pragma unroll
      for (int k = 0; k < kFillPer; ++k) h[k] = on[k] ? key_hash(keys, W[c[k]], seed) : 0;
    }
    // the key's other two cells: claimed in a later round or never, so no
    // thread of this launch writes them
#pragma unroll
    for (int k = 0; k < kFillPer; ++k) {
      v[k] = 0;
      if (on[k]) {
        u64 cs[3];
        cell_indices(h[k], block, recip, cs);
        on[k] = cells_ok(cs, block);
        const int own = cs[0] == c[k] ? 0 : cs[1] == c[k] ? 1 : 2;
        if (on[k]) v[k] = W[own == 0 ? cs[1] : cs[0]] ^ W[own == 2 ? cs[1] : cs[2]];
      }
    }
#pragma unroll
    for (int k = 0; k < kFillPer; ++k)
      if (on[k]) W[c[k]] = (v[k] ^ h[k]) & mask;
  }
}

// remove_key for the scan form (index and hash from the cell word and keys).
__device__ __forceinline__ void remove_key_scan(unsigned long long* W, const u64* keys, u64 seed,
                                                u64 block, u64 recip, u64 c) {
  const u64 idx = W[c] & kSumMask;
  u64 cs[3];
  cell_indices(key_hash(keys, idx, seed), block, recip, cs);
  if (!cells_ok(cs, block) || !S615_KEY_OK(idx)) return;
#pragma unroll
  for (int t = 0; t < 3; ++t)
    if (cs[t] != c) atomicAdd(W + cs[t], (unsigned long long)(0 - upd(idx)));
  W[c] = idx;   // count 0; the index stays for the fill
}

// Does cell c (count 1) claim its key?  The key's lower count-1 cells win.
__device__ __forceinline__ bool claims(const unsigned long long* W, const u64* keys, u64 seed,
                                       u64 block, u64 recip, u64 c, u64 w) {
  u64 cs[3];
  cell_indices(key_hash(keys, w & kSumMask, seed), block, recip, cs);
  if (!cells_ok(cs, block)) return false;
#pragma unroll
  for (int t = 0; t < 3; ++t)
    if (cs[t] < c && cnt_of(W[cs[t]]) == 1) return false;
  return true;
}

// The scan form: claims of round r tagged in round[], apply and fill by tag.
__global__ void k_claim_scan(const unsigned long long* __restrict__ W, const u64* __restrict__ keys,
                             u64 seed, u16* __restrict__ round, u64 m, u64 block, u64 recip, u16 r,
                             unsigned long long* n_claimed) {
  for (u64 c0 = blockIdx.x * (u64)blockDim.x; c0 < m; c0 += (u64)gridDim.x * blockDim.x) {
    const u64 c = c0 + threadIdx.x;
    bool claim = false;
    if (c < m) {
      const u64 w = W[c];
      claim = cnt_of(w) == 1 && claims(W, keys, seed, block, recip, c, w);
      if (claim) round[c] = r;
    }
    const bool take[1] = {claim};
    u64 pos[1];
    block_positions<1>(take, n_claimed, pos);   // counts the claims (every thread, every pass)
  }
}

__global__ void k_apply_scan(unsigned long long* W, const u64* __restrict__ keys, u64 seed,
                             const u16* __restrict__ round, u64 m, u64 block, u64 recip, u16 r) {
  for (u64 c = blockIdx.x * (u64)blockDim.x + threadIdx.x; c < m;
       c += (u64)gridDim.x * blockDim.x) {
    if (round[c] == r) remove_key_scan(W, keys, seed, block, recip, c);
  }
}

__global__ void k_fill_scan(unsigned long long* W, const u64* __restrict__ keys, u64 seed,
                            const u16* __restrict__ round, u64 m, u64 block, u64 recip, u16 r,
                            u64 mask) {
  for (u64 c = blockIdx.x * (u64)blockDim.x + threadIdx.x; c < m;
       c += (u64)gridDim.x * blockDim.x)
    if (round[c] == r) fill_cell(W, key_hash(keys, W[c], seed), block, recip, mask, c);
}

__global__ void k_narrow(const u64* __restrict__ in, u32* __restrict__ out, u64 m) {
  for (u64 c = blockIdx.x * (u64)blockDim.x + threadIdx.x; c < m;
       c += (u64)gridDim.x * blockDim.x)
    out[c] = (u32)in[c];
}

struct Buf {
  s615_ctx* ctx;
  void* p = nullptr;
  size_t n = 0;
  explicit Buf(s615_ctx* c) : ctx(c) {}
  bool own = true;
  int alloc(size_t bytes) { n = bytes; own = true; return dev_alloc(ctx, &p, bytes); }
  // n bytes of another buffer, which outlives this one
  void view(void* at, size_t bytes) { release(); p = at; n = bytes; own = false; }
  void release() { if (p && own) dev_free(ctx, p, n); p = nullptr; n = 0; }
  ~Buf() { release(); }
};

// The scratch of a partition into at most S slices by G blocks: per-block
// counts and bases, slice totals and offsets.
struct PartScratch {
  u32* bhist;
  unsigned long long *brel, *total, *soff;
  static size_t bytes(size_t G, size_t S) { return G * S * 12 + (2 * S + 1) * 8 + 64; }
  PartScratch(void* p, size_t G, size_t S) {
    brel = static_cast<unsigned long long*>(p);
    total = brel + G * S;
    soff = total + S;
    bhist = reinterpret_cast<u32*>(soff + S + 1);
  }
};

// Count: the items of elements [k0, k1) per slice, in ps.total and ps.brel.
template <class Src>
int part_count(s615_ctx* ctx, const Src& src, u64 k0, u64 k1, u32 G, u32 S, const PartScratch& ps,
               cudaStream_t st) {
  k_part_count<Src><<<G, kPartThreads, S * sizeof(u32), st>>>(src, k0, (k1 - k0 + G - 1) / G, k1, S, ps.bhist);
  k_part_scan<<<S, 256, 0, st>>>(ps.bhist, G, S, ps.brel, ps.total);
  ctx->launches += 2;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

// Scatter the items of slices [s0, s1) (counted by part_count over the same
// elements) to out, slice after slice; ps.soff[s0 .. s1] are their offsets.
template <class Src>
int part_scatter(s615_ctx* ctx, const Src& src, u64 k0, u64 k1, u32 G, u32 S, u32 s0, u32 s1,
                 const PartScratch& ps, unsigned long long* out, cudaStream_t st) {
  S615_CU(cudaFuncSetAttribute(k_part_scatter<Src>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)part_smem(kMaxSlices)));
  k_part_offsets<<<1, 1024, 0, st>>>(ps.total, s0, s1, ps.soff);
  k_part_scatter<Src><<<G, kPartThreads, part_smem(S), st>>>(src, k0, (k1 - k0 + G - 1) / G, k1, S,
                                                             ps.brel, ps.soff, out);
  ctx->launches += 2;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

// Blocks of a partition pass: two per SM, fewer for few elements.
u32 part_blocks(const s615_ctx* ctx, u64 n) {
  return (u32)std::min<u64>((u64)ctx->num_sms * 2, std::max<u64>(1, n / (4 * kTile)));
}

// Incidence of keys [0, n) for one seed through the slice bins, in chunks of
// keys whose updates fit the entry buffers (ent_cap updates).
int incidence_binned(s615_ctx* ctx, const u64* keys, u64 n, u64 seed, u64 m, u64 block, u64 recip,
                     unsigned long long* ent, u64 ent_cap, unsigned long long* W, void* scratch,
                     cudaStream_t st) {
  u32 sbits = 21;
  while (((m + (1ull << sbits) - 1) >> sbits) > kMaxSlices) ++sbits;
  const u32 S = (u32)((m + (1ull << sbits) - 1) >> sbits);
  const u64 chunk = std::max<u64>(1, std::min<u64>(ent_cap / 3, 1ull << 32));
  for (u64 k0 = 0; k0 < n; k0 += chunk) {
    const u64 k1 = std::min(n, k0 + chunk);
    const u32 G = part_blocks(ctx, k1 - k0);
    const PartScratch ps(scratch, G, S);
    const UpdateSource src{keys, k0, seed, block, recip, sbits};
    if (const int s = part_count(ctx, src, k0, k1, G, S, ps, st)) return s;
    if (const int s = part_scatter(ctx, src, k0, k1, G, S, 0, S, ps, ent, st)) return s;
    int per_sm = 0;
    S615_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bin_apply<true>, 256, 0));
    const dim3 grid(ctx->num_sms * std::max(per_sm, 1));
    {   // cooperative: every block resident at once (the launch is refused otherwise)
      const unsigned long long* a_ent = ent;
      const unsigned long long* a_soff = ps.soff;
      u64 a_k0 = k0;
      u32 a_sbits = sbits, a_S = S;
      void* args[] = {(void*)&a_ent, (void*)&a_k0, (void*)&a_soff, (void*)&a_sbits, (void*)&a_S,
                      (void*)&W};
      if (cudaLaunchCooperativeKernel((const void*)k_bin_apply<true>, grid, dim3(256), args, 0, st) !=
          cudaSuccess) {
        cudaGetLastError();
        k_bin_apply<false><<<grid, 256, 0, st>>>(ent, k0, ps.soff, sbits, S, W);
      }
    }
    ctx->launches++;
    S615_CU(cudaGetLastError());
  }
  return S615_OK;
}

// The distinct keys of src (at most cap) to out; *n their number.  Slices of
// about 1.5 million keys, so that a slice's hash set (32 MB, and the next one's
// being cleared) stays in L2; more and smaller ones when HBM is short, and
// then as many passes over the source as the partition buffer needs.
// `given`, when it has room for every key, is used as the partition buffer.
int unique_keys(s615_ctx* ctx, KeySource src, u64 n_raw, size_t avail, const Buf* given, u64* out,
                u64 cap, u64* n, cudaStream_t st) {
  constexpr u64 kSliceKeys = 3ull << 19, kMost = 4096;
  u64 S = std::min<u64>(kMost, (n_raw + kSliceKeys - 1) / kSliceKeys);
  S = std::max<u64>(S, 1);
  // two tables of up to four slots a key, in at most a quarter of the room
  while (S < kMost && (n_raw / S + 1) * 8 * 8 > avail / 4) S = std::min<u64>(kMost, 2 * S);
  const u32 G = part_blocks(ctx, src.n);
  src.S = (u32)S;
  src.s_lo = 0;
  src.s_hi = (u32)S;
  Buf scratch(ctx), part(ctx), tables(ctx);
  int s = scratch.alloc(PartScratch::bytes(G, S) + 64);
  if (s) return s;
  auto* d_n = static_cast<unsigned long long*>(scratch.p);           // [0] count
  u32* d_flags = reinterpret_cast<u32*>(d_n + 1);                    // all-ones key, full table
  const PartScratch ps(static_cast<char*>(scratch.p) + 64, G, S);
  S615_CU(cudaMemsetAsync(scratch.p, 0, 64, st));
  if ((s = part_count(ctx, src, 0, src.n, G, (u32)S, ps, st))) return s;
  std::vector<unsigned long long> total(S);
  S615_CU(cudaMemcpyAsync(total.data(), ps.total, S * 8, cudaMemcpyDeviceToHost, st));
  S615_CU(cudaStreamSynchronize(st));
  u64 most = 0, all = 0;
  for (u64 t : total) { most = std::max<u64>(most, t); all += t; }
  u64 slots = 1024;
  while (slots < 2 * most) slots *= 2;
  if ((s = tables.alloc(2 * slots * 8))) return s;
  auto* T = static_cast<unsigned long long*>(tables.p);
  S615_CU(cudaMemsetAsync(T, 0xFF, 2 * slots * 8, st));
  // the partition buffer: every key when there is room, else what there is
  const size_t held = 2 * slots * 8 + PartScratch::bytes(G, S);
  const u64 room = avail > held ? (avail - held) / 8 : 0;
  u64 part_cap = std::max<u64>(std::min<u64>(all, room), std::max<u64>(most, 1));
  if (given && given->n / 8 >= all) part.view(given->p, given->n), part_cap = given->n / 8;
  else if ((s = part.alloc(part_cap * 8))) return s;
  auto* P = static_cast<unsigned long long*>(part.p);
  u32 flip = 0;
  for (u32 s0 = 0; s0 < S;) {
    u32 s1 = s0;
    u64 held_keys = 0;
    while (s1 < S && (s1 == s0 || held_keys + total[s1] <= part_cap)) held_keys += total[s1++];
    src.s_lo = s0;
    src.s_hi = s1;
    if ((s = part_scatter(ctx, src, 0, src.n, G, (u32)S, s0, s1, ps, P, st))) return s;
    u64 at = 0;
    for (u32 sl = s0; sl < s1; ++sl) {
      if (!total[sl]) continue;
      k_dedupe<<<blocks_for(total[sl], 256 * kDedupPer), 256, 0, st>>>(
          reinterpret_cast<const u64*>(P + at), total[sl], T + flip * slots, slots - 1,
          reinterpret_cast<ulonglong2*>(T + (flip ^ 1) * slots), out, cap, d_n, d_flags);
      ctx->launches++;
      flip ^= 1;
      at += total[sl];
    }
    S615_CU(cudaGetLastError());
    s0 = s1;
  }
  unsigned long long h[2] = {0, 0};
  S615_CU(cudaMemcpyAsync(h, d_n, 16, cudaMemcpyDeviceToHost, st));
  S615_CU(cudaStreamSynchronize(st));
  if (h[0] > cap || (h[1] >> 32)) return S615_E_BUILD;   // more keys than out holds, or a full table
  *n = h[0];
  if (h[1] & 0xFFFFFFFFull) {   // the all-ones key stays out of the hash set (out has room for it)
    const u64 e = kEmpty;
    S615_CU(cudaMemcpy(out + *n, &e, 8, cudaMemcpyHostToDevice));
    ++*n;
  }
  return S615_OK;
}

// S615_TRACE: per-phase device times of a build on stderr (CUDA events on
// the build stream).
struct PhaseTrace {
  bool on = std::getenv("S615_TRACE") != nullptr;
  cudaStream_t st;
  std::vector<std::pair<const char*, cudaEvent_t>> marks;
  explicit PhaseTrace(cudaStream_t s) : st(s) {}
  void mark(const char* name) {
    nvtxMarkA(name);   // the phase boundary on a profiler's timeline
    if (!on) return;
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) { cudaGetLastError(); return; }
    cudaEventRecord(e, st);
    marks.emplace_back(name, e);
  }
  void report(u64 n, u64 m, int rounds) {
    if (!on || marks.size() < 2) return;
    cudaEventSynchronize(marks.back().second);
    std::fprintf(stderr, "[xor-build] keys=%llu cells=%llu rounds=%d", (unsigned long long)n,
                 (unsigned long long)m, rounds);
    for (size_t i = 1; i < marks.size(); ++i) {
      float ms = 0;
      cudaEventElapsedTime(&ms, marks[i - 1].second, marks[i].second);
      std::fprintf(stderr, " %s=%.1fms", marks[i].first, ms);
    }
    std::fprintf(stderr, "\n");
  }
  ~PhaseTrace() {
    for (auto& m : marks) cudaEventDestroy(m.second);
  }
};

}  // namespace

int build_xor_device(s615_ctx* ctx, const u64* d_pair_vals, u64 n_vals, const u64* d_keys,
                     u64 n_keys, int r, const u64* seeds, int n_seeds, int N, int layout,
                     DevTable* out, u32 shards, u32 shard) {
  cudaStream_t st = ctx->stream;
  const bool pairs = d_pair_vals != nullptr;
  if (shards < 1) shards = 1;
  if (shard >= shards) return S615_E_ARG;
  const u64 n_all = pairs ? n_vals * (n_vals + 1) / 2 : n_keys;
  // one shard's share of the keys, with room for the binomial spread
  const u64 n_raw = shards == 1 ? n_all
                                : std::min<u64>(n_all, n_all / shards +
                                                           8 * (u64)std::sqrt((double)n_all) + 4096);

  PhaseTrace trace(st);
  trace.mark("start");
  // ---- 1. unique keys ----
  // With room to spare, the scratch of the whole build is one allocation for
  // at most n_raw keys: their array, the entry buffer (the partition's before
  // the incidence, the claim list's after it), the candidate lists and the bin
  // counts.  (Allocating and freeing 58 GB in five pieces for N = 48,000 took
  // 50 to 150 ms of the build, with what had been freed just before.)
  const size_t bin_bytes = PartScratch::bytes((size_t)ctx->num_sms * 2, kMaxSlices);
  const u64 m_most = capacity_for(n_raw);
  const auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t a_keys = up((n_raw + 1) * 8), a_ent = up(24 * (n_raw + 1)),
               a_front = up(10 * std::max<u64>(4096, m_most / 8));
  release_run_batch(ctx);   // a table needs the room more than s615_run's kept buffers
  Buf arena(ctx), keys(ctx), ent(ctx), front(ctx), bins(ctx);
  u64 n = 0;
  {
    size_t free_b = 0, total_b = 0;
    S615_CU(cudaMemGetInfo(&free_b, &total_b));
    const size_t all_bytes = a_keys + a_ent + a_front + up(bin_bytes);
    if (n_raw < (1ull << 32) &&
        std::min(free_b, budget_room(ctx)) > all_bytes + m_most * 8 + ((size_t)3 << 30) &&
        !arena.alloc(all_bytes)) {
      char* at = static_cast<char*>(arena.p);
      keys.view(at, a_keys);
      ent.view(at + a_keys, a_ent);
      front.view(at + a_keys + a_ent, a_front);
      bins.view(at + a_keys + a_ent + a_front, bin_bytes);
    } else {
      arena.p = nullptr;
    }
  }
  {
    // +1: the all-ones key is kept out of the hash set and appended last
    int s = arena.p ? 0 : keys.alloc((n_raw + 1) * sizeof(u64));
    if (s) return s;
    size_t free_b = 0, total_b = 0;
    S615_CU(cudaMemGetInfo(&free_b, &total_b));
    size_t avail = std::min(free_b, budget_room(ctx));
    if (avail > ((size_t)2 << 30)) avail -= (size_t)2 << 30;
    KeySource src{};
    src.vals = d_pair_vals;
    src.keys = d_keys;
    src.nv = n_vals;
    src.n = n_all;
    src.row_recip = mod_recip(n_vals + 1);
    src.shards = shards;
    src.shard = shard;
    src.srecip = mod_recip(shards);
    if ((s = unique_keys(ctx, src, n_raw, avail, arena.p ? &ent : nullptr, static_cast<u64*>(keys.p),
                         n_raw, &n, st)))
      return s;
  }

  std::memset(&out->hdr, 0, sizeof out->hdr);
  out->hdr.magic = kMagic; out->hdr.version = kVersion; out->hdr.kind = 1;
  out->hdr.r = (u32)r; out->hdr.N = (u32)(N > 0 ? N : 0);
  out->hdr.shard_count = shards;
  out->hdr.shard_index = shard;
  if (n == 0) {
    out->hdr.mix_seed = seeds[0];
    out->layout = S615_LAYOUT_WIDE; out->cell_bytes = 8;
    out->d_cells = nullptr; out->bytes = 0;
    return S615_OK;
  }

  trace.mark("unique");
  // ---- 2-4. per seed: incidence, peel, fill ----
  const u64 m = capacity_for(n);
  const u64 block = m / 3, recip = mod_recip(block);
  if (n > kMaxKeys) return S615_E_BUILD;   // key indices must stay below 2^34
#ifdef S615_CHECKED
  S615_CU(cudaMemcpyToSymbolAsync(g_check_nkeys, &n, sizeof n, 0, cudaMemcpyHostToDevice, st));
  S615_CU(cudaMemcpyToSymbolAsync(g_check_ncells, &m, sizeof m, 0, cudaMemcpyHostToDevice, st));
#endif
  Buf cells(ctx), rounds(ctx), scratch(ctx), order(ctx);
  int s = cells.alloc(m * sizeof(u64));
  if (s) return s;
  // Peel over lists (claimed cells in round order, two candidate lists of
  // m/8 cells each; a round whose candidates overflow scans every cell), or,
  // without room for the lists, over full scans by round tag.
  // Candidate lists: two of m/8 entries (5 bytes each: offset + third).
  const u64 fcap = std::max<u64>(4096, m / 8);
  bool lists = block < (1ull << 32);
  if (lists && !arena.p && front.alloc(2 * fcap * 5)) {
    front.release();
    lists = false;
  }
  if ((s = scratch.alloc(64 + sizeof(PeelState)))) return s;
  auto* W = static_cast<unsigned long long*>(cells.p);
  const u64* K = static_cast<const u64*>(keys.p);
  // scratch: [0] max count, [4] list overflow, [8] n_claimed, [16] n_next, then the peel's state
  u32* d_max = static_cast<u32*>(scratch.p);
  u32* d_lover = reinterpret_cast<u32*>(static_cast<char*>(scratch.p) + 4);
  auto* d_norder = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch.p) + 8);
  auto* d_nnext = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch.p) + 16);
  auto* d_peel = reinterpret_cast<PeelState*>(static_cast<char*>(scratch.p) + 64);
  const int g = grid_for(ctx, m, 256);
  // Entry buffers of the binned incidence: all 3n updates when HBM allows,
  // else chunks of keys; with no room for a useful chunk the incidence adds
  // directly into the cell words (k_incidence).  The peel's own buffers come
  // first: the round tags of the scan form, or (when the entry buffers will
  // not hold 2n entries for the recorded claim list) the claimed-cell list.
  auto avail_now = [&]() -> size_t {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) { cudaGetLastError(); return 0; }
    size_t a = std::min(free_b, budget_room(ctx));
    const size_t margin = (size_t)2 << 30;
    return a > margin ? a - margin : 0;
  };
  // the recorded claim list needs 17 bytes per key in the entry buffers
  // (offset, third, u32 index, hash) and n < 2^32; otherwise the claimed
  // cells alone (5 bytes per key) are taken now, before the entry buffers
  const bool rich_possible = n < (1ull << 32);
  if (lists && !arena.p && (!rich_possible || avail_now() < bin_bytes + 24 * n) && order.alloc(n * 5)) {
    order.release(); front.release();
    lists = false;
  }
  if (!lists && (s = rounds.alloc(m * sizeof(u16)))) return s;
  u64 ent_cap = 0;   // of ent: one 8-byte word per update (index << 32 | slice offset)
  if (arena.p) {
    ent_cap = 3 * n;
  } else {
    const size_t avail = avail_now();
    if (avail > bin_bytes) {
      ent_cap = std::min<u64>(3 * n, (avail - bin_bytes) / 8);
      ent_cap = ent_cap / 3 * 3;
    }
    if (ent_cap >= std::min<u64>(3 * n, 3ull << 20)) {
      if ((s = ent.alloc(ent_cap * 8)) || (s = bins.alloc(bin_bytes))) {
        ent.release(); bins.release();
        ent_cap = 0;
      }
    } else {
      ent_cap = 0;
    }
  }
  // The claim list: in the entry buffer (idle after the incidence) with each
  // key's index and hash when it has room, else cells only.  Its layout:
  // offsets (4n bytes), indices (4n), thirds (n), then the hashes (8n) from
  // the next 8-byte boundary.
  ClaimList claim_list{{nullptr, nullptr}, nullptr, nullptr};
  const u64 hash_at = (9 * n + 7) / 8 * 8;
  if (lists && rich_possible && ent_cap * 8 >= hash_at + 8 * n && !order.p) {
    u32* o = static_cast<u32*>(ent.p);
    claim_list = ClaimList{{o, reinterpret_cast<u8*>(o + 2 * n)}, o + n,
                           reinterpret_cast<unsigned long long*>(static_cast<char*>(ent.p) + hash_at)};
  } else if (lists && (order.p || !order.alloc(n * 5))) {
    u32* o = static_cast<u32*>(order.p);
    claim_list.cells = CellList{o, reinterpret_cast<u8*>(o + n)};
  } else if (lists) {   // no room for any list: scan, with round tags in the entry buffers' place
    order.release(); front.release();
    ent.release(); bins.release();
    ent_cap = 0;
    lists = false;
    if ((s = rounds.alloc(m * sizeof(u16)))) return s;
  }
  bool built = false;
  u64 used_seed = 0;
  int trace_rounds = 0;
  for (int si = 0; si < n_seeds && !built; ++si) {
    const u64 seed = seeds[si];
    S615_CU(cudaMemsetAsync(W, 0, m * sizeof(u64), st));
    if (!lists) S615_CU(cudaMemsetAsync(rounds.p, 0, m * sizeof(u16), st));
    S615_CU(cudaMemsetAsync(scratch.p, 0, 64 + sizeof(PeelState), st));
    if (ent_cap) {
      if ((s = incidence_binned(ctx, K, n, seed, m, block, recip,
                                static_cast<unsigned long long*>(ent.p), ent_cap, W, bins.p, st)))
        return s;
    } else {
      k_incidence<<<grid_for(ctx, n, 256), 256, 0, st>>>(K, n, seed, block, recip, W);
      ctx->launches++;
      S615_CU(cudaGetLastError());
    }
    k_max_count<<<g, 256, 0, st>>>(W, m, d_max);
    ctx->launches++;
    u32 mx = 0;
    S615_CU(cudaMemcpyAsync(&mx, d_max, 4, cudaMemcpyDeviceToHost, st));
    S615_CU(cudaStreamSynchronize(st));
    if (mx > 255) return S615_E_BUILD;   // the index sums could reach the count bits
    trace.mark("incidence");
    const u64 mask = fp_mask((u32)r);
    if (lists) {

      u32* fo = static_cast<u32*>(front.p);
      u8* ft = reinterpret_cast<u8*>(fo + 2 * fcap);
      const CellList fr[2] = {CellList{fo, ft}, CellList{fo + fcap, ft + fcap}};
      std::vector<u64> off{0};
      u64 total = 0, ncand = m;
      CellList cand{nullptr, nullptr};   // round 1 scans every cell
      int cur = 0;
      // S615_TRACE: per round, the candidates, the keys claimed and the host
      // time of its claim and apply (each ends in a sync here anyway; a batch's
      // time is spread evenly over its rounds, as apply)
      using TClock = std::chrono::steady_clock;
      const auto ms_since = [](TClock::time_point a) {
        return std::chrono::duration<double, std::milli>(TClock::now() - a).count();
      };
      std::vector<std::array<double, 4>> rounds_trace;
      bool over = false;   // the candidates of the next round overflowed their list
      while (off.size() <= 0xFFFE) {
        const auto t_claim = TClock::now();
        PeelState h{};
        if (cand.off && ncand <= kBatchCand && off.size() + kRounds <= 0xFFFE) {
          // a batch of rounds; sizes on the device, the grids for half as many again
          h.norder = h.end[0] = total;
          h.ncand[0] = ncand;
          S615_CU(cudaMemcpyAsync(d_peel, &h, sizeof h, cudaMemcpyHostToDevice, st));
          const u64 grid_for_n = ncand + ncand / 2;
          for (int j = 0; j < kRounds; ++j) {
            k_claim_list<<<blocks_for(grid_for_n, 256 * kClaimPer), 256, 0, st>>>(
                fr[cur ^ (j & 1)], 0, W, K, seed, block, recip, claim_list, &d_peel->norder, n,
                d_lover, d_peel, j);
            k_apply_list<<<blocks_for(grid_for_n, 256 * kApplyPer), 256, 0, st>>>(
                claim_list, 0, W, K, seed, block, recip, fr[cur ^ (j & 1) ^ 1], &d_peel->ncand[j + 1],
                fcap, &d_peel->over[j + 1], d_peel, j);
            ctx->launches += 2;
          }
          S615_CU(cudaGetLastError());
          S615_CU(cudaMemcpyAsync(&h, d_peel, sizeof h, cudaMemcpyDeviceToHost, st));
          S615_CU(cudaStreamSynchronize(st));
          bool more = true;
          for (int j = 0; j < kRounds && more; ++j) {
            const u64 L = h.end[j + 1] - h.end[j];
            if (trace.on) rounds_trace.push_back({(double)h.ncand[j], (double)L, 0, ms_since(t_claim) / kRounds});
            if (L == 0) { more = false; break; }
            total += L;
            off.push_back(total);
            cur ^= 1;
            ncand = h.ncand[j + 1];
            over = h.over[j + 1] != 0;
            more = ncand != 0 || over;
            if (over) break;
          }
          if (!more) break;
        } else {
          k_claim_list<<<blocks_for(ncand, 256 * kClaimPer), 256, 0, st>>>(
              cand, ncand, W, K, seed, block, recip, claim_list, &d_peel->norder, n, d_lover, nullptr, 0);
          ctx->launches++;
          S615_CU(cudaMemcpyAsync(&h.norder, &d_peel->norder, 8, cudaMemcpyDeviceToHost, st));
          S615_CU(cudaStreamSynchronize(st));
          const u64 L = h.norder - total;
          const double claim_ms = trace.on ? ms_since(t_claim) : 0.0;
          const auto t_apply = TClock::now();
          if (L == 0) break;
          unsigned long long h_next = 0;
          u32 h_lover = 0;
          S615_CU(cudaMemsetAsync(d_nnext, 0, 8, st));
          S615_CU(cudaMemsetAsync(d_lover, 0, 4, st));
          k_apply_list<<<blocks_for(L, 256 * kApplyPer), 256, 0, st>>>(
              claim_list.at(total), L, W, K, seed, block, recip, fr[cur ^ 1], d_nnext, fcap, d_lover,
              nullptr, 0);
          ctx->launches++;
          S615_CU(cudaGetLastError());
          S615_CU(cudaMemcpyAsync(&h_next, d_nnext, 8, cudaMemcpyDeviceToHost, st));
          S615_CU(cudaMemcpyAsync(&h_lover, d_lover, 4, cudaMemcpyDeviceToHost, st));
          S615_CU(cudaStreamSynchronize(st));
          if (trace.on) rounds_trace.push_back({(double)ncand, (double)L, claim_ms, ms_since(t_apply)});
          total += L;
          off.push_back(total);
          cur ^= 1;
          ncand = h_next;
          over = h_lover != 0;
        }
        if (over) {   // candidates overflowed: the next round scans every cell
          cand = CellList{nullptr, nullptr};
          ncand = m;
          S615_CU(cudaMemsetAsync(d_lover, 0, 4, st));
          if (claim_list.hash) {
            k_zero_claimed<<<blocks_for(total, 256), 256, 0, st>>>(claim_list.cells, total, W, block);
            ctx->launches++;
          }
        } else {
          cand = fr[cur];
          if (ncand == 0) break;   // nothing became count 1: the peel is over
        }
      }
      if (trace.on)
        for (size_t q = 0; q < rounds_trace.size(); ++q)
          std::fprintf(stderr, "[xor-build] round %zu: candidates=%.0f claimed=%.0f claim=%.2fms apply=%.2fms\n",
                       q + 1, rounds_trace[q][0], rounds_trace[q][1], rounds_trace[q][2],
                       rounds_trace[q][3]);
      if (total != n) continue;   // 2-core not empty: next seed
      trace.mark("peel");
      for (size_t q = off.size() - 1; q >= 1; --q) {
        const u64 L = off[q] - off[q - 1];
        k_fill_list<<<blocks_for(L, 256 * kFillPer), 256, 0, st>>>(claim_list.at(off[q - 1]), L, W, K,
                                                                   seed, block, recip, mask);
        ctx->launches++;
      }
      trace_rounds = (int)off.size() - 1;
    } else {
      u16* rt = static_cast<u16*>(rounds.p);
      u64 peeled = 0;
      u16 rr = 0;
      for (;;) {
        if (rr == 0xFFFE) break;
        ++rr;
        S615_CU(cudaMemsetAsync(d_norder, 0, 8, st));
        k_claim_scan<<<g, 256, 0, st>>>(W, K, seed, rt, m, block, recip, rr, d_norder);
        ctx->launches++;
        k_apply_scan<<<g, 256, 0, st>>>(W, K, seed, rt, m, block, recip, rr);
        ctx->launches++;
        S615_CU(cudaGetLastError());
        unsigned long long c = 0;
        S615_CU(cudaMemcpyAsync(&c, d_norder, 8, cudaMemcpyDeviceToHost, st));
        S615_CU(cudaStreamSynchronize(st));
        if (c == 0) { --rr; break; }
        peeled += c;
      }
      if (peeled != n) continue;   // 2-core not empty: next seed
      trace.mark("peel");
      for (u16 q = rr; q >= 1; --q) {
        k_fill_scan<<<g, 256, 0, st>>>(W, K, seed, rt, m, block, recip, q, mask);
        ctx->launches++;
      }
      trace_rounds = rr;
    }
    S615_CU(cudaGetLastError());
    trace.mark("fill");
    built = true;
    used_seed = seed;
  }
  if (!built) return S615_E_BUILD;
  S615_CU(cudaStreamSynchronize(st));
  trace.mark("sync");
  keys.release(); rounds.release(); order.release(); front.release();
  ent.release(); bins.release();
  arena.release();
  trace.mark("free");

  out->hdr.n_keys = n;
  out->hdr.m_cells = m;
  out->hdr.mix_seed = used_seed;
  // ---- 5. final HBM layout ----
  if (layout == S615_LAYOUT_PACKED) {
    const u64 len = packed_bytes(m, (u32)r);
    const size_t bytes = ((len + 7) / 8 + 1) * 8;
    void* p = nullptr;
    if ((s = dev_alloc(ctx, &p, bytes))) return s;
    S615_CU(cudaMemsetAsync(p, 0, bytes, st));
    if ((s = launch_pack(ctx, cells.p, 8, m, (u32)r, static_cast<u8*>(p), len, st))) {
      dev_free(ctx, p, bytes);
      return s;
    }
    out->layout = S615_LAYOUT_PACKED; out->cell_bytes = 0;
    out->d_cells = p; out->bytes = bytes;
  } else if (r <= 32) {
    void* p = nullptr;
    const size_t bytes = m * sizeof(u32);
    if ((s = dev_alloc(ctx, &p, bytes))) return s;
    k_narrow<<<g, 256, 0, st>>>(static_cast<const u64*>(cells.p), static_cast<u32*>(p), m);
    ctx->launches++;
    out->layout = S615_LAYOUT_WIDE; out->cell_bytes = 4;
    out->d_cells = p; out->bytes = bytes;
  } else {
    out->layout = S615_LAYOUT_WIDE; out->cell_bytes = 8;
    out->d_cells = cells.p; out->bytes = cells.n;
    cells.p = nullptr; cells.n = 0;   // ownership moves to the table
  }
  trace.mark("layout");
  trace.report(n, m, trace_rounds);
  S615_CU(cudaStreamSynchronize(st));
  S615_CU(cudaGetLastError());
  return S615_OK;
}

namespace {
// Work items by chunk field (its last slice takes every larger one).
struct ItemSource {
  const u64* items;
  u32 S;
  static constexpr int kItems = 1;
  __device__ __forceinline__ void get(u64 t, u64 (&item)[1], u32 (&sl)[1]) const {
    item[0] = items[t];
    sl[0] = min(item_chunk(item[0]), S - 1);
  }
};
}  // namespace

// The builder's partition, with chunks for slices: 18 ms of std::stable_sort on
// the host for 924,000 items of (6,1,7) find4 jobs, 0.1 ms here.
int order_items(s615_ctx* ctx, const u64* in, u64* out, u64 n, void* scratch, cudaStream_t st) {
  const u32 G = part_blocks(ctx, n);
  const PartScratch ps(scratch, G, kItemChunks);
  const ItemSource src{in, kItemChunks};
  if (const int s = part_count(ctx, src, 0, n, G, kItemChunks, ps, st)) return s;
  return part_scatter(ctx, src, 0, n, G, kItemChunks, 0, kItemChunks, ps,
                      reinterpret_cast<unsigned long long*>(out), st);
}
size_t order_items_scratch(const s615_ctx* ctx, u64 n) {
  return PartScratch::bytes(part_blocks(ctx, n), kItemChunks);
}

S615_CHECK_TAKE_DEFINE(check_take_xor_build)

}  // namespace s615
