// staged.cuh -- key pages of the staged probe (staged.cu) and the warp-wide
// push that fills them.
#pragma once
#include <cuda_runtime.h>

#include "s615_device.cuh"

namespace s615 {

// Keys wait in pages of kStagePage 8-byte entries, sorted by bucket: bucket b
// holds the keys whose next cell lies in the b-th slice of 2^sb cells of its
// third.  17 to 32 buckets (stage_geometry), so a lane can stand for each.
constexpr u32 kStagePage = 256;
constexpr u32 kStageBuckets = 32;
constexpr u32 kStageNone = 0xFFFFFFFFu;    // no page open yet
constexpr u32 kStageFull = 0xFFFFFFFEu;    // the bucket has no page left
constexpr u32 kBloomBits = 19;             // positives of a chunk: 2^19 bits, 64 KB

struct StagePages {
  unsigned long long* e;   // [nb * cap][kStagePage]
  u32* fill;               // [nb * cap] entries per page
  u32* npages;             // [nb * kStageStride] pages of a bucket (may pass cap: the rest were refused)
  u32 nb, cap;             // bucket b's pages are b * cap + i
};

// The later steps' keys: bucket b's entries [0, count), laid out in pieces of
// kStagePiece entries (2 MB) that take turns among the buckets, so that the
// ends of all buckets, where a step writes, lie close together (the buckets
// grow alike), and what is read of one bucket at a time lies in a few pieces.
constexpr u32 kStagePieceLog2 = 18;
struct StageRuns {
  unsigned long long* e;
  u32* count;              // [nb * kStageStride] (may pass cap: the rest were refused)
  u32 nb, cap;             // entries of a bucket
  __host__ __device__ __forceinline__ u64 at(u32 b, u32 i) const {
    return (((u64)(i >> kStagePieceLog2) * nb + b) << kStagePieceLog2) |
           (i & ((1u << kStagePieceLog2) - 1u));
  }
};

// Counters of one chunk, cleared together before it starts.  Counters that many
// warps add to at once lie in lines of their own: the adds to one line are
// served one after another (with a bucket's page counters in one line they
// bounded the stages, 23 ps a key).
constexpr u32 kStageStride = 64;   // in u32
struct StageChunk {
  u32 work[5][kStageStride];   // queue cursors: emit, the three stages, resolve
  u32 count[3][kStageBuckets * kStageStride];   // pages emitted; runs of stages 1 and 2
  u32 positives, pad[kStageStride - 1];
  u32 bloom[(1u << kBloomBits) / 32];
};

// sb with 16 * 2^sb < block <= 32 * 2^sb: 17 to 32 slices.
inline u32 stage_shift(u64 block) {
  u32 sb = 0;
  while ((block - 1) >> (sb + 5)) ++sb;
  return sb;
}

// ---- entries ------------------------------------------------------------------
// The first pages hold the key's hash h itself.  Later ones hold the mixed word
// g of the key's next cell (mix64 is a bijection, so h comes back from it)
// without what the bucket says, and the partial xor x of the low bits in the
// four bits that this frees: with g = q * block + (b << sb) + off, the entry is
// (q << sb | off) << 4 | x.  It fits: block > 16 * 2^sb, so q << sb | off < 2^60.
// (A byte array beside the entries took three times the stores' time: scattered
// byte stores are partial writes of a sector each.)
constexpr u64 inv64(u64 a) {   // a odd: a^-1 mod 2^64 by Newton's steps
  u64 x = a;
  for (int i = 0; i < 6; ++i) x *= 2 - a * x;
  return x;
}
__device__ __forceinline__ u64 unmix64(u64 x) {
  constexpr u64 i1 = inv64(0xc4ceb9fe1a85ec53ULL), i2 = inv64(0xff51afd7ed558ccdULL);
  x ^= x >> 33;
  x *= i1;
  x ^= x >> 33;
  x *= i2;
  x ^= x >> 33;
  return x;
}

// The word whose residue mod block is the key's t-th cell offset, and back.
template <int T>
__device__ __forceinline__ u64 cell_word(u64 h) {
  return T == 0 ? h : mix64(h ^ (T == 1 ? kPhi : kSalt2));
}
template <int T>
__device__ __forceinline__ u64 hash_of_word(u64 g) {
  return T == 0 ? g : unmix64(g) ^ (T == 1 ? kPhi : kSalt2);
}

// g = q * block + off (the exact quotient: mulhi undershoots it by at most 1).
__device__ __forceinline__ void split_word(u64 g, u32 block, u64 recip, u64& q, u32& off) {
  q = mulhi64(g, recip);
  u64 r = g - q * block;
  if (r >= block) { r -= block; ++q; }
  off = (u32)r;
}
__device__ __forceinline__ u64 pack_entry(u64 q, u32 off, u32 sb, u32 x) {
  return (((q << sb) | (off & ((1u << sb) - 1u))) << 4) | (x & 15u);
}
__device__ __forceinline__ u64 entry_word(u64 e, u32 b, u32 sb, u32 block) {
  const u64 v = e >> 4;
  return (v >> sb) * block + (((b << sb) | ((u32)v & ((1u << sb) - 1u))));
}

// ---- pages --------------------------------------------------------------------
// A warp gathers kStageHold keys in shared memory, orders them by bucket and
// appends each bucket's run to the page that it keeps open for the bucket (lane
// b holds bucket b's page and fill): a key costs an eighth of a store request
// of 32 lanes over a few runs.
constexpr u32 kStageHold = 256;
struct WarpHold {
  unsigned long long e[kStageHold];
  u16 meta[kStageHold];   // bucket | rank in the bucket's run << 5
};

struct StageOpen {
  u32 page = kStageNone, cnt = kStagePage;
  u32 held = 0;   // keys held by the warp
  u32 acc = 0;    // of bucket `lane`
};

// The held keys to their pages.  `direct(b, e)` probes a key whose bucket has no
// page left.  All lanes call this.
template <class Direct>
__device__ __forceinline__ void stage_flush(const StagePages& O, WarpHold& H, StageOpen& S, u32 lane,
                                            Direct direct) {
  constexpr u32 kFull = 0xFFFFFFFFu;
  if (S.held == 0) return;
  __syncwarp();
  u32 excl = S.acc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(kFull, excl, o);
    if (lane >= (u32)o) excl += y;
  }
  excl -= S.acc;
  unsigned long long e[kStageHold / 32];
  u32 m[kStageHold / 32];
#pragma unroll
  for (u32 k = 0; k < kStageHold / 32; ++k) {
    e[k] = H.e[k * 32 + lane];
    m[k] = H.meta[k * 32 + lane];
  }
  __syncwarp();
#pragma unroll
  for (u32 k = 0; k < kStageHold / 32; ++k) {
    const u32 pos = __shfl_sync(kFull, excl, m[k] & 31u) + (m[k] >> 5);
    if (k * 32 + lane < S.held) {
      H.e[pos] = e[k];
      H.meta[pos] = (u16)(m[k] & 31u);
    }
  }
  if (S.acc && S.cnt + S.acc > kStagePage) {   // acc > 0 only in lanes below nb
    if (S.page < O.cap) O.fill[lane * O.cap + S.page] = S.cnt;
    S.page = atomicAdd(O.npages + lane * kStageStride, 1u);
    S.cnt = 0;
    if (S.page >= O.cap) S.page = kStageFull;
  }
  __syncwarp();
  const bool open = S.page < O.cap;
  const u64 base = open ? ((u64)lane * O.cap + S.page) * kStagePage + S.cnt - excl : ~0ull;
#pragma unroll
  for (u32 k = 0; k < kStageHold / 32; ++k) {
    const u32 p = k * 32 + lane;
    const u32 b = p < S.held ? H.meta[p] : 0u;
    const u64 at = __shfl_sync(kFull, base, b);
    if (p < S.held) {
      if (at != ~0ull) O.e[at + p] = H.e[p];
      else direct(b, (u64)H.e[p]);
    }
  }
  if (open) S.cnt += S.acc;
  else S.cnt = S.page == kStageFull ? 0u : kStagePage;
  S.acc = 0;
  S.held = 0;
  __syncwarp();
}

// All lanes call this: active lanes hand in (b, e).
template <class Direct>
__device__ __forceinline__ void stage_push(const StagePages& O, WarpHold& H, StageOpen& S, bool act,
                                           u32 b, u64 e, u32 lane, Direct direct) {
  constexpr u32 kFull = 0xFFFFFFFFu;
  const u32 all = __ballot_sync(kFull, act), n = __popc(all);
  if (S.held + n > kStageHold) stage_flush(O, H, S, lane, direct);
  u32 own = all, mine = all;   // lanes of bucket `lane`, lanes of this key's bucket
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const u32 B = __ballot_sync(kFull, (b >> i) & 1u);
    own &= ((lane >> i) & 1u) ? B : ~B;
    mine &= ((b >> i) & 1u) ? B : ~B;
  }
  u32 lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  const u32 rank = __shfl_sync(kFull, S.acc, b) + __popc(mine & lt);
  if (act) {
    const u32 at = S.held + __popc(all & lt);
    H.e[at] = e;
    H.meta[at] = (u16)(b | (rank << 5));
  }
  S.acc += __popc(own);
  S.held += n;
}

// At the end of a kernel: the held keys go out, the open pages' fills are recorded.
template <class Direct>
__device__ __forceinline__ void stage_close(const StagePages& O, WarpHold& H, StageOpen& S, u32 lane,
                                            Direct direct) {
  stage_flush(O, H, S, lane, direct);
  if (lane < O.nb && S.page < O.cap) O.fill[lane * O.cap + S.page] = S.cnt;
}

// A key that the table holds: its bit in the chunk's Bloom filter.
__device__ __forceinline__ void stage_positive(StageChunk* C, u64 h) {
  const u32 bit = (u32)(h >> (64 - kBloomBits));
  atomicOr(&C->bloom[bit >> 5], 1u << (bit & 31u));
  atomicAdd(&C->positives, 1u);
}

}  // namespace s615
