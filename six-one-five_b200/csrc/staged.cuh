// staged.cuh -- key lists of the staged probe (staged.cu) and the warp-wide push
// that fills the first.
#pragma once
#include <cuda_runtime.h>

#include "s615_device.cuh"

namespace s615 {

// Keys wait in buckets: bucket b holds the keys whose next cell lies in the b-th
// slice of 2^sb cells of its third.  17 to 32 buckets (stage_shift), so a lane can
// stand for each.  The emitted keys, in no order, are kStageLists lists alike.
constexpr u32 kStageBuckets = 32;
constexpr u32 kStageLists = 16;
constexpr u32 kBloomBits = 19;             // positives of a chunk: 2^19 bits, 64 KB

// Bucket b's entries [0, count), laid out in pieces of
// kStagePiece entries (2 MB) that take turns among the buckets, so that the
// ends of all buckets, where a step writes, lie close together (the buckets
// grow alike), and what is read of one bucket at a time lies in a few pieces.
constexpr u32 kStagePieceLog2 = 18;
struct StageRuns {
  unsigned long long* e;
  u32* count;              // [nb * kStageStride] (may pass cap: those keys were refused)
  u32 nb, cap;             // entries of a bucket
  __host__ __device__ __forceinline__ u64 at(u32 b, u32 i) const {
    return (((u64)(i >> kStagePieceLog2) * nb + b) << kStagePieceLog2) |
           (i & ((1u << kStagePieceLog2) - 1u));
  }
};

// Counters of one chunk, cleared together before it starts.  Counters that many
// warps add to at once lie in lines of their own: the adds to one line are
// served one after another (with the buckets' counters in one line they
// bounded the stages, 23 ps a key).
constexpr u32 kStageStride = 64;   // in u32
struct StageChunk {
  u32 work[6][kStageStride];   // queue cursors: emit, steps 0 to 3, resolve
  u32 count[4][kStageBuckets * kStageStride];   // keys emitted; sorted by cell 0, 1, 2
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
// The emitted entries are the keys' hashes h.  Later ones hold the word g of the
// key's next cell (h, or a mix of it: mix64 is a bijection, so h comes back)
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

// ---- emitted keys -------------------------------------------------------------
// A warp gathers keys in shared memory and appends kStageHold at a time to its
// list: whole lines, and all warps' stores within a window of a few MB that moves
// on, which leaves the first-level TLB to whatever else the kernel reads.
constexpr u32 kStageHold = 256;
struct WarpHold {
  unsigned long long e[kStageHold + 32];
};

// Appends the first n held keys; `direct(e)` probes a key that the list has no
// room for.  All lanes call this.  A full list's counter is put back, so it stays
// within what the warps add at once past the list's end.  Items are dealt to chunks by
// number, and a chunk of the heaviest ones can hold hundreds of times the keys it was
// sized for: with 2^32 for one list the counter would wrap and the list's keys be
// overwritten.
template <class Direct>
__device__ __forceinline__ void stage_append(const StageRuns& O, u32 list, const WarpHold& H, u32 n,
                                             u32 lane, Direct direct) {
  u32 i0 = 0;
  if (lane == 0) {
    i0 = atomicAdd(O.count + list * kStageStride, n);
    if (i0 >= O.cap) atomicSub(O.count + list * kStageStride, n);
  }
  i0 = __shfl_sync(0xFFFFFFFFu, i0, 0);
#pragma unroll 4
  for (u32 p = lane; p < n; p += 32) {
    const u64 e = H.e[p];
    if (i0 + p < O.cap) __stcs(O.e + O.at(list, i0 + p), (unsigned long long)e);
    else direct(e);
  }
}

// All lanes call this: active lanes hand in e.
template <class Direct>
__device__ __forceinline__ void stage_push(const StageRuns& O, u32 list, WarpHold& H, u32& held, bool act,
                                           u64 e, u32 lane, Direct direct) {
  const u32 all = __ballot_sync(0xFFFFFFFFu, act);
  u32 lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  if (act) H.e[held + __popc(all & lt)] = e;
  held += __popc(all);
  if (held < kStageHold) return;
  __syncwarp();
  stage_append(O, list, H, kStageHold, lane, direct);
  held -= kStageHold;
  const u64 rest = H.e[kStageHold + lane];   // fewer than 32
  __syncwarp();
  if (lane < held) H.e[lane] = rest;
  __syncwarp();
}

// At the end of a kernel: the rest goes out.
template <class Direct>
__device__ __forceinline__ void stage_close(const StageRuns& O, u32 list, WarpHold& H, u32 held, u32 lane,
                                            Direct direct) {
  __syncwarp();
  stage_append(O, list, H, held, lane, direct);
}

// A key that the table holds: its bit in the chunk's Bloom filter.
__device__ __forceinline__ void stage_positive(StageChunk* C, u64 h) {
  const u32 bit = (u32)(h >> (64 - kBloomBits));
  atomicOr(&C->bloom[bit >> 5], 1u << (bit & 31u));
  atomicAdd(&C->positives, 1u);
}

}  // namespace s615
