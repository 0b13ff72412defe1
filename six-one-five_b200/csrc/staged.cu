// staged.cu -- the staged probe: large batches against tables past L2.
//
// A probe reads three scattered cells, and a B200 fills at most 4.7e10 of
// them a second from DRAM (21 ps each, 64 of the 64 ps a class-5 probe of the
// 3.2M band takes; the sieve itself is 7 ps).  From L2 the same reads take 3.5
// ps.  So a large batch is probed in chunks, in steps that each read a part
// of the table that stays in L2:
//
//   emit     the peel and the gate (k_peel) append each surviving key's hash to
//            one of 16 lists (for a table whose one-bit plane fits L2 beside
//            this: the keys that its bit leaves);
//   step 0   the keys are sorted by the slice of the first third that their first
//            cell lies in (a 17th to a 32nd of a third: 38 MB of four-bit cells
//            at most for N = 76,667);
//   step 1   slice by slice, four bits of the first cell are read from the plane,
//            which stays in L2, and the key goes on, with them, by the slice of its
//            second cell;
//   step 2   the same with the second and third cells;
//   step 3   the third cell's bits complete the comparison of the four bits; one
//            key in 16 passes and its cells are read in full.  A key that the
//            table holds sets its bit in the chunk's Bloom filter;
//   resolve  only if the chunk has such a key (a false positive of the filter
//            included): the peel runs over the chunk once more and probes the
//            keys whose bit is set, recording hits as ever.
//
// The comparison is the probe's own, cut in parts, so hits and counters are the
// direct probe's.  A key for which a list or bucket has no room is probed where it is.
//
// 12,000 units of the 3.2M class-5 band (20 chunks, 5.2e9 keys): 337 ms probed
// directly, 198 in stages: emit 55, steps 21, 37, 37 and 35, resolve 15.  6,000 units
// of the mixed stream at B <= 2M: 29.1 -> 16.5 ms.  Emit is bound by instruction
// issue, step 3 by the scattered reads of one key in 16, steps 1 and 2 by the chain
// load, plane read, order, store between block barriers (7 ps a key; the floor is
// 3.5 for a plane read and 2.4 for 16 bytes of HBM; 6 blocks of 256 or 10 of 128
// threads a SM: the same, 128 threads with 8 keys each: 230 ms a pass for 200).
// Emitting by slice at once, a page per warp and slice, took 74 ms where emit and
// step 0 take 76, and 12% more on the mixed stream; behind a one-bit plane it took
// 60 ps a key against 14 (page stores all over HBM and the plane's reads shared
// the TLB).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "staged.cuh"

namespace s615 {

int launch_stage_peel(s615_ctx* ctx, const TableView& tv, const s615_batch* b, unsigned flags,
                      cudaStream_t st, bool resolve, u32 lo, u32 hi, const StageRuns& list, StageChunk* chunk);

namespace {

constexpr int kThreads = 256;
constexpr int kPer = 4;        // keys per thread and pass

struct StageParams {
  TableView tv;
  const u32* plane;
  u32 sb;
  u32 bit0;           // the lowest of the four bits that the plane holds
  StageRuns in, out;
  StageChunk* chunk;
};

constexpr u32 kPlaneLb = 2;    // 4 bits of each cell, eight cells to a word

// A step's input as units of kUnit entries of one bucket (a piece is a multiple of
// a unit): warp-wide state.
template <u32 kUnit>
struct UnitOrder {
  u32 incl, n, total;
  __device__ __forceinline__ UnitOrder(const StageParams& P, u32 lane) {
    n = lane < P.in.nb ? (min(P.in.count[lane * kStageStride], P.in.cap) + kUnit - 1) / kUnit : 0u;
    incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= (u32)o) incl += y;
    }
    total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  // Unit g < total: its bucket, first entry and length.
  __device__ __forceinline__ void at(const StageParams& P, u32 g, u32& b, u64& e, u32& len) const {
    b = __popc(__ballot_sync(0xFFFFFFFFu, incl <= g));   // buckets wholly before unit g
    const u32 i = (g - __shfl_sync(0xFFFFFFFFu, incl - n, b)) * kUnit;
    e = P.in.at(b, i);
    len = min(min(P.in.count[b * kStageStride], P.in.cap) - i, kUnit);
  }
};

// Cell kStep - 1 of an entry of bucket b: its index in the table, and its word g.
template <int kStep>
__device__ __forceinline__ u64 stage_open(const StageParams& P, u64 e, u32 b, u64& g) {
  const u32 block = (u32)P.tv.block;
  g = entry_word(e, b, P.sb, block);
  return (u64)(kStep - 1) * block + ((b << P.sb) | ((u32)(e >> 4) & ((1u << P.sb) - 1u)));
}
__device__ __forceinline__ u32 plane_bits(u32 w, u64 c) { return w >> (((u32)c & 7u) << kPlaneLb); }

// Steps 0 to 2: look cell kStep - 1 up (step 0: nothing) and send the key on by cell
// kStep.  The block orders 1,024 keys by bucket in shared memory and appends each bucket's
// run (some 30 to 60 keys) to the bucket.
//
// Scattered accesses run at full rate only within the reach of the first-level
// TLB, which behaves like 128 entries of 2 MB in 8 sets (8 MB of lines in L2 read
// at 2.8e11/s within 128 MB, at 4.5e10/s spread over 1 GB), so input, output and
// plane slice are laid out to lie within that (StageRuns).  With the entries in a
// page per warp and bucket, each bucket in a region of its own, a step took 23 ps a
// key, against 7.
//
// A block always knows its next unit: the queue's answer and the buckets' new
// ends come back while it works.
template <int kStep>
__global__ void __launch_bounds__(kThreads, 5) k_stage(StageParams P) {
  constexpr u32 kNone = 0xFFFFFFFFu, kUnit = kThreads * kPer;
  __shared__ unsigned long long s_e[kUnit];
  __shared__ u8 s_b[kUnit];
  __shared__ u32 s_cnt[kStageBuckets], s_off[kStageBuckets], s_dst[kStageBuckets];
  __shared__ u64 s_at;
  __shared__ u32 s_in, s_len, s_total;
  const u32 tid = threadIdx.x, lane = tid & 31;
  const unsigned long long* in = P.in.e;
  const u32 block = (u32)P.tv.block, sb = P.sb;
  const u64 recip = P.tv.recip;
  const UnitOrder<kUnit> O(P, lane);
  // warp 0: unit g's place to shared memory (s_len = 0: no more units)
  auto place = [&](u32 g) {
    u32 b = 0, len = 0;
    u64 e = 0;
    if (g < O.total) O.at(P, g, b, e, len);
    if (lane == 0) { s_at = e; s_in = b; s_len = len; }
  };
  u32 next = 0;
  if (tid < 32) {
    if (lane == 0) next = atomicAdd(P.chunk->work[kStep + 1], 1u);
    place(__shfl_sync(0xFFFFFFFFu, next, 0));
    if (lane == 0) next = atomicAdd(P.chunk->work[kStep + 1], 1u);
    s_cnt[lane] = 0;
  }
  for (;;) {
    __syncthreads();
    const u32 len = s_len, ib = s_in;
    if (len == 0) break;
    const unsigned long long* src = in + s_at;
    u64 g[kPer];
    u32 w[kPer], x[kPer], at[kPer], act = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const u32 i = (u32)k * kThreads + tid;
      const bool on = i < len;
      g[k] = on ? (u64)__ldcs(src + i) : 0;
      act |= (u32)on << k;
    }
    // the plane's answers come back while the next words are worked out
    if constexpr (kStep > 0) {
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const u32 e = (u32)g[k];
        const u64 c = stage_open<kStep>(P, g[k], ib, g[k]);
        x[k] = (e & 15u) | ((u32)c & 7u) << 6;   // low bits so far | 4 * (cell % 8)
        const bool on = ((act >> k) & 1u) && S615_CHECK(c < 3 * (u64)block, kChkCell);
        w[k] = on ? __ldcg(P.plane + (c >> (5 - kPlaneLb))) : 0u;
      }
    } else {   // the hash's own bits to begin with
#pragma unroll
      for (int k = 0; k < kPer; ++k) { x[k] = (u32)(g[k] >> P.bit0) & 15u; w[k] = 0; }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      u64 q;
      u32 off;
      split_word(cell_word<kStep>(hash_of_word<kStep ? kStep - 1 : 0>(g[k])), block, recip, q, off);
      g[k] = pack_entry(q, off, sb, 0);
      const u32 b = off >> sb;
      at[k] = ((act >> k) & 1u) ? b | (atomicAdd(&s_cnt[b], 1u) << 5) : kNone;
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) g[k] |= (x[k] ^ (w[k] >> (x[k] >> 4))) & 15u;
    __syncthreads();
    u32 base = 0, off0 = 0;
    if (tid < 32) {   // the runs' places: lane b for bucket b
      const u32 r = s_cnt[lane];
      if (r) base = atomicAdd(P.out.count + lane * kStageStride, r);
      s_cnt[lane] = 0;
      u32 incl = r;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (u32)o) incl += y;
      }
      off0 = incl - r;
      s_off[lane] = off0;
      if (lane == 31) s_total = incl;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (at[k] != kNone) {
        const u32 b = at[k] & 31u, pos = s_off[b] + (at[k] >> 5);
        s_e[pos] = g[k];
        s_b[pos] = (u8)b;
      }
    if (tid < 32) {
      place(__shfl_sync(0xFFFFFFFFu, next, 0));
      if (lane == 0) next = atomicAdd(P.chunk->work[kStep + 1], 1u);
      s_dst[lane] = base - off0;   // entry i of the tile goes to place s_dst + i
    }
    __syncthreads();
    const u32 total = s_total;
    for (u32 pos = tid; pos < total; pos += kThreads) {
      const u32 b = s_b[pos], i = s_dst[b] + pos;
      const u64 e = s_e[pos];
      if (i < P.out.cap) {
        __stcs(P.out.e + P.out.at(b, i), (unsigned long long)e);
      } else {   // no room left in the bucket: probed here
        const u64 h = hash_of_word<kStep>(entry_word(e, b, sb, block));
        if (contains_hash<false>(P.tv, h)) stage_positive(P.chunk, h);
      }
    }
  }
}

// Step 3: the last cell's low bits; one key in 16 agrees and is probed in full.
// Warps take units of 1,024 keys, eight keys a lane in flight.  The keys that
// agree gather in shared memory and are probed 32 at a time: probed where they
// come up, two lanes of a warp at a time would wait for their cells, eight times
// for 256 keys (44.5 ms of a 12,000-unit chunk of the 3.2M band; 41.8 ms so).
constexpr u32 kTake = 1024;
constexpr u32 kAgree = 32 + 256;   // at most 31 left over and 256 new
__global__ void __launch_bounds__(kThreads) k_stage_last(StageParams P) {
  __shared__ unsigned long long s_agree[kThreads / 32][kAgree];
  unsigned long long* agree = s_agree[threadIdx.x >> 5];
  const u32 lane = threadIdx.x & 31;
  u32 lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  const UnitOrder<kTake> O(P, lane);
  u32 next = 0, held = 0;
  if (lane == 0) next = atomicAdd(P.chunk->work[4], 1u);
  auto probe = [&](u32 first, u32 n) {   // entries [first, first + n), n <= 32: words of cell 2
    if (lane < n) {
      const u64 h = hash_of_word<2>(agree[first + lane]);
      if (contains_hash<false>(P.tv, h)) stage_positive(P.chunk, h);
    }
  };
  for (;;) {
    const u32 unit = __shfl_sync(0xFFFFFFFFu, next, 0);
    if (unit >= O.total) break;
    if (lane == 0) next = atomicAdd(P.chunk->work[4], 1u);
    u32 b, len;
    u64 at;
    O.at(P, unit, b, at, len);
    for (u32 i0 = 0; i0 < len; i0 += 256u) {
      u64 e[8];
      u32 x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const u32 i = i0 + 32u * k + lane;
        e[k] = i < len ? (u64)__ldcs(P.in.e + at + i) : 0;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const u64 c = 2 * P.tv.block + ((u64)b << P.sb) + ((e[k] >> 4) & ((1ull << P.sb) - 1));
        const bool on = i0 + 32u * k + lane < len && S615_CHECK(c < 3 * P.tv.block, kChkCell);
        x[k] = on ? (u32)e[k] ^ plane_bits(__ldcg(P.plane + (c >> (5 - kPlaneLb))), c) : 1u;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool ok = !(x[k] & 15u);
        const u32 all = __ballot_sync(0xFFFFFFFFu, ok);
        if (ok) agree[held + __popc(all & lt)] = entry_word(e[k], b, P.sb, (u32)P.tv.block);
        held += __popc(all);
      }
      __syncwarp();
      u32 done = 0;
      for (; held - done >= 32u; done += 32u) probe(done, 32u);
      if (done) {   // the rest to the front (fewer than 32)
        const u64 rest = lane < held - done ? (u64)agree[done + lane] : 0;
        __syncwarp();
        if (lane < held - done) agree[lane] = rest;
        held -= done;
        __syncwarp();
      }
    }
  }
  probe(0, held);
}

template <class K>
int launch_stage(s615_ctx* ctx, K kernel, const StageParams& P, cudaStream_t st) {
  int per_sm = 0;
  S615_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0));
  kernel<<<ctx->num_sms * std::max(per_sm, 1), kThreads, 0, st>>>(P);
  ctx->launches++;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

// Keys per chunk: enough that reading the plane once per chunk and the ends of
// seven launches are small beside it, few enough that most chunks of a search hold
// no key of the table (about one in 1e9) and skip the resolve pass.
constexpr u64 kMaxChunkKeys = 1ull << 28, kMinChunkKeys = 1ull << 26;
// The least keys for which the stages pay: below, seven launches and their ends
// cost more than the scattered reads.  Direct / staged, ms, class-5 units:
// 1e7 keys 0.74 / 0.69 (N = 42,000), 0.55 / 0.60 (31,000); 2e7 1.47 / 1.07 and
// 0.99 / 0.91; 2.4e7 1.72 / 1.44 (76,667), but 1.64 / 1.74 with a key of the table
// among them, when the resolve pass runs; 4.4e7 2.93 / 2.22; 1e8 7.2 / 4.4.
constexpr double kMinKeys = 2.5e7;

// Two spaces in turn: the emitted keys, then by first cell, by second (in the first
// space again), by third.
struct Layout {
  u32 nb = 0, list = 0, entries = 0;   // room of an emitted list and of a bucket
  size_t first = 0, second = 0, bytes = 0;
};
Layout layout_for(u64 keys, u32 nb) {
  Layout L;
  L.nb = nb;
  const auto room = [&](u32 parts) {
    return (u32)((((keys + keys / 8) / parts >> kStagePieceLog2) + 1) << kStagePieceLog2);
  };
  L.list = room(kStageLists);
  L.entries = room(nb);
  L.second = (size_t)nb * L.entries * 8;
  L.first = std::max(L.second, (size_t)kStageLists * L.list * 8);
  L.bytes = (sizeof(StageChunk) + 255) / 256 * 256 + L.first + L.second;
  return L;
}
// What a space for chunks of `keys` keys takes, whatever the table (layout_for rounds
// each of at most kStageBuckets parts up by at most a piece).
size_t space_bytes(u64 keys) {
  return (sizeof(StageChunk) + 255) / 256 * 256 +
         2 * 8 * ((size_t)(keys + keys / 8) + ((size_t)kStageBuckets << kStagePieceLog2));
}

constexpr double kSlack = 1.05;   // of the estimated keys

// The context's space, for chunks of `want` keys, or of kMinChunkKeys at least; false:
// there is no room.  It is taken at its largest useful size, a quarter of the room at
// most, by the first run that wants one, so later runs neither allocate nor wait.
// (Grown to each new largest batch, it was freed and allocated inside s615_run_batch,
// behind the work in flight on every stream; and an allocation soon after the free
// stalled: the first pass over the 155,391-unit band after a 300-unit one took 3,140 ms,
// two times of three, where a pass takes 2,530.)  A space that little room made smaller
// is given up for a larger one only when nothing has to be waited for.
bool take_space(s615_ctx* ctx, u64 want) {
  StageSpace& w = ctx->stage;
  const u64 least = std::min(want, kMinChunkKeys);
  const CaptureRelaxed relaxed;
  if (w.p && (w.keys >= want || !device_idle(ctx))) return w.keys >= least;
  const size_t room = w.bytes + hbm_room(ctx) / 4;
  u64 keys = kMaxChunkKeys;
  while (space_bytes(keys) > room && keys > kMinChunkKeys) keys /= 2;
  if (space_bytes(keys) > room) keys = least;
  if (keys <= w.keys) return w.keys >= least;
  if (space_bytes(keys) > room) return false;
  stage_release(ctx);
  void* p = nullptr;
  if (dev_alloc_once(ctx, &p, space_bytes(keys))) return false;
  w.p = p;
  w.bytes = space_bytes(keys);
  w.keys = keys;
  return true;
}

}  // namespace

size_t stage_least_bytes(bool eplane) { return space_bytes((u64)(kMinKeys * kSlack / (eplane ? 2 : 1))); }

void stage_release(s615_ctx* ctx) {
  StageSpace& w = ctx->stage;
  if (w.last) {
    cudaEventSynchronize(w.last);
    cudaEventDestroy(w.last);
    w.last = nullptr;
  }
  dev_free(ctx, w.p, w.bytes);
  w.p = nullptr;
  w.bytes = 0;
  w.keys = 0;
}

// *done = true when the classes 2-5 items of b were probed in stages.
int launch_staged(s615_ctx* ctx, const TableView& tv, s615_batch* b, unsigned flags, cudaStream_t st,
                  bool* done) {
  *done = false;
  double est = b->est_keys;
  if (flags & S615_F_NO_GATE) est *= 37;   // 2.7% of the points pass the gate
  if (!tv.splane || tv.shards > 1 || (flags & S615_F_SHARP) || est < kMinKeys || !b->n_main)
    return S615_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return S615_OK;
  }
  if (tv.eplane) est /= 2;   // the keys that its bit leaves
  std::lock_guard<std::mutex> lock(ctx->stage.mu);
  StageSpace& w = ctx->stage;
  // chunks of at most kMaxChunkKeys keys, smaller when HBM is short
  const u64 want = (u64)std::min<double>(est * kSlack, (double)kMaxChunkKeys);
  if (!take_space(ctx, want)) return S615_OK;
  const u64 keys = std::min(want, w.keys);
  const u32 sb = stage_shift(tv.block);
  const u32 nb = (u32)((tv.block + (1ull << sb) - 1) >> sb);
  const Layout L = layout_for(keys, nb);
  if (!w.last) S615_CU(cudaEventCreateWithFlags(&w.last, cudaEventDisableTiming));
  else S615_CU(cudaStreamWaitEvent(st, w.last, 0));   // the space's last user, on any stream
  *done = true;
  StageChunk* chunk = static_cast<StageChunk*>(w.p);
  char* at = static_cast<char*>(w.p) + (sizeof(StageChunk) + 255) / 256 * 256;
  auto* first = reinterpret_cast<unsigned long long*>(at);
  auto* second = reinterpret_cast<unsigned long long*>(at + L.first);
  const StageRuns list{first, chunk->count[0], kStageLists, L.list};
  const u64 chunks = std::max<u64>(1, (u64)(est / (double)keys + 0.999));
  int s = S615_OK;
  for (u64 c = 0; c < chunks && !s; ++c) {
    const u32 lo = (u32)(b->n_main * c / chunks), hi = (u32)(b->n_main * (c + 1) / chunks);
    if (lo == hi) continue;
    if (cudaMemsetAsync(chunk, 0, sizeof(StageChunk), st) != cudaSuccess) { s = S615_E_DEVICE; break; }
    if ((s = launch_stage_peel(ctx, tv, b, flags, st, false, lo, hi, list, chunk))) break;
    StageParams P{};
    P.tv = tv;
    P.plane = tv.splane;
    P.bit0 = tv.eplane ? 1u : 0u;
    P.sb = sb;
    P.chunk = chunk;
    P.out = list;
    for (int k = 0; k < 3 && !s; ++k) {
      P.in = P.out;
      P.out = StageRuns{k == 1 ? first : second, chunk->count[k + 1], nb, L.entries};
      s = k == 0 ? launch_stage(ctx, k_stage<0>, P, st)
        : k == 1 ? launch_stage(ctx, k_stage<1>, P, st) : launch_stage(ctx, k_stage<2>, P, st);
    }
    if (s) break;
    P.in = P.out;
    if ((s = launch_stage(ctx, k_stage_last, P, st))) break;
    s = launch_stage_peel(ctx, tv, b, flags, st, true, lo, hi, list, chunk);
  }
  cudaEventRecord(w.last, st);
  return s;
}

S615_CHECK_TAKE_DEFINE(check_take_staged)

}  // namespace s615
