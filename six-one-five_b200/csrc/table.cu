// table.cu -- xor-filter query and the packed <-> wide HBM layouts.
//
// k_xor_query is the device form of xor_might_contain
// (spike/ribbon/xor_filter.hpp:472-483, fourcore_cls5_gpu_v4.cu:322-334):
// identical hash, cell indices and fingerprint comparison.  Cell indices are
// 64-bit (the reference's u32 variant in fourcore_find_device.cuh:54-63
// wraps once 3*block > 2^32).
#include <cuda_runtime.h>

#include <algorithm>

#include "s615_device.cuh"

namespace s615 {

namespace {

__global__ void k_xor_query(TableView t, const u64* __restrict__ keys, u64 n,
                            u8* __restrict__ out) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x)
    out[i] = might_contain(t, keys[i]) ? 1 : 0;
}

// One thread per cell: gather r bits from the packed bytes (read as aligned
// 64-bit words) into a 4- or 8-byte wide cell.
__global__ void k_unpack(const unsigned long long* __restrict__ packed, u64 m, u32 r,
                         void* __restrict__ wide, int cell_bytes) {
  const u64 mask = fp_mask(r);
  for (u64 c = blockIdx.x * (u64)blockDim.x + threadIdx.x; c < m;
       c += (u64)gridDim.x * blockDim.x) {
    const u64 bit = c * (u64)r, w = bit >> 6;
    const u32 o = (u32)(bit & 63);
    u64 v = packed[w] >> o;
    if (o + r > 64) v |= packed[w + 1] << (64 - o);
    v &= mask;
    if (cell_bytes == 8) static_cast<u64*>(wide)[c] = v;
    else static_cast<u32*>(wide)[c] = (u32)v;
  }
}

// One thread per output 64-bit word: OR in every cell overlapping bits
// [64w, 64w+64).  No two threads write the same word, so no atomics.
template <typename Cell>
__global__ void k_pack(const Cell* __restrict__ wide, u64 m, u32 r,
                       unsigned long long* __restrict__ packed, u64 n_words) {
  const u64 mask = fp_mask(r);
  for (u64 w = blockIdx.x * (u64)blockDim.x + threadIdx.x; w < n_words;
       w += (u64)gridDim.x * blockDim.x) {
    const u64 lo = w * 64;
    u64 c = lo / r;
    u64 word = 0;
    for (; c < m; ++c) {
      const u64 p = c * (u64)r;
      if (p >= lo + 64) break;
      const u64 v = (u64)wide[c] & mask;
      if (p >= lo) word |= v << (p - lo);
      else word |= v >> (lo - p);
    }
    packed[w] = word;
  }
}

// One thread per 32-bit plane word: 2^lb bits, from bit `shift` on, of its 32 >> lb cells.
__global__ void k_plane(const void* __restrict__ cells, u32 layout, u32 cell_bytes, u32 r, u64 m,
                        u32 lb, u32 shift, u32* __restrict__ plane, u64 n_words) {
  const u32 per = 32u >> lb, bits = 1u << lb;
  const u32 mask = (u32)((1ull << bits) - 1);
  for (u64 w = blockIdx.x * (u64)blockDim.x + threadIdx.x; w < n_words;
       w += (u64)gridDim.x * blockDim.x) {
    const u64 c0 = w * per;
    u32 word = 0;
    for (u32 k = 0; k < per && c0 + k < m; ++k)
      word |= ((u32)(load_cell_at(cells, layout, cell_bytes, r, fp_mask(r), c0 + k) >> shift) & mask) << (k * bits);
    plane[w] = word;
  }
}

// Picoseconds per scattered read over a footprint, the whole GPU reading
// (measured on a B200: 2.85e11 reads/s up to 64 MB, 4.71e10 /s at 28 GB).
double read_ps(double mb) {
  static const double at[][2] = {{64, 3.5},   {80, 4.25},  {96, 6.2},    {112, 8.1},   {128, 9.6},
                                 {160, 11.7}, {192, 13.0}, {256, 14.7},  {384, 16.3},  {512, 17.1},
                                 {1024, 18.5}, {2048, 19.7}, {4096, 20.4}, {8192, 21.1}};
  constexpr int n = sizeof at / sizeof at[0];
  if (mb <= at[0][0]) return at[0][1];
  for (int i = 1; i < n; ++i)
    if (mb <= at[i][0])
      return at[i - 1][1] + (at[i][1] - at[i - 1][1]) * (mb - at[i - 1][0]) / (at[i][0] - at[i - 1][0]);
  return at[n - 1][1];
}

int grid_for(s615_ctx* ctx, u64 n, int threads) {
  const u64 want = (n + threads - 1) / threads;
  const u64 cap = (u64)ctx->num_sms * 16;
  return (int)(want < cap ? (want ? want : 1) : cap);
}

}  // namespace

TableView view_of(const DevTable& t) {
  TableView v{};
  v.shards = 1;
  if (!t.parts.empty()) {   // a shard set: the parts' views live in HBM
    v.shards = t.hdr.shard_count;
    v.block = v.shards;   // the shard index is fast_mod(mix, S, recip)
    v.recip = mod_recip(v.shards);
    v.parts = static_cast<const TableView*>(t.d_views);
    v.shard_seed = kShardSeed;
    size_t bytes = 0;
    for (const DevTable& p : t.parts) bytes += p.bytes;
    const u64 want = t.groups ? t.groups : (bytes + kProbeGroupBytes - 1) / kProbeGroupBytes;
    v.groups = (u32)std::min<u64>(std::max<u64>(want, 1), t.parts.size());
    v.grp_lo = t.shard_lo;   // the shards this set holds; other keys are not its to probe
    v.grp_hi = t.shard_lo + (u32)t.parts.size();
    v.r = t.hdr.r;
    v.fpmask = fp_mask(t.hdr.r);
    return v;
  }
  v.cells = t.d_cells;
  v.block = t.hdr.m_cells / 3;
  v.recip = mod_recip(v.block);
  v.fpmask = fp_mask(t.hdr.r);
  v.seed = t.hdr.mix_seed;
  v.r = t.hdr.r;
  v.layout = (u32)t.layout;
  v.cell_bytes = (u32)t.cell_bytes;
  v.plane = static_cast<const u32*>(t.d_plane);
  v.splane = static_cast<const u32*>(t.d_splane);
  v.eplane = static_cast<const u32*>(t.d_eplane);
  v.plane_lb = t.plane_lb;
  v.plane_mask = (u32)((1ull << (1u << t.plane_lb)) - 1);
  if (t.hdr.n_keys == 0 || t.hdr.m_cells < 3) v.block = 0;
  return v;
}

// Bytes of a plane of 2^lb bits of m cells: whole cells per 32-bit word.
static size_t plane_size(u64 m, int lb) {
  const u64 per = 32u >> lb;
  return (m + per - 1) / per * sizeof(u32);
}

// 2^lb bits of t's cells, from bit `shift` on; *p stays null when there is no room.
static int make_plane(s615_ctx* ctx, const DevTable& t, int lb, u32 shift, cudaStream_t st, void** p,
                      size_t* bytes) {
  const u64 m = t.hdr.m_cells, words = plane_size(m, lb) / sizeof(u32);
  if (dev_alloc_once(ctx, p, words * sizeof(u32))) return S615_OK;
  k_plane<<<grid_for(ctx, words, 256), 256, 0, st>>>(t.d_cells, (u32)t.layout, (u32)t.cell_bytes,
                                                     t.hdr.r, m, (u32)lb, shift,
                                                     static_cast<u32*>(*p), words);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    dev_free(ctx, *p, words * sizeof(u32));
    *p = nullptr;
    return cuda_status(e);
  }
  *bytes = words * sizeof(u32);
  return S615_OK;
}

// A probe costs three scattered reads of cells, or with a plane of b bits
// three reads of the plane and, for 2^-b of the probes, three of cells.  The
// widths tried are 1, 2, 4 and 8 bits, up to 112 MB; the cheapest by read_ps
// is taken when it saves a tenth.  Past 112 MB (N above about 39,000 at one
// bit) the plane is mostly read from DRAM itself: a 4-bit plane of 468 MB gave
// a class-5 pass 7% and took 14% from a mixed one.  Measured, ps per probe
// through the cells alone / with the plane: class 5, N = 12,000 (4 bits) 65.5
// / 43.6, 20,000 (2 bits) 63.2 / 25.5, 24,000 (2 bits) 63.2 / 30.2, 31,000 (1
// bit) 63.1 / 42.9, 36,000 (1 bit) 63.2 / 47.5; (6,1,7), N = 10,476 (8 bits) 54.7 /
// 14.  Three reads of a 64 MB plane are 10.5 ps.
constexpr double kPlaneMaxMB = 112;
// The staged probe takes 33 to 36 ps a key whatever the table, 28 of them after the
// sieve, so tables whose probe costs more than kStagedFrom by this count get its
// planes as well, for their large batches: four bits, and if it is small enough to
// be read at the full rate beside the sieve (58 MB: 14 ps a key; 70 MB 21, 84 MB
// 27), a plane of one bit that keeps half of the keys out of the stages.  2e8
// class-5 keys, ps a key probed directly / in stages: N = 22,000 28.0 / 28.6 (left as
// it is), 24,000 30.8 / 28.3, 26,500 34.7 / 27.6, 28,000 41.5 / 28.6, 29,500 (four bits
// only from here) 42.7 / 33.2, 31,000 43.0 / 32.9, 36,000 47.9 / 35.3, 42,000 61.5 / 34.8,
// 76,667 63.8 / 36.3.
constexpr double kStagedFrom = 29;
constexpr u64 kEPlaneMax = 60ull << 20;
int build_plane(s615_ctx* ctx, DevTable& t, cudaStream_t st) {
  const u64 m = t.hdr.m_cells;
  if (!t.d_cells || t.hdr.n_keys == 0 || m < 3) return S615_OK;
  const double cell_ps = 3 * read_ps((double)t.bytes / 1048576.0);
  double best = 0.9 * cell_ps;
  int lb = -1;
  for (int k = 0; k < 4; ++k) {
    const u32 bits = 1u << k;
    if (bits > t.hdr.r) break;
    const double mb = (double)m * bits / 8 / 1048576.0;
    const double ps = 3 * read_ps(mb) + cell_ps / (double)(1u << bits);
    if (mb <= kPlaneMaxMB && ps < best) { best = ps; lb = k; }
  }
  // (Planes yield: an allocation that finds no room gives them back, release_planes.)
  if (lb >= 0) {
    if (const int s = make_plane(ctx, t, lb, 0, st, &t.d_plane, &t.plane_bytes)) return s;
    t.plane_lb = (u32)lb;
  }
  // The staged probe's plane, when its slices (staged.cuh) fit L2.  Below 16 bits
  // the filter's own false positives (2^-r of the keys) fill the chunk's Bloom
  // filter, and the last pass would probe most keys again.
  if ((t.d_plane ? best : cell_ps) < kStagedFrom || t.bytes < ((size_t)1 << 28) || t.hdr.r < 16 ||
      m / 2 / 3 / 16 > kStageSlice)
    return S615_OK;
  // At most a quarter of the room that is left; and it is of use only to runs that
  // find a quarter of what then remains enough for their keys (launch_staged's rule).
  const bool one_bit = m / 8 <= kEPlaneMax, own = one_bit && !(t.d_plane && lb == 0);
  const size_t want = plane_size(m, 2) + (own ? plane_size(m, 0) : 0);
  const size_t room = hbm_room(ctx);
  if (4 * want > room || 4 * stage_least_bytes(one_bit) > room - want) return S615_OK;
  if (own) {
    if (const int s = make_plane(ctx, t, 0, 0, st, &t.d_eplane, &t.eplane_bytes)) return s;
  } else if (one_bit) {
    t.d_eplane = t.d_plane;
  }
  const int s = make_plane(ctx, t, 2, t.d_eplane ? 1u : 0u, st, &t.d_splane, &t.splane_bytes);
  if (s || t.d_splane) return s;
  if (own) dev_free(ctx, t.d_eplane, t.eplane_bytes);   // of no use alone
  t.d_eplane = nullptr;
  t.eplane_bytes = 0;
  return S615_OK;
}

int launch_xor_query(s615_ctx* ctx, const TableView& tv, const u64* d_keys, size_t n,
                     u8* d_out, cudaStream_t st) {
  if (n == 0) return S615_OK;
  k_xor_query<<<grid_for(ctx, n, 256), 256, 0, st>>>(tv, d_keys, n, d_out);
  ctx->launches++;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

int launch_unpack(s615_ctx* ctx, const u8* d_packed, u64 m, u32 r, void* d_wide, int cell_bytes,
                  cudaStream_t st) {
  if (m == 0) return S615_OK;
  k_unpack<<<grid_for(ctx, m, 256), 256, 0, st>>>(
      reinterpret_cast<const unsigned long long*>(d_packed), m, r, d_wide, cell_bytes);
  ctx->launches++;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

int launch_pack(s615_ctx* ctx, const void* d_wide, int cell_bytes, u64 m, u32 r, u8* d_packed,
                u64 packed_len, cudaStream_t st) {
  const u64 n_words = (packed_len + 7) / 8;
  if (n_words == 0) return S615_OK;
  auto* out = reinterpret_cast<unsigned long long*>(d_packed);
  if (cell_bytes == 8)
    k_pack<<<grid_for(ctx, n_words, 256), 256, 0, st>>>(static_cast<const u64*>(d_wide), m, r, out,
                                                        n_words);
  else
    k_pack<<<grid_for(ctx, n_words, 256), 256, 0, st>>>(static_cast<const u32*>(d_wide), m, r, out,
                                                        n_words);
  ctx->launches++;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

S615_CHECK_TAKE_DEFINE(check_take_table)

}  // namespace s615
