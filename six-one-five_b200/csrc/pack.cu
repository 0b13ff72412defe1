// pack.cu -- unit records and work items made on the device.
//
// make_dev_unit (host_math.cpp) and unit_items (engine.hpp) for the units of
// classes 1-5, of all three kinds, and (6,1,7) find4 jobs, one thread per unit: the
// caller's 72-byte records cross the bus instead of 224-byte ones and 8-byte
// items, and the host works out no residues.  (214,000 reduced-T jobs: 8 of the
// 10 ms of a call were the host's packing and a 48 MB upload, 11 -> 4.4 ms with
// class-1 jobs among them; 100,001 (6,1,7) find4 jobs 25.2 -> 21.5 ms.)  Batches with
// (6,1,7) class-5 candidates are packed on the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "pack.cuh"
#include "s615_device.cuh"

namespace s615 {

namespace {

constexpr u64 kMaxB = 40000000ULL;   // make_dev_unit's bound

// ---- three-limb words, as host_math.cpp's W3 -----------------------------------
__device__ __forceinline__ W3 d_pow6(u64 x) {   // x < 2^32
  const u64 a = x * x;
  const u128 x4 = (u128)a * a, lo = (u128)(u64)x4 * a, hi = (u128)(u64)(x4 >> 64) * a;
  const u128 mid = (lo >> 64) + (u128)(u64)hi;
  return W3{{(u64)lo, (u64)mid, (u64)(hi >> 64) + (u64)(mid >> 64)}};
}
__device__ __forceinline__ bool d_sub(W3& a, const W3& b) {   // a -= b, true on borrow
  u64 br = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const u128 d = (u128)a.l[i] - b.l[i] - br;
    a.l[i] = (u64)d;
    br = (u64)(d >> 64) ? 1 : 0;
  }
  return br != 0;
}
// a mod m for m < 2^33, and floor(a / 21^6) mod 2^64 is not needed beyond its low
// bits: the caller divides exactly.
__device__ __forceinline__ u64 d_mod(const W3& a, u64 m) {
  u128 r = 0;
#pragma unroll
  for (int i = 2; i >= 0; --i) r = ((r << 64) | a.l[i]) % m;
  return (u64)r;
}

// 42^6 | base - (f d0)^6, or the difference is negative (divisible_row234).
__device__ bool row_ok(const W3& base, u32 f, u32 d0) {
  W3 R = base;
  return d_sub(R, d_pow6((u64)f * d0)) || d_mod(R, kM42) == 0;
}
// base - (14 e0)^6 divisible by 21^6 with quotient d0^6 (mod 64), or negative
// (divisible_grid5 with one d0).  The exact quotient mod 64 is R * 21^-6 mod 64.
__device__ bool grid_ok(const W3& base, u32 e0, u32 d0, u32 inv21_64) {
  W3 R = base;
  if (d_sub(R, d_pow6(14ull * e0))) return true;
  if (d_mod(R, kM21) != 0) return false;
  return (((u32)R.l[0] & 63u) * inv21_64 & 63u) == pow6_mod_u32(d0, 64);
}

// A reduced-T job of classes 2-5 that becomes a job row; *find2 for class 5.
__device__ __forceinline__ bool job_row(const s615_unit& u, bool* find2) {
  *find2 = u.cls == 5;
  if (u.kind != S615_KIND_JOB || u.cls < 2 || u.cls > 5) return false;
  return u.cls == 5 || ((u.base[0] | u.base[1]) != 0 && (u.base[1] >> 57) == 0);   // 0 < T < 2^121
}

// Class 1, target T in 1 .. 2^126 - 1: the c4 window [least c with 4 c^6 >= T,
// min(T^(1/6), lim)]; true if it is empty (4 c^6 >= T iff c^6 > floor((T - 1) / 4)).
__device__ bool find4_window(u128 T, u32 lim, DevUnit* out) {
  const u32 hi4 = min(iroot6_u128(T), lim), lo4 = iroot6_u128((T - 1) >> 2) + 1;
  if (hi4 < 1 || lo4 > hi4) return true;
  out->cls = 1;
  out->lim = lim;
  out->base_lo = (u64)T;
  out->base_hi = (u64)(T >> 64);
  out->fmax1 = hi4;
  out->fmax2 = lo4;
  out->nres1 = 1;
  return false;
}
// make_dev_unit1: a class-1 Stage-1 unit or plant.
__device__ int pack_find4(const s615_unit& in, DevUnit* out, bool* skip) {
  W3 R;
  u32 lim = in.lim;
  if (in.kind == 0) {
    const u64 B = in.B, u = in.u;
    if (B < 2 || B > kMaxB || u == 0) return S615_E_FORMAT;
    if (u >= B) { *skip = true; return S615_OK; }
    R = d_pow6(B);
    d_sub(R, d_pow6(u));
    lim = (u32)((B - 1) / 42);
  } else if (in.kind == 1) {
    R = W3{{in.base[0], in.base[1], in.base[2]}};
    if (in.lim >= (1u << 21)) return S615_E_FORMAT;
  } else {
    return S615_E_FORMAT;
  }
  if ((R.l[0] | R.l[1] | R.l[2]) == 0) return S615_E_FORMAT;
  u64 rem = 0;   // T = R / 42^6, exactly
#pragma unroll
  for (int i = 2; i >= 0; --i) {
    const u128 d = ((u128)rem << 64) | R.l[i];
    R.l[i] = (u64)(d / kM42);
    rem = (u64)(d % kM42);
  }
  if (rem != 0 || R.l[2] != 0 || (R.l[1] >> 62) != 0) return S615_E_FORMAT;
  out->B = in.B; out->u = in.u;
  *skip = find4_window(((u128)R.l[1] << 64) | R.l[0], lim, out);
  return S615_OK;
}
// make_dev_unit8: a (6,1,7) find4 job.
__device__ int pack_617_find4(const s615_unit& in, DevUnit* out) {
  if (in.kind != 0 || in.base[2] != 0 || (in.base[1] >> 62) != 0) return S615_E_FORMAT;
  if (in.lim >= (1u << 21) || in.fmax2 < 1 || in.fmax1 < in.fmax2 || in.fmax1 > in.lim)
    return S615_E_FORMAT;
  out->cls = S615_CLS_617_FIND4;
  out->B = in.B; out->u = in.u; out->w = in.w;
  out->base_lo = in.base[0];
  out->base_hi = in.base[1];
  out->lim = in.lim;
  out->fmax1 = in.fmax1;
  out->fmax2 = in.fmax2;
  out->nres1 = 1;
  out->pad1 = in.res_e;
  out->pad2 = in.res_d;
  return S615_OK;
}

// make_dev_unit for the classes above: S615_OK (with *skip for a dropped unit) or
// S615_E_FORMAT, in its order of checks.
__device__ int pack_one(const Roots& R, const s615_unit& in, DevUnit* out, bool* skip) {
  *skip = false;
  const u32 cls = in.cls;
  if (in.kind == S615_KIND_JOB) {
    if (cls < 1 || cls > 5 || in.base[2] != 0) return S615_E_FORMAT;
    const u128 T = ((u128)in.base[1] << 64) | in.base[0];
    const u64 lim = in.lim ? in.lim : (in.B ? (in.B - 1) / 42 : 0);
    if (lim > (kMaxB - 1) / 42) return S615_E_FORMAT;
    out->B = in.B; out->u = in.u;
    out->lim = (u32)lim;
    if (cls == 1) {
      *skip = T == 0 || (T >> 122) != 0 || find4_window(T, (u32)lim, out);
      return S615_OK;
    }
    u128 W;
    if (cls == 5) {
      const u128 M = (u128)15561 << 64;
      if ((T >> 121) == 0 && T + 1 < ((u128)1 << 121)) {
        W = T + 1;
      } else {
        W = ((u128)(in.base[1] % 15561) << 64 | in.base[0]) + 1;   // T mod M, plus 1
        if (W >= M) W -= M;
      }
      if (W == 0) W = M;
      out->w = 1;
    } else {
      if (T == 0 || (T >> 121) != 0) { *skip = true; return S615_OK; }
      W = T;
    }
    out->cls = kClsJobRow;
    out->f = 0;
    out->mod1 = 1;
    out->fmax1 = 1;
    out->nres1 = 1;
    out->res1[0] = 1;
    const u128 base = W * (u128)kM42;
    out->base_lo = (u64)base;
    out->base_hi = (u64)(base >> 64);
    return S615_OK;
  }
  if (cls == 1) return pack_find4(in, out, skip);
  if (cls == S615_CLS_617_FIND4) return pack_617_find4(in, out);
  W3 base;
  out->cls = cls;
  out->f = cls == 2 ? 14 : cls == 3 ? 21 : cls == 4 ? 7 : 0;
  if (in.kind == 0) {
    const u64 B = in.B, u = in.u;
    if (B < 2 || B > kMaxB || u == 0) return S615_E_FORMAT;
    if (u >= B) { *skip = true; return S615_OK; }
    base = d_pow6(B);
    d_sub(base, d_pow6(u));
    out->B = B; out->u = u;
    out->lim = (u32)((B - 1) / 42);
    const u32 b2 = pow6_mod_u32(B, kRootM2), b3 = pow6_mod_u32(B, kRootM3);
    const u32 t_d = (b2 + kRootM2 - pow6_mod_u32(u, kRootM2)) % kRootM2 * R.inv21_2 % kRootM2;
    if (cls == 5) {
      const u32 te = b3 * R.inv14_3 % kRootM3;
      const u32 e0 = R.off3[te], en = R.off3[te + 1] - e0, d0 = R.off2[t_d], dn = R.off2[t_d + 1] - d0;
      if (en == 0 || dn == 0) { *skip = true; return S615_OK; }
      out->mod1 = kModE;
      out->fmax1 = (u32)((B - 1) / 14);
      out->fmax2 = (u32)((B - 1) / 21);
      out->nres1 = min(en, 12u);
      out->nres2 = min(dn, 12u);
      for (u32 i = 0; i < out->nres1; ++i) out->res1[i] = R.r3[e0 + i];
      for (u32 i = 0; i < out->nres2; ++i) out->res2[i] = R.r2[d0 + i];
      if (u % 3 != 0 || pow6_mod_u32(u, kRootM7) != pow6_mod_u32(B, kRootM7)) return S615_E_FORMAT;
    } else {
      u32 n = 0;
      if (cls == 2) {
        const u32 t = b3 * R.inv14_3 % kRootM3, o = R.off3[t];
        n = min(R.off3[t + 1] - o, 24u);
        for (u32 i = 0; i < n; ++i) out->res1[i] = R.r3[o + i];
        out->mod1 = kRootM3; out->fmax1 = (u32)((B - 1) / 14);
      } else if (cls == 3) {
        const u32 o = R.off2[t_d];
        n = min(R.off2[t_d + 1] - o, 24u);
        for (u32 i = 0; i < n; ++i) out->res1[i] = R.r2[o + i];
        out->mod1 = kRootM2; out->fmax1 = (u32)((B - 1) / 21);
      } else {   // every pair of roots mod 2^6 and 3^6, ascending (at most 4 x 6)
        const u32 t2 = b2 * R.inv7_2 % kRootM2, t3 = b3 * R.inv7_3 % kRootM3;
        for (u32 i = R.off2[t2]; i < R.off2[t2 + 1]; ++i)
          for (u32 j = R.off3[t3]; j < R.off3[t3 + 1] && n < 24; ++j) {
            const u32 a = R.r2[i], b = R.r3[j];
            const u32 x = a + kRootM2 * ((b + 2 * kRootM3 - a) % kRootM3 * R.inv64_3 % kRootM3);
            u32 k = n++;
            for (; k > 0 && out->res1[k - 1] > x; --k) out->res1[k] = out->res1[k - 1];
            out->res1[k] = x;
          }
        out->mod1 = kRootM2 * kRootM3; out->fmax1 = (u32)((B - 1) / 7);
      }
      if (n == 0) { *skip = true; return S615_OK; }
      out->nres1 = n;
      for (u32 i = 0; i < n; ++i)
        if (!row_ok(base, out->f, out->res1[i])) return S615_E_FORMAT;
    }
  } else if (in.kind == 1) {
    base = W3{{in.base[0], in.base[1], in.base[2]}};
    if ((base.l[0] | base.l[1] | base.l[2]) == 0 || (in.base[2] >> 24) != 0) return S615_E_FORMAT;
    out->B = in.B; out->u = in.u;
    out->lim = in.lim;
    out->nres1 = 1;
    if (cls == 5) {
      if ((u64)in.fmax1 * 14 > kMaxB || (u64)in.fmax2 * 21 > kMaxB) return S615_E_FORMAT;
      out->mod1 = kModE;
      out->fmax1 = in.fmax1; out->fmax2 = in.fmax2;
      out->nres2 = 1;
      out->res1[0] = in.res_e % kModE;
      out->res2[0] = in.res_d % kModD;
      if (!grid_ok(base, out->res1[0], out->res2[0], R.inv21_2)) return S615_E_FORMAT;
    } else {
      const u32 mod = cls == 2 ? kRootM3 : cls == 3 ? kRootM2 : kRootM2 * kRootM3;
      if ((u64)in.fmax1 * out->f > kMaxB) return S615_E_FORMAT;
      out->mod1 = mod;
      out->fmax1 = in.fmax1;
      out->res1[0] = in.res_d % mod;
      if (!row_ok(base, out->f, out->res1[0])) return S615_E_FORMAT;
    }
  } else {
    return S615_E_FORMAT;
  }
  out->base_lo = base.l[0];
  out->base_hi = base.l[1];
  return S615_OK;
}

// Row chunks of a class 2-5 unit at `rows` rows each.
__device__ __forceinline__ u32 row_items(const DevUnit& d, u32 rows) {
  u32 n = 0;
  for (u32 i = 0; i < d.nres1; ++i) {
    u32 jmin, jend;
    class_rows(d.res1[i], d.mod1, d.fmax1, &jmin, &jend);
    if (jend > jmin) n += (jend - jmin + rows - 1) / rows;
  }
  return n;
}
// Items of the second kernel: chunks of a find4 unit's c4 window.
__device__ __forceinline__ u32 find4_items(const DevUnit& d) {
  return d.cls == 1 || d.cls == S615_CLS_617_FIND4 ? (d.fmax1 - d.fmax2) / kC4Chunk + 1 : 0u;
}
// Does unit k begin a job item?  Consecutive job rows of one kind share items,
// never across a multiple of job_rows.
__device__ __forceinline__ bool job_start(const s615_unit* raw, u32 k, u32 job_rows) {
  bool kind, before;
  if (!job_row(raw[k], &kind)) return false;
  return k % job_rows == 0 || !job_row(raw[k - 1], &before) || before != kind;
}

__global__ void k_pack(Roots R, const s615_unit* __restrict__ raw, u32 n, u32 job_rows,
                       DevUnit* __restrict__ units, FillTotals* tot) {
  const u32 k = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  u32 c5[3] = {0, 0, 0}, c3[3] = {0, 0, 0}, jobs = 0, find4 = 0;
  double keys = 0;
  bool bad = false;
  if (k < n) {
    DevUnit d;
    memset(&d, 0, sizeof d);
    bool skip;
    bad = pack_one(R, raw[k], &d, &skip) != S615_OK;
    d.id = k;
    if (skip) d.cls = 0;
    units[k] = d;
    if (!bad && !skip) {
      find4 = find4_items(d);
      if (d.cls == kClsJobRow) {
        jobs = job_start(raw, k, job_rows);
      } else if (!find4) {
#pragma unroll
        for (int i = 0; i < 3; ++i) (d.cls == 5 ? c5 : c3)[i] = row_items(d, kItemRows >> i);
      }
      if (!find4) keys = unit_keys(d);
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      c5[i] += __shfl_xor_sync(0xFFFFFFFFu, c5[i], o);
      c3[i] += __shfl_xor_sync(0xFFFFFFFFu, c3[i], o);
    }
    jobs += __shfl_xor_sync(0xFFFFFFFFu, jobs, o);
    find4 += __shfl_xor_sync(0xFFFFFFFFu, find4, o);
    keys += __shfl_xor_sync(0xFFFFFFFFu, keys, o);
  }
  bad = __any_sync(0xFFFFFFFFu, bad);
  if (lane == 0) {
    for (int i = 0; i < 3; ++i) {
      if (c5[i]) atomicAdd(&tot->items5[i], (unsigned long long)c5[i]);
      if (c3[i]) atomicAdd(&tot->items234[i], (unsigned long long)c3[i]);
    }
    if (jobs) atomicAdd(&tot->jobs, (unsigned long long)jobs);
    if (find4) atomicAdd(&tot->find4, (unsigned long long)find4);
    if (keys > 0) atomicAdd(&tot->keys, keys);
    if (bad) tot->bad = 1;
  }
}

// The place of this thread's c items in a run of the block's, reserved at `cursor`.
// Every thread of the block calls this.
__device__ __forceinline__ u64 block_place(u32 c, unsigned long long* cursor) {
  __shared__ u32 s_w[8];
  __shared__ unsigned long long s_base;
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32 incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= (u32)o) incl += y;
  }
  __syncthreads();
  if (lane == 31) s_w[wid] = incl;
  __syncthreads();
  u32 before = 0, all = 0;
  for (u32 w = 0; w < 8; ++w) {
    if (w < wid) before += s_w[w];
    all += s_w[w];
  }
  if (threadIdx.x == 0) s_base = all ? atomicAdd(cursor, (unsigned long long)all) : 0ull;
  __syncthreads();
  return s_base + before + incl - c;
}

// The items of 256 units, one after another; the blocks' runs come in the order
// in which the blocks reserve them.  Find4 units' items go to `second` (to be
// ordered by order_items), the others' to `items`.
__global__ void k_items(const s615_unit* __restrict__ raw, const DevUnit* __restrict__ units, u32 n,
                        u32 job_rows, u32 rows, u32 parts3, u64* __restrict__ items, u64 cap,
                        u64* __restrict__ second, u64 cap2, FillTotals* tot) {
  const u32 k = blockIdx.x * blockDim.x + threadIdx.x;
  u32 c = 0, c2 = 0, cls = 0;
  if (k < n) {
    cls = units[k].cls;
    c2 = cls ? find4_items(units[k]) : 0u;
    if (cls == kClsJobRow) c = job_start(raw, k, job_rows);
    else if (cls && !c2) c = row_items(units[k], rows) * (cls == 5 ? 1u : parts3);
  }
  if (second) {   // the same for every thread
    const u64 at2 = block_place(c2, &tot->placed4);
    if (at2 + c2 <= cap2)
      for (u32 i = 0; i < c2; ++i) second[at2 + i] = make_item(k, 0, i);
  }
  u64 at = block_place(c, &tot->placed);
  if (c == 0 || at + c > cap) return;   // cap is the total: never past it
  if (cls == kClsJobRow) {
    bool kind, other;
    job_row(raw[k], &kind);
    u32 run = 1;
    while (k + run < n && (k + run) % job_rows != 0 && job_row(raw[k + run], &other) && other == kind) ++run;
    items[at] = make_item(k, kJobItemTag, (kind ? kJobFind2 : 0u) | run);
    return;
  }
  const DevUnit& d = units[k];
  const u32 parts = cls == 5 ? 1u : parts3;
  for (u32 i = 0; i < d.nres1; ++i) {
    u32 jmin, jend;
    class_rows(d.res1[i], d.mod1, d.fmax1, &jmin, &jend);
    for (u32 ch = 0; jmin + ch * rows < jend; ++ch)
      for (u32 p = 0; p < parts; ++p) items[at++] = make_item(k, i, ch * parts + p);
  }
}

}  // namespace

int launch_pack(s615_ctx* ctx, const s615_unit* d_raw, u32 n, u32 job_rows, DevUnit* units,
                FillTotals* tot, cudaStream_t st) {
  Roots R;
  if (const int s = roots_on_device(ctx, &R)) return s;
  S615_CU(cudaMemsetAsync(tot, 0, sizeof *tot, st));
  k_pack<<<(n + 127) / 128, 128, 0, st>>>(R, d_raw, n, job_rows, units, tot);
  ctx->launches++;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

int launch_items(s615_ctx* ctx, const s615_unit* d_raw, const DevUnit* units, u32 n, u32 job_rows,
                 u32 rows, u32 parts3, u64* items, u64 n_items, u64* second, u64 n_second,
                 FillTotals* tot, cudaStream_t st) {
  k_items<<<(n + 255) / 256, 256, 0, st>>>(d_raw, units, n, job_rows, rows, parts3, items, n_items,
                                           second, n_second, tot);
  ctx->launches++;
  S615_CU(cudaGetLastError());
  return S615_OK;
}

}  // namespace s615
