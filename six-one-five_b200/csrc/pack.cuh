// pack.cuh -- what device-side unit packing (pack.cu) and device Stage-1
// (stage1.cu) share: the root tables and a few modular helpers.
#pragma once
#include <cuda_runtime.h>

#include "engine.hpp"

namespace s615 {

constexpr u32 kRootM2 = 64, kRootM3 = 729, kRootM7 = 117649;

struct Roots {                 // CSR root lists, offsets then roots, per modulus
  const u32 *off2, *r2, *off3, *r3, *off7, *r7;
  u32 inv14_3, inv21_2;        // (14^6)^-1 mod 3^6, (21^6)^-1 mod 2^6
  u32 inv7_2, inv7_3, inv64_3; // (7^6)^-1 mod 2^6 and 3^6, 64^-1 mod 3^6
};
int roots_on_device(s615_ctx* ctx, Roots* R);

__device__ __forceinline__ u32 pow6_mod_u32(u64 x, u32 m) {
  x %= m;
  const u64 x2 = x * x % m, x3 = x2 * x % m;
  return (u32)(x3 * x3 % m);
}

}  // namespace s615
