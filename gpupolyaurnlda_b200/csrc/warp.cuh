// warp.cuh -- warp- and block-level integer scans and reductions, and the exact
// arithmetic of a draw.
#pragma once

#include "common.cuh"

namespace gpulda {

__device__ __forceinline__ u64 warp_incl_scan_u64(u64 x, u32 lane) {
#pragma unroll
  for (u32 o = 1; o < 32; o <<= 1) {
    const u64 y = __shfl_up_sync(kFullMask, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

__device__ __forceinline__ u64 warp_sum_u64(u64 x) {
#pragma unroll
  for (u32 o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFullMask, x, o);
  return x;
}

__device__ __forceinline__ double warp_sum_f64(double x) {
#pragma unroll
  for (u32 o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFullMask, x, o);
  return x;
}

// Inclusive scan over groups of W lanes of the warp: the shuffle's own predicate
// guards the two-word add.
template <u32 W>
__device__ __forceinline__ u64 group_scan(u64 x) {
#pragma unroll
  for (u32 o = 1; o < W; o <<= 1)
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .u32 a0, a1, b0, b1;\n\t"
        "mov.b64 {a0, a1}, %0;\n\t"
        "shfl.sync.up.b32 b0|p, a0, %1, %2, 0xffffffff;\n\t"
        "shfl.sync.up.b32 b1, a1, %1, %2, 0xffffffff;\n\t"
        "@p add.cc.u32 a0, a0, b0;\n\t"
        "@p addc.u32 a1, a1, b1;\n\t"
        "mov.b64 %0, {a0, a1};\n\t"
        "}"
        : "+l"(x)
        : "r"(o), "r"((32 - W) << 8));
  return x;
}

// Integers below 2^52 as doubles, exactly: the integer is the low mantissa of
// 2^52, which is subtracted again.
__device__ __forceinline__ double exact_double(u64 x) {
  return __dadd_rn(__hiloint2double((int)(0x43300000u | (u32)(x >> 32)), (int)(u32)x), -4503599627370496.0);
}

// r / 2^32, exactly, the same way from 2^20.
__device__ __forceinline__ double exact_unit(u32 r) {
  return __dadd_rn(__hiloint2double(0x41300000, (int)r), -1048576.0);
}

// The mixture test: u * (alpha A + B) < B in double, alpha A rounded once.  B is
// below 2^48 (65535 tokens of mass below 2^32).
__device__ __forceinline__ bool sparse_test(u32 r, double aA, u64 B) {
  const double b = exact_double(B);
  return __dmul_rn(exact_unit(r), __dadd_rn(aA, b)) < b;
}

// Block-wide exclusive scan of one u64 per thread; `sh` holds 33 entries.
__device__ __forceinline__ u64 block_excl_scan_u64(u64 v, u64* sh, u64* total) {
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const u64 incl = warp_incl_scan_u64(v, lane);
  if (lane == 31) sh[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    u64 x = lane < nw ? sh[lane] : 0;
    x = warp_incl_scan_u64(x, lane);
    sh[lane] = x;
  }
  __syncthreads();
  const u64 off = warp ? sh[warp - 1] : 0;
  *total = sh[nw - 1];
  __syncthreads();
  return off + incl - v;
}

__device__ __forceinline__ u64 block_sum_u64(u64 v, u64* sh) {
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum_u64(v);
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  u64 t = 0;
  for (u32 i = 0; i < nw; ++i) t += sh[i];
  __syncthreads();
  return t;
}

}  // namespace gpulda
