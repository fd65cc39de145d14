// row_read.cuh -- the search distance of rows read straight from global memory
// (the search kernel's gather, the entry choice's scans).
#pragma once

#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <cstdint>

#include "device_common.cuh"

namespace song {

template <int METRIC>
__device__ __forceinline__ float finish_distance(float t, float len) {
  if (METRIC == 0) return t;
  if (METRIC == 1) return -t;
  // warp_astar_accelerator.h:275-281: sign * tmp * tmp / len in float.
  if (len != 0.0f) {
    float sign = t < 0.0f ? 1.0f : -1.0f;
    return __fdiv_rn(__fmul_rn(__fmul_rn(sign, t), t), len);
  }
  return 0.0f;
}

// ---------------------------------------------------------------------------
// Distances of rows read straight from global memory.
//
// The distance of a row is fixed by the reference's arithmetic: partial p
// (p = 0..31) is the fused multiply-add chain over dimensions p, p+32, ... in
// that order, and the 32 partials meet in the xor butterfly 16, 8, 4, 2, 1.
// Which lane computes a partial is free.  Here four lanes share a row, eight
// partials each, so one pass of the warp takes eight rows: every 32
// dimensions are two 16-byte loads per lane (FP32; 64 contiguous bytes of
// each row per load), already in the register pairs of the paired FP32
// instructions, and the first butterfly levels are adds within a lane.
// Against rows staged by bulk copies and read back one float per lane: no
// barrier, no shared-memory round trip, and 85 instead of 180 warp
// instructions per eight 128-float rows.
// ---------------------------------------------------------------------------

template <int STORAGE>
struct RowRead;

// FP32: lane g of a row's four holds partials 4g..4g+3 and 16+4g..16+4g+3.
template <>
struct RowRead<0> {
  static constexpr bool HALVES = true;
  ulonglong2 a, b;
  __device__ __forceinline__ void load(const uint8_t *row, int j, int g, int width) {
    const ulonglong2 *x = reinterpret_cast<const ulonglong2 *>(row) + (j >> 2) + g;
    a = j + 4 * g < width ? __ldg(x) : make_ulonglong2(0ull, 0ull);
    b = j + 16 + 4 * g < width ? __ldg(x + 4) : make_ulonglong2(0ull, 0ull);
  }
  __device__ __forceinline__ void load_full(const uint8_t *row, int j, int g) {
    const ulonglong2 *x = reinterpret_cast<const ulonglong2 *>(row) + (j >> 2) + g;
    a = __ldg(x);
    b = __ldg(x + 4);
  }
  __device__ __forceinline__ void get(uint64_t (&x)[4], float) const {
    x[0] = a.x;
    x[1] = a.y;
    x[2] = b.x;
    x[3] = b.y;
  }
};

// BF16 and FP8: lane g holds the eight partials 8g..8g+7 (16 or 8
// contiguous bytes), decoded to FP32; an FP8 value is multiplied by the row's
// scale and rounded, so a low-precision search equals an FP32 search over the
// dequantised vectors.
template <>
struct RowRead<1> {
  static constexpr bool HALVES = false;
  uint4 a;
  __device__ __forceinline__ void load(const uint8_t *row, int j, int g, int width) {
    a = j + 8 * g < width ? __ldg(reinterpret_cast<const uint4 *>(row) + (j >> 3) + g) : make_uint4(0u, 0u, 0u, 0u);
  }
  __device__ __forceinline__ void load_full(const uint8_t *row, int j, int g) {
    a = __ldg(reinterpret_cast<const uint4 *>(row) + (j >> 3) + g);
  }
  static __device__ __forceinline__ uint64_t pair(uint32_t w) {
    return f2_pack(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  __device__ __forceinline__ void get(uint64_t (&x)[4], float) const {
    x[0] = pair(a.x);
    x[1] = pair(a.y);
    x[2] = pair(a.z);
    x[3] = pair(a.w);
  }
};

template <>
struct RowRead<2> {
  static constexpr bool HALVES = false;
  uint2 a;
  __device__ __forceinline__ void load(const uint8_t *row, int j, int g, int width) {
    a = j + 8 * g < width ? __ldg(reinterpret_cast<const uint2 *>(row) + (j >> 3) + g) : make_uint2(0u, 0u);
  }
  __device__ __forceinline__ void load_full(const uint8_t *row, int j, int g) {
    a = __ldg(reinterpret_cast<const uint2 *>(row) + (j >> 3) + g);
  }
  static __device__ __forceinline__ uint64_t pair(uint32_t w, float scale) {  // the low 16 bits
    const __half2_raw h =
        __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w & 0xffffu), __NV_E4M3);
    const float2 f = __half22float2(__half2(h));
    return f2_pack(__fmul_rn(f.x, scale), __fmul_rn(f.y, scale));
  }
  __device__ __forceinline__ void get(uint64_t (&x)[4], float scale) const {
    x[0] = pair(a.x, scale);
    x[1] = pair(a.x >> 16, scale);
    x[2] = pair(a.y, scale);
    x[3] = pair(a.y >> 16, scale);
  }
};

// The xor butterfly over a row's 32 partials, four lanes with eight each
// (acc[i]: the pair at 2i, 2i+1 of the lane's eight); the sum in all four
// lanes.  At the first levels a lane keeps half of its values and its
// partner the other half; every sum is the butterfly's own pair (a + b ==
// b + a).
template <bool HALVES>
__device__ __forceinline__ float row_butterfly(const uint64_t (&acc)[4], int lane) {
  const bool h1 = (lane & 2) != 0, h0 = (lane & 1) != 0;
  if (HALVES) {
    // level 16 within the lane; the values left are partials 4g + e
    float e0, e1, e2, e3;
    f2_unpack(f2_add(acc[0], acc[2]), e0, e1);
    f2_unpack(f2_add(acc[1], acc[3]), e2, e3);
    // level 8: lane ^ 2; keep e = 2 h1 + {0, 1}
    float k0 = __fadd_rn(h1 ? e2 : e0, __shfl_xor_sync(FULL, h1 ? e0 : e2, 2));
    float k1 = __fadd_rn(h1 ? e3 : e1, __shfl_xor_sync(FULL, h1 ? e1 : e3, 2));
    // level 4: lane ^ 1; keep e = 2 h1 + h0
    float t = __fadd_rn(h0 ? k1 : k0, __shfl_xor_sync(FULL, h0 ? k0 : k1, 1));
    t = __fadd_rn(t, __shfl_xor_sync(FULL, t, 2));  // level 2
    return __fadd_rn(t, __shfl_xor_sync(FULL, t, 1));  // level 1
  }
  float v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) f2_unpack(acc[i], v[2 * i], v[2 * i + 1]);
  float a[4], c[2];
#pragma unroll
  for (int i = 0; i < 4; ++i)  // level 16: lane ^ 2; keep e = 4 h1 + i
    a[i] = __fadd_rn(h1 ? v[4 + i] : v[i], __shfl_xor_sync(FULL, h1 ? v[i] : v[4 + i], 2));
#pragma unroll
  for (int i = 0; i < 2; ++i)  // level 8: lane ^ 1; keep e = 4 h1 + 2 h0 + i
    c[i] = __fadd_rn(h0 ? a[2 + i] : a[i], __shfl_xor_sync(FULL, h0 ? a[i] : a[2 + i], 1));
  // level 4 (bit 2 of e, held by h1): lane ^ 2; keep i = h1
  float t = __fadd_rn(h1 ? c[1] : c[0], __shfl_xor_sync(FULL, h1 ? c[0] : c[1], 2));
  t = __fadd_rn(t, __shfl_xor_sync(FULL, t, 1));     // level 2 (bit 1, held by h0)
  return __fadd_rn(t, __shfl_xor_sync(FULL, t, 2));  // level 1 (bit 0, held by h1)
}

}  // namespace song
