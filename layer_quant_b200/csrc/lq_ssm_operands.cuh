// Operand access shared by the selective-state update kernels (MX-held and dense state): the
// reference's softplus and the 16-column slices of B / C.
#pragma once

#include "lq_common.cuh"

namespace lq {

// softplus as the reference's kernels compute it (mamba_state_8b_kernel.py:28-30)
__device__ __forceinline__ float softplus_ref(float x) { return x <= 20.0f ? logf(1.0f + expf(x)) : x; }

// 16 consecutive B or C values of (batch b, group grp) starting at column n0, as floats.  Contiguous
// 16-bit operands take two 128-bit loads; anything else goes value by value.
__device__ __forceinline__ void load_bc16(const void* base, const int64_t (&st)[3], int dtype, int b, int grp, int n0, float (&v)[16]) {
  const int64_t off = b * st[0] + grp * st[1] + n0 * st[2];
  if (dtype != LQ_F32 && st[2] == 1 && ((reinterpret_cast<uintptr_t>(base) + 2 * off) & 15) == 0) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + off);
    const uint4 lo = src[0], hi = src[1];  // not the read-only path: a dependent launch may start before these are written
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (dtype == LQ_BF16) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = load_as_float(base, off + i * st[2], dtype);
  }
}

// V (4 or 8) consecutive B or C values starting at column n0
template <int V>
__device__ __forceinline__ void load_bc(const void* base, const int64_t (&st)[3], int dtype, int b, int grp, int n0, float (&v)[V]) {
  const int64_t off = b * st[0] + grp * st[1] + n0 * st[2];
  if (dtype != LQ_F32 && st[2] == 1 && ((reinterpret_cast<uintptr_t>(base) + 2 * off) & (2 * V - 1)) == 0) {
    uint32_t w[V / 2];
    const uint16_t* src = static_cast<const uint16_t*>(base) + off;
    if (V == 8) {
      const uint4 q = *reinterpret_cast<const uint4*>(src);
      w[0] = q.x; w[1] = q.y; w[V / 2 - 2] = q.z; w[V / 2 - 1] = q.w;
    } else {
      const uint2 q = *reinterpret_cast<const uint2*>(src);
      w[0] = q.x; w[1] = q.y;
    }
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      const float2 f = dtype == LQ_BF16 ? make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u))
                                        : __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = load_as_float(base, off + i * st[2], dtype);
  }
}

}  // namespace lq
