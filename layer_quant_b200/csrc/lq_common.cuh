// Shared host/device helpers of the layer_quant_b200 kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/layer_quant_b200.h"

#define LQ_EXPORT extern "C" __attribute__((visibility("default")))

namespace lq {

// ---- host-side error reporting ---------------------------------------------------------------
char* last_error_buffer();  // thread-local, 512 bytes (defined in lq_api.cu)

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buffer(), 512, fmt, ap);
  va_end(ap);
  return code;
}

#define LQ_CHECK_ARG(cond, ...)                                  \
  do {                                                           \
    if (!(cond)) return ::lq::fail(LQ_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
  } while (0)

#define LQ_CHECK_CUDA(expr)                                                                    \
  do {                                                                                         \
    cudaError_t e__ = (expr);                                                                  \
    if (e__ != cudaSuccess)                                                                    \
      return ::lq::fail(LQ_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__));         \
  } while (0)

inline bool valid_dtype(int dt) { return dt == LQ_BF16 || dt == LQ_F16 || dt == LQ_F32; }
inline int dtype_bytes(int dt) { return dt == LQ_F32 ? 4 : 2; }

int sm_count();  // multiprocessors of the current device (cached per device; lq_api.cu)

// floor(n / d) for n < 2^31 without a division: (mulhi(n, magic) + n) >> shift
struct FastDiv {
  uint32_t magic, shift;
};
inline FastDiv fast_div_of(uint32_t d) {
  FastDiv f;
  f.shift = 0;
  while ((1ull << f.shift) < d) ++f.shift;  // ceil(log2 d)
  f.magic = static_cast<uint32_t>(((1ull << (32 + f.shift)) + d - 1) / d - (1ull << 32));
  return f;
}
__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv& f) { return (__umulhi(n, f.magic) + n) >> f.shift; }

// Programmatic dependent launch: the kernel may be scheduled while its predecessor in the stream is still running (its CTAs take
// the slots the predecessor's CTAs leave); before its griddepcontrol.wait, which returns once the predecessor has completed and its writes
// are visible, it reads and writes no global memory but the module's own constants, and only asks for lines in L2 (a prefetch reads nothing).
// Behind the wait operands are read with ordinary loads (the non-coherent ones are for data that nobody writes while the kernel lives).  Whether a kernel lets its own dependents
// start early (pdl_launch_dependents) is a separate choice: the decode and prefill kernels do not.  LQ_MX_PDL=0 switches it off.
bool use_pdl();  // lq_api.cu
template <class... Params, class... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, unsigned block, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_pdl() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- device helpers --------------------------------------------------------------------------
__device__ __forceinline__ float load_as_float(const void* p, int64_t i, int dt) {
  if (dt == LQ_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
  if (dt == LQ_F16) return __half2float(static_cast<const __half*>(p)[i]);
  return static_cast<const float*>(p)[i];
}

__device__ __forceinline__ void store_from_float(void* p, int64_t i, int dt, float v) {
  if (dt == LQ_BF16)
    static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else if (dt == LQ_F16)
    static_cast<__half*>(p)[i] = __float2half_rn(v);
  else
    static_cast<float*>(p)[i] = v;
}

__device__ __forceinline__ float bf16_bits_to_float(uint32_t bits16) { return __uint_as_float(bits16 << 16); }

// Philox4x32-10 (Salmon et al. 2011), the generator behind Triton's tl.rand.
struct Philox4 {
  uint32_t w0, w1, w2, w3;
};

__device__ __forceinline__ Philox4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0,
                                                 uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t pb = static_cast<uint64_t>(0xCD9E8D57u) * c2;
    const uint64_t pa = static_cast<uint64_t>(0xD2511F53u) * c0;
    const uint32_t n0 = static_cast<uint32_t>(pb >> 32) ^ c1 ^ k0;
    const uint32_t n2 = static_cast<uint32_t>(pa >> 32) ^ c3 ^ k1;
    c1 = static_cast<uint32_t>(pb);
    c3 = static_cast<uint32_t>(pa);
    c0 = n0;
    c2 = n2;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return Philox4{c0, c1, c2, c3};
}

// Same generator with the ten round keys precomputed (k0 + r * 0x9E3779B9, k1 + r * 0xBB67AE85 at
// rk[2r], rk[2r + 1]); when rk lives in kernel parameters the keys cost no instruction.
struct PhiloxKeys {
  uint32_t rk[20];
};

inline PhiloxKeys make_philox_keys(uint64_t seed) {
  PhiloxKeys k;
  uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    k.rk[2 * r] = k0;
    k.rk[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return k;
}

__device__ __forceinline__ Philox4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const PhiloxKeys& keys) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t pb = static_cast<uint64_t>(0xCD9E8D57u) * c2;
    const uint64_t pa = static_cast<uint64_t>(0xD2511F53u) * c0;
    const uint32_t n0 = static_cast<uint32_t>(pb >> 32) ^ c1 ^ keys.rk[2 * r];
    const uint32_t n2 = static_cast<uint32_t>(pa >> 32) ^ c3 ^ keys.rk[2 * r + 1];
    c1 = static_cast<uint32_t>(pb);
    c3 = static_cast<uint32_t>(pa);
    c0 = n0;
    c2 = n2;
  }
  return Philox4{c0, c1, c2, c3};
}

// The same generator for counters (c0, c1, step, layer) whose c0 alone changes along a thread's work: what the first rounds
// make of the other three is formed once, and the first product is carried as a sum (pa + n * d for c0 + n), so that a
// block costs 17 wide multiplies (3 cycles of the heavy FMA pipe per scheduler and lane quad each) instead of 20.
constexpr uint32_t kPhiloxM0 = 0xD2511F53u, kPhiloxM1 = 0xCD9E8D57u;
struct PhiloxStream {
  uint64_t pa;                 // kPhiloxM0 * c0; c0 must not pass 2^32
  uint32_t k1, x2, y2, z3;
  __device__ __forceinline__ void init(uint32_t c0, uint32_t c1, uint32_t step, uint32_t layer, const PhiloxKeys& keys) {
    const uint64_t pb1 = static_cast<uint64_t>(kPhiloxM1) * step;
    const uint64_t pa2 = static_cast<uint64_t>(kPhiloxM0) * (static_cast<uint32_t>(pb1 >> 32) ^ c1 ^ keys.rk[0]);
    pa = static_cast<uint64_t>(kPhiloxM0) * c0;
    k1 = layer ^ keys.rk[1];
    x2 = static_cast<uint32_t>(pb1) ^ keys.rk[2];
    y2 = static_cast<uint32_t>(pa2 >> 32) ^ keys.rk[3];
    z3 = static_cast<uint32_t>(pa2) ^ keys.rk[5];
  }
  __device__ __forceinline__ Philox4 block(uint32_t ahead, const PhiloxKeys& keys) const {  // of counter c0 + ahead
    const uint64_t p1 = pa + static_cast<uint64_t>(kPhiloxM0) * ahead;
    const uint64_t p2 = static_cast<uint64_t>(kPhiloxM1) * (static_cast<uint32_t>(p1 >> 32) ^ k1);
    const uint64_t pb3 = static_cast<uint64_t>(kPhiloxM1) * (static_cast<uint32_t>(p1) ^ y2);
    const uint64_t pa3 = static_cast<uint64_t>(kPhiloxM0) * (static_cast<uint32_t>(p2 >> 32) ^ x2);
    uint32_t c0 = static_cast<uint32_t>(pb3 >> 32) ^ static_cast<uint32_t>(p2) ^ keys.rk[4], c1 = static_cast<uint32_t>(pb3);
    uint32_t c2 = static_cast<uint32_t>(pa3 >> 32) ^ z3, c3 = static_cast<uint32_t>(pa3);
#pragma unroll
    for (int r = 3; r < 10; ++r) {
      const uint64_t pb = static_cast<uint64_t>(kPhiloxM1) * c2;
      const uint64_t pq = static_cast<uint64_t>(kPhiloxM0) * c0;
      c0 = static_cast<uint32_t>(pb >> 32) ^ c1 ^ keys.rk[2 * r];
      c2 = static_cast<uint32_t>(pq >> 32) ^ c3 ^ keys.rk[2 * r + 1];
      c1 = static_cast<uint32_t>(pb);
      c3 = static_cast<uint32_t>(pq);
    }
    return Philox4{c0, c1, c2, c3};
  }
};

// Word 0 of the blocks of counters (c0 + i, c1, 0, 0) for small i: what the first rounds make of c1 is formed once, the first product is carried as a
// sum, and the last rounds form only what word 0 needs: 13 wide, 2 high and 1 low multiply per word in place of 17 wide ones.
struct PhiloxWords0 {
  uint64_t pa;  // kPhiloxM0 * c0; c0 + i must not pass 2^32
  uint32_t hi, lo;
  __device__ __forceinline__ void init(uint32_t c0, uint32_t c1, const PhiloxKeys& keys) {
    pa = static_cast<uint64_t>(kPhiloxM0) * c0;
    const uint64_t q = static_cast<uint64_t>(kPhiloxM0) * (c1 ^ keys.rk[0]);
    hi = static_cast<uint32_t>(q >> 32) ^ keys.rk[3];
    lo = static_cast<uint32_t>(q);
  }
  // words first .. first + N - 1: N chains side by side
  template <int N>
  __device__ __forceinline__ void draw(uint32_t first, const PhiloxKeys& keys, uint32_t* w) const {
    uint32_t c0[N], c1[N], c2[N], c3[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t p = pa + static_cast<uint64_t>(kPhiloxM0) * (first + i);
      const uint64_t pb = static_cast<uint64_t>(kPhiloxM1) * (static_cast<uint32_t>(p >> 32) ^ keys.rk[1]);
      c0[i] = static_cast<uint32_t>(pb >> 32) ^ keys.rk[2];
      c1[i] = static_cast<uint32_t>(pb);
      c2[i] = hi ^ static_cast<uint32_t>(p);
      c3[i] = lo;
    }
#pragma unroll
    for (int r = 2; r < 8; ++r)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const uint64_t pb = static_cast<uint64_t>(kPhiloxM1) * c2[i], pq = static_cast<uint64_t>(kPhiloxM0) * c0[i];
        c0[i] = static_cast<uint32_t>(pb >> 32) ^ c1[i] ^ keys.rk[2 * r];
        c2[i] = static_cast<uint32_t>(pq >> 32) ^ c3[i] ^ keys.rk[2 * r + 1];
        c1[i] = static_cast<uint32_t>(pb);
        c3[i] = static_cast<uint32_t>(pq);
      }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      c1[i] = kPhiloxM1 * c2[i];
      c2[i] = __umulhi(kPhiloxM0, c0[i]) ^ c3[i] ^ keys.rk[17];
      w[i] = __umulhi(kPhiloxM1, c2[i]) ^ c1[i] ^ keys.rk[18];
    }
  }
};

// Word -> uniform float in [0, 1) exactly as tl.rand does it: reinterpret as int32, fold the
// negative half with x -> -x - 1, convert (round to nearest) and scale by fp32(4.6566127342e-10).
__device__ __forceinline__ float word_to_uniform(uint32_t w) {
  int x = static_cast<int>(w);
  x = x < 0 ? ~x : x;
  return __int2float_rn(x) * 4.6566127342e-10f;
}

}  // namespace lq
