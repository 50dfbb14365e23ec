// Mamba2 selective-state update on an MX8 / MX4-held recurrent state, fused in one pass, plus the
// stand-alone MX codec kernels.  sm_100a.
//
// In every update kernel one lane owns one 16-value block of a row, so block maximum, pair maxima, exponent
// and micro-exponent bits never leave the thread, and dstate/16 neighbouring lanes own one row.
// mx_state_update_fast_kernel (dense states, every Mamba2 decode step) deals the rows in contiguous slabs to one
// wave of two-warp CTAs; mx_state_update_kernel takes any strides, per-row dt and ragged shapes, one CTA per
// (batch, head).
//
// Both are bound by the dispatch of instructions, not by HBM or by latency: at 18 bytes per block read and written the memory
// system could deliver one value every ~12 issue slots per SM sub-partition, and decode + update + read-out +
// exponent + rounding + random bits need more than that.  What an instruction costs there was measured in random mixes of independent chains
// (the same for two, four and six warps per scheduler): 2 cycles of the logic pipe for byte permutes, logic, shifts and compares, one slot for a
// scalar FMA, two for a packed one (beside byte permutes it takes 3.1 cycles, as two scalar ones do; a packed product with two register operands
// 2.1), and 2.4 cycles of the logic pipe for a wide multiply.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "lq_mx_codec.cuh"
#include "lq_ssm_operands.cuh"

namespace lq {

constexpr int kUpdateThreads = 128;
// the slab kernel runs two warps per CTA, eight CTAs per SM: the same sixteen warps per SM as four CTAs of four warps
// (the register file allows no more), cut into slabs half as large
constexpr int kFastThreads = 64;
constexpr int kFastCtasPerSm = 8;

// ---- block load / store in either storage layout -----------------------------------------------
struct MxRaw {
  uint4 q;        // 16 mantissa bytes (8 for packed MX4: x, y)
  uint32_t e;     // shared exponent byte
  uint32_t mic;   // micro-exponent bits, bit i = pair i
};

template <int BITS, int LAYOUT>
struct MxBlockIO {
  static constexpr bool kNibbles = (BITS == 4 && LAYOUT == LQ_MX_LAYOUT_PACKED);
  static constexpr int kQBytes = kNibbles ? 8 : 16;

  static constexpr int kMicroBytes = (LAYOUT == LQ_MX_LAYOUT_PACKED) ? 1 : 8;

  // One block through plain pointers (dense states: the caller does the address arithmetic once).  The state
  // is streamed: loads go to L2 only, which also keeps them coherent with a predecessor's stores when the
  // kernel was scheduled before that predecessor finished.
  __device__ __forceinline__ static MxRaw load_ptr(const uint8_t* q, const uint8_t* e, const uint8_t* m) {
    MxRaw r;
    if (kNibbles) {
      const uint2 v = __ldcg(reinterpret_cast<const uint2*>(q));
      r.q = make_uint4(v.x, v.y, 0u, 0u);
    } else {
      r.q = __ldcg(reinterpret_cast<const uint4*>(q));
    }
    r.e = __ldcg(e);
    if (LAYOUT == LQ_MX_LAYOUT_PACKED) {
      r.mic = __ldcg(m);
    } else {
      const uint2 mm = __ldcg(reinterpret_cast<const uint2*>(m));
      r.mic = (((mm.x & 0x01010101u) * 0x10204080u) >> 28) | ((((mm.y & 0x01010101u) * 0x10204080u) >> 28) << 4);
    }
    return r;
  }

  // codes: the words as stored (packed nibbles: codes[0..1])
  __device__ __forceinline__ static void store_ptr(uint8_t* q, uint8_t* e, uint8_t* m, const uint32_t (&codes)[4], uint32_t ev,
                                                   uint32_t mic) {
    if (kNibbles) {
      *reinterpret_cast<uint2*>(q) = make_uint2(codes[0], codes[1]);
    } else {
      *reinterpret_cast<uint4*>(q) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
    }
    *e = static_cast<uint8_t>(ev);
    if (LAYOUT == LQ_MX_LAYOUT_PACKED) {
      *m = static_cast<uint8_t>(mic);
    } else {
      const uint32_t lo = ((mic & 0xFu) * 0x00204081u) & 0x01010101u;
      const uint32_t hi = (((mic >> 4) & 0xFu) * 0x00204081u) & 0x01010101u;
      *reinterpret_cast<uint2*>(m) = make_uint2(lo, hi);
    }
  }

  __device__ __forceinline__ static MxRaw load(const lq_mx_state& s, int64_t qrow, int64_t erow, int64_t mrow, int blk) {
    MxRaw r;
    const uint8_t* q = static_cast<const uint8_t*>(s.q_state) + qrow + blk * kQBytes;
    if (kNibbles) {
      const uint2 v = *reinterpret_cast<const uint2*>(q);
      r.q = make_uint4(v.x, v.y, 0u, 0u);
    } else {
      r.q = *reinterpret_cast<const uint4*>(q);
    }
    r.e = s.shared_exp[erow + blk];
    if (LAYOUT == LQ_MX_LAYOUT_PACKED) {
      r.mic = s.micro_exp[mrow + blk];
    } else {
      const uint2 m = *reinterpret_cast<const uint2*>(s.micro_exp + mrow + blk * 8);
      r.mic = (((m.x & 0x01010101u) * 0x10204080u) >> 28) | ((((m.y & 0x01010101u) * 0x10204080u) >> 28) << 4);
    }
    return r;
  }

  __device__ __forceinline__ static void codes_of(const MxRaw& r, uint32_t (&codes)[4]) {
    if (kNibbles) {
      mx4_nibbles_to_bytes(r.q.x, r.q.y, codes);
    } else {
      codes[0] = r.q.x; codes[1] = r.q.y; codes[2] = r.q.z; codes[3] = r.q.w;
    }
  }

  __device__ __forceinline__ static void store(const lq_mx_state& s, int64_t qrow, int64_t erow, int64_t mrow, int blk,
                                               const uint32_t (&codes)[4], uint32_t e, uint32_t mic) {
    uint8_t* q = static_cast<uint8_t*>(s.q_state) + qrow + blk * kQBytes;
    if (kNibbles) {
      uint32_t lo, hi;
      mx4_bytes_to_nibbles(codes, lo, hi);
      *reinterpret_cast<uint2*>(q) = make_uint2(lo, hi);
    } else {
      *reinterpret_cast<uint4*>(q) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
    }
    s.shared_exp[erow + blk] = static_cast<uint8_t>(e);
    if (LAYOUT == LQ_MX_LAYOUT_PACKED) {
      s.micro_exp[mrow + blk] = static_cast<uint8_t>(mic);
    } else {
      const uint32_t lo = ((mic & 0xFu) * 0x00204081u) & 0x01010101u;
      const uint32_t hi = (((mic >> 4) & 0xFu) * 0x00204081u) & 0x01010101u;
      *reinterpret_cast<uint2*>(s.micro_exp + mrow + blk * 8) = make_uint2(lo, hi);
    }
  }
};

// Rounding state that is the same for every block a thread handles.  `numel` = values in the whole
// state: the reference advances its Philox offset by it every step.
struct MxRoundBase {
  uint32_t wrap32, step, layer;
  uint64_t offset;
  const uint32_t* words;
};

__device__ __forceinline__ MxRoundBase make_round_base(const lq_rounding& r, uint64_t numel) {
  MxRoundBase b;
  const uint64_t extra = r.step_counter ? __ldcg(reinterpret_cast<const unsigned long long*>(r.step_counter)) : 0ull;
  b.offset = r.rng_offset + extra * numel;
  b.wrap32 = b.offset < (1ull << 32) ? 1u : 0u;
  b.step = static_cast<uint32_t>(r.step + extra);
  b.layer = r.layer;
  b.words = r.words;
  return b;
}

// Context of the block whose first value has linear index `lin` (a multiple of 16).
template <int MODE>
__device__ __forceinline__ MxRoundCtx round_ctx_at(const MxRoundBase& b, uint64_t lin) {
  MxRoundCtx c;
  c.wrap32 = b.wrap32;
  c.counter = (MODE == LQ_ROUND_PHILOX_LAYERED) ? (lin >> 4) : (MODE == LQ_ROUND_PHILOX_LAYERED4) ? (lin >> 2) : (b.offset + lin);
  c.step = b.step;
  c.layer = b.layer;
  c.words = (MODE == LQ_ROUND_SUPPLIED || MODE == LQ_ROUND_SUPPLIED_FIXED) ? b.words + lin : nullptr;
  return c;
}

struct MxUpdateDerived {
  enum : int32_t { kVec = 1, kAsk = 2 };
  int32_t nblk;        // dstate / 16
  int32_t lpr_log2;    // lanes per row = 1 << lpr_log2 >= nblk
  int32_t dt_uniform;  // dt and dt_bias do not depend on the row (dim) index
  int32_t a_scalar;    // A depends on the head only
  int32_t flags;       // kVec: x, out, B, C in 16 bits, aligned for vectors; D per head, no z; dim a multiple of 4.  kAsk: x, dt, A, B and C are asked for in
                       // L2 ahead of the wait.  (One word: a field more is a launch 1 % longer.)
  int32_t heads_per_cta;  // consecutive heads of one B/C group handled by one CTA
  PhiloxKeys keys;        // round keys of rounding.seed
  uint64_t units_total;   // fast path: batch * heads * dim / rows per pass (< 2^31)
  // fast path: the slab of a CTA without a division.  units_per_cta / units_rem: CTA c owns units_per_cta units, the
  // first units_rem CTAs one more
  uint32_t units_per_cta, units_rem;
  FastDiv div_steps_per_head, div_heads, div_dim, div_heads_per_group, div_groups;
};

// One CTA = `hpc` consecutive heads of one (batch, B/C group): B and C are fetched once and stay in
// registers for hpc * dim rows.  gridDim.x = batch * (heads / hpc).
template <int BITS, int LAYOUT, int MODE>
__global__ void __launch_bounds__(kUpdateThreads, 4) mx_state_update_kernel(const lq_mx_update_args a, const MxUpdateDerived d) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  extern __shared__ float smem_xy[];  // x of the CTA's rows, <h', C> of the rows, per-head dt and exp(A dt)
  const lq_mx_state& s = a.state;
  const int H = s.heads, P = s.dim, N = s.dstate;
  const int hpc = d.heads_per_cta;
  float* sx = smem_xy;
  float* sy = sx + hpc * P;
  float* sdt = sy + hpc * P;
  float* sdA = sdt + hpc;
  const int chunks = H / hpc;
  const int b = blockIdx.x / chunks;
  const int h0 = (blockIdx.x - b * chunks) * hpc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int blk = lane & ((1 << d.lpr_log2) - 1);
  const int rsub = lane >> d.lpr_log2;
  const int rows_per_warp = 32 >> d.lpr_log2;
  const int rows_per_pass = rows_per_warp * (kUpdateThreads / 32);
  const bool blk_ok = blk < d.nblk;
  const int n0 = blk * 16;
  const int grp = h0 / (H / a.ngroups);  // the same for every head of the CTA

  auto row_dt = [&](int h, int p) {
    float dt = load_as_float(a.dt, b * a.dt_stride[0] + h * a.dt_stride[1] + p * a.dt_stride[2], a.dt_dtype);
    if (a.dt_bias) dt += load_as_float(a.dt_bias, h * a.dt_bias_stride[0] + p * a.dt_bias_stride[1], a.dt_bias_dtype);
    if (a.dt_softplus) dt = softplus_ref(dt);
    return dt;
  };
  for (int i = threadIdx.x; i < hpc * P; i += kUpdateThreads) {
    const int hh = i / P, p = i - hh * P;
    sx[i] = load_as_float(a.x, b * a.x_stride[0] + (h0 + hh) * a.x_stride[1] + p * a.x_stride[2], a.x_dtype);
  }
  if (d.dt_uniform && threadIdx.x < hpc) {
    const float dt = row_dt(h0 + threadIdx.x, 0);
    sdt[threadIdx.x] = dt;
    sdA[threadIdx.x] = d.a_scalar ? expf(load_as_float(a.A, (h0 + threadIdx.x) * a.A_stride[0], a.A_dtype) * dt) : 0.0f;
  }

  // B and C of the group, this lane's 16 columns
  float Bv[16], Cv[16];
  if (blk_ok) {
    load_bc16(a.B, a.B_stride, a.B_dtype, b, grp, n0, Bv);
    load_bc16(a.C, a.C_stride, a.C_dtype, b, grp, n0, Cv);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) Bv[i] = Cv[i] = 0.0f;
  }
  const bool hoisted = d.dt_uniform && d.a_scalar;
  const MxRoundBase rb = make_round_base(a.rounding, static_cast<uint64_t>(s.batch) * H * P * N);
  __syncthreads();

#pragma unroll 1
  for (int hh = 0; hh < hpc; ++hh) {
    const int h = h0 + hh;
    const float dt_h = d.dt_uniform ? sdt[hh] : 0.0f;
    const float dA_h = sdA[hh];
    float dBv[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) dBv[i] = __fmul_rn(Bv[i], dt_h);
    const uint64_t lin_head = (static_cast<uint64_t>(b) * H + h) * P * static_cast<uint64_t>(N) + n0;
    const int64_t qbase = b * s.q_stride[0] + h * s.q_stride[1];
    const int64_t ebase = b * s.exp_stride[0] + h * s.exp_stride[1];
    const int64_t mbase = b * s.micro_stride[0] + h * s.micro_stride[1];
    const float* sxh = sx + hh * P;
    float* syh = sy + hh * P;

    int p0 = warp * rows_per_warp;
    MxRaw cur = {make_uint4(0, 0, 0, 0), 127u, 0u};
    if (blk_ok && p0 + rsub < P)
      cur = IO::load(s, qbase + (p0 + rsub) * s.q_stride[2], ebase + (p0 + rsub) * s.exp_stride[2],
                     mbase + (p0 + rsub) * s.micro_stride[2], blk);
#pragma unroll 1
    for (; p0 < P; p0 += rows_per_pass) {
      const int p = p0 + rsub;
      const bool active = blk_ok && p < P;
      // issue the next row's loads before working on this one
      const int pn = p + rows_per_pass;
      MxRaw nxt = {make_uint4(0, 0, 0, 0), 127u, 0u};
      if (blk_ok && pn < P)
        nxt = IO::load(s, qbase + pn * s.q_stride[2], ebase + pn * s.exp_stride[2], mbase + pn * s.micro_stride[2], blk);

      float y = 0.0f;
      if (active) {
        uint32_t codes[4];
        IO::codes_of(cur, codes);
        float hv[16];
        mx_decode_block(codes, cur.e, cur.mic, hv);
        const float xv = sxh[p];
        if (hoisted) {
          const float one[8] = {dA_h};
          y = mx_update_readout16<true>(hv, dBv, Cv, one, xv);  // h' = h exp(A dt) + (B dt) x
        } else {
          const float dt = d.dt_uniform ? dt_h : row_dt(h, p);
          if (d.a_scalar) {
            const float one[8] = {expf(load_as_float(a.A, h * a.A_stride[0], a.A_dtype) * dt)};
            float dBr[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) dBr[i] = __fmul_rn(Bv[i], dt);
            y = mx_update_readout16<true>(hv, dBr, Cv, one, xv);
          } else {
            // All sixteen of A are on their way before the first is used, and the type is asked for once: one after the other behind a question each they were
            // 16 latencies of L2 (us with a dense A, one after the other / now: 64 sequences MX8 231 / 171, MX4 233 / 167, one 13.5 / 9.6).
            const int64_t row = h * a.A_stride[0] + p * a.A_stride[1] + n0 * a.A_stride[2];
            float Ai[16];
            if (a.A_dtype == LQ_F32) {
#pragma unroll
              for (int i = 0; i < 16; ++i) Ai[i] = static_cast<const float*>(a.A)[row + i * a.A_stride[2]];
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) Ai[i] = load_as_float(a.A, row + i * a.A_stride[2], a.A_dtype);
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) hv[i] = fmaf(hv[i], expf(Ai[i] * dt), __fmul_rn(__fmul_rn(Bv[i], dt), xv));
            float y0 = 0.0f, y1 = 0.0f, y2 = 0.0f, y3 = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              y0 = fmaf(hv[i], Cv[i], y0);
              y1 = fmaf(hv[i + 1], Cv[i + 1], y1);
              y2 = fmaf(hv[i + 2], Cv[i + 2], y2);
              y3 = fmaf(hv[i + 3], Cv[i + 3], y3);
            }
            y = (y0 + y1) + (y2 + y3);
          }
        }
        const uint64_t lin = lin_head + static_cast<uint64_t>(static_cast<uint32_t>(p) * static_cast<uint32_t>(N));
        if (a.h_out) {
          float4* dst = reinterpret_cast<float4*>(a.h_out + lin);
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = make_float4(hv[4 * i], hv[4 * i + 1], hv[4 * i + 2], hv[4 * i + 3]);
        }
        const MxRoundCtx ctx = round_ctx_at<MODE>(rb, lin);
        uint32_t e_new, mic_new;
        mx_encode_block<BITS, MODE>(hv, ctx, d.keys, codes, e_new, mic_new);
        IO::store(s, qbase + p * s.q_stride[2], ebase + p * s.exp_stride[2], mbase + p * s.micro_stride[2], blk, codes, e_new,
                  mic_new);
      }
      // y = <h', C> over the row: reduce across the lanes that share it
      for (int o = (1 << d.lpr_log2) >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xFFFFFFFFu, y, o);
      if (active && blk == 0) syh[p] = y;
      cur = nxt;
    }
  }
  __syncthreads();
  // y = <h', C> + D x (* z), stored for all the CTA's rows at once
  for (int i = threadIdx.x; i < hpc * P; i += kUpdateThreads) {
    const int hh = i / P, p = i - hh * P, h = h0 + hh;
    float y = sy[i];
    if (a.D) y += sx[i] * load_as_float(a.D, h * a.D_stride[0] + p * a.D_stride[1], a.D_dtype);
    if (a.z) y *= load_as_float(a.z, b * a.z_stride[0] + h * a.z_stride[1] + p * a.z_stride[2], a.z_dtype);
    store_from_float(a.out, b * a.out_stride[0] + h * a.out_stride[1] + p * a.out_stride[2], a.out_dtype, y);
  }
}

// Fast path of the fused update: the shape every Mamba2 decode step has.  Requirements (checked
// on the host): dense 16-byte aligned state tensors, dt / dt_bias / A per head only, dstate / 16 a power of two,
// dim a multiple of the rows two warps cover, no h_out, fewer than 2^30 units.
//
// A step is 32 consecutive blocks: one per lane, `32 / (dstate / 16)` rows.  A unit is two steps.
// Units are numbered in memory order and dealt out contiguously, U / G to each of the G CTAs and one
// more to the first U mod G: a contiguous slab of the state, balanced to within one unit whatever the batch, the first half of
// its steps for warp 0 and the second for warp 1.  The grid is one wave of resident CTAs whenever the slab's x / y
// staging fits in shared memory.
//
// The state comes through a ring of two stages of four steps per warp (cp.async: a warp synchronises with itself only), so that a
// step has no global address arithmetic for its loads, no copies of prefetched registers, and its loads are one to two stages old.
// B and C of the slab's (batch, group)s and dB = B dt of a warp's current head wait in shared memory as [quarter][block] float4 and are read in every
// step: eight 128-bit loads that share addresses between rows and cost next to nothing beside the arithmetic, for 32 registers.
// A warp's first stage is as long as makes the others start where heads do.  A whole stage of one head with ordinary exponents asks nothing per
// step and takes two steps at a time; anything else goes step by step.
// 272 -> 248 instructions per 16 values (with set-up) and the packed operands of lq_mx_codec.cuh: MX8 1522 -> 1361 us (batch 250, eight layers; on boxes that are at their
// power limit then, 1520 -> 1403 to 1423), 422 -> 381 (64), deterministic rounding 402 -> 354 (60), MX4 417 -> 392 (64).  Four steps at a time,
// or two copies of two, run slower (1455, 1515).
// NBLK_T = dstate / 16 when known at compile time (8 for Nemotron-H: all lane and address arithmetic
// folds to constants), 0 = taken from the arguments.
// kRefAnyOffset: PHILOX_REF with an offset that is no multiple of 16 (a caller's own).  A block's counters may pass 2^32, so every word is drawn by itself.
constexpr int kRefAnyOffset = 64;
constexpr int kRingSteps = 4, kRingStages = 2;
constexpr int kPartialStride = 36;  // floats of a step's read-out partials: 32 and a shift of one 16-byte bank column
constexpr int kPartials = (kFastThreads / 32) * kRingSteps * kPartialStride;  // floats of a stage's, per CTA
template <int BITS, int LAYOUT>
struct MxRing {
  using IO = MxBlockIO<BITS, LAYOUT>;
  static constexpr uint32_t kQ = 32 * IO::kQBytes, kM = 32 * IO::kMicroBytes, kE = 32;  // bytes of a step
  static constexpr uint32_t kEChunks = kRingSteps * kE / 16;
  static constexpr uint32_t kOffE = kRingSteps * kQ, kOffM = kOffE + kRingSteps * kE;
  static constexpr uint32_t kStage = kOffM + kRingSteps * kM;
  static constexpr uint32_t kBytes = (kFastThreads / 32) * kRingStages * kStage;

  // Chunk c of a tensor's part of a stage goes through lane c mod 32 (e: the first kEChunks lanes, m: the next ones, so that packed e and m are
  // one instruction); chunks of steps from `left` on do not exist.  src: q / e or m at the warp's first step, plus 16 bytes per lane.
  struct Source {
    const uint8_t *q, *em, *m;  // em: e, or packed m on the next lanes; m: unpacked micro-exponents
    uint32_t dst_q, dst_em;
    __device__ __forceinline__ Source(uint32_t ring, const uint8_t* q0, const uint8_t* e0, const uint8_t* m0, uint32_t lane) {
      q = q0 + lane * 16;
      em = lane < kEChunks ? e0 + lane * 16 : m0 + (lane - kEChunks) * 16;
      m = m0 + lane * 16;
      dst_q = ring + lane * 16;
      dst_em = ring + (lane < kEChunks ? kOffE + lane * 16 : kOffM + (lane - kEChunks) * 16);
    }
  };
  __device__ __forceinline__ static void cp16(uint32_t dst, const uint8_t* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  }
  // WHOLE: with a form of its own for whole stages (MX8, batch 250: 1412 -> 1361 us; the shorter stages of MX4 and the few of the reference's
  // stream lose a little by the second copy)
  template <bool WHOLE>
  __device__ __forceinline__ static void issue(Source& s, uint32_t stage, uint32_t lane, int left, int advance = kRingSteps) {
    const uint32_t off = stage * kStage;
    if (WHOLE && left >= kRingSteps) {  // a whole stage: nothing to ask per chunk
#pragma unroll
      for (uint32_t c = 0; c < kRingSteps * kQ / 16; c += 32) cp16(s.dst_q + off + c * 16, s.q + c * 16);
      if (LAYOUT != LQ_MX_LAYOUT_PACKED) {
#pragma unroll
        for (uint32_t c = 0; c < kRingSteps * kM / 16; c += 32) cp16(s.dst_q + off + kOffM + c * 16, s.m + c * 16);
      }
      if (lane < (LAYOUT == LQ_MX_LAYOUT_PACKED ? 2 * kEChunks : kEChunks)) cp16(s.dst_em + off, s.em);
      if (LAYOUT != LQ_MX_LAYOUT_PACKED) s.m += advance * kM;
      asm volatile("cp.async.commit_group;" ::: "memory");
      s.q += advance * kQ;
      s.em += advance * kE;
      return;
    }
#pragma unroll
    for (uint32_t c = 0; c < kRingSteps * kQ / 16; c += 32)
      if (static_cast<int>(((c + lane) * 16) / kQ) < left) cp16(s.dst_q + off + c * 16, s.q + c * 16);
    if (lane < (LAYOUT == LQ_MX_LAYOUT_PACKED ? 2 * kEChunks : kEChunks) && static_cast<int>((lane & (kEChunks - 1)) >> 1) < left) cp16(s.dst_em + off, s.em);
    if (LAYOUT != LQ_MX_LAYOUT_PACKED) {
#pragma unroll
      for (uint32_t c = 0; c < kRingSteps * kM / 16; c += 32)
        if (static_cast<int>(((c + lane) * 16) / kM) < left) cp16(s.dst_q + off + kOffM + c * 16, s.m + c * 16);
      s.m += advance * kM;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    s.q += advance * kQ;
    s.em += advance * kE;
  }
  // this lane's block of the step whose mantissas start at `q` + lane * kQBytes and whose exponents at `e` + lane; d: steps further on
  __device__ __forceinline__ static MxRaw read(const uint8_t* q, const uint8_t* e, const uint8_t* m, uint32_t d) {
    MxRaw r;
    if (IO::kNibbles) {
      const uint2 v = *reinterpret_cast<const uint2*>(q + d * kQ);
      r.q = make_uint4(v.x, v.y, 0u, 0u);
    } else {
      r.q = *reinterpret_cast<const uint4*>(q + d * kQ);
    }
    r.e = e[d * kE];
    if (LAYOUT == LQ_MX_LAYOUT_PACKED) {
      r.mic = e[kOffM - kOffE + d * kM];
    } else {
      const uint2 mm = *reinterpret_cast<const uint2*>(m + d * kM);
      r.mic = (((mm.x & 0x01010101u) * 0x10204080u) >> 28) | ((((mm.y & 0x01010101u) * 0x10204080u) >> 28) << 4);
    }
    return r;
  }
};

template <int BITS, int LAYOUT, int MODE, int NBLK_T>
__global__ void __launch_bounds__(kFastThreads, kFastCtasPerSm) mx_state_update_fast_kernel(const lq_mx_update_args a, const MxUpdateDerived d) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  using Ring = MxRing<BITS, LAYOUT>;
  // whole stages two steps at a time; the reference's stream draws sixteen words a step, which leaves nothing to gain by a second copy (batch 32: 795 us
  // against 878)
  constexpr bool kWhole = MODE != LQ_ROUND_PHILOX_REF && MODE != kRefAnyOffset;
  constexpr bool kLongSteps = !kWhole || MODE == LQ_ROUND_PHILOX_LAYERED4;  // several draws a block
  constexpr bool kWholeIssue = kWhole && BITS == 8;
  // With four draws a block a step is long, and the second copy pays only in slabs that mostly stay in it (us of layered4 before there was one / always / from
  // twelve units a CTA on: batch 6 13.3 / 13.9 / 12.8, 8 16.1 / 17.0 / 15.5, 12 22.2 / 22.3 / 21.1, 14 (twelve units) 25.1 / 23.5 / 23.4, 20 34.4 / 33.4 / 33.3).
  const bool whole_pays = !kLongSteps || d.units_per_cta >= 3 * kRingSteps;
  constexpr int kUnroll = 2;
  extern __shared__ __align__(16) uint8_t smem_fast[];
  const lq_mx_state& s = a.state;
  const int H = s.heads, P = s.dim;
  // the warp's number from one lane: the compiler keeps what follows from it in uniform registers (24 layers of batch 1 of the reference's stream
  // 175 -> 172 us, eight of batch 60 with deterministic rounding 354 -> 345)
  const uint32_t lane = threadIdx.x & 31, warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);
  const int nblk = NBLK_T ? NBLK_T : d.nblk;
  const int lpr_log2 = NBLK_T == 8 ? 3 : d.lpr_log2;
  const int dstate = NBLK_T ? NBLK_T * 16 : s.dstate;
  const int blk = lane & (nblk - 1);
  const int rows_per_step = 32 >> lpr_log2;
  const int rows_per_unit = rows_per_step * (kFastThreads / 32);
  const uint32_t steps_per_head = static_cast<uint32_t>(P / rows_per_step);
  const int heads_per_group = H / a.ngroups;

  uint32_t steps[256 / kFastThreads];  // of the module's constants, which no kernel writes
#pragma unroll
  for (int i = 0; i < 256 / kFastThreads; ++i) steps[i] = mx_exp_step<BITS>(threadIdx.x + i * kFastThreads);
  // this CTA's slab: units [u0, u1), rows [R0, R1) of the [batch * heads * dim] row space; the first units_rem CTAs
  // take one unit more than the others
  const uint32_t u0 = blockIdx.x * d.units_per_cta + min(blockIdx.x, d.units_rem);
  const uint32_t n_units = d.units_per_cta + (blockIdx.x < d.units_rem ? 1u : 0u);
  // let the next kernel in the stream be scheduled behind this one (no effect without the launch attribute)
  pdl_launch_dependents();
  if (n_units == 0) return;
  const uint64_t R0 = static_cast<uint64_t>(u0) * rows_per_unit;
  const int n_rows = static_cast<int>(n_units) * rows_per_unit;
  const uint32_t step_first = 2 * u0, step_end = step_first + 2 * n_units;
  const uint32_t bh_first = fast_div(step_first, d.div_steps_per_head);  // first (batch * heads + head) index touched
  const uint32_t bh_last = fast_div(step_end - 1, d.div_steps_per_head);
  const uint32_t bg_first = fast_div(bh_first, d.div_heads_per_group);   // the same for (batch * groups + group)
  const int n_heads = static_cast<int>(bh_last - bh_first) + 1;
  const int n_bg = static_cast<int>(fast_div(bh_last, d.div_heads_per_group) - bg_first) + 1;
  float* const bc = reinterpret_cast<float*>(smem_fast + Ring::kBytes);  // per (batch, group): B, then C
  float* const sdB = bc + n_bg * 2 * dstate;   // per warp: B dt of its current head, laid out as B
  // read-out of a stage's rows where a row spans eight lanes: one partial sum per 16-value block, added up when the stage has been worked
  // through, in the order a butterfly over the eight lanes would add them
  float* const spart = sdB + (kFastThreads / 32) * dstate;
  float* const sx = spart + (NBLK_T == 8 ? kPartials : 0);  // x of the slab's rows
  float* const sy = sx + n_rows;   // <h', C> of the slab's rows
  float* const sdt = sy + n_rows;  // per touched head
  float* const sdA = sdt + n_heads;

  // (batch, head, row) of the slab's first row, once per CTA
  const int p_first = static_cast<int>(step_first - bh_first * steps_per_head) * rows_per_step;
  const int b_first = static_cast<int>(fast_div(bh_first, d.div_heads));
  const int h_first = static_cast<int>(bh_first - static_cast<uint32_t>(b_first) * static_cast<uint32_t>(H));
  auto row_coords = [&](int i, int& b, int& h, int& p) {
    const uint32_t pi = static_cast<uint32_t>(p_first + i);
    const uint32_t hq = fast_div(pi, d.div_dim);
    p = static_cast<int>(pi - hq * static_cast<uint32_t>(P));
    const uint32_t hh = static_cast<uint32_t>(h_first) + hq;
    const uint32_t bq = fast_div(hh, d.div_heads);
    b = b_first + static_cast<int>(bq);
    h = static_cast<int>(hh - bq * static_cast<uint32_t>(H));
  };
  // this warp's steps [0, n_units) start at block `block0` of the state
  const uint32_t my_step0 = step_first + warp * n_units;
  const int n_mine = static_cast<int>(n_units);
  const uint64_t block0 = static_cast<uint64_t>(my_step0) * 32;
  // its first head, the steps left of it, and the steps of its first stage: all of them if they fit one (batch 3 of the reference's stream 284 -> 273 us, 20
  // layers), else what is over stages that start where heads do (if heads are whole stages)
  const uint32_t bh_mine = fast_div(my_step0, d.div_steps_per_head);
  int left = static_cast<int>(steps_per_head - (my_step0 - bh_mine * steps_per_head));
  const int first = n_units <= kRingSteps ? static_cast<int>(n_units) : ((left - 1) & (kRingSteps - 1)) + 1;
  uint8_t* qptr = static_cast<uint8_t*>(s.q_state) + (block0 + lane) * IO::kQBytes;
  uint8_t* eptr = s.shared_exp + block0 + lane;
  uint8_t* mptr = s.micro_exp + (block0 + lane) * IO::kMicroBytes;
  // linear index of the block's first value; in the layered modes the Philox counter (block index / quad index)
  constexpr int kCtrShift = MODE == LQ_ROUND_PHILOX_LAYERED ? 4 : (MODE == LQ_ROUND_PHILOX_LAYERED4 ? 2 : 0);
  constexpr uint32_t dl = 512 >> kCtrShift;
  uint64_t lin = ((block0 + lane) * 16) >> kCtrShift;
  using Table = std::conditional_t<IO::kNibbles, MxPairMasks, MxPairFactors>;
  __shared__ Table table;
  for (int i = threadIdx.x; i < (IO::kNibbles ? 256 : 16); i += kFastThreads) table.fill(i);
  __shared__ uint32_t exp_step[256];
  uint8_t* const ring = smem_fast + warp * (kRingStages * Ring::kStage);
  typename Ring::Source source(static_cast<uint32_t>(__cvta_generic_to_shared(ring)), static_cast<const uint8_t*>(s.q_state) + block0 * IO::kQBytes,
                               s.shared_exp + block0, s.micro_exp + block0 * IO::kMicroBytes, lane);
  // what the first stages will read, asked for in L2 while the predecessor still runs (a prefetch reads nothing): 10.6 -> 10.1 us at
  // batch 8, ...
  if (lane == 0) {
    const uint32_t ahead = min(n_units, static_cast<uint32_t>(kRingSteps));
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const uint8_t*>(s.q_state) + block0 * IO::kQBytes), "r"(ahead * Ring::kQ) : "memory");
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(s.shared_exp + block0), "r"(ahead * Ring::kE) : "memory");
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(s.micro_exp + block0 * IO::kMicroBytes), "r"(ahead * Ring::kM) : "memory");
  }
  // B / C of (batch, group) bgi, block kb; `which` 0: B, 1: C
  const int n_bc = n_bg * nblk * 2;
  auto bc_source = [&](int i, const void*& base, const int64_t*& st, int& dtype, int& b, int& g, int& kb) {
    const int bgi = i >> (lpr_log2 + 1);
    kb = (i >> 1) & (nblk - 1);
    const uint32_t bg = bg_first + bgi;
    b = static_cast<int>(fast_div(bg, d.div_groups));
    g = static_cast<int>(bg) - b * a.ngroups;
    base = i & 1 ? a.C : a.B;
    st = i & 1 ? a.C_stride : a.B_stride;
    dtype = i & 1 ? a.C_dtype : a.B_dtype;
  };
  auto store_bc = [&](int i, const float (&v)[16]) {
    const int kb = (i >> 1) & (nblk - 1);
    float4* dst = reinterpret_cast<float4*>(bc + ((i >> (lpr_log2 + 1)) * 2 + (i & 1)) * dstate) + kb;
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[k * nblk] = make_float4(v[4 * k], v[4 * k + 2], v[4 * k + 1], v[4 * k + 3]);
  };
  auto stage_bc = [&](int i) {
    const void* base; const int64_t* st; int dtype, b, g, kb;
    bc_source(i, base, st, dtype, b, g, kb);
    float v[16];
    const int64_t (&strides)[3] = *reinterpret_cast<const int64_t (*)[3]>(st);
    load_bc16(base, strides, dtype, b, g, kb * 16, v);
    store_bc(i, v);
  };
  auto head_operands = [&](int i, float& dt, float& bias, float& A) {
    const unsigned hh = static_cast<unsigned>(h_first + i);
    const unsigned bq = fast_div(hh, d.div_heads);
    const int h = static_cast<int>(hh - bq * static_cast<unsigned>(H)), b = b_first + static_cast<int>(bq);
    dt = load_as_float(a.dt, b * a.dt_stride[0] + h * a.dt_stride[1], a.dt_dtype);
    bias = a.dt_bias ? load_as_float(a.dt_bias, h * a.dt_bias_stride[0], a.dt_bias_dtype) : 0.0f;
    A = load_as_float(a.A, h * a.A_stride[0], a.A_dtype);
  };
  auto stage_head = [&](int i, float dt, float bias, float A) {
    if (a.dt_bias) dt += bias;
    if (a.dt_softplus) dt = softplus_ref(dt);
    sdt[i] = dt;
    sdA[i] = expf(A * dt);
  };
  const int tid = threadIdx.x;
  // ... and, where the launch says so, the first round of every operand (batch 8: 10.2 -> 9.9 us a launch in a graph whose operands come from HBM).  The launch's word is
  // a predicate of the instruction: as a branch around all of this it changed the code of the steps (MX8 0.8 % slower, MX4 1 to 2 % faster).
  const int asks = d.flags & d.kAsk;
  const auto ask = [&](const void* p, int64_t i, int dtype) {  // a hint: nothing is read
    const uint8_t* const at = static_cast<const uint8_t*>(p) + i * (dtype == LQ_F32 ? 4 : 2);
    if (kLongSteps) asm volatile("prefetch.global.L2 [%0];" ::"l"(at) : "memory");
    else asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %1, 0;\n@p prefetch.global.L2 [%0];\n}" ::"l"(at), "r"(asks) : "memory");
  };
  if (tid < n_heads) {
    const unsigned hh = static_cast<unsigned>(h_first + tid);
    const unsigned bq = fast_div(hh, d.div_heads);
    const int h = static_cast<int>(hh - bq * static_cast<unsigned>(H)), b = b_first + static_cast<int>(bq);
    ask(a.dt, b * a.dt_stride[0] + h * a.dt_stride[1], a.dt_dtype);
    if (a.dt_bias) ask(a.dt_bias, h * a.dt_bias_stride[0], a.dt_bias_dtype);
    ask(a.A, h * a.A_stride[0], a.A_dtype);
  }
  if (4 * tid < n_rows) {
    int b, h, p;
    row_coords(4 * tid, b, h, p);
    ask(a.x, b * a.x_stride[0] + h * a.x_stride[1] + p * a.x_stride[2], a.x_dtype);
  }
  if (tid < n_bc) {
    const void* base; const int64_t* st; int dtype, b, g, kb;
    bc_source(tid, base, st, dtype, b, g, kb);
    ask(base, b * st[0] + g * st[1] + kb * 16 * st[2], dtype);
  }
#pragma unroll
  for (int i = 0; i < 256 / kFastThreads; ++i) exp_step[threadIdx.x + i * kFastThreads] = steps[i];
  // everything above is arithmetic on the arguments; from here on memory the predecessor may have written is read
  pdl_wait();
  // the first stages travel while the operands below are staged
  Ring::template issue<kWholeIssue>(source, 0, lane, min(n_mine, first), first);

  if (NBLK_T == 8 && (d.flags & d.kVec)) {
    // 16-bit operands in vectors.  The first round of every kind is requested before any of it is used: one latency, not three
    auto x_vec = [&](int i) {
      int b, h, p;
      row_coords(4 * i, b, h, p);
      return *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(a.x) + b * a.x_stride[0] + h * a.x_stride[1] + p);
    };
    auto to_float4 = [&](uint2 w) {
      if (a.x_dtype == LQ_BF16)
        return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xFFFF0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xFFFF0000u));
      const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
      return make_float4(lo.x, lo.y, hi.x, hi.y);
    };
    uint2 x0 = make_uint2(0u, 0u);
    float dt = 0.0f, bias = 0.0f, A = 0.0f;
    if (tid < n_heads) head_operands(tid, dt, bias, A);
    if (4 * tid < n_rows) x0 = x_vec(tid);
    if (tid < n_bc) stage_bc(tid);
    if (4 * tid < n_rows) reinterpret_cast<float4*>(sx)[tid] = to_float4(x0);
    if (tid < n_heads) stage_head(tid, dt, bias, A);
    for (int i = tid + kFastThreads; 4 * i < n_rows; i += kFastThreads) reinterpret_cast<float4*>(sx)[i] = to_float4(x_vec(i));
  } else {
    if (tid < n_bc) stage_bc(tid);
    for (int i = tid; i < n_rows; i += kFastThreads) {
      int b, h, p;
      row_coords(i, b, h, p);
      sx[i] = load_as_float(a.x, b * a.x_stride[0] + h * a.x_stride[1] + p * a.x_stride[2], a.x_dtype);
    }
    if (tid < n_heads) {
      float dt, bias, A;
      head_operands(tid, dt, bias, A);
      stage_head(tid, dt, bias, A);
    }
  }
  for (int i = tid + kFastThreads; i < n_bc; i += kFastThreads) stage_bc(i);
  for (int i = tid + kFastThreads; i < n_heads; i += kFastThreads) {
    float dt, bias, A;
    head_operands(i, dt, bias, A);
    stage_head(i, dt, bias, A);
  }
  const MxRoundBase rb = make_round_base(a.rounding, static_cast<uint64_t>(s.batch) * H * P * dstate);
  // layered modes: the counters of the whole state fit 32 bits (fast_update_applies), so the stream carries them
  constexpr bool kStream = MODE == LQ_ROUND_PHILOX_LAYERED || MODE == LQ_ROUND_PHILOX_LAYERED4;
  constexpr bool kDrawn = MODE == LQ_ROUND_PHILOX_REF;  // a block's 16 counters do not pass 2^32 (kRefAnyOffset otherwise)
  PhiloxStream stream;
  if (kStream) stream.init(static_cast<uint32_t>(lin), 0u, rb.step, rb.layer, d.keys);

  for (int i = 1; i < kRingStages; ++i) Ring::template issue<kWholeIssue>(source, i, lane, n_mine - first - (i - 1) * kRingSteps);
  __syncthreads();

  // current head of this warp: its operands, and the steps left in it
  const float* head = sdt + (bh_mine - bh_first);
  const uint32_t bg_mine = fast_div(bh_mine, d.div_heads_per_group);
  int h_in_group = static_cast<int>(bh_mine - bg_mine * static_cast<uint32_t>(heads_per_group));
  const float4* bcp = reinterpret_cast<const float4*>(bc + (bg_mine - bg_first) * 2 * dstate);
  float4* const dBp = reinterpret_cast<float4*>(sdB + warp * dstate);
  float dA;
  uint32_t e_max;
  auto read16 = [&](const float4* src, float (&v)[16]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 f = src[k * nblk];
      v[4 * k] = f.x; v[4 * k + 2] = f.y; v[4 * k + 1] = f.z; v[4 * k + 3] = f.w;
    }
  };
  auto load_head = [&]() {
    const float dt = head[0];
    dA = head[n_heads];
    e_max = dA <= 1048576.0f ? 228u : 0u;
    __syncwarp();  // the head before has been read
    for (int i = lane; i < dstate / 4; i += 32) {
      const float4 f = bcp[i];
      dBp[i] = make_float4(__fmul_rn(f.x, dt), __fmul_rn(f.y, dt), __fmul_rn(f.z, dt), __fmul_rn(f.w, dt));
    }
    __syncwarp();
  };
  load_head();

  auto next_head = [&]() {  // B / C change only with the (batch, group)
    left = steps_per_head;
    ++head;
    if (++h_in_group == heads_per_group) {
      h_in_group = 0;
      bcp += dstate / 2;
    }
    load_head();
  };

  const float* xp = sx + warp * n_mine * rows_per_step + (lane >> lpr_log2);
  float* yp = sy + warp * n_mine * rows_per_step + (NBLK_T == 8 ? lane : lane >> lpr_log2);
  float* const part = spart + warp * (kRingSteps * kPartialStride);
  uint32_t stage = 0;
  // One step, the k-th from where the running pointers are: this lane's block; returns its share of <h', C>.
  const uint8_t *rq = ring, *re = ring, *rm = ring;  // where the current step's block lies in the ring
  auto step = [&](auto known, int k) {
    const MxRaw now = Ring::read(rq, re, rm, k);
    // The reference's stream: the block's words first, four chains at a time, while few registers are in use.  (Drawn where they are used,
    // the chains ran almost one behind the other: 1 / 4 / 32 sequences 8.3 / 19.1 / 113 -> 7.6 / 17.5 / 103 us a launch.)
    uint32_t words[16];
    if (kDrawn) {
      const MxRoundCtx rc = round_ctx_at<MODE>(rb, lin);
      PhiloxWords0 words0;
      words0.init(static_cast<uint32_t>(rc.counter), rc.wrap32 ? 0u : static_cast<uint32_t>(rc.counter >> 32), d.keys);
#pragma unroll
      for (int i = 0; i < 16; i += 4) words0.draw<4>(i, d.keys, words + i);
#pragma unroll
      for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(words[i]));  // stay here
    }
    float hv[16], sd[8], dB[16], Cv[16];
    mx_decode_scaled<decltype(known)::value>(now.q, now.e, now.mic, dA, e_max, table, hv, sd);
    read16(dBp + blk, dB);
    read16(bcp + dstate / 4 + blk, Cv);
    const float y = mx_update_readout16<IO::kNibbles>(hv, dB, Cv, sd, xp[k * rows_per_step]);  // h' = h exp(A dt) + (B dt) x
    MxRoundCtx ctx = round_ctx_at<MODE>(rb, lin);
    ctx.exp_step = exp_step;
    if (kStream) ctx.stream = &stream;
    if (kDrawn) ctx.drawn = words;
    uint32_t codes[4], e_new, mic_new;
    mx_encode_block<BITS, MODE, IO::kNibbles>(hv, ctx, d.keys, codes, e_new, mic_new);
    IO::store_ptr(qptr + k * Ring::kQ, eptr + k * Ring::kE, mptr + k * Ring::kM, codes, e_new, mic_new);
    if (kStream) stream.pa += static_cast<uint64_t>(kPhiloxM0) * dl; else lin += dl;
    return y;
  };
  float* part_k = part;
  auto advance = [&](int k) {
    rq += k * Ring::kQ; re += k * Ring::kE; rm += k * Ring::kM;
    qptr += k * Ring::kQ; eptr += k * Ring::kE; mptr += k * Ring::kM;
    xp += k * rows_per_step;
    part_k += k * kPartialStride;
    if (NBLK_T != 8) yp += k * rows_per_step;
  };
  auto put_y = [&](int k, float y) {
    if (NBLK_T == 8) {
      part_k[k * kPartialStride] = y;
    } else {
      for (int o = nblk >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xFFFFFFFFu, y, o);
      if (blk == 0) yp[k * rows_per_step] = y;
    }
  };
#pragma unroll 1
  for (int todo = n_mine, len = first; todo > 0; todo -= len, len = kRingSteps) {  // steps to do from this stage on, steps in it
    asm volatile("cp.async.wait_group %0;" ::"n"(kRingStages - 1) : "memory");
    __syncwarp();
    const uint8_t* const buf = ring + stage * Ring::kStage;
    rq = buf + lane * IO::kQBytes;
    re = buf + Ring::kOffE + lane;
    rm = buf + Ring::kOffM + lane * IO::kMicroBytes;
    part_k = part + lane;
    const int n = min(len, todo);
    if (left == 0) next_head();
    // A whole stage of one head whose stored exponents are ordinary (four a lane: nonzero, the two top bits not both set; dA likewise) needs no
    // question per step.
    const uint32_t e4 = reinterpret_cast<const uint32_t*>(buf + Ring::kOffE)[lane];
    const bool odd = ((((e4 - 0x01010101u) & ~e4) | (e4 & (e4 << 1))) & 0x80808080u) != 0u;
    if (kWhole && whole_pays && n == kRingSteps && left >= kRingSteps && e_max != 0u && !__any_sync(0xFFFFFFFFu, odd)) {
      left -= kRingSteps;
#pragma unroll 1
      for (int k0 = 0; k0 < kRingSteps; k0 += kUnroll) {
        float y[kUnroll];
#pragma unroll
        for (int k = 0; k < kUnroll; ++k) y[k] = step(std::true_type{}, k);
#pragma unroll
        for (int k = 0; k < kUnroll; ++k) put_y(k, y[k]);
        advance(kUnroll);
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < n; ++k) {
        if (left == 0) next_head();
        --left;
        put_y(0, step(std::false_type{}, 0));
        advance(1);
      }
    }
    __syncwarp();  // the stage has been read
    if (NBLK_T == 8 && lane < 4 * kRingSteps) {  // row lane & 3 of step lane / 4; of steps that do not exist: stale sums into rows that do not
      const float4* p = reinterpret_cast<const float4*>(part + (lane >> 2) * kPartialStride + (lane & 3) * 8);
      const float4 p0 = p[0], p1 = p[1];
      if (static_cast<int>(lane >> 2) < n) yp[0] = ((p0.x + p1.x) + (p0.z + p1.z)) + ((p0.y + p1.y) + (p0.w + p1.w));
    }
    Ring::template issue<kWholeIssue>(source, stage, lane, todo - len - (kRingStages - 1) * kRingSteps);
    if (NBLK_T == 8) yp += n * rows_per_step;
    stage ^= 1u;
  }
  __syncthreads();
  // y = <h', C> + D x (* z), stored for the whole slab at once
  if (NBLK_T == 8 && (d.flags & d.kVec)) {  // a thread takes the four rows of a step
    for (int i = tid; 4 * i < n_rows; i += kFastThreads) {
      int b, h, p;
      row_coords(4 * i, b, h, p);
      const float4 sum = reinterpret_cast<const float4*>(sy)[i];
      float y[4] = {sum.x, sum.y, sum.z, sum.w};
      if (a.D) {
        const float D = load_as_float(a.D, h * a.D_stride[0], a.D_dtype);
        const float4 x = reinterpret_cast<const float4*>(sx)[i];
        y[0] += x.x * D; y[1] += x.y * D; y[2] += x.z * D; y[3] += x.w * D;
      }
      uint2 w;
      if (a.out_dtype == LQ_BF16) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[1]), hi = __floats2bfloat162_rn(y[2], y[3]);
        w = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      } else {
        const __half2 lo = __floats2half2_rn(y[0], y[1]), hi = __floats2half2_rn(y[2], y[3]);
        w = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
      *reinterpret_cast<uint2*>(static_cast<uint16_t*>(a.out) + b * a.out_stride[0] + h * a.out_stride[1] + p) = w;
    }
    return;
  }
  for (int i = tid; i < n_rows; i += kFastThreads) {
    int b, h, p;
    row_coords(i, b, h, p);
    float y = sy[i];
    if (a.D) y += sx[i] * load_as_float(a.D, h * a.D_stride[0] + p * a.D_stride[1], a.D_dtype);
    if (a.z) y *= load_as_float(a.z, b * a.z_stride[0] + h * a.z_stride[1] + p * a.z_stride[2], a.z_dtype);
    store_from_float(a.out, b * a.out_stride[0] + h * a.out_stride[1] + p * a.out_stride[2], a.out_dtype, y);
  }
}

// ---- stand-alone codec kernels: one thread per 16-value block ----------------------------------
template <int BITS, int LAYOUT, int MODE>
__global__ void mx_quantize_kernel(const lq_mx_state s, const void* __restrict__ src, int src_dtype, int64_t src_row_stride,
                                   const lq_rounding rnd, const PhiloxKeys keys, int64_t total_blocks) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  const int nblk = s.dstate / 16;
  const MxRoundBase rb = make_round_base(rnd, static_cast<uint64_t>(s.batch) * s.heads * s.dim * s.dstate);
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total_blocks;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = t / nblk;
    const int blk = static_cast<int>(t - row * nblk);
    const int p = static_cast<int>(row % s.dim);
    const int64_t bh = row / s.dim;
    const int h = static_cast<int>(bh % s.heads);
    const int64_t b = bh / s.heads;
    float hv[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) hv[i] = load_as_float(src, row * src_row_stride + blk * 16 + i, src_dtype);
    const uint64_t lin = static_cast<uint64_t>(row) * s.dstate + blk * 16;
    const MxRoundCtx ctx = round_ctx_at<MODE>(rb, lin);
    uint32_t codes[4], e, mic;
    mx_encode_block<BITS, MODE>(hv, ctx, keys, codes, e, mic);
    IO::store(s, b * s.q_stride[0] + h * s.q_stride[1] + p * s.q_stride[2],
              b * s.exp_stride[0] + h * s.exp_stride[1] + p * s.exp_stride[2],
              b * s.micro_stride[0] + h * s.micro_stride[1] + p * s.micro_stride[2], blk, codes, e, mic);
  }
}

// Dense state and source: block t of one is block t of the other, 32 or 64 bytes in and one block out for each of a thread's two blocks,
// nothing divided.
// Bound by latency and instruction issue at the sizes of a prompt's end (8 x 128 x 64 x 128 values from bf16, 26 MB, 4 us at the copy rate): rounding by
// the addition that forms the code, in place of a rounding instruction of an eighth of the rate, and the source asked for in L2 before the wait:
// twelve launches behind two appends 102.5 -> 97.5 us, of fp32 states 116 -> 110.
template <int BITS, int LAYOUT, int MODE, int SRC>
__global__ void __launch_bounds__(128) mx_quantize_dense_kernel(const lq_mx_state s, const void* src, const lq_rounding rnd, const PhiloxKeys keys,
                                                                int64_t total_blocks, uint64_t numel) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  pdl_launch_dependents();
  constexpr int N = SRC == LQ_F32 ? 4 : 2;  // 16-byte loads of a block
  const int64_t t0 = blockIdx.x * 256ll + threadIdx.x;
  if ((threadIdx.x & (N == 2 ? 3 : 1)) == 0) {  // a thread per 128 bytes asks for them in L2 while the predecessor still runs (a prefetch reads nothing)
#pragma unroll
    for (int j = 0; j < 2; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint4*>(src) + min(t0 + 128 * j, total_blocks - 1) * N));
  }
  pdl_wait();
  uint4 raw[2][N];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint4* p = static_cast<const uint4*>(src) + min(t0 + 128 * j, total_blocks - 1) * N;
#pragma unroll
    for (int i = 0; i < N; ++i) raw[j][i] = p[i];
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int64_t t = t0 + 128 * j;
    if (t >= total_blocks) return;
    float hv[16];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint32_t w[4] = {raw[j][i].x, raw[j][i].y, raw[j][i].z, raw[j][i].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (SRC == LQ_F32) {
          hv[(4 * i + k) & 15] = __uint_as_float(w[k]);
        } else {
          const float2 f = SRC == LQ_BF16 ? make_float2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xFFFF0000u))
                                          : __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
          hv[(8 * i + 2 * k) & 15] = f.x;
          hv[(8 * i + 2 * k + 1) & 15] = f.y;
        }
      }
    }
    const MxRoundCtx ctx = round_ctx_at<MODE>(make_round_base(rnd, numel), static_cast<uint64_t>(t) * 16);
    uint32_t codes[4], e, mic;
    mx_encode_block<BITS, MODE, IO::kNibbles>(hv, ctx, keys, codes, e, mic);
    IO::store_ptr(static_cast<uint8_t*>(s.q_state) + t * IO::kQBytes, s.shared_exp + t, s.micro_exp + t * IO::kMicroBytes, codes, e, mic);
  }
}

template <int BITS, int LAYOUT>
__global__ void mx_dequantize_kernel(const lq_mx_state s, float* __restrict__ dst, int64_t dst_row_stride, int64_t total_blocks) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  const int nblk = s.dstate / 16;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total_blocks;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = t / nblk;
    const int blk = static_cast<int>(t - row * nblk);
    const int p = static_cast<int>(row % s.dim);
    const int64_t bh = row / s.dim;
    const int h = static_cast<int>(bh % s.heads);
    const int64_t b = bh / s.heads;
    const MxRaw r = IO::load(s, b * s.q_stride[0] + h * s.q_stride[1] + p * s.q_stride[2],
                             b * s.exp_stride[0] + h * s.exp_stride[1] + p * s.exp_stride[2],
                             b * s.micro_stride[0] + h * s.micro_stride[1] + p * s.micro_stride[2], blk);
    uint32_t codes[4];
    IO::codes_of(r, codes);
    float hv[16];
    mx_decode_block(codes, r.e, r.mic, hv);
#pragma unroll
    for (int i = 0; i < 16; ++i) dst[row * dst_row_stride + blk * 16 + i] = hv[i];
  }
}

template <int BITS, int SRC_LAYOUT, int DST_LAYOUT>
__global__ void mx_convert_kernel(const lq_mx_state src, const lq_mx_state dst, int64_t total_blocks) {
  using IOS = MxBlockIO<BITS, SRC_LAYOUT>;
  using IOD = MxBlockIO<BITS, DST_LAYOUT>;
  const int nblk = src.dstate / 16;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total_blocks;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = t / nblk;
    const int blk = static_cast<int>(t - row * nblk);
    const int p = static_cast<int>(row % src.dim);
    const int64_t bh = row / src.dim;
    const int h = static_cast<int>(bh % src.heads);
    const int64_t b = bh / src.heads;
    const MxRaw r = IOS::load(src, b * src.q_stride[0] + h * src.q_stride[1] + p * src.q_stride[2],
                              b * src.exp_stride[0] + h * src.exp_stride[1] + p * src.exp_stride[2],
                              b * src.micro_stride[0] + h * src.micro_stride[1] + p * src.micro_stride[2], blk);
    uint32_t codes[4];
    IOS::codes_of(r, codes);
    IOD::store(dst, b * dst.q_stride[0] + h * dst.q_stride[1] + p * dst.q_stride[2],
               b * dst.exp_stride[0] + h * dst.exp_stride[1] + p * dst.exp_stride[2],
               b * dst.micro_stride[0] + h * dst.micro_stride[1] + p * dst.micro_stride[2], blk, codes, r.e, r.mic);
  }
}

__global__ void counter_add_kernel(unsigned long long* counter, unsigned long long inc) { *counter += inc; }

// ---- host side --------------------------------------------------------------------------------
static int validate_state(const lq_mx_state& s, const char* who) {
  LQ_CHECK_ARG(s.q_state && s.shared_exp && s.micro_exp, "%s: null state pointer", who);
  LQ_CHECK_ARG(s.format_bits == 8 || s.format_bits == 4, "%s: Only MX8 and MX4 state quantization are supported, got format_bits=%d",
               who, s.format_bits);
  LQ_CHECK_ARG(s.layout == LQ_MX_LAYOUT_REFERENCE || s.layout == LQ_MX_LAYOUT_PACKED, "%s: unknown layout %d", who, s.layout);
  LQ_CHECK_ARG(s.batch > 0 && s.heads > 0 && s.dim > 0 && s.dstate > 0, "%s: empty state [%d,%d,%d,%d]", who, s.batch,
               s.heads, s.dim, s.dstate);
  LQ_CHECK_ARG(s.dstate % 16 == 0, "%s: MX%d state dim must be divisible by 16, got %d", who, s.format_bits, s.dstate);
  LQ_CHECK_ARG(static_cast<int64_t>(s.batch) * s.heads < (1ll << 31), "%s: batch*heads too large", who);
  const bool nib = s.format_bits == 4 && s.layout == LQ_MX_LAYOUT_PACKED;
  const int qalign = nib ? 8 : 16;
  LQ_CHECK_ARG(reinterpret_cast<uintptr_t>(s.q_state) % qalign == 0, "%s: q_state must be %d-byte aligned", who, qalign);
  for (int i = 0; i < 3; ++i)
    LQ_CHECK_ARG(s.q_stride[i] % qalign == 0, "%s: q_state strides must be multiples of %d bytes", who, qalign);
  if (s.layout == LQ_MX_LAYOUT_REFERENCE) {
    LQ_CHECK_ARG(reinterpret_cast<uintptr_t>(s.micro_exp) % 8 == 0, "%s: micro_exp must be 8-byte aligned", who);
    for (int i = 0; i < 3; ++i) LQ_CHECK_ARG(s.micro_stride[i] % 8 == 0, "%s: micro_exp strides must be multiples of 8", who);
  }
  return LQ_OK;
}

static int validate_rounding(const lq_rounding& r, const char* who) {
  LQ_CHECK_ARG(r.mode >= LQ_ROUND_HALF_UP && r.mode <= LQ_ROUND_PHILOX_LAYERED4, "%s: unknown rounding mode %d", who, r.mode);
  if (r.mode == LQ_ROUND_SUPPLIED || r.mode == LQ_ROUND_SUPPLIED_FIXED) {
    LQ_CHECK_ARG(r.words != nullptr, "%s: rounding mode %d needs words", who, r.mode);
    LQ_CHECK_ARG(reinterpret_cast<uintptr_t>(r.words) % 16 == 0, "%s: rounding words must be 16-byte aligned", who);
  }
  LQ_CHECK_ARG(reinterpret_cast<uintptr_t>(r.step_counter) % 8 == 0, "%s: step_counter must be 8-byte aligned", who);
  return LQ_OK;
}

template <int BITS, int LAYOUT>
static bool fast_update_applies(const lq_mx_update_args& a, const MxUpdateDerived& d) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  const lq_mx_state& s = a.state;
  const int64_t q_row = static_cast<int64_t>(d.nblk) * IO::kQBytes, m_row = static_cast<int64_t>(d.nblk) * IO::kMicroBytes;
  const int rows_per_pass = (32 >> d.lpr_log2) * (kFastThreads / 32);
  const bool dense = s.q_stride[2] == q_row && s.q_stride[1] == q_row * s.dim && s.q_stride[0] == q_row * s.dim * s.heads &&
                     s.exp_stride[2] == d.nblk && s.exp_stride[1] == static_cast<int64_t>(d.nblk) * s.dim &&
                     s.exp_stride[0] == static_cast<int64_t>(d.nblk) * s.dim * s.heads && s.micro_stride[2] == m_row &&
                     s.micro_stride[1] == m_row * s.dim && s.micro_stride[0] == m_row * s.dim * s.heads;
  // the ring's 16-byte copies (q_state is aligned in any case)
  const bool aligned = reinterpret_cast<uintptr_t>(s.q_state) % 16 == 0 && reinterpret_cast<uintptr_t>(s.shared_exp) % 16 == 0 &&
                       reinterpret_cast<uintptr_t>(s.micro_exp) % 16 == 0;
  // fewer than 2^30 units (2^31 steps) keep the kernel's index arithmetic in 32 bits and its multiply-high divisions exact
  const uint64_t units = static_cast<uint64_t>(s.batch) * s.heads * (s.dim / rows_per_pass);
  // Philox counters of the layered modes stay in 32 bits
  const int counter_log2 = a.rounding.mode == LQ_ROUND_PHILOX_LAYERED4 ? 2 : 4;
  const uint64_t counters = a.rounding.mode == LQ_ROUND_PHILOX_LAYERED || a.rounding.mode == LQ_ROUND_PHILOX_LAYERED4
                                ? (static_cast<uint64_t>(s.batch) * s.heads * s.dim * s.dstate) >> counter_log2 : 0;
  return dense && d.dt_uniform && d.a_scalar && a.h_out == nullptr && (1 << d.lpr_log2) == d.nblk &&
         s.dim % rows_per_pass == 0 && aligned && units < (1ull << 30) && counters <= (1ull << 32);
}

// Units of a CTA's slab at most; LQ_MX_MAX_UNITS (a tuning aid) is read once.
static uint64_t max_slab_units() {
  static const uint64_t units = [] {
    const char* env = getenv("LQ_MX_MAX_UNITS");
    return static_cast<uint64_t>(env ? std::min(400, std::max(1, atoi(env))) : 192);
  }();
  return units;
}

template <int BITS, int LAYOUT>
static void launch_update_mode(const lq_mx_update_args& a, const MxUpdateDerived& d, cudaStream_t st) {
  using IO = MxBlockIO<BITS, LAYOUT>;
  if (fast_update_applies<BITS, LAYOUT>(a, d)) {
    // One wave of resident CTAs when a CTA's slab stays within max_units units (its x / y staging: 8 bytes per row, as much as
    // lets kFastCtasPerSm CTAs share an SM's 228 KB); more waves of equally sized slabs otherwise.  Longer slabs have less set-up: batch 250
    // 1385 us with 64 units at most, 1372 with 80 to 192.
    const int rows_per_pass = (32 >> d.lpr_log2) * (kFastThreads / 32);
    const auto smem_of = [&](uint64_t units) {
      const uint64_t heads = units / (a.state.dim / rows_per_pass) + 2, groups = heads / (a.state.heads / a.ngroups) + 2;
      return MxRing<BITS, LAYOUT>::kBytes + sizeof(float) * (2 * units * rows_per_pass + 2 * heads + a.state.dstate * (2 * groups + kFastThreads / 32) +
                                                             (d.nblk == 8 ? kPartials : 0));
    };
    const size_t budget = 228 * 1024 / kFastCtasPerSm - 1024 - 1024 - (IO::kNibbles ? sizeof(MxPairMasks) : sizeof(MxPairFactors));
    uint64_t max_units = max_slab_units();
    while (max_units > 1 && smem_of(max_units) > budget) --max_units;
    MxUpdateDerived dd = d;
    const auto vec16 = [](const void* p, int dtype, const int64_t* st, int mult) {  // 16-bit, innermost contiguous, `mult` elements aligned
      return dtype != LQ_F32 && st[2] == 1 && st[0] % mult == 0 && st[1] % mult == 0 && reinterpret_cast<uintptr_t>(p) % (2 * mult) == 0;
    };
    const bool vec = vec16(a.x, a.x_dtype, a.x_stride, 4) && vec16(a.out, a.out_dtype, a.out_stride, 4) && vec16(a.B, a.B_dtype, a.B_stride, 8) &&
             vec16(a.C, a.C_dtype, a.C_stride, 8) && a.state.dim % 4 == 0 && !a.z && (!a.D || a.D_stride[1] == 0);
    dd.units_total = static_cast<uint64_t>(a.state.batch) * a.state.heads * (a.state.dim / rows_per_pass);
    const uint64_t wave = static_cast<uint64_t>(kFastCtasPerSm) * sm_count();
    uint64_t ctas = std::min<uint64_t>(dd.units_total, wave);
    if (dd.units_total > ctas * max_units) {
      ctas = (dd.units_total + max_units - 1) / max_units;
      ctas = (ctas + wave - 1) / wave * wave;
    }
    dd.units_per_cta = static_cast<uint32_t>(dd.units_total / ctas);
    dd.units_rem = static_cast<uint32_t>(dd.units_total % ctas);
    // Several CTAs an SM of one unit each are through before their askings are, which then stand in the way, most of all where all ask for the same lines of B and
    // C.  us with / without, operands in HBM: two sequences of 48 heads x 96 and one group 5.31 / 4.76 (MX4 5.32 / 4.74), one of 128 x 64 4.65 / 4.57 (MX4 4.39
    // / 4.33); with one CTA an SM (24 x 40) 3.71 / 3.86.  (Streams of several draws a block ask in any case: their steps are long, the reference's
    // 7.13 / 7.33.)
    const bool ask = dd.units_total > ctas || ctas <= static_cast<uint64_t>(sm_count());
    dd.flags = (vec ? dd.kVec : 0) | (ask ? dd.kAsk : 0);
    dd.div_steps_per_head = fast_div_of(static_cast<uint32_t>(2 * (a.state.dim / rows_per_pass)));
    dd.div_groups = fast_div_of(static_cast<uint32_t>(a.ngroups));
    dd.div_heads = fast_div_of(static_cast<uint32_t>(a.state.heads));
    dd.div_dim = fast_div_of(static_cast<uint32_t>(a.state.dim));
    dd.div_heads_per_group = fast_div_of(static_cast<uint32_t>(a.state.heads / a.ngroups));
    const unsigned grid = static_cast<unsigned>(ctas);
    const size_t smem = smem_of((dd.units_total + ctas - 1) / ctas);
    const MxUpdateDerived& d = dd;
#define LQ_FAST_LAUNCH(MODE_)                                                                         \
  do {                                                                                               \
    if (d.nblk == 8) launch_dependent(mx_state_update_fast_kernel<BITS, LAYOUT, MODE_, 8>, grid, kFastThreads, smem, st, a, d); \
    else launch_dependent(mx_state_update_fast_kernel<BITS, LAYOUT, MODE_, 0>, grid, kFastThreads, smem, st, a, d); \
  } while (0)
    switch (a.rounding.mode) {
      case LQ_ROUND_HALF_UP: LQ_FAST_LAUNCH(LQ_ROUND_HALF_UP); break;
      case LQ_ROUND_HALF_EVEN: LQ_FAST_LAUNCH(LQ_ROUND_HALF_EVEN); break;
      case LQ_ROUND_PHILOX_REF:  // the state's size, by which a step counter moves the offset, is a multiple of 16
        if (a.rounding.rng_offset % 16 == 0) LQ_FAST_LAUNCH(LQ_ROUND_PHILOX_REF); else LQ_FAST_LAUNCH(kRefAnyOffset);
        break;
      case LQ_ROUND_SUPPLIED: LQ_FAST_LAUNCH(LQ_ROUND_SUPPLIED); break;
      case LQ_ROUND_PHILOX_LAYERED: LQ_FAST_LAUNCH(LQ_ROUND_PHILOX_LAYERED); break;
      case LQ_ROUND_PHILOX_LAYERED4: LQ_FAST_LAUNCH(LQ_ROUND_PHILOX_LAYERED4); break;
      default: LQ_FAST_LAUNCH(LQ_ROUND_SUPPLIED_FIXED); break;
    }
#undef LQ_FAST_LAUNCH
    return;
  }
  const dim3 grid(a.state.batch * (a.state.heads / d.heads_per_cta)), block(kUpdateThreads);
  const size_t smem = sizeof(float) * (2 * static_cast<size_t>(d.heads_per_cta) * a.state.dim + 2 * d.heads_per_cta);
  switch (a.rounding.mode) {
    case LQ_ROUND_HALF_UP: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_HALF_UP><<<grid, block, smem, st>>>(a, d); break;
    case LQ_ROUND_HALF_EVEN: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_HALF_EVEN><<<grid, block, smem, st>>>(a, d); break;
    case LQ_ROUND_PHILOX_REF: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_PHILOX_REF><<<grid, block, smem, st>>>(a, d); break;
    case LQ_ROUND_SUPPLIED: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_SUPPLIED><<<grid, block, smem, st>>>(a, d); break;
    case LQ_ROUND_PHILOX_LAYERED: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_PHILOX_LAYERED><<<grid, block, smem, st>>>(a, d); break;
    case LQ_ROUND_PHILOX_LAYERED4: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_PHILOX_LAYERED4><<<grid, block, smem, st>>>(a, d); break;
    default: mx_state_update_kernel<BITS, LAYOUT, LQ_ROUND_SUPPLIED_FIXED><<<grid, block, smem, st>>>(a, d); break;
  }
}

template <int BITS, int LAYOUT>
static void launch_quantize_mode(const lq_mx_state& s, const void* src, int dt, int64_t stride, const lq_rounding& r,
                                 int64_t total, cudaStream_t st) {
  const int block = 128;
  const int grid = static_cast<int>(std::min<int64_t>((total + block - 1) / block, 1 << 20));
  const PhiloxKeys keys = make_philox_keys(r.seed);
  using IO = MxBlockIO<BITS, LAYOUT>;
  const int64_t nblk = s.dstate / 16, rows_b = static_cast<int64_t>(s.heads) * s.dim;
  const bool dense = stride == s.dstate && s.q_stride[2] == nblk * IO::kQBytes && s.exp_stride[2] == nblk && s.micro_stride[2] == nblk * IO::kMicroBytes &&
                     (s.heads == 1 || (s.q_stride[1] == s.dim * s.q_stride[2] && s.exp_stride[1] == s.dim * nblk && s.micro_stride[1] == s.dim * s.micro_stride[2])) &&
                     (s.batch == 1 || (s.q_stride[0] == rows_b * s.q_stride[2] && s.exp_stride[0] == rows_b * nblk && s.micro_stride[0] == rows_b * s.micro_stride[2]));
  // the rounding of the one-off quantiser; the other modes (tests, tools) stay on the general kernel
  if (r.mode == LQ_ROUND_HALF_EVEN && dense && reinterpret_cast<uintptr_t>(src) % 16 == 0 && total < (1ll << 37)) {
    const unsigned g = static_cast<unsigned>((total + 255) / 256);
    const uint64_t numel = static_cast<uint64_t>(total) * 16;
    if (dt == LQ_BF16) launch_dependent(mx_quantize_dense_kernel<BITS, LAYOUT, LQ_ROUND_HALF_EVEN, LQ_BF16>, g, 128, 0, st, s, src, r, keys, total, numel);
    else if (dt == LQ_F16) launch_dependent(mx_quantize_dense_kernel<BITS, LAYOUT, LQ_ROUND_HALF_EVEN, LQ_F16>, g, 128, 0, st, s, src, r, keys, total, numel);
    else launch_dependent(mx_quantize_dense_kernel<BITS, LAYOUT, LQ_ROUND_HALF_EVEN, LQ_F32>, g, 128, 0, st, s, src, r, keys, total, numel);
    return;
  }
  switch (r.mode) {
    case LQ_ROUND_HALF_UP: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_HALF_UP><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
    case LQ_ROUND_HALF_EVEN: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_HALF_EVEN><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
    case LQ_ROUND_PHILOX_REF: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_PHILOX_REF><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
    case LQ_ROUND_SUPPLIED: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_SUPPLIED><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
    case LQ_ROUND_PHILOX_LAYERED: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_PHILOX_LAYERED><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
    case LQ_ROUND_PHILOX_LAYERED4: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_PHILOX_LAYERED4><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
    default: mx_quantize_kernel<BITS, LAYOUT, LQ_ROUND_SUPPLIED_FIXED><<<grid, block, 0, st>>>(s, src, dt, stride, r, keys, total); break;
  }
}

#define LQ_DISPATCH_BITS_LAYOUT(bits, layout, CALL)                                   \
  do {                                                                                \
    if ((bits) == 8 && (layout) == LQ_MX_LAYOUT_REFERENCE) { CALL(8, LQ_MX_LAYOUT_REFERENCE); } \
    else if ((bits) == 8) { CALL(8, LQ_MX_LAYOUT_PACKED); }                           \
    else if ((layout) == LQ_MX_LAYOUT_REFERENCE) { CALL(4, LQ_MX_LAYOUT_REFERENCE); } \
    else { CALL(4, LQ_MX_LAYOUT_PACKED); }                                            \
  } while (0)

}  // namespace lq

using namespace lq;

LQ_EXPORT int lq_mx_state_update(const lq_mx_update_args* args, void* cuda_stream) {
  LQ_CHECK_ARG(args != nullptr, "lq_mx_state_update: null args");
  const lq_mx_update_args& a = *args;
  if (int rc = validate_state(a.state, "lq_mx_state_update")) return rc;
  if (int rc = validate_rounding(a.rounding, "lq_mx_state_update")) return rc;
  LQ_CHECK_ARG(a.x && a.dt && a.A && a.B && a.C && a.out, "lq_mx_state_update: null operand");
  LQ_CHECK_ARG(valid_dtype(a.x_dtype) && valid_dtype(a.dt_dtype) && valid_dtype(a.A_dtype) && valid_dtype(a.B_dtype) &&
                   valid_dtype(a.C_dtype) && valid_dtype(a.out_dtype),
               "lq_mx_state_update: bad dtype");
  LQ_CHECK_ARG(!a.dt_bias || valid_dtype(a.dt_bias_dtype), "lq_mx_state_update: bad dt_bias dtype");
  LQ_CHECK_ARG(!a.D || valid_dtype(a.D_dtype), "lq_mx_state_update: bad D dtype");
  LQ_CHECK_ARG(!a.z || valid_dtype(a.z_dtype), "lq_mx_state_update: bad z dtype");
  LQ_CHECK_ARG(a.ngroups > 0 && a.state.heads % a.ngroups == 0, "lq_mx_state_update: heads=%d not divisible by ngroups=%d",
               a.state.heads, a.ngroups);
  MxUpdateDerived d;
  d.nblk = a.state.dstate / 16;
  if (d.nblk > 32) return fail(LQ_ERR_UNSUPPORTED, "lq_mx_state_update: dstate=%d > 512 is not implemented", a.state.dstate);
  if (a.state.dim > 4096) return fail(LQ_ERR_UNSUPPORTED, "lq_mx_state_update: dim=%d > 4096 is not implemented", a.state.dim);
  d.lpr_log2 = 0;
  while ((1 << d.lpr_log2) < d.nblk) ++d.lpr_log2;
  d.dt_uniform = (a.dt_stride[2] == 0 && (!a.dt_bias || a.dt_bias_stride[1] == 0)) ? 1 : 0;
  d.a_scalar = (a.A_stride[1] == 0 && a.A_stride[2] == 0) ? 1 : 0;
  d.keys = make_philox_keys(a.rounding.seed);
  {
    // Heads per CTA: as many heads of one B/C group as keeps the grid at >= 4 CTAs per SM (B and C
    // are then fetched, and dt / exp(A dt) evaluated, once for all of them), and shared memory small.
    const int per_group = a.state.heads / a.ngroups;
    const int64_t want_ctas = 4ll * sm_count();
    int hpc = per_group;
    while (hpc > 1 && (static_cast<int64_t>(a.state.batch) * (a.state.heads / hpc) < want_ctas || hpc * a.state.dim > 4096 ||
                       per_group % hpc != 0))
      --hpc;
    d.heads_per_cta = hpc;
  }
  if (a.h_out) LQ_CHECK_ARG(reinterpret_cast<uintptr_t>(a.h_out) % 16 == 0, "lq_mx_state_update: h_out must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
#define LQ_CALL(B_, L_) launch_update_mode<B_, L_>(a, d, st)
  LQ_DISPATCH_BITS_LAYOUT(a.state.format_bits, a.state.layout, LQ_CALL);
#undef LQ_CALL
  LQ_CHECK_CUDA(cudaGetLastError());
  return LQ_OK;
}

LQ_EXPORT int lq_mx_quantize(const lq_mx_state* state, const void* src, int32_t src_dtype, int64_t src_row_stride,
                              const lq_rounding* rounding, void* cuda_stream) {
  LQ_CHECK_ARG(state && src && rounding, "lq_mx_quantize: null argument");
  if (int rc = validate_state(*state, "lq_mx_quantize")) return rc;
  if (int rc = validate_rounding(*rounding, "lq_mx_quantize")) return rc;
  LQ_CHECK_ARG(valid_dtype(src_dtype), "lq_mx_quantize: bad dtype");
  LQ_CHECK_ARG(src_row_stride >= state->dstate, "lq_mx_quantize: src_row_stride=%lld < dstate", (long long)src_row_stride);
  const int64_t total = static_cast<int64_t>(state->batch) * state->heads * state->dim * (state->dstate / 16);
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
#define LQ_CALL(B_, L_) launch_quantize_mode<B_, L_>(*state, src, src_dtype, src_row_stride, *rounding, total, st)
  LQ_DISPATCH_BITS_LAYOUT(state->format_bits, state->layout, LQ_CALL);
#undef LQ_CALL
  LQ_CHECK_CUDA(cudaGetLastError());
  return LQ_OK;
}

LQ_EXPORT int lq_counter_add(uint64_t* counter, uint64_t inc, void* cuda_stream) {
  LQ_CHECK_ARG(counter != nullptr && reinterpret_cast<uintptr_t>(counter) % 8 == 0, "lq_counter_add: counter must be an 8-byte aligned device pointer");
  counter_add_kernel<<<1, 1, 0, static_cast<cudaStream_t>(cuda_stream)>>>(reinterpret_cast<unsigned long long*>(counter), inc);
  LQ_CHECK_CUDA(cudaGetLastError());
  return LQ_OK;
}

LQ_EXPORT int lq_mx_dequantize(const lq_mx_state* state, float* dst, int64_t dst_row_stride, void* cuda_stream) {
  LQ_CHECK_ARG(state && dst, "lq_mx_dequantize: null argument");
  if (int rc = validate_state(*state, "lq_mx_dequantize")) return rc;
  LQ_CHECK_ARG(dst_row_stride >= state->dstate, "lq_mx_dequantize: dst_row_stride < dstate");
  const int64_t total = static_cast<int64_t>(state->batch) * state->heads * state->dim * (state->dstate / 16);
  const int block = 128;
  const int grid = static_cast<int>(std::min<int64_t>((total + block - 1) / block, 1 << 20));
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
#define LQ_CALL(B_, L_) mx_dequantize_kernel<B_, L_><<<grid, block, 0, st>>>(*state, dst, dst_row_stride, total)
  LQ_DISPATCH_BITS_LAYOUT(state->format_bits, state->layout, LQ_CALL);
#undef LQ_CALL
  LQ_CHECK_CUDA(cudaGetLastError());
  return LQ_OK;
}

LQ_EXPORT int lq_mx_convert_layout(const lq_mx_state* src, const lq_mx_state* dst, void* cuda_stream) {
  LQ_CHECK_ARG(src && dst, "lq_mx_convert_layout: null argument");
  if (int rc = validate_state(*src, "lq_mx_convert_layout(src)")) return rc;
  if (int rc = validate_state(*dst, "lq_mx_convert_layout(dst)")) return rc;
  LQ_CHECK_ARG(src->format_bits == dst->format_bits && src->batch == dst->batch && src->heads == dst->heads &&
                   src->dim == dst->dim && src->dstate == dst->dstate,
               "lq_mx_convert_layout: source and destination differ in shape or format");
  const int64_t total = static_cast<int64_t>(src->batch) * src->heads * src->dim * (src->dstate / 16);
  const int block = 128;
  const int grid = static_cast<int>(std::min<int64_t>((total + block - 1) / block, 1 << 20));
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  const int bits = src->format_bits;
#define LQ_CONV(B_, S_, D_) mx_convert_kernel<B_, S_, D_><<<grid, block, 0, st>>>(*src, *dst, total)
  if (bits == 8) {
    if (src->layout == LQ_MX_LAYOUT_REFERENCE && dst->layout == LQ_MX_LAYOUT_PACKED) LQ_CONV(8, LQ_MX_LAYOUT_REFERENCE, LQ_MX_LAYOUT_PACKED);
    else if (src->layout == LQ_MX_LAYOUT_PACKED && dst->layout == LQ_MX_LAYOUT_REFERENCE) LQ_CONV(8, LQ_MX_LAYOUT_PACKED, LQ_MX_LAYOUT_REFERENCE);
    else if (src->layout == LQ_MX_LAYOUT_PACKED) LQ_CONV(8, LQ_MX_LAYOUT_PACKED, LQ_MX_LAYOUT_PACKED);
    else LQ_CONV(8, LQ_MX_LAYOUT_REFERENCE, LQ_MX_LAYOUT_REFERENCE);
  } else {
    if (src->layout == LQ_MX_LAYOUT_REFERENCE && dst->layout == LQ_MX_LAYOUT_PACKED) LQ_CONV(4, LQ_MX_LAYOUT_REFERENCE, LQ_MX_LAYOUT_PACKED);
    else if (src->layout == LQ_MX_LAYOUT_PACKED && dst->layout == LQ_MX_LAYOUT_REFERENCE) LQ_CONV(4, LQ_MX_LAYOUT_PACKED, LQ_MX_LAYOUT_REFERENCE);
    else if (src->layout == LQ_MX_LAYOUT_PACKED) LQ_CONV(4, LQ_MX_LAYOUT_PACKED, LQ_MX_LAYOUT_PACKED);
    else LQ_CONV(4, LQ_MX_LAYOUT_REFERENCE, LQ_MX_LAYOUT_REFERENCE);
  }
#undef LQ_CONV
  LQ_CHECK_CUDA(cudaGetLastError());
  return LQ_OK;
}
