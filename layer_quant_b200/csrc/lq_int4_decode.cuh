// q_len = 1 GQA decode attention over the packed INT4 KV cache: one CTA per (split, kv head, batch), of four warps or, where an SM gets one CTA anyway, of as
// many as an SM holds, each warp on a contiguous part of the CTA's tokens with a ring of its own.
//
// The arithmetic of a 16-token step is that of lq_int4_mma.cuh (S^T = K Q^T and O^T = V^T (P v_scale)^T on mma.sync, the unpacked
// nibbles as A operand in registers); what differs is everything around it.  A warp stages 32 tokens at a time with cp.async and
// synchronises with itself only, so the warps of a CTA drift apart and their unpacking (ALU), exponentials and products overlap, and
// the per-stage work (addresses, waits, issue) is shared by two steps.
// What bounds it: about 320 instructions per 16 tokens, half of them on the integer pipe (73 logic operations and 48 shifts unpack bf16 nibbles; moves and multiplies
// share its cycles) with three warps per scheduler, then HBM.
// Batch 64 x 32768, group 32: 541 -> 468 us (5.74 TB/s); batch 16 x 8191: 51 -> 45 -> 40 us; fp16 query, 200 x 8000, group 128: 461 -> 348 us.
#pragma once

#include "lq_int4_mma.cuh"

namespace lq {
namespace mma {

constexpr int kStageTok = 32, kStagesD = 3;

template <int GS, int NW>
struct WarpStage {
  static constexpr int kG = kD / GS;
  static constexpr int kCodeBytes = kStageTok * 64, kScaleBytes = kStageTok * kG * 4;
  static constexpr int kKc = 0, kVc = kCodeBytes, kKs = 2 * kCodeBytes, kVs = kKs + kScaleBytes;
  static constexpr int kBytes = kVs + kScaleBytes;
  static constexpr int kWarp = kStagesD * kBytes;
  static constexpr int kMergeBytes = NW * 8 * kD * 4;  // [warps][heads][128] floats, later the split factors
  static constexpr int kSmem = (NW * kWarp > kMergeBytes ? NW * kWarp : kMergeBytes) + TileLayout<GS>::kNewBytes;
};

__device__ __forceinline__ void mma_f16_from(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                             float c0, float c1, float c2, float c3) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
// Nibbles as fp16 pairs: those at bits 0..3 of each half exactly (1032 + n under the pattern of 1024, then the offset taken off);
// those at bits 4..7 as 72 + n under the pattern of 64, where bit 4 counts one: no shift.
// Mask and pattern in one instruction, one of them in a register: left to itself the compiler takes two, 32 more per 16 tokens on the logic pipe,
// which bounds the step (fp16 queries, 24 x 3001 with a mask, group 64: 35.2 -> 33.2 us; 16 x 8191, group 128: 45.4 -> 41.3).
__device__ __forceinline__ uint32_t and_xor(uint32_t x, uint32_t mask, uint32_t pattern) {
  uint32_t v;
  asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(v) : "r"(x), "r"(mask), "r"(pattern));
  return v;
}
__device__ __forceinline__ uint32_t nib_pair_f16(uint32_t x) {
  const uint32_t v = and_xor(x, 0x000F000Fu, 0x64086408u);
  const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&v), __float2half2_rn(-1032.0f));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t nib_pair_f16_plus72(uint32_t x) { return and_xor(x, 0x00F000F0u, 0x54805480u); }

enum QueryMode { kQBf16 = 0, kQF16 = 1, kQF32 = 2 };

// QM: a bf16 query is multiplied as it is; an fp16 query with the K codes in fp16; an fp32 query as bf16 hi + lo (two products).
// NW: warps of the CTA, 4, or as many as an SM holds (kWideWarps; the rule and what it gives stand at wide_pays).
template <int R, int QM>
constexpr int kWideWarps = R <= 4 && QM != kQF32 ? 12 : 8;
template <int R, int GS, bool HAS_MASK, int QM, int NW>
__global__ void __launch_bounds__(NW * 32, kWideWarps<R, QM> / NW) int4_decode_warp_kernel(const DecodeParams p) {
  static_assert(R <= 8, "at most eight head columns");
  constexpr int kWarpsM = NW, kThreadsM = NW * 32;
  constexpr bool QSPLIT = QM == kQF32;
  using L = WarpStage<GS, NW>;
  using N = TileLayout<GS>;
  constexpr int G = L::kG;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int s_is_last;
  __shared__ float s_m[kWarpsM][8], s_l[kWarpsM][8];

  const lq_int4_decode_args& a = p.a;
  const lq_int4_cache& c = a.cache;
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;  // mma fragment coordinates: row / column group
  constexpr bool DUP = R <= 4;            // columns 4..7 repeat columns 0..3: hi and lo part of P * v_scale in one n-tile
  constexpr int NT = DUP ? 1 : 2;
  const int hrow = DUP ? (g & 3) : g;
  const bool is_lo = DUP && t >= 2;
  const uint32_t lo_mul = is_lo ? 65536u : 0u, lo_mask = is_lo ? 0xFFFF0000u : 0u;
  uint8_t* const newtile = smem + L::kSmem - N::kNewBytes;
  // Nothing is asked for in L2 ahead of the wait: it took longer than the loads themselves at every size (us with / without: 64 x 600 24.7 / 21.3, 24 x 1000 17.3 / 15.2,
  // 16 x 1000 9.7 / 9.6, 200 x 600 53.2 / 47.2).
  pdl_wait();
  const RunLengths rl = run_lengths(p);
  const bool do_new = a.k_new != nullptr && split == p.splits - 1;
  if (threadIdx.x == 0) s_is_last = 0;
  const int64_t kp_base = b * c.kp_stride[0] + kvh * c.kp_stride[1];
  const int64_t vp_base = b * c.vp_stride[0] + kvh * c.vp_stride[1];
  const int64_t ks_base = b * c.ks_stride[0] + kvh * c.ks_stride[1];
  const int64_t vs_base = b * c.vs_stride[0] + kvh * c.vs_stride[1];

  // this warp's tokens [tok, tok_end): a contiguous run of 16-token steps of the CTA's tiles
  int tok, tok_end;
  {
    const int cta_begin = min(split * rl.tiles_per_split * kTileTok, rl.ctx_len);
    const int cta_end = min(cta_begin + rl.tiles_per_split * kTileTok, rl.ctx_len);
    const unsigned steps = static_cast<unsigned>(cta_end - cta_begin + 15) >> 4;
    const int each = static_cast<int>(steps / NW), more = static_cast<int>(steps % NW);
    tok = cta_begin + 16 * (warp * each + min(warp, more));
    tok_end = min(tok + 16 * (each + (warp < more ? 1 : 0)), cta_end);
  }

  // ---- staging: chunk 32 k + lane of a stage's K codes is row 8 k + lane / 4, 16-byte chunk lane & 3 (V the same); the swizzle does
  // not depend on k.  Scale chunk `lane` of K and of V (the first kScaleBytes / 16 lanes).
  constexpr int kScaleChunks = L::kScaleBytes / 16;
  const uint32_t ring = s2u(smem) + warp * L::kWarp;
  const uint32_t code_dst = ring + swz(lane >> 2, lane & 3);
  const uint8_t* k_src = c.k_packed + kp_base + static_cast<int64_t>(tok) * 64 + lane * 16;
  const uint8_t* v_src = c.v_packed + vp_base + static_cast<int64_t>(tok) * 64 + lane * 16;
  const uint8_t* ks_src = reinterpret_cast<const uint8_t*>(c.k_scale + ks_base + static_cast<int64_t>(tok) * G) + lane * 16;
  const uint8_t* vs_src = reinterpret_cast<const uint8_t*>(c.v_scale + vs_base + static_cast<int64_t>(tok) * G) + lane * 16;
  int ahead = tok_end - tok;      // tokens not yet requested
  uint32_t fill = 0;              // byte offset of the stage to fill next
  auto issue = [&]() {
    if (ahead >= kStageTok) {
#pragma unroll
      for (int k = 0; k < 4; ++k) cp_async16_full(code_dst + fill + L::kKc + k * 512, k_src + k * 512);
#pragma unroll
      for (int k = 0; k < 4; ++k) cp_async16_full(code_dst + fill + L::kVc + k * 512, v_src + k * 512);
      if (kScaleChunks == 32 || lane < kScaleChunks) {
        cp_async16_full(ring + fill + L::kKs + lane * 16, ks_src);
        cp_async16_full(ring + fill + L::kVs + lane * 16, vs_src);
      }
    } else if (ahead > 0) {  // rows past the end are zero-filled; the address of a copy of nothing is the stage's first byte
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = 8 * k + (lane >> 2) < ahead;
        cp_async16(code_dst + fill + L::kKc + k * 512, k_src + (ok ? k * 512 : -lane * 16), ok ? 16u : 0u);
        cp_async16(code_dst + fill + L::kVc + k * 512, v_src + (ok ? k * 512 : -lane * 16), ok ? 16u : 0u);
      }
      if (lane < kScaleChunks) {
        const int left = ahead * G * 4 - lane * 16;
        const uint32_t n = left >= 16 ? 16u : (left > 0 ? static_cast<uint32_t>(left) : 0u);
        cp_async16(ring + fill + L::kKs + lane * 16, ks_src - (n ? 0 : lane * 16), n);
        cp_async16(ring + fill + L::kVs + lane * 16, vs_src - (n ? 0 : lane * 16), n);
      }
    }
    cp_async_commit();
    ahead -= kStageTok;
    k_src += kStageTok * 64;
    v_src += kStageTok * 64;
    ks_src += kStageTok * G * 4;
    vs_src += kStageTok * G * 4;
    fill = fill == (kStagesD - 1) * L::kBytes ? 0u : fill + L::kBytes;
  };
  // start the ring now: the first stages travel while the new row is quantised and the Q fragments are built
#pragma unroll
  for (int i = 0; i < kStagesD - 1; ++i) issue();

  // the new row's values are fetched now and quantised after the Q fragments, so that the two sets of
  // loads are in flight together
  float xnew[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (do_new && warp < 2) {
    const void* src = warp == 0 ? a.k_new : a.v_new;
    const int64_t* ss = warp == 0 ? a.k_new_stride : a.v_new_stride;
#pragma unroll
    for (int i = 0; i < 4; ++i) xnew[i] = load_as_float(src, b * ss[0] + kvh * ss[1] + (lane * 4 + i) * ss[2], a.dtype);
  }
  if (do_new) {
    for (int i = threadIdx.x; i < N::kNewBytes / 16; i += kThreadsM) reinterpret_cast<uint4*>(newtile)[i] = make_uint4(0, 0, 0, 0);
  }

  // ---- Q^T fragments (B operand of S^T), in the k order the K unpack produces ------------------------------
  // chunk i, k-step s (0: nibbles 0,4,1,5; 1: nibbles 2,6,3,7 of this thread's 8-nibble word).  The unpacked K codes carry an offset
  // (136 in bf16; 72 on the odd nibbles in fp16), so an accumulator starts at -offset * (sum of the q that meet it) instead (two
  // mma per accumulator, so no long cancellation); the sum is taken over the values the fragments actually hold.
  uint32_t qa[4][2][2];
  uint32_t ql[QSPLIT ? 4 : 1][2][2];  // lo halves
  float qoff[4];
  auto bf_lo = [](uint32_t v) { return __uint_as_float(v << 16); };
  auto bf_hi = [](uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); };
  auto pair_sum = [&](uint32_t v) {
    if (QM != kQF16) return bf_lo(v) + bf_hi(v);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
    return f.x + f.y;
  };
  // a 16-bit query whose head dims are contiguous and 16-byte aligned arrives as one 128-bit load per
  // chunk (the lane's eight dims 32 i + 8 t .. + 7), anything else as scalar loads
  const bool q_row_valid = hrow < R;
  const int64_t q_row_base = b * a.q_stride[0] + (kvh * R + hrow % R) * a.q_stride[1];
  const bool q_vec = !QSPLIT && a.q_stride[2] == 1 &&
                     ((reinterpret_cast<uintptr_t>(a.q) | (static_cast<uint64_t>(a.q_stride[0]) * 2) | (static_cast<uint64_t>(a.q_stride[1]) * 2)) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float qs = 0.0f, qs_lo = 0.0f;
    uint4 qw = make_uint4(0u, 0u, 0u, 0u);
    if (q_vec && q_row_valid) qw = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.q) + q_row_base + 32 * i + 8 * t);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int d0 = 32 * i + 8 * t + 2 * s;
      uint32_t pa, pb;
      float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
      if (q_vec) {  // (dim d0, d0 + 4) and (d0 + 1, d0 + 5) out of the eight loaded values
        const uint32_t wl = s == 0 ? qw.x : qw.y, wh = s == 0 ? qw.z : qw.w;
        pa = __byte_perm(wl, wh, 0x5410);
        pb = __byte_perm(wl, wh, 0x7632);
      } else {
        if (q_row_valid) {
          q0 = load_as_float(a.q, q_row_base + (d0 + 0) * a.q_stride[2], a.dtype);
          q1 = load_as_float(a.q, q_row_base + (d0 + 4) * a.q_stride[2], a.dtype);
          q2 = load_as_float(a.q, q_row_base + (d0 + 1) * a.q_stride[2], a.dtype);
          q3 = load_as_float(a.q, q_row_base + (d0 + 5) * a.q_stride[2], a.dtype);
        }
        if (QM == kQF16) {
          const __half2 ha = __floats2half2_rn(q0, q1), hb = __floats2half2_rn(q2, q3);  // exact
          pa = *reinterpret_cast<const uint32_t*>(&ha);
          pb = *reinterpret_cast<const uint32_t*>(&hb);
        } else {
          pa = pack_bf16x2(q0, q1);
          pb = pack_bf16x2(q2, q3);
        }
      }
      qa[i][s][0] = pa;  // k = 2t, 2t+1
      qa[i][s][1] = pb;  // k = 2t+8, 2t+9
      qs += QM == kQF16 ? pair_sum(pb) : pair_sum(pa) + pair_sum(pb);
      if (QSPLIT) {
        const uint32_t la = pack_bf16x2(q0 - bf_lo(pa), q1 - bf_hi(pa)), lb = pack_bf16x2(q2 - bf_lo(pb), q3 - bf_hi(pb));
        ql[QSPLIT ? i : 0][s][0] = la;
        ql[QSPLIT ? i : 0][s][1] = lb;
        qs_lo += pair_sum(la) + pair_sum(lb);
      }
    }
    qs += qs_lo;
    qs += __shfl_xor_sync(0xFFFFFFFFu, qs, 1);  // the chunk's 32 dims live in the four lanes of row g
    qs += __shfl_xor_sync(0xFFFFFFFFu, qs, 2);
    qoff[i] = (QM == kQF16 ? -72.0f : -136.0f) * qs;
  }
  // accumulator start values of this lane's two columns (the sums live in the lanes of row g = column)
  float qstart[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    qstart[i][0] = __shfl_sync(0xFFFFFFFFu, qoff[i], 8 * t);      // lane (g = 2t, t = 0)
    qstart[i][1] = __shfl_sync(0xFFFFFFFFu, qoff[i], 8 * t + 4);  // lane (g = 2t + 1, t = 0)
  }
  // ---- fused append: quantise the new K / V row, write it to the cache and into a 16-row tile -------
  if (do_new) {
    __syncthreads();  // the tile of the new row is zeroed
    if (warp < 2) {
      float amax = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) amax = fmaxf(amax, fabsf(xnew[i]));
#pragma unroll
      for (int o = GS / 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
      const float scale = int4_scale(amax);
      uint32_t half = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) half |= int4_code(xnew[i], scale) << (4 * i);
      const int pos = rl.seq_len - 1;
      uint8_t* gcodes = (warp == 0 ? c.k_packed + kp_base + static_cast<int64_t>(pos) * c.kp_stride[2]
                                   : c.v_packed + vp_base + static_cast<int64_t>(pos) * c.vp_stride[2]);
      reinterpret_cast<uint16_t*>(gcodes)[lane] = static_cast<uint16_t>(half);
      reinterpret_cast<uint16_t*>(newtile + (warp == 0 ? N::kNewKc : N::kNewVc))[lane] = static_cast<uint16_t>(half);  // row 0: no swizzle
      if ((lane * 4) % GS == 0) {
        float* gsc = (warp == 0 ? c.k_scale + ks_base + static_cast<int64_t>(pos) * c.ks_stride[2]
                                : c.v_scale + vs_base + static_cast<int64_t>(pos) * c.vs_stride[2]);
        gsc[lane * 4 / GS] = scale;
        reinterpret_cast<float*>(newtile + (warp == 0 ? N::kNewKs : N::kNewVs))[lane * 4 / GS] = scale;
      }
    }
  }

  const float scale_sm = 1.4426950408889634f / sqrtf(static_cast<float>(kD));
  // O^T accumulators: m-tile (chunk i, half sp) has row g = dim 32 i + 4 g + 2 sp and row g + 8 = that
  // dim + 1; columns 2t, 2t+1 are heads (DUP: head c & 3, hi part for c < 4, lo part for c >= 4).
  float oacc[4][2][NT][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int sp = 0; sp < 2; ++sp)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) oacc[i][sp][nt][e] = 0.0f;
  const int col_head0 = DUP ? ((2 * t) & 3) : 2 * t;  // head column of accumulator column 2t (column 2t+1: the next one)
  float m_run[2] = {kNegBigM, kNegBigM}, l_run[2] = {0.0f, 0.0f};  // this lane's two columns (l: this lane's share)

  // Offsets inside 16 rows: ldmatrix row addresses for K (second half: + 512) and V (two chunk pairs), scale rows of
  // the tokens this thread owns in the S^T fragments (rows g and g + 8)
  const uint32_t koff = swz(lane & 7, lane >> 3);
  uint32_t voff[2];
#pragma unroll
  for (int cp = 0; cp < 2; ++cp) voff[cp] = swz(8 * ((lane >> 3) & 1) + (lane & 7), 2 * cp + (lane >> 4));
  const uint32_t soff = g * G * 4;

  // One 16-token step.  kc / vc: shared-memory addresses of 16 rows of codes, ksc / vsc: of their scales.
  // FULL: all 16 rows hold tokens; otherwise the first `valid` do, and the rest were zero-filled.
  auto step16 = [&](auto full_tag, uint32_t kc, uint32_t vc, const uint8_t* ksc, const uint8_t* vsc, int valid, const float (&bias)[2]) {
    constexpr bool FULL = decltype(full_tag)::value;
    float sacc[4][4];
    {
      uint32_t kr0[4], kr1[4];
      ldmatrix_x4(kr0, kc + koff);
      ldmatrix_x4(kr1, kc + koff + 512);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t w0 = kr0[i], w1 = kr1[i];
        const float c0 = qstart[i][0], c1 = qstart[i][1];
        if (QM == kQF16) {
          const uint32_t y0 = w0 >> 8, y1 = w1 >> 8;
          mma_f16_from(sacc[i], nib_pair_f16(w0), nib_pair_f16(w1), nib_pair_f16_plus72(w0), nib_pair_f16_plus72(w1), qa[i][0][0], qa[i][0][1], c0,
                       c1, c0, c1);
          mma_f16_from(sacc[i], nib_pair_f16(y0), nib_pair_f16(y1), nib_pair_f16_plus72(y0), nib_pair_f16_plus72(y1), qa[i][1][0], qa[i][1][1],
                       sacc[i][0], sacc[i][1], sacc[i][2], sacc[i][3]);
        } else {
          const uint32_t a0 = nib_pair_biased(w0), a1 = nib_pair_biased(w1), a2 = nib_pair_biased(w0 >> 4), a3 = nib_pair_biased(w1 >> 4);
          const uint32_t b0 = nib_pair_biased(w0 >> 8), b1 = nib_pair_biased(w1 >> 8), b2 = nib_pair_biased(w0 >> 12), b3 = nib_pair_biased(w1 >> 12);
          mma_bf16_from(sacc[i], a0, a1, a2, a3, qa[i][0][0], qa[i][0][1], c0, c1, c0, c1);
          if (QSPLIT) mma_bf16(sacc[i], a0, a1, a2, a3, ql[QSPLIT ? i : 0][0][0], ql[QSPLIT ? i : 0][0][1]);
          mma_bf16(sacc[i], b0, b1, b2, b3, qa[i][1][0], qa[i][1][1]);
          if (QSPLIT) mma_bf16(sacc[i], b0, b1, b2, b3, ql[QSPLIT ? i : 0][1][0], ql[QSPLIT ? i : 0][1][1]);
        }
      }
    }
    // scores of tokens g (r = 0) and g + 8 (r = 1) for this lane's two columns
    float sv[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float sc[G];
      load_scales(ksc + soff + r * (8 * G * 4), sc);
      // both columns of the token at once: packed fp32x2 FMA / MUL (sm_100), same rounding per component
      float2 sum2 = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float k = sc[(32 * i) / GS];
        sum2 = __ffma2_rn(make_float2(k, k), make_float2(sacc[i][2 * r], sacc[i][2 * r + 1]), sum2);
      }
      sum2 = __fmul2_rn(sum2, make_float2(scale_sm, scale_sm));
      if (HAS_MASK) sum2 = make_float2(sum2.x + bias[r], sum2.y + bias[r]);
      const bool ok = FULL || g + 8 * r < valid;
      sv[r][0] = ok ? sum2.x : -INFINITY;
      sv[r][1] = ok ? sum2.y : -INFINITY;
    }
    // online softmax per column; the running max of a column is shared by the eight lanes that hold it.
    // Columns without a head (zero Q) run along harmlessly and are never read.
    const float smax0 = fmaxf(sv[0][0], sv[1][0]), smax1 = fmaxf(sv[0][1], sv[1][1]);
    if (__any_sync(0xFFFFFFFFu, smax0 > m_run[0] + kSlackM || smax1 > m_run[1] + kSlackM)) {
      float rm0 = smax0, rm1 = smax1;
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        rm0 = fmaxf(rm0, __shfl_xor_sync(0xFFFFFFFFu, rm0, o));
        rm1 = fmaxf(rm1, __shfl_xor_sync(0xFFFFFFFFu, rm1, o));
      }
      const float n0 = fmaxf(m_run[0], rm0), n1 = fmaxf(m_run[1], rm1);
      const float alpha0 = fast_exp2(m_run[0] - n0), alpha1 = fast_exp2(m_run[1] - n1);
      l_run[0] *= alpha0;
      l_run[1] *= alpha1;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int sp = 0; sp < 2; ++sp)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            oacc[i][sp][nt][0] *= alpha0;
            oacc[i][sp][nt][1] *= alpha1;
            oacc[i][sp][nt][2] *= alpha0;
            oacc[i][sp][nt][3] *= alpha1;
          }
      m_run[0] = n0;
      m_run[1] = n1;
    }
    float pv[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        pv[r][cc] = fast_exp2(sv[r][cc] - m_run[cc]);  // 0 for masked / padded tokens
        l_run[cc] += pv[r][cc];
      }
    // B operand of O^T: (P * v_scale)^T per scale group, k = the tokens 2t, 2t+1 (+8), n = column g.  What
    // this lane has is the other way round (token g / g + 8, columns 2t, 2t+1), so each packed pair goes
    // through movmatrix.  A lane of columns 0..3 keeps the bf16 rounding of the product, a lane of
    // columns 4..7 the bf16 rounding of what that left over (one formula: the part taken off is masked
    // to zero on the hi lanes).
    uint32_t pb[G][2][NT];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float vs[G];
      load_scales(vsc + soff + r * (8 * G * 4), vs);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const float2 pp = __fmul2_rn(make_float2(pv[r][0], pv[r][1]), make_float2(vs[q], vs[q]));
        const uint32_t hi = pack_bf16x2(pp.x, pp.y);
        if (DUP) {
          const float2 lo = __ffma2_rn(make_float2(__uint_as_float(hi * lo_mul), __uint_as_float(hi & lo_mask)), make_float2(-1.0f, -1.0f), pp);
          pb[q][r][0] = movmatrix_trans(pack_bf16x2(lo.x, lo.y));
        } else {
          const float2 lo = __ffma2_rn(make_float2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xFFFF0000u)), make_float2(-1.0f, -1.0f), pp);
          pb[q][r][0] = movmatrix_trans(hi);
          pb[q][r][NT - 1] = movmatrix_trans(pack_bf16x2(lo.x, lo.y));
        }
      }
    }
    // O^T += V^T (P * v_scale)^T, chunk by chunk: the unpacked codes are the A operand
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      uint32_t vr[4];
      ldmatrix_x4_trans(vr, vc + voff[cp]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = 2 * cp + h;
        const int q = (32 * i) / GS;
        const uint32_t w0 = vr[2 * h], w1 = vr[2 * h + 1];
#pragma unroll
        for (int sp = 0; sp < 2; ++sp) {
          const uint32_t a0 = nib_pair_to_bf16x2(w0 >> (8 * sp)), a1 = nib_pair_to_bf16x2(w0 >> (8 * sp + 4));
          const uint32_t a2 = nib_pair_to_bf16x2(w1 >> (8 * sp)), a3 = nib_pair_to_bf16x2(w1 >> (8 * sp + 4));
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_bf16(oacc[i][sp][nt], a0, a1, a2, a3, pb[q][0][nt], pb[q][1][nt]);
        }
      }
    }
  };

  // ---- main loop -------------------------------------------------------------------------------------------
  // The biases of a stage's tokens (rows g and g + 8 of its two steps) are fetched a stage ahead: a mask read where it is used
  // would put a global load into every step.
  uint2 raw_next[2][2];
  auto fetch_mask = [&](int first) {
#pragma unroll
    for (int st = 0; st < 2; ++st)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int n = first + 16 * st + 8 * r + g;
        if (n < min(tok_end, a.mask_k_len)) raw_next[st][r] = mask_load(a, b, n);
      }
  };
  if (HAS_MASK) fetch_mask(tok);
  uint32_t cur = 0;
#pragma unroll 1
  while (tok < tok_end) {
    cp_async_wait<kStagesD - 2>();
    __syncwarp();  // the stage has landed for the whole warp, and the whole warp is done with the one before
    issue();
    float bias[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
    if (HAS_MASK) {
#pragma unroll
      for (int st = 0; st < 2; ++st)
#pragma unroll
        for (int r = 0; r < 2; ++r) bias[st][r] = tok + 16 * st + 8 * r + g < a.mask_k_len ? mask_value(a, raw_next[st][r]) : -INFINITY;
      fetch_mask(tok + kStageTok);
    }
    const uint8_t* const stage = smem + warp * L::kWarp + cur;
    const uint32_t sb = ring + cur;
    if (tok_end - tok >= kStageTok) {
#pragma unroll
      for (int st = 0; st < 2; ++st)
        step16(std::true_type{}, sb + L::kKc + st * 1024, sb + L::kVc + st * 1024, stage + L::kKs + st * (16 * G * 4),
               stage + L::kVs + st * (16 * G * 4), 16, bias[st]);
    } else {
#pragma unroll 1
      for (int st = 0; st < 2 && tok + 16 * st < tok_end; ++st) {
        const float bs[2] = {st ? bias[1][0] : bias[0][0], st ? bias[1][1] : bias[0][1]};
        step16(std::false_type{}, sb + L::kKc + st * 1024, sb + L::kVc + st * 1024, stage + L::kKs + st * (16 * G * 4),
               stage + L::kVs + st * (16 * G * 4), tok_end - tok - 16 * st, bs);
      }
    }
    tok += kStageTok;
    cur = cur == (kStagesD - 1) * L::kBytes ? 0u : cur + L::kBytes;
  }
  cp_async_wait<0>();
  __syncthreads();
  if (do_new && warp == 0) {
    const uint32_t nb = s2u(newtile);
    const float bs[2] = {HAS_MASK ? mask_bias(a, b, rl.seq_len - 1) : 0.0f, 0.0f};
    step16(std::false_type{}, nb + N::kNewKc, nb + N::kNewVc, newtile + N::kNewKs, newtile + N::kNewVs, 1, bs);
  }

  // ---- merge the warps -------------------------------------------------------------------------------------
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {  // a column's denominator: over the eight lanes (token rows) that share it
    l_run[0] += __shfl_xor_sync(0xFFFFFFFFu, l_run[0], o);
    l_run[1] += __shfl_xor_sync(0xFFFFFFFFu, l_run[1], o);
  }
  float* s_acc = reinterpret_cast<float*>(smem);  // [warps][R][128], reuses the rings
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int sp = 0; sp < 2; ++sp)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float v;
        if (DUP) {
          v = oacc[i][sp][0][e];
          v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);  // hi columns (t < 2) + lo columns (t >= 2) of the same heads
        } else {
          v = oacc[i][sp][0][e] + oacc[i][sp][NT - 1][e];
        }
        const int head = col_head0 + (e & 1);
        const int dim = 32 * i + 4 * g + 2 * sp + (e >> 1);
        if ((!DUP || t < 2) && head < R) s_acc[(warp * R + head) * kD + dim] = v;
      }
  if (g == 0 && (!DUP || t < 2)) {
#pragma unroll
    for (int cc = 0; cc < 2; ++cc)
      if (col_head0 + cc < R) {
        s_m[warp][col_head0 + cc] = m_run[cc];
        s_l[warp][col_head0 + cc] = l_run[cc];
      }
  }
  __syncthreads();
  const int hq0 = kvh * R;
  for (int o = threadIdx.x; o < R * kD; o += kThreadsM) {
    const int r = o / kD, d = o - r * kD;
    float M = kNegBigM;
#pragma unroll
    for (int w = 0; w < kWarpsM; ++w) M = fmaxf(M, s_m[w][r]);
    float Lsum = 0.0f, O = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarpsM; ++w) {
      const float fct = exp2f(s_m[w][r] - M);
      Lsum = fmaf(s_l[w][r], fct, Lsum);
      O = fmaf(s_acc[(w * R + r) * kD + d], fct, O);
    }
    if (p.splits == 1) {
      store_from_float(a.out, b * a.out_stride[0] + (hq0 + r) * a.out_stride[1] + d * a.out_stride[2], a.dtype, O / Lsum);
    } else {
      const int64_t slot = (static_cast<int64_t>(b) * a.q_heads + hq0 + r) * p.splits + split;
      p.part_acc[slot * kD + d] = O;
      if (d == 0) {
        p.part_ml[slot * 2] = M;
        p.part_ml[slot * 2 + 1] = Lsum;
      }
    }
  }
  if (p.splits == 1) return;

  // Ticket: the CTA that completes the set merges the splits.  No CTA waits for another.
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int ticket = atomicAdd(&p.counters[b * c.kv_heads + kvh], 1);
    s_is_last = (ticket == p.splits - 1) ? 1 : 0;
  }
  __syncthreads();
  if (!s_is_last) return;
  __threadfence();
  // (1) one warp per head: the maximum over the splits, each split's factor (to shared memory) and the
  // denominator; (2) one thread per output: the weighted sum, its loads independent of one another.
  float* s_f = reinterpret_cast<float*>(smem);  // [R][kMaxSplitsM], reuses the rings
  float* s_den = s_f + R * kMaxSplitsM;         // [R]
  for (int r = warp; r < R; r += kWarpsM) {
    const float* ml = p.part_ml + (static_cast<int64_t>(b) * a.q_heads + hq0 + r) * p.splits * 2;
    float M = kNegBigM;
    for (int s = lane; s < p.splits; s += 32) M = fmaxf(M, __ldcg(ml + 2 * s));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, o));
    float den = 0.0f;
    for (int s = lane; s < p.splits; s += 32) {
      const float fct = exp2f(__ldcg(ml + 2 * s) - M);
      s_f[r * kMaxSplitsM + s] = fct;
      den = fmaf(__ldcg(ml + 2 * s + 1), fct, den);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xFFFFFFFFu, den, o);
    if (lane == 0) s_den[r] = den;
  }
  __syncthreads();
  // four outputs per thread: the splits' partial results arrive as independent 128-bit loads, eight in flight per thread
  for (int o = threadIdx.x; o < R * (kD / 4); o += kThreadsM) {
    const int r = o / (kD / 4), d = (o - r * (kD / 4)) * 4;
    const float4* acc = reinterpret_cast<const float4*>(p.part_acc + (static_cast<int64_t>(b) * a.q_heads + hq0 + r) * p.splits * kD + d);
    float4 O = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
    for (int s = 0; s < p.splits; ++s) {
      const float4 v = __ldcg(acc + static_cast<int64_t>(s) * (kD / 4));
      const float f = s_f[r * kMaxSplitsM + s];
      O.x = fmaf(v.x, f, O.x); O.y = fmaf(v.y, f, O.y); O.z = fmaf(v.z, f, O.z); O.w = fmaf(v.w, f, O.w);
    }
    const float den = s_den[r];
    const int64_t ob = b * a.out_stride[0] + (hq0 + r) * a.out_stride[1] + d * a.out_stride[2];
    store_from_float(a.out, ob, a.dtype, O.x / den);
    store_from_float(a.out, ob + a.out_stride[2], a.dtype, O.y / den);
    store_from_float(a.out, ob + 2 * a.out_stride[2], a.dtype, O.z / den);
    store_from_float(a.out, ob + 3 * a.out_stride[2], a.dtype, O.w / den);
  }
  if (threadIdx.x == 0) p.counters[b * c.kv_heads + kvh] = 0;  // ready for the next launch
}

}  // namespace mma
}  // namespace lq
