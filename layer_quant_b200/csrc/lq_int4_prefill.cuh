// Causal attention of many query positions over the packed INT4 KV cache on the 5th-generation tensor cores.  sm_100a.
//
// One CTA = 256 (position, query head) rows of one (batch, kv head): the query heads that share a kv head are rows of the
// same tile, so a cache tile is unpacked once for 256 / R positions.  Thirteen warps:
//   0 .. 7    softmax, two groups of 128 rows, one row per thread (= one TMEM lane)
//   8 .. 11   unpack 64-token tiles of K and V from global memory to fp16 in shared memory, two stages each
//   12        issues the tcgen05.mma of both groups: O += P V of a tile, then S of the group's next tile into the columns
//             that P has just been read from (the tensor pipe takes one thread's products in order)
// Registers: launched with 128 a thread; the softmax groups raise theirs to 168, the other two groups go down to 88.
// TMEM (all 512 columns, so addresses start at 0; 256 per group): O 128, Q 64 (fp16, A operand), S 64; P replaces S (A operand).
//
// Precision.  A dequantised value n * scale (n in [-8, 7]) is held as two fp16 numbers: the leading 8 bits of the scale
// times n, exact in fp16, and the rest of the scale times n, rounded to fp16: 2^-20 relative in all.  P is split
// the same way: 2^-22 of a weight or 2^-35 of the row's largest, whichever is more.  (The mma.sync kernel keeps 2^-17 of every
// weight.  The absolute part adds up to less than that over 2^17 tokens.)  Q is exact in fp16 for 16-bit queries.
// S = Q Khi + Q Klo, O = Phi Vhi + Plo Vhi + Phi Vlo: five products per tile pair, all in fp32 accumulators.
// Token factors (FACTORS, groups of 128, where a token has one scale): the mantissa of the scale goes to the softmax, which multiplies the scores (K) and
// the weights after their sum is taken (V) by it in fp32; the operands are then a code times a power of two, exact in fp16, and need no lo part: three
// products per tile pair in place of five.  The error against 64 bits goes down with the lo parts: fp16 outputs that are
// not the correctly rounded value 1.08 % -> 0.27 % of 2 x 700 tokens, 3.9 -> 1.5 % of 2 x 500 behind 3000, 8.1 -> 3.6 % of 1 x 300 behind 8000.  (Groups of 64 could leave out one product of five, Phi Vlo and Q Klo of the first group.
// Dropped: it pays only in rows of long launches, and a rule on the launch's size made a sequence's bits depend on what shares its launch.)
// Range.  Powers of two are taken out of every row of Q and of the K and V scales of every 16 tokens, so the
// fp16 operands sit at the top of their range; the exponents come back for free, in the factor and the offset of the
// exp2 argument.  With p' = 2^(s + Ev - m) the V exponent Ev is part of the running maximum m.
// Sixteen tokens whose largest scales lie more than 2^kSpread apart or are not all finite ("wide") get an exponent each, applied in a pass
// of its own over the tile's scores: a very large K or V changes nothing for the rows before it.  (With every tile wide 8 x 1024
// tokens take 400 us instead of 161.)  An infinite or NaN scale is
// stored as zero; the rows that attend to it get a NaN score (K) or NaN in the 32 dims (V).
// What remains relative to the largest: inside a token the group scales below 2^-15 of its largest lose bits, and a weight times
// V counts with the row's largest (first item), whichever group that is in.
//
// What bounds it: the chain of a softmax group.  Per 256 x 64 tile the five products take 2620 tensor cycles (5/2 of a bf16 attention), shared memory
// moves 230 KB (1800 cycles, which is why Q is an operand in TMEM) and the exp2 take 1024; a tile takes 4230 cycles in 2 x 2000 tokens behind 6001, starts and
// ends of blocks included, and with token factors, 1570 tensor cycles, still 3630.  No pipe is full: within a
// softmax group S, softmax, P, the products with V and the next S follow one another (P replaces S), and two groups fill one another's
// gaps only in part (tensor pipe active in 53 % of the cycles at 8 x 1024).  In long rows of launches the board's power limit comes on top: five products at
// 1243 TFLOP/s (of measured 1425 sustained) run at 1695 MHz, 954 us in place of 844 for a few launches on a cool board; three products hold 1942 MHz, 715 us
// and 710.  Other schedules of the five, such as a third score buffer for the two groups, took less cycles per tile (3650) at a clock lower by as much.
#pragma once

#include "lq_common.cuh"

namespace lq {
namespace prefill {

constexpr int kTok = 64;                      // tokens per tile
constexpr int kGroupRows = 128;               // rows of a softmax group
constexpr int kCtaRows = 2 * kGroupRows;
constexpr int kThreads = 512;                 // four warp groups; warps 13 .. 15 only fill the last one
constexpr int kPart = kTok * 128 * 2;         // 16 KB: fp16 [64 tokens][128 dims], as two 128-byte-swizzled halves of 64 dims
constexpr int kStageBytes = 2 * kPart;        // hi and lo part
constexpr int kSmemBytes = 4 * kStageBytes + 1024;  // K stages 0, 1, V stages 0, 1; alignment of the swizzle atoms
constexpr uint32_t kColO = 0, kColQ = 128, kColS = 192, kColsPerGroup = 256;
constexpr int kSpread = 8;                    // binades that the tokens of 16 may lie apart under one exponent
constexpr float kScaleFloor = 1.0e-8f;        // of the codec
// The running maximum is raised when a score exceeds it by more than kSlack (log2 units), and weights are held times 2^kLift: what
// fp16 cannot hold is the absolute 2^-24, so the top of its range has to be used.  2^(kSlack + kLift) must stay below 65504.  A wider slack
// raises the maximum less often and leaves less lift: with 8 and 0 weights below 2^-25 of the largest were lost altogether, at 969 us
// against 977 for 2 x 2000 tokens behind 6001.
// With token factors (below 2) on the weights the slack is a quarter less: 2^15.75.
constexpr float kLift = 11.0f;
template <bool FACTORS>
constexpr float kSlack = FACTORS ? 3.75f : 4.0f;
// A score and the maximum part in one FMA, so the rounding of the maximum is in the difference; beyond scores of 2^24 that would
// overflow P.  Queries below kLargeQ and K scales below kLargeK (values below 8 kLargeK) keep scores below 2^21.3; larger ones are rounded
// before the difference is taken, in the pass that wide tiles take.
constexpr float kLargeQ = 512.0f, kLargeK = 32.0f;

struct Params {
  lq_int4_prefill_args a;
  int32_t ratio_log2;   // query heads per kv head
  int32_t gs_log2;      // group size
  int32_t nqb;          // row blocks per (batch, kv head)
  int32_t kv_len;       // rows of the cache that hold tokens: first_len + q_len - 1
  int32_t whole;        // entries of the work list that are whole row blocks; the rest are halves of one softmax group each
  int32_t entries;
};

// An entry of the work list.  Heaviest row blocks first: a block's work grows with its last position.
struct Block {
  int b, kvh, pos0, groups, ntiles;
};
__device__ __forceinline__ Block block_at(const Params& p, int i) {
  const int bh = p.a.cache.batch * p.a.cache.kv_heads;
  int rows = kCtaRows >> p.ratio_log2, first = 0;
  if (i >= p.whole) {
    rows >>= 1;
    first = (i - p.whole) & 1 ? rows : 0;
    i = p.whole + ((i - p.whole) >> 1);
  }
  const int qb = p.nqb - 1 - i / bh, rest = i % bh;
  Block k;
  k.b = rest / p.a.cache.kv_heads;
  k.kvh = rest % p.a.cache.kv_heads;
  k.pos0 = qb * (kCtaRows >> p.ratio_log2) + first;
  k.groups = rows == (kCtaRows >> p.ratio_log2) && k.pos0 + (rows >> 1) < p.a.q_len ? 2 : 1;  // softmax groups with a position of their own
  k.ntiles = (p.a.first_len + min(k.pos0 + rows - 1, p.a.q_len - 1) + kTok - 1) / kTok;
  return k;
}
// Round r of this CTA: the list is dealt forwards and backwards in turn, so that long and short blocks even out
__device__ __forceinline__ int entry_of(int r) {
  return r * static_cast<int>(gridDim.x) + static_cast<int>(r & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}

// ---- tcgen05 ---------------------------------------------------------------------------------------------------------
#define LQ_R8(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
#define LQ_I8(r, o) "r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7])

// columns of this warp's 32 lanes; the wait is part of the statement, so no use can move before it
__device__ __forceinline__ void tmem_load16(uint32_t (&r)[16], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : LQ_R8(r, 0), LQ_R8(r, 8)
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_load32(uint32_t (&r)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\ttcgen05.wait::ld.sync.aligned;"
      : LQ_R8(r, 0), LQ_R8(r, 8), LQ_R8(r, 16), LQ_R8(r, 24)
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_load64(uint32_t (&r)[64], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,"
      "%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n\ttcgen05.wait::ld.sync.aligned;"
      : LQ_R8(r, 0), LQ_R8(r, 8), LQ_R8(r, 16), LQ_R8(r, 24), LQ_R8(r, 32), LQ_R8(r, 40), LQ_R8(r, 48), LQ_R8(r, 56)
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_store32(uint32_t addr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::LQ_I8(r, 0), LQ_I8(r, 8), LQ_I8(r, 16), LQ_I8(r, 24), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_store16(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::LQ_I8(r, 0), LQ_I8(r, 8), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_store8(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::LQ_I8(r, 0), "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One thread of a converged warp.  The compiler knows that the branch on it is taken by one thread and keeps the operands of the
// products in uniform registers: 16 cycles of issue per product, where a branch on the lane index costs 54 to 64, longer
// than a product of 64 columns runs (32).
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred q;\n\t.reg .b32 x;\n\telect.sync x|q, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r));
  return r != 0;
}
// D[128 x N] (+)= A B, A from TMEM, B from shared memory, fp16 in, fp32 accumulate
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate ? 1u : 0u)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// fp16 inputs, fp32 accumulators, M = 128; K tile: N = 64 tokens, dims contiguous; V tile: N = 128 dims, dims contiguous (N-major)
constexpr uint32_t kIdescS = (1u << 4) | ((64u / 8) << 17) | ((128u / 16) << 24);
constexpr uint32_t kIdescO = (1u << 4) | (1u << 16) | ((128u / 8) << 17) | ((128u / 16) << 24);
// Shared-memory matrix descriptor, 128-byte swizzle.  Stride offset 1024: the next eight rows of 128 bytes; lbo: the next
// 64 dims of an N-major tile.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo) {
  return static_cast<uint64_t>((addr & 0x3FFFF) >> 4) | (static_cast<uint64_t>(lbo >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

struct Shared {
  // Few barriers: the thread that issues products runs only a few of them ahead of the tensor pipe, so every wait and commit of
  // its loop can cost tensor time.  Unit j of the unpacking warps is V of tile j and K of tile j + 1, what the products of
  // iteration j read; s_done of a tile also says that all products before it are done, O of the tile before among them.
  // The tiles of a CTA's blocks are counted through, and K of the next block's first tile is part of the last unit of a block.
  uint64_t k_first, full[2], empty[2], s_done[2], p_ready[2], q_ready[2];
  // Per 16 tokens: 2^Ek, Ev and 2^-Ev of the tile, four tiles deep (they are written a unit ahead of V)
  float k_factor[5][4], v_exp[5][4], v_inv[5][4];  // slot 4: 1, 0, 0
  alignas(16) float k_lead[4][kTok], v_lead[4][kTok];  // token factors, where there are any
  // A byte per 16 tokens, bit 0: they are wide, bit 1: large K scales.  Then for wide ones the same per token (k_factor NaN: the
  // scale is not finite), and the 32-dim chunks of V whose scale is not finite, a bit each
  uint32_t wide[4];
  float k_factor_tok[4][kTok], v_exp_tok[4][kTok], v_inv_tok[4][kTok];
  uint8_t v_bad_tok[4][kTok];
  uint32_t tmem;
};

// Polls with a limit; a wait that runs out is recorded in the device status word.  The result is the same for the whole warp.
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity) {
  bool done = false;
  for (uint32_t i = 0; i < kWaitLimit && !done; ++i) done = mbar_try_wait(bar, parity);
  if (__all_sync(0xFFFFFFFFu, done)) return true;
  atomicOr(&g_int4_device_status, 1);
  return false;
}

__device__ __forceinline__ float pow2_of(int e) { return __uint_as_float(static_cast<uint32_t>(e + 127) << 23); }
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// ---- unpacking -------------------------------------------------------------------------------------------------------
// One 32-bit word (8 nibbles) -> four fp16 pairs in the order (0,4) (1,5) (2,6) (3,7), exact.  The dims of K, Q and V are
// all kept in this order; the output is put right when it is stored.  (x & M) ^ K lays a nibble with its top bit
// flipped (n + 8) under the fp16 pattern of 1024: at bit 0 it counts ones, at bit 4 sixteens.
__device__ __forceinline__ void unpack8(uint32_t x, __half2 (&n)[4]) {
  const uint32_t y = x >> 8;
  const uint32_t b0 = (x & 0x000F000Fu) ^ 0x64086408u, b1 = (x & 0x00F000F0u) ^ 0x64806480u;
  const uint32_t b2 = (y & 0x000F000Fu) ^ 0x64086408u, b3 = (y & 0x00F000F0u) ^ 0x64806480u;
  const __half2 off = __float2half2_rn(-1032.0f), sixteenth = __float2half2_rn(0.0625f), off16 = __float2half2_rn(-72.0f);
  n[0] = __hadd2(*reinterpret_cast<const __half2*>(&b0), off);
  n[1] = __hfma2(*reinterpret_cast<const __half2*>(&b1), sixteenth, off16);
  n[2] = __hadd2(*reinterpret_cast<const __half2*>(&b2), off);
  n[3] = __hfma2(*reinterpret_cast<const __half2*>(&b3), sixteenth, off16);
}

// The exponent that brings a scale (its bits) to [2^11, 2^12): n * scale then stays below 2^15
__device__ __forceinline__ int exponent_of(uint32_t bits) {
  const int field = static_cast<int>(bits >> 23);
  return field == 0 ? 0 : max(field - 127 - 11, -110);
}
// The scales of a warp's 16 tokens, two tokens of one chunk per lane (the chunks eight lanes apart): one exponent, that of the largest, or
// where they are wide one per token.  large: of K (kLargeK).  bad: a ballot of the scales that are not finite, per token of the lane; these become 0.
struct Exponents {
  int e[2];
  uint32_t bad[2];
  bool wide, large;
};
__device__ __forceinline__ Exponents exponents_of(float (&sc)[2]) {
  Exponents r;
  const uint32_t b[2] = {__float_as_uint(sc[0]), __float_as_uint(sc[1])};  // a negative scale counts as out of range here; its tokens are wide
  const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, max(b[0], b[1]));
  r.e[0] = r.e[1] = exponent_of(hi);
  r.bad[0] = r.bad[1] = 0u;
  r.large = hi >= __float_as_uint(kLargeK);
  const uint32_t least = min(b[0] - 1, b[1] - 1);  // 0 (a row without a token) does not count
  r.wide = false;
  if (__any_sync(0xFFFFFFFFu, hi >= 0x7F800000u || (hi >> 23) > (least >> 23) + kSpread)) {
    // some scale is small: are there tokens whose largest is?  (A group beside larger ones of its token has no use for an exponent of the
    // token's own, nor has a token at the codec's floor, whose values are below 7.5e-8 and usually 0.)
    uint32_t m[2];
    bool out = false;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const bool finite = (b[i] & 0x7FFFFFFFu) < 0x7F800000u;
      r.bad[i] = __ballot_sync(0xFFFFFFFFu, !finite);
      if (!finite) sc[i] = 0.0f;
      m[i] = finite ? b[i] & 0x7FFFFFFFu : 0u;
      m[i] = max(m[i], __shfl_xor_sync(0xFFFFFFFFu, m[i], 8));
      m[i] = max(m[i], __shfl_xor_sync(0xFFFFFFFFu, m[i], 16));
      out |= !finite || (m[i] > __float_as_uint(kScaleFloor) && (hi >> 23) > (m[i] >> 23) + kSpread);
    }
    r.wide = __any_sync(0xFFFFFFFFu, out);
    if (r.wide) {
      r.e[0] = exponent_of(m[0]);
      r.e[1] = exponent_of(m[1]);
    }
  }
  return r;
}

// The token factor of a scale (its exponent taken out): its mantissa, so that the rest is a power of two.  The sign stays with the power: the codec
// writes positive scales, a caller's own cache may hold others
__device__ __forceinline__ float lead_of(float s) {
  const uint32_t b = __float_as_uint(s);
  return (b & 0x7FFFFFFFu) < 0x00800000u ? 1.0f : __uint_as_float((b & 0x007FFFFFu) | 0x3F800000u);
}
// 32 dims of one token -> shared memory: 64 bytes of the hi part and, unless s is a power of two, of the lo part
template <bool LO>
__device__ __forceinline__ void store_chunk(uint8_t* part_hi, int token, int chunk, const uint4& raw, float s) {
  const __half2 hi = __float2half2_rn(__uint_as_float(__float_as_uint(s) & 0xFFFF0000u));
  const __half2 lo = __float2half2_rn(s - __low2float(hi));
  const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
  uint8_t* row = part_hi + (chunk >> 1) * (kPart / 2) + token * 128;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    __half2 n[4];
    unpack8(words[w], n);
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 a = __hmul2(n[i], hi), b = __hmul2(n[i], lo);
      h[i] = *reinterpret_cast<const uint32_t*>(&a);
      if (LO) l[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    uint8_t* dst = row + ((((chunk & 1) * 4 + w) ^ (token & 7)) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    if (LO) *reinterpret_cast<uint4*>(dst + kPart) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

template <bool FACTORS>
__device__ __forceinline__ void unpack_tiles(const Params& p, Shared& sh, uint8_t* smem) {
  const lq_int4_cache& c = p.a.cache;
  const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  // lanes 0..7 hold eight tokens of chunk 0, lanes 8..15 the same tokens of chunk 1, ...: 512 contiguous bytes per load, and
  // the eight lanes of a shared-memory store phase hit eight different swizzle positions
  const int chunk = lane >> 3, row = 16 * warp + (lane & 7);
  const int groups_log2 = 7 - p.gs_log2, grp = (chunk * 32) >> p.gs_log2;
  // where the loads stand: a tile of a block; behind the last block no token is in range
  constexpr int kNoToken = 0x7FFF0000;
  int round = 0, tok = 0, tok_end = 0;
  const uint8_t *kp = nullptr, *vp = nullptr;
  const float *ks = nullptr, *vs = nullptr;
  auto open_block = [&]() {
    tok = row;
    if (entry_of(round) >= p.entries) {
      tok += kNoToken;
      tok_end = 0x7FFFFFFF;
      return;
    }
    const Block k = block_at(p, entry_of(round));
    tok_end = k.ntiles * kTok;
    kp = c.k_packed + k.b * c.kp_stride[0] + k.kvh * c.kp_stride[1] + chunk * 16;
    vp = c.v_packed + k.b * c.vp_stride[0] + k.kvh * c.vp_stride[1] + chunk * 16;
    ks = c.k_scale + k.b * c.ks_stride[0] + k.kvh * c.ks_stride[1] + grp;
    vs = c.v_scale + k.b * c.vs_stride[0] + k.kvh * c.vs_stride[1] + grp;
  };
  auto advance = [&]() {
    if (tok >= kNoToken) return;
    tok += kTok;
    if (tok >= tok_end) {
      ++round;
      open_block();
    }
  };
  // 16 bytes (32 dims) of this lane's two tokens of a tile, and their scales.  Ordinary loads, here and of the query: the non-coherent ones are for
  // data that nobody writes while the kernel lives, and a dependent launch lives while its predecessor writes these
  auto fetch = [&](const uint8_t* codes, int token, uint4 (&raw)[2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      raw[i] = token + 8 * i < p.kv_len ? *reinterpret_cast<const uint4*>(codes + static_cast<int64_t>(token + 8 * i) * 64) : make_uint4(0, 0, 0, 0);
  };
  auto fetch_scales = [&](const float* scales, int token, float (&sc)[2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) sc[i] = token + 8 * i < p.kv_len ? scales[static_cast<int64_t>(token + 8 * i) << groups_log2] : 0.0f;
  };
  auto publish = [&](int tile, const Exponents& ek, const Exponents& ev) {
    const int f = tile & 3;
    const bool wide = ek.wide || ev.wide;
    if (lane == 0) {
      sh.k_factor[f][warp] = pow2_of(ek.e[0]);
      sh.v_exp[f][warp] = static_cast<float>(ev.e[0]);
      sh.v_inv[f][warp] = pow2_of(-ev.e[0]);
      reinterpret_cast<uint8_t*>(&sh.wide[f])[warp] = (wide ? 1 : 0) | (ek.large ? 2 : 0);
    }
    if (wide && chunk == 0) {
      constexpr uint32_t kChunks = 0x01010101u;  // a token's bits of a ballot
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t v_bad = (ev.bad[i] >> lane) & kChunks;
        sh.k_factor_tok[f][row + 8 * i] = (ek.bad[i] >> lane) & kChunks ? __uint_as_float(0x7FC00000u) : pow2_of(ek.e[i]);
        sh.v_exp_tok[f][row + 8 * i] = static_cast<float>(ev.e[i]);
        sh.v_inv_tok[f][row + 8 * i] = pow2_of(-ev.e[i]);
        sh.v_bad_tok[f][row + 8 * i] = static_cast<uint8_t>((v_bad | v_bad >> 7 | v_bad >> 14 | v_bad >> 21) & 15u);
      }
    }
  };
  // Takes the exponent out of the lane's two scales, and the token's factor, which goes to `lead` of the tile
  auto take_out = [&](float (&sc)[2], const int (&e)[2], float* lead) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      sc[i] *= pow2_of(-e[i]);
      if (FACTORS) {
        if (chunk == 0) lead[row + 8 * i] = lead_of(sc[i]);
        sc[i] = __uint_as_float(__float_as_uint(sc[i]) & 0xFF800000u);
      }
    }
  };
  auto store = [&](int stage, const uint4 (&raw)[2], const float (&s)[2]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) store_chunk<!FACTORS>(smem + stage * kStageBytes, row + 8 * i, chunk, raw[i], s[i]);
  };
  auto arrive = [&](uint64_t* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  uint4 k[2], v[2], k_next[2], v_next[2];
  float ks_cur[2], vs_cur[2], vs_ahead[2], ks_next[2], vs_next[2];  // scales of k and v above (of v with its exponents taken out); of V one tile further
  open_block();
  fetch(kp, tok, k);
  fetch_scales(ks, tok, ks_cur);
  fetch_scales(vs, tok, vs_cur);
  fetch(vp, tok, v);
  advance();
  fetch(kp, tok, k_next);
  fetch_scales(ks, tok, ks_next);
  fetch_scales(vs, tok, vs_ahead);
  {
    const Exponents ek = exponents_of(ks_cur), ev = exponents_of(vs_cur);
    publish(0, ek, ev);
    take_out(ks_cur, ek.e, sh.k_lead[0]);
    take_out(vs_cur, ev.e, sh.v_lead[0]);
    store(0, k, ks_cur);
    arrive(&sh.k_first);
  }
  int total = 0;  // tiles of all blocks of this CTA
  for (int r = 0; entry_of(r) < p.entries; ++r) total += block_at(p, entry_of(r)).ntiles;
  for (int j = 0; j < total; ++j) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      k[i] = k_next[i];
      ks_cur[i] = ks_next[i];
    }
    fetch(vp, tok, v_next);
    advance();
    fetch(kp, tok, k_next);
    fetch_scales(ks, tok, ks_next);
    fetch_scales(vs, tok, vs_next);
    const Exponents ek = exponents_of(ks_cur), ev_ahead = exponents_of(vs_ahead);
    // iteration j - 2 is done (its last products are S of tile j - 1); unit 0 finds its stages empty, unit 1 waits for S of tile 0
    if (!wait_bar(&sh.empty[j & 1], ((j >> 1) ^ j ^ 1) & 1)) return;
    publish(j + 1, ek, ev_ahead);
    take_out(ks_cur, ek.e, sh.k_lead[(j + 1) & 3]);
    take_out(vs_ahead, ev_ahead.e, sh.v_lead[(j + 1) & 3]);
    store(2 + (j & 1), v, vs_cur);
    if (j + 1 < total) store((j + 1) & 1, k, ks_cur);
    arrive(&sh.full[j & 1]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      v[i] = v_next[i];
      vs_cur[i] = vs_ahead[i];
      vs_ahead[i] = vs_next[i];
    }
  }
}

// ---- products --------------------------------------------------------------------------------------------------------
template <bool FACTORS>
__device__ __forceinline__ void issue_products(const Params& p, Shared& sh, uint8_t* smem) {
  const uint64_t k_desc = smem_desc(smem_u32(smem), 16), v_desc = smem_desc(smem_u32(smem) + 2 * kStageBytes, kPart / 2);
  // S = Q Khi + Q Klo; 16 dims per product: 32 bytes inside a half of 64 dims.  With token factors there is no lo part
  auto issue_s = [&](int g, int j) {
    const uint32_t tm = g * kColsPerGroup;
    const uint64_t d = k_desc + (j & 1) * (kStageBytes >> 4);
#pragma unroll
    for (int hl = 0; hl < (FACTORS ? 1 : 2); ++hl)
#pragma unroll
      for (int k = 0; k < 8; ++k)
        mma_ts(tm + kColS, tm + kColQ + 8 * k, d + ((hl * kPart + (k >> 2) * (kPart / 2) + (k & 3) * 32) >> 4), kIdescS, hl + k > 0);
  };
  // O += Phi Vhi + Plo Vhi + Phi Vlo; 16 tokens per product: 2048 bytes
  auto issue_o = [&](int g, int j, bool first) {
    const uint32_t tm = g * kColsPerGroup;
    const uint64_t d = v_desc + (j & 1) * (kStageBytes >> 4);
#pragma unroll
    for (int t = 0; t < (FACTORS ? 2 : 3); ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        mma_ts(tm + kColO, tm + kColS + (t == 1 ? 32 : 0) + 8 * k, d + (((t == 2 ? kPart : 0) + k * 2048) >> 4), kIdescO, !first || t + k > 0);
  };
  uint32_t p_parity = 0, q_parity = 0;  // bit g
  // S of a block's first tile, once the groups have put their query rows into TMEM
  auto open_block = [&](int groups, int tile) {
    for (int g = 0; g < groups; ++g) {
      if (!wait_bar(&sh.q_ready[g], (q_parity >> g) & 1)) return false;
      q_parity ^= 1u << g;
      fence_after();
      if (elect_one()) {
        issue_s(g, tile);
        mma_commit(&sh.s_done[g]);
        if (g == groups - 1) mma_commit(&sh.empty[(tile - 1) & 1]);
      }
      __syncwarp();
    }
    return true;
  };
  if (!wait_bar(&sh.k_first, 0)) return;
  Block k = block_at(p, entry_of(0));
  if (!open_block(k.groups, 0)) return;
  int tile = 0;
  for (int r = 0;;) {
    for (int j = 0; j < k.ntiles; ++j, ++tile) {
      const bool more = j + 1 < k.ntiles;
      if (!wait_bar(&sh.full[tile & 1], (tile >> 1) & 1)) return;
      for (int g = 0; g < k.groups; ++g) {
        if (!wait_bar(&sh.p_ready[g], (p_parity >> g) & 1)) return;
        p_parity ^= 1u << g;
        fence_after();
        if (elect_one()) {
          issue_o(g, tile, j == 0);
          if (more) issue_s(g, tile + 1);
          mma_commit(&sh.s_done[g]);
          if (more && g == k.groups - 1) mma_commit(&sh.empty[tile & 1]);
        }
        __syncwarp();
      }
    }
    ++r;
    if (entry_of(r) >= p.entries) return;
    k = block_at(p, entry_of(r));
    if (!open_block(k.groups, tile)) return;
  }
}

// ---- softmax ---------------------------------------------------------------------------------------------------------
// 128 dims of a query row in the caller's 16-bit type, two per word
__device__ __forceinline__ void load_query_row(const lq_int4_prefill_args& a, int64_t base, bool vec, uint32_t (&raw)[64]) {
  if (vec) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.q) + base);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint4 v = src[i];
      raw[4 * i] = v.x; raw[4 * i + 1] = v.y; raw[4 * i + 2] = v.z; raw[4 * i + 3] = v.w;
    }
  } else {
    const uint16_t* src = static_cast<const uint16_t*>(a.q) + base;
#pragma unroll
    for (int i = 0; i < 64; ++i) raw[i] = src[2 * i * a.q_stride[3]] | (static_cast<uint32_t>(src[(2 * i + 1) * a.q_stride[3]]) << 16);
  }
}
__device__ __forceinline__ float2 unpack16x2(uint32_t w, bool bf16) {
  if (bf16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

// Query row -> fp16 in TMEM, its largest value brought to [2^14, 2^15); returns the factor of a product of this row,
// 2^Eq log2(e) / sqrt(128).  large: of any row of the warp, as bits of Shared::wide
__device__ __forceinline__ float load_query(const lq_int4_prefill_args& a, int64_t base, bool live, uint32_t tm_q, uint32_t& large) {
  uint32_t raw[64];
  const bool bf16 = a.dtype == LQ_BF16;
  if (live) {
    load_query_row(a, base, a.q_stride[3] == 1 && ((reinterpret_cast<uintptr_t>(a.q) + 2 * base) & 15) == 0, raw);
  } else {
#pragma unroll
    for (int i = 0; i < 64; ++i) raw[i] = 0u;
  }
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 64; ++i) {
    const float2 v = unpack16x2(raw[i], bf16);
    amax = max3(amax, fabsf(v.x), fabsf(v.y));
  }
  large = __any_sync(0xFFFFFFFFu, amax >= kLargeQ) ? 0x02020202u : 0u;
  int field = static_cast<int>(__float_as_uint(amax) >> 23);
  field = field == 0 ? 141 : min(max(field, 15), 254);  // a row of zeros keeps the factor 1
  const float to_half = __uint_as_float(static_cast<uint32_t>(268 - field) << 23);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t q[32];
#pragma unroll
    for (int w = 0; w < 8; ++w) {  // word of eight dims: pairs (0,4) (1,5) (2,6) (3,7)
      float d[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 v = unpack16x2(raw[32 * half + 4 * w + i], bf16);
        d[2 * i] = v.x * to_half;
        d[2 * i + 1] = v.y * to_half;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) q[4 * w + i] = pack_half2(d[i], d[i + 4]);
    }
    tmem_store32(tm_q + 32 * half, q);
  }
  tmem_wait_store();
  return __uint_as_float(static_cast<uint32_t>(field - 14) << 23) * (1.4426950408889634f * 0.08838834764831845f);
}

// bad: a bit per 32 dims that are NaN
__device__ __forceinline__ void store_output(const lq_int4_prefill_args& a, int64_t ob, uint32_t tm_o, float inv_row, uint32_t bad, bool live) {
  const bool vec = a.out_stride[3] == 1 && ((reinterpret_cast<uintptr_t>(a.out) + 2 * ob) & 15) == 0;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    uint32_t o[32];
    tmem_load32(o, tm_o + 32 * q);
    if (!live) continue;
    const float inv = (bad >> q) & 1 ? __uint_as_float(0x7FC00000u) : inv_row;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      float d[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) d[(i >> 1) + 4 * (i & 1)] = __uint_as_float(o[8 * w + i]) * inv;
      const int dim = 32 * q + 8 * w;
      if (vec) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (a.dtype == LQ_BF16) {
            const __nv_bfloat162 r = __floats2bfloat162_rn(d[2 * i], d[2 * i + 1]);
            v[i] = *reinterpret_cast<const uint32_t*>(&r);
          } else {
            v[i] = pack_half2(d[2 * i], d[2 * i + 1]);
          }
        }
        *reinterpret_cast<uint4*>(static_cast<uint16_t*>(a.out) + ob + dim) = make_uint4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) store_from_float(a.out, ob + (dim + i) * a.out_stride[3], a.dtype, d[i]);
      }
    }
  }
}

// One row of scores of one block, a tile at a time: S -> P in place, running maximum and sum.  tile: the block's first, counted over
// all blocks; parity: of the next wait for products of this group; l_run: the sum; bad: the 32-dim chunks for which the row has
// attended to a V that is not finite.  False after a wait that ran out.
template <bool FACTORS>
__device__ __forceinline__ bool softmax_rows(const Params& p, Shared& sh, int pos0, int ntiles, int tile, uint32_t& parity, float cq, uint32_t large_q,
                                             float& l_run, uint32_t& bad) {
  const lq_int4_prefill_args& a = p.a;
  const int group = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int row = warp * 32 + lane;  // = TMEM lane
  const int pos = pos0 + ((group * kGroupRows + row) >> p.ratio_log2);
  const int limit = a.first_len + min(pos, a.q_len - 1);  // tokens this row sees
  // the tokens that every row of the warp sees
  const int warp_limit = a.first_len + min(pos0 + ((group * kGroupRows + warp * 32) >> p.ratio_log2), a.q_len - 1);
  const uint32_t tm = group * kColsPerGroup + (static_cast<uint32_t>(warp * 32) << 16);
  float m_run = 0.0f;
  l_run = 0.0f;
  bad = 0u;
  for (int j = 0; j < ntiles; ++j) {
    const int tok0 = j * kTok, f = (tile + j) & 3;
    if (!wait_bar(&sh.s_done[group], parity)) return false;
    parity ^= 1;
    fence_after();
    const uint32_t wide = sh.wide[f] | large_q;
    uint32_t s[64];
    tmem_load64(s, tm + kColS);
    if (FACTORS) {
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float4 k = *reinterpret_cast<const float4*>(&sh.k_lead[f][i]);
        const float2 a = __fmul2_rn(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), make_float2(k.x, k.y));
        const float2 b = __fmul2_rn(make_float2(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])), make_float2(k.z, k.w));
        s[i] = __float_as_uint(a.x); s[i + 1] = __float_as_uint(a.y); s[i + 2] = __float_as_uint(b.x); s[i + 3] = __float_as_uint(b.y);
      }
    }
    // Rare cases share the branches that are there anyway: with branches of their own 1 x 128 behind 4000 took 115 us instead of 109.
    if (tok0 + kTok > warp_limit || wide != 0u) {
      if (wide != 0u) {  // the finished score of every token in place of the raw one
#pragma unroll 1
        for (int w = 0; w < 4; ++w) {
          const bool own = (wide >> (8 * w)) & 1u;
          const float* const kf = own ? &sh.k_factor_tok[f][16 * w] : &sh.k_factor[f][w];
          const float* const ve = own ? &sh.v_exp_tok[f][16 * w] : &sh.v_exp[f][w];
          uint32_t raw[16];
          tmem_load16(raw, tm + kColS + 16 * w);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            raw[i] = __float_as_uint(fmaf(__uint_as_float(raw[i]) * (FACTORS ? sh.k_lead[f][16 * w + i] : 1.0f), cq * kf[own ? i : 0], ve[own ? i : 0]));
            if (own && tok0 + 16 * w + i < limit) bad |= sh.v_bad_tok[f][16 * w + i];
          }
          tmem_store16(tm + kColS + 16 * w, raw);
        }
        tmem_wait_store();
        tmem_load64(s, tm + kColS);
      }
#pragma unroll
      for (int i = 0; i < 64; ++i)
        if (tok0 + i >= limit) s[i] = 0xFF800000u;  // -inf
    }
    const int slot = wide != 0u ? 4 : f;  // 4: scores are finished, the sum is taken further down
    const float cq_tile = wide != 0u ? 1.0f : cq;
    float cw[4], ev[4], mt[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      cw[w] = fmaxf(cq_tile * sh.k_factor[slot][w], 1.17549435e-38f);  // never 0: -inf * 0 would be NaN
      ev[w] = sh.v_exp[slot][w];
      const auto at = [&](int i) { return __uint_as_float(s[16 * w + i]); };
      const float m0 = max3(at(0), at(1), at(2)), m1 = max3(at(3), at(4), at(5)), m2 = max3(at(6), at(7), at(8));
      const float m3 = max3(at(9), at(10), at(11)), m4 = max3(at(12), at(13), at(14));
      mt[w] = fmaf(max3(max3(m0, m1, m2), max3(m3, m4, at(15)), m2), cw[w], ev[w]);
    }
    const float m_tile = fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3]));
    if (j == 0) {
      m_run = m_tile;  // every row sees token 0
    }
    if (__any_sync(0xFFFFFFFFu, m_tile > m_run + kSlack<FACTORS> || wide != 0u)) {
      if (j > 0) {
        // rare: the running sums of this warp's rows move to a larger maximum (the products into O of the tile before are done)
        const float m_new = fmaxf(m_run, m_tile), alpha = exp2f(m_run - m_new);
        m_run = m_new;
        l_run *= alpha;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          uint32_t o[32];
          tmem_load32(o, tm + kColO + 32 * q);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_store32(tm + kColO + 32 * q, o);
        }
      }
      if (wide != 0u) {  // the sum of the very weights that are stored below
#pragma unroll 1
        for (int w = 0; w < 4; ++w) {
          const bool own = (wide >> (8 * w)) & 1u;
          const float* const vi = own ? &sh.v_inv_tok[f][16 * w] : &sh.v_inv[f][w];
          uint32_t x[16];
          tmem_load16(x, tm + kColS + 16 * w);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (tok0 + 16 * w + i < limit) l_run = fmaf(mma::fast_exp2(__uint_as_float(x[i]) + (kLift - m_run)), vi[own ? i : 0], l_run);
        }
      }
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float off = ev[w] + (kLift - m_run);
      float2 sum = make_float2(0.0f, 0.0f);
      uint32_t hi[8], lo[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 x = __ffma2_rn(make_float2(__uint_as_float(s[16 * w + 2 * i]), __uint_as_float(s[16 * w + 2 * i + 1])), make_float2(cw[w], cw[w]),
                                    make_float2(off, off));
        float2 pr = make_float2(mma::fast_exp2(x.x), mma::fast_exp2(x.y));
        sum = __fadd2_rn(sum, pr);
        if (FACTORS) pr = __fmul2_rn(pr, *reinterpret_cast<const float2*>(&sh.v_lead[f][16 * w + 2 * i]));
        // leading 11 bits by truncation (exact in fp16 from 2^-14 on), the rest rounded to fp16
        const float2 top = make_float2(__uint_as_float(__float_as_uint(pr.x) & 0xFFFFE000u), __uint_as_float(__float_as_uint(pr.y) & 0xFFFFE000u));
        const float2 rest = __ffma2_rn(top, make_float2(-1.0f, -1.0f), pr);
        hi[i] = pack_half2(top.x, top.y);
        lo[i] = pack_half2(rest.x, rest.y);
      }
      tmem_store8(tm + kColS + 8 * w, hi);
      tmem_store8(tm + kColS + 32 + 8 * w, lo);
      l_run = fmaf(sum.x + sum.y, sh.v_inv[slot][w], l_run);
    }
    tmem_wait_store();
    fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.p_ready[group]);
  }
  return true;
}

template <bool FACTORS>
__device__ __forceinline__ void softmax_blocks(const Params& p, Shared& sh) {
  const lq_int4_prefill_args& a = p.a;
  const int group = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int row = threadIdx.x & 127, in_block = static_cast<int>(threadIdx.x) >> p.ratio_log2;
  const uint32_t tm = group * kColsPerGroup + (static_cast<uint32_t>(warp * 32) << 16);
  const auto head_of = [&](const Block& k) { return (k.kvh << p.ratio_log2) + (row & ((1 << p.ratio_log2) - 1)); };
  float cq = 0.0f, l_run;
  uint32_t large_q = 0u, bad;
  // the group's query rows of its first block from round r on, none of whose S has been asked for yet
  const auto load_next = [&](int r) {
    for (; entry_of(r) < p.entries; ++r) {
      const Block k = block_at(p, entry_of(r));
      if (group >= k.groups) continue;
      const int pos = k.pos0 + in_block;
      const int64_t base = k.b * a.q_stride[0] + head_of(k) * a.q_stride[1] + static_cast<int64_t>(pos) * a.q_stride[2];
      cq = load_query(a, base, pos < a.q_len, tm + kColQ, large_q);
      fence_before();
      __syncwarp();
      return true;
    }
    return false;
  };
  uint32_t parity = 0;
  int tile = 0;
  if (load_next(0) && lane == 0) mbar_arrive(&sh.q_ready[group]);
#pragma unroll 1
  for (int r = 0; entry_of(r) < p.entries; ++r) {
    const Block k = block_at(p, entry_of(r));
    if (group < k.groups) {
      if (!softmax_rows<FACTORS>(p, sh, k.pos0, k.ntiles, tile, parity, cq, large_q, l_run, bad)) return;
      const bool more = load_next(r + 1);  // all S of this block are done; its last products run meanwhile
      // the wait stands before the arrival that lets the next S be asked for: s_done is never two phases ahead of a warp
      if (!wait_bar(&sh.s_done[group], parity)) return;
      parity ^= 1;
      fence_after();
      if (more && lane == 0) mbar_arrive(&sh.q_ready[group]);
      const int pos = k.pos0 + in_block;
      const int64_t ob = k.b * a.out_stride[0] + head_of(k) * a.out_stride[1] + static_cast<int64_t>(pos) * a.out_stride[2];
      store_output(a, ob, tm + kColO, 1.0f / l_run, bad, pos < a.q_len);
    }
    tile += k.ntiles;
  }
}

// One CTA per SM works through a list of row blocks, and a block's start overlaps the end of the one before: its first tiles are
// unpacked, its query rows loaded and its first scores made while the last products run and the output is stored.  A tile
// takes 2.05 us; as one CTA per block, start and end added 8 to 9 us to every block.  8 x 1024 tokens: 185 -> 160 us; 2 x 2000 behind 6001: 884 -> 855; 16 x 256: 53 -> 43; 1 x 128 behind 4000 (halves): 135 -> 110.
// Dropped: two score buffers of 32 tokens per group, which would let the tensor pipe run ahead of the softmax (a product of 32 columns
// takes as long as one of 64: 2.31 us a tile), and starting the products of a tile's first half while its second is made (2.1 us).
template <bool FACTORS>
__global__ void __launch_bounds__(kThreads, 1) int4_prefill_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Shared sh;  // no early trigger: dependents that start as this kernel's CTAs leave cost 1 to 4 % of a launch of many blocks (lq_int4_kv.cu)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5;
  if (warp == 12) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sh.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x < 4) {
    sh.k_factor[4][threadIdx.x] = 1.0f;
    sh.v_exp[4][threadIdx.x] = sh.v_inv[4][threadIdx.x] = 0.0f;
  }
  if (threadIdx.x == 0) {
    mbar_init(&sh.k_first, 4);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.full[i], 4);
      mbar_init(&sh.empty[i], 1);
      mbar_init(&sh.s_done[i], 1);
      mbar_init(&sh.p_ready[i], 4);
      mbar_init(&sh.q_ready[i], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  pdl_wait();  // nothing above reads memory; below, what the predecessor has written (the packed rows as a rule) is read
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp < 12) unpack_tiles<FACTORS>(p, sh, smem);
    else if (warp == 12) issue_products<FACTORS>(p, sh, smem);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    softmax_blocks<FACTORS>(p, sh);
  }
  fence_before();
  __syncthreads();
  if (warp == 12) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(sh.tmem));
  }
}

}  // namespace prefill
}  // namespace lq
