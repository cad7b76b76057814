// out[M,N] = x[M,K] * w[N,K]^T in 32 bits on the tensor cores, for many rows.
//
// A 32-bit number is the sum of three bfloat16 numbers, exactly (its 24 bits are three times 8; each
// piece is what rounding leaves of the one before; Henry, Tang and Heinecke, "Leveraging the bfloat16
// artificial intelligence datatype for higher-precision computations", 2019). A product of two such sums
// is nine products of pieces; six go through tcgen05.mma (bf16 x bf16, whose products are exact in 32
// bits), the other three, below 2^-24 of |x w| each, are dropped. Tensor memory truncates where it
// accumulates, so a sum stays there for 32 of K only, its small products first, and the partial sums
// are added in registers, rounded to nearest. Relative error against 64 bits (2-norm, normal
// operands): K = 2048 1.6e-7 (1.0e-7 where four pairs share K), K = 8192 2.9e-7 (1.6e-7); FFMA tiles
// (gemm_f32.cu) 8.1e-7 or 2.9e-7, and 5.8e-7. Sums over 64 of K: 3.3e-7, hence 32.
//
// Bound by the tensor pipe, six bf16 products for one, and close behind it by the issue slots of the
// warps that split and add (two more instructions an operand: 777 rows of 2048 -> 16384 280 us). 777
// rows of 2048 -> 16384 257 us (203 TFLOP/s of the product, 1.22 PFLOP/s of bf16) where FFMA tiles took
// 1524, -> 3072 59 for 311, 8192 -> 2048 156 for 789; 64 rows of 2048 -> 2048 23 for 33; 2048 rows ->
// 16384 700 for 3010 (74 TFLOP/s is all that FFMA could give). The weights are split tile by tile, not
// once to memory, which would move 16 bytes an element where this moves 4.
//
// Two SMs share a tile of 256 weight rows (the instruction's rows) and up to 208 tokens (its N): each
// loads 128 weight rows and half of the tokens. The weights' pieces go to tensor memory, as the
// instruction's first operand, the tokens' to shared memory: with both in shared memory, its
// bandwidth was the bound (raw tiles in and out, pieces in, and out again for six products; 777 rows
// -> 16384 473 us). Roles of a CTA's 20 warps: TMA producer, MMA issuer (leader only), two idle, 8
// that split raw 32-bit stages, 8 that add accumulators up in registers and store. Every wait is
// bounded, as elsewhere.
//
// What pieces cannot carry is summed again behind all tiles, as chains of FMAs (`repair`): results that are
// not finite (an infinity's pieces are not numbers, and what overflows has to do so where 32 bits do),
// and those of operands so small that their pieces, or products of them, fall below the smallest normal
// number, which the tensor cores take as zero: x of 1e-36 times w of 1e10 would be off by 1e-3. The
// splitting warps keep the largest first piece (half an instruction an operand; 777 rows of 2048 ->
// 16384 252 -> 257 us); unless it is huge, a finite result of 2^-64 or more stands, and the rows of the
// others are looked at, which settles most (`falls`). Zeros cost that look: a token in seven of zeros,
// 777 rows of 8192 -> 16384 990 -> 1,320 us; all of x NaN 1,500, all of it infinite 26,000.
#define FB_STATUS_KERNEL 5
#include "gemm_f32.h"
#include "tcgen05_pair.cuh"

namespace {

constexpr int KB = 32;            // K of a stage: 128 bytes of a raw row, 64 of a piece's
constexpr int W_ROWS = 128;       // weight rows of a CTA
constexpr int PIECES = 3;
constexpr int MAX_STAGES = 8, MAX_PIECE_STAGES = 4;
constexpr int MAX_SHARES = 4;     // pairs of a cluster (8 CTAs, the portable size)
// Rounds of tiles that are kept apart in what a CTA notes of them (the others share, round % ROUNDS), and
// words for a bit a token of a tile.
constexpr int ROUNDS = 32, TOKEN_WORDS = 7;
constexpr int SPLIT_WARPS = 8, SUM_WARPS = 8;
constexpr int THREADS = 32 * (4 + SPLIT_WARPS + SUM_WARPS);
// Tensor memory: two accumulators of tn columns, then the weights' pieces, 16 columns each.
constexpr int W_PIECE_COLS = KB / 2, TMEM_COLS = 512, MAX_TN = 208, RUNS = (MAX_TN / 16 + 1) / 2;
// registers a thread of the five warpgroups: loads and MMAs, 2 x splitting, 2 x sums (112 sums a
// thread); their total stays below what the block is launched with (the launcher looks, and leaves it)
constexpr int REGS_LOAD = 48, REGS_SPLIT = 56, REGS_SUM = 160;
constexpr int REGS_ALL = REGS_LOAD + 2 * REGS_SPLIT + 2 * REGS_SUM;
constexpr int SMEM_DYNAMIC = 227 * 1024 - 1536 /*barriers and notes*/, SMEM_TILES = SMEM_DYNAMIC - 1024 /*align*/;

struct Params {
  const float* x;
  const float* w;
  float* out;
  int M, N, K;
  long long ldx, ldw, ldo;
  int tn, tiles_t, units;    // tokens of a tile (a multiple of 16), tiles of them, all tiles
  int stages, piece_stages;  // raw ones, split ones
  int shares;                // pairs that share a tile's K
};

__host__ __device__ constexpr int raw_bytes(int tn) { return (W_ROWS + tn / 2) * KB * 4; }
__host__ __device__ constexpr int piece_bytes(int tn) { return PIECES * (tn / 2) * KB * 2; }

// Descriptor of a K-major tile with rows of 64 bytes in the 64-byte swizzle: 8-row groups are 512
// bytes apart; otherwise as make_desc.
__device__ __forceinline__ uint64_t make_desc64(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(512u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}

// Takes the next bfloat16 piece off two numbers (the first in the lower half).
__device__ __forceinline__ uint32_t take_piece(float& a, float& b) {
  uint32_t h;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
  a -= __uint_as_float(h << 16);
  b -= __uint_as_float(h & 0xffff0000u);
  return h;
}
__device__ __forceinline__ uint32_t last_piece(float a, float b) {
  uint32_t h;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
  return h;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t yes;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(yes));
  return yes != 0;
}
__device__ __forceinline__ float4 ld_shared(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7])
      : "memory");
}
// The pair's product with A (lane = row, a column two neighbouring k) in tensor memory.
__device__ __forceinline__ void umma_pair_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b,
                                                 uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void st_shared(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
               ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Waits for the loads from tensor memory that this warp has under way; `r` is what came.
__device__ __forceinline__ void tmem_arrived(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]),
                 "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

// tc_commit_pair for a pair anywhere in its cluster; `lead_cta`: the pair's first CTA.
__device__ __forceinline__ void commit_to_pair(uint64_t* bar, uint32_t lead_cta) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)(3u << lead_cta))
      : "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void max_cluster(uint32_t addr, uint32_t v) {
  asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void or_cluster(uint32_t addr, uint32_t bits) {
  asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(addr), "r"(bits) : "memory");
}

// A warp's wait for two barriers, asked after together (one after the other cost twice the latency).
__device__ __forceinline__ bool wait_both(uint64_t* bar_a, uint32_t parity_a, int where_a, uint64_t* bar_b,
                                          uint32_t parity_b, int where_b, volatile int* abort_flag,
                                          int kb) {
  uint32_t both;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
      "and.pred p, p, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(both)
      : "r"(smem_u32(bar_a)), "r"(parity_a), "r"(smem_u32(bar_b)), "r"(parity_b)
      : "memory");
  bool ok = both != 0;
  if (!ok)
    ok = mbar_wait(bar_a, parity_a, abort_flag, where_a, kb) &&
         mbar_wait(bar_b, parity_b, abort_flag, where_b, kb);
  return __all_sync(0xffffffffu, ok);
}

template <int N>
__device__ __forceinline__ void more_registers() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void fewer_registers() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// The roles end in branches of their own (a role's registers are its own there): all threads of the
// cluster meet, with shares twice.
__device__ __forceinline__ void shares_meet() { cluster_barrier(); }
__device__ __forceinline__ void roles_meet() {
  tc_fence_before();
  __syncwarp();
  asm volatile("barrier.cta.sync 0;" ::: "memory");
  cluster_barrier();  // nothing of the peers' may still be on its way to this CTA; results are stored
}
__device__ __forceinline__ void all_meet(const Params& p) {
  if (p.shares > 1) shares_meet();
  roles_meet();
}

// Whether a sum of pieces needs no look at its operands: finite, and of 2^-64 or more (see above).
__device__ __forceinline__ bool stands(float v) {
  return (__float_as_uint(v) & 0x7fffffffu) - 0x1f800000u < 0x7f800000u - 0x1f800000u;
}

// The larger magnitudes of two pairs of first pieces (of a number and a NaN the number's).
__device__ __forceinline__ uint32_t larger_pieces(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t largest_of_warp(uint32_t pieces) {  // as the bits of a float
  const uint32_t a = (pieces & 0x7fffu) << 16, b = pieces & 0x7fff0000u;
  return __reduce_max_sync(0xffffffffu, max(a, b));
}
// Whether a row is zeros alone, by one warp.
__device__ __forceinline__ bool is_zero_row(const float* row, int K, int lane) {
  for (int k0 = lane * 4; __any_sync(0xffffffffu, k0 < K); k0 += 16 * 128) {
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (k0 + 128 * i < K) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(row + k0 + 128 * i));
        bits |= (__float_as_uint(v.x) | __float_as_uint(v.y)) | (__float_as_uint(v.z) | __float_as_uint(v.w));
      }
    if (__any_sync(0xffffffffu, bits << 1 != 0)) return false;  // (a zero has a sign)
  }
  return true;
}

// What a row of operands is: the largest magnitude (not a NaN's), the smallest that is not zero (as twice
// its bits less one, so that a zero is the largest), whether it holds a NaN.
struct RowFacts {
  float most;
  uint32_t least;
  int nan;
};
constexpr float LEAST_WHOLE = 1.0f / (1 << 30) / (1 << 30) / (1 << 30) / (1 << 12);  // 2^-102

// Whether a result is to be summed again. Pieces and products of pieces below 2^-126 may have been taken as
// zero: nothing beyond 2^-24 of an operand of 2^-102 or more, nothing beyond 2^-25 of a product of 2^-98
// or more; else K terms lose up to 2^-126 of the largest other operand each way, and six products of
// 2^-126. The result stands where it is 2^24 times that. (A row with a NaN has its results.)
__device__ __forceinline__ bool falls(float v, const RowFacts& w, const RowFacts& x, int K) {
  if (w.nan || x.nan) return false;
  const float size = fabsf(v);
  if (!(size <= 3.402823466e38f)) return true;
  if (w.least == 0xffffffffu || x.least == 0xffffffffu) return false;  // a row of zeros
  const float least_w = __uint_as_float((w.least >> 1) + 1u), least_x = __uint_as_float((x.least >> 1) + 1u);
  if (least_w >= LEAST_WHOLE && least_x >= LEAST_WHOLE && least_w * least_x >= 16.f * LEAST_WHOLE) return false;
  return !(size >= (float)K * LEAST_WHOLE * (w.most + x.most + 8.f));
}
// Whether one operand's row alone settles a result: all are NaN, or it is the zero that a row of zeros makes.
__device__ __forceinline__ bool settles(const RowFacts& of, float v) {
  return of.nan || (of.least == 0xffffffffu && v == 0.f);
}
// One warp looks at two rows side by side (a null row is left), up to 16 loads under way.
__device__ __forceinline__ void look_at_rows(RowFacts* to_a, const float* a, RowFacts* to_b, const float* b,
                                             int K, int lane) {
  float most[2] = {0.f, 0.f};
  uint32_t least[2] = {0xffffffffu, 0xffffffffu};
  bool nan[2] = {false, false};
  if (a == nullptr && b == nullptr) return;
  for (int k0 = lane * 4; k0 < K; k0 += 8 * 128) {
    float4 v[2][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = k0 + 128 * i;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      v[0][i] = a != nullptr && k < K ? __ldcg(reinterpret_cast<const float4*>(a + k)) : zero;
      v[1][i] = b != nullptr && k < K ? __ldcg(reinterpret_cast<const float4*>(b + k)) : zero;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float x[4] = {v[r][i].x, v[r][i].y, v[r][i].z, v[r][i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          most[r] = fmaxf(most[r], fabsf(x[e]));
          least[r] = min(least[r], 2u * __float_as_uint(x[e]) - 1u);
          nan[r] = nan[r] || !(x[e] == x[e]);
        }
      }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const RowFacts facts = {__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most[r]))),
                            __reduce_min_sync(0xffffffffu, least[r]), __any_sync(0xffffffffu, nan[r])};
    if (lane == 0 && (r == 0 ? a : b) != nullptr) *(r == 0 ? to_a : to_b) = facts;
  }
}

// The summing warps' threads meet; whether one of them said yes.
__device__ __forceinline__ bool any_of_sums(bool mine) {
  uint32_t any;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"((uint32_t)mine), "n"(32 * SUM_WARPS)
      : "memory");
  return any != 0;
}

// A run of 16 tokens (from t0) by this CTA's weight rows (from f0) once more, results that fall as chains of
// FMAs over K: 256 threads, a weight row and 8 tokens each, REPAIR_K of K at a time through shared memory.
// All of it is behind all tiles, where nobody waits for these warps. Which results fall: of those that do
// not stand by themselves (or of all; not the zeros of tokens that are not `busy`, which are zeros) the
// rows are looked at, first the operand's of which fewer are asked about (weight rows once a tile), then,
// for what is left, the other's.
constexpr int REPAIR_K = 256, REPAIR_PITCH = REPAIR_K + 4, REPAIR_ROWS = W_ROWS + 16;
static_assert(REPAIR_ROWS % 48 == 0, "whole rounds of loads");
struct RepairRoom {
  float stage[REPAIR_ROWS * REPAIR_PITCH];  // weight rows, then tokens
  RowFacts facts[REPAIR_ROWS];
  uint32_t asked[W_ROWS / 32 + 1], known[W_ROWS / 32];  // weight rows (tokens last); weight rows looked at
};
static_assert(sizeof(RepairRoom) <= SMEM_TILES, "room for the repair");
// Whether the result of weight row f and a tile's token t is to be looked at: no zero of a token of zeros.
__device__ __forceinline__ bool falls_maybe(const Params& p, const uint32_t* busy, bool all, int f, int tile0, int t) {
  if (tile0 + t >= p.M || f >= p.N) return false;
  const float v = __ldcg(p.out + (long long)(tile0 + t) * p.ldo + f);
  return v == 0.f ? busy[t >> 5] >> (t & 31) & 1u : all || !stands(v);
}
__device__ __forceinline__ void repair(const Params& p, RepairRoom& room, const uint32_t* busy, bool all, int f0,
                                       int tile0, int run0) {
  const int t0 = tile0 + run0;
  constexpr int WORDS = W_ROWS / 32;
  const int tid = (int)threadIdx.x - 32 * (4 + SPLIT_WARPS);
  const int row = tid % W_ROWS, half = tid / W_ROWS, f = f0 + row;
  RowFacts* facts = room.facts;
  auto result = [&](int e) { return __ldcg(p.out + (long long)(t0 + half * 8 + e) * p.ldo + f); };
  uint32_t wanted = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (falls_maybe(p, busy, all, f, tile0, run0 + half * 8 + e)) wanted |= 1u << e;
  auto ask = [&]() {
    if (tid <= WORDS) room.asked[tid] = 0;
    if (!any_of_sums(wanted != 0)) return false;
    if (wanted != 0) {
      atomicOr(&room.asked[row / 32], 1u << (row % 32));
      atomicOr(&room.asked[WORDS], wanted << (8 * half));
    }
    any_of_sums(false);
    return true;
  };
  auto look = [&](bool tokens) {  // a warp takes rows SUM_WARPS apart, two at once
    const uint32_t* known = tokens ? nullptr : room.known;
    const float* base = tokens ? p.x + (long long)t0 * p.ldx : p.w + (long long)f0 * p.ldw;
    const long long pitch = tokens ? p.ldx : p.ldw;
    const int first = tokens ? W_ROWS : 0, end = tokens ? W_ROWS + 16 : W_ROWS;
    for (int r = first + tid / 32; r < end; r += 2 * SUM_WARPS) {
      auto place = [&](int r) -> const float* {
        const bool asked = room.asked[r / 32] >> (r % 32) & 1u;
        return asked && (tokens || !(known[r / 32] >> (r % 32) & 1u)) ? base + (long long)(r - first) * pitch
                                                                      : nullptr;
      };
      const int s = r + SUM_WARPS;
      const float *a = place(r), *b = place(s);
      look_at_rows(facts + r, a, facts + s, b, p.K, tid & 31);
      __syncwarp();
      if (!tokens && (tid & 31) == 0) {
        if (a != nullptr) atomicOr(&room.known[r / 32], 1u << (r % 32));
        if (b != nullptr) atomicOr(&room.known[s / 32], 1u << (s % 32));
      }
    }
    any_of_sums(false);
  };
  if (!ask()) return;
  int rows = 0;
#pragma unroll
  for (int i = 0; i < WORDS; ++i) rows += __popc(room.asked[i] & ~room.known[i]);
  const bool tokens_first = any_of_sums(__popc(room.asked[WORDS]) <= rows);
  look(tokens_first);
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if ((wanted >> e & 1u) && settles(facts[tokens_first ? W_ROWS + half * 8 + e : row], result(e)))
      wanted &= ~(1u << e);
  if (!ask()) return;
  look(!tokens_first);
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if ((wanted >> e & 1u) && !falls(result(e), facts[row], facts[W_ROWS + half * 8 + e], p.K))
      wanted &= ~(1u << e);
  if (!any_of_sums(wanted != 0)) return;
  float* stage = room.stage;
  float* xs = stage + W_ROWS * REPAIR_PITCH;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < p.K; k0 += REPAIR_K) {
    const int k = k0 + tid % 64 * 4;
    any_of_sums(false);  // the numbers before have been read
    for (int r0 = tid / 64; r0 < REPAIR_ROWS; r0 += 48) {  // weight rows, then tokens; 12 loads at once
      float4 v[12];
#pragma unroll
      for (int i = 0; i < 12; ++i) {
        const int r = r0 + 4 * i, at = r < W_ROWS ? f0 + r : t0 + r - W_ROWS;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at < (r < W_ROWS ? p.N : p.M) && k < p.K)
          v[i] = __ldcg(reinterpret_cast<const float4*>(
              r < W_ROWS ? p.w + (long long)at * p.ldw + k : p.x + (long long)at * p.ldx + k));
      }
#pragma unroll
      for (int i = 0; i < 12; ++i)
        *reinterpret_cast<float4*>(stage + (r0 + 4 * i) * REPAIR_PITCH + tid % 64 * 4) = v[i];
    }
    any_of_sums(false);
    const int some = min(REPAIR_K, p.K - k0);
#pragma unroll 4
    for (int q = 0; q < some; q += 4) {
      const float4 w = *reinterpret_cast<const float4*>(stage + row * REPAIR_PITCH + q);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 x = *reinterpret_cast<const float4*>(xs + (half * 8 + e) * REPAIR_PITCH + q);
        acc[e] = fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, acc[e]))));
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (wanted >> e & 1u) p.out[(long long)(t0 + half * 8 + e) * p.ldo + f] = acc[e];
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap map_w,
                     const __grid_constant__ CUtensorMap map_x, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int half = p.tn / 2, stage_raw = raw_bytes(p.tn), stage_pieces = piece_bytes(p.tn);
  const int x_piece = half * KB * 2;  // bytes of one piece's tile
  uint8_t* pieces = tiles + p.stages * stage_raw;
  __shared__ __align__(8) uint64_t raw_full[MAX_STAGES], raw_empty[MAX_STAGES];
  __shared__ __align__(8) uint64_t piece_full[MAX_PIECE_STAGES];  // used in the leader
  __shared__ __align__(8) uint64_t piece_empty[MAX_PIECE_STAGES];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];  // acc_empty: used in the leader
  __shared__ uint32_t tmem_slot;
  // of this CTA's tiles, round by round: runs of 16 tokens in which a result does not stand; of a tile: its
  // tokens that are not zeros alone, the runs in which a result of theirs does not stand
  __shared__ uint32_t fallen[ROUNDS], busy[TOKEN_WORDS], odd;
  __shared__ uint32_t largest[2];  // first piece of a weight, of a token that the cluster multiplied
  __shared__ int s_abort;
  volatile int* abort_flag = &s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a cluster is the pairs that share a tile: one, which then walks tiles, or up to MAX_SHARES
  const uint32_t cta = cluster_cta_rank(), rank = cta & 1u, share = cta >> 1, lead_cta = cta & ~1u;
  const bool leader = rank == 0;
  const int ctas = 2 * p.shares;
  const int cluster = (int)blockIdx.x / ctas, clusters = (int)gridDim.x / ctas;
  const int stages_k = (p.K + KB - 1) / KB, kb0 = stages_k * (int)share / p.shares;
  const int nkb = stages_k * ((int)share + 1) / p.shares - kb0;  // this pair's part of K

  if (threadIdx.x < ROUNDS) fallen[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], SPLIT_WARPS / 2);
    }
    for (int b = 0; b < p.piece_stages; ++b) {
      mbar_init(&piece_full[b], SPLIT_WARPS);  // half of each CTA's
      mbar_init(&piece_empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * SUM_WARPS);
    }
    largest[0] = largest[1] = 0u;
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  cluster_barrier();  // the peer is there, and its barriers exist before anything arrives on them
  if (warp == 1) tmem_alloc_pair(&tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const uint32_t tmem_w = tmem_base + (uint32_t)(2 * p.tn);  // the weights' pieces
  const int total = nkb * ((p.units - cluster + clusters - 1) / clusters);  // stages of this pair

  if (warp < 4) {
    fewer_registers<REGS_LOAD>();
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------- TMA producer
      // the first unit's weights are asked for before this kernel waits for the one in front
      const int early = cluster < p.units ? min(nkb, p.stages) : 0;
      auto load_w = [&](int s, int u, int kb) {
        tma_load_2d(tiles + s * stage_raw, &map_w, &raw_full[s], (kb0 + kb) * KB,
                    (u / p.tiles_t) * 2 * W_ROWS + (int)rank * W_ROWS);
      };
      auto load_x = [&](int s, int u, int kb) {
        tma_load_2d(tiles + s * stage_raw + W_ROWS * KB * 4, &map_x, &raw_full[s], (kb0 + kb) * KB,
                    (u % p.tiles_t) * p.tn + (int)rank * half);
      };
      for (int i = 0; i < early; ++i) {
        mbar_expect_tx(&raw_full[i], (uint32_t)stage_raw);
        load_w(i, cluster, i);
      }
      fb_pdl_wait();
      for (int i = 0; i < early; ++i) load_x(i, cluster, i);
      int use = early, s = early % p.stages;
      uint32_t phase = (uint32_t)(early / p.stages) & 1u;
      bool ok = true;
      for (int u = cluster; u < p.units && ok; u += clusters) {
        for (int kb = u == cluster ? early : 0; kb < nkb; ++kb, ++use) {
          ok = mbar_wait(&raw_empty[s], phase ^ 1u, abort_flag, 1, kb);
          if (!ok) break;
          mbar_expect_tx(&raw_full[s], (uint32_t)stage_raw);
          load_w(s, u, kb);
          load_x(s, u, kb);
          if (++s == p.stages) { s = 0; phase ^= 1u; }
        }
      }
    } else if (warp == 1 && leader) {
      // -------------------------- MMA issuer (leader only): the whole warp, one thread of it issues
      const uint32_t idesc = make_idesc(2 * W_ROWS, p.tn);
      int b = 0, sum = 0;  // piece stage, accumulator
      uint32_t phase = 0, sum_phase = 0;
      for (int it = 0; it < total; ++it) {
        if (!wait_both(&piece_full[b], phase, 2, &acc_empty[sum], sum_phase ^ 1u, 4, abort_flag, it)) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t x0 = make_desc64(smem_u32(pieces) + b * stage_pieces);
          const uint32_t w0 = tmem_w + (uint32_t)(b * PIECES * W_PIECE_COLS);
          const uint32_t d_tmem = tmem_base + (uint32_t)(sum * p.tn);
          auto multiply = [&](int i, int j, bool fresh) {
#pragma unroll
            for (int k = 0; k < KB / 16; ++k)
              umma_pair_a_tmem(d_tmem, w0 + (uint32_t)(i * W_PIECE_COLS + k * 8),
                               x0 + (uint64_t)((j * x_piece + k * 32) >> 4), idesc,
                               fresh && k == 0 ? 0u : 1u);
          };
          multiply(2, 0, true);  // 2^-16 of the result
          multiply(0, 2, false);
          multiply(1, 1, false);
          multiply(1, 0, false);  // 2^-8
          multiply(0, 1, false);
          multiply(0, 0, false);
          commit_to_pair(&piece_empty[b], lead_cta);
          commit_to_pair(&acc_full[sum], lead_cta);
        }
        __syncwarp();
        if (++b == p.piece_stages) { b = 0; phase ^= 1u; }
        if ((sum ^= 1) == 0) sum_phase ^= 1u;
      }
    }
    all_meet(p);
    if (warp == 1) {
      tc_fence_after();
      tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
  } else if (warp < 4 + SPLIT_WARPS) {
    // ---------------------------------------------------------------- splitting
    fewer_registers<REGS_SPLIT>();
    // Four warps take every other stage each: a thread one weight row of it (its lane of tensor
    // memory), and 8 neighbouring k of a token, or of up to four.
    const int which = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t piece_full_leader = cluster_address(&piece_full[0], lead_cta);
    const uint32_t w_lanes = tmem_w + ((uint32_t)((warp & 3) * 32) << 16);
    int s = which, b = which;
    uint32_t raw_phase = 0, phase = 0;
    uint32_t most_w = 0, most_x = 0;
    for (int it = which; it < total; it += 2) {
      if (!wait_both(&raw_full[s], raw_phase, 5, &piece_empty[b], phase ^ 1u, 6, abort_flag, it)) break;
      tc_fence_after();
      // raw rows of 128 bytes in the 128-byte swizzle: weights first, then tokens
      const uint32_t raw = smem_u32(tiles) + s * stage_raw;
#pragma unroll
      for (int h = 0; h < KB / 16; ++h) {
        float v[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 t = ld_shared(raw + row * 128 + (((4 * h + q) ^ (row & 7)) << 4));
          v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
        }
#pragma unroll
        for (int piece = 0; piece < PIECES; ++piece) {
          uint32_t to[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            to[e] = piece + 1 < PIECES ? take_piece(v[2 * e], v[2 * e + 1])
                                       : last_piece(v[2 * e], v[2 * e + 1]);
          if (piece == 0) {
#pragma unroll
            for (int e = 0; e < 8; ++e) most_w = larger_pieces(most_w, to[e]);
          }
          tmem_st8(w_lanes + (uint32_t)((b * PIECES + piece) * W_PIECE_COLS + h * 8), to);
        }
      }
      const uint32_t raw_x = raw + W_ROWS * KB * 4, stage = smem_u32(pieces) + b * stage_pieces;
#pragma unroll 2
      for (int i = row; i < half * 4; i += 128) {
        const int r = i >> 2, q = i & 3;
        const uint32_t src = raw_x + r * 128;
        const float4 lo = ld_shared(src + (((2 * q) ^ (r & 7)) << 4));
        const float4 hi = ld_shared(src + (((2 * q + 1) ^ (r & 7)) << 4));
        float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        uint32_t dst = stage + r * 64 + ((q ^ ((r >> 1) & 3)) << 4);
#pragma unroll
        for (int piece = 0; piece < PIECES; ++piece, dst += x_piece) {
          uint32_t to[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            to[e] = piece + 1 < PIECES ? take_piece(v[2 * e], v[2 * e + 1])
                                       : last_piece(v[2 * e], v[2 * e + 1]);
          if (piece == 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) most_x = larger_pieces(most_x, to[e]);
          }
          st_shared(dst, make_uint4(to[0], to[1], to[2], to[3]));
        }
      }
      tmem_st_wait();
      tc_fence_before();
      fence_async_smem();  // the tensor core reads the pieces
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&raw_empty[s]);
        mbar_arrive_pair(piece_full_leader + (uint32_t)(b * 8));
      }
      if ((s += 2) >= p.stages) { s -= p.stages; raw_phase ^= 1u; }
      if ((b += 2) >= p.piece_stages) { b -= p.piece_stages; phase ^= 1u; }
    }
    const uint32_t of_w = largest_of_warp(most_w), of_x = largest_of_warp(most_x);
    if (lane < 2 * p.shares) {  // a lane tells a CTA of the cluster
      const uint32_t at = cluster_address(&largest[0], (uint32_t)lane);
      max_cluster(at, of_w);
      max_cluster(at + 4, of_x);
    }
    all_meet(p);
  } else {
    // --------------------------------------------------------------------- sums
    more_registers<REGS_SUM>();
    const int quarter = warp & 3, which = (warp - 4 - SPLIT_WARPS) >> 2;
    const uint32_t acc_empty_leader = cluster_address(&acc_empty[0], lead_cta);
    const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
    fb_pdl_wait();
    int b = 0, round = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int u = cluster; u < p.units && ok; u += clusters, ++round) {
      float acc[RUNS][16];  // this thread's weight row, every other run of 16 tokens
#pragma unroll
      for (int g = 0; g < RUNS; ++g)
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[g][e] = 0.f;
      for (int kb = 0; kb < nkb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], phase, abort_flag, 3, kb));
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = lanes + (uint32_t)(b * p.tn + which * 16);
        uint32_t r[2][16];  // the next run is on its way while one is added
        tmem_ld16(taddr, r[0]);
#pragma unroll
        for (int g = 0; g < RUNS; ++g) {
          if (g > 0 && (2 * g + which) * 16 >= p.tn) break;
          tmem_arrived(r[g & 1]);
          if (g + 1 < RUNS && (2 * g + 2 + which) * 16 < p.tn)
            tmem_ld16(taddr + (uint32_t)(32 * g + 32), r[(g + 1) & 1]);
#pragma unroll
          for (int e = 0; e < 16; ++e) acc[g][e] += __uint_as_float(r[g & 1][e]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_pair(acc_empty_leader + (uint32_t)(b * 8));
        if ((b ^= 1) == 0) phase ^= 1u;
      }
      if (!ok) break;
      const int f = (u / p.tiles_t) * 2 * W_ROWS + (int)rank * W_ROWS + quarter * 32 + lane;
      const int t0 = (u % p.tiles_t) * p.tn;
      if (p.shares > 1) {  // the only tile: its sums wait in shared memory, [token][weight row]
        float* mine = reinterpret_cast<float*>(tiles) + quarter * 32 + lane;
#pragma unroll
        for (int g = 0; g < RUNS; ++g) {
          const int c = (2 * g + which) * 16;
          if (c >= p.tn) break;
#pragma unroll
          for (int e = 0; e < 16; ++e) mine[(c + e) * W_ROWS] = acc[g][e];
        }
      } else if (f < p.N) {
        uint32_t fell = 0;
#pragma unroll
        for (int g = 0; g < RUNS; ++g) {
          const int c = (2 * g + which) * 16;
          if (c >= p.tn) break;
          bool whole = true;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int t = t0 + c + e;
            if (t < p.M) {
              p.out[(long long)t * p.ldo + f] = acc[g][e];
              whole = whole && stands(acc[g][e]);
            }
          }
          if (!whole) fell |= 1u << (2 * g + which);
        }
        if (fell != 0) atomicOr(&fallen[round % ROUNDS], fell);
      }
    }
    if (p.shares > 1) {
      shares_meet();  // every share's sums are in place
      const int f = (cluster / p.tiles_t) * 2 * W_ROWS + (int)rank * W_ROWS + quarter * 32 + lane;
      const int t0 = (cluster % p.tiles_t) * p.tn, tokens = min(p.tn, p.M - t0);
      uint32_t from[MAX_SHARES];
#pragma unroll
      for (int i = 0; i < MAX_SHARES; ++i)
        from[i] = cluster_address(tiles, (uint32_t)min(i, p.shares - 1) * 2 + rank);
      uint32_t fell = 0;
      // every pair stores its tokens of the tile: the sums of all shares, in their order
#pragma unroll 4
      for (int t = (int)share * 2 + which; t < tokens; t += ctas) {
        const uint32_t at = (uint32_t)(t * W_ROWS + quarter * 32 + lane) * 4;
        float v = ld_cluster(from[0] + at);
#pragma unroll
        for (int i = 1; i < MAX_SHARES; ++i)
          if (i < p.shares) v += ld_cluster(from[i] + at);
        if (f < p.N) {
          p.out[(long long)(t0 + t) * p.ldo + f] = v;
          if (!stands(v)) fell |= 1u << (t >> 4);
        }
      }
      if (fell != 0)  // every pair repairs some runs of the tile, whoever stored them
        for (int i = 0; i < p.shares; ++i)
          or_cluster(cluster_address(&fallen[0], (uint32_t)i * 2 + rank), fell);
    }
    roles_meet();
    if (!*abort_flag) {
      // A result of 2^-64 and more stands by itself while K terms of 2^-102 of the largest operands stay
      // below that (a first piece is off by 2^-8 at most); else every result is looked at.
      const float most = __uint_as_float(largest[0]) + __uint_as_float(largest[1]);
      const bool all = !((float)p.K * (1.01f * most + 8.f) < 274877906944.f);  // 2^38
      RepairRoom& room = *reinterpret_cast<RepairRoom*>(tiles);
      round = 0;
      for (int u = cluster; u < p.units; u += clusters, ++round) {
        const uint32_t fell = all ? (1u << (p.tn / 16)) - 1u : fallen[round % ROUNDS];
        if (fell == 0) continue;
        const int f0 = (u / p.tiles_t) * 2 * W_ROWS + (int)rank * W_ROWS, t0 = (u % p.tiles_t) * p.tn;
        const int me = warp - 4 - SPLIT_WARPS, tid = me * 32 + lane;
        // Mostly zeros of tokens of zeros (padding, in a step), which one look at those settles. (Where a
        // weight is infinite, such a token's results are NaN, by pieces as by FMAs.)
        any_of_sums(false);  // the tile before is done
        if (tid < TOKEN_WORDS) busy[tid] = 0;
        if (tid < W_ROWS / 32) room.known[tid] = 0;
        if (tid == 0) odd = 0;
        any_of_sums(false);
#pragma unroll 1
        for (int t = me; t < p.tn && t0 + t < p.M; t += SUM_WARPS)
          if ((fell >> (t >> 4) & 1u) && (t >> 4) % p.shares == (int)share &&
              !is_zero_row(p.x + (long long)(t0 + t) * p.ldx, p.K, lane) && lane == 0)
            atomicOr(&busy[t >> 5], 1u << (t & 31));
        any_of_sums(false);
#pragma unroll 1
        for (int run = (int)share; fell >> run != 0; run += p.shares)
          if ((fell >> run & 1u) && (busy[run >> 1] >> (16 * (run & 1)) & 0xffffu) != 0) {
            bool mine = false;
#pragma unroll
            for (int e = 0; e < 8; ++e)
              mine = mine || falls_maybe(p, busy, all, f0 + tid % W_ROWS, t0, run * 16 + tid / W_ROWS * 8 + e);
            if (mine) atomicOr(&odd, 1u << run);
          }
        any_of_sums(false);
        const uint32_t left = odd;
        for (int run = (int)share; left >> run != 0; run += p.shares)
          if (left >> run & 1u) repair(p, room, busy, all, f0, t0, run * 16);
      }
    }
  }
}

// A [rows, cols] float32 matrix in boxes of box_rows x 32 with the 128-byte swizzle; out-of-range
// elements read 0.
int make_map_f32(CUtensorMap* map, const void* ptr, long long rows, long long cols, long long ld,
                 int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fb_fail(3, "gemm_f32: cuTensorMapEncodeTiled is not available in this driver");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {(cuuint32_t)KB, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(ptr), dims, strides, box,
                  elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fb_fail(3, "gemm_f32: cuTensorMapEncodeTiled failed with %d", (int)r);
  return 0;
}

}  // namespace

int fb_gemm_f32_tc_launch(const FbGemmF32& p, cudaStream_t stream) {
  bind_status_mirror(stream);
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM_DYNAMIC;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // Tiles of 256 weight rows and about 128 tokens (fewer don't take less time, see below); where
  // they occupy half of the pairs or fewer, several share a tile's K, if each keeps 16 stages of it.
  // Rows count in whole 128s, so that a step padded to a bucket sums as the plain one does.
  const int tiles_w = (p.N + 2 * W_ROWS - 1) / (2 * W_ROWS), stages_k = (p.K + KB - 1) / KB;
  const long long natural = (long long)tiles_w * ((p.M + 127) / 128);
  int shares = (int)(sm_count() / 2 / natural);
  if (shares > stages_k / 16) shares = stages_k / 16;
  shares = shares > MAX_SHARES ? MAX_SHARES : shares < 1 ? 1 : shares;
  attr[0].val.clusterDim.x = 2 * shares;

  static int clusters_of_device[64][MAX_SHARES] = {};  // clusters that run at once
  int device = 0;
  cudaGetDevice(&device);
  if (device < 0 || device >= 64) device = 63;
  int& clusters_max = clusters_of_device[device][shares - 1];
  if (clusters_max == 0) {
    cudaFuncAttributes have;
    cudaError_t e = cudaFuncGetAttributes(&have, gemm_f32_pair_kernel);
    if (e != cudaSuccess) return fb_fail(2, "gemm_f32: attributes: %s", cudaGetErrorString(e));
    if (have.numRegs * (THREADS / 128) < REGS_ALL) return FB_GEMM_F32_NOT_HERE;  // the roles would wait
    e = cudaFuncSetAttribute(gemm_f32_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)cfg.dynamicSmemBytes);
    if (e != cudaSuccess)
      return fb_fail(2, "gemm_f32: shared memory opt-in: %s", cudaGetErrorString(e));
    cfg.gridDim = dim3(sm_count() / (2 * shares) * (2 * shares));
    cfg.numAttrs = 1;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, gemm_f32_pair_kernel, &cfg);
    if (e != cudaSuccess) return fb_fail(2, "gemm_f32: occupancy: %s", cudaGetErrorString(e));
    if (n <= 0) return FB_GEMM_F32_NOT_HERE;
    clusters_max = n;
  }
  // Tokens of a tile: the count that costs the fewest rounds times a stage's time, which is 6 * tn
  // cycles of the tensor pipe, but no less than the issuing warp needs for a stage, about 700. A
  // result does not depend on it.
  int tn = 0;
  long long best = 0;
  for (int cuts = (p.M + MAX_TN - 1) / MAX_TN; cuts <= (p.M + 31) / 32; ++cuts) {
    const int size = ((p.M + cuts - 1) / cuts + 15) / 16 * 16;
    const long long rounds = ((long long)tiles_w * cuts + clusters_max - 1) / clusters_max;
    const long long cost = rounds * (6 * size > 700 ? 6 * size : 700);
    if (tn == 0 || cost < best) {
      best = cost;
      tn = size;
    }
  }
  if (tn < 32) tn = 32;
  Params q = {p.x, p.w, p.out, p.M, p.N, p.K, p.ldx, p.ldw, p.ldo, tn, (p.M + tn - 1) / tn, 0, 0, 0,
              shares};
  q.units = tiles_w * q.tiles_t;
  q.piece_stages = (TMEM_COLS - 2 * tn) / (PIECES * W_PIECE_COLS);
  if (q.piece_stages > MAX_PIECE_STAGES) q.piece_stages = MAX_PIECE_STAGES;
  q.stages = (SMEM_TILES - q.piece_stages * piece_bytes(tn)) / raw_bytes(tn);
  if (q.stages > MAX_STAGES) q.stages = MAX_STAGES;
  CUtensorMap mw, mx;
  int rc = make_map_f32(&mw, p.w, p.N, p.K, p.ldw, W_ROWS);
  if (!rc) rc = make_map_f32(&mx, p.x, p.M, p.K, p.ldx, tn / 2);
  if (rc) return rc;
  const int clusters = shares > 1 || q.units < clusters_max ? q.units : clusters_max;
  cfg.gridDim = dim3(2 * shares * clusters);
  cfg.numAttrs = g_fb_pdl ? 2 : 1;
  cudaLaunchKernelEx(&cfg, gemm_f32_pair_kernel, mw, mx, q);
  return fb_check_launch("gemm_f32_pair");
}

// As fb_gemm_tc_status, for the kernel of this file.
FB_API int fb_gemm_f32_status(int* detail) {
  int host[4] = {0, 0, 0, 0};
  cudaError_t e = cudaMemcpyFromSymbol(host, g_status, sizeof(host));
  if (e != cudaSuccess) return fb_fail(2, "gemm_f32_status: %s", cudaGetErrorString(e));
  if (detail) { detail[0] = host[1]; detail[1] = host[2]; detail[2] = host[3]; }
  if (host[0]) {
    int zero[4] = {0, 0, 0, 0};
    cudaMemcpyToSymbol(g_status, zero, sizeof(zero));
  }
  return host[0] ? host[1] : 0;
}
