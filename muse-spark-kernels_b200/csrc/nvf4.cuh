// Grouped GEMMs of the routed experts on the FP4 tensor cores, for token tiles of up to 16 rows: both GEMMs in one
// cooperative launch behind the sort.
//
// D[128 weight rows, N columns] = W[128, K] * B[N, K]^T with tcgen05.mma.kind::mxf4nvf4 (E2M1 operands, one E4M3 scale per 16
// K). The packed weights are that operand already: a stage of the ring goes from memory to the tensor core as it lies (octet
// blocks are the core matrices of an unswizzled K-major operand), only its scale bytes pass through registers into TMEM. No weight
// is decoded, so the kernel keeps pace with memory: the tcgen05 kernel of gemm.cuh, which decodes to F16 and passes every half
// stage through a TMEM slot, needs 1500 cycles and more for a stage that memory delivers in 1400, and power for it: long rows of
// steps run into the card's limit, where its clock falls. 64 tokens, all of 128 experts (1.3 GB), both GEMMs: 230 us there, 208 here; a
// row of whole steps 279 and 241 (both sides of the other sizes: nv_takes() in msk_moe.cu). Bound by memory, some 7.1 TB/s between the
// first MMA and the last, and by the 11 to 13 us before it (tables, split of the token rows) and 4 after.
//
// Activations enter exactly as in the F16 kernels: every F16 value, whatever lies beside it (tested bit for bit). A token row becomes nine E2M1
// rows of its own, the digits of a fixed-point number: in a block of 16 K an element is x = 2^u * (d0 + d1 / 8 + ... + d8 / 8^8), digits
// -4 .. 3 (the first to 4), which E2M1 holds exactly (as d / 2). The block's 2^u is its E4M3 scale, one byte for all nine rows; 8^-p is applied to
// the FP32 accumulators, which each digit has to itself, in the epilogue. These 27 bits hold all F16 values of blocks with magnitudes below 4, and
// BF16 values down to 2^-17 of the block's largest. What is left over of others, whole steps of 2^-24, is split in the same way with the
// scale 2^-9: its last two digits as a second level, four more as a third one that only blocks with magnitudes from 128 on can need.
// Levels add up in the accumulators of their digits, so a K stage with such an element has another pass of MMAs on the same weights. Which
// stages have one is kept in words per tile. Products are exact and accumulate in FP32. Measured against 64 bits (relative 2-norm of the raw
// down sums, K = 1536, this / the F16 form): SwiGLU values 3.7e-8 / 9.0e-7; beside channels 100 times as large that the weights ignore
// 4.1e-8 / 8.3e-7. (Seven digits and no levels lost bits beside large channels: 1.0e-4 there. Eight digits, with tiles of up to 24 rows:
// a third of the K stages of SwiGLU values have a second level, whole steps of 64 tokens 234 us for 229 now; a few experts taking most tokens,
// 8 tokens 67 for 64, 32 tokens 96 for 92.)
// NaN elements make the block's scale NaN; weight scales with a sign bit (no quantiser writes them) turn the signs of their
// 16 codes in shared memory, because the hardware's scales are unsigned.
//
// Per CTA (512 threads, one CTA per SM):
//   warp 0       draws units from a counter and streams their weights: one bulk copy per K stage (two tiles of 128 rows) into a ring;
//   warp 1       MMA issuer (and TMEM allocation): per pass 2 tiles x 4 MMAs of 64 K, one commit;
//   warp 2       token rows of the unit's tile, split and laid out beforehand: one bulk copy per K stage and level;
//   warps 4-7    scales: shared memory -> TMEM, each warp for its lane quarter (the hardware wants four copies);
//   warps 8-11   epilogue: digits summed, SwiGLU / scale, rows to global memory;
//   warp 3       counts stored gate/up units for their tiles;
//   warps 12-15  split `inter`: pieces of two to eight rows x 256 columns of a token tile, dealt over the CTAs in the order of the tiles, as each tile's
//                gate/up units are all stored. Whole tiles, split by the CTA that stored their last unit, kept a rank's 24-token step waiting
//                for some 20 us.
// Warps 4-15 first split the token rows, a row or a part of one per CTA at a time, while the first weights are on their way.
//
// Work is dealt one unit at a time, gate/up units before down units, as in pair.cuh (but a unit is drawn while the weights of the one before it are
// fetched, not further ahead); a down unit waits for its tile's rows. Units of an expert with several tiles are ordered pair
// first, so that the second tile finds the weights in L2.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "gemm.cuh"
#include "layout.cuh"
#include "ptx.cuh"

namespace msk {

constexpr int NV_THREADS = 512;
constexpr int NV_ROWS = 16;                                // most token rows of a tile
constexpr int NV_PARTS = 9;                                // digits of an activation
// Levels of a K stage of eight token rows (1 KB a digit, 128 bytes of scales each): their digits, the accumulators of the first
// one, their place in the stage.
constexpr int NV_LEVELS = 3;
__host__ __device__ constexpr int nv_digits(int level) { return level == 0 ? NV_PARTS : level == 1 ? 2 : 4; }
__host__ __device__ constexpr int nv_first(int level) { return level == 0 ? 0 : level == 1 ? 6 : 2; }
__host__ __device__ constexpr int nv_level_at(int level) { return level == 0 ? 0 : level == 1 ? nv_digits(0) * 1024 + 128 : (nv_digits(0) + nv_digits(1)) * 1024 + 256; }
constexpr int NV_LEVEL_BYTES = nv_level_at(1);             // of the first level, the widest
constexpr int NV_GROUP_BYTES = nv_level_at(2) + nv_digits(2) * 1024 + 128;   // eight token rows x 256 K
constexpr int NV_W_STAGES = 4, NV_S_STAGES = 2;            // rings: weights, scales in TMEM
constexpr int NV_MARKS = 8;                                // passes whose MMAs have a barrier of their own
constexpr int NV_UNITS = 4;
constexpr int NV_SPLIT_WARP = 4, NV_SPLIT_THREADS = NV_THREADS - NV_SPLIT_WARP * 32;
constexpr int NV_MAX_BLOCKS = 512;                         // blocks of 16 K in a token row: H <= 8192
constexpr int NV_CONV_WARPS = 4;
constexpr int NV_AHEAD = 8;                                // stages of the first unit that are fetched to L2 ahead of the ring

// Token tiles of an expert with c rows: even shares in steps of 8. Width of a tile: its groups of eight rows.
__host__ __device__ inline int nv_tiles(int c) { return (c + NV_ROWS - 1) / NV_ROWS; }
__host__ __device__ inline int nv_tile_rows(int c, int n) { return n <= 1 ? c : ((c + n - 1) / n + 7) & ~7; }
__host__ __device__ inline int nv_width(int rows) { return (rows + 7) >> 3; }
// Rows that its image and its MMAs have room for: up to four rows take four. (The second level's two digits of four rows are the narrowest MMA; room for
// twelve needs scale columns of their own and was 1 to 2 % slower.) With room for eight only, a row of steps in turn on one box, before / after: 8
// tokens 106.4 / 103.7 us, 16: 163.8 / 159.2, 32: 214.9 / 209.9, 64: 242.6 / 238.2; fewer columns and token rows' bytes, and with them less power.
__host__ __device__ inline int nv_room(int rows) { return rows <= 4 ? 4 : 8 * nv_width(rows); }
// Groups that the image of an expert's rows takes: all tiles but the last have whole ones.
constexpr int NV_GROUPS = NV_ROWS / 8;
__host__ __device__ inline int nv_groups(int c) { return nv_width(c); }
// Rows of a piece of inter (x 256 columns), as a power of two, given how many pieces eight rows would make: eight, or two while there are as
// many warps as half of those to split them. Two rows take a warp 2 us, eight 7, for which the down units of a step of few tiles stood still
// (a few experts taking most tokens, 12: 68.4 -> 65.5 us a step, 24: 83.6 -> 81.0; four rows in between gained nothing, 32: 89.9 -> 90.4).
__device__ __forceinline__ int nv_piece_bits(int eights, int n_ctas) { return eights * 2 <= NV_CONV_WARPS * n_ctas ? 1 : 3; }
// A bound on their sum over experts with `rows` rows in all: nv_groups(c) <= 1 + (c - 1) / 8.
inline size_t nv_groups_bound(size_t rows, size_t experts) {
  const size_t e = rows < experts ? rows : experts;
  return e + (rows - e) / 8;
}

// Counters of a tile, a cache line for each: CTAs that wait for a tile poll another line than those that count for its neighbours.
constexpr int NV_TILE_WORDS = 64;
enum : int {
  NV_DONE = 0,     // stored gate/up units
  NV_READY = 8,    // pieces of inter that are split, of two rows each or four times that
  NV_SEEN = 16,    // down units that have fetched them all
  NV_MORE = 32,    // bit per K stage, a word for 32 of them: stages with a second level, a third level; token rows, then inter
  NV_MORE_INTER = NV_MORE + 2 * (NV_MAX_BLOCKS * 16 / KS / 32),
};
constexpr int NV_MAX_INTER = (NV_TILE_WORDS - NV_MORE_INTER) / 2 * 32 * KS;   // 122880

struct NvParams {
  const uint8_t* w[2];
  const float* gs[2];
  const __nv_bfloat16* x;                // [T, H]
  const __nv_bfloat16* pre_w;            // nullable: pre-expert RMS norm
  const int32_t* ids;                    // [T, k]
  const int32_t* inv;                    // [T, k]
  const int32_t* cnt;
  const int32_t* off;
  const __nv_bfloat16* post_norm_w;      // nullable
  __half* inter;                         // [R, I]
  float* y;                              // [R, H]
  uint8_t* img[2];                       // split rows (see the split below): token rows, rows of inter
  int32_t* status;
  unsigned long long* trace;
  unsigned int* ctr;                     // [0] units drawn, [1] CTAs that have left, [2] CTAs that have split their token rows
  unsigned int* tiles;                   // NV_TILE_WORDS a tile: NV_DONE and so on, all zero between launches
  float pre_eps;
  int K[2], n_pairs[2];
  int nloc, lo, H, I, T, k;
  int share_rows;                        // a token row may be read by several CTAs
};

struct alignas(16) NvUnit {
  int phase;                             // -1: no more units
  int expert, row0, rows, pair, tile;
  int group, width;                      // its tile's place in the image, in groups of eight rows, and how many of them it is wide
};

struct NvCtrl {
  uint64_t w_full[NV_W_STAGES], b_full[NV_MARKS], s_full[NV_S_STAGES];
  uint64_t done[NV_MARKS];               // the MMAs of pass n (n % 8): its places for scales and token rows are free
  uint64_t w_done[NV_W_STAGES];          // those of a stage's last pass: its weights' place is
  uint64_t d_full[2], d_empty[2];
  uint64_t u_full[NV_UNITS], u_empty[NV_UNITS];
  uint64_t stored[NV_UNITS];             // the epilogue has stored its values of a unit
  NvUnit unit[NV_UNITS];
  uint4 route[MAX_TOP_K];                // of the token row that is split: place of its digits in the image, its tile's room, tile, row in it
  float red[NV_SPLIT_THREADS / 32];
  int n_routes;
  uint32_t tmem_base;
  int abort_word;
  int b_stages, b_bytes;                 // ring of token rows: places, bytes of one
  int b_pass[NV_MARKS];                  // what a place holds: its level, and NV_LAST in the last pass of a K stage
};
static_assert(sizeof(NvCtrl) <= 1024 && offsetof(NvCtrl, unit) % 16 == 0, "control block");

constexpr int NV_LAST = 4;
__host__ __device__ constexpr int nv_place_bytes(int room) { return (room * (NV_LEVEL_BYTES / 8) + 1023) / 1024 * 1024; }

struct NvCfg {
  static constexpr int TABLE_INTS = MAX_LOCAL_EXPERTS + 4;
  // The ring of token rows has places for the widest tile of the launch (whole swizzle atoms of 1 KB): 4 of them, 7 where no tile has more than eight rows, 8 (as
  // many as there are marks) where none has more than four. (Places of each pass's
  // own size, more of them: 1 % slower; three of them, and three stages of weights ahead: 2 %.)
  static constexpr int B_RING = 76 * 1024;
  static constexpr int W_OFF = 0, B_OFF = NV_W_STAGES * STAGE_W_BYTES, CTL_OFF = B_OFF + B_RING, TABLE_OFF = CTL_OFF + 1024;
  static constexpr int SMEM_BYTES = TABLE_OFF + 4 * TABLE_INTS * 4;
  static_assert(SMEM_BYTES <= 232448 && 4 * nv_place_bytes(NV_ROWS) <= B_RING, "shared memory of a CTA");
  // TMEM: accumulators of two tiles (digits x rows columns each; those of a tile of eight rows twice), two stages of scales
  static constexpr int D_WIDE = NV_PARTS * NV_ROWS, D_NARROW = NV_PARTS * 8;
  static constexpr int S_BASE = 2 * D_WIDE, S_COLS = 32, S_B = S_BASE + NV_S_STAGES * S_COLS;   // 4 x 4 columns per weight tile, 4 x 8 for the token rows
  static_assert(4 * D_NARROW <= S_BASE && (D_WIDE + 31) / 32 <= 8, "TMEM layout");
  static_assert(S_B + NV_S_STAGES * S_COLS <= TMEM_COLS, "TMEM budget");
};

__host__ __device__ constexpr uint32_t idesc_nvf4(uint32_t N) {   // E2M1 x E2M1, E4M3 scales, M = 128
  return (1u << 7) | (1u << 10) | ((N >> 3) << 17) | (8u << 24);
}
// D[tmem] (+)= A[smem, 128 x 256] * B[smem, N x 256]^T for the two tiles of a stage, four MMAs of 64 K each: a scale per row and 16 K in
// TMEM, lane r % 32 (in every lane quarter), column r / 32, the four bytes of 64 K. `sf`: 4 x 4 columns of tile 0, of tile 1, 4 x 8 of the
// token rows. By one elected lane, with the commit that hands the pass's places back (done_bar) and, with `last`, the one for the weights
// (w_done_bar); the answer of a probe of `next_full` (true: complete) is asked for before the MMAs and read behind them. In one block of assembly: as separate calls in a branch of that lane
// the operands went to the issue unit one by one, some 150 cycles an MMA.
#define NV_MMA "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X"
__device__ __forceinline__ bool mma_nvf4_stage(uint32_t d0, uint32_t d1, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate,
                                               uint32_t done_bar, uint32_t w_done_bar, uint32_t last, uint32_t next_full, uint32_t parity) {
  static_assert(OCT_BYTES / 16 == 72, "the second tile's octet blocks");
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred q, e, acc, t, l;\n\t.reg .b64 a, b, c;\n\t.reg .b32 f, g, h;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%9], %10;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 acc, %8, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 a, %3;\n\tmov.b64 b, %4;\n\tmov.b32 f, %6;\n\tmov.b32 g, %13;\n\t"
      "@e " NV_MMA " [%1], a, b, %5, [f], [g], acc;\n\t"
      "add.s64 c, a, 72;\n\tadd.u32 h, f, 16;\n\t"
      "@e " NV_MMA " [%2], c, b, %5, [h], [g], acc;\n\t"
      "add.s64 a, a, 16;\n\tadd.s64 b, b, 2;\n\tadd.u32 f, f, 4;\n\tadd.u32 g, g, 8;\n\t"
      "@e " NV_MMA " [%1], a, b, %5, [f], [g], t;\n\t"
      "add.s64 c, a, 72;\n\tadd.u32 h, f, 16;\n\t"
      "@e " NV_MMA " [%2], c, b, %5, [h], [g], t;\n\t"
      "add.s64 a, a, 16;\n\tadd.s64 b, b, 2;\n\tadd.u32 f, f, 4;\n\tadd.u32 g, g, 8;\n\t"
      "@e " NV_MMA " [%1], a, b, %5, [f], [g], t;\n\t"
      "add.s64 c, a, 72;\n\tadd.u32 h, f, 16;\n\t"
      "@e " NV_MMA " [%2], c, b, %5, [h], [g], t;\n\t"
      "add.s64 a, a, 16;\n\tadd.s64 b, b, 2;\n\tadd.u32 f, f, 4;\n\tadd.u32 g, g, 8;\n\t"
      "@e " NV_MMA " [%1], a, b, %5, [f], [g], t;\n\t"
      "add.s64 c, a, 72;\n\tadd.u32 h, f, 16;\n\t"
      "@e " NV_MMA " [%2], c, b, %5, [h], [g], t;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
      "setp.ne.and.b32 l, %12, 0, e;\n\t"
      "@l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%11];\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(d0), "r"(d1), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(done_bar), "r"(accumulate), "r"(next_full), "r"(parity), "r"(w_done_bar), "r"(last), "r"(sfb)
      : "memory");
  return ok != 0u;
}
#undef NV_MMA

// ---- the split. Image of a tile (room for R rows, K): per K stage of 256 and level, digits [9, 2 or 4][R rows][128 bytes], the eight
// 16-byte chunks of a row in the order of the 128-byte swizzle (chunk c of row n = digit * R + r at c ^ (n & 7): a row's digit is one line to
// write), then scales [R rows][16]; one contiguous copy a level, NV_GROUP_BYTES / 8 * R bytes a stage.
__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((e + 127) << 23); }
constexpr int NV_MAX_EXP = 14;   // of a block's unit: 65504 is below four of 2^14
constexpr int NV_MIN_EXP = 0;    // its ninth digit is a step of 2^-24, the smallest there is
constexpr float NV_SUM_SCALE = 128.f;   // what sums are multiplied by: units of 2^14 have scale 2^8, and codes are d / 2

// Largest magnitude of sixteen values; NaN if one of them is.
__device__ __forceinline__ float nv_block_max(const uint32_t (&h)[8]) {
  __half2 m = __habs2(*reinterpret_cast<const __half2*>(&h[0]));
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax2_nan(m, __habs2(*reinterpret_cast<const __half2*>(&h[i])));
  return __half2float(__hmax_nan(__low2half(m), __high2half(m)));
}

// d digits of -4 .. 3 that are all 4 in the bits of a number: what is added so that they come out as 0 .. 7.
__host__ __device__ constexpr uint32_t nv_bias(int d) { return ((1u << (3 * d)) - 1u) / 7u * 4u; }

struct NvBlock {
  int u;              // its unit is 2^u, the smallest with its largest magnitude below four units (as far as NV_MIN_EXP)
  uint32_t scale;     // as E4M3
  uint32_t levels;    // bit per level that it needs
};
// Sixteen values -> for each the number of steps of 2^-24 units nearest to it, biased: digits + 4 in three bits each, the first of 0 .. 8.
// What is left is at most half a step, 2^13 steps of 2^-24: the lowest two digits of that number are the second level, the four above
// them the third.
__device__ __forceinline__ NvBlock nv_fixed16(const uint32_t (&h)[8], uint32_t (&f)[16]) {
  NvBlock k;
  const float bm = nv_block_max(h);
  k.u = min(max((__float_as_int(bm) >> 23) - 128, NV_MIN_EXP), NV_MAX_EXP);
  const float scale = exp2_int(3 * (NV_PARTS - 1) - k.u);
  float hi = 0.f, lo = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
    const float x0 = v.x * scale, x1 = v.y * scale;
    const int q0 = __float2int_rn(x0), q1 = __float2int_rn(x1);
    f[2 * i] = static_cast<uint32_t>(q0) + nv_bias(NV_PARTS);
    f[2 * i + 1] = static_cast<uint32_t>(q1) + nv_bias(NV_PARTS);
    const float r0 = x0 - static_cast<float>(q0), r1 = x1 - static_cast<float>(q1);
    hi = fmaxf(hi, fmaxf(r0, r1));
    lo = fminf(lo, fminf(r0, r1));
  }
  const float steps = exp2_int(k.u - NV_MIN_EXP);
  k.levels = bm != bm || (hi == 0.f && lo == 0.f) ? 1u : hi * steps <= 27.f && lo * steps >= -36.f ? 3u : 7u;
  const int e = k.u - (NV_MAX_EXP - 8);
  k.scale = bm != bm ? 0x7Fu : e >= -6 ? static_cast<uint32_t>(e + 7) << 3 : 1u << (e + 9);
  return k;
}
// The number of steps of 2^-24 that is left of each, biased by six digits.
__device__ __forceinline__ void nv_rest16(const uint32_t (&h)[8], int u, uint32_t (&f)[16]) {
  const float scale = exp2_int(3 * (NV_PARTS - 1) - u), steps = exp2_int(u - NV_MIN_EXP);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
    const float x0 = v.x * scale, x1 = v.y * scale;
    f[2 * i] = static_cast<uint32_t>(__float2int_rn((x0 - rintf(x0)) * steps)) + nv_bias(6);
    f[2 * i + 1] = static_cast<uint32_t>(__float2int_rn((x1 - rintf(x1)) * steps)) + nv_bias(6);
  }
}
// The last digits of the sixteen (bits `mask` of the numbers) as E2M1 codes, a nibble each; the numbers lose three bits.
__device__ __forceinline__ uint2 nv_next_digit(uint32_t (&f)[16], uint32_t mask) {
  uint32_t q[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t t = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      t += (f[8 * c + i] & mask) * (1u << (4 * i));
      f[8 * c + i] >>= 3;
    }
    const uint32_t pos = (((t >> 2) | (t >> 3)) & 0x11111111u) * 15u;   // nibbles of digits >= 0: the digit; of the others: sign and magnitude 4 - t
    q[c] = (((t & 0x33333333u) | ((t >> 1) & 0x44444444u)) & pos) | ((0xCCCCCCCCu - t) & ~pos);
  }
  return make_uint2(q[0], q[1]);
}
// A lane's block (where `mine`; called by whole warps): put(0, digit, codes) for `n` digits of the first level, the last of them `to` - 1, and where
// `rest` put_scales(bytes of the three levels, 0 for one that it does not need) and put(level, digit, codes) for the others. more1, more2: the
// lanes whose blocks have a second, a third level. (The loops over the digits are not unrolled: this code runs from a cold instruction cache
// while the weights stream, where a line takes a microsecond; all digits in line made the steps 5 to 20 us longer.)
template <class PutScales, class Put>
__device__ __forceinline__ void nv_split_block(const uint32_t (&h)[8], bool mine, int n, int to, bool rest, unsigned& more1, unsigned& more2,
                                               PutScales put_scales, Put put) {
  uint32_t f[16];
  const NvBlock k = nv_fixed16(h, f);
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] >>= 3 * (NV_PARTS - to);
  more1 = __ballot_sync(0xffffffffu, mine && rest && (k.levels & 2u) != 0u);
  more2 = __ballot_sync(0xffffffffu, mine && rest && (k.levels & 4u) != 0u);
  if (mine && rest) put_scales(k.scale, (k.levels >> 1) & 1u, k.levels >> 2);
  const int levels = more2 != 0u ? 3 : more1 != 0u ? 2 : 1;   // (a third level has a second one in front)
#pragma unroll 1
  for (int level = 0; level < levels; ++level) {
    if (level > 0) {
      n = to = nv_digits(level);
      mine = mine && rest;
      if (level == 1) nv_rest16(h, k.u, f);
    }
    const bool has = mine && ((k.levels >> level) & 1u) != 0u;
#pragma unroll 1
    for (int i = 1; i <= n; ++i) {
      const uint2 w = nv_next_digit(f, level == 0 && i == to ? 15u : 7u);
      if (has) put(level, to - i, w);
    }
  }
}

// Where a row of a tile lies in a digit, a block's codes in its row, its scale in a level.
__device__ __forceinline__ int nv_digit_at(int room, int level, int d) { return room * (nv_level_at(level) / 8 + d * 128); }
__device__ __forceinline__ int nv_code_at(int room, int level, int d, int slot, int blk) {
  return nv_digit_at(room, level, d) + slot * 128 + (((blk & 15) >> 1) ^ ((d * room + slot) & 7)) * 16 + (blk & 1) * 8;
}
__device__ __forceinline__ int nv_scale_at(int room, int level, int slot, int blk) {
  return nv_digit_at(room, level, nv_digits(level)) + slot * 16 + (blk & 15);
}

// Which accumulators the units take in turn: tiles of up to eight rows one or the other, wider ones both (as PairBuffers).
struct NvBuffers {
  uint32_t next = 0, par0 = 0, par1 = 0;
  bool wide;
  uint32_t buf, p0, p1;
  __device__ __forceinline__ void take(int width) {
    wide = width > 1;
    buf = wide ? 0u : next;
    p0 = par0;
    p1 = par1;
    if (wide || buf == 0u) par0 ^= 1u;
    if (wide || buf == 1u) par1 ^= 1u;
    next = wide ? 0u : (next ^ 1u);
  }
  __device__ __forceinline__ bool uses(uint32_t b) const { return wide || buf == b; }
  __device__ __forceinline__ uint32_t col() const { return buf * 2 * NvCfg::D_NARROW; }
  __device__ __forceinline__ uint32_t tile_cols() const { return wide ? NvCfg::D_WIDE : NvCfg::D_NARROW; }
};

// grid_counter_wait for the warps that wait through most of the gate/up phase: they look less often.
__device__ __forceinline__ bool nv_tile_wait(const unsigned int* ctr, unsigned int target, volatile int* abort_word) {
  const uint64_t t0 = globaltimer_ns();
  uint32_t polls = 0;
  while (true) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
    if (v >= target) return true;
    __nanosleep(400);
    if ((++polls & 7u) == 0u) {
      if (*abort_word != 0) return false;
      if (globaltimer_ns() - t0 > MSK_WAIT_LIMIT_NS) {
        *abort_word = 1;
        return false;
      }
    }
  }
}

__global__ void __launch_bounds__(NV_THREADS, 1) moe_nvf4_kernel(const __grid_constant__ NvParams p) {
  using C = NvCfg;
  extern __shared__ __align__(1024) uint8_t nv_smem[];
  uint8_t* w_ring = nv_smem + C::W_OFF;
  uint8_t* b_ring = nv_smem + C::B_OFF;
  NvCtrl& ctl = *reinterpret_cast<NvCtrl*>(nv_smem + C::CTL_OFF);
  int* tile_start = reinterpret_cast<int*>(nv_smem + C::TABLE_OFF);   // per expert: first tile, first group, rows, first row
  int* group_start = tile_start + C::TABLE_INTS;
  int* cnt_s = group_start + C::TABLE_INTS;
  int* off_s = cnt_s + C::TABLE_INTS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_ctas = static_cast<int>(gridDim.x);

  // ---------------------------------------------------------------- set-up
  if (tid == 0) {
    MSK_TR(TR_START);
    for (int i = 0; i < NV_W_STAGES; ++i) {
      mbar_init(&ctl.w_full[i], 1);
      mbar_init(&ctl.w_done[i], 1);
    }
    for (int i = 0; i < NV_S_STAGES; ++i) mbar_init(&ctl.s_full[i], 4);
    for (int i = 0; i < NV_MARKS; ++i) {
      mbar_init(&ctl.b_full[i], 2);
      mbar_init(&ctl.done[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl.d_full[i], 1);
      mbar_init(&ctl.d_empty[i], 4);
    }
    for (int i = 0; i < NV_UNITS; ++i) {
      mbar_init(&ctl.u_full[i], 1);
      mbar_init(&ctl.u_empty[i], 11);   // MMA issuer, token rows, warp 3, four warps of scales, four of the epilogue
      mbar_init(&ctl.stored[i], 4);
    }
    ctl.abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl.tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  // The first token row (or its part) of this CTA, as F16 values: it does not depend on the sort, and the launch before the sort
  // has completed (the sort lets this launch begin only behind its own wait).
  constexpr int NT = NV_SPLIT_THREADS, NW = NT / 32, HALVES = NT / 16, PER = (NV_MAX_BLOCKS + NT - 1) / NT;
  const int th = tid - NV_SPLIT_WARP * 32, nb = p.H / 16;
  // up to 74 tokens several CTAs share a row: each reads all of it, as the norm needs, and splits some of the K stages (not over
  // PCIe, where every reader costs the bytes again: 8 rows in host memory, a whole step 121 us shared, 103 not, 119 by the other kernel)
  const int parts = p.share_rows ? max(1, min(n_ctas / p.T, p.H / KS)) : 1, items = p.T * parts;
  uint32_t h[PER][8];
  uint4* row_s = reinterpret_cast<uint4*>(b_ring);   // the row's F16 values, while no token row is fetched yet
  auto fetch_row = [&](int t) {
    const uint4* src = reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(t) * p.H);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = th + i * NT;
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u), v0 = b < nb ? src[2 * b] : zero, v1 = b < nb ? src[2 * b + 1] : zero;
      h[i][0] = v0.x; h[i][1] = v0.y; h[i][2] = v0.z; h[i][3] = v0.w;
      h[i][4] = v1.x; h[i][5] = v1.y; h[i][6] = v1.z; h[i][7] = v1.w;
    }
  };
  auto finish_row = [&]() {   // norm, F16 values
    if (p.pre_w != nullptr) {   // x * rsqrt(mean(x^2) + eps) * (1 + pre_w), one BF16 rounding (copy_rows_kernel)
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float lo = __uint_as_float(h[i][j] << 16), hi = __uint_as_float(h[i][j] & 0xFFFF0000u);
          ss += lo * lo + hi * hi;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) ctl.red[warp - NV_SPLIT_WARP] = ss;
      named_bar_sync(1, NT);
      float tot = 0.f;
#pragma unroll
      for (int i = 0; i < NW; ++i) tot += ctl.red[i];
      const float rs = rsqrtf(tot / static_cast<float>(p.H) + p.pre_eps);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int b = th + i * NT;
        if (b >= nb) continue;
        const uint4 g0 = __ldg(reinterpret_cast<const uint4*>(p.pre_w) + 2 * b), g1 = __ldg(reinterpret_cast<const uint4*>(p.pre_w) + 2 * b + 1);
        const uint32_t g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float lo = __uint_as_float(h[i][j] << 16) * rs * (1.0f + __uint_as_float(g[j] << 16));
          const float hi = __uint_as_float(h[i][j] & 0xFFFF0000u) * rs * (1.0f + __uint_as_float(g[j] & 0xFFFF0000u));
          const __nv_bfloat162 r = __floats2bfloat162_rn(lo, hi);
          h[i][j] = *reinterpret_cast<const uint32_t*>(&r);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = th + i * NT;
#pragma unroll
      for (int j = 0; j < 8; ++j) h[i][j] = bf16x2_to_f16x2(h[i][j]);
      if (b < nb) {
        row_s[2 * b] = make_uint4(h[i][0], h[i][1], h[i][2], h[i][3]);
        row_s[2 * b + 1] = make_uint4(h[i][4], h[i][5], h[i][6], h[i][7]);
      }
    }
  };
  if (warp >= NV_SPLIT_WARP && static_cast<int>(blockIdx.x) < items) {
    fetch_row(static_cast<int>(blockIdx.x) / parts);
    finish_row();
  }
  pdl_wait();
  pdl_launch_dependents();
  int q = -1, id = 0;                              // lane s of the first of these warps: route s of the row
  auto fetch_route = [&](int t) {
    if (th >= 0 && th < p.k) {
      q = __ldcg(p.inv + static_cast<size_t>(t) * p.k + th);
      id = __ldcg(p.ids + static_cast<size_t>(t) * p.k + th);
    }
  };
  if (static_cast<int>(blockIdx.x) < items) fetch_route(static_cast<int>(blockIdx.x) / parts);
  if (warp == 2) {   // exclusive prefixes of the experts' tiles and image groups
    constexpr int PE = (MAX_LOCAL_EXPERTS + 31) / 32;
    int cn[PE], of[PE], tiles = 0, groups = 0, most = 0;
#pragma unroll
    for (int i = 0; i < PE; ++i) {   // (all loads first: one round trip to memory)
      const int e = i * 32 + lane;
      cn[i] = e < p.nloc ? __ldcg(p.cnt + e) : 0;
      of[i] = e < p.nloc ? __ldcg(p.off + e) : 0;
    }
#pragma unroll
    for (int i = 0; i < PE; ++i) {
      const int e = i * 32 + lane;
      if (i * 32 >= p.nloc) break;
      most = max(most, cn[i]);
      int t = nv_tiles(cn[i]), g = nv_groups(cn[i]);
      const int t0 = t, g0 = g;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, t, o), b = __shfl_up_sync(0xffffffffu, g, o);
        if (lane >= o) { t += a; g += b; }
      }
      if (e < p.nloc) {
        tile_start[e] = tiles + t - t0;
        group_start[e] = groups + g - g0;
        cnt_s[e] = cn[i];
        off_s[e] = of[i];
      }
      tiles += __shfl_sync(0xffffffffu, t, 31);
      groups += __shfl_sync(0xffffffffu, g, 31);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) {
      tile_start[p.nloc] = tiles;
      group_start[p.nloc] = groups;
      ctl.b_bytes = nv_place_bytes(nv_room(min(most, NV_ROWS)));   // (no tile at all: places that nobody uses)
      ctl.b_stages = min(NV_MARKS, C::B_RING / ctl.b_bytes);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem = ctl.tmem_base;
  volatile int* abortw = &ctl.abort_word;
  const uint32_t b_stages = static_cast<uint32_t>(ctl.b_stages), b_bytes = static_cast<uint32_t>(ctl.b_bytes);
  if (tid == 0) MSK_TR(TR_SETUP);

  // Units, as every role behind the producer walks them. Whole warps wait with one outcome (mbar_wait_warp).
  uint32_t ui = 0;
  auto wait_unit = [&](NvUnit& u, auto wait) -> bool {
    const uint32_t s = ui % NV_UNITS;
    if (!wait(&ctl.u_full[s], (ui / NV_UNITS) & 1u, abortw)) return false;
    const int4 a = *reinterpret_cast<const int4*>(&ctl.unit[s]), b = *(reinterpret_cast<const int4*>(&ctl.unit[s]) + 1);
    u.phase = a.x; u.expert = a.y; u.row0 = a.z; u.rows = a.w;
    u.pair = b.x; u.tile = b.y; u.group = b.z; u.width = b.w;
    ++ui;
    return true;
  };
  auto done_unit = [&]() { mbar_arrive(&ctl.u_empty[(ui - 1u) % NV_UNITS]); };
  auto expert_of = [&](int tile) -> int {          // largest e with tile_start[e] <= tile
    int lo = 0, hi = p.nloc;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile_start[mid] <= tile) lo = mid; else hi = mid;
    }
    return lo;
  };
  auto set_tile = [&](NvUnit& u, int e, int ti) {   // tile ti of expert e
    const int c = cnt_s[e], per = nv_tile_rows(c, nv_tiles(c));
    u.expert = e;
    u.tile = tile_start[e] + ti;
    u.row0 = off_s[e] + ti * per;
    u.rows = min(per, c - ti * per);
    u.width = nv_width(u.rows);
    u.group = group_start[e] + ti * (per >> 3);
  };

  if (warp >= NV_SPLIT_WARP) {
    // ------------------------------------------------- split of the token rows
    int item = static_cast<int>(blockIdx.x);
    while (item < items) {
      const int part = item % parts, next = item + n_ctas;
      if (th < 32) {   // where its local routes' rows go
        const unsigned have = __ballot_sync(0xffffffffu, q >= 0);
        if (q >= 0) {
          const int e = id - p.lo, c = cnt_s[e], per = nv_tile_rows(c, nv_tiles(c)), r = q - off_s[e], ti = r / per, slot = r - ti * per;
          const int group = group_start[e] + ti * (per >> 3), room = nv_room(min(per, c - ti * per));
          ctl.route[__popc(have & ((1u << th) - 1u))] =
              make_uint4(static_cast<uint32_t>(group * (p.H / KS) * NV_GROUP_BYTES), static_cast<uint32_t>(room),
                         static_cast<uint32_t>(tile_start[e] + ti), static_cast<uint32_t>(slot));
        }
        if (th == 0) ctl.n_routes = __popc(have);
      }
      named_bar_sync(1, NT);
      const int n_routes = ctl.n_routes;
      if (next < items) {                          // on its way while this one is split
        fetch_row(next / parts);
        q = -1;
        fetch_route(next / parts);
      }
      // Half a warp to a K stage, a part of its routes and, with few tokens, a third of the digits: as many shares as there are half warps. (With the
      // thread that holds a block writing all its digits to all routes, 16 threads did 8 tokens' work: first MMA after 11.8 us, now 10.8; 64
      // tokens 14.5 and 13.2.)
      const int stages = (p.H / KS - part + parts - 1) / parts, by_route = max(1, min(HALVES / stages, n_routes));
      const int by_digit = HALVES / (stages * by_route) >= 3 ? 3 : 1, shares = n_routes != 0 ? stages * by_route * by_digit : 0;
#pragma unroll 1
      for (int first = (warp - NV_SPLIT_WARP) * 2; first < shares; first += HALVES) {
        const int share = min(first + (lane >> 4), shares - 1), j = share / stages, stage = part + (share - j * stages) * parts;
        const int third = j / by_route, r0 = j - third * by_route, b = stage * 16 + (lane & 15);
        const uint4 v0 = row_s[2 * b], v1 = row_s[2 * b + 1];
        const uint32_t g[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        auto at = [&](const uint4& to) { return p.img[0] + (to.x + to.y * static_cast<uint32_t>(stage * (NV_GROUP_BYTES / 8))); };
        unsigned more[2];
        nv_split_block(g, first + (lane >> 4) < shares, NV_PARTS / by_digit, NV_PARTS / by_digit * (third + 1), third == 0, more[0], more[1],
            [&](uint32_t s0, uint32_t s1, uint32_t s2) {
#pragma unroll 1
              for (int s = r0; s < n_routes; s += by_route) {
                const uint4 to = ctl.route[s];
                const int room = static_cast<int>(to.y), slot = static_cast<int>(to.w);
                uint8_t* img = at(to);
                img[nv_scale_at(room, 0, slot, b)] = static_cast<uint8_t>(s0);
                img[nv_scale_at(room, 1, slot, b)] = static_cast<uint8_t>(s1);
                img[nv_scale_at(room, 2, slot, b)] = static_cast<uint8_t>(s2);
              }
            },
            [&](int level, int d, uint2 w) {
#pragma unroll 1
              for (int s = r0; s < n_routes; s += by_route) {
                const uint4 to = ctl.route[s];
                *reinterpret_cast<uint2*>(at(to) + nv_code_at(static_cast<int>(to.y), level, d, static_cast<int>(to.w), b)) = w;
              }
            });
#pragma unroll
        for (int m = 0; m < 2; ++m) {              // (lane i of a half: its share's i-th route)
          const int s = r0 + (lane & 15) * by_route;
          if (((more[m] >> (lane & 16)) & 0xFFFFu) != 0u && s < n_routes)
            atomicOr(p.tiles + ctl.route[s].z * NV_TILE_WORDS + NV_MORE + m, 1u << stage);
        }
      }
      item = next;
      if (item < items) {
        named_bar_sync(1, NT);                     // the row's and the routes' places may be written again
        finish_row();
      }
    }
    named_bar_sync(1, NT);
    if (th == 0) {
      red_release_add(p.ctr + 2, 1u);   // (the image's readers put the fence between their acquire and their bulk copies)
      MSK_TR(TR_CONVERTED);
    }
  }

  if (warp == 0) {
    // ------------------------------------------------------- units and weights
    if (lane == 0) {
      const uint64_t pol = policy_evict_first();
      const int tiles = tile_start[p.nloc], n0 = tiles * p.n_pairs[0], n = n0 + tiles * p.n_pairs[1];
      uint32_t st = 0;                              // K stages
      auto publish = [&](NvUnit& u, uint32_t i, int x) -> bool {   // unit x becomes the i-th of this CTA
        u.phase = -1;
        if (x < n) {
          u.phase = x >= n0 ? 1 : 0;
          const int np = p.n_pairs[u.phase], v = u.phase ? x - n0 : x;
          const int e = expert_of(v / np), idx = v - tile_start[e] * np, nt = nv_tiles(cnt_s[e]);
          u.pair = idx / nt;
          set_tile(u, e, idx - u.pair * nt);
        }
        const uint32_t s = i % NV_UNITS;
        if (!mbar_wait_inline(&ctl.u_empty[s], ((i / NV_UNITS) & 1u) ^ 1u, abortw)) return false;
        *reinterpret_cast<int4*>(&ctl.unit[s]) = make_int4(u.phase, u.expert, u.row0, u.rows);
        *(reinterpret_cast<int4*>(&ctl.unit[s]) + 1) = make_int4(u.pair, u.tile, u.group, u.width);
        mbar_arrive(&ctl.u_full[s]);
        return true;
      };
      NvUnit u;
      bool ok = publish(u, 0u, static_cast<int>(blockIdx.x));   // the first unit, then what the counter gives
      for (uint32_t i = 0; ok && u.phase >= 0; ++i) {
        const int x = n_ctas + static_cast<int>(atomicAdd(p.ctr, 1u));   // the next one: its number is back before the third stage
        NvUnit next;
        const int nst = p.K[u.phase] / KS;
        const uint8_t* src = p.w[u.phase] + static_cast<size_t>(u.expert * p.n_pairs[u.phase] + u.pair) * nst * STAGE_W_BYTES;
        for (int ks = 0; ks < nst; ++ks, ++st) {
          const uint32_t ws = st % NV_W_STAGES;
          if (st == NV_W_STAGES && i == 0u) {
            // While the token rows are split memory would stand still once the ring is full: the next stages go to L2, at the pace of memory
            // (all at once they held up the reading of the rows, 3 us) and until the first MMAs are done.
            for (int a = 0; a < min(nst - ks, NV_AHEAD) && !mbar_test(&ctl.done[0], 0u); ++a) {
              bulk_prefetch_l2(src + a * STAGE_W_BYTES, STAGE_W_BYTES);
              __nanosleep(700);
            }
          }
          if (!mbar_wait_inline(&ctl.w_done[ws], ((st / NV_W_STAGES) & 1u) ^ 1u, abortw)) { ok = false; break; }
          mbar_arrive_expect_tx(&ctl.w_full[ws], STAGE_W_BYTES);
          bulk_g2s(w_ring + ws * STAGE_W_BYTES, src, STAGE_W_BYTES, &ctl.w_full[ws], pol);
          if (st == 0u) MSK_TR(TR_FIRST_BULK);
          src += STAGE_W_BYTES;
          // The next unit is published early in this one: the word of its tile's levels and its first token rows are fetched meanwhile (published
          // with its first weights it cost 8 tokens 1.5 us).
          if (ks == min(2, nst - 1) && !publish(next, i + 1u, x)) { ok = false; break; }
        }
        u = next;
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------- MMA issuer
    const uint64_t a0 = smem_desc_kmajor_noswz(smem_u32(w_ring), 128, 2 * OCT_BYTES);
    const uint64_t b0 = smem_desc_kmajor_sw128(smem_u32(b_ring));
    NvBuffers db;
    uint32_t st = 0, wst = 0, bs = 0;            // passes, K stages
    bool ok = true, ready = false;               // ready: the next pass was seen complete
    NvUnit u;
    while (ok && wait_unit(u, mbar_wait_warp)) {
      __syncwarp();
      if (lane == 0) done_unit();
      if (u.phase < 0) break;
      db.take(u.width);
      if (db.uses(0) && !mbar_wait_warp(&ctl.d_empty[0], db.p0 ^ 1u, abortw)) break;
      if (db.uses(1) && !mbar_wait_warp(&ctl.d_empty[1], db.p1 ^ 1u, abortw)) break;
      const uint32_t d0 = tmem + db.col(), d1 = d0 + db.tile_cols();
      const int nst = p.K[u.phase] / KS;
      uint32_t accumulate = 0u;
      for (int ks = 0; ok && ks < nst; ++ks, ++wst) {
        const uint32_t ws = wst % NV_W_STAGES;
        for (uint32_t last = 0u; last == 0u;) {     // the stage's levels
          const uint32_t ss = st % NV_S_STAGES;
          // the scales; the warps that write them have seen the stage's weights and token rows land
          if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(&ctl.s_full[ss], (st / NV_S_STAGES) & 1u, abortw)) { ok = false; break; }
          tc_fence_after();
          if (st == 0u && lane == 0) MSK_TR(TR_FIRST_MMA);
          const int pass = ctl.b_pass[bs], level = pass & 3;
          last = static_cast<uint32_t>(pass & NV_LAST);
          const uint32_t mark = st % NV_MARKS, rows = static_cast<uint32_t>(nv_room(u.rows)), first = static_cast<uint32_t>(nv_first(level)) * rows;
          ++st;
          ready = mma_nvf4_stage(d0 + first, d1 + first, a0 + ((ws * STAGE_W_BYTES) >> 4), b0 + ((bs * b_bytes) >> 4),
                                 idesc_nvf4((static_cast<uint32_t>(nv_digits(level)) * rows + 7u) & ~7u), tmem + C::S_BASE + (wst % NV_S_STAGES) * C::S_COLS,
                                 tmem + C::S_B + ss * C::S_COLS, accumulate,
                                 smem_u32(&ctl.done[mark]), smem_u32(&ctl.w_done[ws]), last, smem_u32(&ctl.s_full[st % NV_S_STAGES]), (st / NV_S_STAGES) & 1u);
          accumulate = 1u;
          if (++bs == b_stages) bs = 0;
        }
      }
      if (ok && elect_one()) {
        if (db.uses(0)) tc_commit(&ctl.d_full[0]);
        if (db.uses(1)) tc_commit(&ctl.d_full[1]);
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------- token rows
    if (lane == 0) {
      const uint64_t keep = policy_evict_last();   // re-read by every pair of the expert
      uint32_t st = 0, bs = 0;
      int last_tile = -1;
      const int n_stages = p.I / KS;
      bool ok = true, split = false;
      NvUnit u;
      while (ok && wait_unit(u, mbar_wait_inline)) {
        done_unit();
        if (u.phase < 0) break;
        if (u.phase == 0 && !split) {
          if (!grid_counter_wait(p.ctr + 2, static_cast<unsigned>(n_ctas), abortw)) break;
          fence_proxy_async_all();                 // ordinary stores of other SMs, about to be read by bulk copies
          split = true;
        }
        unsigned int* tile = p.tiles + u.tile * NV_TILE_WORDS;
        if (u.phase == 1) {
          if (u.tile != last_tile) {
            if (!grid_counter_wait(tile + NV_READY, static_cast<unsigned>(u.width * n_stages * 4), abortw)) break;
            fence_proxy_async_all();
            last_tile = u.tile;
          }
        }
        const int nst = p.K[u.phase] / KS, room = nv_room(u.rows);
        const uint8_t* src = p.img[u.phase] + static_cast<size_t>(u.group) * nst * NV_GROUP_BYTES;
        const unsigned int* flags = tile + (u.phase == 0 ? NV_MORE : NV_MORE_INTER);
        unsigned int more1 = 0u, more2 = 0u;
        for (int ks = 0; ok && ks < nst; ++ks, more1 >>= 1, more2 >>= 1, src += room * (NV_GROUP_BYTES / 8)) {
          if ((ks & 31) == 0) {
            more1 = __ldcg(flags + ks / 16);
            more2 = __ldcg(flags + ks / 16 + 1);
          }
          for (int level = 0; level < NV_LEVELS; ++level) {
            if ((level == 1 && (more1 & 1u) == 0u) || (level == 2 && (more2 & 1u) == 0u)) continue;
            const uint32_t before = st - b_stages;
            if (st >= b_stages && !mbar_wait_inline(&ctl.done[before % NV_MARKS], (before / NV_MARKS) & 1u, abortw)) { ok = false; break; }
            const uint32_t bytes = static_cast<uint32_t>(room * (nv_digits(level) * 128 + 16));
            mbar_arrive_expect_tx(&ctl.b_full[bs], bytes);
            bulk_g2s(b_ring + bs * b_bytes, src + nv_digit_at(room, level, 0), bytes, &ctl.b_full[bs], keep);
            const bool last = level == 2 || ((level == 1 || (more1 & 1u) == 0u) && (more2 & 1u) == 0u);
            ctl.b_pass[bs] = level | (last ? NV_LAST : 0);
            mbar_arrive(&ctl.b_full[bs]);
            ++st;
            if (++bs == b_stages) bs = 0;
          }
        }
        if (ok && u.phase == 1) {
          // the last down unit of the tile to have fetched its rows puts its counters back for the next launch
          const unsigned seen = atomicAdd(tile + NV_SEEN, 1u);
          if (seen == static_cast<unsigned>(p.n_pairs[1]) - 1u) {
            atomicExch(tile + NV_DONE, 0u);
            atomicExch(tile + NV_READY, 0u);
            atomicExch(tile + NV_SEEN, 0u);
            for (int i = NV_MORE; i < NV_MORE_INTER + 2 * ((nst + 31) / 32); ++i) atomicExch(tile + i, 0u);
          }
        }
      }
    }
  } else if (warp == 3) {
    // ----------------------------------------- counts stored gate/up units for their tiles
    // The fence that covers a unit's stores takes a microsecond and more while the memory system streams: here it holds up nobody. (This
    // warp hands back the unit's record as well, so that its barrier is not met twice in a phase.)
    NvUnit u;
    while (lane == 0 && wait_unit(u, mbar_wait_inline) && u.phase >= 0) {
      const uint32_t i = ui - 1u;
      if (!mbar_wait_inline(&ctl.stored[i % NV_UNITS], (i / NV_UNITS) & 1u, abortw)) break;
      if (u.phase == 0) {
        __threadfence();
        red_release_add(p.tiles + u.tile * NV_TILE_WORDS + NV_DONE, 1u);
      }
      done_unit();
    }
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ scales
    const uint32_t quarter = static_cast<uint32_t>((warp & 3) * 32) << 16;
    uint32_t st = 0, wst = 0, bs = 0, bpar = 0;   // passes, K stages
    bool ok = true;
    NvUnit u;
    while (ok && wait_unit(u, mbar_wait_warp)) {
      __syncwarp();
      if (lane == 0) done_unit();
      if (u.phase < 0) break;
      const int nst = p.K[u.phase] / KS;
      // This lane's token row: column c of a stage's scales is that of the MMA's columns 32 c + lane, digit after digit of the tile's
      // rows: with room for four, eight or sixteen all columns are alike.
      const int room = nv_room(u.rows);
      const uint32_t row_at = static_cast<uint32_t>(lane & (room - 1)) * 16u;
      for (int ks = 0; ok && ks < nst; ++ks, ++wst) {
        const uint32_t ws = wst % NV_W_STAGES;
        if (!mbar_wait_warp(&ctl.w_full[ws], (wst / NV_W_STAGES) & 1u, abortw)) { ok = false; break; }
        uint8_t* stage = w_ring + ws * STAGE_W_BYTES;
        uint32_t r[2][16], neg = 0u;   // [tile][64 K x row quarter]: the scales of row 32 c + lane
#pragma unroll
        for (int g = 0; g < 2; ++g) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v = *reinterpret_cast<const uint4*>(stage + (2 * (4 * c + (lane >> 3)) + g) * OCT_BYTES + OCT_CODE_BYTES + (lane & 7) * 16);
            r[g][c] = v.x; r[g][4 + c] = v.y; r[g][8 + c] = v.z; r[g][12 + c] = v.w;
            neg |= v.x | v.y | v.z | v.w;
          }
        }
        if (__any_sync(0xffffffffu, (neg & 0x80808080u) != 0u)) {
          // negative scales: each of the four warps turns the signs of the codes of its own 32 rows
          const int c = warp & 3;
#pragma unroll 1
          for (int g = 0; g < 2; ++g) {
            uint8_t* row = stage + (2 * (4 * c + (lane >> 3)) + g) * OCT_BYTES + (lane & 7) * 16;
#pragma unroll 1
            for (int j = 0; j < 16; ++j) {
              if ((row[OCT_CODE_BYTES + j] & 0x80) == 0) continue;
              uint2* code = reinterpret_cast<uint2*>(row + (j >> 1) * 128 + (j & 1) * 8);
              *code = make_uint2(code->x ^ 0x88888888u, code->y ^ 0x88888888u);
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            r[0][j] &= 0x7F7F7F7Fu;
            r[1][j] &= 0x7F7F7F7Fu;
          }
          fence_proxy_async_smem();
        }
        for (bool last = false; !last; ++st) {     // the stage's levels, each beside the same weights
          const uint32_t ss = st % NV_S_STAGES;
          if (!mbar_wait_warp(&ctl.b_full[bs], bpar, abortw)) { ok = false; break; }
          const int pass = ctl.b_pass[bs];
          last = (pass & NV_LAST) != 0;
          const uint8_t* sc = b_ring + bs * b_bytes + nv_digits(pass & 3) * 128 * room;
          const uint4 v = *reinterpret_cast<const uint4*>(sc + row_at);
          const uint32_t before = st - NV_S_STAGES;
          if (st >= NV_S_STAGES && !mbar_wait_warp(&ctl.done[before % NV_MARKS], (before / NV_MARKS) & 1u, abortw)) { ok = false; break; }
          tc_fence_after();
          if ((pass & 3) == 0) {                   // (the passes of the stage before last are done too: the weights' place is free)
            const uint32_t at = tmem + quarter + C::S_BASE + (wst % NV_S_STAGES) * C::S_COLS;
            tmem_st16(at, r[0]);
            tmem_st16(at + 16, r[1]);
          }
          const uint32_t lo[16] = {v.x, v.x, v.x, v.x, v.x, v.x, v.x, v.x, v.y, v.y, v.y, v.y, v.y, v.y, v.y, v.y};
          const uint32_t hi[16] = {v.z, v.z, v.z, v.z, v.z, v.z, v.z, v.z, v.w, v.w, v.w, v.w, v.w, v.w, v.w, v.w};
          const uint32_t at_b = tmem + quarter + C::S_B + ss * C::S_COLS;
          tmem_st16(at_b, lo);
          tmem_st16(at_b + 16, hi);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.s_full[ss]);
          if (++bs == b_stages) { bs = 0; bpar ^= 1u; }
        }
      }
    }
  } else if (warp >= 8 && warp < 12) {
    // ---------------------------------------------------------------- epilogue
    const int row = (warp & 3) * 32 + lane;
    const uint32_t quarter = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool leader = tid == 8 * 32;
    NvBuffers db;
    uint32_t n_unit = 0;
    bool ok = true;
    NvUnit u;
    while (ok && wait_unit(u, mbar_wait_warp)) {
      __syncwarp();
      if (lane == 0) done_unit();
      if (u.phase < 0) break;
      db.take(u.width);
      const float gsc = p.gs[u.phase][u.expert] * NV_SUM_SCALE;
      const int col = u.phase == 0 ? u.pair * 128 + row : 2 * u.pair * 128 + row;
      float o0 = gsc, o1 = gsc;
      if (u.phase == 1 && p.post_norm_w != nullptr) {
        o0 *= 1.0f + __bfloat162float(p.post_norm_w[col]);
        o1 *= 1.0f + __bfloat162float(p.post_norm_w[col + 128]);
      }
      if (db.uses(0) && !mbar_wait_warp(&ctl.d_full[0], db.p0, abortw)) { ok = false; break; }
      if (db.uses(1) && !mbar_wait_warp(&ctl.d_full[1], db.p1, abortw)) { ok = false; break; }
      tc_fence_after();
      if (leader) { if (n_unit == 0u) MSK_TR(TR_FIRST_DFULL); MSK_TR(TR_LAST_DFULL); }
      const uint32_t d0 = tmem + quarter + db.col(), d1 = d0 + db.tile_cols();
      const int room = nv_room(u.rows);
#pragma unroll 1
      for (int c0 = 0; c0 < u.rows; c0 += 8) {
        const int left = u.rows - c0;
        float a0[8], a1[8];
        {
          uint32_t v[NV_PARTS][8];
#pragma unroll
          for (int q = 0; q < NV_PARTS; ++q) tmem_ld8(d0 + q * room + c0, v[q]);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            a0[j] = __uint_as_float(v[NV_PARTS - 1][j]);
#pragma unroll
            for (int q = NV_PARTS - 2; q >= 0; --q) a0[j] = fmaf(a0[j], 0.125f, __uint_as_float(v[q][j]));
          }
#pragma unroll
          for (int q = 0; q < NV_PARTS; ++q) tmem_ld8(d1 + q * room + c0, v[q]);
          tmem_wait_ld();
          if (left <= 8) {                         // the accumulators are read
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if (db.uses(0)) mbar_arrive(&ctl.d_empty[0]);
              if (db.uses(1)) mbar_arrive(&ctl.d_empty[1]);
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            a1[j] = __uint_as_float(v[NV_PARTS - 1][j]);
#pragma unroll
            for (int q = NV_PARTS - 2; q >= 0; --q) a1[j] = fmaf(a1[j], 0.125f, __uint_as_float(v[q][j]));
          }
        }
        if (u.phase == 0) {
          __half* out = p.inter + static_cast<size_t>(u.row0 + c0) * p.I + col;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < left) out[static_cast<size_t>(j) * p.I] = inter_value(silu_f(a0[j] * gsc) * (a1[j] * gsc));
        } else {
          float* out = p.y + static_cast<size_t>(u.row0 + c0) * p.H + col;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j < left) {
              out[static_cast<size_t>(j) * p.H] = a0[j] * o0;
              out[static_cast<size_t>(j) * p.H + 128] = a1[j] * o1;
            }
          }
        }
      }
      if (leader && n_unit == 0u) MSK_TR(TR_FIRST_EPI_DONE);
      ++n_unit;
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.stored[(ui - 1u) % NV_UNITS]);
    }
  } else if (warp >= 12) {
    // ---------------------------------------------------------- split of inter
    // A warp takes a piece, half a warp to a row. Early tiles are split while later ones are still at their gate/up units, so the first down
    // units wait for nothing.
    const int n_stages = p.I / KS, eights = group_start[p.nloc] * n_stages, bits = nv_piece_bits(eights, n_ctas);
    for (int i = static_cast<int>(blockIdx.x) + (warp - 12) * n_ctas; i < eights << (3 - bits); i += NV_CONV_WARPS * n_ctas) {
      const int eight = i >> (3 - bits), group = eight / n_stages, blk = (eight - group * n_stages) * 16 + (lane & 15);
      int lo = 0, hi = p.nloc;                     // largest e with group_start[e] <= group
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (group_start[mid] <= group) lo = mid; else hi = mid;
      }
      NvUnit u;
      const int at_row = (group - group_start[lo]) * 8;
      set_tile(u, lo, at_row / nv_tile_rows(cnt_s[lo], nv_tiles(cnt_s[lo])));
      const int first = (group - u.group) * 8 + ((i << bits) & 7);   // row of the tile
      if (first >= u.rows) continue;
      const bool go = lane != 0 || nv_tile_wait(p.tiles + u.tile * NV_TILE_WORDS + NV_DONE, static_cast<unsigned>(p.n_pairs[0]), abortw);
      if (!__all_sync(0xffffffffu, go)) break;
      __syncwarp();   // the vote orders no memory: the other lanes read rows that lane 0 has acquired
      uint4 v0, v1;
      auto load = [&](int slot) {   // stored by other SMs: from L2
        const uint4* src = reinterpret_cast<const uint4*>(p.inter + static_cast<size_t>(u.row0 + min(slot, u.rows - 1)) * p.I + blk * 16);
        v0 = __ldcg(src);
        v1 = __ldcg(src + 1);
      };
      const int last = min(first + (1 << bits), u.rows);
      unsigned any1 = 0u, any2 = 0u;
      const int room = nv_room(u.rows);
      uint8_t* stage = p.img[1] + static_cast<size_t>(u.group) * n_stages * NV_GROUP_BYTES + static_cast<size_t>((blk >> 4) * room) * (NV_GROUP_BYTES / 8);
      load(first + (lane >> 4));
#pragma unroll 1
      for (int r0 = first; r0 < last; r0 += 2) {
        const int slot = r0 + (lane >> 4);
        const uint32_t h8[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        load(slot + 2);                            // the next two rows, while these are split
        unsigned more1, more2;
        nv_split_block(h8, slot < last, NV_PARTS, NV_PARTS, true, more1, more2,
            [&](uint32_t s0, uint32_t s1, uint32_t s2) {
              stage[nv_scale_at(room, 0, slot, blk)] = static_cast<uint8_t>(s0);
              stage[nv_scale_at(room, 1, slot, blk)] = static_cast<uint8_t>(s1);
              stage[nv_scale_at(room, 2, slot, blk)] = static_cast<uint8_t>(s2);
            },
            [&](int level, int d, uint2 w) { *reinterpret_cast<uint2*>(stage + nv_code_at(room, level, d, slot, blk)) = w; });
        any1 |= more1;
        any2 |= more2;
      }
      if (any1 != 0u && lane < 2 && (lane == 0 || any2 != 0u))
        atomicOr(p.tiles + u.tile * NV_TILE_WORDS + NV_MORE_INTER + (blk >> 9) * 2 + lane, 1u << ((blk >> 4) & 31));
      __syncwarp();
      // a piece counts as the two rows that it has, or four times that; the tile's last one for the rows behind it as well (the counter's
      // readers put the fence between their acquire and their bulk copies)
      const unsigned twos = bits == 3 ? 4u : first + 2 < u.rows ? 1u : 4u - ((first & 7) >> 1);
      if (lane == 0) red_release_add(p.tiles + u.tile * NV_TILE_WORDS + NV_READY, twos);
    }
  }

  // -------------------------------------------------------------- teardown
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (tid == 0) MSK_TR(TR_END);
  if (tid == 0 && ctl.abort_word == 0) {
    // the last CTA to leave puts the counters back to zero for the next launch
    if (atomicAdd(p.ctr + 1, 1u) == gridDim.x - 1u) {
      atomicExch(p.ctr, 0u);
      atomicExch(p.ctr + 1, 0u);
      atomicExch(p.ctr + 2, 0u);
    }
  }
  if (ctl.abort_word != 0) {
    // give copies and MMAs still in flight time to land before shared memory and TMEM are released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    if (tid == 0) atomicExch(p.status, MSK_DEV_ERR_TIMEOUT);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

}  // namespace msk
