// Grouped GEMMs of the routed experts on the FP4 tensor cores, for token tiles of up to 24 rows: both GEMMs in one
// cooperative launch behind the sort.
//
// D[128 weight rows, N columns] = W[128, K] * B[N, K]^T with tcgen05.mma.kind::mxf4nvf4 (E2M1 operands, one E4M3 scale per 16
// K). The packed weights are that operand already: a stage of the ring goes from memory to the tensor core as it lies (octet
// blocks are the core matrices of an unswizzled K-major operand), only its scale bytes pass through registers into TMEM. No weight
// is decoded, so the kernel keeps pace with memory: the tcgen05 kernel of gemm.cuh, which decodes to F16 and passes every half
// stage through a TMEM slot, needs 1500 cycles and more for a stage that memory delivers in 1400, and power for it: long rows of
// steps run into the card's limit, where its clock falls. 64 tokens, all of 128 experts (1.3 GB), both GEMMs: 229 us there, 200 here; a
// row of whole steps 288 and 240 (both sides of the other sizes: nv_takes() in msk_moe.cu). Bound by memory, some 6.8 TB/s between the
// first MMA and the last, and by the 10 us before it (tables, split of the token rows) and 6 after.
//
// Activations. A token row (F16 values, as in gemm.cuh) enters as seven E2M1 rows of its own, the digits of a fixed-point
// number: in a block of 16 K an element is x = 2^u * (d0 + d1 / 8 + ... + d6 / 8^6), digits -4 .. 3, which E2M1 holds exactly (as
// d / 2). The block's exponent u, relative to the row's, is its E4M3 scale, one byte for all seven rows; 8^-p and the row's
// power of two are applied to the FP32 accumulators, which each digit has to itself, in the epilogue. An element is exact to
// 2^-20 of the largest of its block of 16 (BF16 values are held exactly down to 2^-12 of it), blocks keep that down to 2^-17
// of the row's largest value. Products are exact and accumulate in FP32. Measured against 64 bits (relative 2-norm of the raw
// sums, this / the F16 form): gate/up sums of normal rows, K = 4096, 1e-7 / 1.5e-6; down sums of SwiGLU values, K = 1536,
// 1.6e-7 / 9.0e-7; the rounding of the values to BF16 behind them is 1.7e-3. (Six digits: 5e-7 and 2.8e-6; the seventh costs some 4
// cycles of 56 an MMA.)
// NaN elements make the block's scale NaN; weight scales with a sign bit (no quantiser writes them) turn the signs of their
// 16 codes in shared memory, because the hardware's scales are unsigned.
//
// Per CTA (512 threads, one CTA per SM):
//   warp 0       draws units from a counter and streams their weights: one bulk copy per K stage (two tiles of 128 rows) into a ring;
//   warp 1       MMA issuer (and TMEM allocation): per stage 2 tiles x 4 MMAs of 64 K, one commit;
//   warp 2       token rows of the unit's tile, split and laid out beforehand: one bulk copy per K stage;
//   warps 4-7    scales: shared memory -> TMEM, each warp for its lane quarter (the hardware wants four copies);
//   warps 8-11   epilogue: digits summed, SwiGLU / scale, rows to global memory;
//   warp 3       counts stored gate/up units for their tiles;
//   warps 12-15  split `inter`: pieces of eight rows x 256 columns of a token tile, dealt over the CTAs in the order of the tiles, as each tile's
//                gate/up units are all stored (a row's power of two needs its largest value). Whole tiles, split by the CTA that
//                stored their last unit, kept a rank's 24-token step waiting for some 20 us.
// Warps 4-15 first split the token rows, a row or a part of one per CTA at a time, while the first weights are on their way.
//
// Work is dealt one unit at a time, gate/up units before down units, as in pair.cuh (but a unit is drawn when its weights are next to
// be fetched, not further ahead); a down unit waits for its tile's rows. Units of an expert with several tiles are ordered pair
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
constexpr int NV_ROWS = 24;                                // most token rows of a tile
constexpr int NV_PARTS = 7;                                // digits of an activation
constexpr int NV_GROUP_BYTES = NV_PARTS * 1024 + 128;      // eight token rows x 256 K: digits, scales
constexpr int NV_W_STAGES = 4, NV_S_STAGES = 2;            // rings: weights, scales in TMEM
constexpr int NV_MARKS = 8;                                // stages whose MMAs have a barrier of their own
constexpr int NV_UNITS = 4;
constexpr int NV_SPLIT_WARP = 4, NV_SPLIT_THREADS = NV_THREADS - NV_SPLIT_WARP * 32;
constexpr int NV_MAX_BLOCKS = 512;                         // blocks of 16 K in a token row: H <= 8192
constexpr int NV_CONV_WARPS = 4;
constexpr int NV_AHEAD = 8;                                // stages of the first unit that are fetched to L2 ahead of the ring

// Token tiles of an expert with c rows: even shares in steps of 8. Width of a tile: its groups of eight rows.
__host__ __device__ inline int nv_tiles(int c) { return (c + NV_ROWS - 1) / NV_ROWS; }
__host__ __device__ inline int nv_tile_rows(int c, int n) { return n <= 1 ? c : ((c + n - 1) / n + 7) & ~7; }
__host__ __device__ inline int nv_width(int rows) { return (rows + 7) >> 3; }
// Groups that the image of an expert's rows takes (every tile but a lone one has room for three).
constexpr int NV_GROUPS = NV_ROWS / 8;
__host__ __device__ inline int nv_groups(int c) { return c <= NV_ROWS ? nv_width(c) : NV_GROUPS * nv_tiles(c); }
// A bound on their sum over experts with `rows` rows in all: nv_groups(c) <= 1 + (c - 1) * 7 / 32.
inline size_t nv_groups_bound(size_t rows, size_t experts) {
  const size_t e = rows < experts ? rows : experts;
  return e + ((rows - e) * 7 + 31) / 32;
}

// Counters of a tile, a cache line for each: CTAs that wait for a tile poll another line than those that count for its neighbours.
constexpr int NV_TILE_WORDS = 32;
enum : int {
  NV_DONE = 0,     // stored gate/up units
  NV_READY = 8,    // pieces of inter that are split
  NV_SEEN = 16,    // down units that have seen all of them
};

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
  float* rs[2];                          // [R] the rows' powers of two: token rows, rows of inter
  __half* part_max;                      // [R, I / 32] largest magnitude in 32 columns of a row of inter
  int32_t* status;
  unsigned long long* trace;
  unsigned int* ctr;                     // [0] units drawn, [1] CTAs that have left, [2] CTAs that have split their token rows
  unsigned int* tiles;                   // NV_TILE_WORDS a tile: counters NV_DONE, NV_READY, NV_SEEN, all zero between launches
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
  uint64_t done[NV_MARKS];               // the MMAs of stage n (n % 8): its places in all three rings are free
  uint64_t d_full[2], d_empty[2];
  uint64_t u_full[NV_UNITS], u_empty[NV_UNITS];
  uint64_t stored[NV_UNITS];             // the epilogue has stored its values of a unit
  NvUnit unit[NV_UNITS];
  uint4 route[MAX_TOP_K];                // of the token row that is split: place of its digits in the image, width, row in its group, row
  float red[2][NV_SPLIT_THREADS / 32];
  int n_routes;
  uint32_t tmem_base;
  int abort_word;
  int b_stages, b_bytes;                 // ring of token rows: places, bytes of one
};
static_assert(sizeof(NvCtrl) <= 1024 && offsetof(NvCtrl, unit) % 16 == 0, "control block");

__host__ __device__ constexpr int nv_place_bytes(int width) { return (width * NV_GROUP_BYTES + 1023) / 1024 * 1024; }

struct NvCfg {
  static constexpr int TABLE_INTS = MAX_LOCAL_EXPERTS + 4;
  // The ring of token rows has places for the widest tile of the launch (whole swizzle atoms of 1 KB): 3, 5 or 8 of them.
  static constexpr int B_RING = 75 * 1024;
  static constexpr int W_OFF = 0, B_OFF = NV_W_STAGES * STAGE_W_BYTES, CTL_OFF = B_OFF + B_RING, TABLE_OFF = CTL_OFF + 1024;
  static constexpr int SMEM_BYTES = TABLE_OFF + 4 * TABLE_INTS * 4;
  static_assert(SMEM_BYTES <= 232448 && 3 * nv_place_bytes(NV_GROUPS) <= B_RING, "shared memory of a CTA");
  // TMEM: accumulators of two tiles (digits x rows columns each; those of a tile of eight rows twice), two stages of scales
  static constexpr int D_WIDE = NV_PARTS * NV_ROWS, D_NARROW = NV_PARTS * 8;
  static constexpr int S_BASE = 2 * D_WIDE, S_COLS = 64, S_B = 32;   // 4 x 4 columns per weight tile, 4 x 8 for the token rows
  static_assert(4 * D_NARROW <= S_BASE && (D_WIDE + 31) / 32 <= 8, "TMEM layout");
  static_assert(S_BASE + NV_S_STAGES * S_COLS <= TMEM_COLS, "TMEM budget");
};

__host__ __device__ constexpr uint32_t idesc_nvf4(uint32_t N) {   // E2M1 x E2M1, E4M3 scales, M = 128
  return (1u << 7) | (1u << 10) | ((N >> 3) << 17) | (8u << 24);
}
// D[tmem] (+)= A[smem, 128 x 256] * B[smem, N x 256]^T for the two tiles of a stage, four MMAs of 64 K each: a scale per row and 16 K in
// TMEM, lane r % 32 (in every lane quarter), column r / 32, the four bytes of 64 K. `sf`: 4 x 4 columns of tile 0, of tile 1, 4 x 8 of the
// token rows. By one elected lane, with the commit that hands the stage back (done_bar); the answer of a probe of `next_full` (true:
// complete) is asked for before the MMAs and read behind them. In one block of assembly: as separate calls in a branch of that lane
// the operands went to the issue unit one by one, some 150 cycles an MMA.
#define NV_MMA "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X"
__device__ __forceinline__ bool mma_nvf4_stage(uint32_t d0, uint32_t d1, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sf, uint32_t accumulate,
                                               uint32_t done_bar, uint32_t next_full, uint32_t parity) {
  static_assert(OCT_BYTES / 16 == 72, "the second tile's octet blocks");
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred q, e, acc, t;\n\t.reg .b64 a, b, c;\n\t.reg .b32 f, g, h;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%9], %10;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 acc, %8, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 a, %3;\n\tmov.b64 b, %4;\n\tmov.b32 f, %6;\n\tadd.u32 g, %6, 32;\n\t"
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
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(d0), "r"(d1), "l"(a), "l"(b), "r"(idesc), "r"(sf), "r"(done_bar), "r"(accumulate), "r"(next_full), "r"(parity)
      : "memory");
  return ok != 0u;
}
#undef NV_MMA

// ---- the split. Image of a tile (width W groups, K): per K stage of 256, digits [7][W][8 rows][128 bytes], the eight 16-byte
// chunks of a row in the order of the 128-byte swizzle (chunk c of row r at c ^ r: a row's digit is one line to write), then
// scales [8 W rows][16]; NV_GROUP_BYTES * W bytes a stage, one contiguous copy.

// Exponent of a block's unit: its largest magnitude m is at most 3.4 units (digits reach 24 / 7 upwards).
__device__ __forceinline__ int nv_unit_exp(float m) {
  const int b = __float_as_int(m);
  return m > 0.f ? (b >> 23) - 127 - ((b & 0x7fffff) > 0x599999 ? 0 : 1) : -200;
}
__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((e + 127) << 23); }
// The row's, from its largest magnitude (zero and NaN: that of the smallest F16 value).
__device__ __forceinline__ int nv_row_exp(float m) { return max(nv_unit_exp(m), -25); }
// The power of two that a row's sums are multiplied by, from its unit exponent: the largest block has scale 2^8 (and its codes are d / 2).
__device__ __forceinline__ float nv_row_scale(int U) { return exp2_int(U - 7); }

// Largest magnitude of sixteen values; NaN if one of them is.
__device__ __forceinline__ float nv_block_max(const uint32_t (&h)[8]) {
  __half2 m = __habs2(*reinterpret_cast<const __half2*>(&h[0]));
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax2_nan(m, __habs2(*reinterpret_cast<const __half2*>(&h[i])));
  return __half2float(__hmax_nan(__low2half(m), __high2half(m)));
}

// Sixteen values -> for each the number x * 8^6 / unit as 21 bits that hold digit + 4 in each three; returns the scale byte. bm: the
// block's largest magnitude, U: the row's unit exponent.
__device__ __forceinline__ uint32_t nv_fixed16(const uint32_t (&h)[8], float bm, int U, uint32_t (&f)[16]) {
  const int u = max(nv_unit_exp(bm), U - 17), e = u - U + 8;
  const float scale = exp2_int(3 * (NV_PARTS - 1) - u);
  constexpr float BIAS = 12582912.f + 4.f * ((1 << (3 * NV_PARTS)) - 1) / 7.f;   // rounds by the addition; 4 in every digit
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
    f[2 * i] = __float_as_uint(fmaf(v.x, scale, BIAS));
    f[2 * i + 1] = __float_as_uint(fmaf(v.y, scale, BIAS));
  }
  return bm != bm ? 0x7Fu : e >= -6 ? static_cast<uint32_t>(e + 7) << 3 : 1u << (e + 9);
}
// The last digits of the sixteen as E2M1 codes, a nibble each; the numbers lose them. (The loops over the digits are not unrolled: this
// code runs from a cold instruction cache while the weights stream, where a line takes a microsecond; all digits in line made
// the steps 5 to 20 us longer.)
__device__ __forceinline__ uint2 nv_next_digit(uint32_t (&f)[16]) {
  uint32_t q[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t t = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      t += (f[8 * c + i] & 7u) * (1u << (4 * i));
      f[8 * c + i] >>= 3;
    }
    const uint32_t pos = ((t >> 2) & 0x11111111u) * 15u;   // nibbles of digits >= 0: the digit; of the others: sign and magnitude 4 - t
    q[c] = (t & 0x33333333u & pos) | ((0xCCCCCCCCu - t) & ~pos);
  }
  return make_uint2(q[0], q[1]);
}

// Where block `blk`'s stage begins in the image of a tile; in it the block's digit 0 and its scale for row `slot`.
__device__ __forceinline__ uint8_t* nv_stage(uint8_t* img, int group, int width, int K, int blk) {
  return img + (static_cast<size_t>(group) * (K / KS) + static_cast<size_t>(blk >> 4) * width) * NV_GROUP_BYTES;
}
__device__ __forceinline__ int nv_row_at(int slot) { return (slot >> 3) * 1024 + (slot & 7) * 128; }
__device__ __forceinline__ int nv_digit_at(int slot, int blk) {
  return nv_row_at(slot) + ((((blk & 15) >> 1) ^ (slot & 7)) * 16) + (blk & 1) * 8;
}
__device__ __forceinline__ int nv_scale_at(int width, int slot, int blk) { return NV_PARTS * width * 1024 + slot * 16 + (blk & 15); }

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
    for (int i = 0; i < NV_W_STAGES; ++i) mbar_init(&ctl.w_full[i], 1);
    for (int i = 0; i < NV_S_STAGES; ++i) mbar_init(&ctl.s_full[i], 4);
    for (int i = 0; i < NV_MARKS; ++i) {
      mbar_init(&ctl.b_full[i], 1);
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
  // The first token row (or its part) of this CTA, up to its largest value: it does not depend on the sort, and the launch before the sort
  // has completed (the sort lets this launch begin only behind its own wait).
  constexpr int NT = NV_SPLIT_THREADS, NW = NT / 32, PER = (NV_MAX_BLOCKS + NT - 1) / NT;
  const int th = tid - NV_SPLIT_WARP * 32, nb = p.H / 16;
  // up to 74 tokens several CTAs share a row: each reads all of it for its largest value and splits some of the K stages (not over
  // PCIe, where every reader costs the bytes again: 8 rows in host memory, a whole step 121 us shared, 103 not, 119 by the other kernel)
  const int parts = p.share_rows ? max(1, min(n_ctas / p.T, p.H / KS)) : 1, items = p.T * parts;
  uint32_t h[PER][8];
  float bm[PER];
  int U = 0;
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
  auto finish_row = [&]() {   // norm, F16 values, the row's exponent
    const int sw = warp - NV_SPLIT_WARP;
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
      if (lane == 0) ctl.red[1][sw] = ss;
      named_bar_sync(1, NT);
      float tot = 0.f;
#pragma unroll
      for (int i = 0; i < NW; ++i) tot += ctl.red[1][i];
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
    float rm = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) h[i][j] = bf16x2_to_f16x2(h[i][j]);
      bm[i] = nv_block_max(h[i]);
      rm = fmaxf(rm, bm[i]);
    }
    rm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(rm)));
    if (lane == 0) ctl.red[0][sw] = rm;
    named_bar_sync(1, NT);
#pragma unroll
    for (int i = 0; i < NW; ++i) rm = fmaxf(rm, ctl.red[0][i]);
    U = nv_row_exp(rm);
  };
  if (warp >= NV_SPLIT_WARP && static_cast<int>(blockIdx.x) < items) {
    fetch_row(static_cast<int>(blockIdx.x) / parts);
    finish_row();
  }
  pdl_wait();
  pdl_launch_dependents();
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
      ctl.b_bytes = nv_place_bytes(nv_width(min(most, NV_ROWS)));
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
    u.group = group_start[e] + ti * NV_GROUPS;
  };

  if (warp >= NV_SPLIT_WARP) {
    // ------------------------------------------------- split of the token rows
    int q = -1, id = 0;                            // lane s of the first of these warps: route s of the row
    auto fetch_route = [&](int t) {
      if (th < p.k) {
        q = __ldcg(p.inv + static_cast<size_t>(t) * p.k + th);
        id = __ldcg(p.ids + static_cast<size_t>(t) * p.k + th);
      }
    };
    int item = static_cast<int>(blockIdx.x);
    if (item < items) fetch_route(item / parts);
    while (item < items) {
      const int part = item % parts, next = item + n_ctas;
      if (th < 32) {   // where its local routes' rows go
        const unsigned have = __ballot_sync(0xffffffffu, q >= 0);
        if (q >= 0) {
          const int e = id - p.lo, c = cnt_s[e], per = nv_tile_rows(c, nv_tiles(c)), r = q - off_s[e], ti = r / per, slot = r - ti * per;
          const int group = group_start[e] + ti * NV_GROUPS, width = nv_width(min(per, c - ti * per));
          ctl.route[__popc(have & ((1u << th) - 1u))] =
              make_uint4(static_cast<uint32_t>(group * (p.H / KS) * NV_GROUP_BYTES + nv_row_at(slot)), static_cast<uint32_t>(width),
                         static_cast<uint32_t>(slot & 7), static_cast<uint32_t>(slot));
          if (part == 0) p.rs[0][q] = nv_row_scale(U);
        }
        if (th == 0) ctl.n_routes = __popc(have);
      }
      named_bar_sync(1, NT);
      const int n_routes = ctl.n_routes, row_exp = U;
      uint32_t g[PER][8];
      float gm[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        gm[i] = bm[i];
#pragma unroll
        for (int j = 0; j < 8; ++j) g[i][j] = h[i][j];
      }
      if (next < items) {                          // on its way while this one is split
        fetch_row(next / parts);
        q = -1;
        fetch_route(next / parts);
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int b = th + i * NT;
        if (b >= nb || n_routes == 0 || (parts > 1 && (b >> 4) % parts != part)) continue;
        uint32_t f[16];
        const uint32_t sf = nv_fixed16(g[i], gm[i], row_exp, f), chunk = (b & 15) >> 1;
#pragma unroll 1
        for (int d = NV_PARTS - 1; d >= -1; --d) {   // digits, then the scale
          const uint2 w = nv_next_digit(f);
#pragma unroll 1
          for (int s = 0; s < n_routes; ++s) {
            const uint4 to = ctl.route[s];
            uint8_t* row = p.img[0] + to.x + to.y * ((b >> 4) * NV_GROUP_BYTES);
            if (d >= 0) *reinterpret_cast<uint2*>(row + to.y * (d * 1024) + (chunk ^ to.z) * 16 + (b & 1) * 8) = w;
            else row[nv_scale_at(to.y, to.w, b) - nv_row_at(to.w)] = static_cast<uint8_t>(sf);
          }
        }
      }
      item = next;
      if (item < items) finish_row();              // (with a barrier, behind which the routes' places may be written again)
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
      int x = static_cast<int>(blockIdx.x);         // the first unit, then what the counter gives
      uint32_t st = 0;
      bool ok = true;
      for (uint32_t i = 0; ok; ++i) {
        NvUnit u;
        u.phase = -1;
        if (x < n) {
          u.phase = x >= n0 ? 1 : 0;
          const int np = p.n_pairs[u.phase], v = u.phase ? x - n0 : x;
          const int e = expert_of(v / np), idx = v - tile_start[e] * np, nt = nv_tiles(cnt_s[e]);
          u.pair = idx / nt;
          set_tile(u, e, idx - u.pair * nt);
        }
        const uint32_t s = i % NV_UNITS;
        if (!mbar_wait_inline(&ctl.u_empty[s], ((i / NV_UNITS) & 1u) ^ 1u, abortw)) break;
        *reinterpret_cast<int4*>(&ctl.unit[s]) = make_int4(u.phase, u.expert, u.row0, u.rows);
        *(reinterpret_cast<int4*>(&ctl.unit[s]) + 1) = make_int4(u.pair, u.tile, u.group, u.width);
        mbar_arrive(&ctl.u_full[s]);
        if (u.phase < 0) break;
        x = n_ctas + static_cast<int>(atomicAdd(p.ctr, 1u));   // the next one: its number is back long before this one's last stage
        const int nst = p.K[u.phase] / KS;
        const uint8_t* src = p.w[u.phase] + static_cast<size_t>(u.expert * p.n_pairs[u.phase] + u.pair) * nst * STAGE_W_BYTES;
        for (int ks = 0; ks < nst; ++ks, ++st) {
          const uint32_t ws = st % NV_W_STAGES;
          const uint32_t before = st - NV_W_STAGES;   // the stage whose place this one takes
          if (st == NV_W_STAGES && i == 0u) {
            // While the token rows are split memory would stand still once the ring is full: the next stages go to L2, at the pace of memory
            // (all at once they held up the reading of the rows, 3 us) and until the first MMAs are done.
            for (int a = 0; a < min(nst - ks, NV_AHEAD) && !mbar_test(&ctl.done[0], 0u); ++a) {
              bulk_prefetch_l2(src + a * STAGE_W_BYTES, STAGE_W_BYTES);
              __nanosleep(700);
            }
          }
          if (st >= NV_W_STAGES && !mbar_wait_inline(&ctl.done[before % NV_MARKS], (before / NV_MARKS) & 1u, abortw)) { ok = false; break; }
          mbar_arrive_expect_tx(&ctl.w_full[ws], STAGE_W_BYTES);
          bulk_g2s(w_ring + ws * STAGE_W_BYTES, src, STAGE_W_BYTES, &ctl.w_full[ws], pol);
          if (st == 0u) MSK_TR(TR_FIRST_BULK);
          src += STAGE_W_BYTES;
        }
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------- MMA issuer
    const uint64_t a0 = smem_desc_kmajor_noswz(smem_u32(w_ring), 128, 2 * OCT_BYTES);
    const uint64_t b0 = smem_desc_kmajor_sw128(smem_u32(b_ring));
    NvBuffers db;
    uint32_t st = 0, bs = 0;
    bool ok = true, ready = false;               // ready: the next stage was seen complete
    NvUnit u;
    while (ok && wait_unit(u, mbar_wait_warp)) {
      __syncwarp();
      if (lane == 0) done_unit();
      if (u.phase < 0) break;
      db.take(u.width);
      if (db.uses(0) && !mbar_wait_warp(&ctl.d_empty[0], db.p0 ^ 1u, abortw)) break;
      if (db.uses(1) && !mbar_wait_warp(&ctl.d_empty[1], db.p1 ^ 1u, abortw)) break;
      const uint32_t idesc = idesc_nvf4(static_cast<uint32_t>(NV_PARTS * 8 * u.width));
      const uint32_t d0 = tmem + db.col(), d1 = d0 + db.tile_cols();
      const int nst = p.K[u.phase] / KS;
      for (int ks = 0; ks < nst; ++ks) {
        const uint32_t ws = st % NV_W_STAGES, ss = st % NV_S_STAGES;
        // the scales; the warps that write them have seen the stage's weights and token rows land
        if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(&ctl.s_full[ss], (st / NV_S_STAGES) & 1u, abortw)) { ok = false; break; }
        tc_fence_after();
        if (st == 0u && lane == 0) MSK_TR(TR_FIRST_MMA);
        const uint32_t mark = st % NV_MARKS;
        ++st;
        ready = mma_nvf4_stage(d0, d1, a0 + ((ws * STAGE_W_BYTES) >> 4), b0 + ((bs * b_bytes) >> 4), idesc, tmem + C::S_BASE + ss * C::S_COLS,
                               ks > 0 ? 1u : 0u, smem_u32(&ctl.done[mark]), smem_u32(&ctl.s_full[st % NV_S_STAGES]), (st / NV_S_STAGES) & 1u);
        if (++bs == b_stages) bs = 0;
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
        if (u.phase == 1) {
          unsigned int* tile = p.tiles + u.tile * NV_TILE_WORDS;
          if (u.tile != last_tile) {
            if (!grid_counter_wait(tile + NV_READY, static_cast<unsigned>(u.width * (p.I / KS)), abortw)) break;
            fence_proxy_async_all();
            last_tile = u.tile;
          }
          // the last down unit of the tile to have seen it complete puts its counters back for the next launch
          const unsigned seen = atomicAdd(tile + NV_SEEN, 1u);
          if (seen == static_cast<unsigned>(p.n_pairs[1]) - 1u) {
            atomicExch(tile + NV_DONE, 0u);
            atomicExch(tile + NV_READY, 0u);
            atomicExch(tile + NV_SEEN, 0u);
          }
        }
        const int nst = p.K[u.phase] / KS;
        const uint32_t bytes = static_cast<uint32_t>(u.width * NV_GROUP_BYTES);
        const uint8_t* src = p.img[u.phase] + static_cast<size_t>(u.group) * nst * NV_GROUP_BYTES;
        for (int ks = 0; ks < nst; ++ks, ++st) {
          const uint32_t before = st - b_stages;
          if (st >= b_stages && !mbar_wait_inline(&ctl.done[before % NV_MARKS], (before / NV_MARKS) & 1u, abortw)) { ok = false; break; }
          mbar_arrive_expect_tx(&ctl.b_full[bs], bytes);
          bulk_g2s(b_ring + bs * b_bytes, src, bytes, &ctl.b_full[bs], keep);
          src += bytes;
          if (++bs == b_stages) bs = 0;
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
    uint32_t st = 0, bs = 0, bpar = 0;
    bool ok = true;
    NvUnit u;
    while (ok && wait_unit(u, mbar_wait_warp)) {
      __syncwarp();
      if (lane == 0) done_unit();
      if (u.phase < 0) break;
      const int nst = p.K[u.phase] / KS;
      // This lane's token rows: column c of a stage's scales is that of the MMA's columns 32 c + lane, digit after digit of the tile's
      // rows. With one or two groups of eight all columns are alike, with three they repeat after three.
      const uint32_t b_off = static_cast<uint32_t>(NV_PARTS * 1024 * u.width), n_row = static_cast<uint32_t>(8 * u.width);
      const uint32_t row0 = (lane % n_row) * 16u, row1 = ((lane + 32u) % n_row) * 16u, row2 = ((lane + 64u) % n_row) * 16u;
      const bool three = u.width == 3;
      for (int ks = 0; ks < nst; ++ks, ++st) {
        const uint32_t ws = st % NV_W_STAGES, ss = st % NV_S_STAGES;
        if (!mbar_wait_warp(&ctl.w_full[ws], (st / NV_W_STAGES) & 1u, abortw)) { ok = false; break; }
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
        if (!mbar_wait_warp(&ctl.b_full[bs], bpar, abortw)) { ok = false; break; }
        const uint8_t* sc = b_ring + bs * b_bytes + b_off;
        const uint4 v = *reinterpret_cast<const uint4*>(sc + row0);
        uint4 v1 = v, v2 = v;
        if (three) {
          v1 = *reinterpret_cast<const uint4*>(sc + row1);
          v2 = *reinterpret_cast<const uint4*>(sc + row2);
        }
        const uint32_t before = st - NV_S_STAGES;
        if (st >= NV_S_STAGES && !mbar_wait_warp(&ctl.done[before % NV_MARKS], (before / NV_MARKS) & 1u, abortw)) { ok = false; break; }
        tc_fence_after();
        const uint32_t at = tmem + quarter + C::S_BASE + ss * C::S_COLS;
        tmem_st16(at, r[0]);
        tmem_st16(at + 16, r[1]);
        const uint32_t lo[16] = {v.x, v1.x, v2.x, v.x, v1.x, v2.x, v.x, v1.x, v.y, v1.y, v2.y, v.y, v1.y, v2.y, v.y, v1.y};
        const uint32_t hi[16] = {v.z, v1.z, v2.z, v.z, v1.z, v2.z, v.z, v1.z, v.w, v1.w, v2.w, v.w, v1.w, v2.w, v.w, v1.w};
        tmem_st16(at + C::S_B, lo);
        tmem_st16(at + C::S_B + 16, hi);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.s_full[ss]);
        if (++bs == b_stages) { bs = 0; bpar ^= 1u; }
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
      const float gsc = p.gs[u.phase][u.expert];
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
      const float my_rs = lane < u.rows ? __ldcg(p.rs[u.phase] + u.row0 + lane) : 0.f;   // lane r: row r's power of two
#pragma unroll 1
      for (int c0 = 0; c0 < u.rows; c0 += 8) {
        const int left = u.rows - c0;
        float rs[8], a0[8], a1[8];
        {
          uint32_t v[NV_PARTS][8];
#pragma unroll
          for (int q = 0; q < NV_PARTS; ++q) tmem_ld8(d0 + q * 8 * u.width + c0, v[q]);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            a0[j] = __uint_as_float(v[NV_PARTS - 1][j]);
#pragma unroll
            for (int q = NV_PARTS - 2; q >= 0; --q) a0[j] = fmaf(a0[j], 0.125f, __uint_as_float(v[q][j]));
          }
#pragma unroll
          for (int q = 0; q < NV_PARTS; ++q) tmem_ld8(d1 + q * 8 * u.width + c0, v[q]);
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
#pragma unroll
        for (int j = 0; j < 8; ++j) rs[j] = __shfl_sync(0xffffffffu, my_rs, c0 + j);
        if (u.phase == 0) {
          __half* out = p.inter + static_cast<size_t>(u.row0 + c0) * p.I + col;
          __half2 most[4];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float f = gsc * rs[j];
            const __half v = inter_value(silu_f(a0[j] * f) * (a1[j] * f));
            if (j < left) out[static_cast<size_t>(j) * p.I] = v;
            if (j & 1) most[j >> 1].y = __habs(v); else most[j >> 1].x = __habs(v);
          }
          // (a place for every warp's 32 columns: atomic maxima of the rows, from all CTAs in a few cache lines, took 10 us a round of units)
#pragma unroll
          for (int b = 16; b > 0; b >>= 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) most[j] = __hmax2(most[j], __shfl_xor_sync(0xffffffffu, most[j], b));
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (lane == j && j < left) p.part_max[static_cast<size_t>(u.row0 + c0 + j) * (p.I / 32) + 4 * u.pair + (warp & 3)] = j & 1 ? most[j >> 1].y : most[j >> 1].x;
        } else {
          float* out = p.y + static_cast<size_t>(u.row0 + c0) * p.H + col;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j < left) {
              out[static_cast<size_t>(j) * p.H] = a0[j] * (o0 * rs[j]);
              out[static_cast<size_t>(j) * p.H + 128] = a1[j] * (o1 * rs[j]);
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
    // A warp takes a piece: eight rows of a tile, 256 columns, half a warp to a row. Early tiles are split while later ones are still at their
    // gate/up units, so the first down units wait for nothing.
    const int pieces = p.I / KS, n = group_start[p.nloc] * pieces;
    for (int i = static_cast<int>(blockIdx.x) + (warp - 12) * n_ctas; i < n; i += NV_CONV_WARPS * n_ctas) {
      const int group = i / pieces, blk = (i - group * pieces) * 16 + (lane & 15);
      int lo = 0, hi = p.nloc;                     // largest e with group_start[e] <= group
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (group_start[mid] <= group) lo = mid; else hi = mid;
      }
      NvUnit u;
      set_tile(u, lo, (group - group_start[lo]) / NV_GROUPS);   // (an expert with one tile has at most three groups, others three a tile)
      const int first = (group - u.group) * 8;     // row of the tile
      if (first >= u.width * 8) continue;          // room behind an expert's last tile
      const bool go = lane != 0 || nv_tile_wait(p.tiles + u.tile * NV_TILE_WORDS + NV_DONE, static_cast<unsigned>(p.n_pairs[0]), abortw);
      if (!__all_sync(0xffffffffu, go)) break;
      __syncwarp();   // the vote orders no memory: the other lanes read rows that lane 0 has acquired
      if (first < u.rows) {
        uint4 v0, v1, m;
        auto load = [&](int slot) {   // stored by other SMs: from L2
          const int r = u.row0 + min(slot, u.rows - 1);
          const uint4* src = reinterpret_cast<const uint4*>(p.inter + static_cast<size_t>(r) * p.I + blk * 16);
          v0 = __ldcg(src);
          v1 = __ldcg(src + 1);
          const uint4* mp = reinterpret_cast<const uint4*>(p.part_max + static_cast<size_t>(r) * (p.I / 32));
          m = make_uint4(0u, 0u, 0u, 0u);
          if ((lane & 15) < p.I / 256) m = __ldcg(mp + (lane & 15));
#pragma unroll 1
          for (int c = (lane & 15) + 16; c < p.I / 256; c += 16) {
            const uint4 x = __ldcg(mp + c);
            m = make_uint4(__vmaxu2(m.x, x.x), __vmaxu2(m.y, x.y), __vmaxu2(m.z, x.z), __vmaxu2(m.w, x.w));   // magnitudes compare as their bits
          }
        };
        const int last = min(first + 8, u.rows);
        load(first + (lane >> 4));
#pragma unroll 1
        for (int r0 = first; r0 < last; r0 += 2) {
          const int slot = r0 + (lane >> 4);
          const uint32_t h8[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
          uint32_t mm = __vmaxu2(__vmaxu2(m.x, m.y), __vmaxu2(m.z, m.w));
          mm = max(mm & 0xFFFFu, mm >> 16);
          load(slot + 2);                            // the next two rows, while these are split
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) mm = max(mm, __shfl_xor_sync(0xffffffffu, mm, o));
          const int U = nv_row_exp(__half2float(__ushort_as_half(static_cast<unsigned short>(mm))));
          uint32_t f[16];
          const uint32_t sf = nv_fixed16(h8, nv_block_max(h8), U, f);
          if (slot < last) {
            if (blk == 0) p.rs[1][u.row0 + slot] = nv_row_scale(U);
            uint8_t* stage = nv_stage(p.img[1], u.group, u.width, p.I, blk);
            uint8_t* at = stage + nv_digit_at(slot, blk);
#pragma unroll 1
            for (int d = NV_PARTS - 1; d >= 0; --d) *reinterpret_cast<uint2*>(at + d * u.width * 1024) = nv_next_digit(f);
            stage[nv_scale_at(u.width, slot, blk)] = static_cast<uint8_t>(sf);
          }
        }
      }
      __syncwarp();
      if (lane == 0) red_release_add(p.tiles + u.tile * NV_TILE_WORDS + NV_READY, 1u);   // (its readers put the fence between their acquire and their bulk copies)
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
