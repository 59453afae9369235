// Grouped GEMM of the routed experts on pairs of SMs, for token tiles of up to 256 rows.
//
// D[256 weight rows, N tokens] = W[256, K] * X[N, K]^T with tcgen05.mma.cta_group::2: a cluster of two CTAs works
// on one unit (token tile, pair of 128-row weight tiles). Each CTA decodes 128 of the 256 weight rows (64 of either
// tile) into its TMEM and fetches half of the token rows into its shared memory; CTA 0 issues MMAs that read both CTAs'
// halves and accumulate 128 rows x N columns in either CTA's TMEM.
//
// Why pairs: with one CTA to a tile the accumulators of (gate, up) x 128 tokens and the decoded weights share TMEM
// half and half, so every weight is decoded once per 128 tokens, and decode, its hand-over to the MMAs and the MMAs
// take turns at the A ring. Here the accumulators of 128 rows x 256 tokens fit the same half: the decode of a weight serves 256
// tokens, the activation bytes of a unit are fetched once for two SMs, and the A ring holds 512 K and more ahead of the MMAs.
//
// Per CTA (640 threads, one CTA per SM):
//   warp 0        weight producer: half a K stage (18,432 contiguous bytes, layout.cuh) per bulk copy into a ring;
//   warp 1        CTA 0: MMA issuer (one thread); both: TMEM allocation;
//   warp 2        activations (one thread): a TMA copy (4 x 64 K x half the tile's rows, 128-byte swizzle) per K stage; the copies of
//                 both CTAs complete on CTA 0's barrier;
//   warp 3        CTA 0: scheduler: draws units from a counter in global memory and hands them to both CTAs; both: counts
//                 drained gate/up units for their token tile;
//   warps 4-19    decode: group g = 0..3 of four warps fills every fourth A slot (128 K) of the ring; the same warps drain the
//                 accumulators.
// TMEM lanes 32q .. 32q+15 hold rows of the first tile of the pair (gate, or the even row tile), lanes 32q+16 .. 32q+31 the
// same rows of the second, so that the two values of a SwiGLU sit in one warp, sixteen lanes apart.
//
// Work is dealt one unit at a time from one list, gate/up units (phase 0) before down units (phase 1), ordered (token tile,
// pair). Units differ in cost by the rows of their tile (an expert's rows are split evenly over its tiles), so a fixed
// deal leaves SMs idle at the end of each GEMM; drawn from a counter, the down units fill the end of the gate/up
// phase. A down unit waits for the gate/up units of its token tile: those are drawn before any down unit, by clusters
// that are running, and a cluster stores its last gate/up unit whether or not the MMAs of its first down unit can start
// (pair_slots_before_drain), so the wait ends whatever part of the grid is resident. Which cluster computes a unit does not
// change its bits.
//
// MMAs are as wide as a tile's rows in steps of sixteen (eight rows in either CTA). kind::f16 with cta_group::2 and M = 256 takes N from 16
// to 256 in steps of 16, whichever memory A lies in: the check of tcgen05 operations in CUTLASS's CuTe DSL (MmaOp in cute/nvgpu/tcgen05/mma.py, which cites
// the PTX manual's section; its exceptions are 8-bit operands) makes no difference between them. Its C++ wrapper for A in tensor memory asserts
// 32, the one for A in shared memory 16. Every width is compared with the oracle (tests). In steps of 32 a row of steps took, before / after:
// 777 tokens at H4096 I1536 E128 422 / 411 us, 1500 tokens whose routes favour a few experts 619 / 607, 3012 skewed tokens of a rank 533 / 526,
// 8192 tokens of one rank of eight, H7168 I2048, 733 / 712.
//
// Numerics as in gemm.cuh: the same products, FP32 accumulation along K, the same roundings (the same bits as its tiles).
//
// Measured (both GEMMs, us, against one CTA to a tile of up to 128 tokens, which this replaces): 8192 tokens of Zipf routes at
// H4096 I1536 E128 1997 -> 1928; 8192 tokens at one rank of eight, H7168 I2048, 605 -> 540; 3012 skewed tokens at a rank, H4096 I4096,
// 462 -> 444; 777 tokens, 49 rows an expert, 397 -> 369. Bound by the hand-over of the K stages of the rings (activation rows and A
// slots come back, are refilled over L2 and by the decode warps, 1100 cycles a stage at the least) and, with full tiles, by the MMAs
// and the power limit; the tensor core also stands still while an accumulator of more than 128 columns is drained.
// Two K stages of token rows are in flight with tiles of more than 128 rows; narrower ones, which take one of a stage's two places, have four
// (pair_b_place). With two for all, the loads of 64 to 96 rows an expert, evenly spread, were up to 4 % behind the kernel replaced:
// whole steps at H4096 I1536 E128 with that kernel / two stages / four, 64 rows 468 / 471 / 458 us, 80 rows 552 / 560 / 541, 96
// rows 565 / 586 / 572; 32 of 256 experts at H7168 I2048, 80 rows 305 / 313 / 300, 128 rows 387 / 374 / 364.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gemm.cuh"
#include "layout.cuh"
#include "pair_sched.h"
#include "ptx.cuh"

namespace msk {

constexpr int PAIR_THREADS = 640;
constexpr int PAIR_DQ_WARP = 4;          // first decode warp
constexpr int PAIR_DQ_WARPS = 16;
constexpr int PAIR_SLOT_COLS = PAIR_SLOT_K / 2;
constexpr int PAIR_MAPS = 16;            // tensor maps per phase: boxes of 8, 16 .. 128 rows

struct PairCfg {
  static constexpr int BH = PAIR_BH;
  static constexpr int MAX_ROWS = 2 * BH;
  // TMEM: accumulators in the low columns (two buffers of BH columns, or both for a tile of more rows than that), the A ring above
  static constexpr int NSLOT = PAIR_NSLOT;
  static constexpr int A_BASE = TMEM_COLS - NSLOT * PAIR_SLOT_COLS;
  static constexpr int B_SUB_BYTES = BH * 128;           // 64 K of BH rows
  static constexpr int B_SLOT_BYTES = 2 * B_SUB_BYTES;
  static constexpr int NST = PAIR_NST;
  static constexpr int CTRL_BYTES = 1024;
  static constexpr int TABLE_INTS = MAX_LOCAL_EXPERTS + 4;
  static constexpr int SMEM_BYTES = NSLOT * B_SLOT_BYTES + NST * TILE_BYTES + CTRL_BYTES + 3 * TABLE_INTS * 4 + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory of a CTA");
  static_assert(2 * BH <= A_BASE, "TMEM budget");
};

struct PairParams {
  CUtensorMap tmap[2][PAIR_MAPS];        // per phase: f16 rows as [K / 64][rows][64], boxes 4 x 8(i + 1) x 64, 128-byte swizzle
  const uint8_t* w[2];                   // packed tiles
  const float* gs[2];
  __half* inter;                         // [R, I]
  __nv_bfloat16* y;                      // [R, H]
  const __nv_bfloat16* post_norm_w;      // nullable
  const int32_t* cnt;
  const int32_t* off;
  int32_t* status;
  unsigned long long* trace;             // nullable, stamps as in gemm.cuh
  unsigned int* ctr;                     // [0] next unit, [1] clusters that have left; zero between launches
  unsigned int* tile_done;               // per token tile: CTAs whose half of a gate/up unit is stored, zero between launches
  unsigned int* tile_seen;               // per token tile: CTAs of down units that have seen the count complete
  int K[2];
  int n_pairs[2];
  int nloc;
  int H, I;
  int first, last;                       // phases of this launch
};

struct alignas(16) PairUnit {              // written and read 16 bytes at a time
  int phase;                             // -1: no more units
  int expert, row0, rows, pair, tile;
  int nmma;                              // rows rounded up to 16
  int again;                             // its weights are read by other tiles of the expert as well
};

struct PairCtrl {
  uint64_t raw_full[PairCfg::NST], raw_empty[PairCfg::NST];  // weight stages (local)
  uint64_t full[PAIR_MARKS / 2];         // CTA 0: A and B of two slots (a K stage), from both CTAs
  uint64_t empty[PAIR_MARKS];            // the MMAs of a slot are done, committed into both CTAs
  uint64_t d_full[2];                    // committed into both CTAs
  uint64_t d_empty[2];                   // CTA 0: drained by both CTAs
  uint64_t u_full[PAIR_UNITS];           // local
  uint64_t u_empty[PAIR_UNITS];          // CTA 0: CTA 1 is done with the unit
  uint64_t u_done[PAIR_UNITS];           // local: the decode warps have stored their values of a unit, and every role has read its record
  PairUnit unit[PAIR_UNITS];
  int owed_tile[PAIR_UNITS];             // scheduler: tile to announce when a place's gate/up unit is stored, else -1
  uint32_t tmem_base;
  int abort_word;
};
static_assert(sizeof(PairCtrl) <= 1024 && offsetof(PairCtrl, unit) % 16 == 0, "control block");

// The accumulator buffer of each unit in turn: a tile of up to BH rows takes one of two buffers of BH columns, a wider
// one takes both. MMA issuer and decode warps walk the same sequence.
struct PairBuffers {
  uint32_t next = 0, par0 = 0, par1 = 0;
  bool wide;
  uint32_t buf, p0, p1;
  __device__ __forceinline__ void take(int nmma) {
    wide = nmma > PairCfg::BH;
    buf = wide ? 0u : next;
    p0 = par0;
    p1 = par1;
    if (wide || buf == 0u) par0 ^= 1u;
    if (wide || buf == 1u) par1 ^= 1u;
    next = wide ? 0u : (next ^ 1u);
  }
  __device__ __forceinline__ bool uses(uint32_t b) const { return wide || buf == b; }
};

// Accumulators of a unit -> SwiGLU values (phase 0) or output rows (phase 1) for one decode warp: lane quarter q, a quarter
// (`part`) of the columns, up to four steps of sixteen. The MMAs of a unit that needs the accumulators wait for release(), so
// it comes before the stores and arithmetic of the last two steps, whose values wait in registers; the first two are only
// brought down to packed results before it. (All four as raw values would need 64 registers beside the main loop's.)
template <typename Release>
__device__ __forceinline__ void pair_epilogue(const PairParams& p, const PairUnit& u, uint32_t d_tmem, int rank, int q, int part,
                                              int lane, Release release) {
  const int nc = ((u.nmma >> 2) + 15) & ~15, c0 = part * nc;   // whole steps of sixteen columns
  if (c0 >= u.rows) {
    release();
    return;
  }
  const int t = lane >> 4, r = rank * 64 + q * 16 + (lane & 15);   // tile of the pair, row inside it
  const int lim = min(nc, u.rows - c0);                            // columns this warp owes
  const uint32_t src = d_tmem + c0;
  const float gsc = p.gs[u.phase][u.expert];
  uint32_t a[2][16];
  auto load = [&](int c) {
    tmem_ld16(src + c, a[0]);
    if (c + 16 < lim) tmem_ld16(src + c + 16, a[1]);
    tmem_wait_ld();
  };
  if (u.phase == 0) {
    size_t ld = static_cast<size_t>(p.I);
    asm volatile("" : "+l"(ld));   // or its multiples are kept (and spilled) through the main loop
    __half* outp = p.inter + static_cast<size_t>(u.row0 + c0 + t * 8) * ld + u.pair * 128 + r;
    int left = lim - t * 8;        // columns from this lane's next one on
    uint32_t h[8];
    // lanes 0-15 hold the gate row, lanes 16-31 the up row; the lower half takes columns 0-7, the upper 8-15
    auto swiglu = [&](const uint32_t (&v)[16], int at) {
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const uint32_t s0 = __shfl_xor_sync(0xffffffffu, t ? v[j] : v[8 + j], 16);
        const uint32_t s1 = __shfl_xor_sync(0xffffffffu, t ? v[j + 1] : v[9 + j], 16);
        h[at + j / 2] = inter_pair(t ? s0 : v[j], t ? v[8 + j] : s0, t ? s1 : v[j + 1], t ? v[9 + j] : s1, gsc);
      }
    };
    auto store = [&](int at) {
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        if (left > j) *outp = __ushort_as_half(static_cast<unsigned short>(h[at + j / 2]));
        outp += ld;
        if (left > j + 1) *outp = __ushort_as_half(static_cast<unsigned short>(h[at + j / 2] >> 16));
        outp += ld;
      }
      outp += 8 * ld;
      left -= 16;
    };
    load(0);
    if (lim > 32) {
      swiglu(a[0], 0);
      swiglu(a[1], 4);
      load(32);
      release();
      store(0);
      store(4);
    } else {
      release();
    }
    const int rest = lim > 32 ? lim - 32 : lim;
    swiglu(a[0], 0);
    store(0);
    if (rest > 16) {
      swiglu(a[1], 4);
      store(4);
    }
  } else {
    size_t ld = static_cast<size_t>(p.H);
    asm volatile("" : "+l"(ld));
    const int col = (2 * u.pair + t) * 128 + r;
    float osc = gsc;
    if (p.post_norm_w != nullptr) osc *= 1.0f + __bfloat162float(p.post_norm_w[col]);
    __nv_bfloat16* outp = p.y + static_cast<size_t>(u.row0 + c0) * ld + col;
    int left = lim;
    auto store = [&](const uint32_t (&v)[16]) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (left > j) *outp = __float2bfloat16_rn(__uint_as_float(v[j]) * osc);
        outp += ld;
      }
      left -= 16;
    };
    load(0);
    if (lim > 32) {
      store(a[0]);
      store(a[1]);
      load(32);
    }
    release();
    store(a[0]);
    if (left > 0) store(a[1]);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1) moe_pair_kernel(const __grid_constant__ PairParams p) {
  using C = PairCfg;
  constexpr int BH = C::BH, NST = C::NST, NSLOT = C::NSLOT;
  extern __shared__ __align__(1024) uint8_t pair_smem[];
  uint8_t* b_ring = pair_smem;
  uint8_t* w_ring = pair_smem + NSLOT * C::B_SLOT_BYTES;
  PairCtrl& ctl = *reinterpret_cast<PairCtrl*>(w_ring + NST * TILE_BYTES);
  int* tile_start = reinterpret_cast<int*>(w_ring + NST * TILE_BYTES + C::CTRL_BYTES);
  int* cnt_s = tile_start + C::TABLE_INTS;
  int* off_s = cnt_s + C::TABLE_INTS;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();

  // ---------------------------------------------------------------- set-up
  if (tid == 0) {
    MSK_TR(TR_START);
    for (int i = 0; i < NST; ++i) {
      mbar_init(&ctl.raw_full[i], 1);
      mbar_init(&ctl.raw_empty[i], 8);             // two decode groups read a stage
    }
    for (int i = 0; i < PAIR_MARKS; ++i) {
      mbar_init(&ctl.empty[i], 1);
      if (i < PAIR_MARKS / 2) mbar_init(&ctl.full[i], 1 + 16);   // CTA 0's activation warp (with the bytes of both), eight decode warps of either CTA
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl.d_full[i], 1);
      mbar_init(&ctl.d_empty[i], 2 * PAIR_DQ_WARPS);
    }
    for (int i = 0; i < PAIR_UNITS; ++i) {
      mbar_init(&ctl.u_full[i], 1);
      mbar_init(&ctl.u_empty[i], 1);
      mbar_init(&ctl.u_done[i], PAIR_DQ_WARPS + 3 - rank);   // producer, activations and, in CTA 0, the MMA issuer
    }
    ctl.abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 2 && lane < PAIR_MAPS) prefetch_tensormap(&p.tmap[p.first][lane]);
  if (warp == 1) {
    tmem_alloc_pair(&ctl.tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                  // the other CTA's barriers are set up
  tc_fence_after();
  pdl_wait();                                      // tables and token rows of the kernels before
  pdl_launch_dependents();

  const uint32_t tmem = ctl.tmem_base;
  const uint32_t lead = map_to_rank(smem_u32(&ctl), 0u);   // CTA 0's control block as a cluster address
  volatile int* abortw = &ctl.abort_word;
  if (tid == 0) MSK_TR(TR_SETUP);
  auto lead_bar = [&](const uint64_t* bar) -> uint32_t { return lead + (smem_u32(bar) - smem_u32(&ctl)); };

  // Units, as the roles beside the decode warps walk them: wait_unit() waits for the next one and copies it (for a single
  // lane, or for a whole warp with one outcome), done_unit() hands its place back. Every wait of a whole warp is mbar_wait_warp:
  // what follows are full-warp instructions (elect, tcgen05.ld / st, __syncwarp).
  uint32_t ui = 0;
  auto wait_unit = [&](PairUnit& u, auto wait) -> bool {
    const uint32_t s = ui % PAIR_UNITS;
    if (!wait(&ctl.u_full[s], (ui / PAIR_UNITS) & 1u, abortw)) return false;
    const int4 x = *reinterpret_cast<const int4*>(&ctl.unit[s]), y = *(reinterpret_cast<const int4*>(&ctl.unit[s]) + 1);
    u.phase = x.x; u.expert = x.y; u.row0 = x.z; u.rows = x.w;
    u.pair = y.x; u.tile = y.y; u.nmma = y.z; u.again = y.w;
    ++ui;
    return true;
  };
  auto done_unit = [&]() { mbar_arrive(&ctl.u_done[(ui - 1u) % PAIR_UNITS]); };

  if (warp == 0) {
    // ------------------------------------------------------- weight producer
    if (lane == 0) {
      // Weights that one tile reads leave L2 first. Those of an expert with several tiles are read again within microseconds: first to leave
      // as well, they came from memory for each tile (8192 tokens of Zipf routes 2436 -> 2366 us in a row of steps, evenly spread 2400 -> 2327, one rank
      // of eight, H7168 I2048, 729 -> 716, 3012 skewed tokens of a rank 537 -> 527).
      const uint64_t once = policy_evict_first(), several = policy_evict_normal();
      uint32_t ws = 0, wpar = 0;
      bool ok = true;
      PairUnit u;
      while (ok && wait_unit(u, mbar_wait_inline)) {
        done_unit();
        if (u.phase < 0) break;
        const int nst = p.K[u.phase] / KS;
        const uint8_t* src = p.w[u.phase] + static_cast<size_t>(u.expert * p.n_pairs[u.phase] + u.pair) * nst * STAGE_W_BYTES + rank * TILE_BYTES;
        const uint64_t pol = u.again != 0 ? several : once;
        for (int ks = 0; ks < nst; ++ks) {
          if (!mbar_wait_inline(&ctl.raw_empty[ws], wpar ^ 1u, abortw)) { ok = false; break; }
          mbar_arrive_expect_tx(&ctl.raw_full[ws], TILE_BYTES);
          bulk_g2s(w_ring + ws * TILE_BYTES, src, TILE_BYTES, &ctl.raw_full[ws], pol);
          if (ui == 1u && ks == 0) MSK_TR(TR_FIRST_BULK);
          src += STAGE_W_BYTES;
          if (++ws == NST) { ws = 0; wpar ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------- MMA issuer
    if (rank == 0 && elect_one()) {                // one thread walks the whole loop (ptx.cuh, MSK_MMA_STEP)
      const uint64_t b_desc0 = smem_desc_kmajor_sw128(smem_u32(b_ring));   // slots and K steps advance its address field
      PairBuffers db;
      uint32_t st = 0;                             // K stage, through all units
      bool ready = false;                          // stage st was seen full while the one before was issued
      bool ok = true;
      PairUnit u;
      while (ok && wait_unit(u, mbar_wait_inline)) {
        done_unit();
        if (u.phase < 0) break;
        const uint32_t idesc = idesc_f16(FMT_F16, FMT_F16, 256, static_cast<uint32_t>(u.nmma));
        db.take(u.nmma);
        if (db.uses(0) && !mbar_wait_inline(&ctl.d_empty[0], db.p0 ^ 1u, abortw)) { ok = false; break; }
        if (db.uses(1) && !mbar_wait_inline(&ctl.d_empty[1], db.p1 ^ 1u, abortw)) { ok = false; break; }
        const uint32_t d_tmem = tmem + db.buf * static_cast<uint32_t>(BH);
        tc_fence_after();
        const uint32_t sub = static_cast<uint32_t>(u.nmma) * 4u;   // half of the rows, 128 bytes each, in units of 16 bytes
        uint32_t accumulate = 0u;
        for (int left = p.K[u.phase] / KS; left > 0; --left) {
          if (!ready && !mbar_wait_inline(&ctl.full[st & 3u], (st >> 2) & 1u, abortw)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sn = st + 1u, sl = (st & 1u) * 2u;
          const uint32_t place = pair_b_place(st, u.nmma) * C::B_SLOT_BYTES;
          ready = mma_stage_pair(d_tmem, tmem + C::A_BASE + sl * PAIR_SLOT_COLS, b_desc0 + (place >> 4), idesc, accumulate,
                                 smem_u32(&ctl.empty[(st & 3u) * 2u]), smem_u32(&ctl.full[sn & 3u]), (sn >> 2) & 1u, sub);
          st = sn;
          accumulate = 1u;
        }
        if (ok) {
          if (db.uses(0)) tc_commit_pair(&ctl.d_full[0]);
          if (db.uses(1)) tc_commit_pair(&ctl.d_full[1]);
        }
      }
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------- activations
    // One thread, one wait and one copy a K stage: as a warp that elects a lane for four copies, each half a stage behind a wait of its
    // own, this role took 850 cycles a stage beside the decode warps, and set the pace of tiles of few rows.
    const uint64_t keep = policy_evict_last();     // token rows are re-read by every pair of the expert
    uint32_t st = 0, wide_end = 0;                 // K stage, through all units; the one behind the last wide tile's
    bool ok = true;
    if (elect_one()) {
      int last_tile = -1;
      PairUnit u;
      while (ok && wait_unit(u, mbar_wait_inline)) {
        done_unit();
        if (u.phase < 0) break;
        const int half = u.nmma >> 1;
        const CUtensorMap* map = &p.tmap[u.phase][half / 8 - 1];
        const int row = u.row0 + static_cast<int>(rank) * half, K = p.K[u.phase];
        const uint32_t bytes = static_cast<uint32_t>(half) * 256u * 2u * 2u;   // 256 K of both CTAs' rows
        if (u.phase == 1 && p.first == 0) {
          if (u.tile != last_tile) {
            if (!grid_counter_wait(p.tile_done + u.tile, 2u * static_cast<unsigned>(p.n_pairs[0]), abortw)) { ok = false; break; }
            fence_proxy_async_all();               // ordinary stores of other SMs, about to be read by bulk copies
            last_tile = u.tile;
          }
          // the last CTA to have seen the count complete puts both counters back for the next launch
          const unsigned seen = atomicAdd(p.tile_seen + u.tile, 1u);
          if (seen == 2u * static_cast<unsigned>(p.n_pairs[1]) - 1u) {
            atomicExch(p.tile_done + u.tile, 0u);
            atomicExch(p.tile_seen + u.tile, 0u);
          }
        }
        for (int k = 0; k < K; k += KS, ++st) {
          const uint32_t before = pair_b_waits_for(st, u.nmma, wide_end);   // (of the first stages: a barrier that nothing has completed, parity 1)
          if (!mbar_wait_inline(&ctl.empty[before & 7u], (before >> 3) & 1u, abortw)) { ok = false; break; }
          if (rank == 0) mbar_arrive_expect_tx(&ctl.full[st & 3u], bytes);
          tma_load_3d_pair(b_ring + pair_b_place(st, u.nmma) * C::B_SLOT_BYTES, map, 0, row, k >> 6, lead_bar(&ctl.full[st & 3u]), keep);
        }
        if (u.nmma > BH) wide_end = st;
      }
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, ok);
    uint32_t n = 2u * __reduce_max_sync(0xffffffffu, st);
    // the commits of the last slots arrive in this CTA's shared memory: it stays until they have
    for (int i = 0; ok && i < PAIR_MARKS; ++i) {
      --n;
      if (!mbar_wait_warp(&ctl.empty[n & 7u], (n >> 3) & 1u, abortw)) break;
    }
  } else if (warp == 3) {
    // ------------------------------------------- scheduler; announces stored gate/up units
    // What the other roles do with a unit they release to this CTA only (u_done). From here the decode warps' stores are released to
    // the other SMs, and CTA 1's reads of the unit's record to CTA 0, which writes the next one there: a fence of that scope costs
    // a round trip to memory per unit, in the decode warps or the MMA issuer 1 to 5 % of the kernel. A place of the unit list is
    // handed back behind the drain of its unit, so a barrier is not met twice in a phase.
    auto announce = [&](int tile) {
      fence_proxy_async_all();                     // the rows' readers are bulk copies
      red_release_add(p.tile_done + tile, 1u);
    };
    if (rank != 0) {
      PairUnit u;
      while (lane == 0 && wait_unit(u, mbar_wait_inline) && u.phase >= 0) {
        const uint32_t i = ui - 1u;
        if (!mbar_wait_inline(&ctl.u_done[i % PAIR_UNITS], (i / PAIR_UNITS) & 1u, abortw)) break;
        if (u.phase == 0 && p.last == 1) announce(u.tile);
        mbar_arrive_release_cluster(lead_bar(&ctl.u_empty[i % PAIR_UNITS]));
      }
    } else {
      int carry = 0;
      for (int base = 0; base < p.nloc; base += 32) {   // exclusive prefix of per-expert tile counts
        const int e = base + lane;
        const int cn = e < p.nloc ? __ldcg(p.cnt + e) : 0;
        const int c = (cn + C::MAX_ROWS - 1) / C::MAX_ROWS;
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (e < p.nloc) {
          tile_start[e] = carry + incl - c;
          cnt_s[e] = cn;
          off_s[e] = __ldcg(p.off + e);
        }
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) tile_start[p.nloc] = carry;
      __syncwarp();
      if (lane == 0) {
        const int n0 = p.first == 0 ? carry * p.n_pairs[0] : 0;
        const int n = n0 + (p.last == 1 ? carry * p.n_pairs[1] : 0);
        const uint32_t peer = map_to_rank(smem_u32(&ctl), 1u);
        uint32_t i = 0;
        bool more = true;
        bool ok = true;
        while (more) {
          const int x = static_cast<int>(atomicAdd(p.ctr, 1u));
          int4 a = make_int4(-1, 0, 0, 0), b = make_int4(0, 0, 0, 0);
          more = x < n;
          if (more) {
            const int phase = (p.first == 1 || x >= n0) ? 1 : 0;
            const int v = phase ? x - n0 : x;
            const int tile = v / p.n_pairs[phase], pair = v - tile * p.n_pairs[phase];
            int lo = 0, hi = p.nloc;               // largest e with tile_start[e] <= tile
            while (hi - lo > 1) {
              const int mid = (lo + hi) >> 1;
              if (tile_start[mid] <= tile) lo = mid; else hi = mid;
            }
            const int nt = tile_start[lo + 1] - tile_start[lo], c = cnt_s[lo];
            const int per = pair_tile_rows(c, nt), at = (tile - tile_start[lo]) * per;
            const int rows = min(per, c - at);
            a = make_int4(phase, lo, off_s[lo] + at, rows);
            b = make_int4(pair, tile, pair_cols(rows), nt > 1 ? 1 : 0);
          }
          const uint32_t s = i % PAIR_UNITS;
          const uint32_t par = ((i / PAIR_UNITS) & 1u) ^ 1u;   // of the unit whose place this one takes
          if (i >= PAIR_UNITS) {
            if (!mbar_wait_inline(&ctl.u_done[s], par, abortw)) { ok = false; break; }
            if (ctl.owed_tile[s] >= 0) announce(ctl.owed_tile[s]);
          }
          if (!mbar_wait_cluster(&ctl.u_empty[s], par, abortw)) { ok = false; break; }
          const uint32_t at = smem_u32(&ctl.unit[s]) - smem_u32(&ctl), bar = smem_u32(&ctl.u_full[s]) - smem_u32(&ctl);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint32_t to = r ? peer : lead;
            mbar_arrive_expect_tx_cluster(to + bar, 32u);
            st_async_v4(to + at, a, to + bar);
            st_async_v4(to + at + 16, b, to + bar);
          }
          ctl.owed_tile[s] = more && a.x == 0 && p.last == 1 ? b.y : -1;
          ++i;
        }
        for (uint32_t j = i >= PAIR_UNITS ? i - PAIR_UNITS : 0u; ok && j < i; ++j) {   // the units still in the list
          const uint32_t s = j % PAIR_UNITS;
          if (ctl.owed_tile[s] < 0) continue;
          ok = mbar_wait_inline(&ctl.u_done[s], (j / PAIR_UNITS) & 1u, abortw);
          if (ok) announce(ctl.owed_tile[s]);
        }
      }
    }
  } else {
    // ------------------------------------------------- decode and epilogue
    const int g = (warp - PAIR_DQ_WARP) >> 2, q = warp & 3;
    const int kh = g & 1;                          // K half of a stage this group decodes
    // lane -> row of the stage: octet 2q + (lane >> 3 & 1) of this CTA's eight, tile lane >> 4 of the pair
    const uint32_t row_off = static_cast<uint32_t>((2 * (2 * q + ((lane >> 3) & 1)) + (lane >> 4)) * OCT_BYTES + (lane & 7) * 16);
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t a_tmem = tmem + lane_base + C::A_BASE + static_cast<uint32_t>(g * PAIR_SLOT_COLS);
    const uint32_t full_bar = lead_bar(&ctl.full[0]);
    uint32_t turn = 0;                             // slots this group has filled: always A slot g
    uint32_t ws = static_cast<uint32_t>(g >> 1), wpar = 0;   // stage of this group's next slot
    uint32_t sc = 0;                               // slots of the units before
    PairBuffers db;
    bool ok = true, owe = false;
    uint32_t di = 0;                               // next unit to drain; its record stays in the list until then
    int owed_cols = 0, owed_phase = 0;
    auto drain = [&]() -> bool {
      const PairUnit& r = ctl.unit[di % PAIR_UNITS];
      PairUnit u;
      u.phase = r.phase; u.expert = r.expert; u.row0 = r.row0; u.rows = r.rows; u.pair = r.pair; u.nmma = r.nmma;
      db.take(u.nmma);
      if (db.uses(0) && !mbar_wait_warp(&ctl.d_full[0], db.p0, abortw)) return false;
      if (db.uses(1) && !mbar_wait_warp(&ctl.d_full[1], db.p1, abortw)) return false;
      tc_fence_after();
      if (tid == PAIR_DQ_WARP * 32) { if (di == 0u) MSK_TR(TR_FIRST_DFULL); MSK_TR(TR_LAST_DFULL); }
      pair_epilogue(p, u, tmem + lane_base + db.buf * static_cast<uint32_t>(BH), static_cast<int>(rank), q, g, lane, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (db.uses(0)) mbar_arrive_cluster(lead_bar(&ctl.d_empty[0]));
          if (db.uses(1)) mbar_arrive_cluster(lead_bar(&ctl.d_empty[1]));
        }
      });
      __syncwarp();
      if (tid == PAIR_DQ_WARP * 32 && di == 0u) MSK_TR(TR_FIRST_EPI_DONE);
      if (lane == 0) mbar_arrive(&ctl.u_done[di % PAIR_UNITS]);   // (releases to this CTA only, which waits for no store)
      ++di;
      owe = false;
      return true;
    };
    bool more = true;
    while (ok && more) {
      const uint32_t us = ui % PAIR_UNITS;
      if (!mbar_wait_warp(&ctl.u_full[us], (ui / PAIR_UNITS) & 1u, abortw)) break;
      ++ui;
      const int phase = ctl.unit[us].phase, cols = ctl.unit[us].nmma;
      more = phase >= 0;
      const int nsl = more ? p.K[phase] / PAIR_SLOT_K : 0;
      // the unit before is drained once this warp has decoded ahead for this one, at the latest when its slots are done
      int ahead = pair_slots_before_drain(owed_phase, owed_cols, phase, cols);
      int s = static_cast<int>((static_cast<uint32_t>(g) - sc) & 3u);
      sc += static_cast<uint32_t>(nsl);
      while (true) {
        const bool slot = s < nsl;
        if (slot) {
          if (!mbar_wait_warp(&ctl.raw_full[ws], wpar, abortw)) { ok = false; break; }
          const uint32_t tile_row = smem_u32(w_ring + ws * TILE_BYTES) + row_off;
          uint32_t sf[2];
          asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(sf[0]), "=r"(sf[1]) : "r"(tile_row + OCT_CODE_BYTES + kh * 8));
          uint32_t o[2][16];
          auto decode = [&](int c, uint32_t (&d)[16]) {
            uint32_t w[4];
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                         : "r"(tile_row + (kh * 4 + c) * 128));
            const uint32_t sfw = sf[c >> 1];
            decode_chunk(w, (c & 1) ? (sfw >> 16) : sfw, d);
          };
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            decode(c, o[c]);
#pragma unroll
            for (int j = 0; j < 16; ++j) asm volatile("" : "+r"(o[c][j]));   // here, not behind the wait
          }
          // the slot this group filled last, NSLOT before this one
          if (!mbar_wait_warp(&ctl.empty[g + ((turn & 1u) ? 0 : NSLOT)], ((turn - 1u) >> 1) & 1u, abortw)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c >= 2) decode(c, o[c & 1]);
            tmem_st16(a_tmem + c * 16, o[c & 1]);
          }
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive_cluster(full_bar + (static_cast<uint32_t>(g >> 1) + (turn & 1u) * 2u) * 8u);
            mbar_arrive(&ctl.raw_empty[ws]);
          }
          ++turn;
          ws += 2;
          if (ws >= NST) { ws -= NST; wpar ^= 1u; }
          s += PAIR_GROUPS;
          --ahead;
        }
        if (owe && (!slot || ahead == 0) && !drain()) { ok = false; break; }
        if (!slot) break;
      }
      owed_cols = cols;
      owed_phase = phase;
      owe = true;
    }
  }

  // -------------------------------------------------------------- teardown
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (ctl.abort_word != 0) {
    // give copies and MMAs still in flight time to land before shared memory and TMEM are released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    if (tid == 0) atomicExch(p.status, MSK_DEV_ERR_TIMEOUT);
  }
  __syncthreads();
  cluster_sync();                                  // nothing of this CTA is still written or read by the other one
  if (tid == 0) MSK_TR(TR_END);
  if (rank == 0 && tid == 0) {
    // the last cluster to leave puts the unit counter back to zero for the next launch
    if (atomicAdd(p.ctr + 1, 1u) == gridDim.x / 2u - 1u) {
      atomicExch(p.ctr, 0u);
      atomicExch(p.ctr + 1, 0u);
    }
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, TMEM_COLS);
  }
}

}  // namespace msk
