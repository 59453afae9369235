// The whole routed-expert step of a few tokens in one cooperative launch: two or three, up to six with the pre-expert
// norm (the rule is few_takes() in msk_moe.cu; the tables below hold eight).
//
// There the step streams 85 to 300 MB of weights and every microsecond in which nothing
// streams counts: the kernel is built around a short prologue and as few hand-overs as possible, not around the
// tensor pipe. Weights go from shared memory to registers, are decoded there and multiplied with mma.sync
// (m16n8k16: 8 + 8 weight rows by up to 8 tokens), so there is no TMEM to allocate and no descriptor.
//
// Twelve working warps, one CTA per SM. A warp streams its part of a unit through a private ring of small bulk
// copies that its own lane 0 issues, and keeps the accumulators in registers. A gate/up unit (8 gate + 8 up rows
// over all of K) is the work of a team of two warps, half of K each; they meet
// once per unit, where one of them adds the two partials and runs the epilogue while the other goes on. A
// down unit (16 rows) is one warp's. So at most six units of a CTA are open at a time and the tiles of `inter`
// complete one after the other, before the last weights have arrived.
// (The tcgen05 kernel of gemm.cuh passes every half stage through a TMEM slot, and the pace of those
// hand-overs set its time: one token 40 us, of which 11.5 before the first MMA. Also built and slower than
// this form: all sixteen warps on one unit, with reducing warps behind them, 45 us at one token and 250 at
// eight (1 us per unit for the meeting alone); a warp per gate/up unit, 30 and 116: every tile completes at
// the very end, and 85 units do not go round 16 warps evenly.)
//
// Work. Gate/up units are dealt in order over the CTAs, so the shares differ by one unit (37 KB at K = 4096;
// whole tile pairs were 590 KB, and 96 of them left 52 SMs idle at one token). For the down GEMM every CTA
// owns output rows instead: groups of 16 rows for all tiles, so that the combine needs no further exchange
// between CTAs. Groups do not divide evenly (256 over 148 at H = 4096); the CTAs with fewer groups are
// dealt more gate/up units (FewDeal), which evens out the bytes per CTA. A CTA's gate/up units go round its
// teams and then its down units round its warps. A warp's ring runs ahead into its down weights while `inter` is
// not complete yet.
// `inter` is handed over per tile by a counter, as in gemm.cuh; with the post-expert norm the CTAs exchange
// one partial sum of squares per routed row before they combine. Every sum has a fixed order.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gemm.cuh"
#include "layout.cuh"
#include "ptx.cuh"
#include "route_sort.cuh"

namespace msk {

constexpr int FEW_WARPS = 12;
constexpr int FEW_TEAM = 2;                                // warps of a gate/up unit
constexpr int FEW_TEAMS = FEW_WARPS / FEW_TEAM;
constexpr int FEW_ROUTE_WARPS = 8;                         // route and sort; the others fetch the token rows
constexpr int FEW_THREADS = (FEW_WARPS + 1) * 32;         // the last warp signals finished units
constexpr int FEW_TOKENS = 8;                              // rows of a tile, and most tokens the tables hold
constexpr int FEW_ENTRIES = FEW_TOKENS * MAX_TOP_K;        // (token, slot) entries, and tiles
constexpr int FEW_KB_BYTES = 2 * OCT_BYTES;                // one K block of 8 + 8 rows
// Ring of a warp. More than some fifty bulk copies outstanding per SM slow the stream down, and 50 to 70 KB in flight
// are enough (measured, 16 warps with private rings, copies x slots: 4608 x 2 7.0 TB/s, 2304 x 2 7.0, 2304 x 3 6.7,
// 2304 x 5 5.2, 1152 x 10 3.1): two slots of two K blocks, or three of one where shared memory is short. (The K blocks of a
// slice are 2304-byte pieces, so a slot of two takes two copies. Slots of one block, three or four of them, with
// 12 warps: one token 35.8 and 35.6 us against 33.0, two with norms and router 64.0 and 59.6 against 57.5.)
constexpr int FEW_MAX_SLOTS = 3;

struct FewParams {
  const uint8_t* w13;
  const uint8_t* w2;
  const float* gs13;
  const float* gs2;
  const __nv_bfloat16* x;
  const __nv_bfloat16* pre_w;    // nullable: pre-expert RMS norm
  const __nv_bfloat16* post_w;   // nullable: post-expert RMS norm
  __half* xs;                    // shared F16 copy of x (share_x only)
  __half* inter;
  float* y;
  __nv_bfloat16* out;
  const float* logits;           // route == 1
  const float* bias;
  const int32_t* ids_in;         // route == 2
  const float* tw_in;
  int32_t* ids_out;
  float* tw_out;
  int32_t* cnt;
  int32_t* off;
  int32_t* perm;
  int32_t* inv;
  int32_t* status;
  unsigned int* tile_done;       // [tiles], zero between launches
  unsigned int* ctl;             // [0] CTAs that are done, [1] CTAs whose norm sums are written, [2] slices of xs written
  float* norm_part;              // [CTAs][rows]
  float* logits_copy;            // [T][E], with share_x and logits in host memory: one CTA fetches them, all read its copy; else null
  int32_t* ids_copy;             // [T][k] ids, [T][k] weights behind them: the same where both are given
  unsigned long long* trace;
  float pre_eps, post_eps, route_scale;
  int H, I, T, E, k, lo, nloc, mode, route;
  int share_x;                   // x lies in host memory: each CTA fetches a slice, all read the F16 copy
  int n_slots, slot_kb;          // ring slots of a warp, K blocks per slot
  uint32_t inv_oct1;             // ceil(2^32 / (I / 8))
  int part_bytes;                // partial sums of a warp: 128 bytes per two tile columns
  int n_light, w_light, w_heavy; // FewDeal
  int xb_off, ys_off, part_off, ctl_off;   // shared memory
};

struct FewCtl {
  uint64_t full[FEW_WARPS][FEW_MAX_SLOTS];
  uint64_t part_full[FEW_TEAMS][2], part_empty[FEW_TEAMS][2];
  float ss[FEW_WARPS - FEW_ROUTE_WARPS];
  int mail[FEW_TEAMS];                          // tile of a team's finished gate/up unit + 1, until it is signalled
  int abort_word;
  int n_tiles, n_rows;
  int ids[FEW_ENTRIES];
  float tw[FEW_ENTRIES];
  __align__(16) int key[FEW_ENTRIES];    // local expert << 8 | entry; INT_MAX without a local expert
  __align__(16) int lead[FEW_ENTRIES];   // the key of an entry that starts a tile, else INT_MAX
  short inv[FEW_ENTRIES];                // sorted row of an entry, or -1
  uint8_t row_entry[FEW_ENTRIES];        // entry of a sorted row
  int row_x[FEW_ENTRIES];                // byte offset of its token row in the x region
  short tile_expert[FEW_ENTRIES], tile_row0[FEW_ENTRIES];
  uint8_t tile_rows[FEW_ENTRIES];
};

// Waits of a whole warp. Every lane polls for itself (and so acquires what the barrier publishes), but the warp
// has one outcome: lanes that gave up one by one would leave the others behind in full-warp instructions, and
// without lane 0 a copy would start on a barrier that expects no bytes.
__device__ __forceinline__ bool warp_mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_word)) != 0;
}

// Lane 0 waits for a counter in global memory; the barrier behind the broadcast, which orders no memory by itself,
// passes on to the other lanes what lane 0 acquired.
__device__ __forceinline__ bool warp_counter_wait(const unsigned int* ctr, unsigned int target, volatile int* abort_word, int lane) {
  int ok = 1;
  if (lane == 0) ok = grid_counter_spin(ctr, target, abort_word) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();
  return ok != 0;
}

// Lane 0 puts `value` into a mailbox once it is empty (a bounded wait); the outcome goes to the whole warp.
__device__ __forceinline__ bool warp_mail_post(int* box, int value, volatile int* abort_word, int lane) {
  int ok = 1;
  if (lane == 0) {
    uint64_t t0 = 0;
    uint32_t polls = 0;
    while (ld_acquire_cta(box) != 0) {
      if ((++polls & 1023u) != 0u) continue;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > MSK_WAIT_LIMIT_NS) *abort_word = 1;
      if (*abort_word != 0) { ok = 0; break; }
    }
    if (ok) st_release_cta(box, value);
  }
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// Which gate/up units a CTA takes. CTAs below n_light take w_light units in every super-round, the others
// w_heavy (they own one group of output rows more); pass after pass in CTA order, so that neighbouring
// units stream at the same time and tiles complete in order.
struct FewDeal {
  int c, shares, n_light, w, wh, n_units, round;   // round: units of one super-round
  __host__ __device__ FewDeal(int cta, int n_ctas, int light, int w_light, int w_heavy, int units)
      : c(cta), shares(n_ctas), n_light(light), w(cta < light ? w_light : w_heavy), wh(w_heavy), n_units(units),
        round(w_heavy * n_ctas + (w_light - w_heavy) * light) {}
  // place of this CTA's unit number `pass` (below w) inside a super-round
  __host__ __device__ int place(int pass) const { return (pass < wh ? pass * shares : wh * shares + (pass - wh) * n_light) + c; }
  __host__ __device__ int count() const {
    const int full = n_units / round, rest = n_units - full * round;
    int n = full * w;
    for (int i = 0; i < w; ++i) n += place(i) < rest ? 1 : 0;
    return n;
  }
};

// The units of one warp in order: of the CTA's gate/up units every n_teams-th from its team's number on, then
// its down units (tile-major, own groups within a tile) number j, j + FEW_WARPS, ...
struct FewIter {
  int left;                 // gate/up units of this CTA from the current one on
  int base, pass;           // the current one's place in the deal
  int j;                    // down unit number
  __device__ void start(const FewDeal& d, int n_gate, int warp) {
    left = n_gate - warp / FEW_TEAM;
    base = 0;
    pass = warp / FEW_TEAM;
    if (left > 0) wrap(d);
    // the first down unit goes to the team behind the last gate/up unit
    j = (warp - n_gate % FEW_TEAMS * FEW_TEAM + FEW_WARPS) % FEW_WARPS;
  }
  __device__ void wrap(const FewDeal& d) {
    while (pass >= d.w) {
      pass -= d.w;
      base += d.round;
    }
  }
  __device__ bool gate() const { return left > 0; }
  __device__ int unit(const FewDeal& d) const { return base + d.place(pass); }
  __device__ void advance(const FewDeal& d) {
    if (left > 0) {
      left -= FEW_TEAMS;
      pass += FEW_TEAMS;
      if (left > 0) wrap(d);
    } else {
      j += FEW_WARPS;
    }
  }
};

// Top-k of one token by one warp: k rounds of two hardware warp reductions (largest orderable score, then the
// lowest expert that has it), the weights as route_one_token forms them. Same ids and weights, bit for bit.
template <int PER>
__device__ __forceinline__ void few_route(const float* row, const float* __restrict__ bias, int* ids_s,
                                          float* tw_s, int E, int k, int mode, float scale, int lane) {
  uint32_t key[PER];
  float raw[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    key[i] = 0u;
    raw[i] = 0.f;
    if (e < E) raw[i] = __ldcg(row + e);   // (may be another CTA's copy)
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    if (e < E) {
      float sel = raw[i];
      if (mode == 1) {
        raw[i] = 1.0f / (1.0f + expf(-raw[i] * scale));
        sel = raw[i] + (bias ? bias[e] : 0.f);
      }
      key[i] = max(orderable_u32(sel), 1u);   // 0 marks a taken or absent expert
    }
  }
  float my_val = 0.f;
  int my_id = 0;
#pragma unroll 1
  for (int s = 0; s < k; ++s) {
    uint32_t m = 0u;
#pragma unroll
    for (int i = 0; i < PER; ++i) m = max(m, key[i]);
    const uint32_t best = __reduce_max_sync(0xffffffffu, m);
    uint32_t at = 0xffffffffu;
#pragma unroll
    for (int i = PER - 1; i >= 0; --i)
      if (key[i] == best) at = i * 32 + lane;
    const int e = static_cast<int>(__reduce_min_sync(0xffffffffu, at));
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (i * 32 + lane == e) {
        v = raw[i];
        key[i] = 0u;
      }
    }
    v = __shfl_sync(0xffffffffu, v, e & 31);
    if (lane == s) {
      my_val = v;
      my_id = e;
    }
  }
  float w;
  if (mode == 0) {
    float m = lane < k ? my_val : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float ex = lane < k ? expf(my_val - m) : 0.f;
    float sum = ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    w = ex / sum;
  } else {
    float sum = lane < k ? my_val : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    w = my_val / (sum + 1e-15f);
  }
  if (lane < k) {
    ids_s[lane] = my_id;
    tw_s[lane] = w;
  }
}

// One K block (256) of a unit: decode the 8 + 8 weight rows and multiply. `wg`, `wu`: the two octet blocks in
// shared memory; `xk`: this lane's activation row at the block's first K, plus 16 bytes per word of the
// quad. Lane (row r, word q) holds codes K 8q .. 8q+7 of each 32-K chunk; the K order inside a chunk is the same for
// weights and activations, so 16 bytes of the activation row are the B operands of both MMAs of a chunk.
// The activations come from shared memory (xk) or, with REG_X, from registers loaded a block ahead (xr).
template <bool REG_X>
__device__ __forceinline__ void few_block(float (&d0)[4], float (&d1)[4], const uint8_t* wg, const uint8_t* wu,
                                          const uint8_t* xk, const uint4 (&xr)[8], int lane) {
  const uint32_t sel = (lane & 2) ? 0x7531u : 0x6420u;   // words 0, 1 of a chunk lie in its first scale block, 2, 3 in its second
  uint32_t s[8];   // chunk c: F16 scales (gate row, up row)
  {
    const uint4 g = *reinterpret_cast<const uint4*>(wg + OCT_CODE_BYTES + (lane >> 2) * 16);
    const uint4 v = *reinterpret_cast<const uint4*>(wu + OCT_CODE_BYTES + (lane >> 2) * 16);
    const uint32_t g4[2] = {prmt(g.x, g.y, sel), prmt(g.z, g.w, sel)}, v4[2] = {prmt(v.x, v.y, sel), prmt(v.z, v.w, sel)};
#pragma unroll
    for (int c = 0; c < 8; ++c)
      s[c] = cvt_e4m3x2_f16(static_cast<uint16_t>(prmt(g4[c >> 2], v4[c >> 2], 0x40u + 0x11u * (c & 3))));
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t a = *reinterpret_cast<const uint32_t*>(wg + c * 128 + lane * 4);
    const uint32_t b = *reinterpret_cast<const uint32_t*>(wu + c * 128 + lane * 4);
    const uint4 x = REG_X ? xr[c] : *reinterpret_cast<const uint4*>(xk + c * 64);
    const uint32_t s0 = prmt(s[c], s[c], 0x1010u), s1 = prmt(s[c], s[c], 0x3232u);
    uint32_t h[4], g[4];
    cvt_e2m1x8_f16(a, h[0], h[1], h[2], h[3]);
    cvt_e2m1x8_f16(b, g[0], g[1], g[2], g[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      h[j] = hmul2_f16(h[j], s0);
      g[j] = hmul2_f16(g[j], s1);
    }
    mma_16816(d0, h[0], g[0], h[1], g[1], x.x, x.y);
    mma_16816(d1, h[2], g[2], h[3], g[3], x.z, x.w);
  }
}

__global__ void __launch_bounds__(FEW_THREADS, 1) moe_few_kernel(const __grid_constant__ FewParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  FewCtl& ctl = *reinterpret_cast<FewCtl*>(smem + p.ctl_off);
  uint8_t* xb = smem + p.xb_off;
  float* ys = reinterpret_cast<float*>(smem + p.ys_off);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cta = static_cast<int>(blockIdx.x), n_ctas = static_cast<int>(gridDim.x);
  const int n_entries = p.T * p.k;
  const int x_stride = p.H * 2 + 64;   // 64 bytes of skew: two rows of a quarter-warp in different banks
  volatile int* abortw = &ctl.abort_word;
  const bool shared_routes = p.logits_copy != nullptr || p.ids_copy != nullptr;

  if (tid < FEW_TEAMS) ctl.mail[tid] = 0;
  if (tid == 0) {
    MSK_TR(TR_START);
    ctl.abort_word = 0;
    ctl.n_tiles = 0;
    ctl.n_rows = 0;
  }
  if (lane == 0 && warp < FEW_WARPS) {
    for (int i = 0; i < p.n_slots; ++i) mbar_init(&ctl.full[warp][i], 1);
    if (warp < FEW_TEAMS) {
      for (int i = 0; i < 2; ++i) {
        mbar_init(&ctl.part_full[warp][i], FEW_TEAM);
        mbar_init(&ctl.part_empty[warp][i], 1);
      }
    }
    fence_mbar_init();
  }
  if (tid < FEW_ENTRIES) {
    ctl.key[tid] = 0x7fffffff;
    ctl.lead[tid] = 0x7fffffff;
  }
  pdl_wait();
  if (p.share_x) {
    const int n8 = p.T * (p.H / 8);
    const uint4* src = reinterpret_cast<const uint4*>(p.x);
    uint4* dst = reinterpret_cast<uint4*>(p.xs);
    for (int i = cta * FEW_THREADS + tid; i < n8; i += n_ctas * FEW_THREADS) {
      const uint4 v = src[i];
      dst[i] = make_uint4(bf16x2_to_f16x2(v.x), bf16x2_to_f16x2(v.y), bf16x2_to_f16x2(v.z), bf16x2_to_f16x2(v.w));
    }
    // The logits once over PCIe as well: 148 CTAs that fetched a row of 512 bytes each had it after 3 to 8.5 us, behind which
    // their slices of the rows queued too. A step from and to pinned memory, 128 experts: 1 token 42.9 -> 39.4 us, 2 tokens
    // 57.8 -> 53.4 us, together with the one warp that polls below. Given ids and weights in the same way: 1 token 43 - 50 -> 38.7 us, 2 tokens
    // 60 - 65 -> 55.0 us.
    if (p.logits_copy != nullptr && cta == n_ctas - 1)
      for (int i = tid; i < p.T * p.E; i += FEW_THREADS) p.logits_copy[i] = p.logits[i];
    if (p.ids_copy != nullptr && cta == n_ctas - 1 && tid < n_entries) {
      p.ids_copy[tid] = p.ids_in[tid];
      p.ids_copy[n_entries + tid] = __float_as_int(p.tw_in[tid]);
    }
    __threadfence();
  }
  __syncthreads();
  if (p.share_x && tid == 0) atomicAdd(p.ctl + 2, 1u);

  if (warp < FEW_ROUTE_WARPS) {
    // ---- routing (a warp per token) and the stable sort (brute force: at most 128 entries)
    if (shared_routes) named_bar_sync(3, FEW_WARPS * 32);   // behind the wait below, of the warps that fetch the rows
    if (p.route == 1) {
      if (warp < p.T) {
        const float* row = (p.logits_copy != nullptr ? p.logits_copy : p.logits) + static_cast<size_t>(warp) * p.E;
        int* ids_s = ctl.ids + warp * p.k;
        float* tw_s = ctl.tw + warp * p.k;
        if (p.E <= 128) few_route<4>(row, p.bias, ids_s, tw_s, p.E, p.k, p.mode, p.route_scale, lane);
        else few_route<MAX_EXPERTS / 32>(row, p.bias, ids_s, tw_s, p.E, p.k, p.mode, p.route_scale, lane);
      }
      named_bar_sync(1, 256);
    } else if (tid < n_entries) {
      ctl.ids[tid] = p.ids_copy != nullptr ? __ldcg(p.ids_copy + tid) : p.ids_in[tid];
      ctl.tw[tid] = p.ids_copy != nullptr ? __int_as_float(__ldcg(p.ids_copy + n_entries + tid)) : p.tw_in[tid];
    }
    if (tid == 0) MSK_TR(TR_TOPK);
    int l = -1, key = 0x7fffffff, q = 0, r = 0, c = 0;
    if (tid < n_entries) {
      l = local_expert(ctl.ids[tid], p.lo, p.nloc);
      if (l >= 0) key = (l << 8) | tid;
      ctl.key[tid] = key;
    }
    named_bar_sync(1, 256);
    if (l >= 0) {
      for (int j = 0; j < n_entries; j += 4) {
        const int4 kk = *reinterpret_cast<const int4*>(&ctl.key[j]);
        const int kv[4] = {kk.x, kk.y, kk.z, kk.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const bool below = kv[m] < key, same = (kv[m] >> 8) == l;
          q += below ? 1 : 0;
          r += (below && same) ? 1 : 0;
          c += same ? 1 : 0;
        }
      }
      ctl.row_entry[q] = static_cast<uint8_t>(tid);
      ctl.row_x[q] = tid / p.k * x_stride;
      if ((r & (FEW_TOKENS - 1)) == 0) {
        ctl.lead[tid] = key;
        atomicAdd(&ctl.n_tiles, 1);
      }
      atomicAdd(&ctl.n_rows, 1);
    }
    if (tid < n_entries) ctl.inv[tid] = static_cast<short>(l >= 0 ? q : -1);
    named_bar_sync(1, 256);
    if (l >= 0 && (r & (FEW_TOKENS - 1)) == 0) {
      int t = 0;
      for (int j = 0; j < n_entries; j += 4) {
        const int4 kk = *reinterpret_cast<const int4*>(&ctl.lead[j]);
        t += (kk.x < key ? 1 : 0) + (kk.y < key ? 1 : 0) + (kk.z < key ? 1 : 0) + (kk.w < key ? 1 : 0);
      }
      ctl.tile_expert[t] = static_cast<short>(l);
      ctl.tile_row0[t] = static_cast<short>(q);
      ctl.tile_rows[t] = static_cast<uint8_t>(min(FEW_TOKENS, c - r));
    }
    if (tid == 0) MSK_TR(TR_ROUTED);
  } else if (warp < FEW_WARPS) {
    // ---- token rows as F16 into shared memory, up to four warps per row
    constexpr int XW = FEW_WARPS - FEW_ROUTE_WARPS;
    const int xw = warp - FEW_ROUTE_WARPS, wpr = p.T == 1 ? XW : p.T == 2 ? XW / 2 : 1;
    const int i_first = (xw % wpr) * 32 + lane, i_step = wpr * 32, n16 = p.H / 8;
    if (p.share_x) {
      // One warp polls, the others wait for it: with four of each of 148 CTAs on the counter's line, the counts behind which they
      // wait came microseconds late.
      if (xw == 0) warp_counter_wait(p.ctl + 2, static_cast<unsigned int>(n_ctas), abortw, lane);
      named_bar_sync(3, shared_routes ? FEW_WARPS * 32 : XW * 32);
      const bool go = __all_sync(0xffffffffu, *abortw == 0);
      for (int t = xw / wpr; t < p.T && go; t += XW / wpr) {
        const uint4* src = reinterpret_cast<const uint4*>(p.xs + static_cast<size_t>(t) * p.H);
        uint4* dst = reinterpret_cast<uint4*>(xb + t * x_stride);
        for (int i = i_first; i < n16; i += i_step) dst[i] = __ldcg(src + i);
      }
    } else
    for (int t = xw / wpr; t < p.T; t += XW / wpr) {
      uint4* dst = reinterpret_cast<uint4*>(xb + t * x_stride);
      const uint4* src = reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(t) * p.H);
      float ss = 0.f;
      for (int i0 = i_first; i0 < n16; i0 += 8 * i_step) {
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (i0 + j * i_step < n16) v[j] = __ldg(src + i0 + j * i_step);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (i0 + j * i_step >= n16) continue;
          if (p.pre_w == nullptr) {
            dst[i0 + j * i_step] = make_uint4(bf16x2_to_f16x2(v[j].x), bf16x2_to_f16x2(v[j].y), bf16x2_to_f16x2(v[j].z),
                                              bf16x2_to_f16x2(v[j].w));
          } else {
            dst[i0 + j * i_step] = v[j];
            const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const float lo = __uint_as_float(w[m] << 16), hi = __uint_as_float(w[m] & 0xFFFF0000u);
              ss += lo * lo + hi * hi;
            }
          }
        }
      }
      if (p.pre_w != nullptr) {   // x * rsqrt(mean(x^2) + eps) * (1 + pre_w), one BF16 rounding (copy_rows_kernel)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        float tot = ss;
        if (wpr > 1) {   // one row per group of warps: no warp comes round twice
          if (lane == 0) ctl.ss[xw] = ss;
          named_bar_sync(2, XW * 32);
          tot = 0.f;
          for (int w = 0; w < wpr; ++w) tot += ctl.ss[xw / wpr * wpr + w];   // fixed order
        }
        const float rs = rsqrtf(tot / static_cast<float>(p.H) + p.pre_eps);
        const uint4* g = reinterpret_cast<const uint4*>(p.pre_w);
        for (int i = i_first; i < n16; i += i_step) {
          const uint4 v = dst[i], gv = __ldg(g + i);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w}, gw[4] = {gv.x, gv.y, gv.z, gv.w};
          uint32_t o4[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const float lo = __uint_as_float(w[m] << 16) * rs * (1.0f + __uint_as_float(gw[m] << 16));
            const float hi = __uint_as_float(w[m] & 0xFFFF0000u) * rs * (1.0f + __uint_as_float(gw[m] & 0xFFFF0000u));
            const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
            o4[m] = bf16x2_to_f16x2(*reinterpret_cast<const uint32_t*>(&b));
          }
          dst[i] = make_uint4(o4[0], o4[1], o4[2], o4[3]);
        }
      }
    }
  }
  __syncthreads();

  // ---- units
  const int n_kb1 = p.H / KS, n_kb2 = p.I / KS;
  const int oct1 = p.I / OCT_ROWS, groups = p.H / (2 * OCT_ROWS);
  const int first_group = n_ctas - 1 - cta;                      // this CTA's groups: first_group + g * n_ctas
  const int n_own = first_group < groups ? (groups - first_group + n_ctas - 1) / n_ctas : 0;
  const int n_tiles = ctl.n_tiles, n_down = n_tiles * n_own;
  const FewDeal deal(cta, n_ctas, p.n_light, p.w_light, p.w_heavy, n_tiles * oct1);
  const int n_gate = deal.count();
  if (warp == FEW_WARPS) {
    // ---- signals: a fence that covers a unit's stores takes a microsecond or two while the memory system
    // streams; this warp waits for it in place of the warp that computes (eight tokens: 125 -> 118 us)
    int left = n_gate;
    uint32_t polls = 0;
    uint64_t t0 = globaltimer_ns();
    while (left > 0) {
      const int m = lane < FEW_TEAMS ? ld_acquire_cta(&ctl.mail[lane]) : 0;
      const unsigned have = __ballot_sync(0xffffffffu, m != 0);
      if (have != 0u) {
        __threadfence();
        if (m != 0) {
          red_release_add(p.tile_done + (m - 1), 1u);
          st_release_cta(&ctl.mail[lane], 0);
        }
        left -= __popc(have);
        __syncwarp();
        polls = 0;
        t0 = globaltimer_ns();
      } else {
        __nanosleep(32);
        if ((++polls & 255u) == 0u) {
          int stop = 0;
          if (lane == 0) {
            if (*abortw == 0 && globaltimer_ns() - t0 > MSK_WAIT_LIMIT_NS) *abortw = 1;
            stop = *abortw;
          }
          if (__shfl_sync(0xffffffffu, stop, 0) != 0) break;
        }
      }
    }
  } else {
    const int r = lane >> 2, q = lane & 3;
    const int slot_kb = p.slot_kb, slot_bytes = slot_kb * FEW_KB_BYTES;
    uint8_t* ring = smem + warp * p.n_slots * slot_bytes;
    uint64_t* full = ctl.full[warp];
    const int team = warp / FEW_TEAM, part = warp % FEW_TEAM;
    const int kb_a = part * n_kb1 / FEW_TEAM, kb_b = (part + 1) * n_kb1 / FEW_TEAM;   // this warp's K blocks of a gate/up unit
    // issue side: the next piece to fetch
    FewIter is;
    is.start(deal, n_gate, warp);
    const uint64_t pol = policy_evict_first();
    const uint8_t* src = nullptr;   // next K block to fetch
    int is_left = 0;   // K blocks left of the unit being fetched
    bool begun = false;
    auto issue = [&](int slot) {    // warp-uniform; lane 0 copies
      while (is_left <= 0) {
        if (begun) is.advance(deal);
        begun = true;
        if (is.gate()) {
          const int u = is.unit(deal), t = static_cast<int>(__umulhi(static_cast<uint32_t>(u), p.inv_oct1));
          const int o = u - t * oct1;
          src = p.w13 + (static_cast<size_t>(ctl.tile_expert[t]) * (oct1 >> 4) + (o >> 4)) * n_kb1 * STAGE_W_BYTES + kb_a * STAGE_W_BYTES +
                (o & 15) * FEW_KB_BYTES;
          is_left = kb_b - kb_a;
        } else if (is.j < n_down) {
          const int t = is.j / n_own, g = is.j - t * n_own;
          const int grp = first_group + g * n_ctas;
          src = p.w2 + (static_cast<size_t>(ctl.tile_expert[t]) * (groups >> 4) + (grp >> 4)) * n_kb2 * STAGE_W_BYTES +
                (grp & 15) * FEW_KB_BYTES;
          is_left = n_kb2;
        } else {
          return;
        }
      }
      const int n = min(slot_kb, is_left);
      // a K block per lane (one lane issuing both took longer than the copies overlap: one token 34.8 against 33.0 us,
      // two with norms and router 62 against 57.5)
      if (lane == 0) mbar_arrive_expect_tx(&full[slot], static_cast<uint32_t>(n * FEW_KB_BYTES));
      __syncwarp();
      if (lane < n)
        bulk_g2s(ring + slot * slot_bytes + lane * FEW_KB_BYTES, src + lane * STAGE_W_BYTES, FEW_KB_BYTES, &full[slot], pol);
      src += n * STAGE_W_BYTES;
      is_left -= slot_kb;
    };
    for (int i = 0; i < p.n_slots; ++i) issue(i);
    if (tid == 0) MSK_TR(TR_FIRST_BULK);
    // consume side
    FewIter it;
    it.start(deal, n_gate, warp);
    int slot = 0;
    uint32_t par = 0;
    bool ok = __all_sync(0xffffffffu, *abortw == 0);
    const uint4 no_x[8] = {};
    uint8_t* parts = smem + p.part_off + (2 * team * FEW_TEAM) * p.part_bytes;
    uint32_t n_unit = 0;
    for (; ok && it.gate(); it.advance(deal), ++n_unit) {
      const int u = it.unit(deal), t = static_cast<int>(__umulhi(static_cast<uint32_t>(u), p.inv_oct1)), o = u - t * oct1;
      const int rows = ctl.tile_rows[t], row0 = ctl.tile_row0[t];
      const float gs = p.gs13[ctl.tile_expert[t]];
      const uint8_t* xk = xb + ctl.row_x[row0 + min(r, rows - 1)] + q * 16 + kb_a * (KS * 2);
      float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
      for (int kb = kb_a; kb < kb_b; kb += slot_kb) {
        if (!warp_mbar_wait(&full[slot], par, abortw)) { ok = false; break; }
        const uint8_t* w = ring + slot * slot_bytes;
        for (int b = min(slot_kb, kb_b - kb); b > 0; --b, xk += KS * 2, w += FEW_KB_BYTES)
          few_block<false>(d0, d1, w, w + OCT_BYTES, xk, no_x, lane);
        __syncwarp();
        issue(slot);
        if (++slot == p.n_slots) { slot = 0; par ^= 1u; }
      }
      if (!ok) break;
      // the team meets: its warps take turns in adding the two partials (in K order) and finishing the unit
      const uint32_t pb = n_unit & 1u, pp = (n_unit >> 1) & 1u;
      if (!warp_mbar_wait(&ctl.part_empty[team][pb], pp ^ 1u, abortw)) { ok = false; break; }
      uint8_t* pbuf = parts + pb * FEW_TEAM * p.part_bytes + (q * 8 + r) * 16;
      if (2 * q < rows)
        *reinterpret_cast<float4*>(pbuf + part * p.part_bytes) = make_float4(d0[0] + d1[0], d0[1] + d1[1], d0[2] + d1[2], d0[3] + d1[3]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.part_full[team][pb]);
      if (part == static_cast<int>(n_unit % FEW_TEAM)) {
        if (!warp_mbar_wait(&ctl.part_full[team][pb], pp, abortw)) { ok = false; break; }
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (2 * q < rows) {
#pragma unroll
          for (int w = 0; w < FEW_TEAM; ++w) {
            const float4 v = *reinterpret_cast<const float4*>(pbuf + w * p.part_bytes);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.part_empty[team][pb]);
        __half* dst = p.inter + static_cast<size_t>(row0 + 2 * q) * p.I + o * OCT_ROWS + r;
        if (2 * q < rows) dst[0] = inter_value(silu_f(s.x * gs) * (s.z * gs));
        if (2 * q + 1 < rows) dst[p.I] = inter_value(silu_f(s.y * gs) * (s.w * gs));
        __syncwarp();
        // (the box is empty unless the signalling warp lags a whole unit behind)
        if (!warp_mail_post(&ctl.mail[team], t + 1, abortw, lane)) { ok = false; break; }
      }
    }
    if (tid == 0) MSK_TR(TR_LAST_DFULL);
    uint4 xn[8];              // rows of inter from L2, a K block ahead of its use
    for (; ok && it.j < n_down; it.advance(deal)) {
      const int t = it.j / n_own, g = it.j - t * n_own;
      const int rows = ctl.tile_rows[t], row0 = ctl.tile_row0[t];
      const float gs = p.gs2[ctl.tile_expert[t]];
      const int grp = first_group + g * n_ctas, col = (grp >> 4) * 256 + (grp & 15) * OCT_ROWS + r;
      float o0 = gs, o1 = gs;
      if (p.post_w != nullptr) {
        o0 *= 1.0f + __bfloat162float(p.post_w[col]);
        o1 *= 1.0f + __bfloat162float(p.post_w[col + 128]);
      }
      const uint8_t* xk = reinterpret_cast<const uint8_t*>(p.inter + static_cast<size_t>(row0 + min(r, rows - 1)) * p.I) + q * 16;
      if (!warp_counter_wait(p.tile_done + t, static_cast<unsigned int>(oct1), abortw, lane)) { ok = false; break; }
#pragma unroll
      for (int c = 0; c < 8; ++c) xn[c] = __ldcg(reinterpret_cast<const uint4*>(xk + c * 64));
      float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
      for (int kb = 0; kb < n_kb2; kb += slot_kb) {
        if (!warp_mbar_wait(&full[slot], par, abortw)) { ok = false; break; }
        const uint8_t* w = ring + slot * slot_bytes;
        for (int b = 0; b < min(slot_kb, n_kb2 - kb); ++b, w += FEW_KB_BYTES) {
          uint4 xc[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) xc[c] = xn[c];
          xk += KS * 2;
          if (kb + b + 1 < n_kb2) {
#pragma unroll
            for (int c = 0; c < 8; ++c) xn[c] = __ldcg(reinterpret_cast<const uint4*>(xk + c * 64));
          }
          few_block<true>(d0, d1, w, w + OCT_BYTES, nullptr, xc, lane);
        }
        __syncwarp();
        issue(slot);
        if (++slot == p.n_slots) { slot = 0; par ^= 1u; }
      }
      if (!ok) break;
      const int row = row0 + 2 * q;
      float* yd = p.y + static_cast<size_t>(row) * p.H + col;
      float* sd = ys + (row * n_own + g) * 16 + r;
      if (2 * q < rows) {
        yd[0] = sd[0] = (d0[0] + d1[0]) * o0;
        yd[128] = sd[8] = (d0[2] + d1[2]) * o1;
      }
      if (2 * q + 1 < rows) {
        yd[p.H] = sd[n_own * 16] = (d0[1] + d1[1]) * o0;
        yd[p.H + 128] = sd[n_own * 16 + 8] = (d0[3] + d1[3]) * o1;
      }
    }
  }
  if (cta == 0) {   // tables and routing for whoever asks for them later
    for (int e = tid; e <= p.nloc; e += FEW_THREADS) {
      int below = 0, here = 0;
      for (int j = 0; j < n_entries; ++j) {
        const int le = ctl.key[j] >> 8;
        below += le < e ? 1 : 0;
        here += le == e ? 1 : 0;
      }
      p.off[e] = below;
      if (e < p.nloc) p.cnt[e] = here;
    }
    for (int i = tid; i < n_entries; i += FEW_THREADS) {
      p.inv[i] = ctl.inv[i];
      if (i < ctl.n_rows) p.perm[i] = ctl.row_entry[i];
      if (p.route == 1) {
        p.ids_out[i] = ctl.ids[i];
        p.tw_out[i] = ctl.tw[i];
      }
    }
  }

  // ---- combine of the rows this CTA owns
  __syncwarp();
  __syncthreads();
  const int n_rows = ctl.n_rows;
  if (p.post_w != nullptr && ctl.abort_word == 0 && n_own > 0) {
    constexpr int NW = FEW_THREADS / 32;
    for (int row = warp; row < n_rows; row += NW) {
      float ss = 0.f;
      for (int i = lane; i < n_own * 16; i += 32) {
        const float v = ys[row * n_own * 16 + i];
        ss += v * v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) p.norm_part[static_cast<size_t>(cta) * n_rows + row] = ss;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      atomicAdd(p.ctl + 1, 1u);
      grid_counter_spin(p.ctl + 1, static_cast<unsigned int>(min(n_ctas, groups)), abortw);
    }
    __syncthreads();
    const int c_first = n_ctas - min(n_ctas, groups);   // CTAs that own rows
    for (int i = warp; i < n_entries; i += NW) {
      const int row = ctl.inv[i];
      if (row < 0) continue;
      float ss = 0.f;
      for (int c = c_first + lane; c < n_ctas; c += 32) ss += __ldcg(p.norm_part + static_cast<size_t>(c) * n_rows + row);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) ctl.tw[i] *= rsqrtf(ss / static_cast<float>(p.H) + p.post_eps);
    }
    __syncthreads();
  }
  if (ctl.abort_word == 0) {
    for (int i = tid; i < p.T * n_own * 16; i += FEW_THREADS) {
      const int rr = i & 15, tg = i >> 4, g = tg % n_own, t = tg / n_own;
      float acc = 0.f;
      for (int s = 0; s < p.k; ++s) {   // slot order
        const int row = ctl.inv[t * p.k + s];
        if (row >= 0) acc += ys[(row * n_own + g) * 16 + rr] * ctl.tw[t * p.k + s];
      }
      const int grp = first_group + g * n_ctas;
      p.out[static_cast<size_t>(t) * p.H + (grp >> 4) * 256 + (rr >> 3) * 128 + (grp & 15) * OCT_ROWS + (rr & 7)] = __float2bfloat16_rn(acc);
    }
    if (tid == 0) {
      MSK_TR(TR_END);
      // the last CTA to leave puts the counters back to zero for the next launch
      const unsigned int old = atomicAdd(p.ctl, 1u);
      if (old == static_cast<unsigned int>(n_ctas) - 1u) {
        for (int t = 0; t < n_tiles; ++t) p.tile_done[t] = 0u;
        p.ctl[1] = 0u;
        p.ctl[2] = 0u;
        __threadfence();
        p.ctl[0] = 0u;
      }
    }
  } else {
    const uint64_t t0 = globaltimer_ns();   // copies still in flight land before shared memory is released
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    if (tid == 0) atomicExch(p.status, MSK_DEV_ERR_TIMEOUT);
  }
}

}  // namespace msk
