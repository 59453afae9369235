// Router logits as a tcgen05 GEMM with the FP32 router weight held as an exact-sum pair of BF16
// matrices: logits[t, e] = sum_h x[t, h] * (hi[e, h] + lo[e, h]), hi = bf16(w), lo = bf16(w - hi),
// BF16 x BF16 products (exact in FP32), FP32 accumulation in TMEM. This is how the reference's layers
// feed their routing (muse_decode_layer/py/05_tune.py:279-286, muse_prefill_layer/py/00_layer.py:369-374:
// the two halves stacked as one [2E, H] weight of their dense BF16 GEMM); its FP32 matvec
// (muse_decode_layer/cuda/router_fp32.cu:4-40) is the few-token form, msk_moe_router_logits here.
//
// A cluster of up to eight CTAs per (128 experts, N tokens), each over its run of K steps: D[128 experts, N tokens]
// in TMEM, both halves accumulated into the same accumulator (per 16-wide K step first the hi product, then the lo
// product: a fixed order). The partial sums meet in the CTAs' shared memory, in rank order. There is one tile
// of experts and few of tokens, so without the split in K a handful of CTAs would each stream the whole weight
// through a ring of four steps: 23 - 31 us for 16 to 2000 tokens (E = 128, H = 4096), 6 - 11 with it; against
// 64 bits the error falls from 9.5e-6 to 2.7e-6 (shorter sums).
//   warp 0   producer: 2-D TMA loads (128-byte swizzle) of the hi tile, the lo tile and the token tile
//            of every 64-wide K step into a ring;
//   warp 1   MMA issuer (tcgen05.mma kind::f16, both operands from shared memory), owns the TMEM allocation;
//   warps 2-5 TMEM -> shared memory [token][128 experts]; then all threads sum a share of the tokens over
//            the cluster and write logits (FP32 [T, E]).
// All waits are bounded (ptx.cuh); a wait that gives up sets the status word and the CTA leaves.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "ptx.cuh"

namespace msk {

constexpr int RG_THREADS = 192;
constexpr int RG_STAGES = 4;
constexpr int RG_KSTEP = 64;                        // K elements per stage: one 128-byte swizzle row
constexpr int RG_A_BYTES = 128 * RG_KSTEP * 2;      // one 128-expert tile of a stage

struct RouterGemmCtrl {
  uint64_t full[RG_STAGES], empty[RG_STAGES], d_full;
  uint32_t tmem_base;
  int abort_word;
};

template <int N>
__global__ void __launch_bounds__(RG_THREADS, 1)
    router_hilo_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                       float* __restrict__ logits, int32_t* status, int T, int E, int H) {
  constexpr int B_BYTES = N * RG_KSTEP * 2;
  constexpr int STAGE_BYTES = 2 * RG_A_BYTES + B_BYTES;
  constexpr uint32_t TCOLS = N < 32 ? 32 : N;       // TMEM columns: a power of two, at least 32
  extern __shared__ __align__(1024) uint8_t rg_smem[];
  uint8_t* ring = rg_smem;
  float* part = reinterpret_cast<float*>(rg_smem);   // [N][128], once the ring is done with
  RouterGemmCtrl& ctl = *reinterpret_cast<RouterGemmCtrl*>(rg_smem + RG_STAGES * STAGE_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = gridDim.x, rank = blockIdx.x;   // a cluster is one row of the grid
  const int e0 = blockIdx.y * 128, t0 = blockIdx.z * N;
  const int all_steps = H / RG_KSTEP, first = rank * all_steps / split, n_steps = (rank + 1) * all_steps / split - first;

  if (tid == 0) {
    for (int i = 0; i < RG_STAGES; ++i) {
      mbar_init(&ctl.full[i], 1);
      mbar_init(&ctl.empty[i], 1);
    }
    mbar_init(&ctl.d_full, 1);
    ctl.abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl.tmem_base, TCOLS);
    tmem_relinquish();
  }
  pdl_wait();   // x may come from the kernel before
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl.tmem_base;
  volatile int* abortw = &ctl.abort_word;

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t keep = policy_evict_last();   // both operands are re-read by the other CTAs of the grid
      for (int ks = 0; ks < n_steps; ++ks) {
        const uint32_t slot = ks % RG_STAGES, par = (ks / RG_STAGES) & 1u;
        if (!mbar_wait(&ctl.empty[slot], par ^ 1u, abortw)) break;
        uint8_t* dst = ring + slot * STAGE_BYTES;
        mbar_arrive_expect_tx(&ctl.full[slot], STAGE_BYTES);
        const int k0 = (first + ks) * RG_KSTEP;
        tma_load_2d(dst, &tmap_w, k0, e0, &ctl.full[slot], keep);                    // hi rows e0 .. e0+127
        tma_load_2d(dst + RG_A_BYTES, &tmap_w, k0, E + e0, &ctl.full[slot], keep);   // lo rows
        tma_load_2d(dst + 2 * RG_A_BYTES, &tmap_x, k0, t0, &ctl.full[slot], keep);   // tokens t0 .. (rows past T read as zero)
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = idesc_f16(FMT_BF16, FMT_BF16, 128, N);
    bool ok = true;
    for (int ks = 0; ks < n_steps && ok; ++ks) {
      const uint32_t slot = ks % RG_STAGES, par = (ks / RG_STAGES) & 1u;
      if (!mbar_wait(&ctl.full[slot], par, abortw)) { ok = false; break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_hi = smem_u32(ring + slot * STAGE_BYTES), a_lo = a_hi + RG_A_BYTES, b = a_hi + 2 * RG_A_BYTES;
#pragma unroll
        for (int kk = 0; kk < RG_KSTEP / 16; ++kk) {
          const uint64_t bd = smem_desc_kmajor_sw128(b + kk * 32);
          mma_ss(tmem, smem_desc_kmajor_sw128(a_hi + kk * 32), bd, idesc, (ks > 0 || kk > 0) ? 1u : 0u);
          mma_ss(tmem, smem_desc_kmajor_sw128(a_lo + kk * 32), bd, idesc, 1u);
        }
        tc_commit(&ctl.empty[slot]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) tc_commit(&ctl.d_full);
    __syncwarp();
  } else {
    // this warp's TMEM lane quarter holds 32 experts; column c is token t0 + c. The ring is free: every copy has landed
    // and every MMA has read it.
    if (mbar_wait(&ctl.d_full, 0u, abortw)) {
      tc_fence_after();
      const int q = warp & 3;
      const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < N; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(taddr + c0, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(c0 + j) * 128 + q * 32 + lane] = __uint_as_float(r[j]);
      }
    }
  }
  __syncwarp();
  cluster_sync();   // reached by every thread, also after a wait that gave up
  {
    const int c_beg = rank * N / split, c_end = min((rank + 1) * N / split, T - t0);
    for (int i = c_beg * 32 + tid; i < c_end * 32; i += RG_THREADS) {
      const int c = i >> 5, e = e0 + (i & 31) * 4;
      const uint32_t addr = smem_u32(part + c * 128 + (i & 31) * 4);
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r = 0; r < split; ++r) {   // rank order
        const float4 v = ld_cluster_f4(addr, static_cast<uint32_t>(r));
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      float* dst = logits + static_cast<size_t>(t0 + c) * E + e;
      const float o[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (e + j < E) dst[j] = o[j];
    }
  }
  cluster_sync();   // no CTA leaves while another one reads its part
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (ctl.abort_word != 0) {
    const uint64_t w0 = globaltimer_ns();
    while (globaltimer_ns() - w0 < 2000000ull) __nanosleep(1000);   // let copies in flight land before smem is released
    if (tid == 0 && status != nullptr) atomicExch(status, 1);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TCOLS);
  }
}

}  // namespace msk
