// C ABI of the routed-expert step (declarations and contracts: include/msk_moe.h).
// Host side: argument validation, workspace carving, plan choice and launches; no torch
// headers, no allocation, no synchronisation except msk_moe_read_status.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/msk_moe.h"
#include "route_sort.cuh"
#include "gemm.cuh"
#include "few.cuh"
#include "pair.cuh"
#include "nvf4.cuh"
#include "router_gemm.cuh"

namespace msk {

// ------------------------------------------------------------ repack kernels
// Octet blocks (layout.cuh) in the order [expert][pair][ks][octet][gu]. Source rows of block (pair j,
// octet o, gu): w13 gu*I + j*128 + o*8 .. +7, w2 (2j + gu)*128 + o*8 .. +7.
struct RepackGeom {
  int rows_total;       // source rows per expert (2I or H)
  int K;                // source K
  int n_pairs;          // rows_total / 256
  int n_stages;         // K / 256
  int interleave_I;     // I for w13 (gate tile j with up tile j), 0 for w2 (row tiles 2j and 2j + 1)
};

// First source row (over all experts) of octet-gu number og = ((expert * n_pairs + pair) * 16 + o) * 2 + gu.
__device__ __forceinline__ long long source_row(const RepackGeom& g, long long og) {
  const int gu = static_cast<int>(og & 1), o = static_cast<int>((og >> 1) & 15);
  const long long ep = og >> 5;
  const int pair = static_cast<int>(ep % g.n_pairs);
  const long long e = ep / g.n_pairs;
  const int row = g.interleave_I > 0 ? gu * g.interleave_I + pair * 128 + o * OCT_ROWS
                                     : (2 * pair + gu) * 128 + o * OCT_ROWS;
  return e * g.rows_total + row;
}

// One warp per (octet, gu): 8 source rows of K/2 code bytes and K/16 scale bytes. Bound by memory: both sides
// move whole 32-byte sectors. Lane = (row r, 16-byte piece c of four): a warp reads 64 contiguous bytes of
// each of the eight rows and writes four full 128-byte lines, eight such steps (4 KB) in flight. The form
// this replaces gave each thread one 16-byte piece with the rows running along the lanes (16 useful bytes
// of every 32-byte sector on the source side): 128 experts of 4096 x 1536, both matrices, 535 us in and
// 722 us back out. Blocks of eight warps on the way in, of one on the way out, where a warp's eight rows are pages of their own: both
// matrices 426 us in, 423 out; with blocks of 32 / 64 / 128 / 256 / 512 / 1024 threads 428 / 430 / 430 / 426 / 431 / 457 in, 423 / 429 / 429 / 445 / 445 / 465 out
// (what has to be read and written takes 416 at the rate of a copy).
template <bool INVERSE> constexpr int REPACK_WARPS = INVERSE ? 1 : 8;
template <bool INVERSE>
__global__ void __launch_bounds__(REPACK_WARPS<INVERSE> * 32) repack_kernel(uint8_t* codes, uint8_t* sf, uint8_t* packed, RepackGeom g,
                                                     long long n_og) {
  const long long og = static_cast<long long>(blockIdx.x) * REPACK_WARPS<INVERSE> + (threadIdx.x >> 5);
  if (og >= n_og) return;
  const int lane = threadIdx.x & 31, r = lane >> 2, c4 = lane & 3;
  const long long srow = source_row(g, og) + r;
  uint8_t* block = packed + (og >> 5) * g.n_stages * STAGE_W_BYTES + (og & 31) * OCT_BYTES;   // K block 0; the next one STAGE_W_BYTES on
  {
    uint4* src = reinterpret_cast<uint4*>(codes + srow * (g.K / 2)) + c4;
    // chunk i*4 + c4 of the row: K block (i*4 + c4) / 8, chunk (i*4 + c4) % 8 inside it
    uint4* dst = reinterpret_cast<uint4*>(block + c4 * 128 + r * 16);
    const int n = g.n_stages * 2;                       // steps of four chunks (128 K)
    for (int i0 = 0; i0 < n; i0 += 8) {
      uint4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j;
        if (i < n) {
          const size_t at = static_cast<size_t>(i >> 1) * (STAGE_W_BYTES / 16) + (i & 1) * 32;
          v[j] = INVERSE ? __ldcs(dst + at) : __ldcs(src + i * 4);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j;
        if (i < n) {
          const size_t at = static_cast<size_t>(i >> 1) * (STAGE_W_BYTES / 16) + (i & 1) * 32;
          if (INVERSE) __stcs(src + i * 4, v[j]); else __stcs(dst + at, v[j]);
        }
      }
    }
  }
  uint4* src = reinterpret_cast<uint4*>(sf + srow * (g.K / 16));
  uint4* dst = reinterpret_cast<uint4*>(block + OCT_CODE_BYTES + r * 16);
  for (int ks = c4; ks < g.n_stages; ks += 4) {
    if (INVERSE) __stcs(src + ks, __ldcs(dst + ks * (STAGE_W_BYTES / 16)));
    else __stcs(dst + ks * (STAGE_W_BYTES / 16), __ldcs(src + ks));
  }
}

// Packed tiles -> BF16 e2m1*e4m3 matrices, through the decode routine of the GEMM kernel (the
// F16 products are exact and convert to BF16 without rounding).
__global__ void __launch_bounds__(128) dequant_packed_kernel(const uint8_t* packed, __nv_bfloat16* out, RepackGeom g,
                                                             long long n_og) {
  // a block per 16 octet-gus of one K block: thread = (octet-gu, row)
  const int ks = static_cast<int>(blockIdx.x % g.n_stages);
  const long long og = (blockIdx.x / g.n_stages) * 16 + (threadIdx.x >> 3);
  if (og >= n_og) return;
  const int r = threadIdx.x & 7;
  const uint8_t* block = packed + ((og >> 5) * g.n_stages + ks) * STAGE_W_BYTES + (og & 31) * OCT_BYTES;
  const uint4 sfw = *reinterpret_cast<const uint4*>(block + OCT_CODE_BYTES + r * 16);
  const uint32_t sfa[4] = {sfw.x, sfw.y, sfw.z, sfw.w};
  __nv_bfloat16* orow = out + (source_row(g, og) + r) * g.K + ks * KS;
  for (int chunk = 0; chunk < 8; ++chunk) {
    const uint4 qv = *reinterpret_cast<const uint4*>(block + chunk * 128 + r * 16);
    const uint32_t q[4] = {qv.x, qv.y, qv.z, qv.w};
    const uint32_t sw = sfa[chunk >> 1] >> ((chunk & 1) * 16);
    uint32_t o[16];
    decode_chunk(q, sw, o);
    for (int j = 0; j < 16; ++j) {
      const __half2 h = *reinterpret_cast<const __half2*>(&o[j]);
      orow[chunk * 32 + 2 * j] = __float2bfloat16_rn(__low2float(h));
      orow[chunk * 32 + 2 * j + 1] = __float2bfloat16_rn(__high2float(h));
    }
  }
}

// --------------------------------------------------------------- row copy
// F16 copy of the token rows, a block per token. With `inv` a row goes to each of its routes' places in sorted
// (expert-major) order, xs[inv[t, s]] = f16(x[t]), so that wide token tiles can be fetched as plain TMA boxes (the
// reference's prefill path gathers rows into per-expert tiles, muse_prefill_layer/cuda/prefill.cu:1446-1608, fused with
// its pre-expert norm); without it xs[t] = f16(x[t]), for the narrow token tiles that gather rows through the permutation.
// F16 is the operand type of the MMA (layout.cuh).
// With pre_w the pre-expert RMS norm of the layer callers is applied on the way:
// x' = bf16( x * rsqrt(mean(x^2) + eps) * (1 + pre_w) ), FP32 arithmetic on the row the block holds in
// registers (muse_decode_layer/py/04_triton_kernels.py:556-568: the reference's routing kernel does the
// same before it stores the expert input). The sum of squares is a fixed shuffle tree followed by a
// fixed-order sum of the eight warp partials.
// Bound by memory: a row is read and normalised once however many routes it has, and the row and its routes are loaded
// side by side. Going by sorted row instead (its entry first, then the row, each as often as it has routes) took 154 us for
// 8192 tokens of 8 routes at H = 4096 where this takes 102 (600 MB, 5.9 TB/s), and 18.3 for 777 tokens with the norm (14.3).
// look_first: a rank that holds a part of the experts has no route of many a token, whose row is then not read.
constexpr int COPY_THREADS = 256;
__global__ void __launch_bounds__(COPY_THREADS) copy_rows_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* inv, int top_k,
                                                                 int look_first, int H, __half* __restrict__ xs,
                                                                 const __nv_bfloat16* __restrict__ pre_w, float pre_eps) {
  __shared__ float wsum[COPY_THREADS / 32];
  constexpr int MAXV = 4;   // 8 values per uint4, 256 threads: H <= 8192
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  int dst_row = -1;         // lane s: the place of route s
  if (inv == nullptr) {
    if (lane == 0) dst_row = t;
  } else if (lane < top_k) {
    dst_row = __ldcg(inv + static_cast<size_t>(t) * top_k + lane);   // by an earlier launch of the chain: a coherent load
  }
  if (look_first && __ballot_sync(0xffffffffu, dst_row >= 0) == 0u) return;   // the same in every warp of the block
  const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(t) * H);
  uint4 v[MAXV];
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int i = j * COPY_THREADS + threadIdx.x;
    v[j] = make_uint4(0u, 0u, 0u, 0u);
    if (i < H / 8) v[j] = src[i];
  }
  unsigned routes = __ballot_sync(0xffffffffu, dst_row >= 0);
  if (routes == 0u) return;
  if (pre_w == nullptr) {
#pragma unroll
    for (int j = 0; j < MAXV; ++j)
      v[j] = make_uint4(bf16x2_to_f16x2(v[j].x), bf16x2_to_f16x2(v[j].y), bf16x2_to_f16x2(v[j].z), bf16x2_to_f16x2(v[j].w));
  } else {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float lo = __uint_as_float(w[c] << 16), hi = __uint_as_float(w[c] & 0xFFFF0000u);
        ss += lo * lo + hi * hi;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) wsum[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < COPY_THREADS / 32; ++w8) tot += wsum[w8];
    const float rs = rsqrtf(tot / static_cast<float>(H) + pre_eps);
    const uint4* gsrc = reinterpret_cast<const uint4*>(pre_w);
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = j * COPY_THREADS + threadIdx.x;
      if (i >= H / 8) continue;
      const uint4 gv = gsrc[i];
      const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
      const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
      uint32_t o4[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float lo = __uint_as_float(w[c] << 16) * rs * (1.0f + __uint_as_float(gw[c] << 16));
        const float hi = __uint_as_float(w[c] & 0xFFFF0000u) * rs * (1.0f + __uint_as_float(gw[c] & 0xFFFF0000u));
        const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);   // the expert input is BF16
        o4[c] = bf16x2_to_f16x2(*reinterpret_cast<const uint32_t*>(&b));
      }
      v[j] = make_uint4(o4[0], o4[1], o4[2], o4[3]);
    }
  }
  for (; routes != 0u; routes &= routes - 1u) {
    const int q = __shfl_sync(0xffffffffu, dst_row, __ffs(routes) - 1);
    uint4* dst = reinterpret_cast<uint4*>(xs + static_cast<size_t>(q) * H);
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = j * COPY_THREADS + threadIdx.x;
      if (i < H / 8) dst[i] = v[j];
    }
  }
}

// xh = f16(x), one 16-byte chunk per thread, in small blocks: the row copy in front of a gate/up
// kernel that routes itself (few tokens). It waits for whatever precedes the step, then lets its
// dependents start: the gate/up kernel's prologue (routing, sort) overlaps this copy and only its
// activation gather waits for it.
__global__ void __launch_bounds__(64) convert_rows_kernel(const __nv_bfloat16* __restrict__ x, __half* __restrict__ xh,
                                                          int n_chunks) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.x * 64 + threadIdx.x;
  if (i >= n_chunks) return;
  const uint4 v = reinterpret_cast<const uint4*>(x)[i];
  reinterpret_cast<uint4*>(xh)[i] =
      make_uint4(bf16x2_to_f16x2(v.x), bf16x2_to_f16x2(v.y), bf16x2_to_f16x2(v.z), bf16x2_to_f16x2(v.w));
}

// ---------------------------------------------------------------- combine
// out[t] = bf16( sum over slots in index order of w[t,s] * norm_s * y[inv[t,s]] ), norm_s =
// rsqrt(mean(y^2) + eps) when the post-expert norm is on (y already carries 1 + post_norm_w), else 1
// (muse_moe_w4a16/cuda/moe.cu:2604-2766; muse_decode_layer/py/04_triton_kernels.py:616-632).
// Slots without a local route (inv < 0) are squeezed out first, keeping their order, so an expert-parallel rank
// that owns one or two of a token's eight routes reads only those rows, and a token without any
// local route only gets zeros. Bound by memory for many tokens (8192 tokens, eight rows each: 0.6 GB).

// Eight consecutive y values of a row, FP32 or BF16 (the pair kernel's), in registers while in flight.
template <bool YB> struct YOct;
template <> struct YOct<false> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* y, size_t at) {
    a = __ldcs(reinterpret_cast<const float4*>(y + at));
    b = __ldcs(reinterpret_cast<const float4*>(y + at) + 1);
  }
  __device__ __forceinline__ void add_to(float (&acc)[8], float w) const {
    acc[0] += a.x * w; acc[1] += a.y * w; acc[2] += a.z * w; acc[3] += a.w * w;
    acc[4] += b.x * w; acc[5] += b.y * w; acc[6] += b.z * w; acc[7] += b.w * w;
  }
  __device__ __forceinline__ float squares() const {
    return ((a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w)) + ((b.x * b.x + b.y * b.y) + (b.z * b.z + b.w * b.w));
  }
};
template <> struct YOct<true> {
  uint4 a;
  __device__ __forceinline__ void load(const float* y, size_t at) {
    a = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(y) + at));
  }
  __device__ __forceinline__ void add_to(float (&acc)[8], float w) const {
    const uint32_t v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[2 * i] += __uint_as_float(v[i] << 16) * w;
      acc[2 * i + 1] += __uint_as_float(v[i] & 0xFFFF0000u) * w;
    }
  }
  __device__ __forceinline__ float squares() const {
    const uint32_t v[4] = {a.x, a.y, a.z, a.w};
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float lo = __uint_as_float(v[i] << 16), hi = __uint_as_float(v[i] & 0xFFFF0000u);
      s += lo * lo + hi * hi;
    }
    return s;
  }
};

// Without the post-expert norm the columns do not depend on one another: a warp per (token, C * 256 columns), G rows of
// them in flight, no block-wide step. G = 8, C = 1 where most of a token's routes are local (8192 tokens of eight rows:
// 106 us with a block per token, 98 with this); with two or fewer expected, G = 2, C = 4, or the warps would spend
// their time on the table (8192 tokens of H = 7168 with one local route each: 68 us with a block per token, 78 with G = 8,
// C = 1, 47 with G = 2, C = 4).
constexpr int COMBINE_COLS_WARPS = 4;
template <bool YB, int G, int C>
__global__ void __launch_bounds__(COMBINE_COLS_WARPS * 32)
    combine_cols_kernel(const float* y, const int32_t* inv, const float* tw, __nv_bfloat16* __restrict__ out, int T, int H,
                        int k) {   // (what earlier launches of the chain write is not __restrict__: coherent loads)
  const int lane = threadIdx.x & 31, chunks = (H + C * 256 - 1) / (C * 256);
  const long long item = static_cast<long long>(blockIdx.x) * COMBINE_COLS_WARPS + (threadIdx.x >> 5);
  const int t = static_cast<int>(item / chunks), col = static_cast<int>(item % chunks) * (C * 256) + lane * 8;
  pdl_wait();  // y and inv come from the kernels before this one
  if (t >= T) return;
  const int q = lane < k ? inv[static_cast<size_t>(t) * k + lane] : -1;
  const float w = lane < k ? tw[static_cast<size_t>(t) * k + lane] : 0.f;
  unsigned have = __ballot_sync(0xffffffffu, q >= 0);
  float acc[C][8] = {};
  while (have != 0u) {
    YOct<YB> v[G][C];
    float wv[G];
    const int n = min(__popc(have), G);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (g < n) {
        const int s = __ffs(have) - 1;
        have &= have - 1u;
        wv[g] = __shfl_sync(0xffffffffu, w, s);
        const size_t at = static_cast<size_t>(__shfl_sync(0xffffffffu, q, s)) * H + col;
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (col + c * 256 < H) v[g][c].load(y, at + c * 256);
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {   // slot order
      if (g < n) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (col + c * 256 < H) v[g][c].add_to(acc[c], wv[g]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    if (col + c * 256 >= H) break;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(acc[c][2 * i], acc[c][2 * i + 1]);
      o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * H + col + c * 256) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// With the post-expert norm: a block of TH threads per token, G rows in registers at a time (NO octets of columns a thread, H <= 8 * TH * NO). The sum of
// squares of a row is a fixed tree over every 1024 columns followed by the sum of those in column order, whatever
// the block's size, so the result depends neither on scheduling nor on how many tokens a step has; the sums run in slot order. Bound by latency (table, rows, reduction, each behind the other), so what counts is rows in flight on
// an SM. Many tokens: blocks of 128 threads (256 beyond 4096 columns), five or four of them on an SM, where blocks of 512 left two tokens to
// one: 3012 tokens with 1.6 local routes each 41 -> 18 us, 777 with eight 22 -> 16, 7000 149 -> 98. Up to 2048 columns two octets a
// thread, which four leave half the block's threads without: 2000 tokens of four at 2048 columns 17 -> 13, 4000 of eight at 1024 39 -> 27. Few
// tokens: 512 threads and as many rows at once as fit (64 tokens of eight 8 -> 6). Every warp reads the table for itself; where given weights lie in
// pinned memory that is no slower than one warp's read that the others wait for (whole steps from pinned rows, ids and weights, H2048 I1024, 16 / 24 / 48 tokens,
// that form / this: 53.6 / 51.7, 59.9 / 58.6, 67.6 / 66.0).
constexpr int COMBINE_FEW_TOKENS = 256;
constexpr int COMBINE_MAX_H = 8192;
template <bool YB, int TH, int NO, int G, int MINB>
__global__ void __launch_bounds__(TH, MINB)
    combine_norm_kernel(const float* y, const int32_t* inv, const float* tw, __nv_bfloat16* __restrict__ out, int H, int k,
                        float eps) {   // (y, inv and tw: as above)
  // A run of 1024 columns is four quarters of 32 octets. Its squares are summed over the quarters, over eight neighbours and over the
  // four groups of neighbours, each as a tree, then run after run: NO = 4 has the quarters of a run in a thread and the run in a warp,
  // NO = 2 half of either, NO = 1 a quarter, and SUM_BITS are the lane bits of the same additions in the same order.
  constexpr int CL = 4 / NO, JW = 32 / CL, NW = TH / 32, LG = G == 8 ? 3 : G == 4 ? 2 : 1;
  constexpr int SUM_BITS[5] = {NO == 4 ? 4 : 16, NO == 4 ? 2 : NO == 2 ? 4 : 8, NO == 4 ? 1 : NO == 2 ? 2 : 4, NO == 4 ? 8 : NO == 2 ? 1 : 2,
                               NO == 4 ? 16 : NO == 2 ? 8 : 1};
  static_assert(G == 1 << LG && (NO == 1 || NO == 2 || NO == 4) && NW % 4 == 0, "two, four or eight rows together");
  __shared__ __align__(16) float part[2][G][NW];   // in turn: a group's parts are read while the next one's are written
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = ((warp / CL) * 128 + (lane / JW) * 32 + (warp % CL) * JW + lane % JW) * 8;   // column of the first octet
  constexpr int STEP = CL * 256;                                                                 // to the next one
  pdl_wait();  // y and inv come from the kernels before this one
  const int q = lane < k ? inv[static_cast<size_t>(t) * k + lane] : -1;
  const float w = lane < k ? tw[static_cast<size_t>(t) * k + lane] : 0.f;
  unsigned have = __ballot_sync(0xffffffffu, q >= 0);   // the same in every warp
  float acc[NO][8] = {};
  for (int turn = 0; have != 0u; turn ^= 1) {
    YOct<YB> v[G][NO];
    float wgt[G], ss[G];
    const int n = min(__popc(have), G);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (g < n) {
        const int s = __ffs(have) - 1;
        have &= have - 1u;
        wgt[g] = __shfl_sync(0xffffffffu, w, s);
        const size_t at = static_cast<size_t>(__shfl_sync(0xffffffffu, q, s)) * H;
#pragma unroll
        for (int c = 0; c < NO; ++c)
          if (first + c * STEP < H) v[g][c].load(y, at + first + c * STEP);
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float sq[NO] = {};
      if (g < n) {
#pragma unroll
        for (int c = 0; c < NO; ++c)
          if (first + c * STEP < H) sq[c] = v[g][c].squares();
      }
      ss[g] = NO == 1 ? sq[0] : NO == 2 ? sq[0] + sq[NO / 2] : (sq[0] + sq[NO / 2]) + (sq[NO / 4] + sq[NO - 1]);
    }
    // G sums over the warp at once: in each of the first steps a lane passes on half of its sums and keeps the other
    // half (the same additions as in G separate trees, but in G + 4 - LG shuffles instead of 5 * G)
    int mine = 0;   // whose sum this lane ends with
    bool first_of = true;
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const int o = SUM_BITS[b], h = G >> (b + 1);
      const bool up = (lane & o) != 0;
      if (b < LG) {
        mine = mine * 2 + (up ? 1 : 0);
#pragma unroll
        for (int g = 0; g < h; ++g) {
          const float keep = up ? ss[g + h] : ss[g], send = up ? ss[g] : ss[g + h];
          ss[g] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      } else {
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], o);
        first_of = first_of && !up;
      }
    }
    if (first_of) part[turn][mine][warp] = ss[0];
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; ++g) {   // slot order
      if (g < n) {
        float tot = 0.f;
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {  // a run is one part, two or four
          const float4 f = reinterpret_cast<const float4*>(part[turn][g])[i];
          if (NO == 1) {
            tot += (f.x + f.y) + (f.z + f.w);
          } else if (NO == 2) {
            tot += f.x + f.y; tot += f.z + f.w;
          } else {
            tot += f.x; tot += f.y; tot += f.z; tot += f.w;
          }
        }
        wgt[g] *= rsqrtf(tot / static_cast<float>(H) + eps);
#pragma unroll
        for (int c = 0; c < NO; ++c)
          if (first + c * STEP < H) v[g][c].add_to(acc[c], wgt[g]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NO; ++c) {
    if (first + c * STEP >= H) break;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(acc[c][2 * i], acc[c][2 * i + 1]);
      o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * H + first + c * STEP) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ------------------------------------------------------------- EP combine
// Expert-parallel combine at the token's home rank: out[t] = bf16( sum over ranks d, in rank
// order, of the partial row rank d returned for token t ), FP32 accumulation. Rank d contributes
// only when one of the token's top-k ids lies in d's expert range, so rows of ranks without a
// route are never read. back is [n, T, H] in rank order; the home rank's own partial may live
// elsewhere (self_rows).
__global__ void __launch_bounds__(256) ep_combine_kernel(const __nv_bfloat16* __restrict__ back,
                                                         const __nv_bfloat16* __restrict__ self_rows, int self_rank,
                                                         const int32_t* __restrict__ ids, int top_k, int per_rank,
                                                         __nv_bfloat16* __restrict__ out, int n, int T, int H) {
  __shared__ unsigned long long present;
  const int t = blockIdx.x;
  if (threadIdx.x == 0) present = 0ull;
  __syncthreads();
  if (threadIdx.x < top_k) {
    const int id = ids[static_cast<size_t>(t) * top_k + threadIdx.x];
    if (id >= 0 && id / per_rank < n) atomicOr(&present, 1ull << (id / per_rank));
  }
  __syncthreads();
  const unsigned long long have = present;
  const int n8 = H / 8;
  for (int i = threadIdx.x; i < n8; i += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int d = 0; d < n; ++d) {
      if (!((have >> d) & 1ull)) continue;
      const __nv_bfloat16* rows = (d == self_rank && self_rows != nullptr)
                                      ? self_rows
                                      : back + static_cast<size_t>(d) * T * static_cast<size_t>(H);
      const uint4 v = *reinterpret_cast<const uint4*>(rows + static_cast<size_t>(t) * H + static_cast<size_t>(i) * 8);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] += __uint_as_float(w[j] << 16);
        acc[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
      }
    }
    uint4 o;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
      ow[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * H + static_cast<size_t>(i) * 8) = o;
  }
}

// Stream memory operations (executed by the stream's front end, no SM): the cross-rank flags of
// the expert-parallel step. Looked up through the runtime, like the tensor-map encoder.
typedef CUresult (*StreamValue32Fn)(CUstream, CUdeviceptr, cuuint32_t, unsigned int);

static int stream_value32(const char* name, void* addr, uint32_t value, unsigned int flags, void* stream) {
  void* ptr = nullptr;
  cudaDriverEntryPointQueryResult qres;
  const cudaError_t e = cudaGetDriverEntryPoint(name, &ptr, cudaEnableDefault, &qres);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (qres != cudaDriverEntryPointSuccess || ptr == nullptr) return static_cast<int>(cudaErrorNotSupported);
  const CUresult r = reinterpret_cast<StreamValue32Fn>(ptr)(static_cast<CUstream>(stream),
                                                            reinterpret_cast<CUdeviceptr>(addr), value, flags);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(cudaErrorInvalidValue);
}

// --------------------------------------------------------------- bw probe
// Every CTA streams its contiguous share of the buffer through a ring of bulk async
// copies, one elected thread issuing, one warp consuming (twin of the reference's
// muse_moe_w4a16/cuda/moe_bw.cu tma_kernel).
__global__ void __launch_bounds__(64) bw_probe_kernel(const uint8_t* src, unsigned long long bytes, int stages,
                                                      int stage_bytes, uint32_t* sink, int skip_release) {
  extern __shared__ __align__(1024) uint8_t psm[];
  __shared__ uint64_t full[8], empty[8];
  __shared__ int abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    abort_word = 0;
    fence_mbar_init();
  }
  __syncthreads();
  const unsigned long long n_chunks = bytes / stage_bytes;
  const unsigned long long per = (n_chunks + gridDim.x - 1) / gridDim.x;
  const unsigned long long c0 = per * blockIdx.x, c1 = min(n_chunks, c0 + per);
  if (warp == 0) {
    if (lane == 0) {
      const uint64_t pol = policy_evict_first();
      uint32_t it = 0;
      for (unsigned long long c = c0; c < c1; ++c, ++it) {
        const uint32_t slot = it % stages, par = (it / stages) & 1u;
        if (!mbar_wait(&empty[slot], par ^ 1u, &abort_word)) break;
        mbar_arrive_expect_tx(&full[slot], stage_bytes);
        bulk_g2s(psm + static_cast<size_t>(slot) * stage_bytes, src + c * stage_bytes, stage_bytes, &full[slot], pol);
      }
    }
  } else {
    uint32_t it = 0, sum = 0;
    for (unsigned long long c = c0; c < c1; ++c, ++it) {
      const uint32_t slot = it % stages, par = (it / stages) & 1u;
      if (!mbar_wait(&full[slot], par, &abort_word)) break;
      sum += *reinterpret_cast<const uint32_t*>(psm + static_cast<size_t>(slot) * stage_bytes + lane * 16);
      __syncwarp();
      // skip_release (test hook): chunk number skip_release of every CTA is never handed back, so the
      // producer's bounded wait for that slot runs out and the kernel leaves through its time-out path
      if (lane == 0 && !(skip_release > 0 && it + 1 == static_cast<uint32_t>(skip_release))) mbar_arrive(&empty[slot]);
    }
    if (sum == 0x9E3779B9u) atomicAdd(sink, sum);  // keeps the reads alive
  }
  __syncthreads();
  if (abort_word != 0) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    if (threadIdx.x == 0) atomicExch(reinterpret_cast<int*>(sink) + 1, MSK_DEV_ERR_TIMEOUT);
  }
}

// ------------------------------------------------------------ host helpers
static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
static inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

static int check_cfg(const MskMoeCfg* c) {
  if (c == nullptr) return MSK_ERR_NULL;
  if (c->hidden <= 0 || c->inter <= 0 || c->hidden % 256 != 0 || c->inter % 256 != 0) return MSK_ERR_SHAPE;
  if (c->hidden > COMBINE_MAX_H) return MSK_ERR_SHAPE;  // combine keeps a row in registers
  if (c->max_tokens < 0) return MSK_ERR_SHAPE;
  if (c->top_k < 1 || c->top_k > MAX_TOP_K) return MSK_ERR_SHAPE;
  if (c->local_count < 1 || c->local_count > MAX_LOCAL_EXPERTS) return MSK_ERR_SHAPE;
  if (c->n_experts < 1 || c->n_experts > MAX_EXPERTS) return MSK_ERR_SHAPE;
  if (c->local_start < 0 || c->local_start + c->local_count > c->n_experts) return MSK_ERR_RANGE;
  if (c->token_tile != 0 && c->token_tile != 16 && c->token_tile != 32 && c->token_tile != 64 && c->token_tile != 128)
    return MSK_ERR_SHAPE;
  if (c->decode_path < 0 || c->decode_path > 4) return MSK_ERR_SHAPE;
  return MSK_OK;
}

static int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// Persistent grid when the caller names none: the SM count of a B200. A constant, so that the
// shares of the weight stream (and with them the order in which a cut unit's pieces are summed)
// depend on the configuration, not on the device the library happens to run on.
constexpr int DEFAULT_CTAS = 148;
// MSK_NO_HANDOVER=1 switches the per-tile hand-over between the two GEMM launches off (measurements).
static bool handover_env_off() {
  static const bool v = [] {
    const char* e = std::getenv("MSK_NO_HANDOVER");
    return e != nullptr && e[0] == '1';
  }();
  return v;
}
constexpr int MAX_CTAS = 512;
constexpr int FLAT_MAX_ROWS = SMALL_SORT_MAX_ENTRIES;  // up to here the weight stream may be cut into equal shares
constexpr int ONE_LAUNCH_MAX_TOKENS = 8;               // up to here the step is one launch by default
constexpr int ONE_LAUNCH_NORM_TOKENS = 4;              // from here on it is not with the post-expert norm (step_form)
constexpr int BOTH_GEMMS_MIN_TOKENS = 9;               // from here on (narrow tiles) both GEMMs share one launch by default

struct Plan {
  int N;         // token tile
  int path;      // 0 one launch, 1 chain of launches, 2 row copy + routing gate/up kernel + combining down kernel
  int flat;      // equal shares of the flat (base unit, K stage) list
  int grid;
  bool both;     // both GEMMs in one launch: path 4, and the 64-token tile of path 1
};

// A form that the configuration asks for is always the asked one.
static bool form_asked(const MskMoeCfg* c) { return c->token_tile != 0 || c->decode_path != 0 || c->flat_shares != 0 || c->stop_after != 0; }

static Plan make_plan(const MskMoeCfg* c, int T) {
  Plan p;
  p.grid = c->num_ctas > 0 ? std::min(c->num_ctas, MAX_CTAS) : DEFAULT_CTAS;
  p.path = 1;
  p.flat = 0;
  if (c->token_tile > 0) {
    p.N = c->token_tile;
  } else {
    const double rpe = static_cast<double>(T) * c->top_k / c->n_experts;  // mean tokens per expert
    // 16 / 64-token tile (us, rows of steps): H2048 I1024 E64 near-even rpe 4 58.9 / 58.8, 6 61.1 / 59.8, 8 63.2 / 61.2, 12 68.9 / 63.0, a few experts
    // taking most tokens 45.3 / 47.0, 51.9 / 51.4, 55.1 / 53.7, 67.0 / 59.6; H4096 I1024 E128 rpe 4 193 / 199 (105 / 90), 6 202 / 205, 8 210 / 208 (158 / 117), 12
    // 238 / 215 (210 / 144); H4096 I1280 E128 rpe 6 247 / 250, 8 254 / 252. Few narrow experts, top-2 of 8, rpe 7.25 / 8 / 10 / 12: H4096 I1024 41.2 / 39.2, 41.3 /
    // 39.2, 41.4 / 39.3, 43.2 / 39.3 (43.3 / 41.4, 43.3 / 42.2, 43.3 / 43.4, 43.3 / 44.9); H1024 I512 28.9 / 27.1 .. 29.0 / 28.8 (29.0 / 28.8 .. 29.1 / 31.0); a rank, 16 of 64 of H2048 I1024, rpe 9 / 12 34.1 / 32.4, 34.5 / 33.9 (36.5 / 38.2, 36.9 / 39.7). 64-token tile / pair kernel: T = 384 (rpe 24) 297 / 341, T = 512 319 / 362, T = 640
    // (rpe 40) 343 / 389; with a few experts taking most tokens 252 / 245, 311 / 287, 359 / 330. Beyond: rpe 48 near-even
    // 406 / 464, 32 of 256 experts at H4096 I4096 255 / 289, a few experts taking most 456 / 420, the same at H2048 I1024 E64
    // 107 / 88; rpe 56 445 / 477, 279 / 295, 508 / 452, 114 / 95; rpe 64 near-even 566 / 505. At rpe 40 the 64-token tile loses 13 %
    // at worst and the pair kernel 18, at 48 it is 21 and 20. The 16-token tile is the
    // fastest per K stage and wins while most experts fit one tile; the 64-token tile wins while most fit one of those. The
    // host does not know the counts, and the less even they are the lower that line lies. The 32-token tile never wins at
    // these shapes (it stays selectable with cfg.token_tile). 128 stands for the pair kernel (pair.cuh). Where a path, flat shares or
    // a part of the step is asked for, the narrow tile, which those are made for, stays up to 12.
    p.N = rpe <= (form_asked(c) ? 12 : 7) ? 16 : rpe <= 40 ? 64 : 128;
  }
  const long long rows = static_cast<long long>(T) * c->top_k;
  // Flat shares are an option, off by default: measured on B200 a cut unit's pieces cost about 6 us of
  // round trips through L2 at the end of each GEMM (store, fence, ticket, reload from a cold instruction
  // cache), as much as the idle CTAs of the last round of whole units cost at these sizes.
  p.flat = (c->flat_shares != 0 && rows <= FLAT_MAX_ROWS && p.N <= 64) ? 1 : 0;
  {
    // the kernels do the share arithmetic in 32 bits: items * shares has to fit
    const long long pairs = std::max(c->inter / 128, c->hidden / 256), nst = std::max(c->hidden, c->inter) / KS;
    if ((rows + 1) * pairs * nst * p.grid >= FLAT_MAX_PRODUCT) p.flat = 0;
  }
  // few tokens: the kernels route, sort and combine themselves
  const bool few = rows <= SMALL_SORT_MAX_ENTRIES && T <= FOLD_MAX_TOKENS && p.N <= 32 && c->stop_after == 0;
  if (few) {
    // measured (H4096 I1536 E128 top-8, cold L2): the one-launch form of the tcgen05 kernel 89 / 136 us at 4 / 8 tokens
    // against 94 / 135 for the chain; at 16 and 32 tokens 195 / 268 against 197 / 249. (Fewer tokens mostly take the
    // few-token kernel, few_takes(); by the tcgen05 kernel 1 / 2 tokens take 47 / 64 against 57 / 72.)
    switch (c->decode_path) {
      case 1: p.path = 1; break;
      case 4: p.path = 1; break;   // becomes 4 below
      case 2: p.path = 2; break;
      case 3: p.path = 0; break;
      default: p.path = T <= ONE_LAUNCH_MAX_TOKENS ? 0 : 1; break;
    }
    if (p.path == 0 && p.grid > sm_count()) p.path = 2;  // the one-launch kernel needs every CTA resident
    if (p.path == 0) p.flat = 0;  // its phases hand over per token tile, which counts whole units
  }
  // Beyond a few tokens, narrow token tiles: the sort launches, then both GEMMs in one cooperative launch
  // (path 4: the weight stream, the dequant ring and the MMA pipeline run on from the gate/up units into the
  // down units, tile by tile, and the kernel makes its own F16 copy of the token rows), then the combine.
  // Measured at H4096 I1536 E128 (stamped runs): 16 / 32 / 64 / 128 tokens 176 / 227 / 253 / 268 us against
  // 186 / 240 / 258 / 270 for two GEMM launches with the per-tile hand-over between them. Same bits.
  const bool resident = p.flat == 0 && c->stop_after == 0 && p.grid <= sm_count();
  if (p.path == 1 && p.N <= 32 && resident &&
      (c->decode_path == 4 || (c->decode_path == 0 && T >= BOTH_GEMMS_MIN_TOKENS)))
    p.path = 4;
  // The 64-token tile keeps the row copy in front of the GEMMs and shares one launch between them as well, unless the
  // chain is asked for: 256 tokens 279 us against 287.
  p.both = p.path == 4 || (p.path == 1 && p.N == 64 && resident && c->decode_path != 1);
  return p;
}

// The kernel on the FP4 tensor cores (nvf4.cuh). It streams weights at the pace of memory and pays some us more in front of the first MMA and
// between the GEMMs, so it gains with the bytes that a step streams: those of the experts that get a token, which the host does not know. Whole
// steps in us, the other kernel / this one, in turn on one box; "uneven": a few experts taking most tokens (Zipf routes).
// All of 128 experts (H4096 I1536 top-8, 10.6 MB each), near-even (uneven): 4 tokens 65 / 69 (54 / 55), 5: 76 / 75 (56 / 57), 6: 87 / 82 (60 / 60), 8:
// 105 / 95 (64 / 61), 9: 115 / 102 (60 / 62), 12: 147 / 125 (64 / 66), 16: 174 / 149 (71 / 72), 20: 200 / 170 (77 / 76), 24: 216 / 180 (84 / 81), 64: 262 / 224
// (134 / 116), 192 (12 rows an expert) 339 / 305 (278 / 246); 224: 320 / 351 (191 / 285), 256: 325 / 382 (213 / 309): beyond 12 rows an expert the other
// one is the 64-token tile, which streams the weights of an expert with many rows once for 64 of them, this one for 16. Uneven steps of 9
// to 16 tokens lose 1 to 3 %, near-even ones, which stream twice the bytes, gain 13 to 17: the line stays at 6.
// With the other kernel's issue by one thread and this one's room for four rows (64-token tile / this one, rows of steps) 64: 288 / 240 (123 / 135), 128: 296 / 272
// (161 / 200), 160: 299 / 292 (182 / 235), 192: 304 / 316 (198 / 263), 256: 316 / 384 (230 / 323); a rank, two experts taking most, 100: 158 / 154, 200: 205 / 213, 384:
// 242 / 281; H7168 I2048, even, 200: 171 / 159, 300: 176 / 175, 384: 178 / 192. By these this one gains 9 % at eight rows an expert of near-even routes and 2 % at
// ten, loses 4 % at twelve, and loses 24, 29 and 33 % there where a few experts take most; a rank's skewed steps lose 4 % at six rows and 16 at twelve, its even ones 8 at twelve. The line at
// twelve is the one of before those two changes and is later than they would have it: six to eight rows, or the counts, which the host does not know.
// A rank (32 of 256, one row a token): H4096 I4096, two experts taking most, 4: 45 / 46, 6: 50 / 49, 8: 59 / 58, 10: 59 / 62, 16: 66 / 67, 18: 69 / 69, 20: 70 / 69,
// 24: 79 / 76, 28: 86 / 80, 64: 138 / 115, 384: 308 / 263 (512: 236 / 310); H7168 I2048, even, 4: 50 / 51, 6: 50 / 53, 8: 56 / 58, 16: 74 / 74, 18: 77 / 77, 20: 81 /
// 79, 24: 83 / 80, 28: 91 / 88, 64: 128 / 114, 384: 201 / 171.
// Layers of less: experts of 3.5 MB (a small model, H2048 I1024 E64 top-4, down units of four K stages) 8: 45 / 44 (38 / 35), 24: 54 / 55 (37 / 39), 64: 58
// / 62 (44 / 47); H2048 I1536 E64 (340 MB in all) 8: 43 / 45 (39 / 38), 24: 64 / 62 (44 / 45), 160: 83 / 93 (78 / 89); H2048 I2048 E64 (453 MB) 24: 76 / 72 (50 / 51),
// 64: 94 / 87 (63 / 67), 160: 103 / 107 (100 / 103); 32 experts of H4096 I1536 (340 MB) 6: 53 / 56 (46 / 44), 32: 71 / 71 (59 / 60). H4096 I1280 E128, 24: 161 / 146
// (83 / 77), would gain. (Fewer than 32 experts: 8 of H4096 I14336 16 tokens 155 / 144.)
// With an expert norm the others take an exchange or a launch more up to eight tokens, and this one, whose combine is a launch anyway, does not.
// Post-expert norm, the 128 experts 3: 70 / 62 (56 / 56), 4: 74 / 70 (75 / 57), 8: 119 / 98 (100 / 63); the small model 4: 35 / 37 (38 / 33), 8: 44 / 41; a rank
// 3: 41 / 45, 4: 50 / 47, 8: 66 / 58, H7168 3: 43 / 50, 4: 54 / 52, 8: 61 / 59. Pre-expert norm, the 128 experts 4: 77 / 69 (51 / 56), 5: 82 / 75 (61 / 58),
// 8: 117 / 95 (68 / 61); H2048 I1536 E64 4: 35 / 40 (27 / 35), 6: 43 / 43 (32 / 37); 32 experts of H4096 I1536 6: 57 / 57 (42 / 45); a rank 4: 42 / 48, 8: 59 / 59, H7168
// 5: 50 / 54, 8: 58 / 59; from nine tokens on the other one has a row copy in front as well: H2048 I1536 E64 9: 51 / 49 (37 / 40), 32: 79 / 68 (49 / 47), a
// rank 12: 66 / 63, H7168 12: 75 / 65.
// Where the few-token kernel takes four tokens and more of a rank (both norms), it keeps them: 4: 45 / 48, 6: 52 / 54.
constexpr int NV_MIN_TOKENS = 6;
constexpr int NV_MIN_NORM_TOKENS = 4;        // with an expert norm
constexpr int NV_MIN_RANK_TOKENS = 20;       // of a rank that holds a part of the experts (with the post-expert norm: beyond the one-launch form's)
constexpr int NV_MAX_MEAN_ROWS = 12;
constexpr int NV_MIN_INTER = 1536;
// Bytes of near-even routes, where all of NV_MANY_EXPERTS experts or more are here: beyond the one-launch form's tokens, up to them, with the
// pre-expert norm alone
constexpr double NV_MIN_BYTES = 460e6, NV_MIN_BYTES_ONE_LAUNCH = 400e6, NV_MIN_BYTES_PRE = 300e6;
constexpr int NV_MANY_EXPERTS = 32;

static int nv_max_tokens(const MskMoeCfg* c, int T) {   // of the steps of up to T tokens that may take it
  if (c->inter < NV_MIN_INTER || c->inter > NV_MAX_INTER || c->hidden > NV_MAX_BLOCKS * 16) return 0;
  return static_cast<int>(std::min(static_cast<long long>(T), static_cast<long long>(NV_MAX_MEAN_ROWS) * c->n_experts / c->top_k));
}

// Weights that near-even routes of T tokens touch, where all experts are here.
static double nv_even_bytes(const MskMoeCfg* c, int T) {
  const double touched = c->n_experts * (1.0 - std::pow(1.0 - static_cast<double>(c->top_k) / c->n_experts, T));
  return touched * 3.0 * c->hidden * c->inter * 0.5625;
}

// Whether a step runs in it; norms: MSK_NVF4_* bits.
static bool nv_takes(const MskMoeCfg* c, int T, const Plan& p, int norms) {
  if (form_asked(c) || p.grid > sm_count() || T > nv_max_tokens(c, T)) return false;
  const bool all = c->local_count == c->n_experts, pre = (norms & MSK_NVF4_PRE_NORM) != 0, post = (norms & MSK_NVF4_POST_NORM) != 0;
  const bool many = c->n_experts >= NV_MANY_EXPERTS;
  if (T <= ONE_LAUNCH_MAX_TOKENS) {
    if (post) return T >= NV_MIN_NORM_TOKENS;
    return all && T >= (pre ? NV_MIN_NORM_TOKENS : NV_MIN_TOKENS) && (!many || nv_even_bytes(c, T) >= (pre ? NV_MIN_BYTES_PRE : NV_MIN_BYTES_ONE_LAUNCH));
  }
  return all ? pre || !many || nv_even_bytes(c, T) >= NV_MIN_BYTES : T >= NV_MIN_RANK_TOKENS;
}

// Workspace carving. Everything is sized for max_tokens with the worst plan.
struct Carve {
  size_t status, trace, cnt, off, perm, inv, tickets, few_ctl, sort_blk, tile_ctr, inter, y, partial, xs, nv_tiles, nv_img[2], nv_end, total;
};
constexpr size_t TRACE_CTAS = 256;
constexpr size_t TRACE_WORDS = TRACE_CTAS * 16 + 3 * 256;

static size_t max_tiles(const MskMoeCfg* c, int T) {
  // ceil(cnt/16) summed over experts <= R/16 + (experts that can hold a row)
  const size_t R = static_cast<size_t>(T) * c->top_k;
  return R / 16 + std::min(static_cast<size_t>(c->local_count), R);
}

// Pieces of cut units (flat shares): two slots per CTA of the largest grid, each the two accumulator
// tiles of the widest token tile that is ever cut (64).
static size_t partial_floats(const MskMoeCfg* c) {
  const size_t grid = c->num_ctas > 0 ? static_cast<size_t>(std::min(c->num_ctas, MAX_CTAS)) : DEFAULT_CTAS;
  return 2 * grid * 2 * 128 * 64;
}

static size_t ticket_ints(const MskMoeCfg* c, int T) {
  return max_tiles(c, T) * static_cast<size_t>(std::max(c->inter / 128, c->hidden / 256));
}

static Carve carve(const MskMoeCfg* c, int T) {
  Carve k;
  const size_t R = static_cast<size_t>(T) * c->top_k;
  size_t o = 0;
  k.status = o; o += 256;
  k.trace = o; o += 2 * TRACE_WORDS * 8;  // two GEMM launches x (CTAs x 16 stamps + 3 x 256 events of CTA 0)
  k.cnt = o; o += round_up(static_cast<size_t>(c->local_count) * 4, 256);
  k.off = o; o += round_up(static_cast<size_t>(c->local_count + 1) * 4, 256);
  k.perm = o; o += round_up(R * 4, 256);
  k.inv = o; o += round_up(R * 4, 256);
  k.tickets = o; o += 2 * round_up(ticket_ints(c, T) * 4, 256);  // one region per GEMM
  k.few_ctl = o; o += 8192;    // few-token paths of the GEMM kernel: tickets [32 tokens][up to 32 pairs] at +0, grid counters [2] at
                               // +4096, per-tile counters [2][up to 384 tiles] at +4352
  k.sort_blk = o; o += static_cast<size_t>(SORT_MULTI_BLOCKS) * MAX_LOCAL_EXPERTS * 4;  // per-CTA counts of the multi-CTA sort
  // tile hand-over between the gate/up and the down launch: per token tile the finished gate/up units and
  // the down units that have seen them all (two counters per tile, zero between steps)
  k.tile_ctr = o; o += round_up(2 * max_tiles(c, T) * 4, 256);
  // the FP4 kernel, for the most tokens it takes: counters of its tiles (no more than it has groups of eight rows)
  const size_t nv_rows = static_cast<size_t>(nv_max_tokens(c, T)) * c->top_k;
  const size_t nv_groups = nv_groups_bound(nv_rows, static_cast<size_t>(c->local_count));
  k.nv_tiles = o; o += round_up(nv_groups * NV_TILE_WORDS * 4, 256);
  // everything above is control state: msk_moe_workspace_init zeroes [0, inter)
  k.inter = o; o += round_up(R * c->inter * 2, 256);
  k.y = o; o += round_up(R * c->hidden * 4, 256);
  k.partial = o; o += 2 * round_up(partial_floats(c) * 4, 256);  // one region per GEMM
  k.xs = o; o += round_up(R * c->hidden * 2, 256);  // F16 copy of the token rows ([T, H], or sorted [R, H] for wide token tiles)
  // The FP4 kernel's split rows, 3.8 times their F16 bytes: where the pieces and the F16 rows lie, which its steps have no use for, and beyond
  // them where there is less room (with a capacity of 8192 tokens there never is). Room that only they need is left out where a form is
  // asked for, whose steps never run there; forward() looks whether it is there.
  const int nv_k[2] = {c->hidden, c->inter};
  k.nv_end = k.partial;
  for (int i = 0; i < 2; ++i) {
    k.nv_img[i] = k.nv_end;
    k.nv_end += round_up(nv_groups * (nv_k[i] / KS) * NV_GROUP_BYTES, 256);
  }
  k.total = form_asked(c) ? o : std::max(o, k.nv_end);
  return k;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (no link against libcuda).
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                      const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                      CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int encode_map(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base, const cuuint64_t* dims,
                      const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  static TensorMapEncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (qres != cudaDriverEntryPointSuccess || ptr == nullptr) return static_cast<int>(cudaErrorNotSupported);
    fn = reinterpret_cast<TensorMapEncodeFn>(ptr);
  }
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = fn(map, dtype, static_cast<cuuint32_t>(rank), const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(cudaErrorInvalidValue);
}

static int encode_act_map(CUtensorMap* map, const void* base, size_t rows, int K, int box_rows,
                          CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_FLOAT16) {
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
  const cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
  return encode_map(map, dtype, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// F16 rows as a tensor [K / 64][rows][64]: a box is a K stage of box_rows rows, four sub-tiles of 64 K one behind the other, so that
// one copy fetches what four boxes of 64 K did.
static int encode_stage_map(CUtensorMap* map, const void* base, size_t rows, int K, int box_rows) {
  const cuuint64_t dims[3] = {64u, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(K / 64)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(K) * 2, 128u};
  const cuuint32_t box[3] = {64u, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(KS / 64)};
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Experiment switch (environment variable MSK_FUSED_PLAIN): launch the one-launch kernel without the
// cooperative attribute. Its grid never exceeds the SM count and it holds an SM per CTA, so its CTAs
// are resident together in practice, and its waits are bounded either way.
static bool fused_plain_launch() {
  static int v = -1;
  if (v < 0) v = std::getenv("MSK_FUSED_PLAIN") != nullptr ? 1 : 0;
  return v == 1;
}

// MODE 2 (one launch for the step) waits on a grid-wide counter, so it is launched cooperatively:
// either every CTA is resident or the launch fails. The other modes are chained with programmatic
// dependent launch (unless pdl == 0).
template <int N, int MODE>
static int launch_gemm(const GemmParams& p, int grid, cudaStream_t st, int pdl) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(moe_gemm_kernel<N, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         GemmCfg<N>::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(static_cast<unsigned>(grid));
  lc.blockDim = dim3(GEMM_THREADS);
  lc.dynamicSmemBytes = GemmCfg<N>::SMEM_BYTES;
  lc.stream = st;
  cudaLaunchAttribute at[1];
  if (MODE == 2 && !fused_plain_launch()) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  } else {
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // may start while its predecessor drains
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  }
  lc.attrs = at;
  lc.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&lc, moe_gemm_kernel<N, MODE>, p));
}

template <int MODE>
static int launch_gemm_n(int N, const GemmParams& p, int grid, cudaStream_t st, int pdl) {
  switch (N) {
    case 16: return launch_gemm<16, MODE>(p, grid, st, pdl);
    case 32: return launch_gemm<32, MODE>(p, grid, st, pdl);
    case 64: return launch_gemm<64, MODE>(p, grid, st, pdl);
    default: return MSK_ERR_SHAPE;
  }
}

static int launch_gemm_fused(int N, const GemmParams& p, int grid, cudaStream_t st) {
  switch (N) {
    case 16: return launch_gemm<16, 2>(p, grid, st, 0);
    case 32: return launch_gemm<32, 2>(p, grid, st, 0);
    case 64: return launch_gemm<64, 2>(p, grid, st, 0);
    default: return MSK_ERR_SHAPE;
  }
}

// The kernel on pairs of SMs (pair.cuh). An odd grid is rounded up to whole pairs.
static int launch_pair(PairParams& p, const __half* xs, size_t rows, int grid, cudaStream_t st, int pdl) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(moe_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  for (int i = 0; i < PAIR_MAPS; ++i) {
    int e = encode_stage_map(&p.tmap[0][i], xs, rows, p.K[0], 8 * (i + 1));
    if (e == 0) e = encode_stage_map(&p.tmap[1][i], p.inter, rows, p.K[1], 8 * (i + 1));
    if (e != 0) return e;
  }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(static_cast<unsigned>((grid + 1) / 2 * 2));
  lc.blockDim = dim3(PAIR_THREADS);
  lc.dynamicSmemBytes = PairCfg::SMEM_BYTES;
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  lc.attrs = at;
  lc.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&lc, moe_pair_kernel, p));
}

static int launch_nvf4(const NvParams& p, int grid, cudaStream_t st, int pdl) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(moe_nvf4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NvCfg::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(static_cast<unsigned>(grid));
  lc.blockDim = dim3(NV_THREADS);
  lc.dynamicSmemBytes = NvCfg::SMEM_BYTES;
  lc.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeCooperative;   // its CTAs wait for one another: all resident, or the launch fails
  at[0].val.cooperative = fused_plain_launch() ? 0 : 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = pdl;
  lc.attrs = at;
  lc.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&lc, moe_nvf4_kernel, p));
}

// ---- the few-token kernel (few.cuh): shapes it takes, its shared memory and its dealing of work
struct FewPlan {
  int n_slots, slot_kb, part_bytes, n_light, w_light, w_heavy;
  int xb_off, ys_off, part_off, ctl_off, smem;
  uint32_t inv_oct1;
};

// False when the step does not fit: more than eight tokens, token rows and owned output rows that leave less than
// two K blocks per warp (55 KB in flight per SM), or so many gate/up units that their tile number by the
// reciprocal of I / 8 could be one too large: u * ceil(2^32 / n) / 2^32 has the integer part u / n as long as u times
// the reciprocal's excess stays below 2^32 (nothing below I = 53,000 is refused by this).
static bool few_plan(const MskMoeCfg* c, int T, bool given_ids, int grid, FewPlan* f) {
  if (T > FEW_TOKENS || T * c->top_k > FEW_ENTRIES) return false;
  const uint64_t oct1 = static_cast<uint64_t>(c->inter) / 8, inv = ((1ull << 32) + oct1 - 1) / oct1;
  if (static_cast<uint64_t>(T) * c->top_k * oct1 * (inv * oct1 - (1ull << 32)) >= (1ull << 32)) return false;
  f->inv_oct1 = static_cast<uint32_t>(inv);
  const int groups = c->hidden / (2 * OCT_ROWS), own = (groups + grid - 1) / grid;
  const int x_bytes = T * (c->hidden * 2 + 64), ys_bytes = T * c->top_k * own * 64;
  // rows of a tile: one per token when the top-k is taken here; given ids may repeat an expert
  f->part_bytes = 128 * ((std::min(FEW_TOKENS, given_ids ? T * c->top_k : T) + 1) / 2);
  const int parts = FEW_WARPS * 2 * f->part_bytes;
  const int left = 227 * 1024 - x_bytes - ys_bytes - parts - static_cast<int>(sizeof(FewCtl));
  const int ring_kb = left < 0 ? 0 : left / (FEW_WARPS * FEW_KB_BYTES);   // K blocks a warp's ring can hold
  if (ring_kb < 2) return false;
  f->slot_kb = ring_kb >= 4 ? 2 : 1;
  f->n_slots = ring_kb >= 4 ? 2 : ring_kb;
  f->xb_off = FEW_WARPS * f->n_slots * f->slot_kb * FEW_KB_BYTES;
  f->ys_off = f->xb_off + x_bytes;
  f->part_off = f->ys_off + ys_bytes;
  f->ctl_off = f->part_off + parts;
  f->smem = f->ctl_off + static_cast<int>(sizeof(FewCtl));
  // gate/up units per super-round: a CTA with one group more of output rows streams that many bytes less of
  // gate/up weights; the smallest pair of weights within 4 % of that ratio
  const int extra = groups % grid;
  f->n_light = extra == 0 ? grid : grid - extra;
  f->w_light = f->w_heavy = 1;
  // (one token has few units per team, and they go round the teams evenly only when every CTA has as many)
  if (T == 1) {
    f->n_light = grid;
  } else if (extra != 0) {
    const double unit = 2.0 * (c->hidden / KS), group = 2.0 * (c->inter / KS), per_cta = (c->inter / 8 * unit + groups * group) / grid;
    const double light = per_cta - (groups / grid) * group, heavy = per_cta - own * group;
    if (heavy <= 0.1 * light) {
      f->w_heavy = 0;
    } else {
      for (int wh = 1; wh <= 6; ++wh) {
        const int wl = static_cast<int>(light / heavy * wh + 0.5);
        f->w_light = wl;
        f->w_heavy = wh;
        if (std::fabs(wl * heavy / (wh * light) - 1.0) <= 0.04) break;
      }
    }
  }
  return true;
}

// Whether a step of path 0 runs in the few-token kernel; inputs: MSK_FEW_* bits. It saves latency (prologue, hand-overs,
// launches) and loses where the decode work in its warps sets the pace: with the touched experts, which the host does not
// know, so the lines lie where independent routes are no slower than in the tcgen05 kernel. rows: routed rows expected
// for this rank's experts, T * k * nloc / E. Measured, whole steps in us, this kernel / the other: all of 128 experts
// (H4096 I1536 top-8, eight rows a token) 3 tokens 62 / 63, with the post-expert norm 69 / 69 (Zipf routes 46 / 55); a
// rank with one row a token (H4096 I4096) 3: 38 / 50, (H7168 I2048) 32 / 39; a small model (H2048 I1024, four rows) 24 / 38.
//   Pre-expert norm (the other: three launches): eight rows 4: 89 / 90, 5: 99 / 92 (Zipf, 6: 78 / 96); one row, H4096
// 5: 59 / 65, H7168 6: 62 / 56 (each CTA holds and norms six such rows); four rows 6: 34 / 41.
//   Token rows in host memory: the CTAs read them over PCIe once, a slice each, and share an F16 copy, one exchange more,
// and short runs of output columns go back: eight rows 2: 59 / 66, 3: 76 / 73, with given ids and the post-expert norm
// 86 / 78; one row 3: 49 / 56; four rows 3: 35 / 43. With the pre-expert norm every CTA needs whole rows, and 148 times the
// bytes over PCIe cost far more than the kernel saves (eight rows 1: 68 / 44, 6: 265 / 122): another kernel norms them once.
static bool few_takes(const MskMoeCfg* c, int T, int inputs, int grid, FewPlan* f) {
  const bool pre = (inputs & MSK_FEW_PRE_NORM) != 0, host = (inputs & MSK_FEW_HOST_X) != 0;
  const double rows = static_cast<double>(T) * c->top_k * c->local_count / c->n_experts;
  const int most = pre ? (host ? 0 : c->hidden <= 4096 && rows <= 24 ? 6 : 4) : host && rows > 16 ? 2 : 3;
  return T <= most && few_plan(c, T, (inputs & MSK_FEW_GIVEN_IDS) != 0, grid, f);
}

// With the pre-expert norm the other forms have a kernel in front of the GEMMs: the folded form (a row copy by many CTAs, then routes in every CTA
// of both GEMMs) or the chain (a sort launch whose one CTA norms the rows as well, and a combine: a launch more, and nothing that grows with the routes
// but the combine). The chain takes the steps with the post-expert norm that have local routes enough, from five tokens on (few_takes() has those
// below). Folded / chain, us, rows of steps, local routes a token:
//   given ids: a half, H2048 I1024, 8: 26 / 31; one, H2048 8: 29 / 31, H7168 I1280 5: 49 / 52, 8: 55 / 58; two, H2048 8: 34.4 / 32.3, H4096 I1024 48 / 46.5, of less
// than 40 MB of weights H1024 I512 24.5 / 26.1, H2048 I512 29.5 / 29.7; four, H2048 I1024 46 / 43;
//   logits, which every CTA ranks: 64 experts 31.4 / 33.7 (one), 37 / 35.5 (two); 128, H4096 I1024 one 47 / 43, I512 43 / 41; 256, H7168 60 / 55 .. 73 / 62.
// Rows in host memory and routes on the device (many CTAs fetch the rows faster than one): one route, H7168 4: 50 / 70, 8: 59 / 95; four, H2048 8: 44.4 / 46.7; eight,
// H4096 I1024 6: 79 / 79, 8: 104 / 92. Routes in host memory too, which the folded form fetches once a CTA (35 to 70 us for one step from
// run to run): eight 1: 41 - 55 / 52, 3: 71 - 110 / 70, 8: 115 - 165 / 95; four 3: 35 - 69 / 41, 8: 65 - 87 / 51; one, H7168 2: 49 - 102 / 70, 8: 88 - 155 / 107.
static bool chain_with_pre_norm(const MskMoeCfg* c, int T, int inputs) {
  const bool host_x = (inputs & MSK_FEW_HOST_X) != 0;
  const double mean = static_cast<double>(c->top_k) * c->local_count / c->n_experts;   // local routes of a token
  if (host_x && (inputs & MSK_STEP_HOST_ROUTES) != 0) return mean > 2.0 && T >= 3;
  if ((inputs & MSK_STEP_POST_NORM) == 0 || T <= ONE_LAUNCH_NORM_TOKENS) return false;
  if (host_x) return mean > 4.0;
  return mean > 2.0 || (mean == 2.0 && T * mean * 3.0 * c->hidden * c->inter * 0.5625 >= 40e6) ||
         ((inputs & MSK_FEW_GIVEN_IDS) == 0 && c->n_experts >= 128 && mean >= 1.0);
}

// The form that a step runs in, MSK_FORM_*, and with the few-token kernel its plan; inputs: MSK_FEW_* and MSK_STEP_* bits. nv_room: whether
// the workspace has room for the FP4 kernel's split rows.
// With the post-expert norm the one launch ends with tickets per token and a combine by whole CTAs; from four tokens on the sort, both
// GEMMs and the combine as launches of their own are faster (one launch / those, us, rows of steps): H2048 I1024 E64 top-4 4: 35.6 /
// 33.7, 5: 36.6 / 34.6, 6: 42.5 / 38.2, 8: 46.2 / 40.2; a rank of H4096 I4096 4: 41.7 / 39.5, 8: 52.0 /
// 49.6; 8 of 64 experts of H2048 I1024 8: 31.8 / 29.1 (two launches more are 1.3 us where no route is local: 12.5 / 13.8). Without the norm, whose tickets are per token and columns: 4: 31.4 / 32.8, 8: 39.7 / 39.2, H4096 I1536 E128 5: 78.6 / 80.0.
// Rows in host memory: every CTA of the one launch reads the logits or ids over PCIe, the sort launch once, H2048 I1024 4: 50 - 53 / 39.0,
// 8: 65 / 46.8, given ids 8: 59 - 71 / 44.2; H4096 I1536 E128 4: 95 / 78.5, given ids 3: 71 - 76 / 62.2, 4: 92 - 98 / 73.
static int step_form(const MskMoeCfg* c, int T, const Plan& p, int inputs, bool nv_room, FewPlan* few) {
  const bool pre = (inputs & MSK_FEW_PRE_NORM) != 0, post = (inputs & MSK_STEP_POST_NORM) != 0, host_x = (inputs & MSK_FEW_HOST_X) != 0;
  const bool nv = nv_room && nv_takes(c, T, p, (pre ? MSK_NVF4_PRE_NORM : 0) | (post ? MSK_NVF4_POST_NORM : 0));
  if (p.path == 0 && !(nv && c->local_count == c->n_experts) && few_takes(c, T, inputs, p.grid, few)) return MSK_FORM_FEW;
  if (nv) return MSK_FORM_NVF4;
  if (p.path == 2) return MSK_FORM_FOLDED;
  if (p.path == 0) {
    if (pre) return c->decode_path == 0 && chain_with_pre_norm(c, T, inputs) ? MSK_FORM_CHAIN : MSK_FORM_FOLDED;
    return c->decode_path == 0 && (host_x || (post && T >= ONE_LAUNCH_NORM_TOKENS)) ? MSK_FORM_BOTH_GEMMS : MSK_FORM_ONE_LAUNCH;
  }
  if (p.N == 128) return c->decode_path == 1 || c->stop_after == 2 ? MSK_FORM_CHAIN : MSK_FORM_BOTH_GEMMS;
  return p.both && (p.N == 64 || !pre) ? MSK_FORM_BOTH_GEMMS : MSK_FORM_CHAIN;   // narrow tiles: the pre-expert norm needs the row-copy kernel
}

static bool in_host_memory(const void* p) {   // page-locked, or pageable where the device can read that
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();   // not this call's error
    return false;
  }
  return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeUnregistered;
}

static int launch_few(const FewParams& p, int grid, int smem, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(moe_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(static_cast<unsigned>(grid));
  lc.blockDim = dim3(FEW_THREADS);
  lc.dynamicSmemBytes = static_cast<size_t>(smem);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;   // its CTAs wait for one another: all resident, or the launch fails
  at[0].val.cooperative = fused_plain_launch() ? 0 : 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&lc, moe_few_kernel, p));
}

static RepackGeom geom13(const MskMoeCfg* c) {
  return RepackGeom{2 * c->inter, c->hidden, c->inter / 128, c->hidden / KS, c->inter};
}
static RepackGeom geom2(const MskMoeCfg* c) {
  return RepackGeom{c->hidden, c->inter, c->hidden / 256, c->inter / KS, 0};
}
static long long n_og_of(const MskMoeCfg* c, const RepackGeom& g) {   // octet-gus: 8-row slices of all experts
  return static_cast<long long>(c->local_count) * g.n_pairs * 2 * TILE_OCTETS;
}

template <int N>
static int launch_router_hilo(const CUtensorMap& mw, const CUtensorMap& mx, float* logits, int32_t* status, int T, int E,
                              int H, int pdl, cudaStream_t st) {
  const int smem = RG_STAGES * (2 * RG_A_BYTES + N * RG_KSTEP * 2) + static_cast<int>(sizeof(RouterGemmCtrl));
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(router_hilo_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t lc{};
  // as many CTAs per tile (of K) as the machine has room for: one wave
  const int tiles = ((E + 127) / 128) * ((T + N - 1) / N);
  int split = 8;
  while (split > 1 && (split * tiles > DEFAULT_CTAS || split > H / RG_KSTEP)) split /= 2;
  lc.gridDim = dim3(static_cast<unsigned>(split), static_cast<unsigned>((E + 127) / 128), static_cast<unsigned>((T + N - 1) / N));
  lc.blockDim = dim3(RG_THREADS);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = static_cast<unsigned>(split);
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&lc, router_hilo_kernel<N>, mw, mx, logits, status, T, E, H));
}

}  // namespace msk

using namespace msk;

extern "C" {

int msk_moe_packed_bytes(const MskMoeCfg* cfg, size_t* host_w13_bytes, size_t* host_w2_bytes) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (host_w13_bytes == nullptr || host_w2_bytes == nullptr) return MSK_ERR_NULL;
  *host_w13_bytes = static_cast<size_t>(n_og_of(cfg, geom13(cfg))) * (cfg->hidden / KS) * OCT_BYTES;
  *host_w2_bytes = static_cast<size_t>(n_og_of(cfg, geom2(cfg))) * (cfg->inter / KS) * OCT_BYTES;
  return MSK_OK;
}

static int repack_common(const MskMoeCfg* cfg, void* w13, void* w13_sf, void* w2, void* w2_sf, void* packed13,
                         void* packed2, void* stream, bool inverse) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!w13 || !w13_sf || !w2 || !w2_sf || !packed13 || !packed2) return MSK_ERR_NULL;
  if (!aligned16(w13) || !aligned16(w13_sf) || !aligned16(w2) || !aligned16(w2_sf) || !aligned16(packed13) ||
      !aligned16(packed2))
    return MSK_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const RepackGeom g13 = geom13(cfg), g2 = geom2(cfg);
  const long long n13 = n_og_of(cfg, g13), n2 = n_og_of(cfg, g2);
  auto launch = [&](auto kern, int warps, void* codes, void* sf, void* packed, const RepackGeom& g, long long n) {
    kern<<<static_cast<unsigned>((n + warps - 1) / warps), warps * 32, 0, st>>>(static_cast<uint8_t*>(codes), static_cast<uint8_t*>(sf),
                                                                               static_cast<uint8_t*>(packed), g, n);
  };
  if (!inverse) {
    launch(repack_kernel<false>, REPACK_WARPS<false>, w13, w13_sf, packed13, g13, n13);
    launch(repack_kernel<false>, REPACK_WARPS<false>, w2, w2_sf, packed2, g2, n2);
  } else {
    launch(repack_kernel<true>, REPACK_WARPS<true>, w13, w13_sf, packed13, g13, n13);
    launch(repack_kernel<true>, REPACK_WARPS<true>, w2, w2_sf, packed2, g2, n2);
  }
  return static_cast<int>(cudaGetLastError());
}

int msk_moe_repack(const MskMoeCfg* cfg, const void* w13, const void* w13_sf, const void* w2, const void* w2_sf,
                   void* packed13, void* packed2, void* stream) {
  return repack_common(cfg, const_cast<void*>(w13), const_cast<void*>(w13_sf), const_cast<void*>(w2),
                       const_cast<void*>(w2_sf), packed13, packed2, stream, false);
}

int msk_moe_unpack(const MskMoeCfg* cfg, const void* packed13, const void* packed2, void* w13, void* w13_sf,
                   void* w2, void* w2_sf, void* stream) {
  return repack_common(cfg, w13, w13_sf, w2, w2_sf, const_cast<void*>(packed13), const_cast<void*>(packed2), stream,
                       true);
}

int msk_moe_dequant_packed(const MskMoeCfg* cfg, const void* packed13, const void* packed2, void* dq13, void* dq2,
                           void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!packed13 || !packed2 || !dq13 || !dq2) return MSK_ERR_NULL;
  if (!aligned16(packed13) || !aligned16(packed2) || !aligned16(dq13) || !aligned16(dq2)) return MSK_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const RepackGeom g13 = geom13(cfg), g2 = geom2(cfg);
  const long long n13 = n_og_of(cfg, g13), n2 = n_og_of(cfg, g2);
  dequant_packed_kernel<<<static_cast<unsigned>(n13 / 16 * g13.n_stages), 128, 0, st>>>(
      static_cast<const uint8_t*>(packed13), static_cast<__nv_bfloat16*>(dq13), g13, n13);
  dequant_packed_kernel<<<static_cast<unsigned>(n2 / 16 * g2.n_stages), 128, 0, st>>>(
      static_cast<const uint8_t*>(packed2), static_cast<__nv_bfloat16*>(dq2), g2, n2);
  return static_cast<int>(cudaGetLastError());
}

int msk_moe_router_logits(const MskMoeCfg* cfg, const void* x, const float* router_w, float* logits, int n_tokens,
                          void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!x || !router_w || !logits) return MSK_ERR_NULL;
  if (n_tokens < 0) return MSK_ERR_SHAPE;
  if (n_tokens == 0) return MSK_OK;
  auto* kern = aligned16(x) && aligned16(router_w) ? router_logits_kernel<true> : router_logits_kernel<false>;
  const dim3 grid(static_cast<unsigned>(cfg->n_experts),
                  static_cast<unsigned>(std::min((n_tokens + ROUTER_TOKENS - 1) / ROUTER_TOKENS, 65535)));
  kern<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), router_w, logits, n_tokens, cfg->hidden, cfg->n_experts);
  return static_cast<int>(cudaGetLastError());
}

int msk_moe_router_logits_hilo(const MskMoeCfg* cfg, const void* x, const void* router_hilo, float* logits,
                               int32_t* status_word, int n_tokens, void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!x || !router_hilo || !logits) return MSK_ERR_NULL;
  if (!aligned16(x) || !aligned16(router_hilo) || !aligned16(logits)) return MSK_ERR_ALIGN;
  if (n_tokens < 0) return MSK_ERR_SHAPE;
  if (n_tokens == 0) return MSK_OK;
  if (n_tokens < 16) return MSK_ERR_SHAPE;   // fewer tokens than the narrowest MMA tile: use msk_moe_router_logits
  // (below 2048 tokens tiles of 64 fill the machine better: eight CTAs per tile)
  const int N = n_tokens >= 2048 ? 128 : n_tokens >= 64 ? 64 : n_tokens >= 32 ? 32 : 16;
  CUtensorMap mw, mx;
  int e = encode_act_map(&mw, router_hilo, static_cast<size_t>(2) * cfg->n_experts, cfg->hidden, 128,
                         CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
  if (e != 0) return e;
  e = encode_act_map(&mx, x, static_cast<size_t>(n_tokens), cfg->hidden, N, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
  if (e != 0) return e;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int pdl = cfg->no_pdl ? 0 : 1;
  switch (N) {
    case 128: return launch_router_hilo<128>(mw, mx, logits, status_word, n_tokens, cfg->n_experts, cfg->hidden, pdl, st);
    case 64: return launch_router_hilo<64>(mw, mx, logits, status_word, n_tokens, cfg->n_experts, cfg->hidden, pdl, st);
    case 32: return launch_router_hilo<32>(mw, mx, logits, status_word, n_tokens, cfg->n_experts, cfg->hidden, pdl, st);
    default: return launch_router_hilo<16>(mw, mx, logits, status_word, n_tokens, cfg->n_experts, cfg->hidden, pdl, st);
  }
}

static int launch_topk(const MskMoeCfg* cfg, const float* logits, const float* bias, int32_t* ids, float* tw, int n_tokens, cudaStream_t st) {
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(static_cast<unsigned>((n_tokens + 7) / 8));
  lc.blockDim = dim3(256);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = cfg->no_pdl ? 0 : 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&lc, route_topk_kernel, logits, bias, ids, tw, n_tokens, static_cast<int>(cfg->n_experts),
                                             static_cast<int>(cfg->top_k), static_cast<int>(cfg->routing_mode), cfg->route_scale));
}

int msk_moe_route(const MskMoeCfg* cfg, const float* logits, const float* bias, int32_t* topk_ids,
                  float* topk_weights, int n_tokens, void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!logits || !topk_ids || !topk_weights) return MSK_ERR_NULL;
  if (n_tokens < 0 || cfg->top_k > cfg->n_experts) return MSK_ERR_SHAPE;
  if (n_tokens == 0) return MSK_OK;
  return launch_topk(cfg, logits, bias, topk_ids, topk_weights, n_tokens, static_cast<cudaStream_t>(stream));
}

static int launch_sort(const MskMoeCfg* cfg, const int32_t* ids, int n_tokens, int32_t* cnt, int32_t* off,
                       int32_t* perm, int32_t* inv, cudaStream_t st, const __nv_bfloat16* x = nullptr,
                       __half* xh = nullptr, const void* pre_w = nullptr, float pre_eps = 0.f) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(SortSmem)));
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(1);
  lc.blockDim = dim3(SORT_THREADS);
  lc.dynamicSmemBytes = sizeof(SortSmem);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = cfg->no_pdl ? 0 : 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&lc, sort_kernel, ids, static_cast<int>(n_tokens * cfg->top_k),
                                             static_cast<int>(cfg->local_start), static_cast<int>(cfg->local_count),
                                             cnt, off, perm, inv, x, xh, n_tokens, static_cast<int>(cfg->hidden),
                                             static_cast<const __nv_bfloat16*>(pre_w), pre_eps));
}

// Top-k (when logits are given; otherwise ids is only read) and sort on several CTAs (route_sort.cuh).
static int launch_sort_multi(const MskMoeCfg* cfg, const float* logits, const float* bias, int32_t* ids, float* tw, int n_tokens,
                             int32_t* cnt, int32_t* off, int32_t* perm, int32_t* inv, int32_t* blk, cudaStream_t st) {
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(static_cast<unsigned>(std::min(SORT_MULTI_BLOCKS, (n_tokens + SORT_MULTI_TOKENS - 1) / SORT_MULTI_TOKENS)));
  lc.blockDim = dim3(SORT_THREADS);
  lc.dynamicSmemBytes = sizeof(SortSmem);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = cfg->no_pdl ? 0 : 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  const int k = static_cast<int>(cfg->top_k), lo = static_cast<int>(cfg->local_start), nloc = static_cast<int>(cfg->local_count);
  const int e = static_cast<int>(cudaLaunchKernelEx(&lc, sort_multi_count_kernel, logits, bias, ids, tw, n_tokens,
                                                    static_cast<int>(cfg->n_experts), k, static_cast<int>(cfg->routing_mode),
                                                    cfg->route_scale, lo, nloc, blk));
  if (e != 0) return e;
  return static_cast<int>(cudaLaunchKernelEx(&lc, sort_multi_scatter_kernel, static_cast<const int32_t*>(ids), n_tokens, k, lo,
                                             nloc, static_cast<const int32_t*>(blk), cnt, off, perm, inv));
}

constexpr int FUSED_ROUTE_MAX_TOKENS = 32;  // up to here one CTA routes and sorts in a single launch

static bool sort_on_several_ctas(const MskMoeCfg* cfg, int n_tokens) {
  const long long entries = static_cast<long long>(n_tokens) * cfg->top_k;
  return n_tokens > FUSED_ROUTE_MAX_TOKENS &&
         (entries >= SORT_MULTI_MIN || entries * cfg->local_count >= static_cast<long long>(SORT_MULTI_MIN_LOCAL) * cfg->n_experts);
}

static int launch_route_sort(const MskMoeCfg* cfg, const float* logits, const float* bias, int32_t* ids, float* tw,
                             int n_tokens, int32_t* cnt, int32_t* off, int32_t* perm, int32_t* inv, cudaStream_t st,
                             const __nv_bfloat16* x, __half* xh, const void* pre_w = nullptr, float pre_eps = 0.f) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(route_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(SortSmem)));
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(1);
  lc.blockDim = dim3(SORT_THREADS);
  lc.dynamicSmemBytes = sizeof(SortSmem);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = cfg->no_pdl ? 0 : 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&lc, route_sort_kernel, logits, bias, ids, tw, n_tokens,
                                             static_cast<int>(cfg->n_experts), static_cast<int>(cfg->top_k),
                                             static_cast<int>(cfg->routing_mode), cfg->route_scale,
                                             static_cast<int>(cfg->local_start), static_cast<int>(cfg->local_count),
                                             cnt, off, perm, inv, x, xh, static_cast<int>(cfg->hidden),
                                             static_cast<const __nv_bfloat16*>(pre_w), pre_eps));
}

int msk_moe_sort(const MskMoeCfg* cfg, const int32_t* topk_ids, int n_tokens, int32_t* cnt, int32_t* off,
                 int32_t* perm, int32_t* inv, void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!cnt || !off || !perm || !inv) return MSK_ERR_NULL;
  if (n_tokens < 0) return MSK_ERR_SHAPE;
  if (n_tokens > 0 && !topk_ids) return MSK_ERR_NULL;
  return launch_sort(cfg, topk_ids, n_tokens, cnt, off, perm, inv, static_cast<cudaStream_t>(stream));
}

int msk_moe_workspace_bytes(const MskMoeCfg* cfg, size_t* host_bytes) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!host_bytes) return MSK_ERR_NULL;
  if (cfg->max_tokens < 1) return MSK_ERR_SHAPE;
  *host_bytes = carve(cfg, cfg->max_tokens).total;
  return MSK_OK;
}

int msk_moe_workspace_init(const MskMoeCfg* cfg, void* workspace, size_t workspace_bytes, void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!workspace) return MSK_ERR_NULL;
  if (cfg->max_tokens < 1) return MSK_ERR_SHAPE;
  const Carve k = carve(cfg, cfg->max_tokens);
  if (k.total > workspace_bytes) return MSK_ERR_WORKSPACE;
  // status word, tables and split-K tickets all sit below `inter`
  return static_cast<int>(cudaMemsetAsync(workspace, 0, k.inter, static_cast<cudaStream_t>(stream)));
}

int msk_moe_workspace_view(const MskMoeCfg* cfg, void* workspace, int which, void** host_ptr) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!workspace || !host_ptr) return MSK_ERR_NULL;
  if (cfg->max_tokens < 1) return MSK_ERR_SHAPE;
  const Carve k = carve(cfg, cfg->max_tokens);
  uint8_t* b = static_cast<uint8_t*>(workspace);
  switch (which) {
    case 0: *host_ptr = b + k.cnt; break;
    case 1: *host_ptr = b + k.off; break;
    case 2: *host_ptr = b + k.perm; break;
    case 3: *host_ptr = b + k.inv; break;
    case 4: *host_ptr = b + k.inter; break;
    case 5: *host_ptr = b + k.y; break;
    case 6: *host_ptr = b + k.trace; break;
    case 7: *host_ptr = b + k.tickets; break;
    case 8: *host_ptr = b + k.few_ctl; break;
    case 9: *host_ptr = b + k.sort_blk; break;
    case 10: *host_ptr = b + k.tile_ctr; break;
    default: return MSK_ERR_SHAPE;
  }
  return MSK_OK;
}

// y_bf16: the pair kernel keeps y in BF16 (half the bytes written and read back).
static int launch_combine(const MskMoeCfg* cfg, bool y_bf16, const float* y, const int32_t* inv, const float* tw, void* out,
                          int n_tokens, bool post_norm, int pdl, cudaStream_t st) {
  cudaLaunchConfig_t lc{};
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl;
  lc.attrs = at;
  lc.numAttrs = 1;
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  const int H = static_cast<int>(cfg->hidden), k = static_cast<int>(cfg->top_k);
  const bool few_local = static_cast<long long>(k) * cfg->local_count <= 2LL * cfg->n_experts;   // two or fewer of a token's routes expected
  if (!post_norm) {
    const int cols = few_local ? 1024 : 256;
    const long long items = static_cast<long long>(n_tokens) * ((H + cols - 1) / cols);
    lc.gridDim = dim3(static_cast<unsigned>((items + COMBINE_COLS_WARPS - 1) / COMBINE_COLS_WARPS));
    lc.blockDim = dim3(COMBINE_COLS_WARPS * 32);
    auto* kern = y_bf16 ? (few_local ? combine_cols_kernel<true, 2, 4> : combine_cols_kernel<true, 8, 1>)
                        : (few_local ? combine_cols_kernel<false, 2, 4> : combine_cols_kernel<false, 8, 1>);
    return static_cast<int>(cudaLaunchKernelEx(&lc, kern, y, inv, tw, o, n_tokens, H, k));
  }
  lc.gridDim = dim3(static_cast<unsigned>(n_tokens));
  const bool narrow = H <= 4096, short_rows = H <= 2048;
  if (n_tokens < COMBINE_FEW_TOKENS) {
    lc.blockDim = dim3(512);
    auto* kern = y_bf16 ? (narrow ? combine_norm_kernel<true, 512, 1, 8, 1> : combine_norm_kernel<true, 512, 2, 8, 1>)
                        : (narrow ? combine_norm_kernel<false, 512, 1, 8, 1> : combine_norm_kernel<false, 512, 2, 4, 1>);
    return static_cast<int>(cudaLaunchKernelEx(&lc, kern, y, inv, tw, o, H, k, cfg->post_norm_eps));
  }
  lc.blockDim = dim3(narrow ? 128 : 256);
  auto* kern = !y_bf16 ? (short_rows ? combine_norm_kernel<false, 128, 2, 4, 4> : narrow ? combine_norm_kernel<false, 128, 4, 2, 4> : combine_norm_kernel<false, 256, 4, 2, 2>)
               : few_local ? (short_rows ? combine_norm_kernel<true, 128, 2, 2, 8> : narrow ? combine_norm_kernel<true, 128, 4, 2, 5> : combine_norm_kernel<true, 256, 4, 2, 3>)
                           : (short_rows ? combine_norm_kernel<true, 128, 2, 4, 6> : narrow ? combine_norm_kernel<true, 128, 4, 4, 4> : combine_norm_kernel<true, 256, 4, 4, 2>);
  return static_cast<int>(cudaLaunchKernelEx(&lc, kern, y, inv, tw, o, H, k, cfg->post_norm_eps));
}

// ev, when given, holds 6 events: [0] before the step, [1] after routing + sort, [5] after the row copy,
// [2] after the gate/up GEMM, [3] after the down GEMM, [4] after the combine.
static int forward_impl(const MskMoeCfg* cfg, const void* packed13, const void* packed2, const float* gs13,
                        const float* gs2, const void* post_norm_w, const void* x, const int32_t* topk_ids,
                        const float* topk_weights, void* out, void* workspace, size_t workspace_bytes, int n_tokens,
                        void* stream, cudaEvent_t* ev, const float* logits = nullptr, const float* bias = nullptr,
                        int32_t* ids_out = nullptr, float* tw_out = nullptr, const void* pre_norm_w = nullptr,
                        float pre_norm_eps = 1e-5f) {
  // with `logits` the routing runs here too: ids_out / tw_out receive it and feed the rest
  if (logits != nullptr) {
    if (!ids_out || !tw_out) return MSK_ERR_NULL;
    topk_ids = ids_out;
    topk_weights = tw_out;
  }
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!packed13 || !packed2 || !gs13 || !gs2 || !workspace) return MSK_ERR_NULL;
  if (n_tokens < 0) return MSK_ERR_SHAPE;
  if (n_tokens == 0) return MSK_OK;
  if (!x || !topk_ids || !topk_weights || !out) return MSK_ERR_NULL;
  if (!aligned16(packed13) || !aligned16(packed2) || !aligned16(x) || !aligned16(out) || !aligned16(workspace))
    return MSK_ERR_ALIGN;
  if (n_tokens > cfg->max_tokens) return MSK_ERR_TOO_LARGE;
  // offsets depend on the capacity only, so control words keep their place from call to call
  const Carve k = carve(cfg, cfg->max_tokens);
  if (k.total > workspace_bytes) return MSK_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* b = static_cast<uint8_t*>(workspace);
  int32_t* status = reinterpret_cast<int32_t*>(b + k.status);
  int32_t* cnt = reinterpret_cast<int32_t*>(b + k.cnt);
  int32_t* off = reinterpret_cast<int32_t*>(b + k.off);
  int32_t* perm = reinterpret_cast<int32_t*>(b + k.perm);
  int32_t* inv = reinterpret_cast<int32_t*>(b + k.inv);
  int32_t* tickets = reinterpret_cast<int32_t*>(b + k.tickets);
  __half* inter = reinterpret_cast<__half*>(b + k.inter);
  float* y = reinterpret_cast<float*>(b + k.y);
  float* partial = reinterpret_cast<float*>(b + k.partial);
  __half* xs = reinterpret_cast<__half*>(b + k.xs);

  Plan plan = make_plan(cfg, n_tokens);
  if (plan.N != 16 && plan.N != 32 && plan.N != 64 && plan.N != 128) return MSK_ERR_SHAPE;
  if (plan.grid < 1 || plan.grid > MAX_CTAS) return MSK_ERR_SHAPE;
  const int pdl = cfg->no_pdl ? 0 : 1;
  const size_t r_max = static_cast<size_t>(cfg->max_tokens) * cfg->top_k;
  unsigned long long* trace = (cfg->trace != 0 && plan.grid <= static_cast<int>(TRACE_CTAS))
                                  ? reinterpret_cast<unsigned long long*>(b + k.trace) : nullptr;

  // what every launch of the two GEMMs shares
  GemmParams p{};
  p.cnt = cnt; p.off = off; p.perm = perm; p.inv = inv; p.status = status; p.trace = trace;
  p.nloc = cfg->local_count; p.top_k = cfg->top_k; p.flat = plan.flat;
  // weights stream through L2 once per token tile; the activation rows are what many CTAs re-read,
  // so the weights must not be the ones L2 keeps
  p.evict_first = 1;
  p.post_norm_w = static_cast<const __nv_bfloat16*>(post_norm_w);
  p.eps = cfg->post_norm_eps;
  FewPlan few;
  const bool host_x = plan.path == 0 && n_tokens <= FEW_TOKENS && in_host_memory(x);
  const bool host_routes = host_x && pre_norm_w != nullptr && in_host_memory(logits != nullptr ? static_cast<const void*>(logits) : topk_ids);
  const int inputs = (logits == nullptr ? MSK_FEW_GIVEN_IDS : 0) | (pre_norm_w != nullptr ? MSK_FEW_PRE_NORM : 0) |
                     (host_x ? MSK_FEW_HOST_X : 0) | (post_norm_w != nullptr ? MSK_STEP_POST_NORM : 0) | (host_routes ? MSK_STEP_HOST_ROUTES : 0);
  const int form = step_form(cfg, n_tokens, plan, inputs, k.nv_end <= workspace_bytes, &few);
  const bool nv = form == MSK_FORM_NVF4;
  if (form == MSK_FORM_FEW) {
    FewParams f{};
    f.w13 = static_cast<const uint8_t*>(packed13); f.w2 = static_cast<const uint8_t*>(packed2);
    f.gs13 = gs13; f.gs2 = gs2;
    f.x = static_cast<const __nv_bfloat16*>(x);
    f.pre_w = static_cast<const __nv_bfloat16*>(pre_norm_w); f.pre_eps = pre_norm_eps;
    f.post_w = static_cast<const __nv_bfloat16*>(post_norm_w); f.post_eps = cfg->post_norm_eps;
    f.xs = xs; f.inter = inter; f.y = y; f.out = static_cast<__nv_bfloat16*>(out);
    f.logits = logits; f.bias = bias; f.ids_in = topk_ids; f.tw_in = topk_weights; f.ids_out = ids_out; f.tw_out = tw_out;
    f.cnt = cnt; f.off = off; f.perm = perm; f.inv = inv; f.status = status;
    f.ctl = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4096);
    f.tile_done = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4352);
    f.norm_part = partial; f.trace = trace;
    // (the second region of pieces, which this kernel has no use for: at least 128 KB, for 8 rows of up to 512 logits)
    float* copies = partial + round_up(partial_floats(cfg) * 4, 256) / 4;
    f.logits_copy = host_x && logits != nullptr && in_host_memory(logits) ? copies : nullptr;
    f.ids_copy = host_x && logits == nullptr && in_host_memory(topk_ids) && in_host_memory(topk_weights) ? reinterpret_cast<int32_t*>(copies) : nullptr;
    f.H = cfg->hidden; f.I = cfg->inter; f.T = n_tokens; f.E = cfg->n_experts; f.k = cfg->top_k;
    f.lo = cfg->local_start; f.nloc = cfg->local_count; f.mode = cfg->routing_mode; f.route_scale = cfg->route_scale;
    f.route = logits != nullptr ? 1 : 2;
    f.share_x = host_x ? 1 : 0;
    f.inv_oct1 = few.inv_oct1;
    f.n_slots = few.n_slots; f.slot_kb = few.slot_kb; f.part_bytes = few.part_bytes; f.part_off = few.part_off;
    f.n_light = few.n_light; f.w_light = few.w_light; f.w_heavy = few.w_heavy;
    f.xb_off = few.xb_off; f.ys_off = few.ys_off; f.ctl_off = few.ctl_off;
    if (ev) { cudaEventRecord(ev[0], st); cudaEventRecord(ev[1], st); cudaEventRecord(ev[5], st); }
    const int e = launch_few(f, plan.grid, few.smem, st);
    if (ev) { cudaEventRecord(ev[2], st); cudaEventRecord(ev[3], st); cudaEventRecord(ev[4], st); }
    return e;
  }
  PhaseParams& g13 = p.ph[0];
  PhaseParams& g2 = p.ph[1];
  g13.w = static_cast<const uint8_t*>(packed13); g13.gs = gs13; g13.act = xs; g13.outp = inter;
  g13.partial = partial; g13.tickets = tickets;
  g13.K = cfg->hidden; g13.out_ld = cfg->inter; g13.n_pairs = cfg->inter / 128;
  g2.w = static_cast<const uint8_t*>(packed2); g2.gs = gs2; g2.act = inter; g2.outp = y;
  g2.partial = partial + round_up(partial_floats(cfg) * 4, 256) / 4;
  g2.tickets = tickets + round_up(ticket_ints(cfg, cfg->max_tokens) * 4, 256) / 4;
  g2.K = cfg->inter; g2.out_ld = cfg->hidden; g2.n_pairs = cfg->hidden / 256;

  if (form == MSK_FORM_ONE_LAUNCH || form == MSK_FORM_FOLDED) {
    // ---- few tokens: the GEMM kernels route, sort and combine themselves
    p.route = logits != nullptr ? 1 : 2;
    p.logits = logits; p.bias = bias; p.ids_in = topk_ids; p.ids_out = ids_out; p.tw_out = tw_out;
    p.T = n_tokens; p.E = cfg->n_experts; p.lo = cfg->local_start; p.mode = cfg->routing_mode;
    p.route_scale = cfg->route_scale;
    p.fold = post_norm_w != nullptr ? 1 : 2; p.tw = topk_weights; p.out = static_cast<__nv_bfloat16*>(out);
    p.tok_tickets = reinterpret_cast<int32_t*>(b + k.few_ctl);
    p.grid_bar = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4096);
    p.tile_done = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4352);
    p.tile_seen = p.tile_done + 384;
    p.x_bf16 = static_cast<const __nv_bfloat16*>(x);
    if (ev) { cudaEventRecord(ev[0], st); cudaEventRecord(ev[1], st); }
    if (form == MSK_FORM_ONE_LAUNCH) {
      if (ev) cudaEventRecord(ev[5], st);
      const int e1 = launch_gemm_fused(plan.N, p, plan.grid, st);
      if (ev) { cudaEventRecord(ev[2], st); cudaEventRecord(ev[3], st); cudaEventRecord(ev[4], st); }
      return e1;
    }
    // F16 copy of the token rows (with the pre-expert norm when asked for), small blocks so that the
    // gate/up kernel's CTAs fit beside them; it waits for what precedes the step and lets go of its
    // dependents after that wait
    int e = 0;
    {
      const bool pre = pre_norm_w != nullptr;
      cudaLaunchConfig_t lc{};
      lc.stream = st;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[0].val.programmaticStreamSerializationAllowed = pdl;
      lc.attrs = at;
      lc.numAttrs = 1;
      if (pre) {
        lc.gridDim = dim3(static_cast<unsigned>(n_tokens));
        lc.blockDim = dim3(256);
        e = static_cast<int>(cudaLaunchKernelEx(&lc, copy_rows_kernel, static_cast<const __nv_bfloat16*>(x),
                                                static_cast<const int32_t*>(nullptr), static_cast<int>(cfg->top_k), 0,
                                                static_cast<int>(cfg->hidden), xs,
                                                static_cast<const __nv_bfloat16*>(pre_norm_w), pre_norm_eps));
      } else {
        const int n8 = n_tokens * (cfg->hidden / 8);
        lc.gridDim = dim3(static_cast<unsigned>((n8 + 63) / 64));
        lc.blockDim = dim3(64);
        e = static_cast<int>(cudaLaunchKernelEx(&lc, convert_rows_kernel, static_cast<const __nv_bfloat16*>(x), xs, n8));
      }
      if (e != 0) return e;
    }
    if (ev) cudaEventRecord(ev[5], st);
    e = launch_gemm_n<0>(plan.N, p, plan.grid, st, pdl);
    if (e != 0) return e;
    if (ev) cudaEventRecord(ev[2], st);
    if (trace) p.trace = trace + TRACE_WORDS;
    e = launch_gemm_n<1>(plan.N, p, plan.grid, st, pdl);
    if (ev) { cudaEventRecord(ev[3], st); cudaEventRecord(ev[4], st); }
    return e;
  }

  // ---- chain of launches: [top-k +] sort, [row copy,] gate/up GEMM, down GEMM, combine
  if (ev) cudaEventRecord(ev[0], st);
  int e = 0;
  // narrow token tiles read an F16 copy of x; for few tokens the sorting CTA makes it
  const bool tma_b = !nv && plan.N >= 64;  // GemmCfg<N>::TMA_B
  const bool both_gemms = form == MSK_FORM_BOTH_GEMMS;   // (N = 128: the pair kernel)
  const bool convert_in_sort = !nv && !tma_b && !both_gemms && n_tokens <= FUSED_ROUTE_MAX_TOKENS;
  const __nv_bfloat16* xin = convert_in_sort ? static_cast<const __nv_bfloat16*>(x) : nullptr;
  __half* xh_in_sort = convert_in_sort ? xs : nullptr;
  if (logits != nullptr && n_tokens <= FUSED_ROUTE_MAX_TOKENS) {
    e = launch_route_sort(cfg, logits, bias, ids_out, tw_out, n_tokens, cnt, off, perm, inv, st, xin, xh_in_sort,
                          pre_norm_w, pre_norm_eps);
  } else if (sort_on_several_ctas(cfg, n_tokens)) {
    e = launch_sort_multi(cfg, logits, bias, const_cast<int32_t*>(topk_ids), tw_out, n_tokens, cnt, off, perm, inv,
                          reinterpret_cast<int32_t*>(b + k.sort_blk), st);
  } else {
    if (logits != nullptr) {
      e = launch_topk(cfg, logits, bias, ids_out, tw_out, n_tokens, st);
      if (e != 0) return e;
    }
    e = launch_sort(cfg, topk_ids, n_tokens, cnt, off, perm, inv, st, xin, xh_in_sort, pre_norm_w, pre_norm_eps);
  }
  if (e != 0) return e;
  if (ev) cudaEventRecord(ev[1], st);
  if (cfg->stop_after == 1) return MSK_OK;

  if (!nv && !convert_in_sort && (tma_b || !both_gemms)) {
    // F16 copy of the token rows: sorted (expert-major) for the TMA tiles, plain [T, H] otherwise
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(static_cast<unsigned>(n_tokens));
    lc.blockDim = dim3(COPY_THREADS);
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl;
    lc.attrs = at;
    lc.numAttrs = 1;
    e = static_cast<int>(cudaLaunchKernelEx(&lc, copy_rows_kernel, static_cast<const __nv_bfloat16*>(x),
                                            static_cast<const int32_t*>(tma_b ? inv : nullptr), static_cast<int>(cfg->top_k),
                                            cfg->local_count < cfg->n_experts ? 1 : 0,
                                            static_cast<int>(cfg->hidden), xs,
                                            static_cast<const __nv_bfloat16*>(pre_norm_w), pre_norm_eps));
    if (e != 0) return e;
    if (tma_b && plan.N != 128) {
      for (int i = 0; (16 << i) <= plan.N; ++i) {
        e = encode_stage_map(&p.tmap_act[0][i], xs, r_max, cfg->hidden, 16 << i);
        if (e == 0) e = encode_stage_map(&p.tmap_act[1][i], inter, r_max, cfg->inter, 16 << i);
        if (e != 0) return e;
      }
    }
  }
  if (ev) cudaEventRecord(ev[5], st);
  if (nv) {
    NvParams q{};
    q.w[0] = g13.w; q.w[1] = g2.w; q.gs[0] = gs13; q.gs[1] = gs2;
    q.x = static_cast<const __nv_bfloat16*>(x);
    q.pre_w = static_cast<const __nv_bfloat16*>(pre_norm_w); q.pre_eps = pre_norm_eps;
    q.ids = topk_ids; q.inv = inv; q.cnt = cnt; q.off = off; q.post_norm_w = p.post_norm_w;
    q.inter = inter; q.y = y; q.status = status; q.trace = trace;
    for (int i = 0; i < 2; ++i) {
      q.img[i] = b + k.nv_img[i];
      q.K[i] = p.ph[i].K; q.n_pairs[i] = p.ph[i].n_pairs;
    }
    q.ctr = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4096);
    q.tiles = reinterpret_cast<unsigned int*>(b + k.nv_tiles);
    q.nloc = cfg->local_count; q.lo = cfg->local_start; q.H = cfg->hidden; q.I = cfg->inter; q.T = n_tokens; q.k = cfg->top_k;
    q.share_rows = in_host_memory(x) ? 0 : 1;
    e = launch_nvf4(q, plan.grid, st, pdl);
    if (e != 0) return e;
    if (ev) { cudaEventRecord(ev[2], st); cudaEventRecord(ev[3], st); }
  } else if (plan.N == 128) {
    // tiles of up to 256 rows on pairs of SMs, both GEMMs in one launch unless two are asked for
    PairParams q{};
    q.w[0] = g13.w; q.w[1] = g2.w; q.gs[0] = gs13; q.gs[1] = gs2;
    q.inter = inter; q.y = reinterpret_cast<__nv_bfloat16*>(y); q.post_norm_w = p.post_norm_w;
    q.cnt = cnt; q.off = off; q.status = status; q.trace = trace;
    q.ctr = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4096);
    q.tile_done = reinterpret_cast<unsigned int*>(b + k.tile_ctr);
    q.tile_seen = q.tile_done + max_tiles(cfg, cfg->max_tokens);
    q.K[0] = g13.K; q.K[1] = g2.K; q.n_pairs[0] = g13.n_pairs; q.n_pairs[1] = g2.n_pairs;
    q.nloc = cfg->local_count; q.H = cfg->hidden; q.I = cfg->inter;
    const bool split = form == MSK_FORM_CHAIN;
    q.first = 0; q.last = split ? 0 : 1;
    e = launch_pair(q, xs, r_max, plan.grid, st, pdl);
    if (e != 0) return e;
    if (ev) cudaEventRecord(ev[2], st);
    if (cfg->stop_after == 2) return MSK_OK;
    if (split) {
      q.first = q.last = 1;
      if (trace) q.trace = trace + TRACE_WORDS;
      e = launch_pair(q, xs, r_max, plan.grid, st, pdl);
      if (e != 0) return e;
    }
    if (ev) cudaEventRecord(ev[3], st);
    if (cfg->stop_after == 3) return MSK_OK;
  } else if (both_gemms) {
    p.route = 0; p.fold = 0; p.flat = 0;
    p.x_bf16 = static_cast<const __nv_bfloat16*>(x);
    p.T = n_tokens;
    p.grid_bar = reinterpret_cast<unsigned int*>(b + k.few_ctl + 4096);
    p.tile_done = reinterpret_cast<unsigned int*>(b + k.tile_ctr);
    p.tile_seen = p.tile_done + max_tiles(cfg, cfg->max_tokens);
    e = launch_gemm_fused(plan.N, p, plan.grid, st);
    if (e != 0) return e;
    if (ev) { cudaEventRecord(ev[2], st); cudaEventRecord(ev[3], st); }
  } else {
  // Tile hand-over: the down GEMM's CTAs start on the SMs the gate/up CTAs leave (programmatic launch) and
  // would then wait for that whole grid, whose last CTAs run a unit longer than the others (the units do not
  // divide evenly): a tenth of the gate/up time with every SM but a few idle. Instead each down unit waits
  // for the gate/up units of its own token tile, and the blocks that start last are dealt fewer down units.
  // Needs every gate/up CTA resident while down CTAs wait (grid within the SM count: a waiting CTA must not
  // keep a producing one off the machine), whole units (a cut unit would be counted once per piece) and
  // both launches of the step. Narrow token tiles only, where the gather warp does the waiting: measured at
  // H4096 I1536 E128, 16 / 32 / 64 / 128 tokens take 187 / 242 / 257 / 270 us with it against 190 / 248 /
  // 266 / 274 without. The 64-token tile shares one launch between its GEMMs.
  p.handover = (pdl != 0 && !tma_b && plan.flat == 0 && plan.grid <= sm_count() && cfg->stop_after == 0) ? 1 : 0;
  if (handover_env_off()) p.handover = 0;
  p.tile_done = reinterpret_cast<unsigned int*>(b + k.tile_ctr);
  p.tile_seen = p.tile_done + max_tiles(cfg, cfg->max_tokens);
  e = launch_gemm_n<0>(plan.N, p, plan.grid, st, pdl);
  if (e != 0) return e;
  if (ev) cudaEventRecord(ev[2], st);
  if (cfg->stop_after == 2) return MSK_OK;

  if (trace) p.trace = trace + TRACE_WORDS;
  e = launch_gemm_n<1>(plan.N, p, plan.grid, st, pdl);
  if (e != 0) return e;
  if (ev) cudaEventRecord(ev[3], st);
  if (cfg->stop_after == 3) return MSK_OK;
  }

  e = launch_combine(cfg, !nv && plan.N == 128, y, inv, topk_weights, out, n_tokens, post_norm_w != nullptr, pdl, st);
  if (ev) cudaEventRecord(ev[4], st);
  return e;
}

int msk_moe_forward(const MskMoeCfg* cfg, const void* packed13, const void* packed2, const float* gs13,
                    const float* gs2, const void* post_norm_w, const void* x, const int32_t* topk_ids,
                    const float* topk_weights, void* out, void* workspace, size_t workspace_bytes, int n_tokens,
                    void* stream) {
  return forward_impl(cfg, packed13, packed2, gs13, gs2, post_norm_w, x, topk_ids, topk_weights, out, workspace,
                      workspace_bytes, n_tokens, stream, nullptr);
}

int msk_moe_forward_logits(const MskMoeCfg* cfg, const void* packed13, const void* packed2, const float* gs13,
                           const float* gs2, const void* post_norm_w, const void* x, const float* logits,
                           const float* bias, int32_t* topk_ids_out, float* topk_weights_out, void* out,
                           void* workspace, size_t workspace_bytes, int n_tokens, void* stream) {
  if (!logits) return MSK_ERR_NULL;
  if (cfg != nullptr && cfg->top_k > cfg->n_experts) return MSK_ERR_SHAPE;
  return forward_impl(cfg, packed13, packed2, gs13, gs2, post_norm_w, x, nullptr, nullptr, out, workspace,
                      workspace_bytes, n_tokens, stream, nullptr, logits, bias, topk_ids_out, topk_weights_out);
}

int msk_moe_forward_prenorm(const MskMoeCfg* cfg, const void* packed13, const void* packed2, const float* gs13,
                            const float* gs2, const void* post_norm_w, const void* pre_norm_w, float pre_norm_eps,
                            const void* x, const float* logits, const float* bias, int32_t* topk_ids,
                            float* topk_weights, void* out, void* workspace, size_t workspace_bytes, int n_tokens,
                            void* stream) {
  if (!pre_norm_w) return MSK_ERR_NULL;
  if (!aligned16(pre_norm_w)) return MSK_ERR_ALIGN;
  if (!(pre_norm_eps > 0.f)) return MSK_ERR_SHAPE;
  if (cfg != nullptr && cfg->hidden > 8192) return MSK_ERR_TOO_LARGE;   // a row is held in registers by 256 threads
  if (logits != nullptr) {
    if (cfg != nullptr && cfg->top_k > cfg->n_experts) return MSK_ERR_SHAPE;
    return forward_impl(cfg, packed13, packed2, gs13, gs2, post_norm_w, x, nullptr, nullptr, out, workspace,
                        workspace_bytes, n_tokens, stream, nullptr, logits, bias, topk_ids, topk_weights, pre_norm_w,
                        pre_norm_eps);
  }
  return forward_impl(cfg, packed13, packed2, gs13, gs2, post_norm_w, x, topk_ids, topk_weights, out, workspace,
                      workspace_bytes, n_tokens, stream, nullptr, nullptr, nullptr, nullptr, nullptr, pre_norm_w,
                      pre_norm_eps);
}

int msk_moe_forward_timed(const MskMoeCfg* cfg, const void* packed13, const void* packed2, const float* gs13,
                          const float* gs2, const void* post_norm_w, const void* x, const int32_t* topk_ids,
                          const float* topk_weights, void* out, void* workspace, size_t workspace_bytes,
                          int n_tokens, void* stream, float* host_ms) {
  if (!host_ms) return MSK_ERR_NULL;
  static cudaEvent_t ev[64][6];
  static bool made[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MSK_ERR_RANGE;
  if (!made[dev]) {
    for (int i = 0; i < 6; ++i) {
      cudaError_t ce = cudaEventCreate(&ev[dev][i]);
      if (ce != cudaSuccess) return static_cast<int>(ce);
    }
    made[dev] = true;
  }
  const int rc = forward_impl(cfg, packed13, packed2, gs13, gs2, post_norm_w, x, topk_ids, topk_weights, out,
                              workspace, workspace_bytes, n_tokens, stream, ev[dev]);
  if (rc != 0) return rc;
  cudaError_t ce = cudaEventSynchronize(ev[dev][4]);
  if (ce != cudaSuccess) return static_cast<int>(ce);
  const int from[5] = {0, 1, 5, 2, 3}, to[5] = {1, 5, 2, 3, 4};  // sort, row copy, gate/up, down, combine
  for (int i = 0; i < 5; ++i) {
    ce = cudaEventElapsedTime(&host_ms[i], ev[dev][from[i]], ev[dev][to[i]]);
    if (ce != cudaSuccess) return static_cast<int>(ce);
  }
  return MSK_OK;
}

// ------------------------------------------------------------------------------------------
// msk_moe_forward_static: the routed-expert step for callers that cannot allocate.
// Some hosts of this library run where no device allocation may happen on the calling path:
// a serving loop that has handed all device memory to its own pool, a plug-in called while the
// application's allocator is locked, a latency-critical thread that must not enter the driver's
// allocator.
// msk_moe_forward needs a caller-allocated workspace; this variant keeps its scratch (sort
// tables, the F16 copy of the token rows, the SwiGLU intermediate and the per-route expert outputs) in one file-scope device
// array instead. The array is part of the loaded library image: every GPU that loads the
// library holds MSK_STATIC_WS_BYTES of it until the process exits.
//  * Limits: n_tokens * top_k <= 128 routed rows, hidden <= 8192, inter <= 4096; anything
//    larger is refused with MSK_ERR_TOO_LARGE. The GEMMs run on whole units here (no cut units, no pieces).
//  * The first call on each device looks up the array's device address (cudaGetSymbolAddress,
//    with that device current). Make that first call outside stream capture.
//  * All calls on a device share the one array and it keeps what the last call left; the status
//    word is cleared on the stream at the start of every call, the tables are rewritten by the
//    sort. Two calls that overlap on the GPU (different streams) race on it: serialise them.
//  * No cudaMalloc, cudaFree or allocating library call is made.
constexpr size_t MSK_STATIC_WS_BYTES = 8u << 20;
constexpr int MSK_STATIC_MAX_ROWS = 128;
static __device__ __align__(256) unsigned char g_static_ws[MSK_STATIC_WS_BYTES];

// Device address of the array on the current device, looked up once per device (in host code the
// symbol's name is a host-side stand-in, not a device address).
static int static_ws_base(unsigned char** out) {
  static unsigned char* base_of[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MSK_ERR_RANGE;
  if (base_of[dev] == nullptr) {
    void* ptr = nullptr;
    const cudaError_t ce = cudaGetSymbolAddress(&ptr, g_static_ws);
    if (ce != cudaSuccess) return static_cast<int>(ce);
    base_of[dev] = static_cast<unsigned char*>(ptr);
  }
  *out = base_of[dev];
  return 0;
}

int msk_moe_static_status(int* host_status, void* stream) {
  if (!host_status) return MSK_ERR_NULL;
  unsigned char* b = nullptr;
  const int ar = static_ws_base(&b);
  if (ar != 0) return ar;
  cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return static_cast<int>(e);
  e = cudaMemcpy(host_status, b, sizeof(int), cudaMemcpyDeviceToHost);
  return static_cast<int>(e);
}

int msk_moe_forward_static(const MskMoeCfg* cfg, const void* packed13, const void* packed2, const float* gs13,
                           const float* gs2, const void* post_norm_w, const void* x, const int32_t* topk_ids,
                           const float* topk_weights, void* out, int n_tokens, void* stream) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!packed13 || !packed2 || !gs13 || !gs2) return MSK_ERR_NULL;
  if (n_tokens < 0) return MSK_ERR_SHAPE;
  if (n_tokens == 0) return MSK_OK;
  if (!x || !topk_ids || !topk_weights || !out) return MSK_ERR_NULL;
  if (!aligned16(packed13) || !aligned16(packed2) || !aligned16(x) || !aligned16(out)) return MSK_ERR_ALIGN;
  const size_t R = static_cast<size_t>(n_tokens) * cfg->top_k;
  if (R > static_cast<size_t>(MSK_STATIC_MAX_ROWS) || cfg->hidden > 8192 || cfg->inter > 4096) return MSK_ERR_TOO_LARGE;
  // carve: [status 256][cnt][off][perm][inv][inter f16 R x I][y fp32 R x H][x as f16 T x H]
  size_t o = 256;
  const size_t o_cnt = o; o += round_up(static_cast<size_t>(cfg->local_count) * 4, 256);
  const size_t o_off = o; o += round_up(static_cast<size_t>(cfg->local_count + 1) * 4, 256);
  const size_t o_perm = o; o += round_up(R * 4, 256);
  const size_t o_inv = o; o += round_up(R * 4, 256);
  const size_t o_inter = o; o += round_up(R * cfg->inter * 2, 256);
  const size_t o_y = o; o += round_up(R * cfg->hidden * 4, 256);
  const size_t o_xh = o; o += round_up(static_cast<size_t>(n_tokens) * cfg->hidden * 2, 256);
  if (o > MSK_STATIC_WS_BYTES) return MSK_ERR_TOO_LARGE;

  unsigned char* b = nullptr;
  const int ar = static_ws_base(&b);
  if (ar != 0) return ar;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t ce = cudaMemsetAsync(b, 0, 256, st);  // status word starts at zero
  if (ce != cudaSuccess) return static_cast<int>(ce);

  int32_t* cnt = reinterpret_cast<int32_t*>(b + o_cnt);
  int32_t* off = reinterpret_cast<int32_t*>(b + o_off);
  int32_t* perm = reinterpret_cast<int32_t*>(b + o_perm);
  int32_t* inv = reinterpret_cast<int32_t*>(b + o_inv);
  __half* inter = reinterpret_cast<__half*>(b + o_inter);
  float* y = reinterpret_cast<float*>(b + o_y);
  __half* xh = reinterpret_cast<__half*>(b + o_xh);

  int e = launch_sort(cfg, topk_ids, n_tokens, cnt, off, perm, inv, st);
  if (e != 0) return e;
  copy_rows_kernel<<<static_cast<unsigned>(n_tokens), COPY_THREADS, 0, st>>>(static_cast<const __nv_bfloat16*>(x), nullptr, cfg->top_k, 0,
                                                                            cfg->hidden, xh, nullptr, 0.f);
  e = static_cast<int>(cudaGetLastError());
  if (e != 0) return e;
  GemmParams p{};
  p.cnt = cnt; p.off = off; p.perm = perm; p.inv = inv;
  p.status = reinterpret_cast<int32_t*>(b); p.trace = nullptr;
  p.nloc = cfg->local_count; p.top_k = cfg->top_k; p.evict_first = 1;
  p.flat = 0;  // whole units only: no pieces, so no partial buffer and no tickets
  p.post_norm_w = static_cast<const __nv_bfloat16*>(post_norm_w);
  const int grid = cfg->num_ctas > 0 ? std::min(cfg->num_ctas, MAX_CTAS) : DEFAULT_CTAS;
  p.ph[0].w = static_cast<const uint8_t*>(packed13); p.ph[0].gs = gs13; p.ph[0].act = xh; p.ph[0].outp = inter;
  p.ph[0].K = cfg->hidden; p.ph[0].out_ld = cfg->inter; p.ph[0].n_pairs = cfg->inter / 128;
  p.ph[1].w = static_cast<const uint8_t*>(packed2); p.ph[1].gs = gs2; p.ph[1].act = inter; p.ph[1].outp = y;
  p.ph[1].K = cfg->inter; p.ph[1].out_ld = cfg->hidden; p.ph[1].n_pairs = cfg->hidden / 256;
  e = launch_gemm_n<0>(16, p, grid, st, 1);
  if (e != 0) return e;
  e = launch_gemm_n<1>(16, p, grid, st, 1);
  if (e != 0) return e;
  return launch_combine(cfg, false, y, inv, topk_weights, out, n_tokens, post_norm_w != nullptr, 0, st);
}

int msk_moe_share_pieces(int n_base, int n_stages, int shares, int flat, int cta, int heavy, int skip, int* host_out,
                         int capacity, int* host_count) {
  if (!host_out || !host_count) return MSK_ERR_NULL;
  if (n_base < 0 || n_stages < 1 || shares < 1 || cta < 0 || cta >= shares || capacity < 0 || heavy < 0 || heavy >= shares ||
      skip < 0)
    return MSK_ERR_SHAPE;
  if (static_cast<long long>(n_base) * n_stages * shares >= FLAT_MAX_PRODUCT) return MSK_ERR_TOO_LARGE;
  PieceIter it = make_piece_iter(flat, n_base, n_stages, cta, shares, heavy, skip);
  const int items = (n_base - it.tail_base) * n_stages;
  int n = 0, base, ks0, ks1;
  while (it.next(base, ks0, ks1)) {
    if (n < capacity) {
      int* o = host_out + 6 * n;
      const bool whole = ks0 == 0 && ks1 == n_stages;
      const int b0 = (base - it.tail_base) * n_stages;
      o[0] = base; o[1] = ks0; o[2] = ks1;
      o[3] = whole ? -1 : piece_slot(cta, ks0 == 0);
      o[4] = whole ? cta : share_owner(items, shares, b0);
      o[5] = whole ? cta : share_owner(items, shares, b0 + n_stages - 1);
    }
    ++n;
  }
  *host_count = n;
  return n <= capacity ? MSK_OK : MSK_ERR_TOO_LARGE;
}

// L2 sweep for cold-cache timing: every thread reads 16-byte words of the buffer with ordinary loads,
// so the lines land in L2 clean and displace what was there. (Zeroing a buffer also displaces it, but
// leaves L2 full of dirty lines whose write-back then competes with the kernel being timed; the
// reference sweeps by reading for the same reason, muse_decode_layer/py/05_tune.py:74-94.)
__global__ void __launch_bounds__(256) l2_sweep_kernel(const uint4* __restrict__ buf, size_t n16, uint32_t* sink) {
  uint32_t acc = 0;
  for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < n16; i += static_cast<size_t>(gridDim.x) * 256) {
    const uint4 v = buf[i];
    acc ^= v.x ^ v.y ^ v.z ^ v.w;
  }
  if (acc == 0x9E3779B9u) atomicAdd(sink, acc);  // keeps the loads alive
}

int msk_l2_sweep(const void* buf, size_t bytes, uint32_t* sink, void* stream) {
  if (!buf || !sink) return MSK_ERR_NULL;
  if (!aligned16(buf)) return MSK_ERR_ALIGN;
  if (bytes < 16) return MSK_OK;
  l2_sweep_kernel<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint4*>(buf), bytes / 16, sink);
  return static_cast<int>(cudaGetLastError());
}

#ifndef MSK_BUILD_ID
#define MSK_BUILD_ID "unknown"
#endif
const char* msk_build_id(void) { return MSK_BUILD_ID; }

int msk_moe_few_fits(const MskMoeCfg* cfg, int n_tokens, int inputs, int* host_fits) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!host_fits) return MSK_ERR_NULL;
  if (n_tokens < 1) return MSK_ERR_SHAPE;
  FewPlan f;
  const Plan p = make_plan(cfg, n_tokens);
  *host_fits = p.path == 0 && few_takes(cfg, n_tokens, inputs, p.grid, &f) ? 1 : 0;
  return MSK_OK;
}

int msk_moe_nvf4_takes(const MskMoeCfg* cfg, int n_tokens, int norms, int* host_takes) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!host_takes) return MSK_ERR_NULL;
  if (n_tokens < 1) return MSK_ERR_SHAPE;
  *host_takes = nv_takes(cfg, n_tokens, make_plan(cfg, n_tokens), norms) ? 1 : 0;
  return MSK_OK;
}

int msk_moe_step_form(const MskMoeCfg* cfg, int n_tokens, int inputs, int* host_form) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!host_form) return MSK_ERR_NULL;
  if (n_tokens < 1) return MSK_ERR_SHAPE;
  FewPlan f;
  *host_form = step_form(cfg, n_tokens, make_plan(cfg, n_tokens), inputs, true, &f);
  return MSK_OK;
}

int msk_moe_plan(const MskMoeCfg* cfg, int n_tokens, int* host_out) {
  const int rc = check_cfg(cfg);
  if (rc != MSK_OK) return rc;
  if (!host_out) return MSK_ERR_NULL;
  if (n_tokens < 1) return MSK_ERR_SHAPE;
  const Plan plan = make_plan(cfg, n_tokens);
  host_out[0] = plan.N; host_out[1] = plan.path; host_out[2] = plan.flat; host_out[3] = plan.grid;
  return MSK_OK;
}

int msk_moe_read_status(const void* workspace, int* host_status, void* stream) {
  if (!workspace || !host_status) return MSK_ERR_NULL;
  cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return static_cast<int>(e);
  e = cudaMemcpy(host_status, workspace, sizeof(int), cudaMemcpyDeviceToHost);
  return static_cast<int>(e);
}

int msk_moe_attrs(int which, int token_tile, int* host_out) {
  if (!host_out) return MSK_ERR_NULL;
  cudaFuncAttributes a{};
  cudaError_t e = cudaSuccess;
  switch (which) {
    case 0: e = cudaFuncGetAttributes(&a, sort_kernel); break;
    case 1: e = cudaFuncGetAttributes(&a, route_topk_kernel); break;
    case 2:
    case 3: {
      const bool ph1 = which == 3;
      switch (token_tile) {
        case 16: e = ph1 ? cudaFuncGetAttributes(&a, moe_gemm_kernel<16, 1>) : cudaFuncGetAttributes(&a, moe_gemm_kernel<16, 0>); break;
        case 32: e = ph1 ? cudaFuncGetAttributes(&a, moe_gemm_kernel<32, 1>) : cudaFuncGetAttributes(&a, moe_gemm_kernel<32, 0>); break;
        case 64: e = ph1 ? cudaFuncGetAttributes(&a, moe_gemm_kernel<64, 1>) : cudaFuncGetAttributes(&a, moe_gemm_kernel<64, 0>); break;
        case 128: e = cudaFuncGetAttributes(&a, moe_pair_kernel); break;   // both GEMMs
        default: return MSK_ERR_SHAPE;
      }
      break;
    }
    case 4: e = cudaFuncGetAttributes(&a, combine_norm_kernel<false, 512, 1, 8, 1>); break;
    default: return MSK_ERR_SHAPE;
  }
  if (e != cudaSuccess) return static_cast<int>(e);
  host_out[0] = a.numRegs;
  host_out[1] = static_cast<int>(a.sharedSizeBytes);
  host_out[2] = a.maxDynamicSharedSizeBytes;
  host_out[3] = static_cast<int>(a.localSizeBytes);
  return MSK_OK;
}

int msk_ep_combine(const void* back, const void* self_rows, int self_rank, const int32_t* ids, int top_k,
                   int experts_per_rank, void* out, int n_ranks, int n_tokens, int hidden, void* stream) {
  if (!back || !ids || !out) return MSK_ERR_NULL;
  if (n_ranks < 1 || n_ranks > 64 || n_tokens < 0 || hidden < 8 || hidden % 8 != 0 || top_k < 1 ||
      top_k > MAX_TOP_K || experts_per_rank < 1)
    return MSK_ERR_SHAPE;
  if (!aligned16(back) || !aligned16(out) || (self_rows && !aligned16(self_rows))) return MSK_ERR_ALIGN;
  if (n_tokens == 0) return MSK_OK;
  ep_combine_kernel<<<static_cast<unsigned>(n_tokens), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(back), static_cast<const __nv_bfloat16*>(self_rows), self_rank, ids, top_k,
      experts_per_rank, static_cast<__nv_bfloat16*>(out), n_ranks, n_tokens, hidden);
  return static_cast<int>(cudaGetLastError());
}

int msk_ep_flag_write(void* addr, uint32_t value, void* stream) {
  if (!addr) return MSK_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(addr) % 4 != 0) return MSK_ERR_ALIGN;
  return stream_value32("cuStreamWriteValue32", addr, value, CU_STREAM_WRITE_VALUE_DEFAULT, stream);
}

int msk_ep_flag_wait(void* addr, uint32_t value, void* stream) {
  if (!addr) return MSK_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(addr) % 4 != 0) return MSK_ERR_ALIGN;
  return stream_value32("cuStreamWaitValue32", addr, value, CU_STREAM_WAIT_VALUE_GEQ, stream);
}

int msk_bw_probe(const void* src, size_t bytes, int stages, int stage_bytes, int num_ctas, uint32_t* sink,
                 int skip_release, void* stream) {
  if (!src || !sink) return MSK_ERR_NULL;
  if (!aligned16(src)) return MSK_ERR_ALIGN;
  if (stages < 1 || stages > 8 || stage_bytes < 16 || stage_bytes % 16 != 0) return MSK_ERR_SHAPE;
  const size_t smem = static_cast<size_t>(stages) * stage_bytes;
  if (smem > 220 * 1024) return MSK_ERR_TOO_LARGE;
  const int grid = num_ctas > 0 ? num_ctas : sm_count();
  cudaError_t e = cudaFuncSetAttribute(bw_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return static_cast<int>(e);
  bw_probe_kernel<<<grid, 64, smem, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(src), static_cast<unsigned long long>(bytes), stages, stage_bytes, sink, skip_release);
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
