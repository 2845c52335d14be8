// The batched Q1_0 x Q8_0 product of matmul_q1_0_q8_0.wgsl:57-293 on the 5th-generation tensor cores, and the
// quantiser (quantize_q8_0.wgsl:49-106) that leaves the activations as the tensor cores read them.
//
// y[m][n] (+)= sum over sub-blocks of 32 inputs, in ascending order, of (a_d * w_d) * f32(sumi), every product
// and sum rounded once. The integer dots are exact whoever computes them; the three roundings per output and
// sub-block are what has to stay on the CUDA cores. So the kernel is built around those three operations:
//   - sumi arrives in TMEM as FP32 (kind::f8f6f4): no conversion. An int8 quant q is two e4m3 values,
//     16 * rint(q / 16) and the remainder in [-8, 8], both exact; weights are +-1; every partial sum is an
//     integer below 2^13, exact in the FP32 accumulator in any order. Two MMAs of 32 inputs per sub-block
//     instead of two f16 MMAs of 16, at the same tensor time, and a weight costs one byte of shared memory;
//   - the three operations are packed FP32 pairs, 1.5 instructions per output. The sum is an FMA with a factor
//     of one that the compiler cannot see (a packed product consumed by a packed add was seen to be contracted,
//     which changes the bits);
//   - the sign bits of a sub-block are one 32-bit word w, and word g of its 32 bytes is (w << g) & 0x80808080
//     xor 0xB8B8B8B8 (e4m3 +-1): two instructions per four weights. That puts input 8 j + 7 - g of a sub-block
//     at byte 4 g + j, and the quantiser writes the activations in the same order.
#include <cuda_fp16.h>

#include "bp_common.cuh"
#include "bp_ptx.cuh"
#include "bp_q1_device.cuh"
#include "bp_q1_ops.cuh"

namespace {

using namespace bp;

constexpr uint32_t TT_M = 128;                    // tokens of a tile = TMEM lanes
constexpr uint32_t TT_PART = TT_M * 128;          // one part (16 rint(q / 16), or the remainder) of a tile's block of 128 inputs
constexpr uint32_t TT_WORKERS = 16;               // worker warps: 4 quarters of the TMEM lanes x 4 groups of columns
constexpr uint32_t TT_THREADS = (1 + TT_WORKERS) * 32;
constexpr uint32_t TT_STAGES = 4;

// ---- activations -------------------------------------------------------------------------------------------
// Tiled activations of a batch: per tile of 128 tokens and block of 128 inputs, 2 x 16 KB: part 0 and part 1 as
// [128 tokens][128 bytes], a token's 16-byte chunks xor-ed with (token mod 8): the layout the MMA reads
// (K-major, 128-byte swizzle), so a stage is ONE bulk copy. Scales: [tile][block][128 tokens][4 sub-blocks].
enum { SRC_PLAIN = 0, SRC_RMS = 1, SRC_SILU = 2 };

// quantize_q8_0.wgsl after nothing, after rms_norm.wgsl:41-85, or after silu_mul.wgsl:18-27: the producing
// operator's f16 results go straight into the quantiser. One CTA per token, 512 threads (the norm's
// invocation count: its sum is per invocation). Four lanes share a sub-block: lane t takes the inputs of output
// words 2 t and 2 t + 1, which are the pairs 8 j + 6 - 2 t, 8 j + 7 - 2 t.
template <int SRC>
__global__ void __launch_bounds__(512) quantize_tiled_kernel(const __half* x, const __half* aux, uint32_t k, float eps, uint8_t* a_t, float* a_d) {
  __shared__ float part[32];
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t row = blockIdx.x, tid = threadIdx.x, nb1 = k / 128u;
  const __half* src = x + static_cast<size_t>(row) * k;
  __half2 inv2 = __float2half2_rn(0.0f);
  if (SRC == SRC_RMS) {
    float s = 0.0f;
    for (uint32_t i = tid; i < k; i += 512) {
      const float v = __half2float(src[i]);
      s = __fadd_rn(s, __fmul_rn(v, v));
    }
    const float total = workgroup_sum<16>(s, part);
    inv2 = __half2half2(__float2half_rn(__frsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(k)), eps))));
  }
  const uint32_t r = row % TT_M, t = tid & 3u;
  const size_t tile0 = static_cast<size_t>(row / TT_M) * nb1;
  for (uint32_t u = tid; u < k / 8u; u += 512) {  // (k / 8 is a multiple of 16: the four lanes of a sub-block stay together)
    const uint32_t sub = u >> 2;
    float v[8];
    float amax = 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
      const uint32_t e = 32u * sub + 8u * j + 6u - 2u * t;
      __half2 h = *reinterpret_cast<const __half2*>(src + e);
      if (SRC == SRC_RMS) h = __hmul2(__hmul2(h, inv2), *reinterpret_cast<const __half2*>(aux + e));
      if (SRC == SRC_SILU) {
        const __half2 up = *reinterpret_cast<const __half2*>(aux + static_cast<size_t>(row) * k + e);
        h = __halves2half2(silu_times_up(__low2half(h), __low2half(up)), silu_times_up(__high2half(h), __high2half(up)));
      }
      v[j] = __high2float(h);      // word 2 t, byte j
      v[4 + j] = __low2float(h);   // word 2 t + 1, byte j
      amax = fmaxf(amax, fmaxf(fabsf(v[j]), fabsf(v[4 + j])));
    }
    const unsigned group = 0xFu << (tid & 28u);
    amax = fmaxf(amax, __shfl_xor_sync(group, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(group, amax, 2));
    const float d = __fdiv_rn(amax, 127.0f);
    const float id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    uint32_t hi[2], lo[2];
#pragma unroll
    for (int w = 0; w < 2; w++) {
      float h16[4], rem[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float q = fminf(fmaxf(rintf(__fmul_rn(v[4 * w + j], id)), -127.0f), 127.0f);
        h16[j] = 16.0f * rintf(q * 0.0625f);
        rem[j] = q - h16[j];
      }
      uint16_t b01, b23;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(b01) : "f"(h16[1]), "f"(h16[0]));
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(b23) : "f"(h16[3]), "f"(h16[2]));
      hi[w] = b01 | (static_cast<uint32_t>(b23) << 16);
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(b01) : "f"(rem[1]), "f"(rem[0]));
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(b23) : "f"(rem[3]), "f"(rem[2]));
      lo[w] = b01 | (static_cast<uint32_t>(b23) << 16);
    }
    const uint32_t kb = sub >> 2, s = sub & 3u;
    uint8_t* dst = a_t + (tile0 + kb) * (2u * TT_PART) + r * 128u + (((2u * s + (t >> 1)) ^ (r & 7u)) << 4) + 8u * (t & 1u);
    *reinterpret_cast<uint2*>(dst) = make_uint2(hi[0], hi[1]);
    *reinterpret_cast<uint2*>(dst + TT_PART) = make_uint2(lo[0], lo[1]);
    if (t == 0) a_d[((tile0 + kb) * TT_M + r) * 4u + s] = d;
  }
}

// ---- product -----------------------------------------------------------------------------------------------
struct TiledTensors {  // up to three weight tensors over the same activations: column tile blockIdx.x belongs to one of them
  const __half* w_d[3];
  const uint8_t* w_qs[3];
  __half* y[3];
  uint32_t n[3];
  uint32_t tile_end[3];  // running total of column tiles
};

__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// 16-byte aligned global -> shared copy of a multiple of 16 bytes, completion on an mbarrier
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
template <uint32_t W>
__device__ __forceinline__ void tmem_ld_w(uint32_t taddr, uint32_t (&r)[16]) {
  static_assert(W == 8 || W == 12 || W == 16, "widths of a load");
  if constexpr (W == 16) {
    tmem_ld16(taddr, r);
  } else {
    tmem_ld8(taddr, reinterpret_cast<uint32_t(&)[8]>(r));
    if constexpr (W == 12) tmem_ld4(taddr + 8, r + 8);
  }
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}

// A CTA owns 128 tokens x 4 NC weight rows and runs alone on its SM.
//   worker warps      stage a block of 128 inputs two blocks ahead (thread = one sub-block of one weight row: a word
//                     of signs -> 32 bytes; one thread requests the activations), then take finished sub-blocks out
//                     of TMEM: thread = token = TMEM lane, NC weight rows, sums in registers over all blocks
//   warp 0, lane 0    issues the MMAs, G sub-blocks per hand-over, into one of two sets of G TMEM buffers
// What bounds it (128 x 112 tile, cycles per sub-block, stamps in the kernel): 855, of them 510 the scaling and adding
// (336 if only the FMA pipe counted), 220 the staging (its proxy fence above all), 120 waiting for the MMAs; the
// tensor pipe is 13 % busy, the issue slots 58 % (gate + up of 512 tokens under ncu). A pass of 512 tokens at the Bonsai-8B shape: 37.9 ms with the
// mma.sync kernel, 29.2 now; 21 tokens: 53 ms with the CUDA-core kernel, 11.8 now. Slower (ms per 512-token pass): four
// sets of one sub-block 32.6, the staging in four warps of its own 30.4, two issuing threads with the next
// hand-over's first load before the last piece is added 30.8, scalar instead of packed sums and products: no change.
// Every wait is bounded; a wait that gives up stores a code in the error word and the CTA winds down: it ends only
// when its own copies have landed and its own MMAs are complete (waits of TT_DRAIN polls, whatever the caller's limit:
// what is waited for there always comes), because the next CTA on the SM gets the same shared memory and TMEM.
constexpr uint32_t TT_DRAIN = 1u << 20;
template <uint32_t NC>
__global__ void __launch_bounds__(TT_THREADS, 1) matmul_q1_tiled_kernel(const TiledTensors tensors, uint32_t k, uint32_t m, const uint8_t* __restrict__ a_t,
                                                                        const float* __restrict__ a_d, uint32_t accumulate, float one, uint32_t* err,
                                                                        uint32_t wait_limit, uint32_t poll_ns) {
  constexpr uint32_t N = 4 * NC, STAGE_B = 2 * TT_PART + N * 128;
  constexpr uint32_t G = NC > 16 ? 2 : 4, STEPS = 4 / G;      // sub-blocks per hand-over, hand-overs per block
  constexpr uint32_t BUFS = 2;                                                             // sets of G TMEM buffers
  constexpr uint32_t COLS = N > 64 ? 128 : N;                 // TMEM columns of one buffer
  constexpr uint32_t W0 = NC < 16 ? NC : 16, W1 = NC - W0, PIECES = W1 != 0 ? 2 : 1;  // columns of a TMEM load
  static_assert(BUFS * G * COLS <= 512, "TMEM has 512 columns");
  extern __shared__ uint8_t tt_raw[];
  __shared__ __align__(8) uint64_t full[TT_STAGES], a_full[TT_STAGES], empty[TT_STAGES], d_full[BUFS], d_empty[BUFS], drained;
  __shared__ __align__(16) float s_wd[TT_WORKERS][2][32];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile uint32_t abort_s;
  const uint32_t smem_base = (smem_u32(tt_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = tt_raw + (smem_base - smem_u32(tt_raw));
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t tile = blockIdx.x;
  const uint32_t which = tile < tensors.tile_end[0] ? 0u : tile < tensors.tile_end[1] ? 1u : 2u;
  // (selects: an indexed parameter array would be copied to local memory)
  auto pick = [&](const auto* v) { return which == 0 ? v[0] : which == 1 ? v[1] : v[2]; };
  const uint32_t n = pick(tensors.n);
  const uint32_t n_base = (tile - (which == 0 ? 0u : which == 1 ? tensors.tile_end[0] : tensors.tile_end[1])) * N, m_base = blockIdx.y * TT_M;
  const uint32_t nb1 = k / 128u;
  if (tid == 0) {
    for (uint32_t i = 0; i < TT_STAGES; i++) {
      mbar_init(smem_u32(&full[i]), TT_WORKERS);
      mbar_init(smem_u32(&a_full[i]), 1);
      mbar_init(smem_u32(&empty[i]), 1);
    }
    for (uint32_t i = 0; i < BUFS; i++) {
      mbar_init(smem_u32(&d_full[i]), 1);
      mbar_init(smem_u32(&d_empty[i]), TT_WORKERS);
    }
    mbar_init(smem_u32(&drained), 1);
    abort_s = 0;
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(smem_u32(&tmem_base_s), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  if (tid == 0) pdl_launch_dependents();
  // A wait that gives up, or finds that another one has, leaves its thread `dead`: the thread runs through the rest of
  // its loop without waiting, copying or writing results. (The flag is a register: a look at abort_s before every wait
  // and every MMA lengthened the chain from hand-over to hand-over by 7 % of the kernel.)
  bool dead = false;
  auto waitb = [&](uint64_t* bar, uint32_t parity, uint32_t ns = 2000u) {  // ns: how long a poll may suspend its thread
    if (dead) return;
    const uint32_t addr = smem_u32(bar);
    for (uint32_t i = 0; i < wait_limit; i++) {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(addr), "r"(parity), "r"(ns)
          : "memory");
      if (ok) return;
      if (abort_s) {
        dead = true;
        return;
      }
    }
    dead = true;
    abort_s = 1;
    atomicExch(err, 6u);
  };

  if (warp == 0) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t IDESC = umma_idesc(1, 0, 0, 0, 0, TT_M, N);  // f32 = e4m3 (K-major) x e4m3 (K-major)
      const uint64_t dk = umma_desc_sw128(0, 16, 1024);
      pdl_wait();  // the polls below count from here: the time of the kernel before this one is not theirs
      for (uint32_t b = 0; b < nb1; b++) {
        const uint32_t slot = b % TT_STAGES;
        waitb(&a_full[slot], (b / TT_STAGES) & 1u, poll_ns);
        waitb(&full[slot], (b / TT_STAGES) & 1u);
        const uint64_t ad = dk + ((smem_base + slot * STAGE_B) >> 4), bd = ad + (2u * TT_PART >> 4);
#pragma unroll
        for (uint32_t h = 0; h < STEPS; h++) {
          const uint32_t j = b * STEPS + h, pb = j % BUFS;
          if (j >= BUFS) waitb(&d_empty[pb], (j / BUFS - 1u) & 1u);
          if (dead) break;
          tc_fence_after();
#pragma unroll
          for (uint32_t g = 0; g < G; g++)
#pragma unroll
            for (uint32_t part = 0; part < 2; part++)  // a sub-block: 32 bytes along the row
              umma_f8(tmem + (pb * G + g) * COLS, ad + part * (TT_PART >> 4) + (h * G + g) * 2u, bd + (h * G + g) * 2u, IDESC, part);
          umma_commit(smem_u32(&d_full[pb]));
        }
        if (dead) break;  // no slot is given back any more: a copy into it could meet the previous one
        umma_commit(smem_u32(&empty[slot]));
      }
    }
  } else {
    // ---------------- workers ----------------
    const __half* __restrict__ w_d = pick(tensors.w_d);
    const uint8_t* __restrict__ w_qs = pick(tensors.w_qs);
    const uint32_t wt = tid - 32u, srow = wt >> 2, ssub = wt & 3u;  // staging: sub-block ssub of weight row srow
    const bool b_stage = srow < N, b_ok = b_stage && n_base + srow < n;
    const uint8_t* b_src = w_qs + static_cast<size_t>(n_base + srow) * nb1 * 16u + 4u * ssub;
    const uint8_t* a_src = a_t + static_cast<size_t>(blockIdx.y) * nb1 * (2u * TT_PART);
    uint32_t rb = 0, rb2 = 0;  // the signs of the block to be staged next, and of the one after it
    uint32_t copies = 0;       // blocks of activations requested (one thread)
    auto fetch = [&](uint32_t b) {
      rb = rb2;
      rb2 = b_ok && b < nb1 ? __ldg(reinterpret_cast<const uint32_t*>(b_src + 16u * b)) : 0u;
    };
    auto store = [&](uint32_t b) {
      const uint32_t slot = b % TT_STAGES;
      if (b >= TT_STAGES) waitb(&empty[slot], ((b / TT_STAGES) - 1u) & 1u);
      if (wt == 0 && !dead) {
        mbar_arrive_expect_tx(smem_u32(&a_full[slot]), 2u * TT_PART);
        bulk_load(smem_base + slot * STAGE_B, a_src + static_cast<size_t>(b) * (2u * TT_PART), 2u * TT_PART, smem_u32(&a_full[slot]));
        copies = b + 1;
      }
      if (b_stage) {
        uint8_t* brow = smem_gen + slot * STAGE_B + 2u * TT_PART + srow * 128u;
        uint32_t o[8];
#pragma unroll
        for (uint32_t g = 0; g < 8; g++) o[g] = ((rb << g) & 0x80808080u) ^ 0xB8B8B8B8u;  // bit set: +1 (0x38), clear: -1 (0xB8)
        *reinterpret_cast<uint4*>(brow + (((2u * ssub) ^ (srow & 7u)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(brow + (((2u * ssub + 1u) ^ (srow & 7u)) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full[slot]));
    };
    const uint32_t quad = warp & 3u, ew = warp - 1u, cg = ew >> 2;  // TMEM lane quarter; columns NC cg ..
    const uint32_t row = quad * 32u + lane, mi = m_base + row;
    const uint32_t t_addr = tmem + ((quad * 32u) << 16) + cg * NC;
    const bool row_ok = mi < m;
    const uint32_t my_col = n_base + cg * NC + lane;  // the weight row whose scale this lane fetches for its warp
    const bool col_ok = lane < NC && my_col < n;
    const float4* ad_src = reinterpret_cast<const float4*>(a_d) + static_cast<size_t>(blockIdx.y) * nb1 * TT_M + row;
    const __half* wd_src = w_d + static_cast<size_t>(my_col) * nb1;
    unsigned long long acc[NC / 2];
#pragma unroll
    for (uint32_t c = 0; c < NC / 2; c++) acc[c] = 0ull;
    const unsigned long long ones = pack2(one, one);
    // fetch(b) requests block b and makes block b - 1, requested one call earlier, the one that store() writes. The
    // weights are constants: the first ones are requested before the kernel waits for its predecessor.
    fetch(0);
    fetch(1);
    float wd_next = col_ok ? __half2float(wd_src[0]) : 0.0f;
    pdl_wait();
    float4 ad_next = row_ok ? *ad_src : make_float4(0.f, 0.f, 0.f, 0.f);
    store(0);
    fetch(2);
    if (nb1 > 1) store(1);
    fetch(3);
    uint32_t d[2][16];
    for (uint32_t b = 0; b < nb1; b++) {
      if (b + 2 < nb1) {
        store(b + 2);
        fetch(b + 4);
      }
      const float adv[4] = {ad_next.x, ad_next.y, ad_next.z, ad_next.w};
      float* wd_s = s_wd[ew][b & 1u];
      wd_s[lane] = wd_next;
      __syncwarp();
      if (b + 1 < nb1) {
        if (row_ok) ad_next = ad_src[static_cast<size_t>(b + 1u) * TT_M];
        if (col_ok) wd_next = __half2float(wd_src[b + 1u]);
      }
#pragma unroll
      for (uint32_t h = 0; h < STEPS; h++) {
        const uint32_t j = b * STEPS + h, pb = j % BUFS;
        waitb(&d_full[pb], (j / BUFS) & 1u);
        tc_fence_after();
        // the pieces of the G sub-blocks, each load in flight while the previous piece is scaled and added
        tmem_ld_w<W0>(t_addr + pb * G * COLS, d[0]);
#pragma unroll
        for (uint32_t q = 0; q < G * PIECES; q++) {
          const uint32_t g = q / PIECES, piece = q % PIECES;
          tmem_ld_wait();
          if (q + 1 < G * PIECES) {
            const uint32_t at = t_addr + (pb * G + (q + 1) / PIECES) * COLS;
            if ((q + 1) % PIECES == 0) {
              tmem_ld_w<W0>(at, d[(q + 1) & 1u]);
            } else if constexpr (W1 != 0) {
              tmem_ld_w<W1>(at + W0, d[(q + 1) & 1u]);
            }
          } else {  // the whole hand-over is in registers: its buffers may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&d_empty[pb]));
          }
          const float ad_s = adv[h * G + g];
          const unsigned long long ad2 = pack2(ad_s, ad_s);
          const uint32_t c0 = piece * W0, width = piece == 0 ? W0 : W1;
#pragma unroll
          for (uint32_t c = 0; c < width; c += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(wd_s + c0 + c);
            const uint32_t* dq = d[q & 1u] + c;
            const unsigned long long q01 = mul2(mul2(ad2, pack2(w4.x, w4.y)), pack2(__uint_as_float(dq[0]), __uint_as_float(dq[1])));
            const unsigned long long q23 = mul2(mul2(ad2, pack2(w4.z, w4.w)), pack2(__uint_as_float(dq[2]), __uint_as_float(dq[3])));
            acc[(c0 + c) / 2] = fma2(q01, ones, acc[(c0 + c) / 2]);
            acc[(c0 + c) / 2 + 1] = fma2(q23, ones, acc[(c0 + c) / 2 + 1]);
          }
        }
      }
    }
    // no copy may still be on its way when the CTA ends (all have landed unless a wait gave up)
    if (wt == 0)
      for (uint32_t b = copies > TT_STAGES ? copies - TT_STAGES : 0; b < copies; b++) (void)mbar_wait(smem_u32(&a_full[b % TT_STAGES]), (b / TT_STAGES) & 1u, TT_DRAIN);
    __syncwarp();
    if (row_ok && !dead) {
      __half* y = pick(tensors.y);
      __half* dst = y + static_cast<size_t>(mi) * n + n_base + cg * NC;
      const bool vec = n % 4u == 0 && reinterpret_cast<uintptr_t>(y) % 8u == 0;
#pragma unroll
      for (uint32_t c = 0; c < NC; c += 4) {
        float v[4];
        unpack2(acc[c / 2], v[0], v[1]);
        unpack2(acc[c / 2 + 1], v[2], v[3]);
        const uint32_t col = n_base + cg * NC + c;
        if (vec) {
          if (col >= n) break;
          __half o[4];
          uint2 raw = make_uint2(0, 0);
          if (accumulate) raw = *reinterpret_cast<const uint2*>(dst + c);
          const __half* old = reinterpret_cast<const __half*>(&raw);
#pragma unroll
          for (int e = 0; e < 4; e++) o[e] = __float2half_rn(accumulate ? __fadd_rn(__half2float(old[e]), v[e]) : v[e]);
          *reinterpret_cast<uint2*>(dst + c) = *reinterpret_cast<const uint2*>(o);
        } else {
#pragma unroll
          for (uint32_t e = 0; e < 4; e++)
            if (col + e < n) dst[c + e] = __float2half_rn(accumulate ? __fadd_rn(__half2float(dst[c + e]), v[e]) : v[e]);
        }
      }
    }
  }
  __syncwarp();  // the lanes of the one-thread roles meet again
  tc_fence_before();
  __syncthreads();
  if (abort_s) {  // the workers have not seen the last MMAs complete
    if (tid == 0) {  // (the thread that issued them)
      umma_commit(smem_u32(&drained));
      (void)mbar_wait(smem_u32(&drained), 0, TT_DRAIN);
    }
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <uint32_t NC>
constexpr uint32_t tt_smem() { return TT_STAGES * (2 * TT_PART + 4 * NC * 128) + 1024; }

template <uint32_t NC>
cudaError_t launch_tiled(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* y, uint32_t n_w, uint32_t m, const uint8_t* a_t,
                         const float* a_d, bool accumulate, uint32_t* err, uint32_t wait_limit) {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    e = cudaFuncSetAttribute(matmul_q1_tiled_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(tt_smem<NC>()));
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  TiledTensors t;
  uint32_t tiles = 0;
  for (uint32_t i = 0; i < 3; i++) {
    const uint32_t j = i < n_w ? i : n_w - 1;  // unused entries repeat the last tensor; their tile range is empty
    t.w_d[i] = w[j].d;
    t.w_qs[i] = w[j].qs;
    t.y[i] = y[j];
    t.n[i] = w[j].n;
    if (i < n_w) tiles += (w[i].n + 4 * NC - 1) / (4 * NC);
    t.tile_end[i] = tiles;
  }
  // (a limit of a few polls is short in time too: the MMA issuer's polls for a copy suspend it for as many ns at most)
  return bp_launch(pdl, matmul_q1_tiled_kernel<NC>, dim3(tiles, (m + TT_M - 1) / TT_M), dim3(TT_THREADS), tt_smem<NC>(), s, t, w[0].k, m, a_t, a_d,
                   accumulate ? 1u : 0u, 1.0f, err, wait_limit, wait_limit < 2000u ? wait_limit : 2000u);
}

}  // namespace

size_t bp_q1_tiled_bytes(uint32_t m, uint32_t k) { return static_cast<size_t>((m + TT_M - 1) / TT_M) * (k / 128u) * 2u * TT_PART; }
size_t bp_q1_tiled_scales(uint32_t m, uint32_t k) { return static_cast<size_t>((m + TT_M - 1) / TT_M) * (k / 128u) * TT_M * 4u; }

cudaError_t bp_q1_quantize_tiled(bool pdl, cudaStream_t s, const __half* x, uint32_t k, uint32_t m, uint8_t* a_t, float* a_d) {
  return bp_launch(pdl, quantize_tiled_kernel<SRC_PLAIN>, dim3(m), dim3(512), 0, s, x, x, k, 0.0f, a_t, a_d);
}
cudaError_t bp_q1_rms_quantize_tiled(bool pdl, cudaStream_t s, const __half* x, const __half* w, float eps, uint32_t k, uint32_t m, uint8_t* a_t, float* a_d) {
  return bp_launch(pdl, quantize_tiled_kernel<SRC_RMS>, dim3(m), dim3(512), 0, s, x, w, k, eps, a_t, a_d);
}
cudaError_t bp_q1_silu_quantize_tiled(bool pdl, cudaStream_t s, const __half* gate, const __half* up, uint32_t k, uint32_t m, uint8_t* a_t, float* a_d) {
  return bp_launch(pdl, quantize_tiled_kernel<SRC_SILU>, dim3(m), dim3(512), 0, s, gate, up, k, 0.0f, a_t, a_d);
}

cudaError_t bp_q1_matmul_tiled(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* y, uint32_t n_w, uint32_t m, const uint8_t* a_t,
                               const float* a_d, bool accumulate, uint32_t* err, uint32_t wait_limit) {
  if (n_w == 0 || n_w > 3) return cudaErrorInvalidValue;
  const uint32_t sms = bp_q1_sm_count();
  // The width of a tile: waves of one CTA per SM, times what a block of a tile of that width takes: us, 512 tokens through
  // the 8B shape's tensors, 96 blocks (down) to 32 (Q/K/V): 2.11 - 2.28, 1.79 - 1.96, 1.58 - 1.71, 1.23 - 1.36, 1.14 - 1.21.
  // The choice was the fastest of the five widths for Q/K/V, Wo, gate + up and down at 21, 128, 173, 300 and 512 tokens.
  const uint32_t widths[5] = {32, 28, 24, 16, 8};
  const float cost[5] = {2.15f, 1.79f, 1.66f, 1.34f, 1.17f};
  float best = 1e30f;
  uint32_t nc = 32;
  for (int c = 0; c < 5; c++) {
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < n_w; i++) tiles += (w[i].n + 4 * widths[c] - 1) / (4 * widths[c]);
    const uint32_t ctas = tiles * ((m + TT_M - 1) / TT_M);
    const float t = cost[c] * static_cast<float>((ctas + sms - 1) / sms);
    if (t < best) {
      best = t;
      nc = widths[c];
    }
  }
  if (bp_q1_tile_width() != 0) nc = bp_q1_tile_width() / 4;
  switch (nc) {
    case 32: return launch_tiled<32>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 28: return launch_tiled<28>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 24: return launch_tiled<24>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 16: return launch_tiled<16>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    default: return launch_tiled<8>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
  }
}
