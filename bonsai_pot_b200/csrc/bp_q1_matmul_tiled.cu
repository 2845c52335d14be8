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
//     at byte 4 g + j, and the quantiser writes the activations in the same order;
//   - the weights are the rows of a tile and the tokens its columns, so a batch pays for its tokens in steps of 16.
//     (With the tokens on the 128 TMEM lanes and a tile of up to 128 weight rows a batch of 21 tokens paid for 128, one of
//     173 for 256. A block of 128 inputs took a tile of 128 x 112 outputs 1.79 us with the staging in the worker warps; here
//     128 x 128 outputs take 1.50, 128 x 64 0.90, 128 x 16 0.59; the three operations alone would take 0.83 of the 1.50.)
#include <cuda_fp16.h>

#include "bp_common.cuh"
#include "bp_ptx.cuh"
#include "bp_q1_device.cuh"
#include "bp_q1_ops.cuh"

namespace {

using namespace bp;

constexpr uint32_t TT_M = 128;                       // weight rows of a tile = TMEM lanes
constexpr uint32_t TT_A = TT_M * 128;                // a block of 128 inputs of a tile's weights: one byte per weight
constexpr uint32_t TT_RAW = TT_M * 16, TT_RAWS = 8;  // sign bits of a block of a tile, and blocks of them on their way

// ---- activations -------------------------------------------------------------------------------------------
// Tiled activations of a batch: per tile of N tokens and block of 128 inputs, part 0 (16 rint(q / 16)) and then part 1
// (the remainder) as [N tokens][128 bytes], a token's 16-byte chunks xor-ed with (token mod 8): the layout the MMA reads
// (K-major, 128-byte swizzle), so a stage is ONE bulk copy. Scales: [tile][block][4 sub-blocks][N tokens].
enum { SRC_PLAIN = 0, SRC_RMS = 1, SRC_SILU = 2 };

// quantize_q8_0.wgsl after nothing, after rms_norm.wgsl:41-85, or after silu_mul.wgsl:18-27: the producing
// operator's f16 results go straight into the quantiser. One CTA per token, 512 threads (the norm's
// invocation count: its sum is per invocation). Four lanes share a sub-block: lane t takes the inputs of output
// words 2 t and 2 t + 1, which are the pairs 8 j + 6 - 2 t, 8 j + 7 - 2 t.
template <int SRC>
__global__ void __launch_bounds__(512) quantize_tiled_kernel(const __half* x, const __half* aux, uint32_t k, float eps, uint32_t n_tok, uint8_t* a_t,
                                                             float* a_d) {
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
  const uint32_t r = row % n_tok, t = tid & 3u, part_b = n_tok * 128u;
  const size_t tile0 = static_cast<size_t>(row / n_tok) * nb1;
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
    uint8_t* dst = a_t + (tile0 + kb) * (2u * part_b) + r * 128u + (((2u * s + (t >> 1)) ^ (r & 7u)) << 4) + 8u * (t & 1u);
    *reinterpret_cast<uint2*>(dst) = make_uint2(hi[0], hi[1]);
    *reinterpret_cast<uint2*>(dst + part_b) = make_uint2(lo[0], lo[1]);
    if (t == 0) a_d[((tile0 + kb) * 4u + s) * n_tok + r] = d;
  }
}

// ---- product -----------------------------------------------------------------------------------------------
struct TiledTensors {  // up to three weight tensors over the same activations: row tile blockIdx.x belongs to one of them
  const __half* w_d[3];
  const uint8_t* w_qs[3];
  __half* y[3];
  uint32_t n[3];
  uint32_t tile_end[3];  // running total of row tiles
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
// 16-byte global -> shared copy; cp_async_arrive: this thread's copies so far arrive (once) on the mbarrier when they have landed
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// 16 TMEM lanes x 8 GROUPS columns: the thread gets, per group of 8 columns, columns 2 (lane mod 4) + {0, 1} of row
// lane / 4 (r[0], r[1]) and of row lane / 4 + 8 (r[2], r[3]).
template <uint32_t GROUPS>
__device__ __forceinline__ void tmem_ld_rows16(uint32_t taddr, uint32_t* r) {
  static_assert(GROUPS == 1 || GROUPS == 2, "groups of a load");
  if constexpr (GROUPS == 1) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
  } else {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
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

// A CTA owns 128 weight rows x N tokens and runs alone on its SM. The weights are the A operand (their rows are
// the TMEM lanes), the tokens the columns, so a batch costs by its tokens in steps of 16.
//   loader warp       sign bits (asynchronous copies) and scales TT_RAWS blocks ahead; one lane requests the activations
//                     and their scales for a free stage
//   stager warps      a block's 128 x 128 sign bits -> one byte per weight
//   issuer warp       one thread issues the MMAs, G sub-blocks per hand-over, into one of BUFS sets of G TMEM buffers
//   worker warps      take finished sub-blocks out of TMEM, scale and add them: sums in registers over all blocks
// Every wait is bounded; a wait that gives up stores a code in the error word and the CTA winds down: it ends only
// when its own copies have landed and its own MMAs are complete (waits of TT_DRAIN polls, whatever the caller's limit:
// what is waited for there always comes), because the next CTA on the SM gets the same shared memory and TMEM.
constexpr uint32_t TT_DRAIN = 1u << 20;

template <uint32_t V>
struct Num {  // a constant as an argument
  static constexpr uint32_t value = V;
};

template <uint32_t N_, uint32_t STAGERS_ = (N_ > 64 ? 2 : 4)>
struct TtLayout {
  static constexpr uint32_t N = N_;
  // Worker warps: 4 quarters of the TMEM lanes x CG groups of NC tokens. Stager warps: as many as leave the workers
  // their registers (a scheduler's 16384 are shared by a quarter of the warps: up to 20 warps have 96 each).
  static constexpr uint32_t CG = N == 16 ? 2 : N == 48 ? 3 : 4, NC = N / CG, WORKERS = 4 * CG;
  static constexpr uint32_t STAGERS = STAGERS_;
  static constexpr uint32_t LOADER = WORKERS + STAGERS, ISSUER = LOADER + 1;  // the warps that request copies and issue MMAs
  static constexpr uint32_t THREADS = (ISSUER + 1) * 32;
  static constexpr uint32_t B = 2 * N * 128, AD = N * 16, WD = TT_M * 4;
  static constexpr uint32_t STAGE = TT_A + B;                         // operands: a multiple of 1024
  static constexpr uint32_t STAGES = N > 64 ? 4 : N == 64 ? 6 : N == 48 ? 7 : 8;
  static constexpr uint32_t OFF_AD = STAGES * STAGE, OFF_WD = OFF_AD + STAGES * AD;
  static constexpr uint32_t OFF_RAW = OFF_WD + STAGES * WD;           // sign bits as they are in memory: [128 rows][16 bytes] per block
  static constexpr uint32_t SMEM = OFF_RAW + TT_RAWS * TT_RAW + 1024;
  static constexpr uint32_t G = N > 64 ? 2 : 4, STEPS = 4 / G;        // sub-blocks per hand-over, hand-overs per block
  static constexpr uint32_t COLS = N > 64 ? 128 : N > 32 ? 64 : N;    // TMEM columns of one buffer
  static constexpr uint32_t BUFS = N > 32 ? 2 : 4;                    // sets of G TMEM buffers
  // a piece is what is loaded from TMEM at a time: up to 16 values of a thread, PS sub-blocks or 1 / PPS of one
  static constexpr uint32_t PS = NC == 8 ? 2 : 1, PPS = NC > 16 ? 2 : 1, Q = G * PPS / PS;
  static_assert(BUFS * G * COLS <= 512 && N % 16 == 0 && NC % 8 == 0 && SMEM <= 227 * 1024 - 1024, "limits of an SM");
};

// The outputs of weight row tile `tile` and of the L::N tokens from number `first` on of token tile `m_tile`, which has NL
// tokens in the activations (first = 0 when L::N = NL). Tensors is a value or a reference: which of them leaves the compiler
// the better code differs (gate + up in tiles of 128: three whole waves 143 / 149 us, five and a cut one 274 / 267).
template <class L, uint32_t NL, class Tensors>
__device__ __forceinline__ void tiled_tile(Tensors tensors, uint32_t k, uint32_t m, const uint8_t* __restrict__ a_t,
                                           const float* __restrict__ a_d, uint32_t accumulate, float one, uint32_t* err, uint32_t wait_limit,
                                           uint32_t poll_ns, uint32_t tile, uint32_t m_tile, uint32_t first) {
  static_assert(NL % L::N == 0, "part of a tile");
  constexpr uint32_t N = L::N;
  constexpr uint32_t NC = L::NC, G = L::G, STEPS = L::STEPS, BUFS = L::BUFS, COLS = L::COLS, STAGES = L::STAGES;
  extern __shared__ uint8_t tt_raw[];
  __shared__ __align__(8) uint64_t full[STAGES], a_full[STAGES], empty[STAGES], d_full[BUFS], d_empty[BUFS], drained;
  __shared__ __align__(8) uint64_t raw_full[TT_RAWS], raw_empty[TT_RAWS];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile uint32_t abort_s;
  const uint32_t smem_base = (smem_u32(tt_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = tt_raw + (smem_base - smem_u32(tt_raw));
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t which = tile < tensors.tile_end[0] ? 0u : tile < tensors.tile_end[1] ? 1u : 2u;
  // (selects: an indexed parameter array would be copied to local memory)
  auto pick = [&](const auto* v) { return which == 0 ? v[0] : which == 1 ? v[1] : v[2]; };
  const uint32_t n = pick(tensors.n);
  const uint32_t n_base = (tile - (which == 0 ? 0u : which == 1 ? tensors.tile_end[0] : tensors.tile_end[1])) * TT_M, m_base = m_tile * NL + first;
  const uint32_t nb1 = k / 128u;
  if (tid == 0) {
    for (uint32_t i = 0; i < STAGES; i++) {
      mbar_init(smem_u32(&full[i]), 2);  // stager and loader
      mbar_init(smem_u32(&a_full[i]), 1);
      mbar_init(smem_u32(&empty[i]), 1 + L::WORKERS);
    }
    for (uint32_t i = 0; i < BUFS; i++) {
      mbar_init(smem_u32(&d_full[i]), 2);  // the MMAs, and the thread that issued them
      mbar_init(smem_u32(&d_empty[i]), L::WORKERS);
    }
    for (uint32_t i = 0; i < TT_RAWS; i++) {
      mbar_init(smem_u32(&raw_full[i]), 32);
      mbar_init(smem_u32(&raw_empty[i]), 1);
    }
    mbar_init(smem_u32(&drained), 1);
    abort_s = 0;
    fence_barrier_init();
  }
  if (warp == L::ISSUER) tmem_alloc(smem_u32(&tmem_base_s), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  if (tid == 0) pdl_launch_dependents();
  // A wait that gives up, or finds that another one has, leaves its thread `dead`: the thread runs through the rest of
  // its loop without waiting, copying or writing results. (The flag is a register: a look at abort_s before every wait
  // and every MMA lengthened the chain from hand-over to hand-over by 7 % of the kernel.)
  bool dead = false;
  // A phase that is complete already is found by a plain test: the poll that may suspend its thread costs some 350 cycles here
  // even then, several times per block (128 x 128 outputs: 1.75 us with it alone, 1.62 with the test first; 128 x 16: 0.84, 0.63).
  auto waitb = [&](uint64_t* bar, uint32_t parity, uint32_t ns = 2000u) {  // ns: how long a poll may suspend its thread
    if (dead) return;
    const uint32_t addr = smem_u32(bar);
    if (mbar_test(addr, parity)) return;
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

  if (warp == L::ISSUER) {
    // ---------------- MMA issuer ----------------
    pdl_wait();  // the polls below count from here: the time of the kernel before this one is not theirs
    if (elect_one()) {
      constexpr uint32_t IDESC = umma_idesc(1, 0, 0, 0, 0, TT_M, N);  // f32 = e4m3 (K-major) x e4m3 (K-major)
      const uint64_t dk = umma_desc_sw128(0, 16, 1024);
      for (uint32_t b = 0; b < nb1; b++) {
        const uint32_t slot = b % STAGES;
        waitb(&a_full[slot], (b / STAGES) & 1u, poll_ns);
        waitb(&full[slot], (b / STAGES) & 1u);
        const uint64_t ad = dk + ((smem_base + slot * L::STAGE) >> 4), bd = ad + (TT_A >> 4);
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
              umma_f8(tmem + (pb * G + g) * COLS, ad + (h * G + g) * 2u, bd + part * (N * 128u >> 4) + (h * G + g) * 2u, IDESC, part);
          umma_commit(smem_u32(&d_full[pb]));
          mbar_arrive(smem_u32(&d_full[pb]));  // passes on what this thread has waited for, the scales among it
        }
        if (dead) break;  // no slot is given back any more: a copy into it could meet the previous one
        if (b + STAGES < nb1) umma_commit(smem_u32(&empty[slot]));  // (no arrival that nobody waits for: it could outlive the CTA)
      }
    }
  } else if (warp == L::LOADER) {
    // ---------------- loader ----------------
    constexpr uint32_t RL = TT_M / 32;  // weight rows of a lane: lane, lane + 32, ..
    const uint8_t* w_qs = pick(tensors.w_qs);
    const __half* w_d = pick(tensors.w_d);
    const uint8_t* a_src = a_t + static_cast<size_t>(m_tile) * nb1 * (2u * NL * 128u) + first * 128u;
    const float* ad_src = a_d + static_cast<size_t>(m_tile) * nb1 * (4u * NL) + first;
    uint32_t at[RL];  // the lane's rows (one beyond the tensor repeats the last: nobody reads its results)
#pragma unroll
    for (uint32_t r = 0; r < RL; r++) at[r] = min(n_base + lane + 32u * r, n - 1u);
    __half scale[TT_RAWS][RL];
    uint32_t copies = 0;  // blocks of activations requested (one lane)
    bool before = true;   // the kernel before this one may still run: the weights are constants, the activations are its results
    for (uint32_t t0 = 0; t0 < nb1 + TT_RAWS; t0 += TT_RAWS) {
#pragma unroll
      for (uint32_t i = 0; i < TT_RAWS; i++) {
        const uint32_t t = t0 + i;
        if (t >= TT_RAWS && t - TT_RAWS < nb1) {  // block t - TT_RAWS into its stage
          const uint32_t b = t - TT_RAWS, slot = b % STAGES;
          if (before) {
            pdl_wait();
            before = false;
          }
          if (b >= STAGES) waitb(&empty[slot], ((b / STAGES) - 1u) & 1u);
          if (lane == 0 && !dead) {
            mbar_arrive_expect_tx(smem_u32(&a_full[slot]), L::B + L::AD);
            constexpr uint32_t PARTS = N == NL ? 1 : 2, SCALES = N == NL ? 1 : 4;  // (what lies together when the tile is whole)
#pragma unroll
            for (uint32_t c = 0; c < PARTS; c++)
              bulk_load(smem_base + slot * L::STAGE + TT_A + c * (N * 128u), a_src + (static_cast<size_t>(b) * 2u + c) * (NL * 128u), L::B / PARTS,
                        smem_u32(&a_full[slot]));
#pragma unroll
            for (uint32_t c = 0; c < SCALES; c++)
              bulk_load(smem_base + L::OFF_AD + slot * L::AD + c * (N * 4u), ad_src + (static_cast<size_t>(b) * 4u + c) * NL, L::AD / SCALES,
                        smem_u32(&a_full[slot]));
            copies = b + 1;
          }
          float* wd = reinterpret_cast<float*>(smem_gen + L::OFF_WD + slot * L::WD);
#pragma unroll
          for (uint32_t r = 0; r < RL; r++) wd[lane + 32u * r] = __half2float(scale[i][r]);
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&full[slot]));
        }
        if (t < nb1) {  // block t requested
          if (t >= TT_RAWS) waitb(&raw_empty[i], ((t / TT_RAWS) - 1u) & 1u);
#pragma unroll
          for (uint32_t r = 0; r < RL; r++) {
            const size_t blk = static_cast<size_t>(at[r]) * nb1 + t;
            cp_async16(smem_base + L::OFF_RAW + i * TT_RAW + (lane + 32u * r) * 16u, w_qs + blk * 16u);
            scale[i][r] = __ldg(w_d + blk);
          }
          cp_async_arrive(smem_u32(&raw_full[i]));
        }
      }
    }
    // no copy may still be on its way when the CTA ends (all have landed unless a wait gave up)
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (lane == 0)
      for (uint32_t b = copies > STAGES ? copies - STAGES : 0; b < copies; b++) (void)mbar_wait(smem_u32(&a_full[b % STAGES]), (b / STAGES) & 1u, TT_DRAIN);
  } else if (warp >= L::WORKERS) {
    // ---------------- stagers ----------------
    // The sign bits of a sub-block are one 32-bit word w, and word g of its 32 bytes is (w << g) & 0x80808080 xor
    // 0xB8B8B8B8 (e4m3 +-1). A warp takes whole blocks, every STAGERS-th. (A stage is waited for by different stagers in
    // turn, but none is ever two uses behind: a stager at block b has seen block b - STAGERS - STAGES released, and
    // stages are released in order.)
    static_assert(L::STAGERS <= STAGES && TT_RAWS % L::STAGERS == 0, "phases that a stager has to follow");
    constexpr uint32_t AHEAD = STAGES < TT_RAWS ? STAGES : TT_RAWS;  // blocks that need nothing of the kernel before this one
    for (uint32_t b = warp - L::WORKERS; b < nb1; b += L::STAGERS) {
      const uint32_t slot = b % STAGES, rs = b % TT_RAWS;
      // Further signs are requested, and stages given back, only behind that kernel: the polls count from its end.
      if (b >= AHEAD && b < AHEAD + L::STAGERS) pdl_wait();
      waitb(&raw_full[rs], (b / TT_RAWS) & 1u);
      uint4 sign[4];
#pragma unroll
      for (uint32_t r = 0; r < 4; r++) sign[r] = *reinterpret_cast<const uint4*>(smem_gen + L::OFF_RAW + rs * TT_RAW + (lane + 32u * r) * 16u);
      __syncwarp();
      if (lane == 0 && b + TT_RAWS < nb1) mbar_arrive(smem_u32(&raw_empty[rs]));
      if (b >= STAGES) waitb(&empty[slot], ((b / STAGES) - 1u) & 1u);
#pragma unroll
      for (uint32_t r = 0; r < 4; r++) {
        uint8_t* row = smem_gen + slot * L::STAGE + (lane + 32u * r) * 128u;
        const uint32_t w[4] = {sign[r].x, sign[r].y, sign[r].z, sign[r].w};
#pragma unroll
        for (uint32_t s = 0; s < 4; s++) {
          uint32_t o[8];
#pragma unroll
          for (uint32_t g = 0; g < 8; g++) o[g] = ((w[s] << g) & 0x80808080u) ^ 0xB8B8B8B8u;  // bit set: +1 (0x38), clear: -1 (0xB8)
          *reinterpret_cast<uint4*>(row + (((2u * s) ^ (lane & 7u)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<uint4*>(row + (((2u * s + 1u) ^ (lane & 7u)) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full[slot]));
    }
  } else {
    // ---------------- workers ----------------
    // thread: rows lane / 4 + {0, 8, 16, 24} of its quarter, token pairs 2 (lane mod 4) + {0, 1} of every 8: a scale that
    // it reads from shared memory serves four rows.
    const uint32_t quad = warp & 3u, cg = warp >> 2, r0 = quad * 32u + (lane >> 2), c2 = 2u * (lane & 3u);
    const uint32_t t_addr = tmem + ((quad * 32u) << 16) + cg * NC;
    unsigned long long acc[NC / 8][4];  // [token pair][row]
#pragma unroll
    for (uint32_t c = 0; c < NC / 8; c++)
#pragma unroll
      for (uint32_t r = 0; r < 4; r++) acc[c][r] = 0ull;
    const unsigned long long ones = pack2(one, one);
    pdl_wait();
    uint32_t d[2][16];
    bool there = false;  // the next hand-over, seen while this one was worked on
    // GC groups of 8 tokens from TMEM column `at` on: [row half][group][4]
    auto load_rows = [&](uint32_t at, auto gc, uint32_t* r) {
      tmem_ld_rows16<decltype(gc)::value>(at, r);
      tmem_ld_rows16<decltype(gc)::value>(at + (16u << 16), r + 4 * decltype(gc)::value);
    };
    for (uint32_t b = 0; b < nb1; b++) {
      const uint32_t slot = b % STAGES;
      const float* wd = reinterpret_cast<const float*>(smem_gen + L::OFF_WD + slot * L::WD) + r0;
      unsigned long long wd2[4];
      const float* ad_s = reinterpret_cast<const float*>(smem_gen + L::OFF_AD + slot * L::AD) + cg * NC + c2;
#pragma unroll
      for (uint32_t h = 0; h < STEPS; h++) {
        const uint32_t j = b * STEPS + h, pb = j % BUFS;
        if (!there) waitb(&d_full[pb], (j / BUFS) & 1u);
        tc_fence_after();
        if (h == 0) {  // (the scales are there: the issuer has waited for them and arrived on d_full since. Waiting for them here took 0.1 us)
#pragma unroll
          for (uint32_t r = 0; r < 4; r++) wd2[r] = pack2(wd[8 * r], wd[8 * r]);
        }
        // the pieces of the G sub-blocks, each load in flight while the previous piece is scaled and added
        auto load = [&](uint32_t q) {
          uint32_t* r = d[q & 1u];
          if constexpr (L::PPS == 2) {
            const uint32_t at = t_addr + (pb * G + q / 2) * COLS;
            if (q % 2 == 0) load_rows(at, Num<2>(), r);
            else load_rows(at + 16, Num<(NC > 16 ? NC - 16 : 8) / 8>(), r);
          } else {
#pragma unroll
            for (uint32_t i = 0; i < L::PS; i++) load_rows(t_addr + (pb * G + q * L::PS + i) * COLS, Num<(NC > 16 ? 16 : NC) / 8>(), r + i * NC);
          }
        };
        load(0);
#pragma unroll
        for (uint32_t q = 0; q < L::Q; q++) {
          tmem_ld_wait();
          if (q + 1 < L::Q) {
            load(q + 1);
          } else {  // the whole hand-over is in registers: its buffers may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&d_empty[pb]));
            // (the answer comes while the last piece is worked on: 128 x 96 outputs 1.22 -> 1.18 us, 128 x 128 1.52 -> 1.50)
            there = mbar_test(smem_u32(&d_full[(j + 1) % BUFS]), ((j + 1) / BUFS) & 1u);
          }
#pragma unroll
          for (uint32_t i = 0; i < L::PS; i++) {
            const uint32_t g = L::PPS == 2 ? q / 2 : q * L::PS + i;
            const uint32_t p0 = L::PPS == 2 ? (q % 2) * 2 : 0, groups = L::PPS == 2 ? (q % 2 == 0 ? 2 : (NC - 16) / 8) : NC / 8;
#pragma unroll
            for (uint32_t c = 0; c < groups; c++) {
              const float2 a2 = *reinterpret_cast<const float2*>(ad_s + (h * G + g) * N + 8 * (p0 + c));
              const unsigned long long ad2 = pack2(a2.x, a2.y);
#pragma unroll
              for (uint32_t r = 0; r < 4; r++) {  // rows of the first 16 lanes, then of the second
                const uint32_t* dq = d[q & 1u] + i * NC + (r >> 1) * 4 * groups + 4 * c + 2 * (r & 1u);
                const unsigned long long t = mul2(mul2(wd2[r], ad2), pack2(__uint_as_float(dq[0]), __uint_as_float(dq[1])));
                acc[p0 + c][r] = fma2(t, ones, acc[p0 + c][r]);
              }
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0 && b + STAGES < nb1) mbar_arrive(smem_u32(&empty[slot]));  // the block's scales are read
    }
    if (!dead) {
      const uint32_t t0 = m_base + cg * NC + c2;
      __half* const y = pick(tensors.y);
#pragma unroll
      for (uint32_t c = 0; c < NC / 8; c++) {
#pragma unroll
        for (uint32_t e = 0; e < 2; e++) {
          const uint32_t t = t0 + 8 * c + e;
          __half* dst = y + static_cast<size_t>(t) * n + n_base + r0;
          __half old[4];
#pragma unroll
          for (uint32_t r = 0; r < 4; r++)
            if (accumulate && t < m && n_base + r0 + 8 * r < n) old[r] = dst[8 * r];
#pragma unroll
          for (uint32_t r = 0; r < 4; r++) {
            float v[2];
            unpack2(acc[c][r], v[0], v[1]);
            if (t < m && n_base + r0 + 8 * r < n) dst[8 * r] = __float2half_rn(accumulate ? __fadd_rn(__half2float(old[r]), v[e]) : v[e]);
          }
        }
      }
    }
  }
  __syncwarp();  // the lanes of the one-thread roles meet again
  tc_fence_before();
  __syncthreads();
  if (abort_s) {  // the workers have not seen the last MMAs complete
    if (warp == L::ISSUER && elect_one()) {  // (the thread that issued them)
      umma_commit(smem_u32(&drained));
      (void)mbar_wait(smem_u32(&drained), 0, TT_DRAIN);
    }
    __syncthreads();
  }
  if (warp == L::ISSUER) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <uint32_t N>
__global__ void __launch_bounds__(TtLayout<N>::THREADS, 1) matmul_q1_tiled_kernel(const TiledTensors tensors, uint32_t k, uint32_t m, const uint8_t* __restrict__ a_t,
                                                                        const float* __restrict__ a_d, uint32_t accumulate, float one, uint32_t* err,
                                                                        uint32_t wait_limit, uint32_t poll_ns) {
  tiled_tile<TtLayout<N>, N, const TiledTensors>(tensors, k, m, a_t, a_d, accumulate, one, err, wait_limit, poll_ns, blockIdx.x, blockIdx.y, 0);
}

// The same with the tiles of the last wave cut into tiles of NS tokens: `whole` CTAs have a tile of N, then come the narrow
// ones. A last wave of few tiles leaves most SMs idle for as long as a full one takes: gate + up of 512 tokens at the 8B
// shape (768 tiles = 5 waves of 148 and 28) 288 -> 267 us, of 128 tokens (148 and 44; tiles of 64 before) 91 -> 82.
template <uint32_t N, uint32_t NS>
__global__ void __launch_bounds__(TtLayout<N>::THREADS, 1) matmul_q1_tiled_cut_kernel(const TiledTensors tensors, uint32_t k, uint32_t m,
                                                                        const uint8_t* __restrict__ a_t, const float* __restrict__ a_d,
                                                                        uint32_t accumulate, float one, uint32_t* err, uint32_t wait_limit,
                                                                        uint32_t poll_ns, uint32_t whole) {
  using Small = TtLayout<NS, TtLayout<N>::STAGERS>;
  static_assert(Small::THREADS == TtLayout<N>::THREADS, "the same warps");
  const uint32_t tiles = tensors.tile_end[2];
  if (blockIdx.x < whole) {
    tiled_tile<TtLayout<N>, N, const TiledTensors&>(tensors, k, m, a_t, a_d, accumulate, one, err, wait_limit, poll_ns, blockIdx.x % tiles, blockIdx.x / tiles, 0);
  } else {
    const uint32_t i = blockIdx.x - whole, at = whole + i / (N / NS), first = i % (N / NS) * NS;
    if (at / tiles * N + first < m)
      tiled_tile<Small, N, const TiledTensors&>(tensors, k, m, a_t, a_d, accumulate, one, err, wait_limit, poll_ns, at % tiles, at / tiles, first);
  }
}

// Tokens of the tiles into which the last wave is cut: as narrow as lets them all run at once; n_tok: it is not cut. (Less
// than one wave is not: plain tiles of that width are up to 7 % faster.)
uint32_t last_wave_tokens(uint32_t n_tok, uint32_t ctas, uint32_t sms) {
  const uint32_t rest = ctas % sms;
  if (n_tok != 128 || ctas < sms || rest == 0) return n_tok;
  return rest * 4 <= sms ? 32 : rest * 2 <= sms ? 64 : 128;
}

template <uint32_t N, uint32_t NS = N>
cudaError_t launch_tiled(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* y, uint32_t n_w, uint32_t m, const uint8_t* a_t,
                         const float* a_d, bool accumulate, uint32_t* err, uint32_t wait_limit) {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  TiledTensors t;
  uint32_t tiles = 0;
  for (uint32_t i = 0; i < 3; i++) {
    const uint32_t j = i < n_w ? i : n_w - 1;  // unused entries repeat the last tensor; their tile range is empty
    t.w_d[i] = w[j].d;
    t.w_qs[i] = w[j].qs;
    t.y[i] = y[j];
    t.n[i] = w[j].n;
    if (i < n_w) tiles += (w[i].n + TT_M - 1) / TT_M;
    t.tile_end[i] = tiles;
  }
  const uint32_t m_tiles = (m + N - 1) / N, ctas = tiles * m_tiles, sms = bp_q1_sm_count();
  if constexpr (N == 128 && NS == N) {
    const uint32_t last = last_wave_tokens(N, ctas, sms);
    if (last == 32) return launch_tiled<N, 32>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    if (last == 64) return launch_tiled<N, 64>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
  }
  using L = TtLayout<N>;
  constexpr uint32_t SMALL = TtLayout<NS, L::STAGERS>::SMEM, SMEM = L::SMEM > SMALL ? L::SMEM : SMALL;
  const void* kernel;
  if constexpr (NS == N) kernel = reinterpret_cast<const void*>(matmul_q1_tiled_kernel<N>);
  else kernel = reinterpret_cast<const void*>(matmul_q1_tiled_cut_kernel<N, NS>);
  if (!configured[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM));
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  // (a limit of a few polls is short in time too: the MMA issuer's polls for a copy suspend it for as many ns at most)
  const uint32_t acc = accumulate ? 1u : 0u, poll_ns = wait_limit < 2000u ? wait_limit : 2000u;
  if constexpr (NS == N) {
    return bp_launch(pdl, matmul_q1_tiled_kernel<N>, dim3(tiles, m_tiles), dim3(L::THREADS), SMEM, s, t, w[0].k, m, a_t, a_d, acc, 1.0f, err, wait_limit,
                     poll_ns);
  } else {
    const uint32_t rest = ctas % sms, whole = ctas - rest;
    return bp_launch(pdl, matmul_q1_tiled_cut_kernel<N, NS>, dim3(whole + rest * (N / NS)), dim3(L::THREADS), SMEM, s, t, w[0].k, m, a_t, a_d, acc, 1.0f,
                     err, wait_limit, poll_ns, whole);
  }
}

}  // namespace

// (a tile may be partly filled: at most 127 rows of no token, whatever its width)
size_t bp_q1_tiled_bytes(uint32_t m, uint32_t k) { return static_cast<size_t>(m + 127u) * k * 2u; }
size_t bp_q1_tiled_scales(uint32_t m, uint32_t k) { return static_cast<size_t>(m + 127u) * (k / 32u); }

cudaError_t bp_q1_quantize_tiled(bool pdl, cudaStream_t s, const __half* x, uint32_t k, uint32_t m, uint32_t n_tok, uint8_t* a_t, float* a_d) {
  return bp_launch(pdl, quantize_tiled_kernel<SRC_PLAIN>, dim3(m), dim3(512), 0, s, x, x, k, 0.0f, n_tok, a_t, a_d);
}
cudaError_t bp_q1_rms_quantize_tiled(bool pdl, cudaStream_t s, const __half* x, const __half* w, float eps, uint32_t k, uint32_t m, uint32_t n_tok,
                                     uint8_t* a_t, float* a_d) {
  return bp_launch(pdl, quantize_tiled_kernel<SRC_RMS>, dim3(m), dim3(512), 0, s, x, w, k, eps, n_tok, a_t, a_d);
}
cudaError_t bp_q1_silu_quantize_tiled(bool pdl, cudaStream_t s, const __half* gate, const __half* up, uint32_t k, uint32_t m, uint32_t n_tok,
                                      uint8_t* a_t, float* a_d) {
  return bp_launch(pdl, quantize_tiled_kernel<SRC_SILU>, dim3(m), dim3(512), 0, s, gate, up, k, 0.0f, n_tok, a_t, a_d);
}

uint32_t bp_q1_tile_tokens(const bp_q1_tensor* w, uint32_t n_w, uint32_t m) {
  if (bp_q1_tile_width() != 0) return bp_q1_tile_width();
  const uint32_t sms = bp_q1_sm_count();
  // Waves of one CTA per SM, times what a block of a tile of that width takes: us, gate + up of 512 tokens at the 8B shape
  // (96 blocks take 7 % less per block, 32 blocks in one wave up to 6 % more, of 16 tokens 20 %).
  const uint32_t widths[6] = {128, 96, 64, 48, 32, 16};
  const float cost[6] = {1.50f, 1.18f, 0.90f, 0.76f, 0.70f, 0.59f};
  uint32_t tiles = 0;
  for (uint32_t i = 0; i < n_w; i++) tiles += (w[i].n + TT_M - 1) / TT_M;
  float best = 1e30f;
  uint32_t n_tok = 128;
  for (int c = 0; c < 6; c++) {
    const uint32_t ctas = tiles * ((m + widths[c] - 1) / widths[c]);
    const uint32_t last = last_wave_tokens(widths[c], ctas, sms);
    const float t = cost[c] * static_cast<float>(ctas / sms) + (ctas % sms == 0 ? 0.0f : last == widths[c] ? cost[c] : last == 64 ? cost[2] : cost[4]);
    if (t < best) {
      best = t;
      n_tok = widths[c];
    }
  }
  return n_tok;
}

cudaError_t bp_q1_matmul_tiled(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* y, uint32_t n_w, uint32_t m, uint32_t n_tok,
                               const uint8_t* a_t, const float* a_d, bool accumulate, uint32_t* err, uint32_t wait_limit) {
  if (n_w == 0 || n_w > 3) return cudaErrorInvalidValue;
  switch (n_tok) {
    case 128: return launch_tiled<128>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 96: return launch_tiled<96>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 64: return launch_tiled<64>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 48: return launch_tiled<48>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 32: return launch_tiled<32>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    case 16: return launch_tiled<16>(pdl, s, w, y, n_w, m, a_t, a_d, accumulate, err, wait_limit);
    default: return cudaErrorInvalidValue;
  }
}
