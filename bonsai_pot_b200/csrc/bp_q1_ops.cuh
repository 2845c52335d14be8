// Launchers of the non-attention operators on Q1_0 weights (bp_q1_ops.cu). A Q1_0 tensor
// [n rows][k inputs] is n * k / 128 blocks of one f16 scale and 128 sign bits; on the device it is
// held as the reference's two arrays (scales, sign bytes: src/model.rs manifest d_offset / qs_offset)
// plus, for the tensors the one-token path multiplies, the sign words re-laid out for the matvec kernels.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

struct bp_q1_tensor {
  const __half* d;      // block scales [n][k / 128]
  const uint8_t* qs;    // sign bytes [n][k / 128][16], bit e of a block = weight e (1 = +d, 0 = -d)
  const void* bits;     // re-laid-out sign words [n][k / 128] (uint4), or null
  uint32_t k, n;
};

uint32_t bp_q1_sm_count();  // of the current device: what the grids are cut for
void bp_q1_set_matvec_rows(uint32_t rows_per_lane);  // tuning aid: 0 = by tensor height, else 1, 2 or 4
cudaError_t bp_q1_relayout(cudaStream_t s, const uint8_t* qs, void* out, uint64_t n_blocks);
cudaError_t bp_q1_matvec(bool pdl, cudaStream_t s, const bp_q1_tensor& w, const __half* x, __half* y, bool accumulate);
cudaError_t bp_q1_matvec_normed(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* out, uint32_t n_ranges,
                                const __half* x, const __half* w_norm, float eps);
cudaError_t bp_q1_matvec_normed_silu(bool pdl, cudaStream_t s, const bp_q1_tensor& w_gate, const bp_q1_tensor& w_up, __half* out,
                                     const __half* x, const __half* w_norm, float eps);
cudaError_t bp_q1_matvec_silu(bool pdl, cudaStream_t s, const bp_q1_tensor& w, const __half* gate, const __half* up, __half* y,
                              bool accumulate);
cudaError_t bp_q1_rms_norm(bool pdl, cudaStream_t s, const __half* in, __half* out, const __half* w, uint32_t group_size,
                           uint32_t n_groups, float eps);
cudaError_t bp_q1_silu_mul(bool pdl, cudaStream_t s, const __half* gate, const __half* up, __half* out, uint64_t n);
cudaError_t bp_q1_embed(bool pdl, cudaStream_t s, const bp_q1_tensor& w, const uint32_t* tokens, uint32_t m, __half* x);
cudaError_t bp_q1_quantize_q8(bool pdl, cudaStream_t s, const __half* x, uint32_t k, uint32_t m, float* d_out, int8_t* qs_out);
// err: device-visible error word that a bounded wait of the tensor-core kernel stores a code in when it gives
// up (null: a word of the library's own, read and cleared by bp_q1_take_error); wait_limit 0 = default.
cudaError_t bp_q1_matmul(bool pdl, cudaStream_t s, const bp_q1_tensor& w, uint32_t m, const float* a_d, const int8_t* a_qs, __half* y,
                         bool accumulate, uint32_t* err = nullptr, uint32_t wait_limit = 0);
cudaError_t bp_q1_matmul_multi(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* y, uint32_t n_w, uint32_t m, const float* a_d,
                               const int8_t* a_qs, bool accumulate, uint32_t* err = nullptr, uint32_t wait_limit = 0);
// The product of a model's batches (bp_q1_matmul_tiled.cu): the quantisers write the activations in the layout the
// kernel reads (sizes in bytes / floats for a batch of m tokens, k inputs).
bool bp_q1_matmul_is_tiled(uint32_t m);
uint32_t bp_q1_tile_width();  // tuning aid: 0 = by the number of tiles
// Tokens of a tile (n_tok below) for the product of these weights with a batch of m tokens.
uint32_t bp_q1_tile_tokens(const bp_q1_tensor* w, uint32_t n_w, uint32_t m);
size_t bp_q1_tiled_bytes(uint32_t m, uint32_t k);
size_t bp_q1_tiled_scales(uint32_t m, uint32_t k);
cudaError_t bp_q1_quantize_tiled(bool pdl, cudaStream_t s, const __half* x, uint32_t k, uint32_t m, uint32_t n_tok, uint8_t* a_t, float* a_d);
cudaError_t bp_q1_rms_quantize_tiled(bool pdl, cudaStream_t s, const __half* x, const __half* w, float eps, uint32_t k, uint32_t m, uint32_t n_tok, uint8_t* a_t, float* a_d);
cudaError_t bp_q1_silu_quantize_tiled(bool pdl, cudaStream_t s, const __half* gate, const __half* up, uint32_t k, uint32_t m, uint32_t n_tok, uint8_t* a_t, float* a_d);
cudaError_t bp_q1_matmul_tiled(bool pdl, cudaStream_t s, const bp_q1_tensor* w, __half* const* y, uint32_t n_w, uint32_t m, uint32_t n_tok,
                               const uint8_t* a_t, const float* a_d, bool accumulate, uint32_t* err, uint32_t wait_limit);
void bp_q1_set_matmul_variant(uint32_t variant);  // tuning aid, see bp_op_set_matmul_variant
cudaError_t bp_q1_take_error(uint32_t* code);     // synchronous; 0 = no wait gave up since the last call
cudaError_t bp_q1_topk(bool pdl, cudaStream_t s, const __half* logits, uint32_t n, uint32_t k, float* out_val, uint32_t* out_idx);
