// Memory-bound model kernels used by the flagship training step (Llama-style
// decoder): RMSNorm, rotary embedding, SwiGLU, softmax cross-entropy fused
// with its gradient, and AdamW on flat fp32 shards. bf16 activations, fp32
// statistics and accumulation. Raw-pointer launch interface.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200c {

// y = x * rsqrt(mean(x^2) + eps) * w ; rstd saved for the backward pass.
// cols must be a multiple of 8; all bf16 pointers of the norm and SwiGLU launches are 16-byte aligned
// (cudaErrorMisalignedAddress otherwise). With `delta` (cols <= 8192) the normalised row is sum = bf16(x + delta), which is
// written as well.
cudaError_t launch_rmsnorm_fwd(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* y, float* rstd,
                               int rows, int cols, float eps, cudaStream_t s, const __nv_bfloat16* delta = nullptr,
                               __nv_bfloat16* sum = nullptr);
// dx, and per-block partial weight gradients `dw_partial` [nblocks, cols]
// (fp32), which `launch_colsum` folds into dw. Returns the number of blocks
// it will use through *nblocks when dw_partial is null (sizing query). `dskip`, if given, is added to dx.
cudaError_t launch_rmsnorm_bwd(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w,
                               const float* rstd, __nv_bfloat16* dx, float* dw_partial, int* nblocks, int rows,
                               int cols, cudaStream_t s, const __nv_bfloat16* dskip = nullptr);
// out[c] = sum_r in[r, c]  (fp32 in, 16-byte aligned, cols a multiple of 4; bf16 out)
cudaError_t launch_colsum_bf16(const float* in, __nv_bfloat16* out, int rows, int cols, cudaStream_t s);

// out[i] = convert(in[i] * scale) for n elements; `in_kind` / `out_kind`: 0 = fp32, 1 = bf16.
// What a collective degenerates to on a single rank (cast, scale, copy) in one pass.
cudaError_t launch_cast_scale(const void* in, int in_kind, void* out, int out_kind, size_t n, float scale, cudaStream_t s);

// Row-wise e4m3 quantisation of bf16 x [rows, cols] (row stride `ld` elements): scale[r] = max(max|x_r|, 1e-8) / 448,
// q[r, c] = e4m3(x[r, c] / scale[r]), q contiguous. Any cols; 16-byte accesses where the layout allows them.
cudaError_t launch_quantize_rows(const __nv_bfloat16* x, int64_t ld, void* q, float* scale, int rows, int cols, cudaStream_t s);

// Rotary embedding of x[tokens, heads, head_dim] with interleaved pairs into the
// contiguous y; pos[t] indexes the cos/sin tables [max_pos, head_dim/2]. `inverse`
// rotates by the negative angle (the backward pass). x may be a slice of a wider
// tensor: element strides of its token and head dimensions, multiples of 8 like
// head_dim; x, y and the tables 16-byte aligned.
cudaError_t launch_rope(const __nv_bfloat16* x, int64_t stride_t, int64_t stride_h, __nv_bfloat16* y, const int* pos,
                        const float* cos_t, const float* sin_t, int tokens, int heads, int head_dim, bool inverse,
                        cudaStream_t s);

// Queries, keys and values out of packed rows [tokens, (heads + 2 kv_heads) x head_dim] (row stride `ld`), queries
// and keys rotated; `backward` goes the other way with the inverse rotation and writes every packed element.
// parts / stride_t / stride_h: the three tensors [tokens, heads or kv_heads, head_dim] and their strides.
// Strides are multiples of 8 elements, all pointers 16-byte aligned.
cudaError_t launch_split_rope(__nv_bfloat16* packed, int64_t ld, __nv_bfloat16* const* parts, const int64_t* stride_t,
                              const int64_t* stride_h, const int* pos, const float* cos_t, const float* sin_t, int tokens,
                              int heads, int kv_heads, int head_dim, bool backward, cudaStream_t s);

// h = silu(gate) * up where gate_up = [rows, 2*ffn] (gate first).
cudaError_t launch_swiglu_fwd(const __nv_bfloat16* gate_up, __nv_bfloat16* h, int rows, int ffn, cudaStream_t s);
cudaError_t launch_swiglu_bwd(const __nv_bfloat16* dh, const __nv_bfloat16* gate_up, __nv_bfloat16* dgate_up,
                              int rows, int ffn, cudaStream_t s);

// Row-wise softmax cross-entropy: writes loss[r] and overwrites logits (row stride `ld` elements) with
// d(loss_sum * grad_scale)/dlogits. Rows whose target is < 0 are ignored.
cudaError_t launch_cross_entropy_fwd_bwd(__nv_bfloat16* logits, int64_t ld, const int64_t* targets, float* loss, int rows,
                                         int vocab, float grad_scale, cudaStream_t s);

// The same where launch_head_logits (tc_gemm.h) left the logits with their statistics: row stride `ld` a multiple of 16,
// logits on a 32-byte boundary; up to 15 elements past a row's last, within its stride, are overwritten. `row_scratch`:
// 2 * rows; *loss becomes loss_scale times the sum of the rows' losses, added to what it holds unless `first`.
cudaError_t launch_head_gradient(__nv_bfloat16* logits, int64_t ld, const int64_t* targets, const float2* stats, const float* fine, int shares,
                                 const float* target_logit, float* row_scratch, float* loss, uint32_t* words, int rows, int vocab,
                                 float grad_scale, float loss_scale, bool first, cudaStream_t s);

// dx[rows, cols] (bf16) = part (fp32) + grad[rows, depth] (row stride `ld`) x w[depth, cols], both bf16; cols % 8 == 0,
// part, w and dx 16-byte aligned.
cudaError_t launch_head_tail(const float* part, const __nv_bfloat16* grad, int64_t ld, const __nv_bfloat16* w, __nv_bfloat16* dx, int rows,
                             int cols, int depth, cudaStream_t s);

// out = in * bf16(*factor) on n bf16 values, the factor read from device memory; in and out 16-byte aligned. Optionally
// a second tensor by the same factor.
cudaError_t launch_scale_bf16(const __nv_bfloat16* in, __nv_bfloat16* out, const float* factor, size_t n, cudaStream_t s,
                              const __nv_bfloat16* in2 = nullptr, __nv_bfloat16* out2 = nullptr, size_t n2 = 0);

// AdamW on flat fp32 tensors, 16-byte aligned from four elements on. `grad_scale` multiplies the gradient first
// (loss scaling / averaging); `step` starts at 1.
cudaError_t launch_adamw(float* p, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2,
                         float eps, float weight_decay, int step, float grad_scale, cudaStream_t s);

// Count of launches made through this header since process start (the
// benchmark reports it).
unsigned long long fused_ops_launch_count();

} // namespace b200c
