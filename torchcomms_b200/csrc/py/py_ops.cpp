// Tensor-level bindings of the fused model kernels (`_comms.ops`).
#include "py_common.hpp"

#include <ATen/SavedTensorHooks.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>

#include "../cuda/driver_api.hpp"
#include "../kernels/fused_ops.h"
#include "../kernels/launch_count.h"
#include "../kernels/tc_gemm.h"
#include "plain_call.hpp"

namespace b200c {

namespace {

const __nv_bfloat16* bf(const at::Tensor& t) {
  return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr());
}
__nv_bfloat16* bf_mut(at::Tensor& t) {
  return reinterpret_cast<__nv_bfloat16*>(t.data_ptr());
}

void want(const at::Tensor& t, at::ScalarType dt, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.is_contiguous(), name, ": contiguous CUDA tensor expected");
  TORCH_CHECK(t.scalar_type() == dt, name, ": expected dtype ", dt, ", got ", t.scalar_type());
}

cudaStream_t cur(const at::Tensor& t) {
  return at::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

bool on16(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }
// The kernels take vectors of 16 bytes. A contiguous view at an odd storage offset (a narrow of a flat buffer, a slice
// of a gradient) does not start on such a boundary, and contiguous() leaves it where it is.
at::Tensor vectorable(const at::Tensor& t) { return on16(t) ? t : t.clone(at::MemoryFormat::Contiguous); }

// The two status words of one product, which its kernel clears. Whoever drops them sees a wait that ran out all the same: as NaN.
at::Tensor status_words(const at::Tensor& like) { return at::empty({2}, like.options().dtype(at::kInt)); }

bool quantizable(const at::Tensor& x) {
  return plain_call(x) && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.numel() > 0 && x.stride(1) == 1 &&
      x.size(0) <= INT32_MAX && x.size(1) <= INT32_MAX;
}
void quantize_into(const at::Tensor& x, at::Tensor& q, at::Tensor& scale) {
  B200C_CUDA_CHECK(launch_quantize_rows(bf(x), x.stride(0), q.data_ptr(), scale.data_ptr<float>(), static_cast<int>(x.size(0)),
                                        static_cast<int>(x.size(1)), cur(x)));
}

// x rotated, contiguous.
at::Tensor rope(const at::Tensor& x, const at::Tensor& pos, const at::Tensor& cos_t, const at::Tensor& sin_t, bool inverse) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16, "x: bf16 CUDA tensor expected");
  want(pos, at::kInt, "pos");
  want(cos_t, at::kFloat, "cos");
  want(sin_t, at::kFloat, "sin");
  TORCH_CHECK(x.dim() >= 3, "x must be [..., tokens, heads, head_dim]");
  const int head_dim = static_cast<int>(x.size(-1));
  const int heads = static_cast<int>(x.size(-2));
  const int64_t per_token = static_cast<int64_t>(head_dim) * heads;
  const int tokens = per_token == 0 ? 0 : static_cast<int>(x.numel() / per_token);
  TORCH_CHECK(pos.numel() == tokens, "pos must have one entry per token");
  TORCH_CHECK(cos_t.size(-1) == head_dim / 2 && sin_t.size(-1) == head_dim / 2, "cos/sin tables: [max_pos, head_dim/2]");
  c10::cuda::CUDAGuard g(x.device());
  at::Tensor y = at::empty_like(x, at::MemoryFormat::Contiguous);
  // A slice of a wider tensor (queries or keys of a fused projection) is read where it is; layouts that
  // 16-byte loads cannot follow are made contiguous first.
  const bool in_place = x.dim() == 3 && x.stride(2) == 1 && x.stride(0) % 8 == 0 && x.stride(1) % 8 == 0 && on16(x);
  const at::Tensor src = in_place ? x : x.clone(at::MemoryFormat::Contiguous);
  const int64_t st = in_place ? src.stride(0) : per_token, sh = in_place ? src.stride(1) : head_dim;
  const at::Tensor c = vectorable(cos_t), sn = vectorable(sin_t);
  B200C_CUDA_CHECK(launch_rope(bf(src), st, sh, bf_mut(y), pos.data_ptr<int>(), c.data_ptr<float>(), sn.data_ptr<float>(), tokens,
                               heads, head_dim, inverse, cur(x)));
  return y;
}

std::pair<at::Tensor, at::Tensor> rmsnorm_fwd(const at::Tensor& x, const at::Tensor& w, double eps) {
  want(x, at::kBFloat16, "x");
  want(w, at::kBFloat16, "w");
  const int cols = static_cast<int>(x.size(-1));
  const int rows = static_cast<int>(x.numel() / cols);
  TORCH_CHECK(w.numel() == cols, "weight must have ", cols, " elements");
  c10::cuda::CUDAGuard g(x.device());
  const at::Tensor xv = vectorable(x), wv = vectorable(w);
  at::Tensor y = at::empty_like(x);
  at::Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  B200C_CUDA_CHECK(launch_rmsnorm_fwd(bf(xv), bf(wv), bf_mut(y), rstd.data_ptr<float>(), rows, cols,
                                      static_cast<float>(eps), cur(x)));
  return std::make_pair(y, rstd);
}

std::pair<at::Tensor, at::Tensor> rmsnorm_bwd(const at::Tensor& dy, const at::Tensor& x, const at::Tensor& w,
                                              const at::Tensor& rstd) {
  want(dy, at::kBFloat16, "dy");
  want(x, at::kBFloat16, "x");
  want(w, at::kBFloat16, "w");
  want(rstd, at::kFloat, "rstd");
  const int cols = static_cast<int>(x.size(-1));
  const int rows = static_cast<int>(x.numel() / cols);
  c10::cuda::CUDAGuard g(x.device());
  int nblocks = 0;
  B200C_CUDA_CHECK(launch_rmsnorm_bwd(nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, &nblocks, rows, cols, cur(x)));
  const at::Tensor dyv = vectorable(dy), xv = vectorable(x), wv = vectorable(w);
  at::Tensor dx = at::empty_like(x);
  at::Tensor partial = at::empty({nblocks, cols}, x.options().dtype(at::kFloat));
  at::Tensor dw = at::empty_like(w);
  B200C_CUDA_CHECK(launch_rmsnorm_bwd(bf(dyv), bf(xv), bf(wv), rstd.data_ptr<float>(), bf_mut(dx),
                                      partial.data_ptr<float>(), &nblocks, rows, cols, cur(x)));
  B200C_CUDA_CHECK(launch_colsum_bf16(partial.data_ptr<float>(), bf_mut(dw), nblocks, cols, cur(x)));
  return std::make_pair(dx, dw);
}

at::Tensor swiglu_fwd(const at::Tensor& gate_up) {
  want(gate_up, at::kBFloat16, "gate_up");
  const int ffn = static_cast<int>(gate_up.size(-1) / 2);
  const int rows = static_cast<int>(gate_up.numel() / (2 * static_cast<int64_t>(ffn)));
  c10::cuda::CUDAGuard g(gate_up.device());
  auto sizes = gate_up.sizes().vec();
  sizes.back() = ffn;
  const at::Tensor guv = vectorable(gate_up);
  at::Tensor h = at::empty(sizes, gate_up.options());
  B200C_CUDA_CHECK(launch_swiglu_fwd(bf(guv), bf_mut(h), rows, ffn, cur(gate_up)));
  return h;
}

at::Tensor swiglu_bwd(const at::Tensor& dh, const at::Tensor& gate_up) {
  want(dh, at::kBFloat16, "dh");
  want(gate_up, at::kBFloat16, "gate_up");
  const int ffn = static_cast<int>(gate_up.size(-1) / 2);
  const int rows = static_cast<int>(gate_up.numel() / (2 * static_cast<int64_t>(ffn)));
  c10::cuda::CUDAGuard g(gate_up.device());
  const at::Tensor dhv = vectorable(dh), guv = vectorable(gate_up);
  at::Tensor d = at::empty_like(gate_up);
  B200C_CUDA_CHECK(launch_swiglu_bwd(bf(dhv), bf(guv), bf_mut(d), rows, ffn, cur(gate_up)));
  return d;
}

// Autograd nodes of the small model kernels. A Python autograd function costs several times what these kernels run
// for at ordinary sizes (its forward, and above all its backward, which takes the interpreter back onto the
// autograd engine's thread); the graph they record is the same. Host time of a forward and backward pass: norm 75 us,
// now 66; rotary embedding of queries and keys 97 us, now 87.
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct RmsNormFn : torch::autograd::Function<RmsNormFn> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& w, double eps) {
    auto [y, rstd] = rmsnorm_fwd(x, w, eps);
    ctx->save_for_backward({x, w, rstd});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    auto [dx, dw] = rmsnorm_bwd(grads[0].contiguous(), saved[0], saved[1], saved[2]);
    return {dx, dw, at::Tensor()};
  }
};

// The norm together with the residual stream it reads: (x, y) or, with a `delta` to add first, (x + delta, y). Both
// results' gradients meet inside the backward kernel instead of in an addition of their own.
bool norm_with_skip_applies(const at::Tensor& x, const at::Tensor& w) {
  return plain_call(x, true) && plain_call(w, true) && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 &&
      w.is_contiguous() && x.dim() >= 1 && x.size(-1) % 8 == 0 && x.size(-1) <= 8192 && x.numel() > 0 && w.numel() == x.size(-1) &&
      x.device() == w.device();
}

variable_list norm_with_skip_backward(const variable_list& grads, const variable_list& saved, at::Tensor* dw) {
  const at::Tensor &x = saved[0], &w = saved[1], &rstd = saved[2];
  const at::Tensor dskip = grads[0].contiguous(), dy = grads[1].contiguous();
  want(dskip, at::kBFloat16, "gradient of the residual");
  want(dy, at::kBFloat16, "dy");
  const int cols = static_cast<int>(x.size(-1)), rows = static_cast<int>(x.numel() / cols);
  c10::cuda::CUDAGuard g(x.device());
  int nblocks = 0;
  B200C_CUDA_CHECK(launch_rmsnorm_bwd(nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, &nblocks, rows, cols, cur(x)));
  const at::Tensor dyv = vectorable(dy), xv = vectorable(x), wv = vectorable(w), skip = vectorable(dskip);
  at::Tensor dx = at::empty_like(x);
  at::Tensor partial = at::empty({nblocks, cols}, x.options().dtype(at::kFloat));
  *dw = at::empty_like(w);
  B200C_CUDA_CHECK(launch_rmsnorm_bwd(bf(dyv), bf(xv), bf(wv), rstd.data_ptr<float>(), bf_mut(dx), partial.data_ptr<float>(), &nblocks,
                                      rows, cols, cur(x), bf(skip)));
  B200C_CUDA_CHECK(launch_colsum_bf16(partial.data_ptr<float>(), bf_mut(*dw), nblocks, cols, cur(x)));
  return {dx};
}

struct SkipRmsNormFn : torch::autograd::Function<SkipRmsNormFn> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& w, double eps) {
    auto [y, rstd] = rmsnorm_fwd(x, w, eps);
    ctx->save_for_backward({x, w, rstd});
    return {x, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    at::Tensor dw;
    const variable_list dx = norm_with_skip_backward(grads, ctx->get_saved_variables(), &dw);
    return {dx[0], dw, at::Tensor()};
  }
};

struct AddRmsNormFn : torch::autograd::Function<AddRmsNormFn> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& delta, const at::Tensor& w, double eps) {
    want(x, at::kBFloat16, "x");
    want(delta, at::kBFloat16, "delta");
    const int cols = static_cast<int>(x.size(-1)), rows = static_cast<int>(x.numel() / cols);
    c10::cuda::CUDAGuard g(x.device());
    const at::Tensor xv = vectorable(x), dv = vectorable(delta), wv = vectorable(w);
    at::Tensor sum = at::empty_like(x), y = at::empty_like(x);
    at::Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
    B200C_CUDA_CHECK(launch_rmsnorm_fwd(bf(xv), bf(wv), bf_mut(y), rstd.data_ptr<float>(), rows, cols, static_cast<float>(eps), cur(x),
                                        bf(dv), bf_mut(sum)));
    ctx->save_for_backward({sum, w, rstd});
    return {sum, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    at::Tensor dw;
    const variable_list dx = norm_with_skip_backward(grads, ctx->get_saved_variables(), &dw);
    return {dx[0], dx[0], dw, at::Tensor()};
  }
};

// Strides a split_rope launch can follow for [tokens, heads, head_dim].
bool followable(const at::Tensor& t) {
  return t.dim() == 3 && t.stride(2) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && on16(t);
}

struct SplitRopeFn : torch::autograd::Function<SplitRopeFn> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& qkv, const at::Tensor& pos, const at::Tensor& cos_t,
                               const at::Tensor& sin_t, int64_t heads, int64_t kv_heads) {
    ctx->save_for_backward({pos, cos_t, sin_t});
    const int64_t tokens = qkv.size(0), hd = qkv.size(1) / (heads + 2 * kv_heads);
    c10::cuda::CUDAGuard g(qkv.device());
    variable_list out{at::empty({tokens, heads, hd}, qkv.options()), at::empty({tokens, kv_heads, hd}, qkv.options()),
                      at::empty({tokens, kv_heads, hd}, qkv.options())};
    launch(qkv, out, pos, cos_t, sin_t, false);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    return {packed_gradient(std::move(grads), saved[0], saved[1], saved[2]), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
  // The gradient of the projection's output from those of queries, keys and values.
  static at::Tensor packed_gradient(variable_list grads, const at::Tensor& pos, const at::Tensor& cos_t, const at::Tensor& sin_t) {
    for (auto& t : grads) {
      if (!followable(t)) t = t.clone(at::MemoryFormat::Contiguous);
      TORCH_CHECK(t.scalar_type() == at::kBFloat16, "split_rope: bf16 gradients expected");
    }
    c10::cuda::CUDAGuard g(grads[0].device());
    at::Tensor dqkv = at::empty({grads[0].size(0), (grads[0].size(1) + 2 * grads[1].size(1)) * grads[0].size(2)}, grads[0].options());
    launch(dqkv, grads, pos, cos_t, sin_t, true);
    return dqkv;
  }
  static void launch(const at::Tensor& packed, const variable_list& part, const at::Tensor& pos, const at::Tensor& cos_t,
                     const at::Tensor& sin_t, bool backward) {
    __nv_bfloat16* p[3];
    int64_t st[3], sh[3];
    for (int i = 0; i < 3; ++i) {
      p[i] = reinterpret_cast<__nv_bfloat16*>(part[i].data_ptr());
      st[i] = part[i].stride(0);
      sh[i] = part[i].stride(1);
    }
    B200C_CUDA_CHECK(launch_split_rope(reinterpret_cast<__nv_bfloat16*>(packed.data_ptr()), packed.stride(0), p, st, sh,
                                       pos.data_ptr<int>(), cos_t.data_ptr<float>(), sin_t.data_ptr<float>(),
                                       static_cast<int>(packed.size(0)), static_cast<int>(part[0].size(1)),
                                       static_cast<int>(part[1].size(1)), static_cast<int>(part[0].size(2)), backward, cur(packed)));
  }
  static bool applies(const at::Tensor& qkv, const at::Tensor& pos, const at::Tensor& cos_t, const at::Tensor& sin_t, int64_t heads,
                      int64_t kv_heads) {
    return plain_call(qkv, true) && qkv.dim() == 2 && qkv.numel() > 0 && qkv.scalar_type() == at::kBFloat16 && qkv.stride(1) == 1 &&
        qkv.stride(0) % 8 == 0 && on16(qkv) && heads >= 1 && kv_heads >= 1 &&
        applies_to(qkv.size(0), qkv.size(1), qkv.device(), pos, cos_t, sin_t, heads, kv_heads);
  }
  // The same for a projection that is yet to be made, contiguous.
  static bool applies_to(int64_t tokens, int64_t cols, at::Device device, const at::Tensor& pos, const at::Tensor& cos_t,
                         const at::Tensor& sin_t, int64_t heads, int64_t kv_heads) {
    if (!plain_call(pos) || !plain_call(cos_t) || !plain_call(sin_t) || cols % (8 * (heads + 2 * kv_heads)) != 0) return false;
    const int64_t hd = cols / (heads + 2 * kv_heads);
    auto table = [&](const at::Tensor& t) {
      return t.scalar_type() == at::kFloat && t.is_contiguous() && t.dim() == 2 && t.size(1) == hd / 2 && t.device() == device && on16(t);
    };
    return table(cos_t) && table(sin_t) && pos.scalar_type() == at::kInt && pos.is_contiguous() && pos.numel() == tokens && pos.device() == device;
  }
};

struct SwiGluFn : torch::autograd::Function<SwiGluFn> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& gate_up) {
    ctx->save_for_backward({gate_up});
    return swiglu_fwd(gate_up);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return {swiglu_bwd(grads[0].contiguous(), ctx->get_saved_variables()[0])};
  }
};

struct RopeFn : torch::autograd::Function<RopeFn> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& pos, const at::Tensor& cos_t,
                            const at::Tensor& sin_t) {
    ctx->save_for_backward({pos, cos_t, sin_t});
    return rope(x, pos, cos_t, sin_t, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    return {rope(grads[0], saved[0], saved[1], saved[2], true), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

// The two halves of a decoder block around its attention, as one node each: what the separate nodes of norms, projections,
// rotary embedding and activation launch, without an allocation, a graph edge and a trip through the engine for each, and with
// the activation in its projection's epilogue. Both take what those nodes take: contiguous bf16 matrices on the
// 16-byte grid, widths that are multiples of 8. Backward they make what is asked for and what that takes, as the engine does of
// separate nodes.
bool block_matrix(const at::Tensor& t, int64_t rows, int64_t cols, const at::Tensor& like) {
  return plain_call(t, true) && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.size(0) == rows && t.size(1) == cols &&
      t.is_contiguous() && on16(t) && t.device() == like.device();
}
// Pairs work in units of 256 rows, the tensor library's kernels in finer ones: whether rows fill theirs to so many percent.
bool filled(int64_t rows, int percent) { return rows * 100 >= (rows + 255) / 256 * 256 * percent; }
bool mostly_empty_rows(int64_t rows) { return rows > 128 && !filled(rows, 70); }
constexpr int64_t kLargeWeight = 12 << 20;
// x w^T of contiguous matrices on the 16-byte grid, widths multiples of 8: this library's product, whose call costs half the
// tensor library's host time (6.5 and 11.5 us) and which starts early, up to a depth of 4096 (deeper sums that fill the GPU less
// than once the tensor library splits better), where that is most of it or units of 256 rows are nine tenths full, and of large
// weights from 450 rows on. In us, both from the host over weights from DRAM, the library's / this one's: 64 x 2048 x 2048 10.0 / 7.7,
// 1000 x 3072 x 2048 13.1 / 13.1, 1552 x 2048 x 2048 17 / 21; 160 x 6144 x 4096 16 / 23, 520 25 / 33, 784 38 / 45, 1000 45 / 47, 1288 59 / 63,
// 1536 68 / 66, 4096 169 / 150; 304 x 4096 x 4096 15 / 19, 1552 52 / 61, 4096 114 / 100.
at::Tensor product(const at::Tensor& x, const at::Tensor& w) {
  const int64_t m = x.size(0), n = w.size(0), k = x.size(1);
  const bool own = k <= 4096 && (n * k > kLargeWeight ? m >= 450 && filled(m, 90) : m * n * k <= 6000000000 || filled(m, 90));
  if (!own) return at::mm(x, w.t());
  at::Tensor y = at::empty({m, n}, x.options()), status = status_words(x);
  B200C_CUDA_CHECK(launch_gemm_bf16_nt(x.data_ptr(), w.data_ptr(), y.data_ptr(), static_cast<int>(m), static_cast<int>(n), static_cast<int>(k),
                                       reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(x)));
  return y;
}
// (x w^T, its activation): in one kernel, but of large weights for up to 128 rows and where units of 256 rows are too empty: less
// than 77 % full, from 768 rows on, where the activation kernel is less of it, 83 %. In us, the tensor library's product and the
// activation kernel / one kernel: 64 x 14336 x 4096 49 / 53, 160 54 / 56, 208 61 / 57, 304 74 / 86, 400 92 / 90, 568 115 / 132, 592
// 172 / 138, 784 159 / 173, 832 184 / 174, 1032 214 / 227, 1288 267 / 254; 64 x 8192 x 2048 20 / 26, 208 24 / 25, 304 31 / 35, 592 41 / 40.
std::pair<at::Tensor, at::Tensor> gated_product(const at::Tensor& x, const at::Tensor& w) {
  const int64_t m = x.size(0), n = w.size(0) / 2, k = x.size(1);
  if (2 * n * k > kLargeWeight && (m <= 128 || !filled(m, m < 768 ? 77 : 83))) {
    at::Tensor gate_up = product(x, w);
    at::Tensor act = swiglu_fwd(gate_up);
    return {gate_up, act};
  }
  at::Tensor gate_up = at::empty({m, 2 * n}, x.options()), act = at::empty({m, n}, x.options()), status = status_words(x);
  B200C_CUDA_CHECK(launch_gemm_gated(x.data_ptr(), w.data_ptr(), gate_up.data_ptr(), act.data_ptr(), static_cast<int>(m), static_cast<int>(n),
                                     static_cast<int>(k), reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(x)));
  return {gate_up, act};
}
// Which products of a backward pass this library makes. With K in both operands' rows (a weight's gradient): all but those of
// few tiles and a long sum, which the tensor library shares out. With K in A's columns (an input's): short sums, which end
// before the next call is made, and from 700 rows on those of up to 96 steps, or 48 where the tiles are few. In us, both from
// the host, the tensor library's / this one's: weights' gradients (columns x columns, rows) 512 x 512, 64 11.1 / 5.7; 28672 x 4096, 1000
// 183 / 156; 4096 x 14336, 4096 324 / 290; 512 x 512, 4096 11.3 / 13.8. Inputs' gradients (rows x K x columns) 64 x 2048 x 8192 11.6 / 10.6,
// 1000 x 4096 x 14336 82.4 / 82.8, 4096 x 4096 x 14336 319 / 294; 300 x 3072 x 2048 9.0 / 12.1, 1000 x 4096 x 512 13.9 / 15.2, 64 x 28672 x
// 4096 42 / 94.
constexpr int64_t kKStep = 64;
bool few_tiles(int64_t m, int64_t n) { return pair_tiles_fit(static_cast<int>(m), static_cast<int>(n), false); }
bool own_by_columns(int64_t m, int64_t n, int64_t k) { return !few_tiles(m, n) || k <= 48 * kKStep; }
bool own_by_rows(int64_t m, int64_t n, int64_t k) {
  if (mostly_empty_rows(m) && n * k > kLargeWeight) return false;
  return k <= 32 * kKStep || (m >= 700 && k <= (few_tiles(m, n) ? 48 : 96) * kKStep);
}
// Elements from row to row. A single row is contiguous whatever its stride says, and then that means nothing.
int64_t row_stride(const at::Tensor& t) { return t.size(0) > 1 ? t.stride(0) : (t.size(1) + 7) / 8 * 8; }
void mn_product_into(at::Tensor& c, const at::Tensor& a, bool by_columns, const at::Tensor& b) {
  at::Tensor status = status_words(b);
  B200C_CUDA_CHECK(launch_gemm_pair_mn(a.data_ptr(), row_stride(a), by_columns, b.data_ptr(), row_stride(b), c.data_ptr(),
                                       static_cast<int>(c.size(0)), static_cast<int>(c.size(1)), static_cast<int>(b.size(0)),
                                       reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(b)));
}
// dy [rows, n] w [n, k] and dy^T x [rows, k], the gradients of a product's operands. The tensor library's where a mode watches the
// backward pass, or a hook has put something else in a tensor's place.
bool plain_rows(const at::Tensor& t, const at::Tensor& like) {
  return plain_call(t) && block_matrix(t, t.size(0), t.size(1), like) && t.size(1) % 8 == 0;
}
at::Tensor input_gradient(const at::Tensor& dy, const at::Tensor& w) {
  if (!plain_rows(dy, dy) || !plain_rows(w, dy) || dy.size(1) != w.size(0) || !own_by_rows(dy.size(0), w.size(1), w.size(0))) {
    return at::mm(dy, w);
  }
  at::Tensor dx = at::empty({dy.size(0), w.size(1)}, w.options());
  mn_product_into(dx, dy, false, w);
  return dx;
}
// The gradient of [gate, up] from that of silu(gate) * up w^T. Where this library makes the product, its epilogue does the rest,
// but for few rows of large weights, whose only tiles end in that epilogue. In us, dy [rows, k] w [k, n], the tensor library's product
// and the kernel / this library's and the kernel / one kernel: 4096 x 4096 x 14336 504 / 512 / 385, 1000 124 / 129 / 112; 2048 x 2048 x
// 8192 96 / 90 / 67, 64 13.7 / 14.3 / 15.9; 1000 x 512 x 2048 13.6 / 10.6 / 9.3.
at::Tensor gated_gradient(const at::Tensor& dy, const at::Tensor& w, const at::Tensor& gate_up) {
  const int64_t m = dy.size(0), n = w.size(1), k = w.size(0);
  if (!plain_rows(dy, dy) || !plain_rows(w, dy) || !plain_rows(gate_up, dy) || dy.size(1) != k || gate_up.size(0) != m ||
      gate_up.size(1) != 2 * n || !own_by_rows(m, n, k) || (m <= 128 && n * k > kLargeWeight)) {
    return swiglu_bwd(input_gradient(dy, w), gate_up);
  }
  at::Tensor d = at::empty_like(gate_up), status = status_words(dy);
  B200C_CUDA_CHECK(launch_gemm_gated_grad(dy.data_ptr(), w.data_ptr(), gate_up.data_ptr(), d.data_ptr(), static_cast<int>(m), static_cast<int>(n),
                                          static_cast<int>(k), reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(dy)));
  return d;
}
at::Tensor weight_gradient(const at::Tensor& dy, const at::Tensor& x) {
  if (!plain_rows(dy, dy) || !plain_rows(x, dy) || dy.size(0) != x.size(0) || !own_by_columns(dy.size(1), x.size(1), x.size(0))) {
    return at::mm(dy.t(), x);
  }
  at::Tensor dw = at::empty({dy.size(1), x.size(1)}, x.options());
  mn_product_into(dw, dy, true, x);
  return dw;
}

// A backward pass that is itself differentiated needs its gradients' history, which the nodes below do not have: what they keep was
// made inside them. There the separate nodes run once more, on the arguments, and the engine differentiates them: the history, and
// the limits (a norm's or an activation's gradient has none), of a block made of them. `forward` gets the arguments under other
// names, so that nothing is counted twice where one argument was made from another.
template <typename F>
variable_list gradients_with_history(AutogradContext* ctx, const std::vector<at::Tensor>& args, variable_list grads, F&& forward) {
  std::vector<at::Tensor> own(args.size());
  variable_list wanted, out(args.size());
  for (size_t i = 0; i < args.size(); ++i) {
    own[i] = args[i].view_as(args[i]);
    if (ctx->needs_input_grad(i)) wanted.push_back(own[i]);
  }
  variable_list results, of_results;
  const variable_list all = forward(own);
  for (size_t i = 0; i < all.size(); ++i) {
    if (!all[i].requires_grad()) continue;  // the residual stream where only the projection is trained
    results.push_back(all[i]);
    of_results.push_back(grads[i]);
  }
  const variable_list made = torch::autograd::grad(results, wanted, of_results, /*retain_graph=*/std::nullopt, /*create_graph=*/true,
                                                   /*allow_unused=*/true);
  for (size_t i = 0, j = 0; i < args.size(); ++i) {
    if (ctx->needs_input_grad(i)) out[i] = made[j++];
  }
  return out;
}

// (x, queries, keys, values) of x [tokens, dim]: norm, fused projection, rotary embedding. x is returned for the residual.
struct BlockInFn : torch::autograd::Function<BlockInFn> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& norm, const at::Tensor& wqkv,
                               const at::Tensor& pos, const at::Tensor& cos_t, const at::Tensor& sin_t, int64_t heads, int64_t kv_heads,
                               double eps) {
    auto [h, rstd] = rmsnorm_fwd(x, norm, eps);
    c10::cuda::CUDAGuard g(x.device());
    const at::Tensor qkv = product(h, wqkv);
    const int64_t tokens = x.size(0), hd = wqkv.size(0) / (heads + 2 * kv_heads);
    variable_list out{at::empty({tokens, heads, hd}, x.options()), at::empty({tokens, kv_heads, hd}, x.options()),
                      at::empty({tokens, kv_heads, hd}, x.options())};
    SplitRopeFn::launch(qkv, out, pos, cos_t, sin_t, false);
    const at::Tensor none;
    ctx->save_for_backward({x, norm, rstd, wqkv.requires_grad() ? h : none, wqkv, pos, cos_t, sin_t});
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["kv_heads"] = kv_heads;
    ctx->saved_data["eps"] = eps;
    return {x, out[0], out[1], out[2]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &h = saved[3], &wqkv = saved[4];
    if (c10::GradMode::is_enabled()) {
      variable_list out = gradients_with_history(ctx, {saved[0], saved[1], wqkv}, grads, [&](const std::vector<at::Tensor>& a) {
        const variable_list normed = SkipRmsNormFn::apply(a[0], a[1], ctx->saved_data["eps"].toDouble());
        variable_list parts = SplitRopeFn::apply(at::linear(normed[1], a[2]), saved[5], saved[6], saved[7], ctx->saved_data["heads"].toInt(),
                                                 ctx->saved_data["kv_heads"].toInt());
        parts.insert(parts.begin(), normed[0]);
        return parts;
      });
      out.resize(9);
      return out;
    }
    const at::Tensor dqkv = SplitRopeFn::packed_gradient({grads[1], grads[2], grads[3]}, saved[5], saved[6], saved[7]);
    const at::Tensor dw = ctx->needs_input_grad(2) ? weight_gradient(dqkv, h) : at::Tensor();
    at::Tensor dx, dnorm;
    if (ctx->needs_input_grad(0) || ctx->needs_input_grad(1)) {
      dx = norm_with_skip_backward({grads[0], input_gradient(dqkv, wqkv)}, {saved[0], saved[1], saved[2]}, &dnorm)[0];
    }
    return {dx, dnorm, dw, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
  static bool applies(const at::Tensor& x, const at::Tensor& norm, const at::Tensor& wqkv, const at::Tensor& pos, const at::Tensor& cos_t,
                      const at::Tensor& sin_t, int64_t heads, int64_t kv_heads) {
    if (heads < 1 || kv_heads < 1 || at::autocast::is_autocast_enabled(at::kCUDA) || !norm_with_skip_applies(x, norm)) return false;
    return x.dim() == 2 && block_matrix(x, x.size(0), x.size(1), x) && wqkv.dim() == 2 && block_matrix(wqkv, wqkv.size(0), x.size(1), x) &&
        SplitRopeFn::applies_to(x.size(0), wqkv.size(0), x.device(), pos, cos_t, sin_t, heads, kv_heads);
  }
};

// x + o wo^T, and on it the norm and the gated MLP: y = s + (silu(gate) * up) w2^T, [gate, up] = norm(s) w13^T, s = x + o wo^T.
struct BlockOutFn : torch::autograd::Function<BlockOutFn> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& o, const at::Tensor& wo, const at::Tensor& norm,
                            const at::Tensor& w13, const at::Tensor& w2, double eps) {
    const int cols = static_cast<int>(x.size(1)), rows = static_cast<int>(x.size(0));
    c10::cuda::CUDAGuard g(x.device());
    const at::Tensor delta = product(o, wo);
    at::Tensor sum = at::empty_like(x), h = at::empty_like(x), rstd = at::empty({rows}, x.options().dtype(at::kFloat));
    B200C_CUDA_CHECK(launch_rmsnorm_fwd(bf(x), bf(norm), bf_mut(h), rstd.data_ptr<float>(), rows, cols, static_cast<float>(eps), cur(x),
                                        bf(delta), bf_mut(sum)));
    const auto [gate_up, act] = gated_product(h, w13);
    at::Tensor y = product(act, w2);
    y.add_(sum);
    // What was made on the way is kept for whoever has a gradient that takes it.
    const at::Tensor none;
    const bool sum_wanted = x.requires_grad() || o.requires_grad() || wo.requires_grad() || norm.requires_grad();
    ctx->save_for_backward({sum_wanted ? sum : none, norm, rstd, o, wo, w13.requires_grad() ? h : none, w13,
                            sum_wanted || w13.requires_grad() ? gate_up : none, w2.requires_grad() ? act : none, w2, x});
    ctx->saved_data["eps"] = eps;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &o = saved[3], &wo = saved[4], &h = saved[5], &w13 = saved[6], &gate_up = saved[7], &act = saved[8], &w2 = saved[9];
    if (c10::GradMode::is_enabled()) {
      variable_list out = gradients_with_history(ctx, {saved[10], o, wo, saved[1], w13, w2}, grads, [&](const std::vector<at::Tensor>& a) {
        const variable_list normed = AddRmsNormFn::apply(a[0], at::linear(a[1], a[2]), a[3], ctx->saved_data["eps"].toDouble());
        return variable_list{normed[0] + at::linear(SwiGluFn::apply(at::linear(normed[1], a[4])), a[5])};
      });
      out.resize(7);
      return out;
    }
    const at::Tensor dy = grads[0].contiguous();
    c10::cuda::CUDAGuard g(dy.device());
    at::Tensor ds, d_o, dwo, dnorm, dw13, dw2;
    if (ctx->needs_input_grad(5)) dw2 = weight_gradient(dy, act);
    const bool sum_wanted = ctx->needs_input_grad(0) || ctx->needs_input_grad(1) || ctx->needs_input_grad(2) || ctx->needs_input_grad(3);
    if (sum_wanted || ctx->needs_input_grad(4)) {
      const at::Tensor dgate_up = gated_gradient(dy, w2, gate_up);
      if (ctx->needs_input_grad(4)) dw13 = weight_gradient(dgate_up, h);
      if (sum_wanted) ds = norm_with_skip_backward({dy, input_gradient(dgate_up, w13)}, {saved[0], saved[1], saved[2]}, &dnorm)[0];
    }
    if (ctx->needs_input_grad(2)) dwo = weight_gradient(ds, o);
    if (ctx->needs_input_grad(1)) d_o = input_gradient(ds, wo);
    return {ds, d_o, dwo, dnorm, dw13, dw2, at::Tensor()};
  }
  static bool applies(const at::Tensor& x, const at::Tensor& o, const at::Tensor& wo, const at::Tensor& norm, const at::Tensor& w13,
                      const at::Tensor& w2) {
    if (at::autocast::is_autocast_enabled(at::kCUDA) || !norm_with_skip_applies(x, norm) || x.dim() != 2 || o.dim() != 2 || w2.dim() != 2) {
      return false;
    }
    const int64_t rows = x.size(0), dim = x.size(1), ffn = w2.size(1);
    return ffn > 0 && ffn % 8 == 0 && o.size(1) > 0 && o.size(1) % 8 == 0 && rows <= INT32_MAX / 2 && ffn <= INT32_MAX / 2 && block_matrix(x, rows, dim, x) &&
        block_matrix(o, rows, o.size(1), x) && block_matrix(wo, dim, o.size(1), x) && block_matrix(w13, 2 * ffn, dim, x) &&
        block_matrix(w2, dim, ffn, x);
  }
};

// Loss and gradients of a head, (loss, dx, dweight), on the framework's own logits kernel. Logits have rows of whole
// 128-byte lines, so that every vocabulary's products are tiled ones: at odd row strides the tensor library's fall
// back to two-element accesses. x: [rows, dim].
bool head_applies(const at::Tensor& x, const at::Tensor& weight, const at::Tensor& targets, int64_t chunk_rows) {
  auto matrix = [&](const at::Tensor& t) {
    return plain_call(t) && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.is_contiguous() && on16(t) && t.device() == x.device();
  };
  return matrix(x) && matrix(weight) && x.size(1) == weight.size(1) && x.size(1) % 8 == 0 && x.numel() > 0 && weight.size(0) > 0 &&
      x.size(0) <= INT32_MAX && x.size(1) <= INT32_MAX && weight.size(0) <= INT32_MAX - 256 && chunk_rows >= 1 &&
      !at::autocast::is_autocast_enabled(at::kCUDA) && plain_call(targets) && targets.scalar_type() == at::kLong &&
      targets.dim() == 1 && targets.size(0) == x.size(0) && targets.is_contiguous() && targets.device() == x.device();
}

// Whether the logits are this library's product, with their statistics: but for large weights where half of a pair's rows would be
// empty, or with more than a unit of 256 rows and 15 % of all, of widths beyond 2048 5 %. The tensor library's product and the
// kernel with two looks take as long then or less. A pass of the head in us, that way / this library's, rows x width x vocabulary:
// 64 x 4096 x 128256 608 / 645, 128 x 2048 x 128256 390 / 397, 128 x 4096 x 32000 215 / 212, 32 x 2048 x 50256 185 / 152; 400 x 4096 x
// 128256 1346 / 1400, 700 1954 / 1994, 200 909 / 910, 512 1520 / 1513, 400 x 4096 x 32000 365 / 376, 1300 889 / 899; 700 x 2048 x
// 128256 1130 / 1123, 400 x 2048 x 50256 304 / 306, 1300 792 / 763.
bool own_logits(int64_t rows, int64_t vocab, int64_t dim) {
  const int64_t weight = vocab * dim;
  if (rows <= 256) return rows > 128 || weight <= 128 << 20;
  return rows * 20 >= (rows + 255) / 256 * 256 * (dim > 2048 ? 19 : 17) || (weight <= 128 << 20 && (dim <= 2048 || weight <= 64 << 20));
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> head(const at::Tensor& x, const at::Tensor& weight, const at::Tensor& targets,
                                                    int64_t chunk_rows) {
  c10::cuda::CUDAGuard g(x.device());
  const int64_t rows = x.size(0), dim = x.size(1), vocab = weight.size(0), chunk = std::min(rows, chunk_rows), ld = (vocab + 63) / 64 * 64;
  at::Tensor dx = at::empty_like(x), dw = at::empty_like(weight), loss = at::empty({}, x.options().dtype(at::kFloat));
  const at::Tensor logits = at::empty({chunk, ld}, x.options());
  // Statistics and what the loss's sums have more (the last chunk may take narrower tiles), then a target's logit and two words of
  // scratch per row, then the kernels' words.
  const int64_t last = rows - (rows - 1) / chunk * chunk;
  const int64_t shares = std::max(chunk * head_row_shares(static_cast<int>(chunk), static_cast<int>(vocab)),
                                  last * head_row_shares(static_cast<int>(last), static_cast<int>(vocab)));
  const at::Tensor scratch = at::empty({3 * shares + 3 * chunk + 4}, x.options().dtype(at::kFloat));
  float *stats = scratch.data_ptr<float>(), *fine = stats + 2 * shares;
  float *target_logit = fine + shares, *row_scratch = target_logit + chunk;
  auto* words = reinterpret_cast<uint32_t*>(row_scratch + 2 * chunk);
  const float mean = 1.0f / static_cast<float>(rows);
  for (int64_t r0 = 0; r0 < rows; r0 += chunk) {
    const int n = static_cast<int>(std::min(chunk, rows - r0));
    const int64_t* t = targets.data_ptr<int64_t>() + r0;
    const at::Tensor xs = r0 == 0 && n == rows ? x : x.narrow(0, r0, n);
    at::Tensor dxs = r0 == 0 && n == rows ? dx : dx.narrow(0, r0, n);
    auto* z = reinterpret_cast<__nv_bfloat16*>(logits.data_ptr());
    at::Tensor grad = logits.as_strided({n, vocab}, {ld, 1});
    if (own_logits(n, vocab, dim)) {
      B200C_CUDA_CHECK(launch_head_logits(xs.data_ptr(), weight.data_ptr(), z, ld, t, n, static_cast<int>(vocab), static_cast<int>(dim),
                                          reinterpret_cast<float2*>(stats), fine, target_logit, words, cur(x)));
      B200C_CUDA_CHECK(launch_head_gradient(z, ld, t, reinterpret_cast<float2*>(stats), fine, head_row_shares(n, static_cast<int>(vocab)),
                                            target_logit, row_scratch, loss.data_ptr<float>(), words, n, static_cast<int>(vocab), mean, mean,
                                            r0 == 0, cur(x)));
    } else {
      at::mm_out(grad, xs, weight.t());
      B200C_CUDA_CHECK(launch_cross_entropy_fwd_bwd(z, ld, t, row_scratch, n, static_cast<int>(vocab), mean, cur(x)));
      const at::Tensor sum = scratch.narrow(0, row_scratch - stats, n).sum().mul_(mean);
      if (r0 == 0) loss = sum;
      else loss.add_(sum);
    }
    // A depth that is no multiple of 8 costs the tensor library's product its tiled loads: the last few columns are added to its
    // fp32 result.
    const int64_t even = vocab / 8 * 8;
    if (own_by_rows(n, dim, vocab)) {
      mn_product_into(dxs, grad, false, weight);
    } else if (even == vocab || even == 0) {
      at::mm_out(dxs, grad, weight);
    } else {
      const at::Tensor part = at::mm(grad.narrow(1, 0, even), weight.narrow(0, 0, even), at::kFloat);
      B200C_CUDA_CHECK(launch_head_tail(part.data_ptr<float>(), z + even, ld, bf(weight) + even * dim, bf_mut(dxs), n, static_cast<int>(dim),
                                        static_cast<int>(vocab - even), cur(x)));
    }
    if (r0 == 0) at::mm_out(dw, grad.t(), xs);  // the first chunk needs no zeroed gradient to add to
    else dw.addmm_(grad.t(), xs);
  }
  return {loss, dx, dw};
}

} // namespace

void bind_ops(py::module_& m) {
  auto ops = m.def_submodule("ops", "fused sm_100a model kernels");

  // Points the storage behind `t` (and so every view of it, including tensors
  // autograd saved) at the memory of `src`, or at nothing. The storage keeps
  // `src` alive. This is how a stage's flat parameter buffer moves between
  // rotating communication buffers without its parameter views being rebuilt.
  ops.def("rebind_storage_", [](at::Tensor t, std::optional<at::Tensor> src) {
    c10::StorageImpl* impl = t.storage().unsafeGetStorageImpl();
    if (!src.has_value()) {
      impl->set_data_ptr_noswap(at::DataPtr(nullptr, t.device()));
      impl->set_nbytes(0);
      return;
    }
    TORCH_CHECK(src->is_contiguous() && src->device() == t.device(), "rebind_storage_: contiguous source on the same device");
    auto* keep = new at::Tensor(*src);
    impl->set_data_ptr_noswap(
        at::DataPtr(src->data_ptr(), keep, [](void* ctx) { delete static_cast<at::Tensor*>(ctx); }, t.device()));
    impl->set_nbytes(src->nbytes());
  }, py::arg("tensor"), py::arg("source") = py::none());

  ops.def("rmsnorm_fwd", &rmsnorm_fwd);
  ops.def("rmsnorm_bwd", &rmsnorm_bwd);

  // x [..., tokens, heads, head_dim] of any strides -> contiguous.
  ops.def("rope", &rope);

  ops.def("swiglu_fwd", &swiglu_fwd);
  ops.def("swiglu_bwd", &swiglu_bwd);

  // The differentiable forms as native autograd nodes, or None where something other than plain autograd wants to
  // see the operation (functorch transforms, forward mode, dispatch and function modes, tracing): the caller then
  // takes the autograd function written in Python.
  ops.def("rms_norm", [](const at::Tensor& x, const at::Tensor& w, double eps) -> std::optional<at::Tensor> {
    if (!plain_call(x, true) || !plain_call(w, true)) return std::nullopt;
    return RmsNormFn::apply(x.contiguous(), w, eps);
  });
  ops.def("rms_norm_skip", [](const at::Tensor& x, const at::Tensor& w, double eps) -> std::optional<std::vector<at::Tensor>> {
    if (!norm_with_skip_applies(x, w)) return std::nullopt;
    return SkipRmsNormFn::apply(x.contiguous(), w, eps);
  });
  ops.def("add_rms_norm", [](const at::Tensor& x, const at::Tensor& delta, const at::Tensor& w, double eps)
              -> std::optional<std::vector<at::Tensor>> {
    if (!norm_with_skip_applies(x, w) || !plain_call(delta, true) || delta.scalar_type() != at::kBFloat16 ||
        delta.sizes() != x.sizes() || delta.device() != x.device()) {
      return std::nullopt;
    }
    return AddRmsNormFn::apply(x.contiguous(), delta.contiguous(), w, eps);
  });
  ops.def("split_rope", [](const at::Tensor& qkv, const at::Tensor& pos, const at::Tensor& cos_t, const at::Tensor& sin_t,
                           int64_t heads, int64_t kv_heads) -> std::optional<std::vector<at::Tensor>> {
    if (!SplitRopeFn::applies(qkv, pos, cos_t, sin_t, heads, kv_heads)) return std::nullopt;
    return SplitRopeFn::apply(qkv, pos, cos_t, sin_t, heads, kv_heads);
  });
  ops.def("block_in", [](const at::Tensor& x, const at::Tensor& norm, const at::Tensor& wqkv, const at::Tensor& pos, const at::Tensor& cos_t,
                         const at::Tensor& sin_t, int64_t heads, int64_t kv_heads, double eps) -> std::optional<std::vector<at::Tensor>> {
    if (!BlockInFn::applies(x, norm, wqkv, pos, cos_t, sin_t, heads, kv_heads)) return std::nullopt;
    return BlockInFn::apply(x, norm, wqkv, pos, cos_t, sin_t, heads, kv_heads, eps);
  });
  ops.def("block_out", [](const at::Tensor& x, const at::Tensor& o, const at::Tensor& wo, const at::Tensor& norm, const at::Tensor& w13,
                          const at::Tensor& w2, double eps) -> std::optional<at::Tensor> {
    if (!BlockOutFn::applies(x, o, wo, norm, w13, w2)) return std::nullopt;
    return BlockOutFn::apply(x, o, wo, norm, w13, w2, eps);
  });
  ops.def("swiglu", [](const at::Tensor& gate_up) -> std::optional<at::Tensor> {
    if (!plain_call(gate_up, true)) return std::nullopt;
    return SwiGluFn::apply(gate_up.contiguous());
  });
  ops.def("apply_rope", [](const at::Tensor& x, const at::Tensor& pos, const at::Tensor& cos_t, const at::Tensor& sin_t)
              -> std::optional<at::Tensor> {
    if (!plain_call(x, true) || !plain_call(pos) || !plain_call(cos_t) || !plain_call(sin_t)) return std::nullopt;
    return RopeFn::apply(x, pos, cos_t, sin_t);
  });

  ops.def("cross_entropy_fwd_bwd_", [](at::Tensor logits, const at::Tensor& targets, double grad_scale) {
    // Contiguous, or rows of a wider buffer.
    const bool padded = logits.dim() == 2 && logits.stride(1) == 1 && logits.stride(0) >= logits.size(1);
    TORCH_CHECK(logits.is_cuda() && (padded || logits.is_contiguous()), "logits: contiguous CUDA tensor expected");
    TORCH_CHECK(logits.scalar_type() == at::kBFloat16, "logits: expected dtype ", at::kBFloat16, ", got ", logits.scalar_type());
    want(targets, at::kLong, "targets");
    const int vocab = static_cast<int>(logits.size(-1));
    const int64_t ld = padded ? logits.stride(0) : vocab;
    const int rows = static_cast<int>(logits.numel() / vocab);
    TORCH_CHECK(targets.numel() == rows, "one target per row");
    c10::cuda::CUDAGuard g(logits.device());
    at::Tensor loss = at::empty({rows}, logits.options().dtype(at::kFloat));
    B200C_CUDA_CHECK(launch_cross_entropy_fwd_bwd(bf_mut(logits), ld, targets.data_ptr<int64_t>(), loss.data_ptr<float>(), rows,
                                                  vocab, static_cast<float>(grad_scale), cur(logits)));
    return loss;
  });

  // (loss, dx, dweight) of a head, or None where its kernels do not apply.
  ops.def("head", [](const at::Tensor& x, const at::Tensor& weight, const at::Tensor& targets, int64_t chunk_rows)
              -> std::optional<std::tuple<at::Tensor, at::Tensor, at::Tensor>> {
    if (!head_applies(x, weight, targets, chunk_rows)) return std::nullopt;
    return head(x, weight, targets, chunk_rows);
  });

  // t * factor.to(t.dtype) for a 0-d factor on the device (the gradient of a loss). `consume`: nobody reads t
  // afterwards, so the product may take its place. scale_both_by: two tensors by one factor, in one launch.
  static const auto scalable = [](const at::Tensor& t, const at::Tensor& factor) {
    return plain_call(t) && plain_call(factor) && t.scalar_type() == at::kBFloat16 && t.is_non_overlapping_and_dense() && on16(t) &&
        factor.dim() == 0 && factor.scalar_type() == at::kFloat && factor.device() == t.device();
  };
  ops.def("scale_both_by", [](const at::Tensor& t, const at::Tensor& u, const at::Tensor& factor, bool consume) {
    if (!scalable(t, factor) || !scalable(u, factor)) return std::make_pair(t * factor.to(t.scalar_type()), u * factor.to(u.scalar_type()));
    c10::cuda::CUDAGuard g(t.device());
    at::Tensor a = consume ? t : at::empty_like(t), b = consume ? u : at::empty_like(u);
    B200C_CUDA_CHECK(launch_scale_bf16(bf(t), bf_mut(a), factor.data_ptr<float>(), static_cast<size_t>(t.numel()), cur(t), bf(u), bf_mut(b),
                                       static_cast<size_t>(u.numel())));
    return std::make_pair(a, b);
  });
  ops.def("scale_by", [](const at::Tensor& t, const at::Tensor& factor, bool consume) {
    if (!scalable(t, factor)) return t * factor.to(t.scalar_type());
    c10::cuda::CUDAGuard g(t.device());
    at::Tensor out = consume ? t : at::empty_like(t);  // same strides: dense tensors map element by element
    B200C_CUDA_CHECK(launch_scale_bf16(bf(t), bf_mut(out), factor.data_ptr<float>(), static_cast<size_t>(t.numel()), cur(t)));
    return out;
  }, py::arg("t"), py::arg("factor"), py::arg("consume") = false);
  // Whether tensors that autograd saves now go through hooks (which may keep them).
  ops.def("saved_tensor_hooks_active", []() { return at::SavedTensorDefaultHooks::get_hooks().has_value(); });

  ops.def("adamw_step_", [](at::Tensor p, const at::Tensor& grad, at::Tensor mom, at::Tensor var, double lr, double beta1,
                            double beta2, double eps, double weight_decay, int step, double grad_scale) {
    want(p, at::kFloat, "p");
    want(grad, at::kFloat, "grad");
    want(mom, at::kFloat, "m");
    want(var, at::kFloat, "v");
    TORCH_CHECK(grad.numel() == p.numel() && mom.numel() == p.numel() && var.numel() == p.numel(), "size mismatch");
    c10::cuda::CUDAGuard g(p.device());
    B200C_CUDA_CHECK(launch_adamw(p.data_ptr<float>(), grad.data_ptr<float>(), mom.data_ptr<float>(), var.data_ptr<float>(),
                                  static_cast<size_t>(p.numel()), static_cast<float>(lr), static_cast<float>(beta1),
                                  static_cast<float>(beta2), static_cast<float>(eps), static_cast<float>(weight_decay), step,
                                  static_cast<float>(grad_scale), cur(p)));
  });

  // Row-wise e4m3 quantisation: (q, scale), or None where the kernel does not apply (the caller then takes the
  // operator-by-operator path, which every device, type and transform understands).
  ops.def("quantize_rows", [](const at::Tensor& x) -> std::optional<std::pair<at::Tensor, at::Tensor>> {
    if (!quantizable(x)) return std::nullopt;
    c10::cuda::CUDAGuard g(x.device());
    at::Tensor q = at::empty({x.size(0), x.size(1)}, x.options().dtype(at::kFloat8_e4m3fn));
    at::Tensor scale = at::empty({x.size(0)}, x.options().dtype(at::kFloat));
    quantize_into(x, q, scale);
    return std::make_pair(q, scale);
  });
  // The same into existing buffers; false where the kernel does not apply.
  ops.def("quantize_rows_into", [](const at::Tensor& x, at::Tensor q, at::Tensor scale) {
    if (!quantizable(x) || q.device() != x.device() || scale.device() != x.device()) return false;
    if (q.sizes() != x.sizes() || q.scalar_type() != at::kFloat8_e4m3fn || !q.is_contiguous()) return false;
    if (scale.numel() != x.size(0) || scale.scalar_type() != at::kFloat || !scale.is_contiguous()) return false;
    c10::cuda::CUDAGuard g(x.device());
    quantize_into(x, q, scale);
    return true;
  });

  ops.def("gemm_bf16_nt", [](const at::Tensor& a, const at::Tensor& b) {
    want(a, at::kBFloat16, "a");
    want(b, at::kBFloat16, "b");
    TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.size(1) == b.size(1), "a: [m, k], b: [n, k]");
    c10::cuda::CUDAGuard g(a.device());
    at::Tensor c = at::empty({a.size(0), b.size(0)}, a.options());
    at::Tensor status = status_words(a);
    B200C_CUDA_CHECK(launch_gemm_bf16_nt(a.data_ptr(), b.data_ptr(), c.data_ptr(), static_cast<int>(a.size(0)),
                                         static_cast<int>(b.size(0)), static_cast<int>(a.size(1)),
                                         reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(a)));
    return std::make_pair(c, status);
  });

  // c[m, n] (bf16) = scale_a[m] * scale_b[n] * (a[m, k] (e4m3) @ b[n, k]^T (e4m3)), fp32 accumulation in tensor memory.
  ops.def("gemm_e4m3_nt", [](const at::Tensor& a, const at::Tensor& b, const at::Tensor& scale_a, const at::Tensor& scale_b) {
    want(a, at::kFloat8_e4m3fn, "a");
    want(b, at::kFloat8_e4m3fn, "b");
    want(scale_a, at::kFloat, "scale_a");
    want(scale_b, at::kFloat, "scale_b");
    TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.size(1) == b.size(1), "a: [m, k], b: [n, k]");
    TORCH_CHECK(scale_a.numel() == a.size(0) && scale_b.numel() == b.size(0), "one scale per row of a and per row of b");
    c10::cuda::CUDAGuard g(a.device());
    at::Tensor c = at::empty({a.size(0), b.size(0)}, a.options().dtype(at::kBFloat16));
    at::Tensor status = status_words(a);
    B200C_CUDA_CHECK(launch_gemm_e4m3_nt(a.data_ptr(), b.data_ptr(), c.data_ptr(), static_cast<int>(a.size(0)),
                                         static_cast<int>(b.size(0)), static_cast<int>(a.size(1)), scale_a.data_ptr<float>(),
                                         scale_b.data_ptr<float>(), reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(a)));
    return std::make_pair(c, status);
  });

  ops.def("gemm_bf16_nt_pair", [](const at::Tensor& a, const at::Tensor& b) {
    want(a, at::kBFloat16, "a");
    want(b, at::kBFloat16, "b");
    TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.size(1) == b.size(1), "a: [m, k], b: [n, k]");
    c10::cuda::CUDAGuard g(a.device());
    at::Tensor c = at::empty({a.size(0), b.size(0)}, a.options());
    at::Tensor status = status_words(a);
    B200C_CUDA_CHECK(launch_gemm_nt_pair(a.data_ptr(), b.data_ptr(), c.data_ptr(), static_cast<int>(a.size(0)),
                                         static_cast<int>(b.size(0)), static_cast<int>(a.size(1)), nullptr, nullptr,
                                         reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(a)));
    return std::make_pair(c, status);
  });

  // a[m, k] b[k, n], or with `by_columns` a[k, m]^T b[k, n], bf16; rows of a may be apart.
  ops.def("gemm_bf16_mn", [](const at::Tensor& a, const at::Tensor& b, bool by_columns) {
    want(b, at::kBFloat16, "b");
    TORCH_CHECK(a.is_cuda() && a.scalar_type() == at::kBFloat16 && a.dim() == 2 && a.stride(1) == 1, "a: bf16 CUDA rows expected");
    TORCH_CHECK(b.dim() == 2 && a.size(by_columns ? 0 : 1) == b.size(0), "a: [m, k] or, by columns, [k, m]; b: [k, n]");
    c10::cuda::CUDAGuard g(a.device());
    const int64_t m = a.size(by_columns ? 1 : 0);
    at::Tensor c = at::empty({m, b.size(1)}, b.options()), status = status_words(b);
    B200C_CUDA_CHECK(launch_gemm_pair_mn(a.data_ptr(), row_stride(a), by_columns, b.data_ptr(), b.size(1), c.data_ptr(), static_cast<int>(m),
                                         static_cast<int>(b.size(1)), static_cast<int>(b.size(0)),
                                         reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(a)));
    return std::make_pair(c, status);
  }, py::arg("a"), py::arg("b"), py::arg("by_columns") = false);

  // The gradient of gate_up[m, 2 n] from dy[m, k] w[k, n], the gradient of silu(gate) * up.
  ops.def("gemm_gated_grad", [](const at::Tensor& dy, const at::Tensor& w, const at::Tensor& gate_up) {
    want(dy, at::kBFloat16, "dy");
    want(w, at::kBFloat16, "w");
    want(gate_up, at::kBFloat16, "gate_up");
    TORCH_CHECK(dy.dim() == 2 && w.dim() == 2 && gate_up.dim() == 2 && dy.size(1) == w.size(0) && gate_up.size(0) == dy.size(0) &&
                    gate_up.size(1) == 2 * w.size(1), "dy: [m, k], w: [k, n], gate_up: [m, 2 n]");
    c10::cuda::CUDAGuard g(dy.device());
    at::Tensor d = at::empty_like(gate_up), status = status_words(dy);
    B200C_CUDA_CHECK(launch_gemm_gated_grad(dy.data_ptr(), w.data_ptr(), gate_up.data_ptr(), d.data_ptr(), static_cast<int>(dy.size(0)),
                                            static_cast<int>(w.size(1)), static_cast<int>(w.size(0)),
                                            reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(dy)));
    return std::make_pair(d, status);
  });

  // (x w^T, silu(gate) * up of it), bf16, gate columns first. `columns` of a tile, gate and up together: 192, 224 or 256 (0: by size).
  ops.def("gemm_gated", [](const at::Tensor& x, const at::Tensor& w, int columns) {
    want(x, at::kBFloat16, "x");
    want(w, at::kBFloat16, "w");
    TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && w.size(0) % 2 == 0, "x: [m, k], w: [2 n, k]");
    c10::cuda::CUDAGuard g(x.device());
    at::Tensor gate_up = at::empty({x.size(0), w.size(0)}, x.options()), act = at::empty({x.size(0), w.size(0) / 2}, x.options());
    at::Tensor status = status_words(x);
    B200C_CUDA_CHECK(launch_gemm_gated(x.data_ptr(), w.data_ptr(), gate_up.data_ptr(), act.data_ptr(), static_cast<int>(x.size(0)),
                                       static_cast<int>(w.size(0) / 2), static_cast<int>(x.size(1)),
                                       reinterpret_cast<uint32_t*>(status.data_ptr<int>()), cur(x), columns));
    return std::make_tuple(gate_up, act, status);
  }, py::arg("x"), py::arg("w"), py::arg("columns") = 0);

  // For tests: the products' kernels with loads that are never complete and waits of `wait_ms`. `kind`: "nt" (a w^T by the kernel that
  // its size takes), "pair", "gated" (a, w) or "gated_grad" (a w, gate_up). Output and status words.
  ops.def("gemm_giving_up", [](const std::string& kind, const at::Tensor& a, const at::Tensor& w, const std::optional<at::Tensor>& gate_up,
                               int wait_ms) {
    want(a, at::kBFloat16, "a");
    want(w, at::kBFloat16, "w");
    const bool grad = kind == "gated_grad";
    TORCH_CHECK(a.dim() == 2 && w.dim() == 2 && a.size(1) == w.size(grad ? 0 : 1) && wait_ms >= 1 && wait_ms <= 1000, "a: [m, k], w: [n, k] or [k, n]");
    const GiveUp give_up{static_cast<unsigned long long>(wait_ms) * 1000000ull, 16};
    c10::cuda::CUDAGuard g(a.device());
    const int m = static_cast<int>(a.size(0)), n = static_cast<int>(w.size(grad ? 1 : 0)), k = static_cast<int>(a.size(1));
    at::Tensor status = status_words(a), out = at::zeros({m, grad ? 2 * n : n}, a.options());
    auto* words = reinterpret_cast<uint32_t*>(status.data_ptr<int>());
    if (kind == "nt") {
      B200C_CUDA_CHECK(launch_gemm_nt(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, nullptr, nullptr, words, cur(a), nullptr, nullptr, &give_up));
    } else if (kind == "pair") {
      B200C_CUDA_CHECK(launch_gemm_nt_pair(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, nullptr, nullptr, words, cur(a), 0, nullptr, &give_up));
    } else if (kind == "gated") {
      TORCH_CHECK(n % 2 == 0, "w: [2 n, k]");
      at::Tensor act = at::zeros({m, n / 2}, a.options());
      B200C_CUDA_CHECK(launch_gemm_gated(a.data_ptr(), w.data_ptr(), out.data_ptr(), act.data_ptr(), m, n / 2, k, words, cur(a), 0, &give_up));
      out = at::cat({out, act}, 1);
    } else {
      TORCH_CHECK(grad && gate_up.has_value(), "kind");
      want(*gate_up, at::kBFloat16, "gate_up");
      TORCH_CHECK(gate_up->dim() == 2 && gate_up->size(0) == m && gate_up->size(1) == 2 * n, "gate_up: [m, 2 n]");
      B200C_CUDA_CHECK(launch_gemm_gated_grad(a.data_ptr(), w.data_ptr(), gate_up->data_ptr(), out.data_ptr(), m, n, k, words, cur(a), &give_up));
    }
    return std::make_pair(out, status);
  }, py::arg("kind"), py::arg("a"), py::arg("w"), py::arg("gate_up") = std::nullopt, py::arg("wait_ms") = 20);

  ops.def("kernel_launch_count", []() { return kernel_launch_count(); });
}

} // namespace b200c
