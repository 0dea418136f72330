// Memory-bound model kernels (sm_100a): RMSNorm fwd/bwd, RoPE, SwiGLU
// fwd/bwd, fused softmax cross-entropy + gradient, AdamW.
//
// All of them stream their operands once with 16-byte accesses and keep
// statistics in fp32; grids are sized to the 148 SMs of a B200 (persistent
// row loops where a reduction over rows is needed).
#include "fused_ops.h"

#include <cuda_fp8.h>

#include <algorithm>
#include <atomic>

#include "activation.cuh"
#include "early_launch.cuh"
#include "launch_count.h"
#include "wide_access.cuh"

namespace b200c {

namespace {

std::atomic<unsigned long long> g_launches{0};

constexpr int kSms = 148;

__device__ __forceinline__ float2 bf2_to_f2(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
__device__ __forceinline__ uint32_t f2_to_bf2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void unpack8(uint4 v, float* f) {
  float2 a = bf2_to_f2(v.x), b = bf2_to_f2(v.y), c = bf2_to_f2(v.z), d = bf2_to_f2(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(f2_to_bf2(f[0], f[1]), f2_to_bf2(f[2], f[3]), f2_to_bf2(f[4], f[5]), f2_to_bf2(f[6], f[7]));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum; every thread gets the result. `scratch` holds 32 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = lane < nw ? scratch[lane] : 0.0f;
  return warp_sum(t);
}
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = lane < nw ? scratch[lane] : -INFINITY;
  return warp_max(t);
}

// ------------------------------------------------------------- RMSNorm ------

constexpr int kNormThreads = 256;
constexpr int kNormMaxVec = 4;  // cols <= 256 * 4 * 8 = 8192 stay in registers

// Sum over the TPR threads that share a row: a warp, or the whole block. `scratch` holds two sets of partial
// sums that alternate from row to row, so one barrier per row is enough.
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float (*scratch)[TPR / 32], int parity) {
  v = warp_sum(v);
  if constexpr (TPR > 32) {
    if ((threadIdx.x & 31) == 0) scratch[parity][threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0f;
#pragma unroll
    for (int w = 0; w < TPR / 32; ++w) v += scratch[parity][w];
  }
  return v;
}

// Rows that fit the registers of TPR threads (VPT vectors of 8 each): one pass, all loads before the reduction.
// Bound by memory; [4096, 4096]: 16.2 us when blocks of 256 walked rows in a fixed stride, 11.9 us (5.6 TB/s) now.
// ADD: the row is x + delta, rounded to bf16 and also written to `sum` (the residual stream).
template <int TPR, int VPT, bool ADD>
__global__ void __launch_bounds__(TPR < 128 ? 128 : TPR) k_rmsnorm_fwd_reg(const __nv_bfloat16* __restrict__ x,
                                                                            const __nv_bfloat16* __restrict__ delta,
                                                                            const __nv_bfloat16* __restrict__ w,
                                                                            __nv_bfloat16* __restrict__ sum,
                                                                            __nv_bfloat16* __restrict__ y,
                                                                            float* __restrict__ rstd, int rows, int cols,
                                                                            float eps) {
  constexpr int kRows = (TPR < 128 ? 128 : TPR) / TPR;
  __shared__ float scratch[2][TPR / 32];
  const int nvec = cols / 8, lane = threadIdx.x % TPR;
  const int r = blockIdx.x * kRows + threadIdx.x / TPR;
  if (r >= rows) return;  // whole warps where a block holds several rows
  const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * cols);
  uint4* yr = reinterpret_cast<uint4*>(y + static_cast<size_t>(r) * cols);
  uint4 keep[VPT], wv[VPT];
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = lane + k * TPR;
    keep[k] = v < nvec ? xr[v] : make_uint4(0u, 0u, 0u, 0u);
  }
  uint4 add[ADD ? VPT : 1];
  if constexpr (ADD) {
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * TPR;
      add[k] = v < nvec ? reinterpret_cast<const uint4*>(delta + static_cast<size_t>(r) * cols)[v] : make_uint4(0u, 0u, 0u, 0u);
    }
  }
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = lane + k * TPR;
    if (v < nvec) wv[k] = reinterpret_cast<const uint4*>(w)[v];
  }
  if constexpr (ADD) {
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * TPR;
      float f[8], g[8];
      unpack8(keep[k], f);
      unpack8(add[k], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += g[i];
      keep[k] = pack8(f);
      if (v < nvec) reinterpret_cast<uint4*>(sum + static_cast<size_t>(r) * cols)[v] = keep[k];
    }
  }
  float ss = 0.0f;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    float f[8];
    unpack8(keep[k], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  ss = row_sum<TPR>(ss, scratch, 0);
  const float rs = rsqrtf(ss / static_cast<float>(cols) + eps);
  if (lane == 0) rstd[r] = rs;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = lane + k * TPR;
    if (v < nvec) {
      float f[8], g[8];
      unpack8(keep[k], f);
      unpack8(wv[k], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rs * g[i];
      yr[v] = pack8(f);
    }
  }
}

// Rows wider than the registers hold: the first kNormMaxVec vectors of every thread stay there between the two looks,
// the remainder is read twice (the second time from L2). Against reading the whole row twice: 41.3 us and 39.1 at 4096
// x 12288, but 49.3 and 53.1 at 4096 x 16384, 53.4 and 62.6 at 2048 x 32768, 10.3 and 12.4 at 8 x 65536.
__global__ void __launch_bounds__(kNormThreads) k_rmsnorm_fwd_wide(const __nv_bfloat16* __restrict__ x,
                                                                    const __nv_bfloat16* __restrict__ w,
                                                                    __nv_bfloat16* __restrict__ y,
                                                                    float* __restrict__ rstd, int rows, int cols,
                                                                    float eps) {
  __shared__ float scratch[32];
  const int nvec = cols / 8, tail = kNormMaxVec * kNormThreads + threadIdx.x;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * cols);
    uint4* yr = reinterpret_cast<uint4*>(y + static_cast<size_t>(r) * cols);
    uint4 keep[kNormMaxVec];  // all there: this kernel's rows are wider than that
#pragma unroll
    for (int k = 0; k < kNormMaxVec; ++k) keep[k] = xr[threadIdx.x + k * kNormThreads];
    float ss = 0.0f;
    auto square = [&](uint4 q) {
      float f[8];
      unpack8(q, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    };
#pragma unroll
    for (int k = 0; k < kNormMaxVec; ++k) square(keep[k]);
    for (int v = tail; v < nvec; v += kNormThreads) square(xr[v]);
    ss = block_sum(ss, scratch);
    const float rs = rsqrtf(ss / static_cast<float>(cols) + eps);
    if (threadIdx.x == 0) rstd[r] = rs;
    auto write = [&](uint4 q, int v) {
      float f[8], g[8];
      unpack8(q, f);
      unpack8(reinterpret_cast<const uint4*>(w)[v], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rs * g[i];
      yr[v] = pack8(f);
    };
#pragma unroll
    for (int k = 0; k < kNormMaxVec; ++k) write(keep[k], threadIdx.x + k * kNormThreads);
    for (int v = tail; v < nvec; v += kNormThreads) write(xr[v], v);
  }
}

// Every group of TPR threads walks rows with a fixed stride and keeps its share of the weight gradient in
// registers (thread t owns vectors t, t + TPR, ...). x and dy of a row are read once; the next row's loads are
// issued before the current row's reduction, so 16 warps per SM keep the memory busy. [4096, 4096]: 38.9 us when
// every row was read twice without looking ahead, 20.7 us (4.9 TB/s) now.
template <int TPR>
constexpr int norm_bwd_threads() { return TPR < kNormThreads ? kNormThreads : TPR; }
// The two widest shapes need more than the 128 registers a thread that two blocks per SM leave.
template <int TPR, int VPT>
constexpr int norm_bwd_per_sm() { return TPR > 256 || (TPR == 32 && VPT == 4) ? 1 : 2; }

// ADD: the row also fed something else, whose gradient `dskip` is added before the one rounding of dx.
template <int TPR, int VPT, bool ADD>
__global__ void __launch_bounds__(norm_bwd_threads<TPR>(), norm_bwd_per_sm<TPR, VPT>()) k_rmsnorm_bwd(const __nv_bfloat16* __restrict__ dy,
                                                                  const __nv_bfloat16* __restrict__ x,
                                                                  const __nv_bfloat16* __restrict__ w,
                                                                  const float* __restrict__ rstd,
                                                                  const __nv_bfloat16* __restrict__ dskip,
                                                                  __nv_bfloat16* __restrict__ dx,
                                                                  float* __restrict__ dw_partial, int rows, int cols) {
  constexpr int kThreads = norm_bwd_threads<TPR>(), kRows = kThreads / TPR;
  __shared__ float scratch[2][TPR / 32];
  const int nvec = cols / 8, lane = threadIdx.x % TPR;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4* wv = reinterpret_cast<const uint4*>(w);
  float dw[VPT][8];
#pragma unroll
  for (int k = 0; k < VPT; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) dw[k][i] = 0.0f;

  uint4 nx[VPT], nd[VPT];
  float nrs = 0.0f;
  auto fetch = [&](int r) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * cols);
    const uint4* dyr = reinterpret_cast<const uint4*>(dy + static_cast<size_t>(r) * cols);
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * TPR;
      nx[k] = v < nvec ? xr[v] : zero;
      nd[k] = v < nvec ? dyr[v] : zero;
    }
    nrs = rstd[r];
  };
  int r = blockIdx.x * kRows + threadIdx.x / TPR;
  const int step = gridDim.x * kRows;
  if (r < rows) fetch(r);
  for (int parity = 0; r < rows; r += step, parity ^= 1) {
    uint4 cx[VPT], cd[VPT];
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      cx[k] = nx[k];
      cd[k] = nd[k];
    }
    const float rs = nrs;
    if (r + step < rows) fetch(r + step);
    uint4 skip[ADD ? VPT : 1];
    if constexpr (ADD) {
#pragma unroll
      for (int k = 0; k < VPT; ++k) {
        const int v = lane + k * TPR;
        skip[k] = v < nvec ? reinterpret_cast<const uint4*>(dskip + static_cast<size_t>(r) * cols)[v] : zero;
      }
    }
    float dot = 0.0f;  // sum(dy * w * x)
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * TPR;
      float fx[8], fd[8], fw[8];
      unpack8(cx[k], fx);
      unpack8(cd[k], fd);
      unpack8(v < nvec ? wv[v] : zero, fw);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot += fd[i] * fw[i] * fx[i];
    }
    dot = row_sum<TPR>(dot, scratch, parity) * rs / static_cast<float>(cols);
    uint4* dxr = reinterpret_cast<uint4*>(dx + static_cast<size_t>(r) * cols);
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * TPR;
      if (v < nvec) {
        float fx[8], fd[8], fw[8], o[8];
        unpack8(cx[k], fx);
        unpack8(cd[k], fd);
        unpack8(wv[v], fw);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xhat = fx[i] * rs;
          o[i] = rs * (fd[i] * fw[i] - xhat * dot);
          dw[k][i] += fd[i] * xhat;
        }
        if constexpr (ADD) {
          float fs[8];
          unpack8(skip[k], fs);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += fs[i];
        }
        dxr[v] = pack8(o);
      }
    }
  }

  float* out = dw_partial + static_cast<size_t>(blockIdx.x) * cols;
  if constexpr (kRows == 1) {
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * TPR;
      if (v < nvec) {
        reinterpret_cast<float4*>(out)[2 * v] = make_float4(dw[k][0], dw[k][1], dw[k][2], dw[k][3]);
        reinterpret_cast<float4*>(out)[2 * v + 1] = make_float4(dw[k][4], dw[k][5], dw[k][6], dw[k][7]);
      }
    }
  } else {
    // The block's row groups add up their shares first.
    __shared__ float share[kRows][VPT * TPR * 8];
#pragma unroll
    for (int k = 0; k < VPT; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) share[threadIdx.x / TPR][(k * 8 + i) * TPR + lane] = dw[k][i];
    __syncthreads();
    for (int c = threadIdx.x; c < cols; c += kThreads) {
      const int v = c / 8, at = ((v / TPR) * 8 + c % 8) * TPR + v % TPR;
      float sum = 0.0f;
#pragma unroll
      for (int g = 0; g < kRows; ++g) sum += share[g][at];
      out[c] = sum;
    }
  }
}

// out[c] = sum_r in[r, c]. A block takes 32 columns with 32 groups of rows side by side: the few hundred partial
// rows of a norm's backward are a chain of a dozen loads instead of one load per row (296 x 4096: 14.2 us, now 4.1).
constexpr int kColsumCols = 32, kColsumGroups = 32;

__global__ void __launch_bounds__(256) k_colsum_bf16(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, int rows, int cols) {
  __shared__ float part[kColsumGroups][kColsumCols + 1];
  const int quad = threadIdx.x % (kColsumCols / 4), group = threadIdx.x / (kColsumCols / 4);
  const int c = blockIdx.x * kColsumCols + quad * 4;
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (c < cols) {
#pragma unroll 4
    for (int r = group; r < rows; r += kColsumGroups) {
      const float4 v = *reinterpret_cast<const float4*>(in + static_cast<size_t>(r) * cols + c);
      s.x += v.x;
      s.y += v.y;
      s.z += v.z;
      s.w += v.w;
    }
  }
  part[group][quad * 4] = s.x;
  part[group][quad * 4 + 1] = s.y;
  part[group][quad * 4 + 2] = s.z;
  part[group][quad * 4 + 3] = s.w;
  __syncthreads();
  // Eight threads per column finish it; they sit side by side in a warp.
  const int col = threadIdx.x / 8, at = threadIdx.x % 8;
  float t = 0.0f;
#pragma unroll
  for (int g = at; g < kColsumGroups; g += 8) t += part[g][col];
  t += __shfl_xor_sync(0xffffffffu, t, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  if (at == 0 && blockIdx.x * kColsumCols + col < cols) out[blockIdx.x * kColsumCols + col] = __float2bfloat16_rn(t);
}

// ---------------------------------------------------------------- RoPE ------

// Quotient by a divisor fixed at launch, for dividends below 2^31: one wide
// multiply instead of the long sequence of an integer division.
struct FastDiv {
  uint32_t mul, shift, d;
};
FastDiv make_fast_div(uint32_t d) {
  // Granlund & Montgomery, "Division by invariant integers using multiplication"
  // (1994): with l = ceil(log2 d), m = floor(2^(31 + l) / d) + 1 gives exact
  // quotients for every n < 2^31.
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  return FastDiv{static_cast<uint32_t>(((1ull << (31 + l)) / d) + 1), l == 0 ? 0u : l - 1, d};
}
__device__ __forceinline__ uint32_t fast_div(uint32_t n, FastDiv f) {
  return f.d == 1 ? n : __umulhi(n, f.mul) >> f.shift;
}

// Rotates the four pairs of a vector. Spelled out, so that every kernel rounds alike.
__device__ __forceinline__ void rotate8(float* f, float4 c4, float4 s4, float sign) {
  const float* c = &c4.x;
  const float* s = &s4.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = f[2 * j], b = f[2 * j + 1], sj = s[j] * sign;
    f[2 * j] = __fmaf_rn(-b, sj, __fmul_rn(a, c[j]));
    f[2 * j + 1] = __fmaf_rn(a, sj, __fmul_rn(b, c[j]));
  }
}

// Bound by memory: every element is read and written once, so the source is read where the caller has it (a
// slice of the fused projection's output) instead of being copied first and rotated in place, and the result is
// the only write. Four vectors of 8 bf16 per thread, all loads before the first use. Queries and keys of 4093 tokens
// (32 + 8 heads of 128, slices of one projection), both directions: 107 us with the copies (73 us of it), 36 us
// (4.6 TB/s) without.
constexpr int kRopeVecs = 4;

__global__ void __launch_bounds__(256) k_rope(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                              const int* __restrict__ pos, const float* __restrict__ cos_t,
                                              const float* __restrict__ sin_t, uint32_t total, FastDiv per_head,
                                              FastDiv heads, int64_t stride_t, int64_t stride_h, float sign) {
  const uint32_t base = blockIdx.x * (256u * kRopeVecs) + threadIdx.x;
  uint4 in[kRopeVecs];
  float4 cs[kRopeVecs], sn[kRopeVecs];
#pragma unroll
  for (int k = 0; k < kRopeVecs; ++k) {
    const uint32_t i = base + k * 256u;
    if (i < total) {
      const uint32_t th = fast_div(i, per_head), v = i - th * per_head.d;
      const uint32_t t = fast_div(th, heads), h = th - t * heads.d;
      in[k] = *reinterpret_cast<const uint4*>(x + t * stride_t + h * stride_h + v * 8);
      const size_t at = static_cast<size_t>(pos[t]) * per_head.d + v;  // tables of head_dim / 2 = 4 * per_head floats
      cs[k] = reinterpret_cast<const float4*>(cos_t)[at];
      sn[k] = reinterpret_cast<const float4*>(sin_t)[at];
    }
  }
#pragma unroll
  for (int k = 0; k < kRopeVecs; ++k) {
    const uint32_t i = base + k * 256u;
    if (i < total) {
      float f[8];
      unpack8(in[k], f);
      rotate8(f, cs[k], sn[k], sign);
      reinterpret_cast<uint4*>(y)[i] = pack8(f);
    }
  }
}

// Both directions of what sits between a fused QKV projection and attention. `packed` is the projection's output
// (or its gradient), rows of (heads + 2 kv_heads) x head_dim; `part[0..2]` are queries, keys and values with their
// own strides. Forward reads `packed`, rotates queries and keys and copies values; backward does the reverse, so
// the gradient of the projection is written once, without rotating pieces first and joining them afterwards.
struct QkvParts {
  __nv_bfloat16* p[3];
  int64_t stride_t[3], stride_h[3];
};

template <bool FWD>
__global__ void __launch_bounds__(256) k_split_rope(__nv_bfloat16* packed, int64_t ld, QkvParts part, const int* __restrict__ pos,
                                                    const float* __restrict__ cos_t, const float* __restrict__ sin_t, uint32_t total,
                                                    FastDiv per_head, FastDiv all_heads, uint32_t heads, uint32_t kv_heads) {
  const uint32_t base = blockIdx.x * (256u * kRopeVecs) + threadIdx.x;
  uint4 in[kRopeVecs];
  float4 cs[kRopeVecs], sn[kRopeVecs];
  uint4* dst[kRopeVecs];
  bool rotate[kRopeVecs];
#pragma unroll
  for (int k = 0; k < kRopeVecs; ++k) {
    const uint32_t i = base + k * 256u;
    dst[k] = nullptr;
    if (i < total) {
      const uint32_t th = fast_div(i, per_head), v = i - th * per_head.d;
      const uint32_t t = fast_div(th, all_heads), h = th - t * all_heads.d;
      const int which = h < heads ? 0 : h < heads + kv_heads ? 1 : 2;
      const uint32_t hp = h - (which == 0 ? 0u : which == 1 ? heads : heads + kv_heads);
      uint4* a = reinterpret_cast<uint4*>(packed + t * ld) + (h * per_head.d + v);
      // selects instead of an indexed parameter, which would go through local memory
      __nv_bfloat16* pp = which == 0 ? part.p[0] : which == 1 ? part.p[1] : part.p[2];
      const int64_t st = which == 0 ? part.stride_t[0] : which == 1 ? part.stride_t[1] : part.stride_t[2];
      const int64_t sh = which == 0 ? part.stride_h[0] : which == 1 ? part.stride_h[1] : part.stride_h[2];
      uint4* b = reinterpret_cast<uint4*>(pp + t * st + hp * sh + v * 8);
      in[k] = FWD ? *a : *b;
      dst[k] = FWD ? b : a;
      rotate[k] = which < 2;
      if (rotate[k]) {
        const size_t at = static_cast<size_t>(pos[t]) * per_head.d + v;
        cs[k] = reinterpret_cast<const float4*>(cos_t)[at];
        sn[k] = reinterpret_cast<const float4*>(sin_t)[at];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kRopeVecs; ++k) {
    if (dst[k] != nullptr && !rotate[k]) {
      *dst[k] = in[k];  // values are copied bit by bit
    } else if (dst[k] != nullptr) {
      float f[8];
      unpack8(in[k], f);
      rotate8(f, cs[k], sn[k], FWD ? 1.0f : -1.0f);
      *dst[k] = pack8(f);
    }
  }
}

// -------------------------------------------------------------- SwiGLU ------

// Both directions stream their operands once and are bound by memory: every thread takes VECS vectors of each
// operand, all loads before the first use, and finds its row with a multiply instead of a 64-bit division.
// [4096, 2 x 14336]: forward 60.8 us, now 53.8 (6.5 TB/s); backward 101.2 us, now 83.5 (7.0 TB/s); a pass of both through autograd
// 146.7 us with a division in the sigmoid, which branches, and 142.5. Two vectors per
// thread once every vector cannot have a resident thread of its own (148 x 2048 threads); below that a pass is one
// chain of latencies, which a second vector's arithmetic makes longer: forward / backward of [100, 2 x 8192] 2.9 / 3.5 us
// with two, 2.3 / 2.8 with one, of [1, 2 x 4096] 2.6 / 3.0 and 2.0 / 2.3; of [700, 2 x 4096] (358 thousand vectors)
// 4.2 / 5.0 with two.
template <int VECS>
__global__ void __launch_bounds__(256) k_swiglu_fwd(const __nv_bfloat16* gate_up, __nv_bfloat16* h, uint32_t total, FastDiv per_row) {
  const uint32_t base = blockIdx.x * (256u * VECS) + threadIdx.x;
  grid_release();
  grid_wait();
  uint4 gv[VECS], uv[VECS];
#pragma unroll
  for (int k = 0; k < VECS; ++k) {
    const uint32_t i = base + k * 256u;
    if (i < total) {
      // row r holds 2 x per_row vectors: gate, then up
      const size_t at = static_cast<size_t>(i) + static_cast<size_t>(fast_div(i, per_row)) * per_row.d;
      gv[k] = reinterpret_cast<const uint4*>(gate_up)[at];
      uv[k] = reinterpret_cast<const uint4*>(gate_up)[at + per_row.d];
    }
  }
#pragma unroll
  for (int k = 0; k < VECS; ++k) {
    const uint32_t i = base + k * 256u;
    if (i < total) {
      float g[8], u[8], o[8];
      unpack8(gv[k], g);
      unpack8(uv[k], u);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = gated(g[j], u[j]);
      reinterpret_cast<uint4*>(h)[i] = pack8(o);
    }
  }
}

template <int VECS>
__global__ void __launch_bounds__(256) k_swiglu_bwd(const __nv_bfloat16* dh, const __nv_bfloat16* gate_up, __nv_bfloat16* dgate_up,
                                                    uint32_t total, FastDiv per_row) {
  const uint32_t base = blockIdx.x * (256u * VECS) + threadIdx.x;
  grid_release();
  grid_wait();
  uint4 gv[VECS], uv[VECS], dv[VECS];
#pragma unroll
  for (int k = 0; k < VECS; ++k) {
    const uint32_t i = base + k * 256u;
    if (i < total) {
      const size_t at = static_cast<size_t>(i) + static_cast<size_t>(fast_div(i, per_row)) * per_row.d;
      gv[k] = reinterpret_cast<const uint4*>(gate_up)[at];
      uv[k] = reinterpret_cast<const uint4*>(gate_up)[at + per_row.d];
      dv[k] = reinterpret_cast<const uint4*>(dh)[i];
    }
  }
#pragma unroll
  for (int k = 0; k < VECS; ++k) {
    const uint32_t i = base + k * 256u;
    if (i < total) {
      const size_t at = static_cast<size_t>(i) + static_cast<size_t>(fast_div(i, per_row)) * per_row.d;
      float g[8], u[8], d[8], dg[8], du[8];
      unpack8(gv[k], g);
      unpack8(uv[k], u);
      unpack8(dv[k], d);
#pragma unroll
      for (int j = 0; j < 8; ++j) gated_gradient(d[j], g[j], u[j], &dg[j], &du[j]);
      reinterpret_cast<uint4*>(dgate_up)[at] = pack8(dg);
      reinterpret_cast<uint4*>(dgate_up)[at + per_row.d] = pack8(du);
    }
  }
}

// ------------------------------------------------------- cross-entropy ------

constexpr int kCeMaxThreads = 512;

// Two looks at every row: the first finds its log-sum-exp, the second writes the gradient over it. What bounds
// it is memory (one read and one write of the logits) as long as the second look hits L2, so no more rows are in
// work at a time than L2 holds (see the launcher), and the exponentials come next: two per element on the
// special-function unit. The rest is kept off the issue slots: one maximum and one comparison per 8 elements,
// and the target's column is looked for per vector. Rows that start off a 16-byte boundary (vocabularies that
// are no multiple of 8) peel up to 7 elements instead of giving up wide accesses. 4096 rows of 128256
// between a head's GEMMs: 698 us with 592 rows in work and a comparison per element, 480 to 570 us now, by the clock
// that the power cap leaves.
__global__ void __launch_bounds__(kCeMaxThreads, 2) k_cross_entropy(__nv_bfloat16* __restrict__ logits,
                                                                    int64_t ld, const int64_t* __restrict__ targets,
                                                                    float* __restrict__ loss, int rows, int vocab,
                                                                    float grad_scale) {
  __shared__ float scratch[32];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    __nv_bfloat16* row = logits + static_cast<int64_t>(r) * ld;
    const int64_t tgt = targets[r];
    const int head = min(vocab, static_cast<int>((16u - (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(row)) & 15u)) & 15u) / 2);
    const int nvec = (vocab - head) / 8, tail = head + nvec * 8;
    uint4* body = reinterpret_cast<uint4*>(row + head);
    // pass 1: running maximum and sum of exponentials per thread, merged across the block
    float mx = -INFINITY, ref = 0.0f, sum = 0.0f;  // ref = mx, or 0 while nothing above -inf was seen
    auto raise = [&](float m) {
      if (m > mx) {
        if (mx != -INFINITY) sum *= __expf(mx - m);
        mx = ref = m;
      }
    };
    auto feed = [&](uint4 q) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
      const __nv_bfloat162 m2 = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
      raise(fmaxf(__low2float(m2), __high2float(m2)));
      float f[8];
      unpack8(q, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += __expf(f[i] - ref);
    };
    int v = tid;
    for (; v + 3 * nt < nvec; v += 4 * nt) {
      uint4 q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = body[v + k * nt];
#pragma unroll
      for (int k = 0; k < 4; ++k) feed(q[k]);
    }
    for (; v < nvec; v += nt) feed(body[v]);
    const int edge = tid < head ? tid : tail + tid - head;  // the elements outside the vectors, one per thread
    if (edge < vocab && (edge < head || edge >= tail)) {
      const float z = __bfloat162float(row[edge]);
      raise(z);
      sum += __expf(z - ref);
    }
    const float gmx = block_max(mx, scratch);
    const float gsum = block_sum(mx == -INFINITY ? sum : sum * __expf(mx - gmx), scratch);
    const float lse = gmx + __logf(gsum);
    const bool ignore = tgt < 0 || tgt >= vocab;
    if (tid == 0) loss[r] = ignore ? 0.0f : lse - __bfloat162float(row[tgt]);
    __syncthreads();  // the target logit was read before anybody overwrites it
    // pass 2: gradient in place
    const float gs = ignore ? 0.0f : grad_scale;
    const int tv = (ignore || tgt < head || tgt >= tail) ? -1 : static_cast<int>(tgt - head) / 8;
    auto grad = [&](uint4 q, int at) {
      float f[8];
      unpack8(q, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = __expf(f[i] - lse);
      if (at == tv) {
        const int c = static_cast<int>(tgt - head) % 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] -= i == c ? 1.0f : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] *= gs;
      __stcs(body + at, pack8(f));  // not read again here
    };
    v = tid;
    for (; v + 3 * nt < nvec; v += 4 * nt) {
      uint4 q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = __ldcs(body + v + k * nt);
#pragma unroll
      for (int k = 0; k < 4; ++k) grad(q[k], v + k * nt);
    }
    for (; v < nvec; v += nt) grad(__ldcs(body + v), v);
    if (edge < vocab && (edge < head || edge >= tail)) {
      const float z = __bfloat162float(row[edge]);
      row[edge] = __float2bfloat16_rn((__expf(z - lse) - (edge == tgt ? 1.0f : 0.0f)) * gs);
    }
  }
}

// Rows whose shares' maxima and sums of exponentials are known (launch_head_logits): the gradient in one look, bound by one
// read and one write of the logits. A block takes a vector of 16 logits per thread and the grid covers the logits once,
// in the order of their addresses: 4096 x 128256 302 us by itself (6.9 TB/s); blocks that walk a row of their own take 338,
// columns from the last, which L2 still holds, to the first 327. Up to kGradFused blocks each puts the log-sum-exp of its
// row together while its logits are on their way (64 x 2000 4.0 us, 512 x 11008 7.4); more of them leave that to k_head_rows
// (5.3 and 8.2 with both; 4096 x 1000 9.0 against 15.2, 4096 x 8000 26.5 against 34).
constexpr int kGradThreads = 256, kGradFused = 2048;

struct HeadGrad {
  __nv_bfloat16* logits;
  int64_t ld;
  const int64_t* targets;
  const float2* stats;
  const float* fine;
  const float* target_logit;
  float* row_lse;   // [rows], where k_head_rows runs
  float* row_loss;
  float* loss;
  uint32_t* words;
  int rows, shares, vocab, parts, first;
  float grad_scale, loss_scale;
};

// What several shares of a row are together: maximum and sum of exponentials of the rounded logits, and what the sum of the
// unrounded ones has more.
struct HeadShare {
  float mx = -INFINITY, sum = 0.0f, fine = 0.0f;
};
__device__ __forceinline__ void head_join(HeadShare& a, HeadShare b) {
  const float top = fmaxf(a.mx, b.mx);
  const float by_a = a.mx == -INFINITY ? 1.0f : __expf(a.mx - top), by_b = b.mx == -INFINITY ? 1.0f : __expf(b.mx - top);
  a = HeadShare{top, a.sum * by_a + b.sum * by_b, a.fine * by_a + b.fine * by_b};
}
__device__ __forceinline__ HeadShare head_share(const HeadGrad& a, int share, int row) {
  const size_t at = static_cast<size_t>(share) * a.rows + row;
  const float2 s = a.stats[at];
  return HeadShare{s.x, s.y, a.fine[at]};
}
// The log-sum-exp that the gradient is made with, of the rounded logits, and the loss's, of the unrounded ones.
__device__ __forceinline__ float head_lse(const HeadGrad& a, HeadShare row) {
  return a.words[0] != 0u ? NAN : row.mx + logf(row.sum);  // the product gave up a wait: its logits are not to be used
}
__device__ __forceinline__ float head_loss(const HeadGrad& a, HeadShare row, int r) {
  return (a.words[0] != 0u ? NAN : row.mx + logf(row.sum + row.fine)) - a.target_logit[r];
}

__device__ __forceinline__ bool head_ignores(const HeadGrad& a, int64_t target) { return target < 0 || target >= a.vocab; }

// Counts `rows` rows whose loss threads of this block have written and fenced; the block that finds all counted adds them up, in an
// order that does not depend on which block it is. Every thread of the block calls it.
__device__ __forceinline__ void head_add_up(const HeadGrad& a, int rows, float* scratch) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(a.words + 2, static_cast<uint32_t>(rows)) + static_cast<uint32_t>(rows) == static_cast<uint32_t>(a.rows);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  float total = 0.0f;
  for (int i = threadIdx.x; i < a.rows; i += blockDim.x) total += __ldcg(a.row_loss + i);
  total = block_sum(total, scratch) * a.loss_scale;
  if (threadIdx.x == 0) *a.loss = a.first != 0 ? total : *a.loss + total;
}

// 32 rows a block, one per lane; the warps take the shares in turn.
__global__ void __launch_bounds__(512) k_head_rows(HeadGrad a) {
  __shared__ float scratch[32];
  __shared__ HeadShare part[16][32];
  grid_release();
  grid_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = blockIdx.x * 32 + lane;
  HeadShare sum;
  if (r < a.rows) {
#pragma unroll 4
    for (int t = warp; t < a.shares; t += 16) head_join(sum, head_share(a, t, r));
  }
  part[warp][lane] = sum;
  __syncthreads();
  if (warp == 0 && r < a.rows) {
    for (int w = 1; w < 16; ++w) head_join(sum, part[w][lane]);
    a.row_lse[r] = head_lse(a, sum);
    a.row_loss[r] = head_ignores(a, a.targets[r]) ? 0.0f : head_loss(a, sum, r);
    __threadfence();
  }
  head_add_up(a, min(32, a.rows - static_cast<int>(blockIdx.x) * 32), scratch);
}

template <bool LSE_KNOWN>
__global__ void __launch_bounds__(kGradThreads) k_head_gradient(HeadGrad a) {
  __shared__ float scratch[32];
  __shared__ float shared_lse;
  grid_release();
  grid_wait();
  const int r = blockIdx.x / a.parts, part = blockIdx.x - r * a.parts, v = part * blockDim.x + threadIdx.x;
  const bool there = v < (a.vocab + 15) / 16;
  __nv_bfloat16* at = a.logits + static_cast<int64_t>(r) * a.ld + static_cast<int64_t>(v) * 16;
  uint4 q[2];
  if (there) ld32(at, q[0], q[1]);
  const int64_t tgt = a.targets[r];
  const bool ignore = head_ignores(a, tgt);
  if (!LSE_KNOWN) {
    if (threadIdx.x < 32) {
      HeadShare sum;
      for (int t = threadIdx.x; t < a.shares; t += 32) head_join(sum, head_share(a, t, r));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        head_join(sum, HeadShare{__shfl_xor_sync(0xffffffffu, sum.mx, o), __shfl_xor_sync(0xffffffffu, sum.sum, o),
                                 __shfl_xor_sync(0xffffffffu, sum.fine, o)});
      }
      if (threadIdx.x == 0) {
        shared_lse = head_lse(a, sum);
        if (part == 0) {
          a.row_loss[r] = ignore ? 0.0f : head_loss(a, sum, r);
          __threadfence();
        }
      }
    }
    __syncthreads();
  }
  const float lse = LSE_KNOWN ? a.row_lse[r] : shared_lse;
  const float gs = ignore ? 0.0f : a.grad_scale;
  if (there) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float f[8];
      unpack8(q[h], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = __expf(f[i] - lse);
      if (!ignore && v * 2 + h == static_cast<int>(tgt / 8)) {
        const int c = static_cast<int>(tgt % 8);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] -= i == c ? 1.0f : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] *= gs;
      q[h] = pack8(f);
    }
    st32(at, q[0], q[1]);
  }
  if (!LSE_KNOWN && part == 0) head_add_up(a, 1, scratch);
}

// dx[r, :] = bf16(part[r, :] + sum over j < depth of grad[r, j] * w[j, :]): the last few (depth < 8) columns of a vocabulary
// that is no multiple of 8, whose product with the others would lose its tiled loads and, summed by itself and rounded,
// its accuracy (512 x 4096 x 6007: 1.78e-3 off, so 1.66e-3 like any product of 8 columns more). Columns in vectors of 8.
__global__ void __launch_bounds__(256) k_head_tail(const float* part, const __nv_bfloat16* grad, int64_t ld, const __nv_bfloat16* w,
                                                    __nv_bfloat16* dx, uint32_t total, FastDiv per_row, int depth) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= total) return;
  const uint32_t r = fast_div(i, per_row), c = i - r * per_row.d;
  float sum[8];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 p = reinterpret_cast<const float4*>(part)[2 * static_cast<size_t>(i) + h];
    sum[4 * h] = p.x;
    sum[4 * h + 1] = p.y;
    sum[4 * h + 2] = p.z;
    sum[4 * h + 3] = p.w;
  }
  for (int j = 0; j < depth; ++j) {
    const float g = __bfloat162float(grad[r * ld + j]);
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(w)[static_cast<size_t>(j) * per_row.d + c], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[k] = __fmaf_rn(g, f[k], sum[k]);
  }
  reinterpret_cast<uint4*>(dx)[i] = pack8(sum);
}

// out = in * bf16(*factor) for n bf16 values, the factor on the device. Both pointers 16-byte aligned; out may be
// in, and then a factor of one (the gradient of a loss that is differentiated directly) leaves nothing to do.
// Blocks stride over the data: with nothing to do, the 64 thousand blocks that cover a 1 GB gradient once take 45 us
// to start and end, these 5.
struct ScaleSpan {
  const __nv_bfloat16* in;
  __nv_bfloat16* out;
  size_t n;
};
__global__ void __launch_bounds__(256) k_scale_bf16(ScaleSpan a, ScaleSpan b, const float* __restrict__ factor) {
  const float f = __bfloat162float(__float2bfloat16_rn(*factor));
  const ScaleSpan span = blockIdx.y == 0 ? a : b;
  const __nv_bfloat16* in = span.in;
  __nv_bfloat16* out = span.out;
  const size_t n = span.n;
  if (f == 1.0f && in == out) return;
  const size_t nvec = n / 8, stride = static_cast<size_t>(gridDim.x) * 256;
  size_t v = blockIdx.x * static_cast<size_t>(256) + threadIdx.x;
  auto one = [&](uint4 q) {
    float x[8];
    unpack8(q, x);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] *= f;
    return pack8(x);
  };
  const uint4* src = reinterpret_cast<const uint4*>(in);
  uint4* dst = reinterpret_cast<uint4*>(out);
  for (; v + 3 * stride < nvec; v += 4 * stride) {
    uint4 q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = __ldcs(src + v + k * stride);
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[v + k * stride] = one(q[k]);
  }
  for (; v < nvec; v += stride) dst[v] = one(src[v]);
  if (blockIdx.x == 0 && threadIdx.x < n % 8) {
    const size_t i = nvec * 8 + threadIdx.x;
    out[i] = __float2bfloat16_rn(__bfloat162float(in[i]) * f);
  }
}

// ------------------------------------------------- row quantisation (e4m3) ---

// q[r, :] = e4m3(x[r, :] / scale[r]) with scale[r] = max(amax_r, 1e-8) / 448. A block per row, which stays in
// registers between the maximum and the division (longer rows re-read the rest from L2): 2 bytes in and 1 byte
// out per element is all that moves. The maximum is taken on the bit patterns, where NaN is above infinity and
// so comes through. VEC elements per access: 16 where base, row stride and cols allow 32-byte loads and 16-byte stores, 8
// where they allow half of that, 1 otherwise; KEEP accesses of a thread stay in registers. In us with 8 and 16: [4096,
// 4096] 10.7 and 8.9 (5.7 TB/s), [4096, 8192] 19.9 and 15.9, [4096, 14336] 27.2 and 26.8 (6.6 TB/s), [67, 4096] 1.9 and 1.4;
// the first and third operator by operator: 890 us.
template <int VEC, int KEEP>
__global__ void __launch_bounds__(256) k_quantize_rows(const __nv_bfloat16* x, int64_t ld, uint8_t* q, float* scale, int cols) {
  constexpr int kQuads = VEC >= 8 ? VEC / 8 : 1;  // 16-byte pieces of an access
  __shared__ uint32_t part[8];
  grid_release();
  grid_wait();
  const int tid = threadIdx.x, nt = blockDim.x;
  const __nv_bfloat16* row = x + static_cast<int64_t>(blockIdx.x) * ld;
  uint8_t* out = q + static_cast<size_t>(blockIdx.x) * cols;
  const int nvec = VEC > 1 ? cols / VEC : 0;
  uint4 keep[KEEP][kQuads];
  uint32_t mx = 0;  // two 16-bit lanes
  auto fetch = [&](int v, uint4* to) {
    if constexpr (VEC == 16) ld32(row + static_cast<int64_t>(v) * 16, to[0], to[1]);
    else to[0] = reinterpret_cast<const uint4*>(row)[v];
  };
  auto look = [&](const uint4* v) {
#pragma unroll
    for (int i = 0; i < kQuads; ++i) {
      mx = __vmaxu2(mx, __vmaxu2(__vmaxu2(v[i].x & 0x7fff7fffu, v[i].y & 0x7fff7fffu), __vmaxu2(v[i].z & 0x7fff7fffu, v[i].w & 0x7fff7fffu)));
    }
  };
  if constexpr (VEC > 1) {
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
#pragma unroll
      for (int i = 0; i < kQuads; ++i) keep[k][i] = make_uint4(0u, 0u, 0u, 0u);
      if (tid + k * nt < nvec) fetch(tid + k * nt, keep[k]);
    }
#pragma unroll
    for (int k = 0; k < KEEP; ++k) look(keep[k]);
    for (int v = tid + KEEP * nt; v < nvec; v += nt) {
      uint4 w[kQuads];
      fetch(v, w);
      look(w);
    }
  } else {
    for (int c = tid; c < cols; c += nt) mx = __vmaxu2(mx, reinterpret_cast<const uint16_t*>(row)[c] & 0x7fffu);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = __vmaxu2(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (nt > 32) {
    if ((tid & 31) == 0) part[tid >> 5] = mx;
    __syncthreads();
    for (int i = 0; i < nt / 32; ++i) mx = __vmaxu2(mx, part[i]);
  }
  const uint32_t top = max(mx & 0xffffu, mx >> 16);
  float amax = __uint_as_float(top << 16);
  amax = amax < 1e-8f ? 1e-8f : amax;  // NaN stays
  const float sc = amax * (1.0f / 448.0f);
  if (tid == 0) scale[blockIdx.x] = sc;
  // x / sc for every element, correctly rounded. All share one divisor, so for finite rows the quotient comes from
  // its reciprocal and one residual correction (Markstein, "Computation of elementary functions on the IBM RISC
  // System/6000 processor", 1990): exact for the 8-bit significands that x and the maximum have, at a third of the
  // instructions of a division. The tests compare every pair of significands with the division.
  const float rc = __frcp_rn(sc);
  auto divide = [&](float v) {
    const float q0 = v * rc;
    return __fmaf_rn(__fmaf_rn(-q0, sc, v), rc, q0);
  };
  auto convert = [&](const uint4* v, int at, auto quotient) {
    uint32_t o[2 * kQuads];
#pragma unroll
    for (int i = 0; i < 2 * kQuads; ++i) {
      const uint4 w = v[i / 2];
      const float2 a = bf2_to_f2(i % 2 == 0 ? w.x : w.z), b = bf2_to_f2(i % 2 == 0 ? w.y : w.w);
      const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(quotient(a.x), quotient(a.y)), __NV_SATFINITE, __NV_E4M3);
      const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(quotient(b.x), quotient(b.y)), __NV_SATFINITE, __NV_E4M3);
      o[i] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
    }
    if constexpr (VEC == 16) reinterpret_cast<uint4*>(out)[at] = make_uint4(o[0], o[1], o[2], o[3]);
    else reinterpret_cast<uint2*>(out)[at] = make_uint2(o[0], o[1]);
  };
  auto write_row = [&](auto quotient) {
    if constexpr (VEC > 1) {
#pragma unroll
      for (int k = 0; k < KEEP; ++k) {
        const int v = tid + k * nt;
        if (v < nvec) convert(keep[k], v, quotient);
      }
      for (int v = tid + KEEP * nt; v < nvec; v += nt) {
        uint4 w[kQuads];
        fetch(v, w);
        convert(w, v, quotient);
      }
    } else {
      for (int c = tid; c < cols; c += nt) {
        out[c] = __nv_cvt_float_to_fp8(quotient(__bfloat162float(row[c])), __NV_SATFINITE, __NV_E4M3);
      }
    }
  };
  if (amax < INFINITY) write_row(divide);
  else write_row([&](float v) { return __fdiv_rn(v, sc); });  // infinities and NaN as the division has them
}

// ------------------------------------------------------------ cast copy -----

constexpr int kCastVecs = 2;

template <typename In, typename Out>
__global__ void __launch_bounds__(256) k_cast_scale(const In* __restrict__ in, Out* __restrict__ out, size_t n, float scale) {
  // kCastVecs vectors of 8 elements per thread, all loads first; the grid covers the data once.
  const size_t nvec = n / 8;
  const size_t base = blockIdx.x * static_cast<size_t>(256 * kCastVecs) + threadIdx.x;
  uint4 raw[kCastVecs][sizeof(In) / 2];
#pragma unroll
  for (int k = 0; k < kCastVecs; ++k) {
    const size_t v = base + k * 256;
    if (v < nvec) {
#pragma unroll
      for (int h = 0; h < static_cast<int>(sizeof(In) / 2); ++h) raw[k][h] = __ldcs(reinterpret_cast<const uint4*>(in) + v * (sizeof(In) / 2) + h);
    }
  }
#pragma unroll
  for (int k = 0; k < kCastVecs; ++k) {
    const size_t v = base + k * 256;
    if (v < nvec) {
      float f[8];
      if constexpr (sizeof(In) == 4) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          f[4 * h] = __uint_as_float(raw[k][h].x);
          f[4 * h + 1] = __uint_as_float(raw[k][h].y);
          f[4 * h + 2] = __uint_as_float(raw[k][h].z);
          f[4 * h + 3] = __uint_as_float(raw[k][h].w);
        }
      } else {
        unpack8(raw[k][0], f);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] *= scale;
      if constexpr (sizeof(Out) == 4) {
        reinterpret_cast<float4*>(out)[2 * v] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4*>(out)[2 * v + 1] = make_float4(f[4], f[5], f[6], f[7]);
      } else {
        reinterpret_cast<uint4*>(out)[v] = pack8(f);
      }
    }
  }
  if (blockIdx.x == 0) {
    for (size_t i = nvec * 8 + threadIdx.x; i < n; i += blockDim.x) {
      float x;
      if constexpr (sizeof(In) == 4) x = reinterpret_cast<const float*>(in)[i];
      else x = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(in)[i]);
      x *= scale;
      if constexpr (sizeof(Out) == 4) reinterpret_cast<float*>(out)[i] = x;
      else reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(x);
    }
  }
}

// --------------------------------------------------------------- AdamW ------

// sqrt and division as the hardware approximations (about 1 ulp): the IEEE
// sequences cost several times the arithmetic of the rest of the update and
// made this memory-bound kernel issue-bound.
__device__ __forceinline__ float fast_sqrt(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float adamw_one(float p, float g, float& m, float& v, float lr, float beta1, float beta2,
                                           float eps, float decay, float inv_bias1, float inv_bias2, float grad_scale) {
  const float gr = g * grad_scale;
  m = beta1 * m + (1.0f - beta1) * gr;
  v = beta2 * v + (1.0f - beta2) * gr * gr;
  const float denom = fast_sqrt(v * inv_bias2) + eps;
  return p * decay - __fdividef(lr * (m * inv_bias1), denom);
}

// Seven streams, each touched once: bound by memory. A block takes a contiguous span, two vectors per thread, and the
// grid covers the tensors once; with blocks that stride through them the streams reach memory in a less even order
// (218112000 elements: 1013 us striding over 1184 blocks, 890 us, 6.9 TB/s, so). Small tensors are one chain of
// latencies, which a second vector makes longer, and take one vector per thread up to three blocks per SM: 50000
// elements 2.3 us with two and 2.1 with one, 400000 2.8 and 2.6, but 800000 3.5 and 3.7.
template <int VECS>
__global__ void __launch_bounds__(256) k_adamw(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                                               float* __restrict__ v, size_t n, float lr, float beta1, float beta2,
                                               float eps, float weight_decay, float bias1, float bias2, float grad_scale) {
  const size_t nvec = n / 4;
  const float inv_bias1 = 1.0f / bias1, inv_bias2 = 1.0f / bias2, decay = 1.0f - lr * weight_decay;
  const size_t base = blockIdx.x * static_cast<size_t>(256 * VECS) + threadIdx.x;
  float4 pp[VECS], gg[VECS], mm[VECS], vv[VECS];
#pragma unroll
  for (int u = 0; u < VECS; ++u) {
    const size_t j = base + u * 256;
    if (j < nvec) {
      pp[u] = reinterpret_cast<float4*>(p)[j];
      gg[u] = __ldcs(reinterpret_cast<const float4*>(g) + j);  // the gradient is not read again
      mm[u] = reinterpret_cast<float4*>(m)[j];
      vv[u] = reinterpret_cast<float4*>(v)[j];
    }
  }
#pragma unroll
  for (int u = 0; u < VECS; ++u) {
    const size_t j = base + u * 256;
    if (j < nvec) {
      float* pa = &pp[u].x;
      const float* ga = &gg[u].x;
      float* ma = &mm[u].x;
      float* va = &vv[u].x;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        pa[k] = adamw_one(pa[k], ga[k], ma[k], va[k], lr, beta1, beta2, eps, decay, inv_bias1, inv_bias2, grad_scale);
      }
      reinterpret_cast<float4*>(p)[j] = pp[u];
      reinterpret_cast<float4*>(m)[j] = mm[u];
      reinterpret_cast<float4*>(v)[j] = vv[u];
    }
  }
  // tail
  if (blockIdx.x == 0 && threadIdx.x < n % 4) {
    const size_t t = nvec * 4 + threadIdx.x;
    p[t] = adamw_one(p[t], g[t], m[t], v[t], lr, beta1, beta2, eps, decay, inv_bias1, inv_bias2, grad_scale);
  }
}

// Blocks that cover `vecs` vectors once, `per_block` each (at least one block, for the elements outside the vectors).
unsigned covering_grid(size_t vecs, size_t per_block) {
  return static_cast<unsigned>(std::max<size_t>(1, (vecs + per_block - 1) / per_block));
}

} // namespace

void note_kernel_launch(int n) { g_launches.fetch_add(static_cast<unsigned long long>(n), std::memory_order_relaxed); }
unsigned long long kernel_launch_count() { return g_launches.load(std::memory_order_relaxed); }
unsigned long long fused_ops_launch_count() { return kernel_launch_count(); }

namespace {

// Vector accesses of 16 bytes (null pointers, as in a sizing query or for an absent operand, count as aligned).
template <typename... P>
bool misaligned16(const P*... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) != 0;
}

template <bool ADD>
void rmsnorm_fwd_rows(const __nv_bfloat16* x, const __nv_bfloat16* delta, const __nv_bfloat16* w, __nv_bfloat16* sum,
                      __nv_bfloat16* y, float* rstd, int rows, int cols, float eps, cudaStream_t s) {
  // Narrow rows: a warp each, four to a block. Above 1024 columns a block per row, wide enough for four vectors a
  // thread. Blocks are handed out as they finish, so no SM waits for a longer share of rows.
  const int quads = (rows + 3) / 4;
  if (cols <= 256) k_rmsnorm_fwd_reg<32, 1, ADD><<<quads, 128, 0, s>>>(x, delta, w, sum, y, rstd, rows, cols, eps);
  else if (cols <= 512) k_rmsnorm_fwd_reg<32, 2, ADD><<<quads, 128, 0, s>>>(x, delta, w, sum, y, rstd, rows, cols, eps);
  else if (cols <= 1024) k_rmsnorm_fwd_reg<32, 4, ADD><<<quads, 128, 0, s>>>(x, delta, w, sum, y, rstd, rows, cols, eps);
  else if (cols <= 2048) k_rmsnorm_fwd_reg<128, 2, ADD><<<rows, 128, 0, s>>>(x, delta, w, sum, y, rstd, rows, cols, eps);
  else if (cols <= 4096) k_rmsnorm_fwd_reg<128, 4, ADD><<<rows, 128, 0, s>>>(x, delta, w, sum, y, rstd, rows, cols, eps);
  else k_rmsnorm_fwd_reg<256, 4, ADD><<<rows, 256, 0, s>>>(x, delta, w, sum, y, rstd, rows, cols, eps);
}

// Rows of the backward as a warp each, eight to a block, or as a block each (every row that needs more than 1024
// columns). A warp holds up to 32 elements of its row and the block then adds up eight shares of the weight gradient;
// with few rows that is a longer chain than a block per row, whose many partial rows cost more from some rows on.
// Warp / block, in us with the column sum: 1 x 776 5.0 / 3.5, 64 x 776 5.4 / 4.1, 148 x 1024 5.4 / 4.5, 200 x 1024
// 5.5 / 5.5, 296 x 1024 5.7 / 6.0; 16 x 512 4.3 / 3.7, 64 x 512 4.5 / 4.2, 148 x 512 4.5 / 4.5, 200 x 512 4.5 / 5.0;
// 1 x 256 3.8 / 3.5.
bool bwd_warp_rows(int rows, int cols) {
  return cols <= 1024 && rows > (cols > 512 ? kSms : cols > 256 ? kSms / 2 : 4);
}

template <bool ADD>
void rmsnorm_bwd_rows(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const float* rstd,
                      const __nv_bfloat16* dskip, __nv_bfloat16* dx, float* part, int blocks, int rows, int cols, cudaStream_t s) {
  if (cols <= 2048 && !bwd_warp_rows(rows, cols)) k_rmsnorm_bwd<256, 1, ADD><<<blocks, kNormThreads, 0, s>>>(dy, x, w, rstd, dskip, dx, part, rows, cols);
  else if (cols <= 256) k_rmsnorm_bwd<32, 1, ADD><<<blocks, kNormThreads, 0, s>>>(dy, x, w, rstd, dskip, dx, part, rows, cols);
  else if (cols <= 512) k_rmsnorm_bwd<32, 2, ADD><<<blocks, kNormThreads, 0, s>>>(dy, x, w, rstd, dskip, dx, part, rows, cols);
  else if (cols <= 1024) k_rmsnorm_bwd<32, 4, ADD><<<blocks, kNormThreads, 0, s>>>(dy, x, w, rstd, dskip, dx, part, rows, cols);
  else if (cols <= 4096) k_rmsnorm_bwd<256, 2, ADD><<<blocks, kNormThreads, 0, s>>>(dy, x, w, rstd, dskip, dx, part, rows, cols);
  else k_rmsnorm_bwd<512, 2, ADD><<<blocks, 512, 0, s>>>(dy, x, w, rstd, dskip, dx, part, rows, cols);
}

} // namespace

cudaError_t launch_rmsnorm_fwd(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* y, float* rstd, int rows,
                               int cols, float eps, cudaStream_t s, const __nv_bfloat16* delta, __nv_bfloat16* sum) {
  if (cols % 8 != 0 || rows <= 0) return cudaErrorInvalidValue;
  if (misaligned16(x, w, y, delta, sum)) return cudaErrorMisalignedAddress;
  if (delta != nullptr) {
    if (cols > kNormThreads * kNormMaxVec * 8 || sum == nullptr) return cudaErrorInvalidValue;
    rmsnorm_fwd_rows<true>(x, delta, w, sum, y, rstd, rows, cols, eps, s);
  } else if (cols <= kNormThreads * kNormMaxVec * 8) {
    rmsnorm_fwd_rows<false>(x, nullptr, w, nullptr, y, rstd, rows, cols, eps, s);
  } else {
    k_rmsnorm_fwd_wide<<<std::min(rows, kSms * 8), kNormThreads, 0, s>>>(x, w, y, rstd, rows, cols, eps);
  }
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_rmsnorm_bwd(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w,
                               const float* rstd, __nv_bfloat16* dx, float* dw_partial, int* nblocks, int rows,
                               int cols, cudaStream_t s, const __nv_bfloat16* dskip) {
  if (cols % 8 != 0 || rows <= 0 || cols > kNormThreads * kNormMaxVec * 8) return cudaErrorInvalidValue;
  const bool warp_rows = bwd_warp_rows(rows, cols);
  const int per_sm = cols > 4096 ? norm_bwd_per_sm<512, 2>() : (cols > 512 && warp_rows) ? norm_bwd_per_sm<32, 4>() : 2;
  const int blocks = std::min(warp_rows ? (rows + 7) / 8 : rows, kSms * per_sm);
  if (nblocks) *nblocks = blocks;
  if (dw_partial == nullptr) return cudaSuccess;
  if (misaligned16(dy, x, w, dx, dskip, dw_partial)) return cudaErrorMisalignedAddress;
  if (dskip != nullptr) rmsnorm_bwd_rows<true>(dy, x, w, rstd, dskip, dx, dw_partial, blocks, rows, cols, s);
  else rmsnorm_bwd_rows<false>(dy, x, w, rstd, nullptr, dx, dw_partial, blocks, rows, cols, s);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_cast_scale(const void* in, int in_kind, void* out, int out_kind, size_t n, float scale, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const size_t in_bytes = in_kind == 0 ? 4 : 2, out_bytes = out_kind == 0 ? 4 : 2;
  // Vector accesses of 8 elements: 32-byte (fp32) or 16-byte (bf16) alignment of the bases.
  if ((reinterpret_cast<uintptr_t>(in) % (8 * in_bytes)) != 0 || (reinterpret_cast<uintptr_t>(out) % (8 * out_bytes)) != 0) {
    return cudaErrorInvalidValue;
  }
  const unsigned grid = covering_grid(n / 8, 256 * kCastVecs);
  if (in_kind == 0 && out_kind == 0) k_cast_scale<float, float><<<grid, 256, 0, s>>>(static_cast<const float*>(in), static_cast<float*>(out), n, scale);
  else if (in_kind == 0 && out_kind == 1) k_cast_scale<float, __nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const float*>(in), static_cast<__nv_bfloat16*>(out), n, scale);
  else if (in_kind == 1 && out_kind == 0) k_cast_scale<__nv_bfloat16, float><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(in), static_cast<float*>(out), n, scale);
  else k_cast_scale<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(in), static_cast<__nv_bfloat16*>(out), n, scale);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_quantize_rows(const __nv_bfloat16* x, int64_t ld, void* q, float* scale, int rows, int cols, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return cudaErrorInvalidValue;
  const uintptr_t xa = reinterpret_cast<uintptr_t>(x), qa = reinterpret_cast<uintptr_t>(q);
  const bool wide = cols % 16 == 0 && ld % 16 == 0 && xa % 32 == 0 && qa % 16 == 0;
  const bool vec = cols % 8 == 0 && ld % 8 == 0 && xa % 16 == 0 && qa % 8 == 0;
  // Enough threads that a row of up to KEEP accesses each stays in registers; with few rows on the GPU more threads
  // shorten the row instead.
  const unsigned threads = cols <= 1024 ? 32 : cols <= 4096 && (wide || rows > kSms * 4) ? 128 : 256;
  const auto kernel = !wide ? (vec ? k_quantize_rows<8, 8> : k_quantize_rows<1, 1>) : cols > 8192 ? k_quantize_rows<16, 4> : k_quantize_rows<16, 2>;
  launch_early(kernel, static_cast<unsigned>(rows), threads, s, x, ld, static_cast<uint8_t*>(q), scale, cols);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_colsum_bf16(const float* in, __nv_bfloat16* out, int rows, int cols, cudaStream_t s) {
  if (cols % 4 != 0 || (reinterpret_cast<uintptr_t>(in) & 15u) != 0) return cudaErrorInvalidValue;
  k_colsum_bf16<<<(cols + kColsumCols - 1) / kColsumCols, 256, 0, s>>>(in, out, rows, cols);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_rope(const __nv_bfloat16* x, int64_t stride_t, int64_t stride_h, __nv_bfloat16* y, const int* pos,
                        const float* cos_t, const float* sin_t, int tokens, int heads, int head_dim, bool inverse,
                        cudaStream_t s) {
  if (head_dim % 8 != 0 || stride_t % 8 != 0 || stride_h % 8 != 0) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(cos_t) |
       reinterpret_cast<uintptr_t>(sin_t)) & 15u) {
    return cudaErrorMisalignedAddress;
  }
  const int per_head = head_dim / 8;
  const size_t per_token = static_cast<size_t>(heads) * per_head;
  if (tokens <= 0 || per_token == 0) return cudaSuccess;
  // 32-bit indices inside a launch: very large tensors go in slices of whole tokens.
  const size_t slice = std::max<size_t>(1, (size_t{1} << 30) / per_token);
  if (per_token > (size_t{1} << 30)) return cudaErrorInvalidValue;
  for (size_t t0 = 0; t0 < static_cast<size_t>(tokens); t0 += slice) {
    const size_t nt = std::min(slice, static_cast<size_t>(tokens) - t0);
    const uint32_t total = static_cast<uint32_t>(nt * per_token);
    const int blocks = static_cast<int>((total + 256u * kRopeVecs - 1) / (256u * kRopeVecs));
    k_rope<<<blocks, 256, 0, s>>>(x + static_cast<int64_t>(t0) * stride_t, y + t0 * per_token * 8, pos + t0, cos_t, sin_t, total,
                                  make_fast_div(per_head), make_fast_div(heads), stride_t, stride_h, inverse ? -1.0f : 1.0f);
    note_kernel_launch();
  }
  return cudaGetLastError();
}

namespace {

// Calls fn(first row, vectors) for slices of whole rows whose vectors fit 32-bit indices (one slice but for tensors
// of many gigabytes).
template <typename Fn>
cudaError_t for_row_slices(int rows, int per_row, Fn fn) {
  if (rows <= 0 || per_row <= 0) return cudaSuccess;
  const int slice = std::max(1, (1 << 30) / per_row);
  for (int r0 = 0; r0 < rows; r0 += std::min(slice, rows - r0)) {
    const uint32_t total = static_cast<uint32_t>(std::min(slice, rows - r0)) * static_cast<uint32_t>(per_row);
    fn(static_cast<size_t>(r0), total);
    note_kernel_launch();
  }
  return cudaGetLastError();
}

// Vectors per thread of the SwiGLU kernels (see there).
unsigned swiglu_vecs(uint32_t total) { return total <= static_cast<uint32_t>(kSms) * 2048u ? 1u : 2u; }

} // namespace

cudaError_t launch_split_rope(__nv_bfloat16* packed, int64_t ld, __nv_bfloat16* const* parts, const int64_t* stride_t,
                              const int64_t* stride_h, const int* pos, const float* cos_t, const float* sin_t, int tokens,
                              int heads, int kv_heads, int head_dim, bool backward, cudaStream_t s) {
  if (head_dim <= 0 || head_dim % 8 != 0 || heads <= 0 || kv_heads <= 0 || ld % 8 != 0) return cudaErrorInvalidValue;
  QkvParts q{};
  uintptr_t bits = reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t);
  for (int i = 0; i < 3; ++i) {
    if (stride_t[i] % 8 != 0 || stride_h[i] % 8 != 0) return cudaErrorInvalidValue;
    q.p[i] = parts[i];
    q.stride_t[i] = stride_t[i];
    q.stride_h[i] = stride_h[i];
    bits |= reinterpret_cast<uintptr_t>(parts[i]);
  }
  if (bits & 15u) return cudaErrorMisalignedAddress;
  const int all = heads + 2 * kv_heads, per_head = head_dim / 8;
  return for_row_slices(tokens, all * per_head, [&](size_t t0, uint32_t total) {
    QkvParts here = q;
    for (int i = 0; i < 3; ++i) here.p[i] += static_cast<int64_t>(t0) * q.stride_t[i];
    const int blocks = static_cast<int>((total + 256u * kRopeVecs - 1) / (256u * kRopeVecs));
    if (backward) {
      k_split_rope<false><<<blocks, 256, 0, s>>>(packed + static_cast<int64_t>(t0) * ld, ld, here, pos + t0, cos_t, sin_t, total,
                                                 make_fast_div(per_head), make_fast_div(all), heads, kv_heads);
    } else {
      k_split_rope<true><<<blocks, 256, 0, s>>>(packed + static_cast<int64_t>(t0) * ld, ld, here, pos + t0, cos_t, sin_t, total,
                                                make_fast_div(per_head), make_fast_div(all), heads, kv_heads);
    }
  });
}

cudaError_t launch_swiglu_fwd(const __nv_bfloat16* gate_up, __nv_bfloat16* h, int rows, int ffn, cudaStream_t s) {
  if (ffn % 8 != 0) return cudaErrorInvalidValue;
  if (misaligned16(gate_up, h)) return cudaErrorMisalignedAddress;
  return for_row_slices(rows, ffn / 8, [&](size_t r0, uint32_t total) {
    const unsigned vecs = swiglu_vecs(total);
    launch_early(vecs == 1 ? k_swiglu_fwd<1> : k_swiglu_fwd<2>, covering_grid(total, 256 * vecs), 256, s, gate_up + r0 * 2 * ffn,
                 h + r0 * ffn, total, make_fast_div(ffn / 8));
  });
}

cudaError_t launch_swiglu_bwd(const __nv_bfloat16* dh, const __nv_bfloat16* gate_up, __nv_bfloat16* dgate_up, int rows,
                              int ffn, cudaStream_t s) {
  if (ffn % 8 != 0) return cudaErrorInvalidValue;
  if (misaligned16(dh, gate_up, dgate_up)) return cudaErrorMisalignedAddress;
  return for_row_slices(rows, ffn / 8, [&](size_t r0, uint32_t total) {
    const unsigned vecs = swiglu_vecs(total);
    launch_early(vecs == 1 ? k_swiglu_bwd<1> : k_swiglu_bwd<2>, covering_grid(total, 256 * vecs), 256, s, dh + r0 * ffn,
                 gate_up + r0 * 2 * ffn, dgate_up + r0 * 2 * ffn, total, make_fast_div(ffn / 8));
  });
}

cudaError_t launch_cross_entropy_fwd_bwd(__nv_bfloat16* logits, int64_t ld, const int64_t* targets, float* loss, int rows,
                                         int vocab, float grad_scale, cudaStream_t s) {
  if (rows <= 0 || vocab <= 0 || ld < vocab) return cudaErrorInvalidValue;
  // Rows in work at a time: 296 rows of a 128k vocabulary are 76 MB, which the 126 MB L2 keeps for the second
  // look; shorter rows take smaller blocks, more of them per SM, and stay below that. Every block has at least 128
  // threads: one for each element outside the vectors.
  const int threads = vocab <= 4096 ? 128 : vocab <= 16384 ? 256 : kCeMaxThreads;
  const int blocks = std::min(rows, kSms * 2 * (kCeMaxThreads / threads));
  k_cross_entropy<<<blocks, threads, 0, s>>>(logits, ld, targets, loss, rows, vocab, grad_scale);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_head_gradient(__nv_bfloat16* logits, int64_t ld, const int64_t* targets, const float2* stats, const float* fine, int shares,
                                 const float* target_logit, float* row_scratch, float* loss, uint32_t* words, int rows, int vocab,
                                 float grad_scale, float loss_scale, bool first, cudaStream_t s) {
  if (rows <= 0 || vocab <= 0 || shares <= 0 || ld % 16 != 0 || ld < vocab) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(logits) & 31u) != 0) return cudaErrorMisalignedAddress;
  const int nvec = (vocab + 15) / 16, threads = std::min(kGradThreads, (nvec + 31) / 32 * 32), parts = (nvec + threads - 1) / threads;
  if (static_cast<int64_t>(rows) * parts > INT32_MAX) return cudaErrorInvalidValue;
  const HeadGrad a{logits, ld, targets, stats, fine, target_logit, row_scratch, row_scratch + rows, loss, words, rows, shares, vocab, parts,
                   first ? 1 : 0, grad_scale, loss_scale};
  const unsigned grid = static_cast<unsigned>(rows) * static_cast<unsigned>(parts);
  if (grid > kGradFused) {
    launch_early(k_head_rows, static_cast<unsigned>((rows + 31) / 32), 512, s, a);
    note_kernel_launch();
    launch_early(k_head_gradient<true>, grid, threads, s, a);
  } else {
    launch_early(k_head_gradient<false>, grid, threads, s, a);
  }
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_head_tail(const float* part, const __nv_bfloat16* grad, int64_t ld, const __nv_bfloat16* w, __nv_bfloat16* dx, int rows,
                             int cols, int depth, cudaStream_t s) {
  if (cols <= 0 || cols % 8 != 0) return cudaErrorInvalidValue;
  if (misaligned16(part, w, dx)) return cudaErrorMisalignedAddress;
  return for_row_slices(rows, cols / 8, [&](size_t r0, uint32_t total) {
    k_head_tail<<<covering_grid(total, 256), 256, 0, s>>>(part + r0 * cols, grad + static_cast<int64_t>(r0) * ld, ld, w, dx + r0 * cols, total,
                                                          make_fast_div(cols / 8), depth);
  });
}

cudaError_t launch_scale_bf16(const __nv_bfloat16* in, __nv_bfloat16* out, const float* factor, size_t n, cudaStream_t s,
                              const __nv_bfloat16* in2, __nv_bfloat16* out2, size_t n2) {
  if (n == 0 && n2 == 0) return cudaSuccess;
  if (misaligned16(in, out, in2, out2)) return cudaErrorMisalignedAddress;
  const dim3 grid(std::min<unsigned>(covering_grid(std::max(n, n2) / 8, 256 * 4), kSms * 8), n2 != 0 ? 2 : 1);
  k_scale_bf16<<<grid, 256, 0, s>>>(ScaleSpan{in, out, n}, ScaleSpan{in2, out2, n2}, factor);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_adamw(float* p, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2,
                         float eps, float weight_decay, int step, float grad_scale, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (n >= 4 && misaligned16(p, g, m, v)) return cudaErrorMisalignedAddress;  // fewer elements use no vectors
  const float bias1 = 1.0f - powf(beta1, static_cast<float>(step));
  const float bias2 = 1.0f - powf(beta2, static_cast<float>(step));
  const unsigned vecs = n / 4 <= static_cast<size_t>(kSms) * 3 * 256 ? 1u : 2u;
  (vecs == 1 ? k_adamw<1> : k_adamw<2>)<<<covering_grid(n / 4, 256 * vecs), 256, 0, s>>>(p, g, m, v, n, lr, beta1, beta2, eps,
                                                                                         weight_decay, bias1, bias2, grad_scale);
  note_kernel_launch();
  return cudaGetLastError();
}

} // namespace b200c
