// MoE expert-parallel dispatch / combine kernels (sm_100a). See moe_ep.h.
#include "moe_ep.h"

#include <cooperative_groups.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <vector>

#include "early_launch.cuh"
#include "launch_count.h"

namespace cg = cooperative_groups;

namespace b200c {

namespace {

constexpr int kEpThreads = 256;
constexpr int kEpWarps = kEpThreads / 32;

__device__ __forceinline__ float2 bf2f(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// Cross-GPU barrier by block 0 of every rank, on flag row 0 of the EP set.
__device__ __forceinline__ bool ep_rank_barrier(const CommDev& c, uint32_t phase) {
  BlockEpoch ep;
  ep.load(c, kFlagSetEp);
  const bool ok = block_barrier(c, kFlagSetEp, ep, phase);
  ep.store(c, kFlagSetEp);
  return ok;
}

struct DispatchArgs {
  const void* x;          // [num_tokens, hidden] bf16
  const int* topk_idx;    // [num_tokens, topk]
  const float* topk_w;    // [num_tokens, topk]
  int num_tokens;
  int per_block;          // single rank: tokens of a block, at most one per warp
};

// 16 bf16 of a lane to e4m3, with one scale per 128 elements (8 neighbouring lanes). Returns the scale.
__device__ __forceinline__ float ep_quantize16(uint4 v0, uint4 v1, uint4* packed) {
  float f[16];
  const uint32_t* p0 = &v0.x;
  const uint32_t* p1 = &v1.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a0 = bf2f(p0[j]), a1 = bf2f(p1[j]);
    f[2 * j] = a0.x;
    f[2 * j + 1] = a0.y;
    f[8 + 2 * j] = a1.x;
    f[8 + 2 * j + 1] = a1.y;
  }
  float amax = 0.0f;
#pragma unroll
  for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
  amax = fmaxf(amax, 1e-4f);
  const float inv = 448.0f / amax;
  uint32_t q[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j] * inv, f[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j + 2] * inv, f[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    q[j] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
  *packed = make_uint4(q[0], q[1], q[2], q[3]);
  return amax / 448.0f;
}

constexpr int kEpChunkCols = 1024;  // columns of one work item of the send loop (a multiple of 512)

// Bound by memory (a bf16 row in, a quantised row out), so what counts is how many bytes are in flight and how
// little happens before the rows move. Tokens are numbered per destination by a thread each: ballots inside a
// warp, one atomic per block and destination. The send loop hands out pieces of rows, so that every warp has the
// same share and issues its whole piece's loads at once. (4096 tokens of 7168 to e4m3 on one rank, when that ran
// here: 49.6 us with a warp per token and more grid-wide meetings, 23.4 us in this form.)
__device__ void ep_dispatch_body(const CommDev& c, const EpDev& e, const DispatchArgs& a) {
  cg::grid_group grid = cg::this_grid();
  __shared__ int s_first[kEpWarps][kMaxRanks];  // tokens of the block's earlier warps, per destination
  __shared__ int s_base[kMaxRanks];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gwarp = blockIdx.x * kEpWarps + warp, nwarps = gridDim.x * kEpWarps;

  trace_mark(c, 0);
  // A. number the tokens per destination rank (e.cnt is zero between calls)
  for (int t0 = blockIdx.x * kEpThreads; t0 < a.num_tokens; t0 += gridDim.x * kEpThreads) {
    const int t = t0 + static_cast<int>(threadIdx.x);
    uint32_t mask = 0;
    if (t < a.num_tokens) {
      const int* ids = a.topk_idx + static_cast<size_t>(t) * e.topk;
      for (int k = 0; k < e.topk; ++k) {
        const int idx = ids[k];
        if (idx >= 0 && idx < e.num_experts) mask |= 1u << (idx / e.experts_per_rank);
      }
    }
    int before[kMaxRanks];
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d) {
      if (d < e.nranks) {
        const uint32_t has = __ballot_sync(0xffffffffu, (mask >> d) & 1u);
        before[d] = __popc(has & ((1u << lane) - 1u));
        if (lane == 0) s_first[warp][d] = __popc(has);
      }
    }
    __syncthreads();
    if (threadIdx.x < e.nranks) {
      int total = 0;
      for (int w = 0; w < kEpWarps; ++w) {
        const int n = s_first[w][threadIdx.x];
        s_first[w][threadIdx.x] = total;
        total += n;
      }
      s_base[threadIdx.x] = total > 0 ? atomicAdd(&e.cnt[threadIdx.x], total) : 0;
    }
    __syncthreads();
    if (t < a.num_tokens) {
#pragma unroll
      for (int d = 0; d < kMaxRanks; ++d) {
        if (d < e.nranks) {
          e.order[static_cast<size_t>(t) * e.nranks + d] = (mask >> d) & 1u ? s_base[d] + s_first[warp][d] + before[d] : -1;
        }
      }
    }
    __syncthreads();
  }
  grid.sync();
  trace_mark(c, 1);

  // B. publish the counts to every rank, learn where this rank's rows start inside each destination's receive
  //    buffer (rows are packed by source).
  if (blockIdx.x == 0) {
    if (threadIdx.x < e.nranks) {
      const int d = threadIdx.x;
      const long long n = e.cnt[d];
      e.cnt[d] = 0;  // nobody else looks at it any more; the next call starts from zero
      for (int p = 0; p < e.nranks; ++p) {
        e.count_matrix[p][e.rank * e.nranks + d] = n;
      }
    }
    ep_rank_barrier(c, 0x91);
    const long long* m = e.count_matrix[e.rank];
    if (threadIdx.x < e.nranks) {
      const int d = threadIdx.x;
      long long b = 0;
      for (int s = 0; s < e.rank; ++s) b += m[s * e.nranks + d];
      e.base[d] = b;
      e.recv_info[1 + d] = static_cast<int>(m[d * e.nranks + e.rank]);  // rows from source d
    }
    if (threadIdx.x == 0) {
      long long total = 0;
      for (int s = 0; s < e.nranks; ++s) total += m[s * e.nranks + e.rank];
      e.recv_info[0] = static_cast<int>(total);
    }
  }
  grid.sync();
  trace_mark(c, 2);

  // C. quantise and send; one work item = one token x kEpChunkCols columns
  const int groups = e.hidden / 128;
  const size_t row_bytes = e.fp8 ? static_cast<size_t>(e.hidden) : static_cast<size_t>(e.hidden) * 2;
  const int nchunks = (e.hidden + kEpChunkCols - 1) / kEpChunkCols;
  for (int item = gwarp; item < a.num_tokens * nchunks; item += nwarps) {
    const int t = item / nchunks, chunk = item - t * nchunks;
    // payload: 16 elements per lane and step, 8 lanes share one 128-element group
    const __nv_bfloat16* xr = static_cast<const __nv_bfloat16*>(a.x) + static_cast<size_t>(t) * e.hidden;
    constexpr int kSteps = kEpChunkCols / 512;
    const int col0 = chunk * kEpChunkCols + lane * 16;
    uint4 v0[kSteps], v1[kSteps];
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      if (col0 + i * 512 < e.hidden) {
        v0[i] = ld16_stream(xr + col0 + i * 512);
        v1[i] = ld16_stream(xr + col0 + i * 512 + 8);
      }
    }
    int slot = -1;
    if (lane < e.nranks) {
      const int n = e.order[static_cast<size_t>(t) * e.nranks + lane];
      if (n >= 0) {
        slot = static_cast<int>(e.base[lane]) + n;
        if (slot >= e.nranks * e.max_tokens) {  // cannot happen with consistent inputs; never write out of bounds
          c.status[0] = c.status[0] | kStatusBadArg;
          slot = -1;
        }
      }
      if (chunk == 0) e.send_slot[static_cast<size_t>(t) * e.nranks + lane] = slot;
    }
    if (chunk == 0) {  // metadata
      const int idx = lane < e.topk ? a.topk_idx[static_cast<size_t>(t) * e.topk + lane] : -1;
      const float w = lane < e.topk ? a.topk_w[static_cast<size_t>(t) * e.topk + lane] : 0.0f;
      for (int d = 0; d < e.nranks; ++d) {
        const int sd = __shfl_sync(0xffffffffu, slot, d);
        if (sd < 0) continue;
        if (lane < e.topk) {
          const bool here = idx >= 0 && idx / e.experts_per_rank == d;
          e.recv_topk_idx[d][static_cast<size_t>(sd) * e.topk + lane] = here ? idx - d * e.experts_per_rank : -1;
          e.recv_topk_w[d][static_cast<size_t>(sd) * e.topk + lane] = here ? w : 0.0f;
        }
        if (lane == 0) e.recv_src[d][sd] = e.rank * e.max_tokens + t;
      }
    }
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      const int e0 = col0 + i * 512;
      if (e0 - lane * 16 >= e.hidden) break;  // hidden is a multiple of 512: the whole warp agrees
      if (!e.fp8) {
        for (int d = 0; d < e.nranks; ++d) {
          const int sd = __shfl_sync(0xffffffffu, slot, d);
          if (sd < 0) continue;
          char* dst = e.recv_x[d] + static_cast<size_t>(sd) * row_bytes + static_cast<size_t>(e0) * 2;
          st16(dst, v0[i]);
          st16(dst + 16, v1[i]);
        }
        continue;
      }
      uint4 packed;
      const float scale = ep_quantize16(v0[i], v1[i], &packed);
      const int group = e0 / 128;
      for (int d = 0; d < e.nranks; ++d) {
        const int sd = __shfl_sync(0xffffffffu, slot, d);
        if (sd < 0) continue;
        st16(e.recv_x[d] + static_cast<size_t>(sd) * row_bytes + e0, packed);
        if ((lane & 7) == 0) e.recv_scales[d][static_cast<size_t>(sd) * groups + group] = scale;
      }
    }
  }
  trace_mark(c, 3);
  grid.sync();
  // D. every rank's rows have landed before anybody returns
  if (blockIdx.x == 0) {
    ep_rank_barrier(c, 0x92);
    trace_mark(c, 4);
  }
}

__global__ void __launch_bounds__(kEpThreads) k_ep_dispatch(CommDev c, EpDev e, DispatchArgs a) {
  ep_dispatch_body(c, e, a);
}
__global__ void __launch_bounds__(kEpThreads) k_ep_dispatch_emu(const CommDev* cs, const EpDev* es, const DispatchArgs* as) {
  ep_dispatch_body(cs[blockIdx.y], es[blockIdx.y], as[blockIdx.y]);
}

// A single rank: rows may stand in any order from 0, so a block numbers its own tokens with one atomic and sends them
// at once, and nobody waits for anybody. The last block to finish leaves the count. An ordinary launch that covers
// the tokens, where the general kernel is a cooperative one with grid-wide meetings (4096 tokens of 7168 to e4m3:
// 23.3 us there, 18.5 us (4.8 TB/s) here; as they are 20.4 (5.8 TB/s)). How many tokens a block takes: solo_blocks().
// Started early, a dispatch and a combine of 128 x 7168 to e4m3 through a communicator take 1.3 us less in a graph and 0.8 on
// the stream, of 4096 x 7168 2.0 and 3.1.

template <int THREADS, int COLS, bool WIDE, bool TRACE>
__global__ void __launch_bounds__(THREADS) k_ep_dispatch_solo(CommDev c, EpDev e, DispatchArgs a) {
  constexpr int kWarps = THREADS / 32, kSteps = COLS / 512;
  __shared__ int s_slot[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = blockIdx.x * a.per_block, here = min(a.per_block, a.num_tokens - t0);
  const int groups = e.hidden / 128, nchunks = (e.hidden + COLS - 1) / COLS;
  const size_t row_bytes = e.fp8 ? static_cast<size_t>(e.hidden) : static_cast<size_t>(e.hidden) * 2;
  grid_release();
  grid_wait();
  trace_mark<TRACE>(c, 0);  // the marks of the general kernel
  uint4 v0[kSteps], v1[kSteps];
  auto load = [&](int item) {
    const int t = t0 + item / nchunks, col0 = (item % nchunks) * COLS + lane * 16;
    const __nv_bfloat16* xr = static_cast<const __nv_bfloat16*>(a.x) + static_cast<size_t>(t) * e.hidden;
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      if (col0 + i * 512 < e.hidden) {
        if constexpr (WIDE) {
          ld32_stream(xr + col0 + i * 512, v0[i], v1[i]);
        } else {
          v0[i] = ld16_stream(xr + col0 + i * 512);
          v1[i] = ld16_stream(xr + col0 + i * 512 + 8);
        }
      }
    }
  };
  int item = warp;
  if (item < here * nchunks) load(item);  // in flight while the tokens are numbered
  int idx = -1;
  float w = 0.0f;
  if (warp < here) {
    const size_t at = static_cast<size_t>(t0 + warp) * e.topk + lane;
    if (lane < e.topk) {
      idx = a.topk_idx[at];
      w = a.topk_w[at];
    }
    const bool sent = __any_sync(0xffffffffu, idx >= 0 && idx < e.num_experts);
    if (lane == 0) s_slot[warp] = sent ? 0 : -1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int i = 0; i < here; ++i) n += s_slot[i] >= 0 ? 1 : 0;
    int next = n > 0 ? atomicAdd(&e.cnt[0], n) : 0;
    for (int i = 0; i < here; ++i) {
      if (s_slot[i] < 0) continue;
      s_slot[i] = next++;
      if (s_slot[i] >= e.max_tokens) {  // cannot happen with consistent inputs; never write out of bounds
        c.status[0] = c.status[0] | kStatusBadArg;
        s_slot[i] = -1;
      }
    }
  }
  __syncthreads();
  trace_mark<TRACE>(c, 1);
  trace_mark<TRACE>(c, 2);  // no counts to exchange
  if (warp < here) {  // metadata
    const int slot = s_slot[warp];
    if (lane == 0) e.send_slot[t0 + warp] = slot;
    if (slot >= 0) {
      if (lane < e.topk) {
        const bool valid = idx >= 0 && idx < e.num_experts;
        e.recv_topk_idx[0][static_cast<size_t>(slot) * e.topk + lane] = valid ? idx : -1;
        e.recv_topk_w[0][static_cast<size_t>(slot) * e.topk + lane] = valid ? w : 0.0f;
      }
      if (lane == 0) e.recv_src[0][slot] = t0 + warp;
    }
  }
  while (item < here * nchunks) {
    const int slot = s_slot[item / nchunks], col0 = (item % nchunks) * COLS + lane * 16;
    if (slot >= 0) {
#pragma unroll
      for (int i = 0; i < kSteps; ++i) {
        const int e0 = col0 + i * 512;
        if (e0 - lane * 16 >= e.hidden) break;  // hidden is a multiple of 512: the whole warp agrees
        if (e.fp8) {
          uint4 packed;
          const float scale = ep_quantize16(v0[i], v1[i], &packed);
          st16(e.recv_x[0] + static_cast<size_t>(slot) * row_bytes + e0, packed);
          if ((lane & 7) == 0) e.recv_scales[0][static_cast<size_t>(slot) * groups + e0 / 128] = scale;
        } else {
          st32(e.recv_x[0] + static_cast<size_t>(slot) * row_bytes + static_cast<size_t>(e0) * 2, v0[i], v1[i]);
        }
      }
    }
    item += kWarps;
    if (item < here * nchunks) load(item);
  }
  trace_mark<TRACE>(c, 3);
  if (threadIdx.x == 0) {
    __threadfence();  // this block's numbers are counted before it reports
    if (atomicAdd(e.ticket, 1) == static_cast<int>(gridDim.x) - 1) {
      __threadfence();
      const int total = __ldcg(e.cnt);
      e.recv_info[0] = total;
      e.recv_info[1] = total;
      e.cnt[0] = 0;
      *e.ticket = 0;
    }
  }
  trace_mark<TRACE>(c, 4);
}

struct CombineArgs {
  void* out;             // [num_tokens, hidden] bf16
  const float* weights;  // [num_tokens, nranks] or nullptr
  const void* bias;      // [num_tokens, hidden] bf16 or nullptr
  int num_tokens;
  const int* send_slot;  // [num_tokens, nranks] handle of the dispatch to undo; nullptr = the last one's
  float* topk_w_out;     // [num_tokens, topk] or nullptr
};

// Pull combine: the token's owner reads the expert output of every rank the
// token went to straight out of that rank's `combine_x` (the row is the slot
// the dispatch recorded in `send_slot`) and forms the weighted sum in
// registers. Each row crosses NVLink once and nothing is staged. Every block
// meets its peers' blocks before (all expert outputs are complete) and after
// (nobody still reads this rank's outputs), so the kernel needs no grid-wide
// synchronisation. Bound by memory: COLS 16-byte columns of every source are in
// flight per lane. One rank (RANKS = 1) has one source per token, so it takes
// four columns and works on pieces of rows, to the same number of loads
// (4096 x 7168: 39.0 us before, now 17.0, 6.9 TB/s).
template <int RANKS, int COLS, bool TRACE>
__device__ void ep_combine_body(const CommDev& c, const EpDev& e, const CombineArgs& a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gwarp = blockIdx.x * kEpWarps + warp, nwarps = gridDim.x * kEpWarps;
  const size_t row_bytes = static_cast<size_t>(e.hidden) * 2;
  const int cap_rows = e.nranks * e.max_tokens;
  const int* send_slot = a.send_slot != nullptr ? a.send_slot : e.send_slot;
  BlockEpoch ep;
  if (RANKS > 1) ep.load(c, kFlagSetEp);
  trace_mark<TRACE>(c, 0);
  bool ok = RANKS == 1 || block_barrier(c, kFlagSetEp, ep, 0x93);
  trace_mark<TRACE>(c, 1);
  if (ok) {
    const int piece = RANKS == 1 ? COLS * 256 : e.hidden;  // columns of one work item
    const int pieces = (e.hidden + piece - 1) / piece;
    for (int item = gwarp; item < a.num_tokens * pieces; item += nwarps) {
      const int t = item / pieces, col_lo = (item - t * pieces) * piece;
      int slot = -1;
      float wt = 1.0f;
      if (lane < e.nranks) {
        slot = send_slot[static_cast<size_t>(t) * e.nranks + lane];
        if (slot >= cap_rows) {  // never read through a bad index
          c.status[0] = c.status[0] | kStatusBadArg;
          slot = -1;
        }
        if (a.weights != nullptr) wt = a.weights[static_cast<size_t>(t) * e.nranks + lane];
      }
      const uint32_t have = __ballot_sync(0xffffffffu, slot >= 0);
      if (a.topk_w_out != nullptr && col_lo == 0) {
        // Per-expert weights travel back with the rows: entry k is non-zero on the one rank that hosts expert k.
        float acc_w = 0.0f;
        for (int d = 0; d < e.nranks; ++d) {
          const int sd = __shfl_sync(0xffffffffu, slot, d);
          if (((have >> d) & 1u) && lane < e.topk) acc_w += e.comb_topk_w[d][static_cast<size_t>(sd) * e.topk + lane];
        }
        if (lane < e.topk) a.topk_w_out[static_cast<size_t>(t) * e.topk + lane] = acc_w;
      }
      const int col_hi = min(e.hidden, col_lo + piece);
      for (int e0 = col_lo + lane * 8; e0 < col_hi; e0 += COLS * 256) {
        uint4 rows[COLS][RANKS];
#pragma unroll
        for (int i = 0; i < RANKS; ++i) {
          if (i < e.nranks) {
            // Start at the next rank so that the ranks read different peers at any time.
            int d = e.rank + 1 + i;
            if (d >= e.nranks) d -= e.nranks;
            const int sd = __shfl_sync(0xffffffffu, slot, d);
            if ((have >> d) & 1u) {
              const char* src = e.combine_x[d] + static_cast<size_t>(sd) * row_bytes + static_cast<size_t>(e0) * 2;
#pragma unroll
              for (int h = 0; h < COLS; ++h) {
                if (e0 + h * 256 < col_hi) rows[h][i] = ld16_stream(src + h * 512);
              }
            }
          }
        }
#pragma unroll
        for (int h = 0; h < COLS; ++h) {
          const int col = e0 + h * 256;
          if (col >= col_hi) break;
          float acc[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
          if (a.bias != nullptr) {
            const uint4 b = ld16(static_cast<const __nv_bfloat16*>(a.bias) + static_cast<size_t>(t) * e.hidden + col);
            const uint32_t* p = &b.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = bf2f(p[i]);
              acc[2 * i] = f.x;
              acc[2 * i + 1] = f.y;
            }
          }
#pragma unroll
          for (int i = 0; i < RANKS; ++i) {
            if (i < e.nranks) {
              int d = e.rank + 1 + i;
              if (d >= e.nranks) d -= e.nranks;
              const float wd = __shfl_sync(0xffffffffu, wt, d);
              if ((have >> d) & 1u) {
                const uint32_t* p = &rows[h][i].x;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const float2 f = bf2f(p[k]);
                  acc[2 * k] += wd * f.x;
                  acc[2 * k + 1] += wd * f.y;
                }
              }
            }
          }
          uint4 o;
          uint32_t* po = &o.x;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
            po[i] = *reinterpret_cast<uint32_t*>(&hh);
          }
          st16(static_cast<__nv_bfloat16*>(a.out) + static_cast<size_t>(t) * e.hidden + col, o);
        }
      }
    }
    trace_mark<TRACE>(c, 2);
    // Nobody overwrites its expert outputs while a peer still reads them.
    ok = RANKS == 1 || block_barrier(c, kFlagSetEp, ep, 0x94);
    trace_mark<TRACE>(c, 3);
  }
  if (RANKS > 1) ep.store(c, kFlagSetEp);
}

__global__ void __launch_bounds__(kEpThreads) k_ep_combine(CommDev c, EpDev e, CombineArgs a) {
  ep_combine_body<kMaxRanks, 2, true>(c, e, a);
}
template <bool TRACE>
__global__ void __launch_bounds__(kEpThreads) k_ep_combine_solo(CommDev c, EpDev e, CombineArgs a) {
  grid_release();
  grid_wait();
  ep_combine_body<1, 4, TRACE>(c, e, a);
}
__global__ void __launch_bounds__(kEpThreads) k_ep_combine_emu(const CommDev* cs, const EpDev* es, const CombineArgs* as) {
  ep_combine_body<kMaxRanks, 2, true>(cs[blockIdx.y], es[blockIdx.y], as[blockIdx.y]);
}

struct PullArgs {
  void* out;             // [out_rows, hidden] bf16
  const int* recv_src;   // [rows] src_rank * max_tokens + token; nullptr = the last dispatch's
  const int* num_rows;   // device count; nullptr = the last dispatch's
  int out_rows;
};

// Cached dispatch: the receiver copies the rows it was sent by an earlier
// dispatch again, this time out of the sources' `stage_x` (bf16, as is). The
// same per-block meeting before and after as in the combine.
__device__ void ep_pull_body(const CommDev& c, const EpDev& e, const PullArgs& a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gwarp = blockIdx.x * kEpWarps + warp, nwarps = gridDim.x * kEpWarps;
  const size_t row_bytes = static_cast<size_t>(e.hidden) * 2;
  const int* recv_src = a.recv_src != nullptr ? a.recv_src : e.recv_src[e.rank];
  BlockEpoch ep;
  ep.load(c, kFlagSetEp);
  bool ok = block_barrier(c, kFlagSetEp, ep, 0x95);
  if (ok) {
    int rows = a.num_rows != nullptr ? a.num_rows[0] : e.recv_info[0];
    if (rows > a.out_rows) rows = a.out_rows;
    for (int r = gwarp; r < rows; r += nwarps) {
      const int src = recv_src[r];
      const int s = src / e.max_tokens, t = src - s * e.max_tokens;
      if (src < 0 || s >= e.nranks) {  // a handle that does not belong to this buffer: skip, never read through it
        if (lane == 0) c.status[0] = c.status[0] | kStatusBadArg;
        continue;
      }
      const char* from = e.stage_x[s] + static_cast<size_t>(t) * row_bytes;
      char* to = static_cast<char*>(a.out) + static_cast<size_t>(r) * row_bytes;
      for (size_t b = static_cast<size_t>(lane) * 16; b < row_bytes; b += 2048) {
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (b + i * 512 < row_bytes) v[i] = ld16_stream(from + b + i * 512);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (b + i * 512 < row_bytes) st16(to + b + i * 512, v[i]);
        }
      }
    }
    // Nobody refills its staging rows while a peer still reads them.
    ok = block_barrier(c, kFlagSetEp, ep, 0x96);
  }
  ep.store(c, kFlagSetEp);
}

__global__ void __launch_bounds__(kEpThreads) k_ep_pull(CommDev c, EpDev e, PullArgs a) {
  ep_pull_body(c, e, a);
}
__global__ void __launch_bounds__(kEpThreads) k_ep_pull_emu(const CommDev* cs, const EpDev* es, const PullArgs* as) {
  ep_pull_body(cs[blockIdx.y], es[blockIdx.y], as[blockIdx.y]);
}

__global__ void k_ep_layout(const int* __restrict__ topk_idx, int num_tokens, int topk, int num_experts, int nranks,
                            int* __restrict__ per_rank, int* __restrict__ per_expert, int* __restrict__ in_rank) {
  const int epr = num_experts / nranks;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < num_tokens; t += gridDim.x * blockDim.x) {
    uint32_t mask = 0;
    for (int k = 0; k < topk; ++k) {
      const int idx = topk_idx[static_cast<size_t>(t) * topk + k];
      if (idx >= 0 && idx < num_experts) {
        atomicAdd(&per_expert[idx], 1);
        mask |= 1u << (idx / epr);
      }
    }
    for (int r = 0; r < nranks; ++r) {
      const int in = (mask >> r) & 1u;
      in_rank[static_cast<size_t>(t) * nranks + r] = in;
      if (in) atomicAdd(&per_rank[r], 1);
    }
  }
}

// One cooperative launch; the grid is sized so that every block is resident.
template <typename Args>
cudaError_t launch_coop(void* real_kernel, void* emu_kernel, const CommDev* comms, const EpDev* eps, int emu_ranks,
                        const std::vector<Args>& args, cudaStream_t stream) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, real_kernel, kEpThreads, 0);
  // Every block of the combine and the cached dispatch also meets its peers' blocks, itself when alone: two blocks per
  // SM (cached dispatch of 4096 x 7168 on one rank: 34.4 us, with four 35.2; of 64 x 7168 18.4 and 19.9).
  per_sm = std::max(1, std::min(per_sm, 2));
  note_kernel_launch();
  if (emu_ranks <= 0) {
    CommDev c = comms[0];
    EpDev e = eps[0];
    Args a = args[0];
    void* params[] = {&c, &e, &a};
    return cudaLaunchCooperativeKernel(real_kernel, dim3(sms * per_sm), dim3(kEpThreads), params, 0, stream);
  }
  CommDev* dc = nullptr;
  EpDev* de = nullptr;
  Args* da = nullptr;
  cudaMalloc(&dc, sizeof(CommDev) * emu_ranks);
  cudaMalloc(&de, sizeof(EpDev) * emu_ranks);
  cudaMalloc(&da, sizeof(Args) * emu_ranks);
  cudaMemcpyAsync(dc, comms, sizeof(CommDev) * emu_ranks, cudaMemcpyHostToDevice, stream);
  cudaMemcpyAsync(de, eps, sizeof(EpDev) * emu_ranks, cudaMemcpyHostToDevice, stream);
  cudaMemcpyAsync(da, args.data(), sizeof(Args) * emu_ranks, cudaMemcpyHostToDevice, stream);
  void* params[] = {&dc, &de, &da};
  const int blocks = std::max(1, sms * per_sm / emu_ranks);
  cudaError_t err = cudaLaunchCooperativeKernel(emu_kernel, dim3(blocks, emu_ranks), dim3(kEpThreads), params, 0, stream);
  cudaError_t e2 = cudaStreamSynchronize(stream);
  cudaFree(dc);
  cudaFree(de);
  cudaFree(da);
  return err != cudaSuccess ? err : e2;
}

// Blocks of the single-rank dispatch. Tokens of a block share its start and its atomic, and a wave of blocks costs that
// start once more. So while there is a shape whose blocks are all resident at once, it is the one with the fewest tokens a
// block: blocks of eight warps that take pieces of 1024 columns, four per SM, with one, two or four tokens; between two and
// four, blocks of four warps with two, which take pieces of 2048 columns, seven per SM (not for rows of 1024, which are half a
// piece). Above, where several waves run anyway, blocks of four warps: more of them start while others move rows, with half as
// many bytes again in flight; four tokens a block, two for bf16 rows of more than 4096 columns, which have more to move. In us a
// launch, replayed from a graph of 24, on eight warps with the best of 2, 4 and 8 tokens, and so: to e4m3 64 x 7168 5.1 and 4.2,
// 2048 x 7168 12.4 and 11.2, 3000 x 4096 12.4 and 10.8, 4096 x 7168 20.5 and 18.5, 6000 x 7168 28.7 and 26.8, 8192 x 4096 23.4
// and 20.3; as they are 4096 x 7168 21.9 and 20.4, 8192 x 2560 17.8 and 16.3. Around the lines, to e4m3: 1185 x 7168 8.8 with
// two tokens on four warps, 8.9 with four on eight, 2072 x 7168 11.5 and 12.7, 2200 x 7168 14.2 and 12.8, 2600 x 4096 10.0 (four
// tokens on four warps) and 10.9, 2048 x 1024 5.3 and 4.8.
struct SoloBlocks {
  int threads, tokens;
};
SoloBlocks solo_blocks(int tokens, int hidden, bool fp8) {
  constexpr int kWide = 148 * 4, kSlim = 148 * 7;  // resident at once: blocks of 256 and of 128 threads
  if (tokens <= 2 * kWide) return {256, tokens <= kWide ? 1 : 2};
  if (tokens <= 4 * kWide) return tokens <= 2 * kSlim && hidden > 1024 ? SoloBlocks{128, 2} : SoloBlocks{256, 4};
  return {128, !fp8 && hidden > 4096 ? 2 : 4};
}

template <bool TRACE>
auto solo_dispatch_kernel(int threads, bool wide) {
  if (threads == 256) return wide ? k_ep_dispatch_solo<256, 1024, true, TRACE> : k_ep_dispatch_solo<256, 1024, false, TRACE>;
  return wide ? k_ep_dispatch_solo<128, 2048, true, TRACE> : k_ep_dispatch_solo<128, 2048, false, TRACE>;
}

} // namespace

cudaError_t launch_ep_dispatch(const CommDev* comms, const EpDev* eps, int emu_ranks, const void* const* x,
                               const int* const* topk_idx, const float* const* topk_w, int num_tokens,
                               cudaStream_t stream) {
  const EpDev& e0 = eps[0];
  if (e0.hidden % 512 != 0 || e0.topk > 32 || e0.nranks > kMaxRanks || num_tokens > e0.max_tokens ||
      e0.num_experts % e0.nranks != 0) {
    return cudaErrorInvalidValue;
  }
  const int n = emu_ranks > 0 ? emu_ranks : 1;
  std::vector<DispatchArgs> args(n);
  for (int i = 0; i < n; ++i) args[i] = {x[i], topk_idx[i], topk_w[i], num_tokens, 0};
  if (emu_ranks <= 0 && e0.nranks == 1) {
    const SoloBlocks by = solo_blocks(num_tokens, e0.hidden, e0.fp8 != 0);  // at most a token per warp
    args[0].per_block = by.tokens;
    const int blocks = std::max(1, (num_tokens + by.tokens - 1) / by.tokens);
    // 32-byte loads (rows are multiples of 1024 bytes).
    const bool wide = reinterpret_cast<uintptr_t>(x[0]) % 32 == 0;
    const auto kernel = comms[0].trace != nullptr ? solo_dispatch_kernel<true>(by.threads, wide) : solo_dispatch_kernel<false>(by.threads, wide);
    launch_early(kernel, static_cast<unsigned>(blocks), static_cast<unsigned>(by.threads), stream, comms[0], e0, args[0]);
    note_kernel_launch();
    return cudaGetLastError();
  }
  return launch_coop<DispatchArgs>(reinterpret_cast<void*>(&k_ep_dispatch), reinterpret_cast<void*>(&k_ep_dispatch_emu),
                                   comms, eps, emu_ranks, args, stream);
}

cudaError_t launch_ep_combine(const CommDev* comms, const EpDev* eps, int emu_ranks, void* const* out,
                              const float* const* weights, const void* const* bias, int num_tokens,
                              cudaStream_t stream, const int* const* send_slot, float* const* topk_w_out) {
  const EpDev& e0 = eps[0];
  if (e0.hidden % 256 != 0 || num_tokens > e0.max_tokens) return cudaErrorInvalidValue;
  const int n = emu_ranks > 0 ? emu_ranks : 1;
  std::vector<CombineArgs> args(n);
  for (int i = 0; i < n; ++i) {
    args[i] = {out[i], weights ? weights[i] : nullptr, bias ? bias[i] : nullptr, num_tokens,
               send_slot ? send_slot[i] : nullptr, topk_w_out ? topk_w_out[i] : nullptr};
  }
  if (emu_ranks <= 0 && e0.nranks == 1) {
    // Nobody to meet: an ordinary launch with a warp per piece of 1024 columns. Four blocks per SM that stride over
    // the pieces (16.9 us for 4096 x 7168) beat a grid that covers them once (18.3).
    const int64_t items = static_cast<int64_t>(num_tokens) * ((e0.hidden + 1023) / 1024);
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((items + kEpWarps - 1) / kEpWarps, 148 * 4));
    launch_early(comms[0].trace != nullptr ? k_ep_combine_solo<true> : k_ep_combine_solo<false>, static_cast<unsigned>(blocks), kEpThreads,
                 stream, comms[0], e0, args[0]);
    note_kernel_launch();
    return cudaGetLastError();
  }
  return launch_coop<CombineArgs>(reinterpret_cast<void*>(&k_ep_combine), reinterpret_cast<void*>(&k_ep_combine_emu),
                                  comms, eps, emu_ranks, args, stream);
}

cudaError_t launch_ep_pull(const CommDev* comms, const EpDev* eps, int emu_ranks, void* const* out,
                           const int* const* recv_src, const int* const* num_rows, int out_rows, cudaStream_t stream) {
  const EpDev& e0 = eps[0];
  if (e0.hidden % 8 != 0 || out_rows < 0) return cudaErrorInvalidValue;
  const int n = emu_ranks > 0 ? emu_ranks : 1;
  std::vector<PullArgs> args(n);
  for (int i = 0; i < n; ++i) {
    args[i] = {out[i], recv_src ? recv_src[i] : nullptr, num_rows ? num_rows[i] : nullptr, out_rows};
  }
  return launch_coop<PullArgs>(reinterpret_cast<void*>(&k_ep_pull), reinterpret_cast<void*>(&k_ep_pull_emu), comms, eps,
                               emu_ranks, args, stream);
}

cudaError_t launch_ep_layout(const int* topk_idx, int num_tokens, int topk, int num_experts, int nranks,
                             int* tokens_per_rank, int* tokens_per_expert, int* is_token_in_rank, cudaStream_t stream) {
  if (num_experts % nranks != 0) return cudaErrorInvalidValue;
  cudaMemsetAsync(tokens_per_rank, 0, sizeof(int) * nranks, stream);
  cudaMemsetAsync(tokens_per_expert, 0, sizeof(int) * num_experts, stream);
  const int blocks = std::max(1, std::min(296, (num_tokens + 255) / 256));
  k_ep_layout<<<blocks, 256, 0, stream>>>(topk_idx, num_tokens, topk, num_experts, nranks, tokens_per_rank,
                                          tokens_per_expert, is_token_in_rank);
  note_kernel_launch();
  return cudaGetLastError();
}

} // namespace b200c
