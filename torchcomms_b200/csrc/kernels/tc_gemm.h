// tcgen05 / TMEM GEMMs (sm_100a) and their fusion with tensor-parallel
// collectives. Raw-pointer launch interface.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "device_prims.cuh"

namespace b200c {

// C[M, N] (bf16) = A[M, K] (bf16, row-major) x B[N, K]^T (bf16, row-major),
// fp32 accumulation in tensor memory. K % 64 == 0, N % 128 == 0.
// `status` (device or mapped host memory, may be null) receives a non-zero
// word if a bounded wait inside the kernel ran out.
cudaError_t launch_gemm_bf16_nt(const void* a, const void* b, void* c, int m, int n, int k, uint32_t* status,
                                cudaStream_t stream);

// The same with fp8 operands: C[M, N] (bf16) = scale_a[m] * scale_b[n] * (A[M, K] (e4m3) x B[N, K]^T (e4m3)),
// one fp32 scale per row of A (per token) and per row of B (per output channel), applied to the fp32
// accumulator in the epilogue. K % 16 == 0. An e4m3 row has the bytes of a bf16 row of half the length, so
// tiles, tensor maps and pipeline are those of the bf16 kernel; only the tcgen05.mma kind differs.
cudaError_t launch_gemm_e4m3_nt(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                                const float* scale_b, uint32_t* status, cudaStream_t stream);
// For tests of waits that run out: every K step's loads are said to be `missing` bytes more than they are, so that none is
// complete, and each wait of the kernel gives up after `wait_ns`. A product whose waits ran out reports kStatusTimeout and stores NaN
// for what it does not have.
struct GiveUp {
  unsigned long long wait_ns;
  int missing;
};

// Common entry of the two above (k in 16-bit units, scales null = bf16), which picks the kernel. `status`: two words, which
// the kernel clears before it reports into them. `layer`: the communicator of a fused layer on one rank, whose status
// words are not the call's own and keep what they hold, and whose phase trace is stamped (start, loads issued, MMAs
// committed, tiles stored, CTA done). `a_copy`: a second [m, k] buffer (16-byte aligned, not overlapping `a`) that receives a copy of A, or
// `a` itself, where it is there already: the same kernel then, and the same bits.
cudaError_t launch_gemm_nt(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                           const float* scale_b, uint32_t* status, cudaStream_t stream, const CommDev* layer = nullptr,
                           void* a_copy = nullptr, const GiveUp* give_up = nullptr);

// The same product where 128 x 128 tiles are too few to fill the GPU: clusters of CTAs split K and sum in
// distributed shared memory. Sets *done when it launched; otherwise (more than kSplitMaxTiles tiles, or a product that
// another kernel is faster at) nothing happened. Argument rules checked by launch_gemm_nt. `layer`, `a_copy`: as above;
// with a copy to make this kernel is taken wherever it fits, since it passes the copy on by the way: over 480 sizes (128 to
// 4096 rows, 256 to 14336 columns, K of 256 to 8192, weights in L2 and in DRAM) in 0.26 to 0.98 of the time of a copy and the
// best of the others, 768 x 2304 x 256 5.4 us against 7.2, 256 x 7168 x 8192 44.4 against 45.3.
constexpr int kSplitMaxTiles = 148;
cudaError_t launch_gemm_nt_split(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                                 const float* scale_b, uint32_t* status, cudaStream_t stream, bool* done,
                                 const CommDev* layer = nullptr, void* a_copy = nullptr, const GiveUp* give_up = nullptr);

// The same product on CTA pairs (clusters of two CTAs, tcgen05 cta_group::2):
// each pair owns a tile of 256 rows and `columns` (128, 192, 224 or 256; 0: pair_columns()) columns and reads every
// B element once. Any m, n % 8 == 0, k % 8 == 0 (in 16-bit units); scales
// non-null = e4m3 operands. `layer`: as above.
cudaError_t launch_gemm_nt_pair(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                                const float* scale_b, uint32_t* status, cudaStream_t stream, int columns = 0,
                                const CommDev* layer = nullptr, const GiveUp* give_up = nullptr);
// Products whose operands do not lie along K, bf16: c[m, n] = A x b[k, n] with A = a[m, k], or the transpose of a[k, m] where it
// lies `by_columns`.
// `lda`, `ldb`: row strides, multiples of 8. Any m and k, n % 8 == 0; all pointers 16-byte aligned. `status`: as above.
cudaError_t launch_gemm_pair_mn(const void* a, int64_t lda, bool a_by_columns, const void* b, int64_t ldb, void* c, int m, int n, int k,
                                uint32_t* status, cudaStream_t stream);
// dgate_up[m, 2 n], the gradient of gate_up, from d = dy[m, k] x w[k, n], that of silu(gate) * up. n, k % 8 == 0; all pointers
// 16-byte aligned.
cudaError_t launch_gemm_gated_grad(const void* dy, const void* w, const void* gate_up, void* dgate_up, int m, int n, int k, uint32_t* status,
                                   cudaStream_t stream, const GiveUp* give_up = nullptr);
// Pairs that the GPU holds at once (0 after an error), and whether the narrow tiles of an m x n product are at most as many.
int pairs_at_once(bool fp8);
// Waves of tiles, of which `at_once` run at a time, in time: a last, partial wave costs half a wave and half of the share it
// fills, since few tiles have the memory to themselves.
double wave_cost(int64_t tiles, int64_t at_once);
// Columns of a pair's tile for a product, or a gated one of n columns each, and what its waves cost.
int pair_columns(int m, int n, bool gated = false, double* cost = nullptr);
bool pair_tiles_fit(int m, int n, bool fp8);

// The first half of a gated MLP on CTA pairs, bf16: gate_up[m, 2 n] = x[m, k] x w[2 n, k]^T (gate columns first) and, from its
// rounded values, act[m, n] = silu(gate) * up. n and k multiples of 8. `status`: as above.
cudaError_t launch_gemm_gated(const void* x, const void* w, void* gate_up, void* act, int m, int n, int k, uint32_t* status,
                              cudaStream_t stream, int columns = 0, const GiveUp* give_up = nullptr);

// Logits of a head on CTA pairs: logits[m, n] (bf16, row stride `ld`, a multiple of 8) = x[m, k] x w[n, k]^T, any n, k % 8 ==
// 0. Also, of the rounded logits, for each of head_row_shares(m, n) shares of a row the maximum and the sum of
// exp(logit - maximum) (`stats`, [shares, m]), what the sum of the unrounded ones has more (`fine`, the same), and the unrounded
// logit of the row's target (`target_logit`, where targets[row] is in [0, n)). `words`: status as above, then a counter that launch_head_gradient counts rows in; all cleared by the kernel.
int head_row_shares(int m, int n);
cudaError_t launch_head_logits(const void* x, const void* w, void* logits, int64_t ld, const int64_t* targets, int m, int n, int k,
                               float2* stats, float* fine, float* target_logit, uint32_t* words, cudaStream_t stream);

// Column-parallel layer fused with the all-gather of its input.
// x_shards[r] is rank r's [m_local, k] bf16 activation shard in symmetric
// memory (x_shards[rank] local); `x_full` is local scratch [nranks*m_local, k]
// that the kernel's copy warps fill from the peers while the tensor cores
// already work on the rows that have arrived (own rows first, then the
// sources in ring order); w is this rank's [n, k] weight shard;
// y [nranks*m_local, n]. m_local % 128 == 0, n % 256 == 0, k % 64 == 0.
// `ctrl`: local device memory of tp_ctrl_words(nranks*m_local) uint32, zeroed
// once when allocated; the kernel keeps its call epoch and arrival counters
// there, so the same launch may be replayed from a CUDA graph.
// The kernel opens and closes with a cross-rank barrier: a peer's shard is
// complete before it is read, and no rank returns while its shard is in use.
struct AgGemmArgs {
  const void* x_shards[kMaxRanks];
  // Single rank only: the activations where the caller has them, read instead of x_shards[0], which receives a copy.
  const void* x_src;
  void* x_full;
  const void* w;
  void* y;
  int m_local, n, k;
  uint32_t* ctrl;
  // fp8 = 1: x shards and w are e4m3 (k counts e4m3 elements, k % 128 == 0). scale_x_shards[r]: rank r's
  // [m_local] fp32 row scales (symmetric, next to its shard); scale_x_full: local scratch [nranks*m_local]
  // that the copy warps fill with the peers' scales; scale_w: [n] fp32.
  int fp8;
  const float* scale_x_shards[kMaxRanks];
  float* scale_x_full;
  const float* scale_w;
};
cudaError_t launch_allgather_gemm(const CommDev& comm, const AgGemmArgs& args, cudaStream_t stream);

// Row-parallel layer fused with the reduce-scatter of its output.
// h [m, k_local] bf16 local, w [n, k_local] local; every rank computes the
// partial product for all m rows; rows [r*m/nranks, (r+1)*m/nranks) belong to
// rank r. The epilogue TMA-stores each partial tile into local memory: a
// tile of this rank's own rows straight into its `partials` staging, a tile
// of another rank's rows into `send_stage` (local, [m, n] bf16), from where
// four forward warps per CTA push it into the owner's `partials` staging with
// plain 16-byte stores over NVLink (symmetric; partials[r] = owner r's buffer
// of [nranks, m/nranks, n] bf16, slot index = source rank) and raise the
// tile's flag there. The same warps then sum the nranks slots of this rank's
// rows in fp32 into `out` [m/nranks, n] bf16 as the flags arrive, while the
// tensor cores finish the remaining tiles. Tiles for the next rank are
// computed first, the rank's own last. m % (128*nranks) == 0, n % 256 == 0,
// k_local % 64 == 0.
// `arrived` (symmetric, arrived[r] on owner r, zeroed once): one uint32 per
// (tile of the owner's rows, source). `ctrl`: as above (tp_ctrl_words(0)).
struct GemmRsArgs {
  const void* h;
  const void* w;
  void* partials[kMaxRanks];
  void* send_stage;   // local [m, n] bf16 (may be null on a single rank)
  uint32_t* arrived[kMaxRanks];
  void* out;
  int m, n, k_local;
  uint32_t* ctrl;
  // fp8 = 1: h and w are e4m3 (k_local % 128 == 0) with scale_h [m] and scale_w [n]; the partial tiles that
  // travel are bf16 as before (already scaled).
  int fp8;
  const float* scale_h;
  const float* scale_w;
};
cudaError_t launch_gemm_reduce_scatter(const CommDev& comm, const GemmRsArgs& args, cudaStream_t stream);

size_t tp_ctrl_words(int m_total);

// Tests: up to 4 ranks in ONE cooperative launch on the current device, each rank on its share of the SMs, on single
// CTAs or (`pairs`: shards of a multiple of 256 rows) on CTA pairs. comms[r] / args[r] describe rank r; all pointers are device memory of this GPU.
cudaError_t launch_allgather_gemm_emu(const CommDev* comms, const AgGemmArgs* args, int nranks, bool pairs, cudaStream_t stream);
cudaError_t launch_gemm_reduce_scatter_emu(const CommDev* comms, const GemmRsArgs* args, int nranks, bool pairs, cudaStream_t stream);

} // namespace b200c
