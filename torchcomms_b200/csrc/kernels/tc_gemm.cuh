// Blackwell (sm_100a) tensor-core building blocks written as inline PTX:
// mbarriers, TMA tile loads (never with cluster multicast), TMEM allocation,
// tcgen05.mma issue / commit and tcgen05.ld, plus the shared-memory and
// instruction descriptors for bf16 x bf16 -> fp32 and e4m3 x e4m3 -> fp32 with
// K-major operands under the 128-byte swizzle. An e4m3 matrix [rows, K] has the
// bytes of a bf16 matrix [rows, K/2]: the tensor maps, the shared-memory tiles
// and the 32-byte K step are the same for both, only the instruction differs.
//
// Every wait is bounded: when its spin budget runs out it returns false, the
// caller records an error word, skips the remaining work and still releases
// its tensor memory.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200c {
namespace tc {

constexpr int kBlockM = 128;
constexpr int kBlockK = 64;                 // 64 bf16 = 128 bytes = one swizzle row
constexpr int kUmmaK = 16;                  // K of one tcgen05.mma for 16-bit inputs
constexpr unsigned long long kLocalWaitNs = 60ull * 1000 * 1000 * 1000;   // wall-time bound of a CTA-local pipeline wait


// ------------------------------------------------------- tensor maps ------
// Host side: row-major bf16 matrix [rows, cols] as a 2-D tiled tensor map
// with a box of [box_rows, 64 columns] and the 128-byte swizzle (the layout
// the shared-memory descriptors above expect). The driver entry point is
// looked up at run time; the extension does not link against libcuda.

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      return reinterpret_cast<EncodeTiledFn>(sym);
    }
    return nullptr;
  }();
  return fn;
}

// The driver encodes maps under the calling thread's context, and refuses where there is none yet: in a thread that has made no call
// of the runtime that binds one. Buffers from PyTorch's cache and what is kept per device need none, so a product in a new
// thread can come here first.
inline void bind_thread() {
  thread_local bool bound = false;
  int device = 0;
  if (!bound) bound = cudaGetDevice(&device) == cudaSuccess && cudaSetDevice(device) == cudaSuccess;
}

// `ld`: elements from row to row, a multiple of 8 (0: rows follow one another).
// `box_cols`: other boxes than of 64 columns are not swizzled.
inline bool make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint64_t ld = 0,
                     uint32_t box_cols = kBlockK) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return false;
  bind_thread();
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {(ld != 0 ? ld : cols) * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == kBlockK ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Rows of the boxes that bring A where it has `m` rows: those of its only tile, in groups of eight (the period of the
// swizzle). A box row past the matrix takes as long as one in it, and longer where few rows are left; what a stage holds
// below the box gives rows of the accumulator that nobody reads. In us with boxes of 128 rows and so: 1 x 6144 x 8192 in e4m3
// 17.7 and 14.2; in bf16 8 x 6144 x 4096 17.2 and 14.0, 1 x 14336 x 4096 39.5 and 26.0, 32 x 6144 x 8192 25.0 and 24.9.
constexpr int a_box_rows(int m) { return m >= kBlockM ? kBlockM : (m + 7) / 8 * 8; }

#ifdef __CUDACC__

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One thread of a converged warp, which the compiler knows to be one. TMA and tcgen05 instructions take their operands from
// uniform registers; under `lane == 0` each of them is wrapped in a loop over the threads that might be there, and a K step of
// four MMAs took 290 ns whatever the tile's width: in a pair kernel of one tile of 128 columns 290 ns and now 144, of 192 290 and
// 214, of 256, which the tensor pipe bounds, 291 and 284.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}

// ---------------------------------------------------------------- mbarrier --

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait; false = gave up. The bound is wall time, not a number of
// polls: how long a poll takes depends on what else the SM is doing, and a
// pipeline stage may legitimately wait while copy warps sit in their own
// (time-bounded) wait for a slow peer. kLocalWaitNs is far above any peer-wait
// budget, so a local wait only runs out when the pipeline is truly stuck.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned long long limit_ns = 0) {
  unsigned long long start = 0;
  for (uint32_t i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (start == 0) {
        start = now;
      } else if (now - start > (limit_ns != 0 ? limit_ns : kLocalWaitNs)) {
        return false;
      }
    }
  }
}
// The same for a converged warp, whose lanes all get the one answer: each leaves the wait by itself, and one might give up where
// the next one still sees the barrier complete.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, unsigned long long limit_ns) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit_ns)) != 0;
}
// Accumulators that will never be there. A plain product whose wait ran out stores NaN wherever it has nothing else: not every
// caller reads the status words (a decoder block has no time to), and what was in the output's memory before passes for numbers.
template <int N>
__device__ __forceinline__ void no_acc(uint32_t (&r)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = 0x7fc00000u;
}
// The two status words of a plain product, cleared by its first block (after grid_wait()) and not by a launch of their own
// in front of it: a kernel node for that costs a captured product 2.5 us (128 x 1024 x 256 in bf16: 7.1 us a replay, with the
// words cleared here 4.5), and nothing starts early behind it. No other block can be ahead of this one: what they report
// is a wait of kLocalWaitNs that ran out.
__device__ __forceinline__ void clear_status(uint32_t* status) {
  if (blockIdx.x == 0 && threadIdx.x < 2) status[threadIdx.x] = 0u;
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// --------------------------------------------------------------------- TMA --

// 2-D tile load, global -> shared, completion counted in bytes on `bar`.
// x is the innermost (contiguous) coordinate in elements; x * elem_size must
// be a multiple of 16 bytes. No multicast.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// 2-D tile store, shared -> global (local or a peer's memory), tracked by the
// issuing thread's bulk async-group. Same alignment rule for x.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// At most N committed groups may still be READING their shared-memory source.
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
// At most N committed groups may still be incomplete (writes not yet done).
template <int N>
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
// Orders this thread's shared-memory writes before later async-proxy reads of them.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// -------------------------------------------------------------------- TMEM --

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by ONE thread.
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
      : "memory");
}
// The same for 8-bit floating-point operands (formats named by the instruction descriptor); K of one
// instruction is 32 elements, which is again 32 bytes of the swizzled row.
__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
      : "memory");
}
// Arrives on `bar` once every tcgen05.mma issued so far by this thread is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 32 lanes x 32 columns of fp32: thread i of the warp gets row i, 32 columns.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ------------------------------------------------ CTA pairs (cta_group::2) --
//
// Two CTAs of a cluster (ranks 0 and 1, rank 0 leads) work on one 256-row
// tile: each holds its own 128 rows of A and half of the B tile in shared
// memory and its own 128 rows of the accumulator in tensor memory; the leader
// issues one tcgen05.mma for both. Shared-memory addresses of the two CTAs
// differ only in bit 24 of the 32-bit shared::cluster address, so clearing
// that bit names the leader's copy of a barrier from either CTA.

constexpr uint32_t kPeerBitMask = 0xFEFFFFFFu;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on the LEADER's copy of `bar` (callable from both CTAs of the pair).
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & kPeerBitMask) : "memory");
}
// Tile load whose completion bytes are counted on the LEADER's barrier. No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar) & kPeerBitMask), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A * B^T over the pair, issued by ONE thread of the leader.
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_f8_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)), "r"(0u)
      : "memory");
}
// Arrives on `bar` in every CTA of `cta_mask` once the leader's MMAs so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t cta_mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(cta_mask)
               : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(uint32_t a, uint32_t b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
  return *reinterpret_cast<uint32_t*>(&h);
}

// ------------------------------------------------------------- descriptors --

// Shared-memory matrix descriptor: K-major tile whose rows are 128 bytes
// (64 bf16), 128-byte swizzle, 8-row groups 1024 bytes apart. The tile base
// must be 1024-byte aligned; stepping along K inside the swizzle row is done
// by adding the byte offset (>> 4) to the low word.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);   // start address
  d |= static_cast<uint64_t>(1) << 16;                        // leading byte offset (unused for swizzled K-major)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                // stride byte offset: 8 rows x 128 B
  d |= static_cast<uint64_t>(1) << 46;                        // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                        // layout: 128-byte swizzle
  return d;
}

// The same for an MN-major tile: 64 rows of K of 64 bf16 each (128 bytes, swizzled), one such block of 8 KB after the other along
// M or N. Eight rows of K are 1024 bytes; stepping along K adds 128 bytes a row.
constexpr int kMnBlock = 64;
constexpr int kMnBlockBytes = kBlockK * kMnBlock * 2;
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(kMnBlockBytes >> 4) << 16;       // leading byte offset: from block to block
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                // stride byte offset: 8 rows of K
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// Instruction descriptor: bf16 x bf16 -> fp32, operands K-major or MN-major.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int m, int n, bool a_mn = false, bool b_mn = false) {
  return (1u << 4)                              // D format: fp32
      | (1u << 7)                               // A format: bf16
      | (1u << 10)                              // B format: bf16
      | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u)
      | (static_cast<uint32_t>(n >> 3) << 17)   // N / 8
      | (static_cast<uint32_t>(m >> 4) << 24);  // M / 16
}

// Instruction descriptor: e4m3 x e4m3 -> fp32 (kind::f8f6f4; operand format 0 = e4m3), both operands K-major.
__host__ __device__ constexpr uint32_t make_idesc_e4m3(int m, int n) {
  return (1u << 4)                              // D format: fp32
      | (static_cast<uint32_t>(n >> 3) << 17)   // N / 8
      | (static_cast<uint32_t>(m >> 4) << 24);  // M / 16
}

// Epilogue of the fp8 products: acc[i] *= row_scale * col_scale[i]; `col_scale`: 16-byte aligned, in shared memory.
__device__ __forceinline__ void scale_acc32(uint32_t (&r)[32], float row_scale, const float* col_scale) {
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const float4 b = reinterpret_cast<const float4*>(col_scale)[v];
    r[4 * v] = __float_as_uint(__uint_as_float(r[4 * v]) * (row_scale * b.x));
    r[4 * v + 1] = __float_as_uint(__uint_as_float(r[4 * v + 1]) * (row_scale * b.y));
    r[4 * v + 2] = __float_as_uint(__uint_as_float(r[4 * v + 2]) * (row_scale * b.z));
    r[4 * v + 3] = __float_as_uint(__uint_as_float(r[4 * v + 3]) * (row_scale * b.w));
  }
}

// The column scales of a tile of BN columns on their way to shared memory: each of the 128 epilogue threads fetches BN / 128
// of them (rounded up) a tile ahead, so that the epilogue does not wait for global memory (zero past column `n`). In e4m3, pairs, in us with every thread
// reading each scale from global memory, and so: 300 x 28672 x 2048 31.1 and 27.1, 384 x 28672 x 512 20.4 and 15.8, 1000 x
// 14336 x 512 19.8 and 15.8.
template <int BN>
struct ColScales {
  static constexpr int kEach = (BN + 127) / 128;
  float v[kEach];
  __device__ __forceinline__ void fetch(const float* col_scale, int col0, int n, int thread) {
#pragma unroll
    for (int i = 0; i < kEach; ++i) {
      const int col = col0 + thread * kEach + i;
      v[i] = col < n ? col_scale[col] : 0.0f;
    }
  }
  // To `to` (kEach * 128 floats), which nobody reads any more; it may be read after the epilogue's next barrier.
  __device__ __forceinline__ void put(float* to, int thread) const {
#pragma unroll
    for (int i = 0; i < kEach; ++i) to[thread * kEach + i] = v[i];
  }
};

#endif // __CUDACC__

} // namespace tc
} // namespace b200c
