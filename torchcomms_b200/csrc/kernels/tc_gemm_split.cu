// Small products on the tensor cores: C = A x B^T with fewer 128 x 128 output
// tiles than the GPU has SMs (a decode batch against one layer's weights). See
// tc_gemm.h.
//
// What bounds them is how fast the weights reach the SMs, and one tile per SM
// would leave most SMs without work. So a cluster of S CTAs takes one tile, each
// CTA a share of K: its TMA -> tcgen05.mma pipeline runs over that share alone,
// the fp32 accumulators meet in distributed shared memory, and every CTA sums,
// scales and stores 1/S of the tile. No workspace, no atomics, a fixed order of
// summation: the same bits at every call. Shares of K make shorter fp32 chains than the persistent kernels', so
// some results round differently and fewer of them away from the exact product's bf16 value (0.07 % of 128 x 3584 x
// 4096, there 0.24 %). m x n x k = 128 x 3584 x 4096 and 128 x 4096 x 1792 in bf16: 31.8 and
// 28.3 us with one 128 x 256 tile on each of 14 and 16 CTAs, 25.1 us for both here
// (28 x 4 and 32 x 4 CTAs); 67 x 6144 x 4096 in e4m3: 15.3 us, now 11.0. Behind another kernel the set-up (barriers,
// tensor memory) overlaps with that one's end: bf16 rows quantised and multiplied, 67 x 6144 x 4096, take 13.8 us a pass,
// 18.4 when every launch and the clearing of the status words waited for the one in front.
//   warp 0, one lane : TMA producer
//   warp 1           : allocates tensor memory; one lane issues tcgen05.mma
//   warps 2..5       : accumulator -> shared memory; then all warps reduce
#include <algorithm>
#include <atomic>

#include "early_launch.cuh"
#include "launch_count.h"
#include "tc_gemm.cuh"
#include "tc_gemm.h"

namespace b200c {

namespace {

using namespace tc;

constexpr int kSplitBN = 128;
constexpr int kSplitStages = 6;
constexpr int kSplitABytes = kBlockM * kBlockK * 2;
constexpr int kSplitBBytes = kSplitBN * kBlockK * 2;
constexpr int kSplitStageBytes = kSplitABytes + kSplitBBytes;
constexpr int kSplitThreads = 192;
constexpr int kSplitPitch = kSplitBN + 4;  // floats per row of the partial tile: 16-byte rows, no bank conflicts
constexpr int kSplitMax = 8;               // portable cluster size
constexpr int kSplitSmemBytes = kSplitStages * kSplitStageBytes + 1024 + 256;
static_assert(kBlockM * kSplitPitch * 4 <= kSplitStages * kSplitStageBytes, "the partial tile reuses the pipeline stages");

struct SplitBarriers {
  uint64_t full[kSplitStages];
  uint64_t empty[kSplitStages];
  uint64_t acc_full;
  uint32_t tmem_base;
  uint32_t failed;
};

struct SplitMaps {
  CUtensorMap a, b;
  CUtensorMap a_copy;  // where the operand A is also wanted (p.copy_a), laid out as A
};

struct SplitParams {
  __nv_bfloat16* c;
  uint32_t* status;
  const float* scale_a;  // e4m3: per row of A, per row of B
  const float* scale_b;
  long long* trace;
  int m, n, k, k_iters, tiles_m;  // k in 16-bit units
  int copy_a;
};

__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <bool FP8, bool TRACE>
__global__ void __launch_bounds__(kSplitThreads, 1) k_gemm_split(const __grid_constant__ SplitMaps maps, SplitParams p) {
  constexpr uint32_t idesc = FP8 ? make_idesc_e4m3(kBlockM, kSplitBN) : make_idesc_bf16(kBlockM, kSplitBN);
  extern __shared__ char smem_raw[];
  char* stages = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  SplitBarriers* bars = reinterpret_cast<SplitBarriers*>(stages + kSplitStages * kSplitStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = static_cast<int>(cluster_nctarank()), part = static_cast<int>(cluster_ctarank());
  const int tile = blockIdx.x / splits;
  const int mi = tile % p.tiles_m, ni = tile / p.tiles_m;
  const int kb0 = static_cast<int>(static_cast<int64_t>(p.k_iters) * part / splits);
  const int kb1 = static_cast<int>(static_cast<int64_t>(p.k_iters) * (part + 1) / splits);

  // The first column of tiles passes its stages of A on (see warp 2 below).
  const bool copies = p.copy_a != 0 && ni == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSplitStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], copies ? 2 : 1);
    }
    mbar_init(&bars->acc_full, 1);
    bars->failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kSplitBN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  grid_release();
  grid_wait();
  if (TRACE && threadIdx.x == 0) trace_stamp_ns(p.trace, 0);

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % kSplitStages;
        const uint32_t ph = (it / kSplitStages) & 1u;
        if (!mbar_wait(&bars->empty[s], ph ^ 1u)) {
          bars->failed = 1;
          break;
        }
        mbar_expect_tx(&bars->full[s], kSplitStageBytes);
        char* sa = stages + s * kSplitStageBytes;
        tma_load_2d(sa, &maps.a, &bars->full[s], kb * kBlockK, mi * kBlockM);
        tma_load_2d(sa + kSplitABytes, &maps.b, &bars->full[s], kb * kBlockK, ni * kSplitBN);
      }
      if (TRACE) trace_stamp_ns(p.trace, 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % kSplitStages;
        const uint32_t ph = (it / kSplitStages) & 1u;
        if (!mbar_wait(&bars->full[s], ph)) {
          bars->failed = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t sa = smem_u32(stages + s * kSplitStageBytes);
        const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + kSplitABytes);
#pragma unroll
        for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) {
          if (FP8) {
            umma_f8(tmem_base, da + static_cast<uint64_t>(kk * 2), db + static_cast<uint64_t>(kk * 2), idesc, (it | kk) != 0);
          } else {
            umma_bf16(tmem_base, da + static_cast<uint64_t>(kk * 2), db + static_cast<uint64_t>(kk * 2), idesc, (it | kk) != 0);
          }
        }
        umma_commit(&bars->empty[s]);
      }
      umma_commit(&bars->acc_full);
      if (TRACE) trace_stamp_ns(p.trace, 2);
    }
  } else {
    // The accumulator is complete, so every stage has been read: the partial tile may overwrite them.
    const int q = warp & 3, row = q * 32 + lane;
    if (copies && warp == 2 && lane == 0) {
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % kSplitStages;
        if (!mbar_wait(&bars->full[s], (it / kSplitStages) & 1u)) {
          bars->failed = 1;
          break;
        }
        tma_store_2d(&maps.a_copy, stages + s * kSplitStageBytes, kb * kBlockK, mi * kBlockM);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&bars->empty[s]);
      }
      tma_store_wait_all<0>();
    }
    __syncwarp();
    float* mine = reinterpret_cast<float*>(stages) + row * kSplitPitch;
    if (mbar_wait(&bars->acc_full, 0)) {
      tc_fence_after_sync();
#pragma unroll
      for (int j = 0; j < kSplitBN / 32; ++j) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(j * 32), r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          *reinterpret_cast<uint4*>(mine + j * 32 + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
        }
      }
    } else {
      bars->failed = 1;
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  cluster_sync_all();  // every CTA's partial tile is in its shared memory
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, kSplitBN);

  // This CTA's share of the tile's 16-byte output vectors: sum over the cluster, scale, round once.
  constexpr int kVecsPerRow = kSplitBN / 8;
  const uint32_t base = smem_u32(stages);
  const int rows_here = min(kBlockM, p.m - mi * kBlockM);
  const int vecs = rows_here * kVecsPerRow;
  for (int v = part * kSplitThreads + static_cast<int>(threadIdx.x); v < vecs; v += splits * kSplitThreads) {
    const int row = v / kVecsPerRow, col = (v % kVecsPerRow) * 8;
    const int gcol = ni * kSplitBN + col;
    if (gcol >= p.n) continue;
    const uint32_t at = base + static_cast<uint32_t>(row * kSplitPitch + col) * 4u;
    float4 lo[kSplitMax], hi[kSplitMax];
#pragma unroll
    for (int s = 0; s < kSplitMax; ++s) {
      if (s < splits) {
        const uint32_t from = map_shared(at, static_cast<uint32_t>(s));
        lo[s] = ld_cluster_f4(from);
        hi[s] = ld_cluster_f4(from + 16u);
      }
    }
    float acc[8] = {lo[0].x, lo[0].y, lo[0].z, lo[0].w, hi[0].x, hi[0].y, hi[0].z, hi[0].w};
#pragma unroll
    for (int s = 1; s < kSplitMax; ++s) {
      if (s < splits) {
        acc[0] += lo[s].x;
        acc[1] += lo[s].y;
        acc[2] += lo[s].z;
        acc[3] += lo[s].w;
        acc[4] += hi[s].x;
        acc[5] += hi[s].y;
        acc[6] += hi[s].z;
        acc[7] += hi[s].w;
      }
    }
    const int grow = mi * kBlockM + row;
    if (FP8) {
      const float ra = p.scale_a[grow];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] *= ra * p.scale_b[gcol + i];
    }
    uint4 o;
    uint32_t* po = &o.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) po[i] = pack_bf16(__float_as_uint(acc[2 * i]), __float_as_uint(acc[2 * i + 1]));
    *reinterpret_cast<uint4*>(p.c + static_cast<size_t>(grow) * p.n + gcol) = o;
  }
  if (TRACE && threadIdx.x == 0) trace_stamp_ns(p.trace, 3);
  if (threadIdx.x == 0 && bars->failed && p.status != nullptr) p.status[0] = p.status[0] | kStatusTimeout;
  __syncwarp();
  cluster_sync_all();  // a peer may still be reading this CTA's partial tile
  if (TRACE && threadIdx.x == 0) trace_stamp_ns(p.trace, 7);
}

__global__ void k_clear_status(uint32_t* status) {
  if (threadIdx.x < 2) status[threadIdx.x] = 0u;
}

cudaLaunchConfig_t split_config(int tiles, int splits, cudaStream_t stream, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * splits));
  cfg.blockDim = dim3(kSplitThreads);
  cfg.dynamicSmemBytes = kSplitSmemBytes;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

constexpr int kDevices = 64;  // whose answers are kept

// Clusters of each size that the current GPU holds at once: they must fit one GPC, so not simply SMs / size, and GPUs
// differ in how their SMs are spread over GPCs. The answer decides the order of summation, so it is kept per device,
// and a query that failed is asked again at the next call.
template <bool FP8>
int resident_clusters(int device, int splits) {
  static std::atomic<int> known[kDevices][kSplitMax + 1];
  std::atomic<int>* kept = device >= 0 && device < kDevices ? &known[device][splits] : nullptr;
  int n = kept != nullptr ? kept->load(std::memory_order_relaxed) : 0;
  if (n == 0) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = split_config(1, splits, nullptr, attr);
    cfg.numAttrs = 1;  // the cluster size
    if (cudaOccupancyMaxActiveClusters(&n, k_gemm_split<FP8, false>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      return 0;
    }
    if (kept != nullptr) kept->store(n, std::memory_order_relaxed);
  }
  return n;
}

// Whether the split kernel beats the others (tc_gemm.cu has their rule); `k` in 16-bit units. Meeting the cluster and
// adding up the shares costs it 2 us more than the direct stores of a full tile, less where the tile has few rows; a K
// step of 64 units is 0.27 us of the others' time and 0.2 us of this one's, over the CTAs that share K.
// Replayed from a graph, best of the others / split in us (bf16 unless e4m3 is said):
//   few rows: 1 x 256 x 256 4.2 / 3.8, 32 x 2560 x 256 4.5 / 4.5, e4m3 1 x 14336 x 256 6.6 / 4.4; up to 64, line at 6
//   steps: 64 x 6144 x 256 5.0 / 5.2, 64 x 2560 x 1024 8.1 / 6.6, e4m3 64 x 2560 x 256 5.0 / 5.4, 64 x 1024 x 1024 6.7 / 5.8
//   K shared, line at 10 steps: e4m3 128 x 4096 x 1024 (8) 6.9 / 7.2, x 2048 (16) 9.3 / 8.5; 384 x 1024 x 1024 (16)
//   8.2 / 8.4, 512 x 1024 x 2048 (32) 12.8 / 10.1; e4m3 1536 x 256 x 8192 (64) 23.0 / 12.0
//   K not shared: half the tile on twice the SMs is worth it only where narrow pair tiles would need a second wave, from
//   20 steps on: e4m3 128 x 14336 x 4096 (32) 19.9 / 18.7; 192 x 8192 x 4096, one wave of pairs, 15.9 / 17.6
bool split_pays(int m, int n, int k_iters, bool fp8, bool shares_k) {
  if (m <= 32) return true;
  if (m <= 64) return k_iters >= 6;
  if (shares_k) return k_iters >= 10;
  return k_iters >= 20 && !pair_tiles_fit(m, n, fp8);
}

template <bool FP8>
cudaError_t launch_split(const SplitMaps& maps, const SplitParams& p, int tiles, cudaStream_t stream, bool* done) {
  // The untraced kernel is the one that resident_clusters asks about: one CTA per SM, as the traced one. Its attribute
  // stays with the device and is set once.
  static std::atomic<bool> ready[kDevices];
  const auto kernel = p.trace != nullptr ? k_gemm_split<FP8, true> : k_gemm_split<FP8, false>;
  int splits = 0, device = 0;
  cudaError_t e = cudaGetDevice(&device);
  const bool kept = device >= 0 && device < kDevices;
  if (e == cudaSuccess && !(kept && ready[device].load(std::memory_order_acquire))) {
    e = cudaFuncSetAttribute(k_gemm_split<FP8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmemBytes);
    if (e == cudaSuccess && kept) ready[device].store(true, std::memory_order_release);
  }
  if (e == cudaSuccess && p.trace != nullptr) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmemBytes);
  }
  if (e != cudaSuccess) return e;
  // As many ways as leave every cluster resident and every CTA at least four K steps (below that the fixed cost of
  // filling the pipeline and meeting the cluster is larger than what another split saves).
  for (int s = 1; s <= kSplitMax; ++s) {
    if (s > 1 && p.k_iters < 4 * s) break;
    if (resident_clusters<FP8>(device, s) >= tiles) splits = s;
  }
  if (splits == 0) return cudaSuccess;  // more tiles than SMs after all: not this kernel's case
  if (p.copy_a == 0 && !split_pays(p.m, p.n, p.k_iters, FP8, splits > 1)) return cudaSuccess;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = split_config(tiles, splits, stream, attr);
  e = cudaLaunchKernelEx(&cfg, kernel, maps, p);
  note_kernel_launch();
  *done = true;
  return e != cudaSuccess ? e : cudaGetLastError();
}

} // namespace

cudaError_t launch_clear_status(uint32_t* status, cudaStream_t stream) {
  k_clear_status<<<1, 32, 0, stream>>>(status);
  note_kernel_launch();
  return cudaGetLastError();
}

cudaError_t launch_gemm_nt_split(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                                 const float* scale_b, uint32_t* status, cudaStream_t stream, bool* done, const CommDev* layer,
                                 void* a_copy) {
  *done = false;
  const int64_t tiles_m = (static_cast<int64_t>(m) + kBlockM - 1) / kBlockM, tiles_n = (static_cast<int64_t>(n) + kSplitBN - 1) / kSplitBN;
  if (tiles_m * tiles_n > kSplitMaxTiles) return cudaSuccess;
  SplitMaps maps;
  if (!make_map(&maps.a, a, m, k, kBlockM) || !make_map(&maps.b, b, n, k, kSplitBN)) return cudaErrorInvalidValue;
  maps.a_copy = maps.a;
  if (a_copy != nullptr && !make_map(&maps.a_copy, a_copy, m, k, kBlockM)) return cudaErrorInvalidValue;
  SplitParams p{};
  p.copy_a = a_copy != nullptr ? 1 : 0;
  p.c = static_cast<__nv_bfloat16*>(c);
  p.status = status;
  p.trace = layer != nullptr ? layer->trace : nullptr;
  p.scale_a = scale_a;
  p.scale_b = scale_b;
  p.m = m;
  p.n = n;
  p.k = k;
  p.k_iters = (k + kBlockK - 1) / kBlockK;
  p.tiles_m = static_cast<int>(tiles_m);
  const int tiles = static_cast<int>(tiles_m * tiles_n);
  return scale_a != nullptr ? launch_split<true>(maps, p, tiles, stream, done) : launch_split<false>(maps, p, tiles, stream, done);
}

} // namespace b200c
