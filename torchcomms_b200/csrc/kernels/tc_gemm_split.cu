// Small products on the tensor cores: C = A x B^T with fewer 128 x 128 output
// tiles than the GPU has SMs (a decode batch against one layer's weights). See
// tc_gemm.h.
//
// What bounds them is how fast the weights reach the SMs, and one tile per SM
// would leave most SMs without work. So a cluster of S CTAs takes one tile, each
// CTA a share of K: its TMA -> tcgen05.mma pipeline runs over that share alone.
// Every CTA then owns 1/S of the tile's columns, sums, scales and stores them: the
// others send their fp32 accumulators of these columns from registers into its
// shared memory (st.async), where one barrier counts the bytes, so nobody meets
// the whole cluster and the sums start as the last share arrives. No workspace, no
// atomics, a fixed order of summation: the same bits at every call. Shares of K
// make shorter fp32 chains than the other kernels', so some results round
// differently and fewer of them away from the exact product's bf16 value (0.07 % of
// 128 x 3584 x 4096, there 0.24 %). 128 x 3584 x 4096 in bf16, operands in L2, in us from the start: loads issued 4.3,
// accumulators complete 5.7, shares sent 7.1 and received 8.1, done 9.1; when the cluster met, read one another's
// accumulators and met again, 11.4. Replayed from a graph, then and now: this 13.4 and 11.2, in e4m3 128 x 6144 x 4096 12.8
// and 10.4. Behind another kernel the set-up (barriers, tensor memory) overlaps with that one's end.
//   warp 0, one lane : TMA producer
//   warp 1           : allocates tensor memory; one lane issues tcgen05.mma
//   warps 2..5       : accumulators -> their owners, then the own columns
// The phase trace has, besides the marks of the other kernels, 4: accumulators complete, 5: shares sent, 6: received.
#include <algorithm>
#include <atomic>

#include "early_launch.cuh"
#include "launch_count.h"
#include "tc_gemm.cuh"
#include "tc_gemm.h"
#include "wide_access.cuh"

namespace b200c {

namespace {

using namespace tc;

constexpr int kSplitBN = 128;
constexpr int kSplitStages = 5;
constexpr int kSplitABytes = kBlockM * kBlockK * 2;
constexpr int kSplitBBytes = kSplitBN * kBlockK * 2;
constexpr int kSplitStageBytes = kSplitABytes + kSplitBBytes;
constexpr int kSplitThreads = 192;
constexpr int kSplitMax = 8;                // portable cluster size
constexpr int kSplitGroups = kSplitBN / 8;  // a tile's columns are shared out among the cluster in groups of eight
// The first group of CTA `o`; `per_split` = groups per CTA, rounded up to 1/65536. The last CTA may own fewer.
__host__ __device__ constexpr int first_group(int o, int per_split) {
  const int g = (o * per_split + 65535) >> 16;
  return g < kSplitGroups ? g : kSplitGroups;
}
constexpr int groups_per_split(int splits) { return (kSplitGroups * 65536 + splits - 1) / splits; }
// Clusters of six and seven would need more room than the others for what a CTA receives.
constexpr bool split_allowed(int splits) { return splits != 6 && splits != 7; }
// What a CTA receives: for its groups, 128 rows of eight fp32 from every other CTA.
constexpr int most_share_bytes() {
  int most = 0;
  for (int s = 1; s <= kSplitMax; ++s) {
    for (int o = 0; o < s && split_allowed(s); ++o) {
      const int own = first_group(o + 1, groups_per_split(s)) - first_group(o, groups_per_split(s));
      const int bytes = (s - 1) * own * kBlockM * 32;
      most = bytes > most ? bytes : most;
    }
  }
  return most;
}
constexpr int kSplitSmemBytes = kSplitStages * kSplitStageBytes + most_share_bytes() + 1024 + 768;
static_assert(kSplitSmemBytes <= 227 * 1024, "shared memory of one CTA");

struct SplitBarriers {
  alignas(16) float scale_b[kSplitBN];  // e4m3: of the tile's columns
  uint64_t full[kSplitStages];
  uint64_t empty[kSplitStages];
  uint64_t acc_full;
  uint64_t shares;  // the other CTAs' shares have arrived
  uint32_t tmem_base;
  uint32_t failed;
};
static_assert(sizeof(SplitBarriers) <= 768, "kSplitSmemBytes");

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
  unsigned long long wait_ns;  // limit of a wait (0: kLocalWaitNs)
  int m, n, k, k_iters, tiles_m;  // k in 16-bit units
  int copy_a, per_split;
  int always;  // (host) this kernel whether it pays or not
  int clear;        // the status words are this call's own
  int stage_bytes;  // of one K step's loads
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
// Four values into another CTA's shared memory; their 16 bytes count on that CTA's barrier.
__device__ __forceinline__ void st_async_f4(uint32_t addr, const uint32_t* r, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// 32 lanes x 16 columns of fp32.
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

template <bool FP8, bool TRACE>
__global__ void __launch_bounds__(kSplitThreads, 1) k_gemm_split(const __grid_constant__ SplitMaps maps, SplitParams p) {
  constexpr uint32_t idesc = FP8 ? make_idesc_e4m3(kBlockM, kSplitBN) : make_idesc_bf16(kBlockM, kSplitBN);
  extern __shared__ char smem_raw[];
  // The same place in every CTA of the cluster: shares are written across.
  char* stages = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  char* received = stages + kSplitStages * kSplitStageBytes;
  SplitBarriers* bars = reinterpret_cast<SplitBarriers*>(received + most_share_bytes());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = static_cast<int>(cluster_nctarank()), part = static_cast<int>(cluster_ctarank());
  const int tile = blockIdx.x / splits;
  const int mi = tile % p.tiles_m, ni = tile / p.tiles_m;
  const int kb0 = static_cast<int>(static_cast<int64_t>(p.k_iters) * part / splits);
  const int kb1 = static_cast<int>(static_cast<int64_t>(p.k_iters) * (part + 1) / splits);
  const int rows = min(kBlockM, p.m - mi * kBlockM);
  const int groups = min(kSplitGroups, (p.n - ni * kSplitBN) / 8);  // n is a multiple of 8
  const int own_lo = first_group(part, p.per_split), own_hi = min(first_group(part + 1, p.per_split), groups);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSplitStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], p.copy_a != 0 ? 2 : 1);  // see warp 2
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->shares, 1);
    bars->failed = 0;
    fence_barrier_init();
    mbar_expect_tx(&bars->shares, static_cast<uint32_t>((splits - 1) * max(own_hi - own_lo, 0) * rows * 32));
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kSplitBN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  cluster_arrive();  // this CTA's barriers exist
  const uint32_t tmem_base = bars->tmem_base;
  grid_release();
  grid_wait();
  if (p.clear != 0) clear_status(p.status);
  if (TRACE && threadIdx.x == 0) trace_stamp_ns(p.trace, 0);

  if (warp == 0) {
    if (elect_one()) {
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % kSplitStages;
        const uint32_t ph = (it / kSplitStages) & 1u;
        if (!mbar_wait(&bars->empty[s], ph ^ 1u, p.wait_ns)) {
          bars->failed = 1;
          break;
        }
        mbar_expect_tx(&bars->full[s], static_cast<uint32_t>(p.stage_bytes));
        char* sa = stages + s * kSplitStageBytes;
        tma_load_2d(sa, &maps.a, &bars->full[s], kb * kBlockK, mi * kBlockM);
        tma_load_2d(sa + kSplitABytes, &maps.b, &bars->full[s], kb * kBlockK, ni * kSplitBN);
      }
      if (TRACE) trace_stamp_ns(p.trace, 1);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      bool cut_short = false;
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % kSplitStages;
        const uint32_t ph = (it / kSplitStages) & 1u;
        if (!mbar_wait(&bars->full[s], ph, p.wait_ns)) {
          bars->failed = 1;
          cut_short = true;
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
      if (!cut_short) umma_commit(&bars->acc_full);  // or not all of K is there: the epilogue waits in vain
      if (TRACE) trace_stamp_ns(p.trace, 2);
    }
  } else {
    if (p.copy_a != 0 && warp == 2 && elect_one()) {
      // Every column of tiles has all of A pass by; each passes the steps on whose turn it is.
      const int tiles_n = static_cast<int>(gridDim.x) / splits / p.tiles_m;
      for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int s = it % kSplitStages;
        if (!mbar_wait(&bars->full[s], (it / kSplitStages) & 1u, p.wait_ns)) {
          bars->failed = 1;
          break;
        }
        if (kb % tiles_n == ni) {
          tma_store_2d(&maps.a_copy, stages + s * kSplitStageBytes, kb * kBlockK, mi * kBlockM);
          tma_store_commit();
          tma_store_wait_read<0>();
        }
        mbar_arrive(&bars->empty[s]);
      }
      tma_store_wait_all<0>();
    }
    __syncwarp();
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t acc = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    float ra = 0.0f;
    if (FP8) {  // the scales come in while the product runs
      if (row < rows) ra = p.scale_a[mi * kBlockM + row];
      bars->scale_b[row] = ni * kSplitBN + row < p.n ? p.scale_b[ni * kSplitBN + row] : 0.0f;
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    // After a failed wait the shares still go out and come in, as NaN, so that no CTA leaves while another one writes to it and no
    // tile passes for complete.
    bool lost = !mbar_wait_warp(&bars->acc_full, 0, p.wait_ns);
    if (lost) bars->failed = 1;
    __syncwarp();  // the cluster barrier and the loads below want the lanes together
    tc_fence_after_sync();
    cluster_wait();  // the peers' barriers exist
    if (TRACE && threadIdx.x == 64) trace_stamp_ns(p.trace, 4);
    // Every CTA runs this part once: a chain of latencies, and some 35 bytes per ns between the CTAs' shared memories. (From
    // there to there by bulk copies: 2.4 us for what takes 1.6 straight from the registers.) Two groups of columns at a
    // time, from `at` on; the last two where one remains. Warps without rows have nothing to do.
    const bool live = q * 32 < rows;
    uint32_t r[16];
#pragma unroll 1
    for (int o = 0; o < splits && live; ++o) {
      if (o == part) continue;
      const int lo = first_group(o, p.per_split), next = first_group(o + 1, p.per_split), hi = min(next, groups);
      const int slot = part < o ? part : part - 1;
      const uint32_t to = map_shared(smem_u32(received) + static_cast<uint32_t>((slot * (next - lo) * 2 * kBlockM + row) * 16), static_cast<uint32_t>(o));
      const uint32_t bar = map_shared(smem_u32(&bars->shares), static_cast<uint32_t>(o));
#pragma unroll 1
      for (int g = lo; g < hi; g += 2) {
        const int at = min(g, kSplitGroups - 2);
        tmem_ld_32x16(acc + static_cast<uint32_t>(at * 8), r);
        tmem_ld_wait();
        if (lost) no_acc(r);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int here = at + v / 2;
          if (row < rows && here >= g && here < hi) st_async_f4(to + static_cast<uint32_t>(((here - lo) * 2 + v % 2) * kBlockM * 16), r + 4 * v, bar);
        }
        __syncwarp();
      }
    }
    if (TRACE && threadIdx.x == 64) trace_stamp_ns(p.trace, 5);
    if (splits > 1) {
      if (!mbar_wait_warp(&bars->shares, 0, p.wait_ns) && !mbar_wait_warp(&bars->shares, 0, p.wait_ns)) {  // longer than a peer's own waits
        bars->failed = 1;
        lost = true;
      }
      asm volatile("fence.acq_rel.cluster;" ::: "memory");
    }
    __syncwarp();
    if (TRACE && threadIdx.x == 64) trace_stamp_ns(p.trace, 6);
    // This CTA's columns: the sum over the cluster in its order, scaled, rounded once.
    const int step = (first_group(part + 1, p.per_split) - own_lo) * 2 * kBlockM;  // from one CTA's share to the next
    const float4* in = reinterpret_cast<const float4*>(received) + row;
    __nv_bfloat16* out = p.c + static_cast<size_t>(mi * kBlockM + row) * p.n + ni * kSplitBN;
    const bool wide = p.n % 16 == 0 && (reinterpret_cast<uintptr_t>(p.c) & 31u) == 0;
#pragma unroll 1
    for (int g = own_lo; g < own_hi && live; g += 2) {
      const int at = min(g, kSplitGroups - 2);
      tmem_ld_32x16(acc + static_cast<uint32_t>(at * 8), r);
      tmem_ld_wait();
      if (lost) no_acc(r);
      const float4* from = in + (at - own_lo) * 2 * kBlockM;
      const bool first = at >= g, second = at + 1 < own_hi;  // which of the two are wanted
      float sum[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
#pragma unroll 1
      for (int s = 0; s < splits; ++s) {
        if (s == part) {
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[i] += __uint_as_float(r[i]);
          continue;
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const float4 f = (v < 2 ? first : second) ? from[v * kBlockM] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          sum[4 * v] += f.x;
          sum[4 * v + 1] += f.y;
          sum[4 * v + 2] += f.z;
          sum[4 * v + 3] += f.w;
        }
        from += step;
      }
      if (FP8) {
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] *= ra * bars->scale_b[at * 8 + i];
      }
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = pack_bf16(__float_as_uint(sum[2 * i]), __float_as_uint(sum[2 * i + 1]));
      if (row < rows) {
        const uint4 lo = make_uint4(o[0], o[1], o[2], o[3]), hi = make_uint4(o[4], o[5], o[6], o[7]);
        if (first && second && wide && at % 2 == 0) {
          st32(out + at * 8, lo, hi);
        } else {
          if (first) *reinterpret_cast<uint4*>(out + at * 8) = lo;
          if (second) *reinterpret_cast<uint4*>(out + at * 8 + 8) = hi;
        }
      }
      __syncwarp();
    }
    if (TRACE && threadIdx.x == 64) trace_stamp_ns(p.trace, 3);
  }

  __syncwarp();
  if (warp < 2) cluster_wait();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, kSplitBN);
  if (threadIdx.x == 0 && bars->failed && p.status != nullptr) p.status[0] = p.status[0] | kStatusTimeout;
  if (TRACE && threadIdx.x == 0) trace_stamp_ns(p.trace, 7);
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

// Whether the split kernel beats the others (tc_gemm.cu has their rule), K being shared by `splits` CTAs. Sending shares to
// their owners costs it 2 us more than a kernel that has its tile to itself, as long as 11 K steps take a pair, or 7 with up to
// 64 rows, which send less; weights from DRAM, as here, favour the kernel with more CTAs to fetch them. Without shares it is ahead
// where pairs are mostly start and end, or leave their second half of rows empty in more tiles than a quarter of the SMs.
// Replayed from a graph over 320 MB of weights, narrow pairs / split in us:
//   K shared, by the steps that a CTA is spared: bf16 256 x 2816 x 1280 (10) 7.7 / 9.0, 384 x 768 x 1024 (12) 6.5 / 7.0, 128 x 4096 x
//   1792 (21) 9.7 / 9.1, 128 x 3584 x 4096 (48) 17.9 / 12.0; e4m3 128 x 4096 x 1408 (6) 6.3 / 6.7, 1152 x 768 x 2304 (9) 7.3 / 7.3, 640 x
//   1792 x 3072 (12) 9.0 / 8.5, 256 x 4608 x 3712 (15) 10.5 / 10.0, 67 x 6144 x 4096 (16) 11.4 / 10.2; few rows: bf16 55 x 4848 x 768
//   (6) 6.0 / 6.1, e4m3 28 x 6440 x 1808 (8) 7.6 / 7.3, 4 x 272 x 1600 (9) 5.7 / 4.9, 1 x 1712 x 3040 (20) 8.2 / 6.0
//   not shared, at most as many tiles as pairs: e4m3 256 x 4352 x 512 (4) 4.8 / 4.6, 640 x 3072 x 896 (7) 6.0 / 5.8, 768 x 2048 x 1152
//   (9) 6.0 / 6.1, 119 x 8376 x 480 (off the lines) 5.8 / 5.0; bf16 1280 x 1536 x 1792 (28) 9.4 / 9.9, 1280 x 1792 x 5120 (80) 21.3 /
//   22.8; off the lines 1014 x 1400 x 3952 (31) 13.3 / 15.9
//   not shared, more tiles than pairs, best of the others / split, weights in L2: bf16 384 x 5376 x 1536 10.5 / 9.5, 128 x 12032 x
//   2304 16.2 / 15.4; e4m3 300 x 6144 x 4096 13.8 / 13.1; off the lines 259 x 5560 x 1872 (15) 10.7 / 10.5, x 2056 in bf16 (33) 18.2 /
//   19.5
bool split_pays(int m, int n, int k, int k_iters, bool fp8, int splits) {
  const bool on_lines = k % kBlockK == 0;
  if (pair_tiles_fit(m, n, fp8)) {
    if (splits == 1) return (on_lines && k_iters <= 7) || (m <= kBlockM && n > 40 * kSplitBN);
    return k_iters - k_iters / splits >= (m > 64 ? 11 : 7);
  }
  if (splits > 1) return fp8 || m <= 64 || k_iters >= 10;
  return on_lines || k_iters <= 17;
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
  // filling the pipeline and exchanging the shares is larger than what another split saves).
  for (int s = 1; s <= kSplitMax; ++s) {
    if (s > 1 && p.k_iters < 4 * s) break;
    if (!split_allowed(s)) continue;
    if (resident_clusters<FP8>(device, s) >= tiles) splits = s;
  }
  if (splits == 0) return cudaSuccess;  // more tiles than SMs after all: not this kernel's case
  if (!p.always && !split_pays(p.m, p.n, p.k, p.k_iters, FP8, splits)) return cudaSuccess;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = split_config(tiles, splits, stream, attr);
  // Clusters of three and five do not pack into the SMs as the kernel in front leaves them, so that fewer are resident than
  // on an empty GPU, and a second wave follows. Where room for less than ten more CTAs is left, they start late instead. In
  // us, early / late, 128 rows x 4096, tiles of 45 in clusters of three: 40 12.9 / 13.9, 42 15.6 / 14.2, 45 18.9 / 14.1; of
  // 26 in clusters of five: 25 11.8 / 12.1, 26 13.4 / 11.8. Even sizes pack: 33 in clusters of four 11.8 / 12.8, 74 in two 15.9 / 17.2.
  if (splits % 2 == 1 && splits > 1 && (resident_clusters<FP8>(device, splits) - tiles) * splits < 10) cfg.numAttrs = 1;
  SplitParams q = p;
  q.per_split = groups_per_split(splits);
  e = cudaLaunchKernelEx(&cfg, kernel, maps, q);
  note_kernel_launch();
  *done = true;
  return e != cudaSuccess ? e : cudaGetLastError();
}

} // namespace

cudaError_t launch_gemm_nt_split(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                                 const float* scale_b, uint32_t* status, cudaStream_t stream, bool* done, const CommDev* layer,
                                 void* a_copy, const GiveUp* give_up) {
  *done = false;
  const int64_t tiles_m = (static_cast<int64_t>(m) + kBlockM - 1) / kBlockM, tiles_n = (static_cast<int64_t>(n) + kSplitBN - 1) / kSplitBN;
  if (tiles_m * tiles_n > kSplitMaxTiles) return cudaSuccess;
  SplitMaps maps;
  if (!make_map(&maps.a, a, m, k, a_box_rows(m)) || !make_map(&maps.b, b, n, k, kSplitBN)) return cudaErrorInvalidValue;
  maps.a_copy = maps.a;
  if (a_copy != nullptr && a_copy != a && !make_map(&maps.a_copy, a_copy, m, k, a_box_rows(m))) return cudaErrorInvalidValue;
  SplitParams p{};
  p.copy_a = a_copy != nullptr && a_copy != a ? 1 : 0;
  p.always = a_copy != nullptr ? 1 : 0;
  p.c = static_cast<__nv_bfloat16*>(c);
  p.status = status;
  p.clear = layer == nullptr && status != nullptr ? 1 : 0;
  p.trace = layer != nullptr ? layer->trace : nullptr;
  p.scale_a = scale_a;
  p.scale_b = scale_b;
  p.m = m;
  p.n = n;
  p.k = k;
  p.stage_bytes = a_box_rows(m) * kBlockK * 2 + kSplitBBytes + (give_up != nullptr ? give_up->missing : 0);
  p.wait_ns = give_up != nullptr ? give_up->wait_ns : 0;
  p.k_iters = (k + kBlockK - 1) / kBlockK;
  p.tiles_m = static_cast<int>(tiles_m);
  const int tiles = static_cast<int>(tiles_m * tiles_n);
  return scale_a != nullptr ? launch_split<true>(maps, p, tiles, stream, done) : launch_split<false>(maps, p, tiles, stream, done);
}

} // namespace b200c
