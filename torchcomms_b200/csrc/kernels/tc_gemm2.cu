// GEMM on CTA pairs (tcgen05 cta_group::2), bf16 or e4m3. See tc_gemm.h.
//
// A cluster of two CTAs owns a 256 x 256 output tile. Each CTA loads its own
// 128 rows of A and HALF of the B tile (128 of the 256 rows of B) per k-step,
// so the pair reads every B element once instead of twice; the leader CTA
// issues one 256 x 256 x 16 MMA for both, accumulating into the tensor memory
// of both. The smaller per-CTA stage (32 KB) also buys a 6-deep TMA ring.
// The tensor pipe bounds a pair with the memory to itself (a K step of 64 units
// in 284 ns), operand traffic from L2 to the SMs all of them together: 4096 x
// 28672 x 4096 in e4m3 318 us in a burst and 369 under the power cap, in bf16
// 577 and 680. Tiles are 256, 224, 192 or 128 columns wide, whichever leaves the
// last wave of pairs fuller (pair_columns), and a wave that stays mostly empty
// all the same is worked on in halves of tiles.
//
// Roles per CTA (192 threads): warp 0 (one thread) TMA producer (both CTAs), warp 1
// tensor-memory allocation (both CTAs) and MMA issue (leader only), warps 2-5
// epilogue (both CTAs: tcgen05.ld -> bf16 -> swizzled staging -> TMA store).
// Barriers: `full` lives in the leader and counts the bytes of all four loads
// of a stage; `empty` and `acc_full` exist in both CTAs and are released by
// the leader's commits (arrival delivered to both CTAs); `acc_empty` lives in
// the leader and collects the eight epilogue warps of the pair.
// No load uses cluster multicast.
//
// With kStats the product is a head's logits, and the epilogue, which holds a row of the tile in every thread, also leaves
// each row's maximum and sum of exponentials over the tile and the logit of its target: the loss then needs one look
// at the logits instead of two. One set of epilogue warps takes 405 us for 4096 x 128256 x 256 with one barrier more a chunk,
// two sets that share a tile's columns 348, two that take the tiles in turn 315 (the plain product 257); 4096 x 128256 x 4096
// 2700 to 2790, by the clock that the exponentials' power leaves (plain 2650). These are of one sum, over the
// accumulators. There are two now: of the rounded logits for the gradient, and what the unrounded ones have more for the loss. Both cost
// a pass of the head 8 % at a width of 256 (1230 and 1335 us) and 0.9 % at 4096 (9900 and 9990), where the exponentials do not
// bound the kernel. With the accumulators' sum under rounded logits a row of probabilities does not sum to one: where a target has
// a probability of 0.95 the gradient was 0.26 of itself off (200 x 256 x 8000; so 0.0155), at 0.9999 140 times itself (0.028); with
// the rounded sum in the loss that is 2.5e-5 off at 4096 x 1024 x 32000, so 1.2e-6.
//
// With kGated the product is the first half of a gated MLP: the second CTA's half of a B tile are the rows of `up` that go with
// the first one's of `gate`, and the epilogue, which then has both of a column, also writes silu(gate) * up. 4096 x 14336 x 4096
// 605 us, the plain product 577 and with the activation kernel behind it 623; 1000 x 14336 x 4096 164, 156 and 169. Staging the
// activation as well costs a stage of the ring (644 us for the first, 638 with plain stores of it).
#include "tc_gemm.h"

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "activation.cuh"
#include "early_launch.cuh"
#include "launch_count.h"
#include "tc_gemm.cuh"

namespace b200c {

namespace {

using namespace tc;

constexpr int kABytes = kBlockM * kBlockK * 2;  // 16 KB: this CTA's 128 rows of A
constexpr int kOutChunkBytes = kBlockM * 64 * 2;  // of the widest chunk
// How the operands lie in memory, K being the rows of B and of A or its columns: A [m, k] and B [n, k], A [m, k] and B [k, n], A [k,
// m] and B [k, n]. The tensor pipe takes either; only the boxes that bring the operands differ.
enum class PairLayout { kNT, kNN, kTN };
// What the epilogue does besides storing the product.
enum Epilogue { kPlain, kStats, kGated, kGatedGrad };
// Warps of the epilogue: four, one for each quarter of the tensor memory's lanes, or two such sets that take the tiles, and
// with them the two accumulators, in turn.
template <Epilogue EPI>
constexpr int epilogue_sets() { return EPI == kStats ? 2 : 1; }
template <Epilogue EPI>
constexpr int pair_threads() { return 64 + 128 * epilogue_sets<EPI>(); }
constexpr int kAccCols = 256;  // tensor-memory columns of one accumulator

// Stages of the TMA ring. With two sets of epilogue warps one of six makes room for two staging buffers each: with six stages and one
// buffer 4096 x 128256 x 256 takes 361 us, so 315; x 4096 the same either way. So it does for two buffers of gate and two of up.
template <Epilogue EPI>
constexpr int pair_stages() { return EPI == kStats || EPI == kGatedGrad ? 5 : 6; }

// Shared memory for tiles of BN columns: each CTA holds half of the B tile. (Eight stages, which tiles of 128 columns
// leave room for, gain nothing: 512 x 4096 x 4096 in e4m3 15.1 us either way.)
template <int BN, Epilogue EPI>
struct PairTile {
  static constexpr int kStages = pair_stages<EPI>(), kOutBuffers = EPI == kStats || EPI == kGatedGrad ? 4 : 2;
  // Columns that are staged and stored at a time: a quarter of the tile, of narrow tiles half. Only whole swizzle rows of 64
  // are swizzled; rows of 56 lie on different banks anyway, rows of 48 two by two on the same.
  static constexpr int kChunk = BN == 128 ? 64 : BN / 4;
  static_assert(kChunk % 8 == 0 && kChunk > 32 && kChunk <= 64, "two reads of 32 columns each");
  static constexpr int kBHalfBytes = (BN / 2) * kBlockK * 2;
  static constexpr int kStageBytes = kABytes + kBHalfBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + kOutBuffers * kOutChunkBytes + 1024 + 256 + 256 * 4;
};

struct PairBarriers {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t gates[2];  // kGatedGrad: a chunk of gate and up has arrived
  uint32_t tmem_base;
  uint32_t failed;
};
static_assert(sizeof(PairBarriers) <= 256, "the column scales lie behind them");

template <Epilogue EPI>
struct PairMaps {
  CUtensorMap a;    // box 128 rows x 64 columns
  CUtensorMap b;    // box BN / 2 rows x 64 columns (half of the B tile)
  CUtensorMap out;  // box 128 rows x 64 columns
  CUtensorMap b_tail;  // box BN / 4 rows x 64 columns
};
// B and the product in halves, gate and up, of n columns each: a tile has BN / 2 columns of both.
template <>
struct PairMaps<kGated> : PairMaps<kPlain> {
  CUtensorMap b_up, out_up, b_up_tail;
};

// Gate and up, n columns each, and their gradients: boxes as of `out`.
template <>
struct PairMaps<kGatedGrad> : PairMaps<kPlain> {
  CUtensorMap out_up, gate, up;
};

struct PairParams {
  uint32_t* status;
  const float* scale_a;  // e4m3: per row of A, per row of B
  const float* scale_b;
  long long* trace;
  unsigned long long wait_ns;  // limit of a wait (0: kLocalWaitNs)
  int m, n, k, gm;  // k in 16-bit units
  int clear;        // the status words are this call's own
  int stage_bytes, tail_bytes;  // of one K step's loads, both CTAs together, of a tile and of half a tile
  int missing;      // (host) bytes more that a step's loads are said to be
  int whole;        // tiles that are worked on whole; the others, too few to keep half of the pairs busy, in halves of their columns
  float2* stats;    // kStats: [shares of a row, m] maximum and sum of exponentials of rounded logits; per row its target and the target's logit
  float* fine;      // [shares of a row, m] what the sum of unrounded ones has more
  const int64_t* targets;
  float* target_logit;
  __nv_bfloat16* act;  // kGated: [m, n] silu(gate) * up
  const __nv_bfloat16* gate_up;  // (host) kGatedGrad: [m, 2 n]
};

// Maximum and sum of exp(x - maximum) of what a row has shown so far, NaN where one was among it. `sum` is of the logits as they
// are stored, rounded to bf16: the gradient is made from those, and its probabilities sum to one only if the sum is of the same
// numbers. `fine` is what the sum of the unrounded ones, which the loss is made from, has more. Two elements per addition and
// product, two per maximum: the exponentials then take more of the time than what is around them.
struct RowStats {
  float mx = -INFINITY, sum = 0.0f, fine = 0.0f;
  __device__ __forceinline__ void feed(const uint32_t (&r)[32], const uint32_t (&packed)[16]) {
    const auto lo = [&](int i) { return __uint_as_float(packed[i] << 16); };
    const auto hi = [&](int i) { return __uint_as_float(packed[i] & 0xffff0000u); };
    float m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = fmaxf(lo(i), hi(i));
      l[i] = fminf(lo(i), hi(i));
    }
#pragma unroll
    for (int i = 4; i < 16; i += 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        m[j] = max3(m[j], lo(i + j), hi(i + j));
        l[j] = min3(l[j], lo(i + j), hi(i + j));
      }
    }
    const float top = fmaxf(max3(m[0], m[1], m[2]), m[3]), bottom = fminf(min3(l[0], l[1], l[2]), l[3]);
    if (top > mx) {
      if (mx != -INFINITY) {
        const float less = __expf(mx - top);
        sum *= less;
        fine *= less;
      }
      mx = top;
    }
    constexpr float kLog2e = 1.44269504f;
    const float shift = mx == -INFINITY ? 0.0f : -mx;
    float2 s[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)}, f[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
    // What rounding took off an element.
    const auto rest = [&](int i, float2 x) {
      return fma2(x, make_float2(-1.0f, -1.0f), make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
    };
    if (fabsf(mx) <= 32.0f && bottom >= -1e4f) {
      // exp(d) - 1 to the third order: d is 2^-9 of the element at most, the fourth order 6e-7 of the exponential. (Where d is larger,
      // far below the maximum, nothing is left of that.)
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 x = make_float2(lo(i), hi(i)), d = rest(i, x);
        const float2 y = mul2(add2(x, make_float2(shift, shift)), make_float2(kLog2e, kLog2e));
        const float2 e = make_float2(exp2_fast(y.x), exp2_fast(y.y));
        s[i % 2] = add2(s[i % 2], e);
        const float2 q = fma2(fma2(d, make_float2(1.0f / 6.0f, 1.0f / 6.0f), make_float2(0.5f, 0.5f)), d, make_float2(1.0f, 1.0f));
        f[i % 2] = fma2(mul2(e, d), q, f[i % 2]);
      }
    } else {
      // An infinity less an infinity is no number, and its exponential zero or none either; logits above 32768 lose up to more than
      // 64, of which the rest stays off.
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 x = make_float2(lo(i), hi(i)), d = rest(i, x);
        const float2 y = mul2(add2(x, make_float2(shift, shift)), make_float2(kLog2e, kLog2e));
        const float2 e = make_float2(exp2_fast(y.x), exp2_fast(y.y));
        s[i % 2] = add2(s[i % 2], e);
        f[i % 2].x += e.x * (__expf(fminf(d.x, 64.0f)) - 1.0f);
        f[i % 2].y += e.y * (__expf(fminf(d.y, 64.0f)) - 1.0f);
      }
    }
    sum += (s[0].x + s[0].y) + (s[1].x + s[1].y);
    fine += (f[0].x + f[0].y) + (f[1].x + f[1].y);
  }
  static __device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
  }
  static __device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
  }
  static __device__ __forceinline__ float exp2_fast(float x) {
    float d;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(x));
    return d;
  }
  static __device__ __forceinline__ unsigned long long both(float2 v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(v.x), "f"(v.y));
    return d;
  }
  static __device__ __forceinline__ float2 apart(unsigned long long v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
  }
  static __device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(both(a)), "l"(both(b)));
    return apart(d);
  }
  static __device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(both(a)), "l"(both(b)), "l"(both(c)));
    return apart(d);
  }
  static __device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(both(a)), "l"(both(b)));
    return apart(d);
  }
};

// Pair-tile `t` of the schedule: groups of `gm` 256-row tiles, n-major inside a group.
__device__ __forceinline__ void pair_tile_at(int t, int tiles_m, int tiles_n, int gm, int* pm, int* pn) {
  const int per_group = gm * tiles_n;
  const int group = t / per_group;
  const int first = group * gm;
  const int gsz = min(gm, tiles_m - first);
  const int rem = t - group * per_group;
  *pm = first + rem % gsz;
  *pn = rem / gsz;
}

// Item `i` of the work of a product: a tile, or half of one of the last.
struct PairItem {
  int pm, col;  // 256-row tile, first column of the output
  bool tail;
};
template <int TILE_COLS>
__device__ __forceinline__ PairItem pair_item(int i, int whole, int tiles_m, int tiles_n, int gm) {
  const bool tail = i >= whole;
  const int half = tail ? (i - whole) & 1 : 0;
  int pm, pn;
  pair_tile_at(tail ? whole + ((i - whole) >> 1) : i, tiles_m, tiles_n, gm, &pm, &pn);
  return PairItem{pm, pn * TILE_COLS + half * (TILE_COLS / 2), tail};
}

// silu(gate) * up of two columns, from the rounded values: the bits of k_swiglu_fwd.
__device__ __forceinline__ uint32_t gated_pair(uint32_t gate, uint32_t up) {
  const float lo = gated(__uint_as_float(gate << 16), __uint_as_float(up << 16));
  const float hi = gated(__uint_as_float(gate & 0xffff0000u), __uint_as_float(up & 0xffff0000u));
  return pack_bf16(__float_as_uint(lo), __float_as_uint(hi));
}

// The gradients of eight columns of gate and up as k_swiglu_bwd has them, but from the fp32 sums of silu(gate) * up's gradient.
__device__ __forceinline__ void gated_gradients(const uint32_t* d, uint4 gate, uint4 up, uint4* dgate, uint4* dup) {
  const uint32_t g[4] = {gate.x, gate.y, gate.z, gate.w}, u[4] = {up.x, up.y, up.z, up.w};
  uint32_t dg[4], du[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float og[2], ou[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float gf = __uint_as_float(j == 0 ? g[i] << 16 : g[i] & 0xffff0000u), uf = __uint_as_float(j == 0 ? u[i] << 16 : u[i] & 0xffff0000u);
      gated_gradient(__uint_as_float(d[2 * i + j]), gf, uf, &og[j], &ou[j]);
    }
    dg[i] = pack_bf16(__float_as_uint(og[0]), __float_as_uint(og[1]));
    du[i] = pack_bf16(__float_as_uint(ou[0]), __float_as_uint(ou[1]));
  }
  *dgate = make_uint4(dg[0], dg[1], dg[2], dg[3]);
  *dup = make_uint4(du[0], du[1], du[2], du[3]);
}

// The 128 threads of one set of epilogue warps.
__device__ __forceinline__ void epilogue_sync(int set) {
  if (set == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}

template <bool FP8, int BN, Epilogue EPI, PairLayout LAYOUT>
__global__ void __launch_bounds__(pair_threads<EPI>(), 1) k_gemm_pair(const __grid_constant__ PairMaps<EPI> maps, PairParams p) {
  constexpr bool STATS = EPI == kStats, GATED = EPI == kGated, GRAD = EPI == kGatedGrad;
  constexpr bool A_MN = LAYOUT == PairLayout::kTN, B_MN = LAYOUT != PairLayout::kNT;
  static_assert(!B_MN || (!FP8 && !STATS && !GATED && BN % 128 == 0), "whole blocks of 64 columns for each CTA");
  constexpr int kTileCols = GATED ? BN / 2 : BN;  // of the output
  constexpr uint32_t idesc = FP8 ? make_idesc_e4m3(2 * kBlockM, BN) : make_idesc_bf16(2 * kBlockM, BN, A_MN, B_MN);
  constexpr uint32_t idesc_tail = FP8 ? make_idesc_e4m3(2 * kBlockM, BN / 2) : make_idesc_bf16(2 * kBlockM, BN / 2, A_MN, B_MN);
  using Tile = PairTile<BN, EPI>;
  constexpr int kChunk = Tile::kChunk;
  constexpr int kStages = Tile::kStages, kStageBytes = Tile::kStageBytes, kOutBuffers = Tile::kOutBuffers;
  extern __shared__ char smem_raw[];
  // The carve-up must be identical in both CTAs (the MMA addresses both with one descriptor).
  char* stages = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  char* obuf = stages + kStages * kStageBytes;
  PairBarriers* bars = reinterpret_cast<PairBarriers*>(obuf + kOutBuffers * kOutChunkBytes);
  float* col_scales = reinterpret_cast<float*>(obuf + kOutBuffers * kOutChunkBytes + 256);  // e4m3: of the tile in the epilogue
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();  // 0 leads
  const bool leader = cta == 0;
  const int cluster_id = blockIdx.x >> 1, nclusters = gridDim.x >> 1;
  const int tiles_m = (p.m - 1) / (2 * kBlockM) + 1, tiles_n = (p.n - 1) / kTileCols + 1;
  const int items = p.whole + 2 * (tiles_m * tiles_n - p.whole);
  const int k_iters = (p.k + kBlockK - 1) / kBlockK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->acc_full[s], 1);
      mbar_init(&bars->acc_empty[s], 8);  // four epilogue warps in each CTA of the pair
      mbar_init(&bars->gates[s], 1);
    }
    bars->failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_base, 2 * kAccCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anybody signals across
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  grid_release();
  grid_wait();  // everything above may run while the kernel in front still does
  if (p.clear != 0) clear_status(p.status);
  if (STATS && blockIdx.x == 0 && threadIdx.x == 2) p.status[2] = 0u;  // rows whose loss is known
  if (threadIdx.x == 0) trace_stamp_ns(p.trace, 0);

  if (warp == 0) {
    // ---------------- TMA producer (each CTA loads its own A rows and its half of B)
    if (elect_one()) {
      uint32_t it = 0;
      for (int i = cluster_id; i < items && !bars->failed; i += nclusters) {
        const PairItem at = pair_item<kTileCols>(i, p.whole, tiles_m, tiles_n, p.gm);
        const int a_row = (at.pm * 2 + static_cast<int>(cta)) * kBlockM;
        // Each CTA loads one half of the B tile: the second one its last rows, or its rows of the second half of B.
        const int b_row = GATED ? at.col : at.col + static_cast<int>(cta) * (at.tail ? BN / 4 : BN / 2);
        const CUtensorMap* b_map = at.tail ? &maps.b_tail : &maps.b;
        if constexpr (GATED) {
          if (!leader) b_map = at.tail ? &maps.b_up_tail : &maps.b_up;
        }
        const uint32_t bytes = static_cast<uint32_t>(at.tail ? p.tail_bytes : p.stage_bytes);
        for (int kb = 0; kb < k_iters; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1u;
          if (!mbar_wait(&bars->empty[s], ph ^ 1u, p.wait_ns)) {
            bars->failed = 1;
            break;
          }
          // The leader's barrier counts all four loads of the stage.
          if (leader) mbar_expect_tx(&bars->full[s], bytes);
          char* sa = stages + s * kStageBytes;
          if constexpr (A_MN) {
#pragma unroll
            for (int j = 0; j < kBlockM / kMnBlock; ++j) {
              tma_load_2d_pair(sa + j * kMnBlockBytes, &maps.a, &bars->full[s], a_row + j * kMnBlock, kb * kBlockK);
            }
          } else {
            tma_load_2d_pair(sa, &maps.a, &bars->full[s], kb * kBlockK, a_row);
          }
          if constexpr (B_MN) {
#pragma unroll
            for (int j = 0; j < BN / 2 / kMnBlock; ++j) {
              if (j > 0 && at.tail) break;  // half a tile: half the columns
              tma_load_2d_pair(sa + kABytes + j * kMnBlockBytes, &maps.b, &bars->full[s], b_row + j * kMnBlock, kb * kBlockK);
            }
          } else {
            tma_load_2d_pair(sa + kABytes, b_map, &bars->full[s], kb * kBlockK, b_row);
          }
        }
      }
      trace_stamp_ns(p.trace, 1);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      uint32_t it = 0, tile_iter = 0;
      bool cut_short = false;
      for (int i = cluster_id; i < items && !bars->failed; i += nclusters, ++tile_iter) {
        const uint32_t shape = i >= p.whole ? idesc_tail : idesc;
        const uint32_t as = tile_iter & 1u, aph = (tile_iter >> 1) & 1u;
        if (!mbar_wait(&bars->acc_empty[as], aph ^ 1u, p.wait_ns)) {
          bars->failed = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tmem_acc = tmem_base + as * kAccCols;
        for (int kb = 0; kb < k_iters; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1u;
          if (!mbar_wait(&bars->full[s], ph, p.wait_ns)) {
            bars->failed = 1;
            cut_short = true;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(stages + s * kStageBytes);
          const uint64_t da = A_MN ? make_smem_desc_mn(sa) : make_smem_desc(sa);
          const uint64_t db = B_MN ? make_smem_desc_mn(sa + kABytes) : make_smem_desc(sa + kABytes);
          // 16 bf16 (or 32 e4m3) further along K: 32 bytes inside the swizzled row, or 16 rows of 128 bytes.
          constexpr uint64_t kNextA = (A_MN ? kUmmaK * 128 : 32) >> 4, kNextB = (B_MN ? kUmmaK * 128 : 32) >> 4;
#pragma unroll
          for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) {
            if (FP8) {
              umma_f8_pair(tmem_acc, da + kk * kNextA, db + kk * kNextB, shape, (kb | kk) != 0);
            } else {
              umma_bf16_pair(tmem_acc, da + kk * kNextA, db + kk * kNextB, shape, (kb | kk) != 0);
            }
          }
          umma_commit_pair(&bars->empty[s], 3);  // both CTAs may refill the stage
        }
        if (cut_short) break;  // not all of K: the epilogues wait in vain
        umma_commit_pair(&bars->acc_full[as], 3);  // both CTAs' epilogues may read
      }
    }
    if (lane == 0) trace_stamp_ns(p.trace, 2);
  } else {
    // ---------------- epilogue (both CTAs, own 128 rows)
    const int q = warp & 3;
    const int row_in_tile = q * 32 + lane;
    constexpr int kSets = epilogue_sets<EPI>();
    const int set = kSets == 1 ? 0 : (warp - 2) >> 2;
    const bool issuer = (warp & 3) == 2 && lane == 0;
    const int et = static_cast<int>(threadIdx.x) - 64;  // (one set: the column scales)
    // Where 16 bytes of a row lie in a staged chunk.
    const auto staged = [](int row, int piece) { return kChunk == 64 ? row * 128 + ((piece ^ (row & 7)) << 4) : row * kChunk * 2 + piece * 16; };
    // What a row brings along is fetched a tile ahead: its scale, or the column its target has in the tile's row of tiles.
    const auto place_of = [&](int i) {
      const PairItem at = pair_item<kTileCols>(i, p.whole, tiles_m, tiles_n, p.gm);
      return make_int2((at.pm * 2 + static_cast<int>(cta)) * kBlockM, at.col);
    };
    ColScales<BN> fetched;
    float next_scale = 0.0f;
    int64_t next_target = -1;
    const auto fetch = [&](int i) {
      const int2 at = place_of(i);
      const int row = at.x + row_in_tile;
      if (FP8) {
        fetched.fetch(p.scale_b, at.y, p.n, et);
        next_scale = row < p.m ? p.scale_a[row] : 0.0f;
      }
      if (STATS) next_target = row < p.m ? p.targets[row] : -1;
    };
    const int first = cluster_id + set * nclusters, step = kSets * nclusters;
    if (first < items) fetch(first);
    // Chunk `n` of gate and up, where its gradients will be: two buffers, the next chunk on its way while one is worked on.
    uint32_t gate_loads = 0;  // made by this thread
    const auto load_gates = [&](uint32_t n, int2 at) {
      if constexpr (GRAD) {
        gate_loads = n + 1;
        char* const to = obuf + 2 * (n & 1u) * kOutChunkBytes;
        tma_store_wait_read<0>();  // the chunk before the last is out of it
        mbar_expect_tx(&bars->gates[n & 1u], 2 * kOutChunkBytes);
        tma_load_2d(to, &maps.gate, &bars->gates[n & 1u], at.y, at.x);
        tma_load_2d(to + kOutChunkBytes, &maps.up, &bars->gates[n & 1u], at.y, at.x);
      }
    };
    if (GRAD && issuer && first < items) load_gates(0, place_of(first));
    uint32_t tile_iter = static_cast<uint32_t>(set), chunk_iter = 0;
    // After a wait that ran out a warp waits no more, and goes on to the end with the others of its set, which meet it at every
    // chunk; what it stores is NaN. `gates_lost`: that of a load of gate and up.
    bool lost = false, gates_lost = false;
    for (int i = first; i < items; i += step, tile_iter += kSets) {
      const uint32_t as = tile_iter & 1u, aph = (tile_iter >> 1) & 1u;
      const int2 at = place_of(i);
      const int out_row = at.x, out_col = at.y;
      const bool tail = i >= p.whole;
      const float row_scale = next_scale;
      const int target = next_target >= 0 && next_target < p.n ? static_cast<int>(next_target) - out_col : -1;  // column of the tile
      if (FP8) {
        fetched.put(col_scales, et);
        epilogue_sync(set);
      }
      if (i + step < items) fetch(i + step);
      lost = lost || !mbar_wait_warp(&bars->acc_full[as], aph, p.wait_ns);
      if (lost) bars->failed = 1;
      tc_fence_after_sync();
      RowStats row_stats;
      const bool row_there = STATS && out_row + row_in_tile < p.m;
      if constexpr (GATED) {
        static_assert(!GATED || kSets == 1, "");
        const int chunks = kTileCols / kChunk / (tail ? 2 : 1);
        const uint32_t to_up = tail ? BN / 4 : BN / 2;
        for (int j = 0; j < chunks; ++j) {
          if (issuer) tma_store_wait_read<0>();
          epilogue_sync(0);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t g[32], u[32];
            const uint32_t from = tmem_base + as * kAccCols + (static_cast<uint32_t>(q * 32) << 16) +
                static_cast<uint32_t>(j * kChunk + half * 32);
            tmem_ld_32x32(from, g);
            tmem_ld_32x32(from + to_up, u);
            tmem_ld_wait();
            if (lost) no_acc(g), no_acc(u);
            if (j == chunks - 1 && half == 1) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive_leader(&bars->acc_empty[as]);
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint32_t pg[4], pu[4], pa[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                pg[i] = pack_bf16(g[8 * v + 2 * i], g[8 * v + 2 * i + 1]);
                pu[i] = pack_bf16(u[8 * v + 2 * i], u[8 * v + 2 * i + 1]);
                pa[i] = gated_pair(pg[i], pu[i]);
              }
              if (half * 4 + v >= kChunk / 8) continue;
              const int at = staged(row_in_tile, half * 4 + v);
              *reinterpret_cast<uint4*>(obuf + at) = make_uint4(pg[0], pg[1], pg[2], pg[3]);
              *reinterpret_cast<uint4*>(obuf + kOutChunkBytes + at) = make_uint4(pu[0], pu[1], pu[2], pu[3]);
              const int col = out_col + j * kChunk + half * 32 + v * 8;
              if (out_row + row_in_tile < p.m && col < p.n) {
                *reinterpret_cast<uint4*>(p.act + static_cast<size_t>(out_row + row_in_tile) * p.n + col) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
              }
            }
          }
          fence_proxy_async_smem();
          epilogue_sync(0);
          const int col = out_col + j * kChunk;
          if (issuer && out_row < p.m && col < p.n) {
            tma_store_2d(&maps.out, obuf, col, out_row);
            tma_store_2d(&maps.out_up, obuf + kOutChunkBytes, col, out_row);
            tma_store_commit();
          }
        }
        continue;
      }
      if constexpr (GRAD) {
        static_assert(!GRAD || (kSets == 1 && kChunk == 64), "");
        const int chunks = BN / kChunk / (tail ? 2 : 1);
        for (int j = 0; j < chunks; ++j, ++chunk_iter) {
          const uint32_t b = chunk_iter & 1u;
          if (issuer && !gates_lost) {
            if (j + 1 < chunks) {
              load_gates(chunk_iter + 1, make_int2(out_row, out_col + (j + 1) * kChunk));
            } else if (i + step < items) {
              load_gates(chunk_iter + 1, place_of(i + step));
            }
          }
          gates_lost = gates_lost || !mbar_wait_warp(&bars->gates[b], (chunk_iter >> 1) & 1u, p.wait_ns);
          if (gates_lost) bars->failed = 1;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t d[32];
            tmem_ld_32x32(tmem_base + as * kAccCols + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(j * kChunk + half * 32), d);
            tmem_ld_wait();
            if (lost || gates_lost) no_acc(d);
            if (j == chunks - 1 && half == 1) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive_leader(&bars->acc_empty[as]);
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4* const gate = reinterpret_cast<uint4*>(obuf + 2 * b * kOutChunkBytes + staged(row_in_tile, half * 4 + v));
              uint4* const up = gate + kOutChunkBytes / 16;
              gated_gradients(d + 8 * v, *gate, *up, gate, up);
            }
          }
          fence_proxy_async_smem();
          epilogue_sync(0);
          const int col = out_col + j * kChunk;
          if (issuer && out_row < p.m && col < p.n) {
            tma_store_2d(&maps.out, obuf + 2 * b * kOutChunkBytes, col, out_row);
            tma_store_2d(&maps.out_up, obuf + (2 * b + 1) * kOutChunkBytes, col, out_row);
            tma_store_commit();
          }
        }
        continue;
      }
      const int chunks = BN / kChunk / (tail ? 2 : 1);
      for (int j = 0; j < chunks; ++j, ++chunk_iter) {
        char* buf = obuf + (2 * set + (chunk_iter & 1u)) * kOutChunkBytes;
        uint32_t acc[2][32];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          tmem_ld_32x32(tmem_base + as * kAccCols + (static_cast<uint32_t>(q * 32) << 16) +
                            static_cast<uint32_t>(j * kChunk + half * 32),
                        acc[half]);
        }
        tmem_ld_wait();
        if (lost) no_acc(acc[0]), no_acc(acc[1]);
        if (j == chunks - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_leader(&bars->acc_empty[as]);
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t(&r)[32] = acc[half];
          if (FP8) scale_acc32(r, row_scale, col_scales + j * kChunk + half * 32);
          if constexpr (STATS) {
            const int past = p.n - out_col - j * kChunk - half * 32;  // columns beyond the last are zeros of the tile, not logits
            if (past < 32) {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = i < past ? r[i] : 0xff800000u;
            }
          }
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) packed[i] = pack_bf16(r[2 * i], r[2 * i + 1]);
          if constexpr (STATS) {
            const int col = j * kChunk + half * 32;
            if (row_there) row_stats.feed(r, packed);
            if (row_there && target >= col && target < col + 32) {
              uint32_t z = 0;
#pragma unroll
              for (int i = 0; i < 32; ++i) z = target == col + i ? r[i] : z;
              p.target_logit[out_row + row_in_tile] = __uint_as_float(z);
            }
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (half * 4 + v >= kChunk / 8) continue;
            *reinterpret_cast<uint4*>(buf + staged(row_in_tile, half * 4 + v)) = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
          }
        }
        fence_proxy_async_smem();
        // The other buffer is free once the store before this one has been read: one meeting per chunk says both that
        // and that this one is full.
        if (issuer) tma_store_wait_read<0>();
        epilogue_sync(set);
        if (issuer && out_row < p.m && out_col + j * kChunk < p.n) {
          tma_store_2d(&maps.out, buf, out_col + j * kChunk, out_row);
          tma_store_commit();
        }
      }
      if (row_there) {
        const size_t at = static_cast<size_t>(out_col / BN) * p.m + out_row + row_in_tile;
        p.stats[at] = make_float2(row_stats.mx, row_stats.sum);
        p.fine[at] = row_stats.fine;
      }
    }
    if (issuer) {
      tma_store_wait_all<0>();
      // Of loads that nobody waited for in the end, the last of each buffer may still be on its way.
      for (uint32_t n = gate_loads; n > 0 && n + 2 > gate_loads; --n) mbar_wait(&bars->gates[(n - 1) & 1u], ((n - 1) >> 1) & 1u, p.wait_ns);
      trace_stamp_ns(p.trace, 3);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // the peer may still be reading this CTA's shared memory / signalling its barriers
  if (warp == 1) {
    tmem_dealloc_pair(tmem_base, 2 * kAccCols);
  }
  if (threadIdx.x == 0 && bars->failed && p.status != nullptr) p.status[0] = p.status[0] | kStatusTimeout;
  if (threadIdx.x == 0) trace_stamp_ns(p.trace, 7);
}

// Whether the tiles of a last, partial wave are worked on in halves of their columns: where at most half of the pairs would
// have one. In us without and so: bf16 4096 x 4096 x 14336 (34 of 74 pairs) 328 and 317, 4096 x 2560 x 2560 (12) 43.0 and 38.7, 1000
// x 28672 x 4096 (4) 161.7 and 156.6; e4m3 4096 x 4096 x 14336 175.7 and 168.2, 640 x 20480 x 2048 (18) 28.7 and 26.8; gated 2048 x
// 14336 x 4096 (8) 313 and 308, 512 x 14336 x 4096 (2) 99.1 and 94.0.
bool tail_in_halves(int64_t tiles, int64_t pairs, int columns) {
  const int64_t rest = tiles % pairs;
  return columns > 128 && rest > 0 && 2 * rest <= pairs;
}

constexpr int kDevices = 64;  // whose answers are kept

// Pairs that the current GPU holds at once (each CTA fills an SM), or 0 after an error. Kept per device; a query that
// failed is asked again at the next call.
template <bool FP8, int BN, Epilogue EPI = kPlain, PairLayout LAYOUT = PairLayout::kNT>
int resident_pairs() {
  static std::atomic<int> known[kDevices];
  int device = 0, n = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return 0;
  std::atomic<int>* kept = device >= 0 && device < kDevices ? &known[device] : nullptr;
  if (kept != nullptr) n = kept->load(std::memory_order_acquire);
  if (n > 0) return n;
  if (cudaFuncSetAttribute(k_gemm_pair<FP8, BN, EPI, LAYOUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairTile<BN, EPI>::kSmemBytes) !=
      cudaSuccess) {
    return 0;
  }
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(pair_threads<EPI>());
  cfg.dynamicSmemBytes = PairTile<BN, EPI>::kSmemBytes;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, k_gemm_pair<FP8, BN, EPI, LAYOUT>, &cfg) != cudaSuccess || n < 1) return 0;
  if (kept != nullptr) kept->store(n, std::memory_order_release);
  return n;
}

void set_limits(PairParams* p, const GiveUp* give_up) {
  if (give_up == nullptr) return;
  p->wait_ns = give_up->wait_ns;
  p->missing = give_up->missing;
}

// `ldc`: row stride of the output in elements (0: n), `lda`, `ldb`: of the operands as they lie in memory (0: rows follow one another).
template <bool FP8, int BN, Epilogue EPI = kPlain, PairLayout LAYOUT = PairLayout::kNT>
cudaError_t launch_pair(const void* a, const void* b, void* c, PairParams p, cudaStream_t stream, int64_t ldc = 0, int64_t lda = 0,
                        int64_t ldb = 0) {
  const int pairs = resident_pairs<FP8, BN, EPI, LAYOUT>();
  if (pairs < 1) {
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
  }
  constexpr int kTileCols = EPI == kGated ? BN / 2 : BN;
  PairMaps<EPI> maps;
  constexpr bool A_MN = LAYOUT == PairLayout::kTN, B_MN = LAYOUT != PairLayout::kNT;
  const bool mapped_a = A_MN ? make_map(&maps.a, a, p.k, p.m, kBlockK, lda) : make_map(&maps.a, a, p.m, p.k, a_box_rows(p.m), lda);
  const bool mapped_b = B_MN ? make_map(&maps.b, b, p.k, p.n, kBlockK, ldb)
                             : make_map(&maps.b, b, p.n, p.k, BN / 2, ldb) && make_map(&maps.b_tail, b, p.n, p.k, BN / 4, ldb);
  if (!mapped_a || !mapped_b || !make_map(&maps.out, c, p.m, p.n, kBlockM, ldc, PairTile<BN, EPI>::kChunk)) {
    return cudaErrorInvalidValue;
  }
  if constexpr (EPI == kGated) {
    const auto* up = static_cast<const char*>(b) + static_cast<size_t>(p.n) * p.k * 2;
    if (!make_map(&maps.b_up, up, p.n, p.k, BN / 2) || !make_map(&maps.b_up_tail, up, p.n, p.k, BN / 4) ||
        !make_map(&maps.out_up, static_cast<char*>(c) + static_cast<size_t>(p.n) * 2, p.m, p.n, kBlockM, ldc, PairTile<BN, EPI>::kChunk)) {
      return cudaErrorInvalidValue;
    }
  }
  if constexpr (EPI == kGatedGrad) {
    constexpr int kCols = PairTile<BN, EPI>::kChunk;
    if (!make_map(&maps.out_up, static_cast<__nv_bfloat16*>(c) + p.n, p.m, p.n, kBlockM, ldc, kCols) ||
        !make_map(&maps.gate, p.gate_up, p.m, p.n, kBlockM, ldc, kCols) || !make_map(&maps.up, p.gate_up + p.n, p.m, p.n, kBlockM, ldc, kCols)) {
      return cudaErrorInvalidValue;
    }
  }
  const int a_bytes = A_MN ? kABytes : a_box_rows(p.m) * kBlockK * 2;
  p.stage_bytes = 2 * (a_bytes + PairTile<BN, EPI>::kBHalfBytes) + p.missing;
  p.tail_bytes = 2 * (a_bytes + PairTile<BN, EPI>::kBHalfBytes / 2) + p.missing;
  const int tiles_m = (p.m - 1) / (2 * kBlockM) + 1, tiles_n = (p.n - 1) / kTileCols + 1;
  const int64_t tiles = static_cast<int64_t>(tiles_m) * tiles_n;
  const bool halves = EPI != kStats && tail_in_halves(tiles, pairs, BN);
  p.whole = static_cast<int>(halves ? tiles - tiles % pairs : tiles);
  // A rows of a group stay in L2 while the pairs sweep over n: at most 8 pair-tiles and ~40 MB. Every group reads B again,
  // so where L2 does not keep that either (above 48 MB) groups are of up to 16 pair-tiles and 32 MB. In us under the power
  // cap with 8 and 16: 4096 x 28672 x 4096 in e4m3 (B of 117 MB) 397 and 390, 8192 x 14336 x 4096 (59 MB) 400 and 392; 4096 x
  // 8192 x 1024 (8 MB) 43.4 and 45.8.
  const size_t a_tile_bytes = static_cast<size_t>(2 * kBlockM) * p.k * 2;
  const bool b_again = static_cast<size_t>(p.n) * p.k * 2 * (BN / kTileCols) > (48u << 20);
  p.gm = std::max(1, std::min({b_again ? 16 : 8, tiles_m, static_cast<int>((b_again ? 32u << 20 : 40u << 20) / std::max<size_t>(a_tile_bytes, 1))}));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * static_cast<unsigned>(std::min<int64_t>(pairs, halves ? tiles + tiles % pairs : tiles)));
  cfg.blockDim = dim3(pair_threads<EPI>());
  cfg.dynamicSmemBytes = PairTile<BN, EPI>::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_gemm_pair<FP8, BN, EPI, LAYOUT>, maps, p);
  note_kernel_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

} // namespace

int pairs_at_once(bool fp8) { return fp8 ? resident_pairs<true, 256>() : resident_pairs<false, 256>(); }

double wave_cost(int64_t tiles, int64_t at_once) {
  const int64_t part = tiles % at_once;
  return static_cast<double>(tiles / at_once) + (part > 0 ? 0.5 + 0.5 * static_cast<double>(part) / static_cast<double>(at_once) : 0.0);
}

// The width whose waves take least. A wave of full width costs 1 and one of half the width 0.575 (the rows of A come in either
// way), a last wave of halves a tenth more. 256 unless another is 1 % ahead. Of 39 sizes, types and epilogues this takes the
// best width or one at most 2 % behind it. In us with 256 / 224 / 192 columns: bf16 1000 x 6144 x 4096 40.1 / 43.0 / 38.9, 1500 x 5000 x
// 2992 38.3 / 34.9 / 40.7, 1024 x 8192 x 1024 16.2 / 15.2 / 15.9, 4096 x 4096 x 14336 318 / 333 / 331; e4m3 1500 x 5000 x 2992 28.0 /
// 26.6 / 31.4, 4096 x 2560 x 2560 23.0 / 24.1 / 23.4; gated 700 x 5000 x 768 16.8 / 15.4 / 16.0.
int pair_columns(int m, int n, bool gated, double* cost) {
  const int64_t pairs = std::max(1, pairs_at_once(false)), tiles_m = (m - 1) / (2 * kBlockM) + 1;
  int best = 256;
  double least = 0.0;
  const auto width_cost = [](int columns) { return 0.15 + 0.85 * columns / 256.0; };
  for (const int columns : {256, 224, 192, 128}) {
    if (gated && columns == 128) break;
    const int64_t tiles = tiles_m * ((n - 1) / (gated ? columns / 2 : columns) + 1), rest = tiles % pairs;
    const double here = (tail_in_halves(tiles, pairs, columns)
                             ? static_cast<double>(tiles / pairs) * width_cost(columns) + 1.1 * wave_cost(2 * rest, pairs) * width_cost(columns / 2)
                             : wave_cost(tiles, pairs) * width_cost(columns)) * (columns == 256 ? 0.99 : 1.0);
    if (columns == 256 || here < least) {
      best = columns;
      least = here;
    }
  }
  if (cost != nullptr) *cost = least;
  return best;
}

bool pair_tiles_fit(int m, int n, bool fp8) {
  const int pairs = fp8 ? resident_pairs<true, 128>() : resident_pairs<false, 128>();
  return static_cast<int64_t>((m - 1) / (2 * kBlockM) + 1) * ((n - 1) / 128 + 1) <= pairs;
}

cudaError_t launch_gemm_nt_pair(const void* a, const void* b, void* c, int m, int n, int k, const float* scale_a,
                                const float* scale_b, uint32_t* status, cudaStream_t stream, int columns, const CommDev* layer,
                                const GiveUp* give_up) {
  if (m <= 0 || n <= 0 || k <= 0 || k % 8 != 0 || n % 8 != 0) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) {
    return cudaErrorInvalidValue;
  }
  PairParams p{};
  set_limits(&p, give_up);
  p.status = status;
  p.clear = layer == nullptr && status != nullptr ? 1 : 0;
  p.scale_a = scale_a;
  p.scale_b = scale_b;
  p.trace = layer != nullptr ? layer->trace : nullptr;
  p.m = m;
  p.n = n;
  p.k = k;
  const auto launch = [&](auto fp8) {
    switch (columns != 0 ? columns : pair_columns(m, n, false)) {
      case 128: return launch_pair<fp8(), 128>(a, b, c, p, stream);
      case 192: return launch_pair<fp8(), 192>(a, b, c, p, stream);
      case 224: return launch_pair<fp8(), 224>(a, b, c, p, stream);
      default: return launch_pair<fp8(), 256>(a, b, c, p, stream);
    }
  };
  return scale_a != nullptr ? launch(std::true_type()) : launch(std::false_type());
}

// Tiles of 128 columns where they are at most a wave, otherwise of 256: the blocks of 64 columns that each CTA brings allow no width
// between. A step brings its operands in up to four boxes, and the tensor pipe takes them as fast as along K: 4096 x 14336 x 4096
// 290 us with both along rows, 294 with one (the tensor library 324 and 319), 1000 x 28672 x 4096 156 (183).
cudaError_t launch_gemm_pair_mn(const void* a, int64_t lda, bool a_by_columns, const void* b, int64_t ldb, void* c, int m, int n, int k,
                                uint32_t* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0 || lda % 8 != 0 || ldb % 8 != 0 || n % 8 != 0 || lda < (a_by_columns ? m : k) || ldb < n) {
    return cudaErrorInvalidValue;
  }
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) {
    return cudaErrorMisalignedAddress;
  }
  PairParams p{};
  p.status = status;
  p.clear = status != nullptr ? 1 : 0;
  p.m = m;
  p.n = n;
  p.k = k;
  const bool narrow = pair_tiles_fit(m, n, false);
  if (a_by_columns) {
    return narrow ? launch_pair<false, 128, kPlain, PairLayout::kTN>(a, b, c, p, stream, 0, lda, ldb)
                  : launch_pair<false, 256, kPlain, PairLayout::kTN>(a, b, c, p, stream, 0, lda, ldb);
  }
  return narrow ? launch_pair<false, 128, kPlain, PairLayout::kNN>(a, b, c, p, stream, 0, lda, ldb)
                : launch_pair<false, 256, kPlain, PairLayout::kNN>(a, b, c, p, stream, 0, lda, ldb);
}

// What it saves is the product's way through memory and a kernel of memory's speed; gate and up come and their gradients go while
// the next tile's product runs. Gate and up by boxes into the buffers that their gradients leave from: rows read by one thread each
// instead were 200 us for 2048 x 14336 x 4096, so 198, and 89 for 2048 x 8192 x 2048, so 67 (two sets of epilogue warps 212 and 91).
cudaError_t launch_gemm_gated_grad(const void* dy, const void* w, const void* gate_up, void* dgate_up, int m, int n, int k, uint32_t* status,
                                   cudaStream_t stream, const GiveUp* give_up) {
  if (m <= 0 || n <= 0 || k <= 0 || n % 8 != 0 || k % 8 != 0 || n > INT32_MAX / 2) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(gate_up) |
       reinterpret_cast<uintptr_t>(dgate_up)) & 15u) {
    return cudaErrorMisalignedAddress;
  }
  PairParams p{};
  set_limits(&p, give_up);
  p.status = status;
  p.clear = status != nullptr ? 1 : 0;
  p.m = m;
  p.n = n;
  p.k = k;
  p.gate_up = static_cast<const __nv_bfloat16*>(gate_up);
  const int64_t ld = 2 * static_cast<int64_t>(n);
  return pair_tiles_fit(m, n, false) ? launch_pair<false, 128, kGatedGrad, PairLayout::kNN>(dy, w, dgate_up, p, stream, ld)
                                     : launch_pair<false, 256, kGatedGrad, PairLayout::kNN>(dy, w, dgate_up, p, stream, ld);
}

int head_row_shares(int m, int n) {
  const int bn = pair_tiles_fit(m, n, false) ? 128 : 256;
  return (n - 1) / bn + 1;
}

cudaError_t launch_head_logits(const void* x, const void* w, void* logits, int64_t ld, const int64_t* targets, int m, int n, int k,
                               float2* stats, float* fine, float* target_logit, uint32_t* words, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0 || k % 8 != 0 || ld % 8 != 0 || ld < n) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(logits)) & 15u) {
    return cudaErrorMisalignedAddress;
  }
  PairParams p{};
  p.status = words;
  p.clear = 1;
  p.m = m;
  p.n = n;
  p.k = k;
  p.stats = stats;
  p.fine = fine;
  p.targets = targets;
  p.target_logit = target_logit;
  return pair_tiles_fit(m, n, false) ? launch_pair<false, 128, kStats>(x, w, logits, p, stream, ld)
                                     : launch_pair<false, 256, kStats>(x, w, logits, p, stream, ld);
}

cudaError_t launch_gemm_gated(const void* x, const void* w, void* gate_up, void* act, int m, int n, int k, uint32_t* status,
                              cudaStream_t stream, int columns, const GiveUp* give_up) {
  if (m <= 0 || n <= 0 || k <= 0 || k % 8 != 0 || n % 8 != 0) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(act)) & 15u) {
    return cudaErrorMisalignedAddress;
  }
  PairParams p{};
  set_limits(&p, give_up);
  p.status = status;
  p.clear = 1;
  p.m = m;
  p.n = n;
  p.k = k;
  p.act = static_cast<__nv_bfloat16*>(act);
  const int64_t ld = 2 * static_cast<int64_t>(n);
  switch (columns != 0 ? columns : pair_columns(m, n, true)) {
    case 192: return launch_pair<false, 192, kGated>(x, w, gate_up, p, stream, ld);
    case 224: return launch_pair<false, 224, kGated>(x, w, gate_up, p, stream, ld);
    default: return launch_pair<false, 256, kGated>(x, w, gate_up, p, stream, ld);
  }
}

} // namespace b200c
