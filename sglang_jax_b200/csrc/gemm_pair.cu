// bf16 GEMM of prefill sizes on pairs of SMs  (tcgen05 cta_group::2):  out[T, N] = x[T, K] . w[N, K]^T (+ bias)
//
// A pair of CTAs works on 256 weight rows (the MMA's M dimension, 128 in each CTA) times up to 256 tokens (N): each CTA fetches its
// half of both operands, the leader's tensor instruction reads both halves.  An SM takes in 64 bytes a clock from L2: the 48 KB that a
// 128 x 256 tile on one SM needs for 64 of K arrive in 0.39 us, longer than the tensor core works on them; a pair's 256 x 256
// tile takes in 32 KB an SM.  With tokens on the N dimension a tile's width follows its tokens in steps of 32, where tiles of 128
// rows computed on padding (293 tokens: 384 rows; experts: half a tile each).
//
// What a slice of K costs beside that: a round through the barriers of the ring 0.17 us, a copy 0.1 us of its issuing thread.  So a
// stage holds 128 of K (two swizzle blocks) and takes one copy for each operand (maps with the blocks of K as a dimension).
// Against one SM's 128 x 256 tiles, operands cold: 293 x 14336 -> 4096 98 -> 59 us, 293 x 4096 -> 6144 39 -> 29, 2500 x 2048 -> 2048
// 35 -> 27, 8192 x 5120 -> 51200 3264 -> 2735 us (1570 TFLOP/s).
//
//   warp 0      TMA producer of its CTA; both halves complete on the leader's barrier
//   warp 1      leader only: issues tcgen05.mma 256 x n x 16, commits to both CTAs' barriers
//   warps 2..5  epilogue of the CTA's 128 rows, two accumulators deep: tensor memory -> shared memory (transposed) -> 16-byte stores
//
// Grouped: rows of x are sorted by group (experts), tiles of at most `bt` rows come from a device-side list.
// GATED: w holds N gate rows, then N up rows; a CTA's 128 rows are 64 of each, and silu(gate) * up leaves the epilogue, from
// the fp32 sums: the activations are written once, at half the width.
//
// No load is multicast; the pair shares the operands inside the tensor instruction.  All waits are bounded.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "gemm_pair.h"

namespace sglb {
namespace {

constexpr int BK = 64;                         // 64 bf16 = one 128-byte swizzle row: a block of K
constexpr int kBlocks = 2;                     // blocks of K per stage
constexpr int kRows = 128;                     // weight rows of one CTA
constexpr int kThreads = 192;
constexpr int kEpiThreads = 128;
constexpr int kBlockA = kRows * BK * 2, kStageA = kBlocks * kBlockA;
constexpr int kMaxStages = 8;
constexpr int kChunk = 32;                     // tokens per epilogue step
constexpr int kTmemCols = 512;                 // two accumulators of up to 256 columns
constexpr int kMaxSmem = 227 * 1024;

struct Bars {
  uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2];
  uint32_t tmem_slot;
  int abort_flag;
};

struct Params {
  __nv_bfloat16* out;
  const __nv_bfloat16* bias;
  Status* status;
  int T, N, blocks;              // N: output columns of one group; blocks of K
  int tiles_w, tiles_t, bt;      // tiles over the output columns / tokens, tokens of a tile at most
  int band;                      // token tiles of a band: a band's tiles are done for all weight rows before the next band's
  int stages, stage_bytes, block_b;   // ring; bytes of a CTA's tokens in one block of K
  const int *group_offsets, *tile_group, *tile_row0, *num_token_tiles;   // grouped (null: dense)
};

struct Item {
  int w0, w_base;                // first output column of the tile; first weight row of the group
  int row0, rows;                // its tokens
};

template <bool GATED>
__device__ __forceinline__ bool get_item(const Params& p, int i, Item& s) {
  constexpr int kCols = GATED ? kRows : 2 * kRows;              // output columns of a pair's tile
  int t, w;
  if (p.group_offsets != nullptr) {
    // all weight tiles of a token tile together, an expert's token tiles one after another: both operands are read from DRAM once
    if (i >= *p.num_token_tiles * p.tiles_w) return false;
    t = i / p.tiles_w;
    w = i - t * p.tiles_w;
    const int g = p.tile_group[t];
    s.row0 = p.tile_row0[t];
    s.rows = min(p.group_offsets[g + 1] - s.row0, p.bt);
    s.w_base = g * p.N * (GATED ? 2 : 1);
  } else {
    if (i >= p.tiles_t * p.tiles_w) return false;
    const int per_band = p.band * p.tiles_w, b = i / per_band, r = i - b * per_band;
    const int in_band = min(p.band, p.tiles_t - b * p.band);
    w = r / in_band;
    t = b * p.band + r - w * in_band;
    s.row0 = t * p.bt;
    s.rows = min(p.bt, p.T - s.row0);
    s.w_base = 0;
  }
  s.w0 = w * kCols;
  return true;
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Named barrier that says whether `ok` holds in every one of its threads.
__device__ __forceinline__ bool bar_all(int id, int threads, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.and.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(id), "r"(threads), "r"(static_cast<uint32_t>(ok)) : "memory");
  return r != 0;
}
// Copies into this CTA's shared memory that complete on a barrier of the pair's leader (no multicast): 64 elements of K x rows (x gate
// and up) x blocks of K.
__device__ __forceinline__ void tma_load_pair_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int row, int block) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(block)
      : "memory");
}
__device__ __forceinline__ void tma_load_pair_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int row, int block) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(block)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs once the tensor instructions issued so far are done.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}

template <bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using Staged = std::conditional_t<GATED, float, __nv_bfloat16>;
  Staged* staging = reinterpret_cast<Staged*>(smem + p.stages * p.stage_bytes);          // [2][kChunk][kRows]
  Bars* bars = reinterpret_cast<Bars*>(staging + 2 * kChunk * kRows);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    prefetch_tmap(&map_w);
    prefetch_tmap(&map_x);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&bars->full[s]), 1);
      mbar_init(smem_u32(&bars->empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bars->acc_full[a]), 1);
      mbar_init(smem_u32(&bars->acc_empty[a]), 8);              // one arrival per epilogue warp of the pair (the leader's counts)
    }
    bars->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&bars->tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      Item it;
      for (int i = pair; !*abort_flag && get_item<GATED>(p, i, it); i += pairs) {
        const int x_row = it.row0 + static_cast<int>(rank) * ((it.rows + 31) / 32 * 16);
        const int w_row = it.w_base + it.w0 + static_cast<int>(rank) * (GATED ? kRows / 2 : kRows);
        for (int kb = 0; kb < p.blocks; kb += kBlocks) {
          if (!mbar_wait(smem_u32(&bars->empty[stage]), phase ^ 1)) {
            report(p.status, kTimeoutEmptyBarrier, i, kb);
            *abort_flag = 1;
            break;
          }
          const uint32_t fb = in_cta(smem_u32(&bars->full[stage]), 0);
          if (rank == 0) mbar_expect_tx(smem_u32(&bars->full[stage]), 2 * p.stage_bytes);
          const uint32_t sa = smem_u32(smem + stage * p.stage_bytes);
          tma_load_pair_4d(sa, &map_w, fb, w_row, kb);
          tma_load_pair_3d(sa + kStageA, &map_x, fb, x_row, kb);
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      Item it;
      for (int i = pair; !*abort_flag && get_item<GATED>(p, i, it); i += pairs) {
        if (!mbar_wait(smem_u32(&bars->acc_empty[acc]), acc_phase ^ 1)) {
          report(p.status, kTimeoutTmemEmpty, i, acc);
          *abort_flag = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t idesc = make_idesc(2 * kRows, (it.rows + 31) / 32 * 32, 1, 1);
        const uint32_t d = tmem + acc * 256;
        bool ok = true;
        for (int kb = 0; kb < p.blocks; kb += kBlocks) {
          if (!mbar_wait(smem_u32(&bars->full[stage]), phase)) {
            report(p.status, kTimeoutFullBarrier, i, kb);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * p.stage_bytes);
          const uint64_t da = make_smem_desc_sw128(sa), db = make_smem_desc_sw128(sa + kStageA);
          const uint64_t next_b = p.block_b >> 4;
          const int n = min(kBlocks, p.blocks - kb);
          for (int j = 0; j < n; ++j) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_pair(d, da + j * (kBlockA >> 4) + 2 * k, db + j * next_b + 2 * k, idesc, (kb + j > 0 || k > 0) ? 1u : 0u);
          }
          commit_pair(smem_u32(&bars->empty[stage]));
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        commit_pair(smem_u32(&bars->acc_full[acc]));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    const int q = warp & 3, row = q * 32 + lane, tid = threadIdx.x - 64;
    int acc = 0, buf = 0;
    uint32_t acc_phase = 0;
    Item it;
    for (int i = pair; get_item<GATED>(p, i, it); i += pairs) {
      bool ok = !*abort_flag;
      if (ok && !mbar_wait(smem_u32(&bars->acc_full[acc]), acc_phase)) {
        report(p.status, kTimeoutTmemFull, i, acc);
        *abort_flag = 1;
        ok = false;
      }
      // all go on or none: they meet at the barriers below
      if (!bar_all(1, kEpiThreads, ok)) break;
      tc_fence_after_sync();
      const uint32_t t_addr = tmem + (static_cast<uint32_t>(q * 32) << 16) + acc * 256;
      const int col0 = it.w0 + static_cast<int>(rank) * (GATED ? kRows / 2 : kRows);
      [[maybe_unused]] float b = 0.f;
      if constexpr (!GATED)
        if (p.bias != nullptr && col0 + row < p.N) b = __bfloat162float(p.bias[col0 + row]);
#pragma unroll 1
      for (int c0 = 0; c0 < it.rows; c0 += kChunk) {
        uint32_t v[32];
        tmem_ld32(t_addr + c0, v);
        tmem_ld_wait();
        if (c0 + kChunk >= it.rows) {
          // drained: the accumulator goes back to the leader's MMA thread
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) arrive_cluster(in_cta(smem_u32(&bars->acc_empty[acc]), 0));
        }
        Staged* st = staging + buf * (kChunk * kRows);
#pragma unroll
        for (int e = 0; e < kChunk; ++e) {
          if constexpr (GATED) st[e * kRows + row] = __uint_as_float(v[e]);
          else st[e * kRows + row] = __float2bfloat16(__uint_as_float(v[e]) + b);
        }
        // one barrier a step: a buffer is written again two steps on, behind the next step's barrier
        named_bar_sync(2, kEpiThreads);
        const int left = it.rows - c0;
        __nv_bfloat16* out = p.out + static_cast<size_t>(it.row0 + c0) * p.N;
        if constexpr (GATED) {
#pragma unroll
          for (int r = 0; r < kChunk * (kRows / 16) / kEpiThreads; ++r) {
            const int vid = r * kEpiThreads + tid, e = vid / (kRows / 16), part = vid % (kRows / 16);
            const int col = col0 + part * 8;
            if (e < left && col < p.N) {
              const float* g = st + e * kRows + part * 8;
              float y[8];
#pragma unroll
              for (int j = 0; j < 8; j += 4) {
                const float4 a = *reinterpret_cast<const float4*>(g + j), u = *reinterpret_cast<const float4*>(g + kRows / 2 + j);
                y[j] = a.x / (1.f + __expf(-a.x)) * u.x;
                y[j + 1] = a.y / (1.f + __expf(-a.y)) * u.y;
                y[j + 2] = a.z / (1.f + __expf(-a.z)) * u.z;
                y[j + 3] = a.w / (1.f + __expf(-a.w)) * u.w;
              }
              *reinterpret_cast<uint4*>(out + static_cast<size_t>(e) * p.N + col) =
                  make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
            }
          }
        } else {
#pragma unroll
          for (int r = 0; r < kChunk * (kRows / 8) / kEpiThreads; ++r) {
            const int vid = r * kEpiThreads + tid, e = vid / (kRows / 8), part = vid % (kRows / 8);
            const int col = col0 + part * 8;
            if (e < left && col < p.N)
              *reinterpret_cast<uint4*>(out + static_cast<size_t>(e) * p.N + col) =
                  *reinterpret_cast<const uint4*>(st + e * kRows + part * 8);
          }
        }
        buf ^= 1;
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // give copies that are still in flight time to land before shared memory is released
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncwarp();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
  cluster_sync();
}

template <bool GATED>
cudaError_t launch(const CUtensorMap& mw, const CUtensorMap& mx, Params& p, long long items, cudaStream_t s) {
  p.block_b = p.bt / 2 * 128;
  p.stage_bytes = kStageA + kBlocks * p.block_b;
  const int fixed = 2 * kChunk * kRows * (GATED ? 4 : 2) + static_cast<int>(sizeof(Bars)) + 1024;
  p.stages = std::min(kMaxStages, (kMaxSmem - fixed) / p.stage_bytes);
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm_pair_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (configured != cudaSuccess) return configured;
  const int pairs = static_cast<int>(std::min<long long>(items, sm_count() / 2));
  return launch_pdl(gemm_pair_kernel<GATED>, dim3(2 * pairs), dim3(kThreads), static_cast<size_t>(p.stages * p.stage_bytes + fixed), s, mw,
                    mx, p);
}

// Tokens of a dense tile.  64 of K cost the tensor core 0.35 us for 256 tokens and the ring 0.2 us at least, a tile about a
// microsecond more; the fewest such units over the pairs' waves win, of nearly equal ones the widest tile (fewer bytes moved: large
// products are bound by power).  293 tokens, 4096 columns: 16 x 4 tiles of 96 on 74 pairs instead of 48 tiles of 128 x 256.
int pick_tile(int T, int cols, int blocks) {
  const int pairs = std::max(sm_count() / 2, 1);
  int best = 256;
  float best_cost = 0.f;
  for (int bt = 256; bt >= 32; bt -= 32) {
    const long long tiles = static_cast<long long>((T + bt - 1) / bt) * cols;
    const float slice = std::max(bt * (0.35f / 256.f), 0.18f + bt * (0.08f / 256.f));
    const float cost = static_cast<float>((tiles + pairs - 1) / pairs) * (blocks * slice + 1.f);
    if (best_cost == 0.f || cost < best_cost * 0.97f) {
      best_cost = cost;
      best = bt;
    }
  }
  return best;
}

// Microseconds of a dense product, fitted to 886 sizes (257 to 8192 tokens, 8 to 28672 columns, K 64 to 14336; operands in L2 where they
// fit).  Here: a start that grows with the tile, blocks of K as in pick_tile, and for each further wave the longer of its products and
// its epilogue (3.9 us for 256 x 256).  On single SMs (gemm_sm100.cu, mode 0): 0.3 us a block of K whatever the tile, a little more once
// operands no longer stay in L2, a further wave of 128 x 256 tiles 2.9 us for its epilogue.  The choice by them is more than 5% off the
// better one at 8 of these sizes, 8.5% at most.
float pair_us(int T, int cols, int blocks) {
  const int bt = pick_tile(T, cols, blocks), pairs = std::max(sm_count() / 2, 1);
  const float share = bt / 256.f, slice = std::max(0.34f * share, 0.14f + 0.11f * share);
  const long long waves = (static_cast<long long>((T + bt - 1) / bt) * cols + pairs - 1) / pairs;
  return 5.1f + 2.6f * share + slice * blocks + (waves - 1) * std::max(3.85f * share, 2.1f * share + 0.95f * slice * blocks);
}
float single_us(int T, int N, int blocks, int bn) {
  const long long waves = (static_cast<long long>((T + 127) / 128) * ((N + bn - 1) / bn) + sm_count() - 1) / sm_count();
  if (bn == 256) return 5.9f + 0.329f * blocks + 0.04f * std::max(blocks - 64, 0) + (waves - 1) * std::max(2.9f, 1.3f + 0.378f * blocks);
  return 4.9f + 0.302f * blocks + (waves - 1) * std::max(1.45f, 0.65f + 0.302f * blocks);
}

}  // namespace

// Pairs are the better choice for most sizes (2500 x 2048 -> 2048 35 -> 27 us, 8192 x 4096 -> 10240 528 -> 441), but not where K is short,
// so that a tile is mostly epilogue (8192 x 64 -> 28672: 141 us on single SMs, 189 here; 4096 x 512 -> 4096 20.8 / 24.3), nor where the tiles
// of single SMs fill one wave as well and theirs are half as large (1000 x 2048 -> 4096: 17.4 / 19.0; 300 x 1536 -> 10240: 14.5 / 16.5).
// Fewer than 64 columns for many tokens, which read the tokens and do little else, are outside the fit: 8192 x 4096 -> 8 23.8 / 32.4, but
// 4096 x 7168 -> 8 47.1 / 37.3.
bool gemm_pair_pays(int T, int N, int K, int single_bn) {
  if (K % BK) return false;
  if (N < 64 && T > 1024 && K <= 4096) return false;
  return pair_us(T, (N + 2 * kRows - 1) / (2 * kRows), K / BK) <= single_us(T, N, K / BK, single_bn);
}

int gemm_pair(const void* x, long long ldx, const void* w, const void* bias, void* out, int T, int N, int K, bool gated,
              const GemmGroups* groups, int bt, cudaStream_t stream) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if (K % BK || N % 8 || ldx % 8 || ldx < K || (gated && bias != nullptr) || bt < 0 || bt > 256 || bt % 32) return -kBadArgument;
  const int cols = gated ? kRows : 2 * kRows;
  Params p{};
  p.out = static_cast<__nv_bfloat16*>(out);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.status = device_status();
  p.T = T;
  p.N = N;
  p.blocks = K / BK;
  p.tiles_w = (N + cols - 1) / cols;
  long long items;
  if (groups != nullptr) {
    if (bt == 0 || groups->offsets == nullptr || groups->tile_group == nullptr || groups->tile_row0 == nullptr ||
        groups->num_tiles == nullptr)
      return -kBadArgument;
    p.group_offsets = groups->offsets;
    p.tile_group = groups->tile_group;
    p.tile_row0 = groups->tile_row0;
    p.num_token_tiles = groups->num_tiles;
    items = (static_cast<long long>(T) / bt + groups->count) * p.tiles_w;          // (an upper bound)
  } else {
    if (bt == 0) bt = pick_tile(T, p.tiles_w, p.blocks);
    p.tiles_t = (T + bt - 1) / bt;
    // bands of 8 token tiles keep a wave's operands in L2 where x as a whole does not stay there
    p.band = static_cast<long long>(T) * K * 2 > (48ll << 20) ? 8 : p.tiles_t;
    items = static_cast<long long>(p.tiles_t) * p.tiles_w;
  }
  if (items > (1ll << 30)) return -kBadArgument;
  p.bt = bt;
  const uint64_t halves = gated ? 2 : 1;
  const uint64_t w_rows = static_cast<uint64_t>(N) * halves * (groups != nullptr ? groups->count : 1);
  const uint64_t row = static_cast<uint64_t>(K) * 2, block = BK * 2;
  CUtensorMap mw, mx;
  {
    // gate and up rows lie N rows apart: a dimension of their own, so that one copy brings 64 of each
    const uint64_t dims[4] = {BK, w_rows - (gated ? N : 0), halves, static_cast<uint64_t>(p.blocks)}, strides[3] = {row, row * N, block};
    const uint32_t box[4] = {BK, static_cast<uint32_t>(kRows / halves), static_cast<uint32_t>(halves), kBlocks};
    if (!encode_tmap_blocks(&mw, w, 4, dims, strides, box)) return -100;
  }
  {
    const uint64_t dims[3] = {BK, static_cast<uint64_t>(T), static_cast<uint64_t>(p.blocks)};
    const uint64_t strides[2] = {static_cast<uint64_t>(ldx) * 2, block};
    const uint32_t box[3] = {BK, static_cast<uint32_t>(bt / 2), kBlocks};
    if (!encode_tmap_blocks(&mx, x, 3, dims, strides, box)) return -101;
  }
  const cudaError_t e = gated ? launch<true>(mw, mx, p, items, stream) : launch<false>(mw, mx, p, items, stream);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

}  // namespace sglb

extern "C" {

// out[T, N] = x[T, K] (rows ldx apart) . w^T + bias; `gated`: w [2 N, K] = gate rows, then up rows, out = silu(gate) * up.  bf16, N and
// ldx whole 16-byte units, K of 128-byte ones, 16-byte aligned.  bt: tokens of a tile, a multiple of 32 up to 256 (0: chosen here).
int sglb_gemm_pair(const void* x, long long ldx, const void* w, const void* bias, void* out, int T, int N, int K, int gated, int bt,
                   cudaStream_t stream) {
  return sglb::gemm_pair(x, ldx, w, bias, out, T, N, K, gated != 0, nullptr, bt, stream);
}

// The same for rows sorted by group: w [groups, N (2 N), K]; the list of token tiles holds tiles of at most `bt` rows.
int sglb_gemm_pair_grouped(const void* x, const void* w, void* out, const int* group_offsets, const int* tile_group, const int* tile_row0,
                           const int* num_token_tiles, int rows, int N, int K, int groups, int gated, int bt, cudaStream_t stream) {
  const sglb::GemmGroups g{group_offsets, tile_group, tile_row0, num_token_tiles, groups};
  return sglb::gemm_pair(x, K, w, nullptr, out, rows, N, K, gated != 0, &g, bt, stream);
}

}  // extern "C"
