// Mixture-of-experts routing and token (un)permutation.
//
//   router_logits  fp32 logits of bf16 tokens and weights on the tensor cores, summed like an fp32 product
//   topk_route     scores = softmax | sigmoid | tanh (fp32) of router logits; optional selection bias
//                  (choose by score + bias, weigh by the unbiased score); optional group-limited
//                  routing (group score = max, or sum of the top 2 when biased; keep `topk_group`
//                  groups); top-k by repeated argmax (ties -> lowest index); optional renormalise;
//                  times `routed_scaling_factor`.
//                  Semantics: python/sgl_jax/srt/layers/gate.py:59-333 and
//                  python/sgl_jax/srt/kernels/{biased_topk,grouped_topk}/v1/kernel.py.
//   moe_align      counts the (token, k) pairs routed to this rank's experts, builds the expert
//                  row offsets, the pair -> sorted-row map and the list of token tiles the grouped
//                  GEMM walks.
//   moe_gather     x_sorted[row] = x[token of row]
//   moe_combine    out[t] = sum_j weight[t, j] * y_sorted[row(t, j)]   (fixed j order: deterministic)
//                  = the unpermute + weighted sum of python/sgl_jax/srt/layers/moe.py:684-760.
#include <float.h>

#include "common.cuh"

namespace sglb {
namespace {

constexpr int kMaxExperts = 512;
constexpr int kMaxTopK = 16;

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Logits of 16 * MT tokens x 8 * NT experts by a CTA.  Its eight warps take every eighth run of 32 lanes of K; products of bf16 are
// exact in fp32, the tensor core adds 32 of them at a time from zero, and all further sums are rounded fp32 additions in a fixed
// order (runs, then warps).  Operands come straight from L2, 16 bytes a load: the order of K inside a run is the same
// permutation for both.  Bound by load latency in decode, by L2 in prefill.  Two casts and an fp32 GEMM on the CUDA cores did this
// before, casting the weights on every call: 25 us at 64 tokens x 128 experts x 2048, 82 us at 4096 tokens.
constexpr int kRouterWarps = 8;

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int MT, int NT>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_logits_kernel(float* __restrict__ out, const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w,
                     const __nv_bfloat16* __restrict__ bias, int T, int E, int K) {
  extern __shared__ float part[];                             // [warp][16 * MT][8 * NT]
  constexpr int kM = 16 * MT, kN = 8 * NT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int t0 = blockIdx.x * kM, e0 = blockIdx.y * kN;
  pdl_wait();
  const __nv_bfloat16 *xa[MT][2], *wb[NT];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) xa[m][h] = x + min(t0 + 16 * m + 8 * h + g, T - 1) * ldx + 8 * t4;
#pragma unroll
  for (int n = 0; n < NT; ++n) wb[n] = w + static_cast<size_t>(min(e0 + 8 * n + g, E - 1)) * K + 8 * t4;
  float sum[MT][NT][4] = {};
  constexpr int kRuns = MT == 1 ? 4 : 1;                     // runs whose loads are in flight together
  for (int k0 = 32 * warp; k0 < K; k0 += 32 * kRouterWarps * kRuns) {
    uint4 a[kRuns][MT][2], b[kRuns][NT];
#pragma unroll
    for (int r = 0; r < kRuns; ++r) {
      const int k = k0 + 32 * kRouterWarps * r;
      const bool in = k < K;                                  // (zeros add nothing)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) a[r][m][h] = in ? __ldg(reinterpret_cast<const uint4*>(xa[m][h] + k)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int n = 0; n < NT; ++n) b[r][n] = in ? __ldg(reinterpret_cast<const uint4*>(wb[n] + k)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int r = 0; r < kRuns; ++r)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          mma_bf16(c, a[r][m][0].x, a[r][m][1].x, a[r][m][0].y, a[r][m][1].y, b[r][n].x, b[r][n].y);
          mma_bf16(c, a[r][m][0].z, a[r][m][1].z, a[r][m][0].w, a[r][m][1].w, b[r][n].z, b[r][n].w);
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[m][n][i] += c[i];
        }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        part[(warp * kM + 16 * m + g + 8 * (i >> 1)) * kN + 8 * n + 2 * t4 + (i & 1)] = sum[m][n][i];
  __syncthreads();
  for (int i = threadIdx.x; i < kM * kN; i += kRouterWarps * 32) {
    const int t = t0 + i / kN, e = e0 + i % kN;
    if (t >= T || e >= E) continue;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < kRouterWarps; ++q) v += part[q * kM * kN + i];
    if (bias != nullptr) v += __bfloat162float(bias[e]);
    out[static_cast<size_t>(t) * E + e] = v;
  }
}

// one warp per token; scores live in shared memory (E floats per warp)
template <typename T>
__global__ void topk_route_kernel(const T* __restrict__ logits, const float* __restrict__ bias,
                                  float* __restrict__ out_w, int* __restrict__ out_ids, int Tn, int E, int k,
                                  int scoring, int renorm, int num_groups, int topk_group, float scale) {
  extern __shared__ float smem[];
  const int warps = blockDim.x >> 5;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * warps + wid;
  if (t >= Tn) return;
  pdl_wait();
  float* sc = smem + wid * 2 * E;     // unbiased scores
  float* ch = sc + E;                 // selection scores (biased / group-masked)
  const T* row = logits + static_cast<size_t>(t) * E;
  // ---- scores
  float mx = -FLT_MAX;
  for (int e = lane; e < E; e += 32) mx = fmaxf(mx, to_f(row[e]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
  for (int e = lane; e < E; e += 32) {
    const float x = to_f(row[e]);
    float s;
    if (scoring == 0) s = __expf(x - mx);
    else if (scoring == 1) s = 1.f / (1.f + __expf(-x));
    else s = tanhf(x);
    sc[e] = s;
    sum += s;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  __syncwarp();
  for (int e = lane; e < E; e += 32) {
    if (scoring == 0) sc[e] = sc[e] / sum;
    ch[e] = sc[e] + (bias != nullptr ? bias[e] : 0.f);
  }
  __syncwarp();
  // ---- group-limited routing
  if (num_groups > 1) {
    const int gs = E / num_groups;
    float gscore = -FLT_MAX;
    if (lane < num_groups) {
      float m1 = -FLT_MAX, m2 = -FLT_MAX;
      for (int i = 0; i < gs; ++i) {
        const float v = ch[lane * gs + i];
        if (v > m1) {
          m2 = m1;
          m1 = v;
        } else if (v > m2) {
          m2 = v;
        }
      }
      gscore = bias != nullptr ? m1 + m2 : m1;
    }
    // keep the topk_group best groups: a group survives if fewer than topk_group groups beat it
    int beaten = 0;
    for (int g = 0; g < num_groups; ++g) {
      const float og = __shfl_sync(0xffffffffu, gscore, g);
      if (og > gscore || (og == gscore && g < lane)) ++beaten;
    }
    const bool keep = lane < num_groups && beaten < topk_group;
    const unsigned keep_mask = __ballot_sync(0xffffffffu, keep);
    for (int e = lane; e < E; e += 32)
      if (!((keep_mask >> (e / gs)) & 1u)) ch[e] = -FLT_MAX;
    __syncwarp();
  }
  // ---- top-k by repeated argmax
  float wsum = 0.f;
  float my_w = 0.f;
  int my_id = 0;
  for (int j = 0; j < k; ++j) {
    float best = -FLT_MAX;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = ch[e];
      if (v > best || (v == best && e < bi)) {
        best = v;
        bi = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if (bi == 0x7fffffff) bi = 0;
    const float w = sc[bi];
    wsum += w;
    if (lane == j) {
      my_w = w;
      my_id = bi;
    }
    __syncwarp();
    if (lane == 0) ch[bi] = -FLT_MAX;
    __syncwarp();
  }
  if (lane < k) {
    float w = my_w;
    if (renorm) w = w / fmaxf(wsum, 1e-20f);
    out_w[static_cast<size_t>(t) * k + lane] = w * scale;
    out_ids[static_cast<size_t>(t) * k + lane] = my_id;
  }
}

// One cluster.  pairs = T * k.  Experts [e0, e0 + E_local) are local.
//   offsets[E_local + 1], pair_row[pairs] (sorted row or -1), row_token[rows_cap] (token of each
//   sorted row), tile lists for the prefill-shaped grouped GEMM (tiles of at most `tile_rows` rows), counts[0] = number of
//   local rows, counts[1] = number of token tiles.
// Every CTA counts its share of the pairs in shared memory, reads the others' counts there and places its pairs behind those of the
// CTAs before it.  Bound by the shared-memory atomics of prefill (one CTA took 50 us for 32768 pairs; eight share them) and by
// latency in decode, where offsets and tiles come out of one scan instead of a loop over the experts in one thread (10 us for 64).
constexpr int kAlignThreads = 1024;
constexpr int kAlignCluster = 8;

__device__ __forceinline__ void align_cluster_sync(int ctas) {
  if (ctas > 1) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kAlignThreads)
moe_align_kernel(const int* __restrict__ topk_ids, int pairs, int k, int e0, int E_local, int tile_rows,
                 int* __restrict__ offsets, int* __restrict__ pair_row, int* __restrict__ row_token,
                 int* __restrict__ tile_group, int* __restrict__ tile_row0, int* __restrict__ counts,
                 int* __restrict__ expert_hist /* [E_local] optional, accumulates */) {
  __shared__ int cnt[kMaxExperts];             // pairs of this CTA's share, read by the others
  __shared__ int next[kMaxExperts];            // next row of this CTA's pairs
  __shared__ int warp_sum[2][kAlignThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ctas = gridDim.x, rank = blockIdx.x;
  const int share = (pairs + ctas - 1) / ctas, lo = rank * share, hi = min(pairs, lo + share);
  for (int e = tid; e < E_local; e += kAlignThreads) cnt[e] = 0;
  __syncthreads();
  pdl_wait();
  for (int i = lo + tid; i < hi; i += kAlignThreads) {
    const int e = topk_ids[i] - e0;
    if (e >= 0 && e < E_local) atomicAdd(&cnt[e], 1);
  }
  align_cluster_sync(ctas);
  // thread e: rows of expert e, those of the CTAs before this one; then rows and tiles of the experts before e (kMaxExperts threads
  // at most have one)
  int total = 0, before = 0;
  if (tid < E_local) {
    if (ctas == 1) {
      total = cnt[tid];
    } else {
      const uint32_t mine = smem_u32(&cnt[tid]);
      for (int r = 0; r < ctas; ++r) {
        uint32_t at;
        int v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(r));
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
        total += v;
        if (r < rank) before += v;
      }
    }
  }
  const int tiles = (total + tile_rows - 1) / tile_rows;
  int row_scan = total, tile_scan = tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, row_scan, o), b = __shfl_up_sync(0xffffffffu, tile_scan, o);
    if (lane >= o) {
      row_scan += a;
      tile_scan += b;
    }
  }
  if (lane == 31) {
    warp_sum[0][warp] = row_scan;
    warp_sum[1][warp] = tile_scan;
  }
  __syncthreads();
  int row0 = row_scan - total, tile0 = tile_scan - tiles;
  if (tid < kMaxExperts)
    for (int w = 0; w < warp; ++w) {
      row0 += warp_sum[0][w];
      tile0 += warp_sum[1][w];
    }
  if (tid < E_local) {
    next[tid] = row0 + before;
    if (rank == 0) {
      offsets[tid] = row0;
      for (int i = 0; i < tiles; ++i) {
        tile_group[tile0 + i] = tid;
        tile_row0[tile0 + i] = row0 + i * tile_rows;
      }
      if (expert_hist != nullptr) expert_hist[tid] += total;
      if (tid == E_local - 1) {
        offsets[E_local] = row0 + total;
        counts[0] = row0 + total;
        counts[1] = tile0 + tiles;
      }
    }
  }
  __syncthreads();
  // Row order inside an expert is whatever the atomics produce; every sorted row is computed
  // independently of its neighbours and the combine step sums in (token, j) order, so results do
  // not depend on it.
  for (int i = lo + tid; i < hi; i += kAlignThreads) {
    const int e = topk_ids[i] - e0;
    if (e >= 0 && e < E_local) {
      const int row = atomicAdd(&next[e], 1);
      pair_row[i] = row;
      row_token[row] = i / k;
    } else {
      pair_row[i] = -1;
    }
  }
  if (ctas > 1) align_cluster_sync(ctas);      // (the others may still read cnt)
}

__global__ void moe_gather_kernel(__nv_bfloat16* __restrict__ x_sorted, const __nv_bfloat16* __restrict__ x,
                                  const int* __restrict__ row_token, const int* __restrict__ counts, int H) {
  const int row = blockIdx.x;
  pdl_wait();
  if (row >= counts[0]) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row_token[row]) * H);
  uint4* dst = reinterpret_cast<uint4*>(x_sorted + static_cast<size_t>(row) * H);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) dst[i] = src[i];
}

// out[t] (+)= sum_j w[t, j] * y[pair_row[t*k + j]]; pairs routed elsewhere contribute nothing.  A thread sums 8 columns of a token; its
// rows come eight at a time, all in flight together (one after another: 10 us for 96 tokens of 2048 columns, now 3).
constexpr int kCombineThreads = 128, kCombineRows = 8;

__global__ void __launch_bounds__(kCombineThreads)
moe_combine_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ y,
                   const float* __restrict__ w, const int* __restrict__ pair_row, int k, int H,
                   const __nv_bfloat16* __restrict__ add /* optional [T, H] (shared expert) */) {
  const size_t t = blockIdx.x;
  const int i = blockIdx.y * kCombineThreads + threadIdx.x;
  pdl_wait();
  if (i >= (H >> 3)) return;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  auto unpack = [](const uint4& v, float (&f)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 p = __bfloat1622float2(h[e]);
      f[2 * e] = p.x;
      f[2 * e + 1] = p.y;
    }
  };
  if (add != nullptr) unpack(reinterpret_cast<const uint4*>(add + t * H)[i], acc);
  for (int j0 = 0; j0 < k; j0 += kCombineRows) {
    int row[kCombineRows];
    float wj[kCombineRows];
    uint4 v[kCombineRows];
#pragma unroll
    for (int j = 0; j < kCombineRows; ++j) {
      const bool in = j0 + j < k;
      row[j] = in ? pair_row[t * k + j0 + j] : -1;
      wj[j] = in ? w[t * k + j0 + j] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kCombineRows; ++j)
      if (row[j] >= 0) v[j] = reinterpret_cast<const uint4*>(y + static_cast<size_t>(row[j]) * H)[i];
#pragma unroll
    for (int j = 0; j < kCombineRows; ++j) {
      if (row[j] < 0) continue;
      float f[8];
      unpack(v[j], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += wj[j] * f[e];
    }
  }
  reinterpret_cast<uint4*>(out + t * H)[i] =
      make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
}

template <int MT, int NT>
cudaError_t launch_router(float* out, const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, const __nv_bfloat16* bias, int T, int E,
                          int K, cudaStream_t s) {
  constexpr int smem = kRouterWarps * 16 * MT * 8 * NT * 4;
  static const cudaError_t configured =
      cudaFuncSetAttribute(router_logits_kernel<MT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (configured != cudaSuccess) return configured;
  return launch_pdl(router_logits_kernel<MT, NT>, dim3((T + 16 * MT - 1) / (16 * MT), (E + 8 * NT - 1) / (8 * NT)),
                    dim3(kRouterWarps * 32), smem, s, out, x, ldx, w, bias, T, E, K);
}

}  // namespace
}  // namespace sglb

extern "C" {

// out fp32 [T, E] = x [T, K] (bf16, rows ldx apart) . w [E, K]^T + bias [E] (bf16 or null), fp32 arithmetic.  K a multiple of 32, ldx of
// 8; x and w 16-byte aligned.
int sglb_router_logits(float* out, const void* x, long long ldx, const void* w, const void* bias, int T, int E, int K, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (E < 1 || K < 32 || K % 32 != 0 || ldx % 8 != 0 || ldx < K || reinterpret_cast<uintptr_t>(x) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(w) % 16 != 0)
    return -kBadArgument;
  auto* xx = static_cast<const __nv_bfloat16*>(x);
  auto* ww = static_cast<const __nv_bfloat16*>(w);
  auto* bb = static_cast<const __nv_bfloat16*>(bias);
  // few tokens: small tiles, so that many SMs share the loads; many: 64 x 32, which reads the operands from L2 four times less often
  return static_cast<int>(T <= 512 ? launch_router<1, 2>(out, xx, ldx, ww, bb, T, E, K, s)
                                   : launch_router<4, 4>(out, xx, ldx, ww, bb, T, E, K, s));
}

// scoring: 0 softmax, 1 sigmoid, 2 tanh.  logits fp32 (dtype_bytes 4) or bf16 (2).  bias fp32 or null.
int sglb_topk_route(const void* logits, int dtype_bytes, const float* bias, float* out_w, int* out_ids, int T, int E,
                    int k, int scoring, int renorm, int num_groups, int topk_group, float scale, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (E > kMaxExperts || k > kMaxTopK || k > 32 || k > E || (num_groups > 1 && (E % num_groups || num_groups > 32)))
    return -kBadArgument;
  const int warps = 4;
  const int blocks = (T + warps - 1) / warps;
  const size_t smem = warps * 2 * E * sizeof(float);
  if (dtype_bytes == 4)
    launch_pdl(topk_route_kernel<float>, dim3(blocks), dim3(warps * 32), smem, s, static_cast<const float*>(logits), bias, out_w,
               out_ids, T, E, k, scoring, renorm, num_groups, topk_group, scale);
  else
    launch_pdl(topk_route_kernel<__nv_bfloat16>, dim3(blocks), dim3(warps * 32), smem, s, static_cast<const __nv_bfloat16*>(logits),
               bias, out_w, out_ids, T, E, k, scoring, renorm, num_groups, topk_group, scale);
  return static_cast<int>(cudaGetLastError());
}

int sglb_moe_align(const int* topk_ids, int pairs, int k, int e0, int E_local, int tile_rows, int* offsets, int* pair_row,
                   int* row_token, int* tile_group, int* tile_row0, int* counts, int* expert_hist, cudaStream_t s) {
  using namespace sglb;
  if (E_local > kMaxExperts || E_local < 1 || tile_rows < 1) return -kBadArgument;
  // up to four pairs a thread one CTA does as well: no barriers across SMs
  const int ctas = pairs <= 4 * kAlignThreads ? 1 : kAlignCluster;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kAlignThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, moe_align_kernel, topk_ids, pairs, k, e0, E_local, tile_rows, offsets, pair_row,
                                             row_token, tile_group, tile_row0, counts, expert_hist));
}

int sglb_moe_gather(void* x_sorted, const void* x, const int* row_token, const int* counts, int max_rows, int H,
                    cudaStream_t s) {
  using namespace sglb;
  if (max_rows <= 0) return 0;
  if (H % 8) return -kBadArgument;
  launch_pdl(moe_gather_kernel, dim3(max_rows), dim3(128), 0, s, static_cast<__nv_bfloat16*>(x_sorted),
             static_cast<const __nv_bfloat16*>(x), row_token, counts, H);
  return static_cast<int>(cudaGetLastError());
}

int sglb_moe_combine(void* out, const void* y, const float* w, const int* pair_row, int T, int k, int H,
                     const void* add, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (H % 8) return -kBadArgument;
  launch_pdl(moe_combine_kernel, dim3(T, (H / 8 + kCombineThreads - 1) / kCombineThreads), dim3(kCombineThreads), 0, s,
             static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(y), w, pair_row, k, H,
             static_cast<const __nv_bfloat16*>(add));
  return static_cast<int>(cudaGetLastError());
}
}
