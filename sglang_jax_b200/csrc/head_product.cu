// Per-head products around the absorbed latent attention (queries into the latent space, its results out of it):
//   out[t, h, n] = sum_k x[t, h, k] w[h, n, k]      bf16 operands, fp32 sums throughout, rounded once
//
// Partial sums never leave fp32, whatever the sizes (a library may add up the pieces of a split product in the type of its result).
// Operands are read where they lie: heads of a token and heads of the weights by strides.
//
//   head_product_few_kernel    decode: 16 tokens x 16 columns of a head a CTA, its warps share K; bound by latency
//   head_product_tile_kernel   more tokens or heads: tiles through a ring in shared memory (cp.async), one tile a CTA; a tile has two to
//                              eight stages, so that it is bound by their latency in a short pipeline, then by L2
//
// 16 heads, 128 -> 512 and 512 -> 128 lanes, weights from DRAM as in a step: 7 tokens 2.5 and 3.0 us, 96 tokens 3.5 and 4.9; a batched library
// product in bf16, whose sums may be split and added up in bf16, 3.5 and 3.8, 3.8 and 4.1; fp32 products on the CUDA cores (weights in L2) 17
// and 20 at 96 tokens.
#include "common.cuh"
#include "mma_sync.cuh"

namespace sglb {
namespace {

struct HeadProductParams {
  const __nv_bfloat16 *x, *w;
  __nv_bfloat16* out;            // [T, H, N]
  long long x_ts, w_hs;          // elements between tokens of x, heads of w
  int x_hs, w_ld;                // between heads of x, rows of w
  int T, H, N, K;
  __device__ __forceinline__ const __nv_bfloat16* x_row(int t, int h) const {      // (rows past the end: the last one again)
    return x + min(t, T - 1) * x_ts + static_cast<long long>(h) * x_hs;
  }
  __device__ __forceinline__ const __nv_bfloat16* w_row(int n, int h) const {
    return w + h * w_hs + static_cast<long long>(min(n, N - 1)) * w_ld;
  }
  __device__ __forceinline__ void store(int t, int h, int n, float v0, float v1) const {      // (N is a multiple of 8: pairs are whole)
    if (t < T && n < N)
      *reinterpret_cast<uint32_t*>(out + (static_cast<long long>(t) * H + h) * N + n) = pack_bf16(v0, v1);
  }
};

constexpr int kFewCols = 16;

// Operands come straight from memory, 16 bytes a load: inside a run of 32 lanes of K both have the same permutation.  A warp has RUNS runs
// in flight, all of K in one go for what is usual (4 warps x 1 run of 128 lanes, 8 x 2 of 512).
template <int WARPS, int RUNS>
__global__ void __launch_bounds__(32 * WARPS)
head_product_few_kernel(const HeadProductParams p) {
  __shared__ float part[WARPS][16][kFewCols];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int t0 = blockIdx.x * 16, n0 = blockIdx.y * kFewCols, h = blockIdx.z;
  pdl_wait();
  const __nv_bfloat16 *xa[2], *wb[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    xa[i] = p.x_row(t0 + 8 * i + g, h) + 8 * t4;
    wb[i] = p.w_row(n0 + 8 * i + g, h) + 8 * t4;
  }
  float c[2][4] = {};
  for (int k0 = 32 * warp; k0 < p.K; k0 += 32 * WARPS * RUNS) {
    uint4 a[RUNS][2], b[RUNS][2];
#pragma unroll
    for (int r = 0; r < RUNS; ++r) {
      const int k = k0 + 32 * WARPS * r;
      const bool in = k + 8 * t4 < p.K;                       // (K is whole groups of 8 lanes; zeros add nothing)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[r][i] = in ? *reinterpret_cast<const uint4*>(xa[i] + k) : make_uint4(0, 0, 0, 0);
        b[r][i] = in ? *reinterpret_cast<const uint4*>(wb[i] + k) : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int r = 0; r < RUNS; ++r) {
      const uint32_t lo[4] = {a[r][0].x, a[r][1].x, a[r][0].y, a[r][1].y}, hi[4] = {a[r][0].z, a[r][1].z, a[r][0].w, a[r][1].w};
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        mma16816(c[n], lo, b[r][n].x, b[r][n].y);
        mma16816(c[n], hi, b[r][n].z, b[r][n].w);
      }
    }
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) part[warp][g + 8 * (i >> 1)][8 * n + 2 * t4 + (i & 1)] = c[n][i];
  __syncthreads();
  if (threadIdx.x >= 16 * kFewCols / 2) return;
  const int t = threadIdx.x / (kFewCols / 2), n = threadIdx.x % (kFewCols / 2) * 2;
  float v0 = 0.f, v1 = 0.f;
#pragma unroll
  for (int q = 0; q < WARPS; ++q) {
    v0 += part[q][t][n];
    v1 += part[q][t][n + 1];
  }
  p.store(t0 + t, h, n0 + n, v0, v1);
}

// byte offset of (row, 16-byte chunk) inside a [rows][64 bf16] block, chunks swizzled so that eight rows lie in different banks
__device__ __forceinline__ uint32_t chunk_at(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool in) {       // 16 bytes, or zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// BM tokens x BN columns of one head, 64 lanes of K a stage, STAGES of the ring; WM x WN warps.
template <int BM, int BN, int WM, int WN, int STAGES>
__global__ void __launch_bounds__(32 * WM * WN)
head_product_tile_kernel(const HeadProductParams p) {
  constexpr int kThreads = 32 * WM * WN, kStage = (BM + BN) * 128, MT = BM / WM / 16, NT = BN / WN / 16;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp / WN * (BM / WM), wn = warp % WN * (BN / WN);
  const int t0 = blockIdx.x * BM, n0 = blockIdx.y * BN, h = blockIdx.z, blocks = (p.K + 63) / 64;
  pdl_wait();
  auto load = [&](int kb) {
    if (kb < blocks) {
      const uint32_t st = base + kb % STAGES * kStage;
#pragma unroll
      for (int i = threadIdx.x; i < (BM + BN) * 8; i += kThreads) {
        const int row = i >> 3, k = kb * 64 + (i & 7) * 8;
        const __nv_bfloat16* src = row < BM ? p.x_row(t0 + row, h) : p.w_row(n0 + row - BM, h);
        const bool in = k < p.K;
        copy16(st + chunk_at(row, i & 7), in ? src + k : src, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");      // (an empty one past the end: the count below stays right)
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load(s);
  float c[MT][NT][2][4] = {};
  for (int kb = 0; kb < blocks; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                          // the stage has landed; the one before it is read
    load(kb + STAGES - 1);
    const uint32_t sa = base + kb % STAGES * kStage, sb = sa + BM * 128;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[MT][4], b[NT][4];
#pragma unroll
      for (int m = 0; m < MT; ++m) ldsm_x4(sa + chunk_at(wm + 16 * m + (lane & 15), 2 * ks + (lane >> 4)), a[m]);
#pragma unroll
      for (int n = 0; n < NT; ++n)
        ldsm_x4(sb + chunk_at(wn + 16 * n + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1)), b[n]);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          mma16816(c[m][n][0], a[m], b[n][0], b[n][1]);
          mma16816(c[m][n][1], a[m], b[n][2], b[n][3]);
        }
    }
  }
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = t0 + wm + 16 * m + g, col = n0 + wn + 16 * n + 8 * j + 2 * t4;
        p.store(t, h, col, c[m][n][j][0], c[m][n][j][1]);
        p.store(t + 8, h, col, c[m][n][j][2], c[m][n][j][3]);
      }
}

template <int WARPS, int RUNS>
cudaError_t launch_few(const HeadProductParams& p, cudaStream_t s) {
  static_assert(32 * WARPS >= 16 * kFewCols / 2, "a thread for every pair of results");
  return launch_pdl(head_product_few_kernel<WARPS, RUNS>, dim3((p.T + 15) / 16, (p.N + kFewCols - 1) / kFewCols, p.H), dim3(32 * WARPS), 0, s,
                    p);
}

template <int BM, int BN, int WM, int WN, int STAGES>
cudaError_t launch_tile(const HeadProductParams& p, cudaStream_t s) {
  constexpr int smem = STAGES * (BM + BN) * 128;
  static const cudaError_t configured =
      cudaFuncSetAttribute(head_product_tile_kernel<BM, BN, WM, WN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (configured != cudaSuccess) return configured;
  return launch_pdl(head_product_tile_kernel<BM, BN, WM, WN, STAGES>, dim3((p.T + BM - 1) / BM, (p.N + BN - 1) / BN, p.H), dim3(32 * WM * WN), smem,
                    s, p);
}

}  // namespace
}  // namespace sglb

extern "C" {

// out [T, H, N] = x . w^T per head: head h of token t at x + t * x_ts + h * x_hs, row n of head h's weights at w + h * w_hs + n * w_ld.
// bf16; K, N and all strides whole 16-byte units, x and w 16-byte aligned.
int sglb_head_product(void* out, const void* x, long long x_ts, int x_hs, const void* w, long long w_hs, int w_ld, int T, int H, int N,
                      int K, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  auto whole = [](long long v) { return v % 8 == 0; };
  if (H < 1 || H > 65535 || N < 8 || K < 8 || !whole(N) || !whole(K) || !whole(x_ts) || !whole(x_hs) || !whole(w_hs) || !whole(w_ld) ||
      (N + kFewCols - 1) / kFewCols > 65535 || reinterpret_cast<uintptr_t>(x) % 16 != 0 || reinterpret_cast<uintptr_t>(w) % 16 != 0)
    return -kBadArgument;
  const HeadProductParams p{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(out),
                            x_ts, w_hs, x_hs, w_ld, T, H, N, K};
  auto ctas = [&](int m, int n) { return static_cast<long long>((T + m - 1) / m) * ((N + n - 1) / n) * H; };
  // (us for weights from DRAM, H heads x T tokens, 128 -> 512 lanes; then 512 -> 128)
  // The small CTAs up to about 900 threads an SM: 16 x 7 2.5 against 2.8 in tiles, 16 x 32 2.8 / 3.0, 16 x 64 4.0 / 3.2; 16 x 64 3.5 / 4.8,
  // 16 x 96 5.2 / 4.9, 128 x 7 6.3 / 5.9.  K up to 128 in four warps: 16 x 7 2.5, in eight 2.6; 512 in eight: 3.0, in four 4.4.
  // Large tiles where more than half of their rows are tokens and most SMs get one: 128 x 96 12.6 against 14.7, 16 x 256 4.7 / 6.4, 16 x 128
  // (64 tiles) 4.4 / 3.9; 128 x 128 10.9 / 14.7, 16 x 256 (32 tiles) 10.2 / 5.8.
  const long long few = ctas(16, kFewCols), sms = sm_count();
  if (K <= 128 && few <= 7 * sms) return static_cast<int>(launch_few<4, 1>(p, s));
  if (K > 128 && 2 * few <= 7 * sms) return static_cast<int>(launch_few<8, 2>(p, s));
  if (T > 64 && 8 * ctas(128, 128) >= 6 * sms) return static_cast<int>(launch_tile<128, 128, 4, 2, 3>(p, s));
  // the ring as deep as helps: 512 lanes 4.9 with five stages, 5.5 with three; 128 lanes (two stages) 3.5 with three, 3.5 with five
  return static_cast<int>(K > 192 ? launch_tile<32, 64, 1, 4, 5>(p, s) : launch_tile<32, 64, 1, 4, 3>(p, s));
}

}  // extern "C"
