// Bandwidth-bound ops of the decoder layer: RMSNorm (+ fused residual add), SiLU-gate,
// embedding gather, greedy argmax, and the fused per-head q/k RMSNorm + RoPE + paged KV write.
// All are single-pass, 16-byte vectorised and keep their statistics in fp32
// (reference semantics: python/sgl_jax/srt/layers/layernorm.py:30-253,
//  python/sgl_jax/srt/layers/embeddings.py:539-601, python/sgl_jax/srt/kernels/update_kv_cache/).
#include <float.h>

#include "common.cuh"

namespace sglb {
namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  const float r = red[0];
  __syncthreads();
  return r;
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

// One CTA per row.  H % 8 == 0.  With ADD: residual <- x + residual (bf16), y <- norm(residual).
// Row data is kept in registers between the two passes (H <= 8 * 8 * blockDim).
template <bool ADD, int VPT>
__global__ void rmsnorm_kernel(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x,
                               __nv_bfloat16* __restrict__ residual, const __nv_bfloat16* __restrict__ w, int H,
                               float eps, int gemma) {
  __shared__ float red[32];
  pdl_wait();
  const size_t row = blockIdx.x;
  const uint4* xv = reinterpret_cast<const uint4*>(x + row * H);
  uint4* rv = ADD ? reinterpret_cast<uint4*>(residual + row * H) : nullptr;
  const uint4* wv = reinterpret_cast<const uint4*>(w);
  uint4* yv = reinterpret_cast<uint4*>(y + row * H);
  const int nvec = H >> 3;
  float vals[VPT][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = threadIdx.x + i * blockDim.x;
    if (idx < nvec) {
      unpack8(xv[idx], vals[i]);
      if (ADD) {
        float r[8];
        unpack8(rv[idx], r);
#pragma unroll
        for (int e = 0; e < 8; ++e) vals[i][e] += r[e];
        const uint4 packed = pack8(vals[i]);
        rv[idx] = packed;
        unpack8(packed, vals[i]);   // normalise the rounded sum, as the unfused sequence would
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += vals[i][e] * vals[i][e];
    }
  }
  const float tot = block_sum(ss, red);
  const float inv = rsqrtf(tot / H + eps);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = threadIdx.x + i * blockDim.x;
    if (idx < nvec) {
      float wf[8], o[8];
      unpack8(wv[idx], wf);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = vals[i][e] * inv * (gemma ? wf[e] + 1.f : wf[e]);
      yv[idx] = pack8(o);
    }
  }
}

// out[t, i] = silu(x[t, i]) * x[t, I + i]
__global__ void silu_mul_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ x, long long T,
                                int I) {
  pdl_wait();
  const int nvec = I >> 3;
  const long long total = T * nvec;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = idx / nvec;
    const int v = static_cast<int>(idx - t * nvec);
    const uint4* row = reinterpret_cast<const uint4*>(x + t * 2 * I);
    float a[8], b[8], o[8];
    unpack8(row[v], a);
    unpack8(row[nvec + v], b);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = a[e] / (1.f + __expf(-a[e])) * b[e];
    reinterpret_cast<uint4*>(out + t * I)[v] = pack8(o);
  }
}

// out[t] = table[ids[t] - vocab_start] (zeros when outside this shard and `masked`)
__global__ void embedding_kernel(__nv_bfloat16* __restrict__ out, const int* __restrict__ ids,
                                 const __nv_bfloat16* __restrict__ table, int H, int rows, int vocab_start,
                                 int masked) {
  pdl_wait();
  const size_t t = blockIdx.x;
  int id = ids[t] - vocab_start;
  const bool ok = id >= 0 && id < rows;
  if (!ok) id = 0;
  const uint4* src = reinterpret_cast<const uint4*>(table + static_cast<size_t>(id) * H);
  uint4* dst = reinterpret_cast<uint4*>(out + t * H);
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) dst[i] = (ok || !masked) ? src[i] : z;
}

// first maximal index per row
template <typename T>
__global__ void argmax_kernel(int* __restrict__ out, const T* __restrict__ logits, int V, long long row_stride) {
  pdl_wait();
  __shared__ float sv[32];
  __shared__ int si[32];
  const T* row = logits + blockIdx.x * row_stride;
  float best = -FLT_MAX;
  int bi = 0x7fffffff;
  int scalar_from = 0;
  if constexpr (sizeof(T) == 2) {
    // 16-byte loads, four in flight per thread, when the row starts on a 16-byte boundary
    if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
      const int nvec = V / 8;
      const uint4* rv = reinterpret_cast<const uint4*>(row);
      constexpr int U = 4;
      for (int base = threadIdx.x; base < nvec; base += blockDim.x * U) {
        uint4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int idx = base + u * blockDim.x;
          q[u] = idx < nvec ? __ldg(rv + idx) : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int idx = base + u * blockDim.x;
          const uint32_t w[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float v = __uint_as_float((e & 1) ? (w[e >> 1] & 0xffff0000u) : (w[e >> 1] << 16));
            const int i = idx * 8 + e;
            if (v > best || (v == best && i < bi)) {
              best = v;
              bi = i;
            }
          }
        }
      }
      scalar_from = nvec * 8;
    }
  }
  for (int i = scalar_from + threadIdx.x; i < V; i += blockDim.x) {
    float v;
    if constexpr (sizeof(T) == 2) v = __bfloat162float(row[i]);
    else v = row[i];
    if (v > best || (v == best && i < bi)) {
      best = v;
      bi = i;
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
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sv[w] = best;
    si[w] = bi;
  }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    best = l < nw ? sv[l] : -FLT_MAX;
    bi = l < nw ? si[l] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if (l == 0) out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
  }
}

#ifdef SGLB_BOUNDS_CHECK
// Checked build only: the extent of the KV buffers and where to report, set by sglb_debug_set_kv_pages().
__device__ int g_dbg_kv_pages = 0;
__device__ Status* g_dbg_status = nullptr;
#endif

// Every (token, head) of a step's queries, keys and values:
//   q heads: optional RMSNorm over the head, RoPE, -> q_out[t, h, :]
//   k heads: optional RMSNorm, RoPE, -> cache[page, 0, h, off, :]
//   v heads: -> cache[page, 1, h, off, :]
struct RopeParams {
  __nv_bfloat16* q_out;
  const __nv_bfloat16 *q, *k, *v;            // head h of token t at q + t * q_ts + h * q_hs, k + t * k_ts + h * D, v likewise
  long long q_ts, k_ts, v_ts;
  int q_hs;
  const int* positions;
  const float* cos_sin;                      // [position][cos | sin], rd / 2 each; null: no rotation
  const __nv_bfloat16 *q_w, *k_w;            // norm weights (+ w_add) or null
  float w_add, eps;
  int Hq, Hkv, rd;
  __nv_bfloat16* kv;
  const int* loc;
  int page_size;
};

// D / 8 lanes hold a head, 16 bytes each; lane u of the first half of the rotary part turns with lane u + rd / 16.  A CTA takes a token (or a
// share of its heads where tokens are few), its threads as many heads at a time as divide them well; where one pass holds the heads of several
// tokens it takes `tokens` of them.  A thread keeps its cosines, sines and norm weights for all heads that it takes.  Bound by memory in prefill, by
// latency in decode.  With 2-byte accesses and a position's row read again for every head / with one token a CTA of 256 threads whatever its
// heads / now, us: 8192 tokens of 64 + 2 x 8 normed heads 173 / 105 / 103, 16 + 2 x 4 of them half rotated 46 / 52 / 40, 8 + 2 of 64 lanes 14 / 23 /
// 9.6, 1 + 2 6.8 / 24 / 6.7; 16 tokens of 8 + 2 2.0 / 2.3 / 1.9, of 40 + 2 x 8 2.4 / 2.4 / 2.0.
constexpr int kRopeThreads = 256;

template <int D>
__global__ void __launch_bounds__(kRopeThreads)
rope_qknorm_kvwrite_kernel(const RopeParams p, int T, int tokens) {
  constexpr int L = D / 8;
  const int u = threadIdx.x % L, lane = threadIdx.x & 31, slot = threadIdx.x / L, slots = blockDim.x / L;
  const int heads = p.Hq + 2 * p.Hkv, half = p.rd / 16;          // vectors in a half
  const int place = tokens > 1 ? slot / heads : 0, t_own = blockIdx.x * tokens + place;
  const bool live = place < tokens && t_own < T;
  const int t = live ? t_own : 0;
  int h = tokens > 1 ? slot - place * heads : blockIdx.y * slots + slot;
  const int step = gridDim.y * slots, passes = tokens > 1 ? 1 : (heads - static_cast<int>(blockIdx.y) * slots + step - 1) / step;
  pdl_wait();
  auto load = [&](int head) {
    if (!live || head >= heads) return make_uint4(0, 0, 0, 0);
    const __nv_bfloat16* src = head < p.Hq ? p.q + t * p.q_ts + static_cast<long long>(head) * p.q_hs
                               : head < p.Hq + p.Hkv ? p.k + t * p.k_ts + static_cast<long long>(head - p.Hq) * D
                                                     : p.v + t * p.v_ts + static_cast<long long>(head - p.Hq - p.Hkv) * D;
    return reinterpret_cast<const uint4*>(src)[u];
  };
  uint4 raw = load(h);                         // (on its way while the position's row is looked up)
  const bool first = u < half, turns = p.cos_sin != nullptr && u < 2 * half;
  const int partner = lane - u + (first ? u + half : u - half);
  float c[8], sn[8];
  if (turns) {
    const float* cs = p.cos_sin + static_cast<long long>(p.positions[t]) * p.rd + 8 * (first ? u : u - half);
#pragma unroll
    for (int e = 0; e < 8; e += 4) {
      const float4 a = *reinterpret_cast<const float4*>(cs + e), b = *reinterpret_cast<const float4*>(cs + p.rd / 2 + e);
      c[e] = a.x, c[e + 1] = a.y, c[e + 2] = a.z, c[e + 3] = a.w;
      sn[e] = b.x, sn[e + 1] = b.y, sn[e + 2] = b.z, sn[e + 3] = b.w;
    }
  }
  uint4 wq = make_uint4(0, 0, 0, 0), wk = wq;
  if (p.q_w != nullptr) wq = reinterpret_cast<const uint4*>(p.q_w)[u];
  if (p.k_w != nullptr) wk = reinterpret_cast<const uint4*>(p.k_w)[u];
  long long slot_at = -1;
  if (p.kv != nullptr) {
    const int at = p.loc[t];
    const int page = at / p.page_size, off = at - page * p.page_size;
    if (at >= 0) slot_at = (static_cast<long long>(page) * 2 * p.Hkv * p.page_size + off) * D;
#ifdef SGLB_BOUNDS_CHECK
    if (g_dbg_kv_pages > 0 && (at < 0 || page >= g_dbg_kv_pages)) {
      if (u == 0 && h == 0) report(g_dbg_status, kOutOfBounds, t, at);
      slot_at = -1;
    }
#endif
  }
  // (all lanes of a warp stay in the loop together: they exchange values)
  for (int i = 0; i < passes; ++i, h += step) {
    if (i > 0) raw = load(h);
    const bool is_q = h < p.Hq, is_k = !is_q && h < p.Hq + p.Hkv, in = live && h < heads;
    const bool norm = is_q ? p.q_w != nullptr : is_k && p.k_w != nullptr;
    if (p.q_w != nullptr || p.k_w != nullptr) {
      float v[8], w[8], ss = 0.f;
      unpack8(raw, v);
      unpack8(is_q ? wq : wk, w);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float inv = rsqrtf(ss / D + p.eps);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = v[e] * inv * (w[e] + p.w_add);
      if (norm) raw = pack8(v);                // rounded like the norm on its own, before the rotation
    }
    if (p.cos_sin != nullptr) {
      const uint4 other = make_uint4(__shfl_sync(0xffffffffu, raw.x, partner), __shfl_sync(0xffffffffu, raw.y, partner),
                                     __shfl_sync(0xffffffffu, raw.z, partner), __shfl_sync(0xffffffffu, raw.w, partner));
      if (turns && (is_q || is_k)) {
        float v[8], o[8];
        unpack8(raw, v);
        unpack8(other, o);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = v[e] * c[e] + o[e] * (first ? -sn[e] : sn[e]);
        raw = pack8(v);
      }
    }
    if (!in) continue;
    if (is_q) {
      reinterpret_cast<uint4*>(p.q_out + (static_cast<long long>(t) * p.Hq + h) * D)[u] = raw;
    } else if (slot_at >= 0) {
      const long long head = static_cast<long long>(h - p.Hq) * p.page_size * D;      // (values behind the keys)
      reinterpret_cast<uint4*>(p.kv + slot_at + head)[u] = raw;
    }
  }
}

// The same for rotations of neighbouring lanes: one warp per (token, head), lane l holds elements l, l + 32, l + 64, ...
template <int D>
__global__ void rope_pairs_kernel(const RopeParams p, long long T) {
  pdl_wait();
  constexpr int E = D / 32;
  const int heads = p.Hq + 2 * p.Hkv;
  const long long wid = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  if (wid >= T * heads) return;
  const int lane = threadIdx.x & 31;
  const long long t = wid / heads;
  const int h = static_cast<int>(wid - t * heads);
  const bool is_q = h < p.Hq;
  const bool is_k = !is_q && h < p.Hq + p.Hkv;
  const int hh = is_k ? h - p.Hq : h - p.Hq - p.Hkv;
  const __nv_bfloat16* src = is_q ? p.q + t * p.q_ts + static_cast<long long>(h) * p.q_hs
                                  : (is_k ? p.k + t * p.k_ts : p.v + t * p.v_ts) + static_cast<long long>(hh) * D;
  float v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = __bfloat162float(src[lane + 32 * j]);
  if (is_q || is_k) {
    const __nv_bfloat16* nw = is_q ? p.q_w : p.k_w;
    if (nw != nullptr) {
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < E; ++j) ss += v[j] * v[j];
      ss = warp_sum(ss);
      const float inv = rsqrtf(ss / D + p.eps);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        // round to bf16 like the unfused norm would before the rotation
        v[j] = __bfloat162float(__float2bfloat16(v[j] * inv * (__bfloat162float(nw[lane + 32 * j]) + p.w_add)));
      }
    }
    const float* cs = p.cos_sin + static_cast<long long>(p.positions[t]) * p.rd;
    const int half = p.rd >> 1;
    // pairs (2i, 2i + 1): the partner sits in the neighbouring lane
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const int i = lane + 32 * j;
      const float other = __shfl_xor_sync(0xffffffffu, v[j], 1);
      if (i < p.rd) {
        const float c = cs[i >> 1], s = cs[half + (i >> 1)];
        v[j] = (i & 1) ? (v[j] * c + other * s) : (v[j] * c - other * s);
      }
    }
  }
  __nv_bfloat16* dst;
  if (is_q) {
    dst = p.q_out + (t * p.Hq + h) * D;
  } else {
    if (p.kv == nullptr) return;
    const int slot = p.loc[t];
    const int page = slot / p.page_size, off = slot - page * p.page_size;
#ifdef SGLB_BOUNDS_CHECK
    if (g_dbg_kv_pages > 0 && (slot < 0 || page >= g_dbg_kv_pages)) {
      if (lane == 0) report(g_dbg_status, kOutOfBounds, static_cast<int>(t), slot);
      return;
    }
#endif
    if (slot < 0) return;
    dst = p.kv + ((((static_cast<long long>(page) * 2 + (is_k ? 0 : 1)) * p.Hkv + hh) * p.page_size) + off) * D;
  }
#pragma unroll
  for (int j = 0; j < E; ++j) dst[lane + 32 * j] = __float2bfloat16(v[j]);
}

template <int D>
cudaError_t launch_rope(const RopeParams& p, long long T, bool pairs, cudaStream_t s) {
  const int heads = p.Hq + 2 * p.Hkv;
  if (pairs) {
    const long long blocks = (T * heads * 32 + 127) / 128;
    return launch_pdl(rope_pairs_kernel<D>, dim3(blocks), dim3(128), 0, s, p, T);
  }
  constexpr int kMost = kRopeThreads / (D / 8), kWarp = 32 / (D / 8);            // heads of a CTA at a time; of a warp
  const long long want = 4ll * sm_count();                                       // CTAs to have at least, if there is work for them
  auto threads = [](int h) { return dim3((h + kWarp - 1) / kWarp * 32); };
  if (heads <= kMost) {
    const long long most = kMost / heads, some = T / want;
    const int tokens = static_cast<int>(some < 1 ? 1 : some < most ? some : most);
    return launch_pdl(rope_qknorm_kvwrite_kernel<D>, dim3(static_cast<unsigned>((T + tokens - 1) / tokens)), threads(tokens * heads), 0, s, p,
                      static_cast<int>(T), tokens);
  }
  // few tokens: a token's passes go to several CTAs
  const int passes = (heads + kMost - 1) / kMost;
  const long long shares = (want + T - 1) / T;
  return launch_pdl(rope_qknorm_kvwrite_kernel<D>, dim3(static_cast<unsigned>(T), static_cast<unsigned>(shares < passes ? shares : passes)),
                    threads((heads + passes - 1) / passes), 0, s, p, static_cast<int>(T), 1);
}

// page_table[rows[i], pos[i]] = ids[i]
__global__ void page_table_scatter_kernel(int* __restrict__ table, int max_pages, const int* __restrict__ rows,
                                          const int* __restrict__ pos, const int* __restrict__ ids, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) table[static_cast<long long>(rows[i]) * max_pages + pos[i]] = ids[i];
}

// ids < 0 are placeholders -slot: replace from the future-token map (overlap scheduling)
__global__ void resolve_future_kernel(int* __restrict__ ids, const int* __restrict__ future_map, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const int v = ids[i];
    if (v < 0) ids[i] = future_map[-v];
  }
}

}  // namespace
}  // namespace sglb

extern "C" {

int sglb_rmsnorm(void* y, const void* x, const void* w, long long T, int H, float eps, int gemma, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (H % 8 || H > 8 * 8 * 1024) return -kBadArgument;
  const int nvec = H / 8;
  int threads = ((nvec + 31) / 32) * 32;
  if (threads > 1024) threads = 1024;
  int vpt = 1;
  while (vpt * threads < nvec) vpt *= 2;
  auto* yy = static_cast<__nv_bfloat16*>(y);
  auto* xx = static_cast<const __nv_bfloat16*>(x);
  auto* ww = static_cast<const __nv_bfloat16*>(w);
  switch (vpt) {
    case 1: launch_pdl(rmsnorm_kernel<false, 1>, dim3(T), dim3(threads), 0, s, yy, xx, nullptr, ww, H, eps, gemma); break;
    case 2: launch_pdl(rmsnorm_kernel<false, 2>, dim3(T), dim3(threads), 0, s, yy, xx, nullptr, ww, H, eps, gemma); break;
    case 4: launch_pdl(rmsnorm_kernel<false, 4>, dim3(T), dim3(threads), 0, s, yy, xx, nullptr, ww, H, eps, gemma); break;
    default: launch_pdl(rmsnorm_kernel<false, 8>, dim3(T), dim3(threads), 0, s, yy, xx, nullptr, ww, H, eps, gemma); break;
  }
  return static_cast<int>(cudaGetLastError());
}

int sglb_fused_add_rmsnorm(void* y, const void* x, void* residual, const void* w, long long T, int H, float eps,
                           int gemma, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (H % 8 || H > 8 * 8 * 1024) return -kBadArgument;
  const int nvec = H / 8;
  int threads = ((nvec + 31) / 32) * 32;
  if (threads > 1024) threads = 1024;
  int vpt = 1;
  while (vpt * threads < nvec) vpt *= 2;
  auto* yy = static_cast<__nv_bfloat16*>(y);
  auto* xx = static_cast<const __nv_bfloat16*>(x);
  auto* rr = static_cast<__nv_bfloat16*>(residual);
  auto* ww = static_cast<const __nv_bfloat16*>(w);
  switch (vpt) {
    case 1: launch_pdl(rmsnorm_kernel<true, 1>, dim3(T), dim3(threads), 0, s, yy, xx, rr, ww, H, eps, gemma); break;
    case 2: launch_pdl(rmsnorm_kernel<true, 2>, dim3(T), dim3(threads), 0, s, yy, xx, rr, ww, H, eps, gemma); break;
    case 4: launch_pdl(rmsnorm_kernel<true, 4>, dim3(T), dim3(threads), 0, s, yy, xx, rr, ww, H, eps, gemma); break;
    default: launch_pdl(rmsnorm_kernel<true, 8>, dim3(T), dim3(threads), 0, s, yy, xx, rr, ww, H, eps, gemma); break;
  }
  return static_cast<int>(cudaGetLastError());
}

int sglb_silu_and_mul(void* out, const void* x, long long T, int I, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (I % 8) return -kBadArgument;
  const long long total = T * (I / 8);
  const int threads = 256;
  long long blocks = (total + threads - 1) / threads;
  if (blocks > 148LL * 16) blocks = 148LL * 16;
  launch_pdl(silu_mul_kernel, dim3(static_cast<int>(blocks)), dim3(threads), 0, s, static_cast<__nv_bfloat16*>(out),
                                                               static_cast<const __nv_bfloat16*>(x), T, I);
  return static_cast<int>(cudaGetLastError());
}

int sglb_embedding(void* out, const int* ids, const void* table, long long T, int H, int rows, int vocab_start,
                   int masked, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (H % 8) return -kBadArgument;
  int threads = H / 8 < 256 ? ((H / 8 + 31) / 32) * 32 : 256;
  launch_pdl(embedding_kernel, dim3(T), dim3(threads), 0, s, static_cast<__nv_bfloat16*>(out), ids,
                                         static_cast<const __nv_bfloat16*>(table), H, rows, vocab_start, masked);
  return static_cast<int>(cudaGetLastError());
}

// dtype_bytes: 4 = fp32 logits, 2 = bf16 logits
int sglb_argmax(int* out, const void* logits, int B, int V, long long row_stride, int dtype_bytes, cudaStream_t s) {
  using namespace sglb;
  if (B <= 0) return 0;
  if (dtype_bytes == 4) launch_pdl(argmax_kernel<float>, dim3(B), dim3(1024), 0, s, out, static_cast<const float*>(logits), V, row_stride);
  else launch_pdl(argmax_kernel<__nv_bfloat16>, dim3(B), dim3(1024), 0, s, out, static_cast<const __nv_bfloat16*>(logits), V, row_stride);
  return static_cast<int>(cudaGetLastError());
}

// Checked build (-DSGLB_BOUNDS_CHECK): tell the KV-write kernel how many pages the KV buffers have; a slot outside
// them is then reported through the status word (code kOutOfBounds, aux = token row, slot) and its store skipped.
// Returns 1 when the library was built with the checks, 0 otherwise (the call is then a no-op).
int sglb_debug_set_kv_pages(int pages) {
#ifdef SGLB_BOUNDS_CHECK
  sglb::Status* st = sglb::device_status();
  if (cudaMemcpyToSymbol(sglb::g_dbg_kv_pages, &pages, sizeof(int)) != cudaSuccess) return -sglb::kBadArgument;
  if (cudaMemcpyToSymbol(sglb::g_dbg_status, &st, sizeof(st)) != cudaSuccess) return -sglb::kBadArgument;
  return 1;
#else
  (void)pages;
  return 0;
#endif
}

// q: head h of token t at q + t * q_ts + h * q_hs; k, v: at k + t * k_ts + h * D, v + t * v_ts + h * D (all 16-byte units).  q_out
// [T, Hq, D]; kv_buffer [pages, 2, Hkv, page_size, D] or null, loc the slots (< 0: not written).  Norm weights [D] (+ w_add) or null.
// cos_sin fp32 [positions, rotary_dim] or null; is_neox: lane i turns with lane i + rotary_dim / 2 (rotary_dim a multiple of 16), else
// neighbours turn.
int sglb_rope_qknorm_kvwrite(void* q_out, const void* q, long long q_ts, int q_hs, const void* k, long long k_ts, const void* v,
                             long long v_ts, const int* positions, const float* cos_sin, const void* q_w, const void* k_w, float w_add,
                             float eps, long long T, int Hq, int Hkv, int D, int rotary_dim, void* kv_buffer, const int* loc,
                             int page_size, int is_neox, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  auto off = [](const void* a) { return reinterpret_cast<uintptr_t>(a) % 16 != 0; };
  if (off(q) || off(k) || off(v) || off(q_out) || off(kv_buffer) || off(q_w) || off(k_w) || off(cos_sin) || q_ts % 8 || q_hs % 8 ||
      k_ts % 8 || v_ts % 8 || T > 0x7fffffffll)
    return -kBadArgument;
  if (cos_sin != nullptr && (rotary_dim > D || rotary_dim % (is_neox ? 16 : 2) != 0)) return -kBadArgument;
  RopeParams p{};
  p.q_out = static_cast<__nv_bfloat16*>(q_out);
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.q_ts = q_ts;
  p.k_ts = k_ts;
  p.v_ts = v_ts;
  p.q_hs = q_hs;
  p.positions = positions;
  p.cos_sin = cos_sin;
  p.q_w = static_cast<const __nv_bfloat16*>(q_w);
  p.k_w = static_cast<const __nv_bfloat16*>(k_w);
  p.w_add = w_add;
  p.eps = eps;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.rd = cos_sin != nullptr ? rotary_dim : 0;
  p.kv = static_cast<__nv_bfloat16*>(kv_buffer);
  p.loc = loc;
  p.page_size = page_size;
  const bool pairs = !is_neox && cos_sin != nullptr;
  switch (D) {
    case 64: return static_cast<int>(launch_rope<64>(p, T, pairs, s));
    case 128: return static_cast<int>(launch_rope<128>(p, T, pairs, s));
    case 256: return static_cast<int>(launch_rope<256>(p, T, pairs, s));
    default: return -kBadArgument;
  }
}

int sglb_page_table_scatter(int* table, int max_pages, const int* rows, const int* pos, const int* ids, int n,
                            cudaStream_t s) {
  if (n <= 0) return 0;
  sglb::page_table_scatter_kernel<<<(n + 255) / 256, 256, 0, s>>>(table, max_pages, rows, pos, ids, n);
  return static_cast<int>(cudaGetLastError());
}

int sglb_resolve_future(int* ids, const int* future_map, int n, cudaStream_t s) {
  if (n <= 0) return 0;
  sglb::resolve_future_kernel<<<(n + 255) / 256, 256, 0, s>>>(ids, future_map, n);
  return static_cast<int>(cudaGetLastError());
}
}
