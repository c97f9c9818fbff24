// Gated delta rule over ragged batches, prefill and decode alike, the recurrence entirely in fp32:
//
//   delta_prep    short causal convolution + SiLU of the q / k / v channels of a fused projection (window = this step's
//                 rows, then the request's stored window, then zeros), unit q (times dim^-1/2) and k vectors, write
//                 strength beta = sigmoid(b) and decay g = exp(-exp(A_log) softplus(a + dt_bias)), one per head or one
//                 per head and key channel (then the next two kernels compute it, the only readers of its input)
//   delta_chunk   prefill: what a chunk of 32 tokens contributes independently of the state in front of it
//   delta_scan    prefill: S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q   chunk by chunk as small matrix
//                 products; columns of S are independent, so a CTA owns 32 columns of one (sequence, head) and keeps
//                 them from the first token to the last.  The result depends on how a prompt is cut by rounding only
//   delta_step    decode: the same for one token per request, the state streaming through once
//                 The convolution windows and the optional checkpoint (state after `track` tokens, for prefix sharing)
//                 are written by the last two.
//   delta_gate    rmsnorm(o) * w * silu(gate) (or sigmoid(gate)) per head, in the projections' type
//
// Both state tensors belong to `RecurrentStatePool`: windows [slots, channels, taps - 1], states [slots, H, D, V].
// Compiled without fast-math substitutions.
#include <math.h>

#include "common.cuh"
#include "recurrent.cuh"

namespace sglb {
namespace {

// Columns of a projection's row.  Heads that share a q / k head are neighbours and form a group; the q and k channels of group g
// begin at column `q + g * qk_step` and `k + g * qk_step`, its value heads' channels at `v + g * v_step`, the inputs of its heads'
// beta and decay at `b + g * ba_step` and `a + g * ba_step`.  One run of q, then k, then v channels: steps of one head (of one
// group's value heads); the checkpoints that keep a group's q, k, v and gate rows together: steps of a whole group.
struct DeltaColumns {
  int q, k, qk_step, v, v_step, b, a, ba_step;
};

struct DeltaParams {
  const void* proj;              // [T, ld]: the q, k and v channels, where `cols` says
  long long ld;
  const void* ba;                // [T, ba_ld]: inputs of beta and decay, where `cols` says
  long long ba_ld;
  DeltaColumns cols;
  const void* conv_w;            // [channels, taps], channels = q | k | v
  const float* a_log;            // [H]
  const float* dt_bias;          // [H]; per channel: [H, D]
  const void* chan_a;            // [T, H, D] inputs of the decays per channel; null: one decay per head, from proj
  void* conv_state;              // [slots, channels, taps - 1]
  float* state;                  // [slots, H, D, V]
  const long long* slots;        // [B]
  const int* cu;                 // [B + 1] first row of every sequence; null: one row each
  const int* prefix;             // [B] tokens before this step (0: start from zero state); null: continue
  const int* track_len;          // [B] tokens after which the state is also stored in track_slot (0: never); may be null
  const int* track_slot;         // [B]
  float* qk;                     // [T, Hk, 2, D] unit q * D^-1/2 | unit k
  float* v;                      // [T, H, V]
  float* gb;                     // [T, H, 2] decay, beta
  float* coef;                   // [T / 32 + 2 B, H, kCoefs], see delta_chunk_kernel
  float* kq;                     // per channel: [T, H, 3, D], see delta_chunk_channel_kernel
  float* gc;                     // per channel: [T / 32 + 2 B, H, D] decay over a whole chunk
  float* o;                      // [T, H, V]
  int B, T, H, Hk, D, V, taps;
  int singles;                   // ragged step: how many sequences bring exactly one token (-1: not known)
};

// One warp per (run of RUN consecutive rows, head): the convolution window slides through registers.  A lane owns the
// channels lane, lane + 32, ... (NPL of them); TAPS >= taps, the kernel and the window are padded in front with zeros.
template <typename T, int NPL, int TAPS>
struct Conv {
  float w[NPL][TAPS], x[NPL][TAPS - 1];                // x[.][TAPS - 2] is the previous row

  __device__ __forceinline__ void load_kernel(const T* __restrict__ kernel, int c0, int width, int taps, int lane) {
#pragma unroll
    for (int i = 0; i < NPL; ++i)
#pragma unroll
      for (int j = 0; j < TAPS; ++j) {
        const int tap = j - (TAPS - taps), c = lane + 32 * i;
        w[i][j] = (tap >= 0 && c < width) ? to_f(kernel[static_cast<long long>(c0 + c) * taps + tap]) : 0.f;
      }
  }
  // window in front of row `start + local` of a sequence whose rows begin at `start`; the channels from c0 on are the columns
  // from `col` on
  __device__ __forceinline__ void load_window(const T* __restrict__ proj, long long ld, const T* __restrict__ stored,
                                              bool fresh, int start, int local, int col, int c0, int width, int taps, int lane) {
    const int win = taps - 1;
#pragma unroll
    for (int i = 0; i < NPL; ++i)
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) {
        const int c = lane + 32 * i, back = TAPS - 1 - j, r = local - back;
        float v = 0.f;
        if (c < width && back <= win) {
          if (r >= 0) v = to_f(proj[(start + r) * ld + col + c]);
          else if (!fresh) v = to_f(stored[static_cast<long long>(c0 + c) * win + win + r]);
        }
        x[i][j] = v;
      }
  }
  // SiLU of the convolution at the next row, whose inputs are `in`
  __device__ __forceinline__ void step(const float (&in)[NPL], float (&out)[NPL]) {
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      float acc = w[i][TAPS - 1] * in[i];
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) acc += w[i][j] * x[i][j];
#pragma unroll
      for (int j = 0; j < TAPS - 2; ++j) x[i][j] = x[i][j + 1];
      x[i][TAPS - 2] = in[i];
      out[i] = acc / (1.f + expf(-acc));
    }
  }
};

template <typename T, int NPL, int TAPS, int RUN>
__global__ void __launch_bounds__(128) delta_prep_kernel(const DeltaParams p) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int units = p.Hk + p.H;
  const long long wid = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const long long runs = (p.T + RUN - 1) / RUN;
  if (wid >= runs * units) return;
  const int run = static_cast<int>(wid / units), unit = static_cast<int>(wid - static_cast<long long>(run) * units);
  const int t0 = run * RUN, t1 = min(t0 + RUN, p.T);
  const int b0 = p.cu != nullptr ? sequence_of(p.cu, p.B, t0) : t0;
  const int channels = 2 * p.Hk * p.D + p.H * p.V, taps = p.taps, win = taps - 1;
  const T* __restrict__ proj = static_cast<const T*>(p.proj);
  const T* __restrict__ kernel = static_cast<const T*>(p.conv_w);
  const T* __restrict__ windows = static_cast<const T*>(p.conv_state);
  // calls fn(t) for every row, after reload(b, start, local) wherever a sequence begins (or the run does)
  auto walk = [&](auto&& reload, auto&& fn) {
    int b = b0, end = t0;
    for (int t = t0; t < t1; ++t) {
      if (t == end || t == t0) {
        int start = t;
        if (p.cu != nullptr) {
          while (b + 1 < p.B && p.cu[b + 1] <= t) ++b;
          start = p.cu[b];
          end = b + 1 < p.B ? p.cu[b + 1] : p.T;
        } else {
          b = t;
          end = t + 1;
        }
        reload(windows + static_cast<long long>(p.slots[b]) * channels * win, p.prefix != nullptr && p.prefix[b] == 0,
               start, t - start);
      }
      fn(t);
    }
  };
  auto rows = [&](int t, int c0, int width, float (&in)[NPL]) {
    const T* src = proj + t * p.ld + c0;
#pragma unroll
    for (int i = 0; i < NPL; ++i) in[i] = lane + 32 * i < width ? to_f(src[lane + 32 * i]) : 0.f;
  };
  if (unit < p.Hk) {
    const int q0 = unit * p.D, k0 = p.Hk * p.D + unit * p.D;             // channels, and the columns they are found in
    const int qc = p.cols.q + unit * p.cols.qk_step, kc = p.cols.k + unit * p.cols.qk_step;
    Conv<T, NPL, TAPS> cq, ck;
    cq.load_kernel(kernel, q0, p.D, taps, lane);
    ck.load_kernel(kernel, k0, p.D, taps, lane);
    const float scale = 1.f / sqrtf(static_cast<float>(p.D));
    float in_q[NPL], in_k[NPL];
    rows(t0, qc, p.D, in_q);
    rows(t0, kc, p.D, in_k);
    walk(
        [&](const T* stored, bool fresh, int start, int local) {
          cq.load_window(proj, p.ld, stored, fresh, start, local, qc, q0, p.D, taps, lane);
          ck.load_window(proj, p.ld, stored, fresh, start, local, kc, k0, p.D, taps, lane);
        },
        [&](int t) {
          float q[NPL], k[NPL];
          cq.step(in_q, q);
          ck.step(in_k, k);
          if (t + 1 < t1) {                            // the next row is on its way while this one is worked on
            rows(t + 1, qc, p.D, in_q);
            rows(t + 1, kc, p.D, in_k);
          }
          float qq = 0.f, kk = 0.f;
#pragma unroll
          for (int i = 0; i < NPL; ++i) {
            qq += q[i] * q[i];
            kk += k[i] * k[i];
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            qq += __shfl_xor_sync(0xffffffffu, qq, o);
            kk += __shfl_xor_sync(0xffffffffu, kk, o);
          }
          const float qs = scale / sqrtf(qq + 1e-6f), ks = 1.f / sqrtf(kk + 1e-6f);
          float* dst = p.qk + (static_cast<long long>(t) * p.Hk + unit) * 2 * p.D;
#pragma unroll
          for (int i = 0; i < NPL; ++i) {
            const int d = lane + 32 * i;
            if (d < p.D) {
              dst[d] = q[i] * qs;
              dst[p.D + d] = k[i] * ks;
            }
          }
        });
  } else {
    const int h = unit - p.Hk, r = p.H / p.Hk, hk = h / r;
    for (int vb = 0; vb < p.V; vb += 32 * NPL) {
      const int v0 = 2 * p.Hk * p.D + h * p.V + vb, width = min(32 * NPL, p.V - vb);
      const int vc = p.cols.v + hk * p.cols.v_step + (h - hk * r) * p.V + vb;
      Conv<T, NPL, TAPS> cv;
      cv.load_kernel(kernel, v0, width, taps, lane);
      float in[NPL];
      rows(t0, vc, width, in);
      walk(
          [&](const T* stored, bool fresh, int start, int local) {
            cv.load_window(proj, p.ld, stored, fresh, start, local, vc, v0, width, taps, lane);
          },
          [&](int t) {
            float v[NPL];
            cv.step(in, v);
            if (t + 1 < t1) rows(t + 1, vc, width, in);
            float* dst = p.v + (static_cast<long long>(t) * p.H + h) * p.V + vb;
#pragma unroll
            for (int i = 0; i < NPL; ++i)
              if (lane + 32 * i < width) dst[lane + 32 * i] = v[i];
          });
    }
    for (int t = t0 + lane; t < t1; t += 32) {
      const T* row = static_cast<const T*>(p.ba) + static_cast<long long>(t) * p.ba_ld + hk * p.cols.ba_step + (h - hk * r);
      float* gb = p.gb + (static_cast<long long>(t) * p.H + h) * 2;
      if (p.chan_a == nullptr) gb[0] = expf(-expf(p.a_log[h]) * softplus(to_f(row[p.cols.a]) + p.dt_bias[h]));
      gb[1] = 1.f / (1.f + expf(-to_f(row[p.cols.b])));
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Prefill works in chunks of kC tokens.  With S the state in front of a chunk, G_t the product of its decays up to and
// including t, and g_tj the product over j + 1 .. t, the recurrence unrolls to
//
//   u_t + sum_{j<t} beta_t g_tj (k_t . k_j) u_j = beta_t (v_t - G_t S^T k_t)
//   o_t = G_t S^T q_t + sum_{j<=t} g_tj (q_t . k_j) u_j          S <- G S + sum_j g_Cj k_j u_j^T
//
// delta_chunk solves the unit lower-triangular system once per (chunk, head), independently of the state, so that the
// sequential part (delta_scan) is matrix products only.  All in fp32; decays are products of decays, never quotients.
constexpr int kC = 32;
constexpr int kCoefRow = kC;                           // coefficient block of a (chunk, head):
constexpr int kCoefB = kC * kC;                        //   [0]      (I + A)^-1 diag(beta), rows t
constexpr int kCoefVec = 2 * kC * kC;                  //   [kCoefB] g_tj (q_t . k_j), rows t
constexpr int kCoefs = 2 * kC * kC + 2 * kC;           //   [kCoefVec] G_t | g_Cj

using Chunks = ChunksOf<kC>;
__host__ __device__ __forceinline__ int chunk_base(int start, int b) { return Chunks::base(start, b); }

// kC rows (of D floats, `tok` floats apart) into smem rows of `ld` floats; rows past m become zeros; below, those of the unit
// q (which = 0) or k (1) vectors.  Lanes past D
// of a row are left alone.
template <int THREADS>
__device__ __forceinline__ void stage_rows(float* dst, int ld, const float* src, long long tok, int D, int m) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < kC; r += THREADS / 32) {
    const bool in = r < m;
    const float* s = src + (in ? r : 0) * tok;
    if (D % 4 == 0)
      for (int e = lane * 4; e < D; e += 128) cp_async16(dst + r * ld + e, s + e, in ? 16 : 0);
    else
      for (int e = lane; e < D; e += 32) cp_async4(dst + r * ld + e, s + e, in ? 4 : 0);
  }
}

// Where chunk `idx` of the launch lies: sequence, first row, rows; none of them for places no sequence uses and for single
// tokens (delta_step).
struct ChunkPlace {
  int row0, m;
  __device__ __forceinline__ ChunkPlace(const DeltaParams& p, int idx) : row0(0), m(0) {
    int lo = 0, hi = p.B - 1;
    while (lo < hi) {                                  // last sequence whose chunks begin at or before idx
      const int mid = (lo + hi + 1) >> 1;
      if (chunk_base(p.cu[mid], mid) <= idx) lo = mid;
      else hi = mid - 1;
    }
    const int start = p.cu[lo];
    const Chunks ch(p.cu[lo + 1] - start, p.track_len != nullptr ? p.track_len[lo] : 0);
    const int ci = idx - chunk_base(start, lo);
    if (ch.n <= 1 || ci >= ch.count()) return;
    row0 = start + ch.first(ci);
    m = ch.len(ci);
  }
};

template <int THREADS>
__device__ __forceinline__ void stage_rows(float* dst, int ld, const DeltaParams& p, int row0, int hk, int which, int m) {
  const long long tok = static_cast<long long>(p.Hk) * 2 * p.D;
  stage_rows<THREADS>(dst, ld, p.qk + row0 * tok + (static_cast<long long>(hk) * 2 + which) * p.D, tok, p.D, m);
}

// One CTA per (chunk, q / k head): products of the chunk's vectors, then the coefficients of every value head that uses
// them (one warp per head).
constexpr int kChunkThreads = 128;
constexpr int kGramLd = kC + 4;

__global__ void __launch_bounds__(kChunkThreads) delta_chunk_kernel(const DeltaParams p, int Dp) {
  extern __shared__ float4 sm4[];
  float* rows = reinterpret_cast<float*>(sm4);         // [k 0..kC-1 | q 0..kC-1][ld]
  const int ld = Dp + 4;
  float* gram = rows + 2 * kC * ld;                    // [k . k | q . k][kC][kGramLd]
  float* line = gram + 2 * kC * kGramLd;               // [warp][kC]
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hk = blockIdx.y;
  const int idx = blockIdx.x;
  const ChunkPlace place(p, idx);
  if (place.m == 0) return;
  const int row0 = place.row0, m = place.m;
  for (int i = tid; i < 2 * kC * (ld - p.D); i += kChunkThreads) rows[(i / (ld - p.D)) * ld + p.D + i % (ld - p.D)] = 0.f;
  stage_rows<kChunkThreads>(rows, ld, p, row0, hk, 1, m);
  stage_rows<kChunkThreads>(rows + kC * ld, ld, p, row0, hk, 0, m);
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  {
    // 64 x 32 products, four rows by four columns per thread
    const int r0 = (tid >> 3) * 4, j0 = tid & 7;       // columns j0, j0 + 8, ...: neighbouring lanes, neighbouring rows
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int d = 0; d < Dp; d += 4) {
      float4 a[4], c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const float4*>(rows + (r0 + i) * ld + d);
        c[i] = *reinterpret_cast<const float4*>(rows + (j0 + 8 * i) * ld + d);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += a[i].x * c[j].x + a[i].y * c[j].y + a[i].z * c[j].z + a[i].w * c[j].w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) gram[(r0 + i) * kGramLd + j0 + 8 * j] = acc[i][j];
  }
  __syncthreads();
  const int r = p.H / p.Hk;
  for (int hh = warp; hh < r; hh += kChunkThreads / 32) {
    const int h = hk * r + hh;
    const float* gb = p.gb + (static_cast<long long>(row0 + lane) * p.H + h) * 2;
    const float g = lane < m ? gb[0] : 1.f, beta = lane < m ? gb[1] : 0.f;
    float* out = p.coef + (static_cast<long long>(idx) * p.H + h) * kCoefs;
    float* a = line + warp * kC;
    float from = 1.f, G = 1.f;                         // lane j: product of the decays j + 1 .. t; product up to t
    float X[kC];                                       // lane c: column c of (I + A)^-1
#pragma unroll
    for (int t = 0; t < kC; ++t) {
      const float gt = __shfl_sync(0xffffffffu, g, t), bt = __shfl_sync(0xffffffffu, beta, t);
      G *= gt;
      if (lane < t) from *= gt;
      __syncwarp();
      a[lane] = lane < t ? bt * from * gram[t * kGramLd + lane] : 0.f;
      out[kCoefB + t * kCoefRow + lane] = lane <= t ? from * gram[(kC + t) * kGramLd + lane] : 0.f;
      if (lane == t) out[kCoefVec + t] = G;
      __syncwarp();
      float x = lane == t ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < t; j += 4) {
        const float4 c = *reinterpret_cast<const float4*>(a + j);
        x -= c.x * X[j];
        if (j + 1 < t) x -= c.y * X[j + 1];
        if (j + 2 < t) x -= c.z * X[j + 2];
        if (j + 3 < t) x -= c.w * X[j + 3];
      }
      X[t] = x;
      out[t * kCoefRow + lane] = x * beta;
    }
    out[kCoefVec + kC + lane] = from;
  }
}

// The same with one decay per head and key channel, one CTA per (chunk, head).  The products need the decay between two
// tokens inside the sum over channels.  A block of tokens is halved down to blocks of four: between the halves the decay is
// split at the last token of the first half, so neither factor exceeds one, and the products are plain ones of scaled
// vectors; inside four tokens the decays are taken pair by pair.  Every exponent is a sum over just the tokens in between,
// never a difference of longer sums, so that strong decays earlier in the chunk do not cost precision.  Scaled vectors for
// delta_scan: k and q times the decay from the chunk's start (what meets the state in front of it), and k times the decay to
// its end (what it leaves behind).
constexpr int kChannelThreads = 256;

struct ChannelShape {
  static constexpr int kRows = 3 * kC + kC + kC / 2;   // k, q, logs of the decays; scaled k, scaled q of second halves
  static int smem(int Dp) { return (kRows * (Dp + 4) + 2 * kC * kGramLd + kC) * 4; }
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T>
__global__ void __launch_bounds__(kChannelThreads, 2) delta_chunk_channel_kernel(const DeltaParams p, int Dp) {
  extern __shared__ float4 sm4[];
  const int ld = Dp + 4;
  float* ks = reinterpret_cast<float*>(sm4);           // [kC][ld]
  float* qs = ks + kC * ld;                            // [kC][ld]
  float* cs = qs + kC * ld;                            // [kC][ld]  binary logarithms of the tokens' decays
  float* sk = cs + kC * ld;                            // [kC][ld]
  float* sq = sk + kC * ld;                            // [kC / 2][ld]
  float* gram = sq + kC / 2 * ld;                      // [beta k . k | q . k][kC][kGramLd]
  float* betas = gram + 2 * kC * kGramLd;              // [kC]
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, hk = h / (p.H / p.Hk), D = p.D;
  const int idx = blockIdx.x;
  const ChunkPlace place(p, idx);
  if (place.m == 0) return;
  const int row0 = place.row0, m = place.m;
  for (int i = tid; i < 3 * kC * (ld - D); i += kChannelThreads) ks[(i / (ld - D)) * ld + D + i % (ld - D)] = 0.f;
  stage_rows<kChannelThreads>(ks, ld, p, row0, hk, 1, m);
  stage_rows<kChannelThreads>(qs, ld, p, row0, hk, 0, m);
  cp_commit();
  if (tid < kC) betas[tid] = tid < m ? p.gb[(static_cast<long long>(row0 + tid) * p.H + h) * 2 + 1] : 0.f;
  // a channel's 32 tokens are shared by two threads, one for each half
  const int shift = 31 - __clz(Dp);
  const float rate = -1.4426950408889634f * expf(p.a_log[h]);
  for (int i = tid; i < 2 * Dp; i += kChannelThreads) {
    const int d = i & (Dp - 1), t0 = (i >> shift) * (kC / 2);
    if (d >= D) continue;
    const T* a = static_cast<const T*>(p.chan_a) + (static_cast<long long>(row0) * p.H + h) * D + d;
    const float bias = p.dt_bias[h * D + d];
#pragma unroll 1
    for (int t = t0; t < t0 + kC / 2; t += 8) {
      float in[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) in[e] = to_f(a[static_cast<long long>(min(t + e, m - 1)) * p.H * D]);
#pragma unroll
      for (int e = 0; e < 8; ++e) cs[(t + e) * ld + d] = t + e < m ? rate * softplus(in[e] + bias) : 0.f;
    }
  }
  for (int i = tid; i < 2 * kC * kGramLd; i += kChannelThreads) gram[i] = 0.f;
  cp_wait<0>();
  __syncthreads();
#pragma unroll
  for (int half = kC / 2; half >= 4; half >>= 1) {
    // scaled vectors: first halves backwards from their last token, second halves forwards from there
    for (int i = tid; i < 2 * Dp; i += kChannelThreads) {
      const int d = i & (Dp - 1), part = i >> shift;
#pragma unroll
      for (int j = 0; j < kC / 2 / half; ++j) {        // this thread's half blocks: every second one
        const int blk = j * 2 * half, t0 = blk + part * half;
        float c = 0.f;
        if (part == 0) {
#pragma unroll 8
          for (int t = t0 + half - 1; t >= t0; --t) {
            sk[t * ld + d] = ks[t * ld + d] * ex2_approx(c);
            c += cs[t * ld + d];
          }
        } else {
#pragma unroll 8
          for (int t = t0; t < t0 + half; ++t) {
            c += cs[t * ld + d];
            const float f = ex2_approx(c);
            sk[t * ld + d] = ks[t * ld + d] * f;
            sq[(t - half - blk / 2) * ld + d] = qs[t * ld + d] * f;
          }
        }
      }
    }
    __syncthreads();
    {
      // kC / 2 second-half rows times `half` columns of their first half, for k and q; neighbouring lanes share the
      // channels of one product
      const int parts = kC / 2 / half, part = tid & (parts - 1), item = tid / parts;
      const int j = item % half, r = item / half;                // r: place among the second-half rows
      const int blk = r / half * 2 * half, t = blk + half + r % half;
      const float *col = sk + (blk + j) * ld, *rk = sk + t * ld, *rq = sq + r * ld;
      float kk = 0.f, qk = 0.f;
#pragma unroll 4
      for (int d = 4 * part; d < Dp; d += 4 * parts) {
        const float4 c = *reinterpret_cast<const float4*>(col + d);
        const float4 a = *reinterpret_cast<const float4*>(rk + d), b = *reinterpret_cast<const float4*>(rq + d);
        kk += a.x * c.x + a.y * c.y + a.z * c.z + a.w * c.w;
        qk += b.x * c.x + b.y * c.y + b.z * c.z + b.w * c.w;
      }
#pragma unroll
      for (int o = parts / 2; o > 0; o >>= 1) {
        kk += __shfl_xor_sync(0xffffffffu, kk, o);
        qk += __shfl_xor_sync(0xffffffffu, qk, o);
      }
      if (part == 0) {
        gram[t * kGramLd + blk + j] = kk;
        gram[(kC + t) * kGramLd + blk + j] = qk;
      }
    }
    if (half > 4) __syncthreads();
  }
  {
    // blocks of four tokens: one warp each, lanes share the channels
    const int blk = warp * 4;
    float kk[6], qk[10];
#pragma unroll
    for (int i = 0; i < 6; ++i) kk[i] = 0.f;
#pragma unroll
    for (int i = 0; i < 10; ++i) qk[i] = 0.f;
    for (int d = lane; d < Dp; d += 32) {
      float k[4], q[4], c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        k[i] = ks[(blk + i) * ld + d];
        q[i] = qs[(blk + i) * ld + d];
        c[i] = cs[(blk + i) * ld + d];
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float e = 0.f;
#pragma unroll
        for (int j = t - 1; j >= 0; --j) {
          e += c[j + 1];
          const float f = ex2_approx(e) * k[j];
          kk[t * (t - 1) / 2 + j] += k[t] * f;
          qk[t * (t + 1) / 2 + j] += q[t] * f;
        }
        qk[t * (t + 1) / 2 + t] += q[t] * k[t];
      }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) kk[i] = warp_sum(kk[i]);
#pragma unroll
    for (int i = 0; i < 10; ++i) qk[i] = warp_sum(qk[i]);
    if (lane == 0)
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int j = 0; j <= t; ++j) {
          if (j < t) gram[(blk + t) * kGramLd + blk + j] = kk[t * (t - 1) / 2 + j];
          gram[(kC + blk + t) * kGramLd + blk + j] = qk[t * (t + 1) / 2 + j];
        }
  }
  __syncthreads();
  float* out = p.coef + (static_cast<long long>(idx) * p.H + h) * kCoefs;
  for (int i = tid; i < kC * kC; i += kChannelThreads) {
    const int t = i / kC, j = i % kC;
    out[kCoefB + i] = gram[(kC + t) * kGramLd + j];
    gram[t * kGramLd + j] *= betas[t];
  }
  __syncthreads();
  if (warp == 0) {
    const float beta = betas[lane];
    float X[kC];                                       // lane c: column c of (I + A)^-1
#pragma unroll
    for (int t = 0; t < kC; ++t) {
      float x[4] = {lane == t ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < t; j += 4) {
        const float4 c = *reinterpret_cast<const float4*>(gram + t * kGramLd + j);
        x[0] -= c.x * X[j];
        if (j + 1 < t) x[1] -= c.y * X[j + 1];
        if (j + 2 < t) x[2] -= c.z * X[j + 2];
        if (j + 3 < t) x[3] -= c.w * X[j + 3];
      }
      X[t] = (x[0] + x[1]) + (x[2] + x[3]);
      out[t * kCoefRow + lane] = X[t] * beta;
    }
  } else if (warp >= 4) {
    for (int d = tid - 128; d < D; d += 128) {
      float* dst = p.kq + (static_cast<long long>(row0) * p.H + h) * 3 * D + d;
      const long long tok = static_cast<long long>(p.H) * 3 * D;
      float c = 0.f, e = 0.f;                          // from the start up to t; behind t to the end
#pragma unroll 8
      for (int t = 0; t < m; ++t) {
        c += cs[t * ld + d];
        const float f = ex2_approx(c);
        dst[t * tok] = ks[t * ld + d] * f;
        dst[t * tok + D] = qs[t * ld + d] * f;
      }
#pragma unroll 8
      for (int t = m - 1; t >= 0; --t) {
        dst[t * tok + 2 * D] = ks[t * ld + d] * ex2_approx(e);
        e += cs[t * ld + d];
      }
      p.gc[(static_cast<long long>(idx) * p.H + h) * D + d] = ex2_approx(c);
    }
  }
}

// ---------------------------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kCols = 32;          // columns of the state per CTA

// Convolution windows of one head's channels after a step of n rows (the q / k channels are written by the first value
// head that uses them), and after its first `track` rows in the checkpoint's slot.
template <typename T>
__device__ __forceinline__ void write_windows(const DeltaParams& p, int b, int h, int start, int n, bool fresh, int track,
                                              int threads) {
  const int D = p.D, V = p.V, win = p.taps - 1, channels = 2 * p.Hk * D + p.H * V, hk = h / (p.H / p.Hk);
  const T* proj = static_cast<const T*>(p.proj) + start * p.ld;
  T* cs = static_cast<T*>(p.conv_state);
  T* own = cs + p.slots[b] * channels * win;
  auto window = [&](int c, int col) {
    T* keep = track > 0 && track <= n ? cs + (static_cast<long long>(p.track_slot[b]) * channels + c) * win : nullptr;
    advance_window(own + static_cast<long long>(c) * win, keep, proj + col, p.ld, win, n, fresh, track);
  };
  const int first = h - hk * (p.H / p.Hk);             // place of the head in its group
  for (int i = threadIdx.x; i < V; i += threads)
    window(2 * p.Hk * D + h * V + i, p.cols.v + hk * p.cols.v_step + first * V + i);
  if (first == 0)
    for (int i = threadIdx.x; i < D; i += threads) {
      window(hk * D + i, p.cols.q + hk * p.cols.qk_step + i);
      window(p.Hk * D + hk * D + i, p.cols.k + hk * p.cols.qk_step + i);
    }
}

// Prefill: one CTA per (sequence, head, 32 columns of the state).  Thread (rg, cp) of 16 x 16 owns RPT rows and the two
// columns 2 cp, 2 cp + 1 of the state (registers, mirrored in shared memory as the operand of the next chunk).  Per chunk:
//   Y = [K; Q] S                    rows 4 rg .. of the 64: warps 0-3 turn K S into the right-hand side, 4-7 keep G Q S
//   U = (I + A)^-1 diag(beta) (V - G K S)
//   O = G Q S + B U                 warps 4-7;         S <- G S + K^T diag(g_C) U   all warps
// With decays per channel (CHAN) the factors sit in three scaled copies of K and Q instead (delta_chunk_channel_kernel).
template <int RPT>
struct ScanShape {
  static constexpr int kDp = 16 * RPT, kLd = kDp + 4;
  static constexpr int kK = kC * kLd;                  // one buffer of k (two of them), and the one of q
  static constexpr int kCo = kC * kGramLd;             // T', B
  static constexpr int kFloats = 3 * kK + kC * kCols + 2 * kCo + 2 * 2 * kC + kDp * kCols + 2 * kC * kCols + kDp;
  static constexpr int kSmem = kFloats * 4;
};

template <typename T, int RPT, bool CHAN>
__global__ void __launch_bounds__(kScanThreads, RPT <= 8 ? 2 : 1) delta_scan_kernel(const DeltaParams p) {
  using Sh = ScanShape<RPT>;
  constexpr int ld = Sh::kLd;
  extern __shared__ float4 sm4[];
  float* ks = reinterpret_cast<float*>(sm4);           // [2][kC][ld]
  float* qs = ks + 2 * Sh::kK;                         // [kC][ld]
  float* vs = qs + Sh::kK;                             // [kC][kCols]
  float* ts = vs + kC * kCols;                         // [kC][kGramLd]  (I + A)^-1 diag(beta)
  float* bs = ts + Sh::kCo;                            // [kC][kGramLd]
  float* vec = bs + Sh::kCo;                           // [2][G_t | g_Cj]
  float* ss = vec + 4 * kC;                            // [kDp][kCols]
  float* us = ss + Sh::kDp * kCols;                    // [kC][kCols]
  float* rs = us + kC * kCols;                         // [kC][kCols]    right-hand side, then diag(g_C) U
  float* gcs = rs + kC * kCols;                        // [kDp]          CHAN: decays over the chunk
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cp = (lane & 15) * 2, rg = warp * 2 + (lane >> 4);
  const int b = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * kCols, hk = h / (p.H / p.Hk);
  const int start = p.cu[b], n = p.cu[b + 1] - start, D = p.D, V = p.V;
  if (n <= 1) return;                                  // single tokens: delta_step
  const bool fresh = p.prefix[b] == 0;
  const int track = p.track_len != nullptr ? p.track_len[b] : 0;
  const Chunks ch(n, track);
  const int nch = ch.count();
  const long long plane = static_cast<long long>(D) * V;
  float* st = p.state + (p.slots[b] * p.H + h) * plane;
  const float* coef = p.coef + (static_cast<long long>(chunk_base(start, b)) * p.H + h) * kCoefs;

  float S[RPT][2];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = rg * RPT + i;
#pragma unroll
    for (int c = 0; c < 2; ++c)
      S[i][c] = (!fresh && r < D && c0 + cp + c < V) ? st[static_cast<long long>(r) * V + c0 + cp + c] : 0.f;
    *reinterpret_cast<float2*>(ss + r * kCols + cp) = make_float2(S[i][0], S[i][1]);
  }
  auto store = [&](float* dst) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = rg * RPT + i;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (r < D && c0 + cp + c < V) dst[static_cast<long long>(r) * V + c0 + cp + c] = S[i][c];
    }
  };
  for (int i = tid; i < 3 * kC * (ld - D); i += kScanThreads) ks[(i / (ld - D)) * ld + D + i % (ld - D)] = 0.f;

  if (CHAN)
    for (int i = tid; i < Sh::kDp - D; i += kScanThreads) gcs[D + i] = 0.f;
  auto scaled = [&](float* dst, int ci, int which) {   // CHAN: one of the three copies of chunk ci
    const long long tok = static_cast<long long>(p.H) * 3 * D;
    stage_rows<kScanThreads>(dst, ld, p.kq + (start + ch.first(ci)) * tok + (static_cast<long long>(h) * 3 + which) * D, tok,
                             D, ch.len(ci));
  };

  auto stage_tokens = [&](int ci) {                    // k, q, v and the decays of chunk ci
    const int row0 = start + ch.first(ci), m = ch.len(ci);
    if constexpr (CHAN) {
      scaled(ks, ci, 0);
      scaled(qs, ci, 1);
    } else {
      stage_rows<kScanThreads>(ks + (ci & 1) * Sh::kK, ld, p, row0, hk, 1, m);
      stage_rows<kScanThreads>(qs, ld, p, row0, hk, 0, m);
    }
    for (int i = tid; i < kC * kCols; i += kScanThreads) {
      const int t = i / kCols, e = i % kCols;
      const bool in = t < m && c0 + e < V;
      cp_async4(vs + i, p.v + (static_cast<long long>(row0 + (in ? t : 0)) * p.H + h) * V + (in ? c0 + e : 0), in ? 4 : 0);
    }
    const float* src = coef + static_cast<long long>(ci) * p.H * kCoefs + kCoefVec;
    if (!CHAN && tid < 2 * kC / 4) cp_async16(vec + (ci & 1) * 2 * kC + tid * 4, src + tid * 4);
    cp_commit();
  };
  auto stage_coefs = [&](int ci) {
    const float* src = coef + static_cast<long long>(ci) * p.H * kCoefs;
    for (int i = tid; i < 2 * kC * kC / 4; i += kScanThreads) {
      const int row = i / (kC / 4), e = (i % (kC / 4)) * 4;              // rows 0..kC-1 of T', then of B
      cp_async16(ts + row * kGramLd + e, src + row * kC + e);
    }
    if constexpr (CHAN) {
      scaled(ks + Sh::kK, ci, 2);
      const float* g = p.gc + (static_cast<long long>(chunk_base(start, b) + ci) * p.H + h) * D;
      for (int i = tid; i < D; i += kScanThreads) cp_async4(gcs + i, g + i);
    }
    cp_commit();
  };

  stage_tokens(0);
  stage_coefs(0);
  for (int ci = 0; ci < nch; ++ci) {
    const float* kb = ks + (CHAN ? 0 : (ci & 1) * Sh::kK);
    const float* ku = CHAN ? ks + Sh::kK : kb;         // what the state's update reads
    const float* gv = vec + (ci & 1) * 2 * kC;
    cp_wait<1>();                                      // the tokens; the coefficients may still be on their way
    __syncthreads();
    float y[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i][0] = y[i][1] = 0.f;
    {
      const float* a = (rg < 8 ? kb + rg * 4 * ld : qs + (rg - 8) * 4 * ld);
#pragma unroll 4
      for (int d = 0; d < Sh::kDp; d += 4) {
        float4 x[4];
        float2 z[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i] = *reinterpret_cast<const float4*>(a + i * ld + d);
          z[i] = *reinterpret_cast<const float2*>(ss + (d + i) * kCols + cp);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          y[i][0] += x[i].x * z[0].x + x[i].y * z[1].x + x[i].z * z[2].x + x[i].w * z[3].x;
          y[i][1] += x[i].x * z[0].y + x[i].y * z[1].y + x[i].z * z[2].y + x[i].w * z[3].y;
        }
      }
    }
    const int t4 = (rg & 7) * 4;                       // first of this thread's four tokens
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (!CHAN) {
        const float G = gv[t4 + i];
        y[i][0] *= G;
        y[i][1] *= G;
      }
      if (rg < 8) {
        const float2 v = *reinterpret_cast<const float2*>(vs + (t4 + i) * kCols + cp);
        *reinterpret_cast<float2*>(rs + (t4 + i) * kCols + cp) = make_float2(v.x - y[i][0], v.y - y[i][1]);
      }
    }
    cp_wait<0>();
    __syncthreads();
    if (ci + 1 < nch) stage_tokens(ci + 1);            // q, v and the other k buffer are free
    {
      float u[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
      const int t2 = rg * 2;
      for (int j = 0; j <= 4 * warp; j += 4) {         // T' is lower triangular; this warp's rows end at 4 warp + 3
        float4 x[2];
        float2 z[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) x[i] = *reinterpret_cast<const float4*>(ts + (t2 + i) * kGramLd + j);
#pragma unroll
        for (int i = 0; i < 4; ++i) z[i] = *reinterpret_cast<const float2*>(rs + (j + i) * kCols + cp);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          u[i][0] += x[i].x * z[0].x + x[i].y * z[1].x + x[i].z * z[2].x + x[i].w * z[3].x;
          u[i][1] += x[i].x * z[0].y + x[i].y * z[1].y + x[i].z * z[2].y + x[i].w * z[3].y;
        }
      }
      __syncthreads();                                 // everyone is done with the right-hand side
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float w = CHAN ? 1.f : gv[kC + t2 + i];
        *reinterpret_cast<float2*>(us + (t2 + i) * kCols + cp) = make_float2(u[i][0], u[i][1]);
        *reinterpret_cast<float2*>(rs + (t2 + i) * kCols + cp) = make_float2(w * u[i][0], w * u[i][1]);
      }
    }
    __syncthreads();
    if (warp >= 4) {
      for (int j = 0; j < 8 * (warp - 3); j += 4) {    // B is lower triangular; this warp's tokens end at 8 (warp - 3) - 1
        float4 x[4];
        float2 z[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i] = *reinterpret_cast<const float4*>(bs + (t4 + i) * kGramLd + j);
          z[i] = *reinterpret_cast<const float2*>(us + (j + i) * kCols + cp);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          y[i][0] += x[i].x * z[0].x + x[i].y * z[1].x + x[i].z * z[2].x + x[i].w * z[3].x;
          y[i][1] += x[i].x * z[0].y + x[i].y * z[1].y + x[i].z * z[2].y + x[i].w * z[3].y;
        }
      }
      const int row0 = start + ch.first(ci), m = ch.len(ci);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (t4 + i >= m) continue;
        float* o = p.o + (static_cast<long long>(row0 + t4 + i) * p.H + h) * V + c0 + cp;
        if (c0 + cp < V) o[0] = y[i][0];
        if (c0 + cp + 1 < V) o[1] = y[i][1];
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const float G = CHAN ? gcs[rg * RPT + i] : gv[kC - 1];
      S[i][0] *= G;
      S[i][1] *= G;
    }
#pragma unroll 4
    for (int j = 0; j < kC; ++j) {
      const float2 w = *reinterpret_cast<const float2*>(rs + j * kCols + cp);
#pragma unroll
      for (int i = 0; i < RPT; i += 4) {
        const float4 k = *reinterpret_cast<const float4*>(ku + j * ld + rg * RPT + i);
        S[i][0] += k.x * w.x;
        S[i][1] += k.x * w.y;
        S[i + 1][0] += k.y * w.x;
        S[i + 1][1] += k.y * w.y;
        S[i + 2][0] += k.z * w.x;
        S[i + 2][1] += k.z * w.y;
        S[i + 3][0] += k.w * w.x;
        S[i + 3][1] += k.w * w.y;
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i)
      *reinterpret_cast<float2*>(ss + (rg * RPT + i) * kCols + cp) = make_float2(S[i][0], S[i][1]);
    if (track > 0 && ch.first(ci) + ch.len(ci) == track)
      store(p.state + (static_cast<long long>(p.track_slot[b]) * p.H + h) * plane);
    __syncthreads();
    if (ci + 1 < nch) stage_coefs(ci + 1);
  }
  store(st);
  if (blockIdx.z == 0) write_windows<T>(p, b, h, start, n, fresh, track, kScanThreads);
}

// Decode, and the sequences of a ragged step that bring one token.  Eight lanes share a column group, RPL rows and CPL adjacent columns of the state per
// lane (D <= 8 * RPL); a CTA owns 16 * CPL columns of one (request, head).  The state streams through once.
constexpr int kLanes = 8;
constexpr int kStepThreads = 128;

template <typename T, int RPL, int CPL, bool CHAN>
__global__ void __launch_bounds__(kStepThreads) delta_step_kernel(const DeltaParams p) {
  __shared__ __align__(16) float qk[CHAN ? 3 : 2][kLanes * RPL];       // q, k, decays per channel
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, rl = lane & (kLanes - 1);
  const int b = blockIdx.x, h = blockIdx.y, hk = h / (p.H / p.Hk), D = p.D, V = p.V;
  int t = b;
  if (p.cu != nullptr) {
    t = p.cu[b];
    if (p.cu[b + 1] - t != 1) return;
  }
  const bool fresh = p.prefix != nullptr && p.prefix[b] == 0;
  const int gc = blockIdx.z * (kStepThreads / kLanes) * CPL + ((tid >> 5) * (32 / kLanes) + lane / kLanes) * CPL;
  const bool vec = V % CPL == 0;                       // whole column groups: wide accesses
  float* st = p.state + (p.slots[b] * p.H + h) * static_cast<long long>(D) * V;
  float S[RPL][CPL];
  auto row_of = [&](int i) { return 4 * ((i >> 2) * kLanes + rl) + (i & 3); };
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = row_of(i);
    const float* d = st + static_cast<long long>(r) * V + gc;
#pragma unroll
    for (int c = 0; c < CPL; ++c) S[i][c] = 0.f;
    if (fresh || r >= D || gc >= V) continue;
    if (CPL == 4 && vec) {
      const float4 v = *reinterpret_cast<const float4*>(d);
      S[i][0] = v.x; S[i][1 % CPL] = v.y; S[i][2 % CPL] = v.z; S[i][3 % CPL] = v.w;
    } else if (CPL == 2 && vec) {
      const float2 v = *reinterpret_cast<const float2*>(d);
      S[i][0] = v.x; S[i][1 % CPL] = v.y;
    } else {
#pragma unroll
      for (int c = 0; c < CPL; ++c)
        if (gc + c < V) S[i][c] = d[c];
    }
  }
  for (int i = tid; i < 2 * kLanes * RPL; i += kStepThreads) {
    const int which = i / (kLanes * RPL), e = i - which * kLanes * RPL;
    qk[which][e] = e < D ? p.qk[((static_cast<long long>(t) * p.Hk + hk) * 2 + which) * D + e] : 0.f;
  }
  const long long bh = static_cast<long long>(t) * p.H + h;
  if constexpr (CHAN) {
    const float rate = -expf(p.a_log[h]);
    for (int e = tid; e < kLanes * RPL; e += kStepThreads)
      qk[CHAN ? 2 : 0][e] = e < D ? expf(rate * softplus(to_f(static_cast<const T*>(p.chan_a)[bh * D + e]) + p.dt_bias[h * D + e]))
                                  : 0.f;
  }
  __syncthreads();
  const float g = CHAN ? 1.f : p.gb[bh * 2], beta = p.gb[bh * 2 + 1];
  if constexpr (CHAN)
#pragma unroll
    for (int i = 0; i < RPL; i += 4) {
      const float4 d = *reinterpret_cast<const float4*>(&qk[CHAN ? 2 : 0][row_of(i)]);
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        S[i][c] *= d.x;
        S[i + 1][c] *= d.y;
        S[i + 2][c] *= d.z;
        S[i + 3][c] *= d.w;
      }
    }
  float kd[CPL], qd[CPL], kq = 0.f, kr[RPL];
#pragma unroll
  for (int c = 0; c < CPL; ++c) kd[c] = qd[c] = 0.f;
#pragma unroll
  for (int i = 0; i < RPL; i += 4) {
    const float4 q = *reinterpret_cast<const float4*>(&qk[0][row_of(i)]), k = *reinterpret_cast<const float4*>(&qk[1][row_of(i)]);
    kr[i] = k.x; kr[i + 1] = k.y; kr[i + 2] = k.z; kr[i + 3] = k.w;
    kq += k.x * q.x + k.y * q.y + k.z * q.z + k.w * q.w;
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      kd[c] += S[i][c] * k.x + S[i + 1][c] * k.y + S[i + 2][c] * k.z + S[i + 3][c] * k.w;
      qd[c] += S[i][c] * q.x + S[i + 1][c] * q.y + S[i + 2][c] * q.z + S[i + 3][c] * q.w;
    }
  }
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) {
    kq += __shfl_xor_sync(0xffffffffu, kq, o);
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      kd[c] += __shfl_xor_sync(0xffffffffu, kd[c], o);
      qd[c] += __shfl_xor_sync(0xffffffffu, qd[c], o);
    }
  }
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    const float v = gc + c < V ? p.v[bh * V + gc + c] : 0.f;
    const float u = beta * (v - g * kd[c]);
    // o = S'^T q with S' = g S + k u^T, that is g (S^T q) + u (k . q)
    if (rl == 0 && gc + c < V) p.o[bh * V + gc + c] = g * qd[c] + u * kq;
#pragma unroll
    for (int i = 0; i < RPL; ++i) S[i][c] = g * S[i][c] + kr[i] * u;
  }
  auto store = [&](float* dst) {
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int r = row_of(i);
      float* d = dst + static_cast<long long>(r) * V + gc;
      if (r >= D || gc >= V) continue;
      if (CPL == 4 && vec) {
        *reinterpret_cast<float4*>(d) = make_float4(S[i][0], S[i][1 % CPL], S[i][2 % CPL], S[i][3 % CPL]);
      } else if (CPL == 2 && vec) {
        *reinterpret_cast<float2*>(d) = make_float2(S[i][0], S[i][1 % CPL]);
      } else {
#pragma unroll
        for (int c = 0; c < CPL; ++c)
          if (gc + c < V) d[c] = S[i][c];
      }
    }
  };
  store(st);
  const int track = p.cu != nullptr && p.track_len != nullptr ? p.track_len[b] : 0;
  if (track == 1) store(p.state + (static_cast<long long>(p.track_slot[b]) * p.H + h) * static_cast<long long>(D) * V);
  if (blockIdx.z == 0) write_windows<T>(p, b, h, t, 1, fresh, track, kStepThreads);
}

// One warp per (token, head); a lane holds NV groups of four adjacent columns (V <= 128 * NV, V % 4 == 0), or takes single
// columns (NV = 0, any V).
// The gates of head h lie at column (h / group) * step + (h % group) * V of a row.
template <typename W>
__device__ __forceinline__ float4 load_weight4(const W* w) {
  if constexpr (sizeof(W) == 2) {
    const uint2 raw = *reinterpret_cast<const uint2*>(w);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
  } else {
    return *reinterpret_cast<const float4*>(w);
  }
}

template <typename T, typename W, int NV, bool SIGMOID>
__global__ void delta_gate_kernel(const float* __restrict__ o, const T* __restrict__ gate, long long ld, int group, int step,
                                  const W* __restrict__ w, T* __restrict__ out, long long T_, int H, int V, float eps) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long wid = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  if (wid >= T_ * H) return;
  const long long t = wid / H;
  const int h = static_cast<int>(wid - t * H);
  const float* src = o + wid * V;
  const T* g = gate + t * ld + static_cast<long long>(h / group) * step + static_cast<long long>(h % group) * V;
  T* dst = out + wid * V;
  auto gated = [](float x, float gv) { return x * ((SIGMOID ? 1.f : gv) / (1.f + expf(-gv))); };
  float ss = 0.f;
  if constexpr (NV > 0) {
    float4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (lane + 32 * i) * 4;
      v[i] = c < V ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
    const float inv = 1.f / sqrtf(warp_sum(ss) / V + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (lane + 32 * i) * 4;
      if (c >= V) continue;
      const float4 wv = load_weight4(w + c);
      if constexpr (sizeof(T) == 2) {
        const uint2 raw = *reinterpret_cast<const uint2*>(g + c);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        *reinterpret_cast<uint2*>(dst + c) =
            make_uint2(pack_bf16(gated(v[i].x * inv * wv.x, a.x), gated(v[i].y * inv * wv.y, a.y)),
                       pack_bf16(gated(v[i].z * inv * wv.z, b.x), gated(v[i].w * inv * wv.w, b.y)));
      } else {
        const float4 a = *reinterpret_cast<const float4*>(g + c);
        *reinterpret_cast<float4*>(dst + c) =
            make_float4(gated(v[i].x * inv * wv.x, a.x), gated(v[i].y * inv * wv.y, a.y),
                        gated(v[i].z * inv * wv.z, a.z), gated(v[i].w * inv * wv.w, a.w));
      }
    }
  } else {
    for (int i = lane; i < V; i += 32) ss += src[i] * src[i];
    const float inv = 1.f / sqrtf(warp_sum(ss) / V + eps);
    for (int i = lane; i < V; i += 32) dst[i] = from_f<T>(gated(src[i] * inv * to_f(w[i]), to_f(g[i])));
  }
}

template <typename T, typename W, bool SIGMOID>
int run_gate(const float* o, const void* gate, long long ld, int group, int step, const W* w, void* out, long long n, int H,
             int V, float eps, cudaStream_t s) {
  const dim3 grid(static_cast<unsigned>((n * H + 3) / 4));
  const T* g = static_cast<const T*>(gate);
  T* d = static_cast<T*>(out);
  const bool vec = V % 4 == 0 && ld % 4 == 0 && step % 4 == 0 && reinterpret_cast<uintptr_t>(gate) % (4 * sizeof(T)) == 0 &&
                   reinterpret_cast<uintptr_t>(w) % (4 * sizeof(W)) == 0;
  if (vec && V <= 128)
    launch_pdl(delta_gate_kernel<T, W, 1, SIGMOID>, grid, dim3(128), 0, s, o, g, ld, group, step, w, d, n, H, V, eps);
  else if (vec && V <= 256)
    launch_pdl(delta_gate_kernel<T, W, 2, SIGMOID>, grid, dim3(128), 0, s, o, g, ld, group, step, w, d, n, H, V, eps);
  else
    launch_pdl(delta_gate_kernel<T, W, 0, SIGMOID>, grid, dim3(128), 0, s, o, g, ld, group, step, w, d, n, H, V, eps);
  return static_cast<int>(cudaGetLastError());
}

template <typename T, bool SIGMOID>
int run_gate(const float* o, const void* gate, long long ld, int group, int step, const void* w, int w_f32, void* out,
             long long n, int H, int V, float eps, cudaStream_t s) {
  if (w_f32) return run_gate<T, float, SIGMOID>(o, gate, ld, group, step, static_cast<const float*>(w), out, n, H, V, eps, s);
  return run_gate<T, __nv_bfloat16, SIGMOID>(o, gate, ld, group, step, static_cast<const __nv_bfloat16*>(w), out, n, H, V, eps, s);
}

template <typename T, int NPL, int TAPS>
int launch_prep(const DeltaParams& p, cudaStream_t s) {
  const int units = p.Hk + p.H;
  auto blocks = [&](int run) {
    return dim3(static_cast<unsigned>(((static_cast<long long>(p.T) + run - 1) / run * units + 3) / 4));
  };
  // long runs reuse the window and the kernel; short steps want the warps.  Eight rows a warp from 16 such warps an SM on (1024 rows of 32
  // units: 78 us a row at a time, 38 so), sixteen from 32 on
  const long long rows = static_cast<long long>(p.T) * units, sms = sm_count();
  if (p.cu != nullptr && rows >= 16 * sms * 32)
    launch_pdl(delta_prep_kernel<T, NPL, TAPS, 16>, blocks(16), dim3(128), 0, s, p);
  else if (p.cu != nullptr && rows >= 8 * sms * 16)
    launch_pdl(delta_prep_kernel<T, NPL, TAPS, 8>, blocks(8), dim3(128), 0, s, p);
  else
    launch_pdl(delta_prep_kernel<T, NPL, TAPS, 1>, blocks(1), dim3(128), 0, s, p);
  return static_cast<int>(cudaGetLastError());
}

template <typename T, int RPT>
int launch_scan_channel(const DeltaParams& p, cudaStream_t s) {
  using Sh = ScanShape<RPT>;
  static bool cfg = false, cfg_chunk = false;
  const int chunk_smem = ChannelShape::smem(Sh::kDp);
  int e = set_smem(delta_chunk_channel_kernel<T>, ChannelShape::smem(ScanShape<16>::kDp), &cfg_chunk);
  if (e == 0) e = set_smem(delta_scan_kernel<T, RPT, true>, Sh::kSmem, &cfg);
  if (e != 0) return e;
  launch_pdl(delta_chunk_channel_kernel<T>, dim3(chunk_base(p.T, p.B), p.H), dim3(kChannelThreads), chunk_smem, s, p,
             static_cast<int>(Sh::kDp));
  e = static_cast<int>(cudaGetLastError());
  if (e != 0) return e;
  launch_pdl(delta_scan_kernel<T, RPT, true>, dim3(p.B, p.H, (p.V + kCols - 1) / kCols), dim3(kScanThreads), Sh::kSmem, s, p);
  return static_cast<int>(cudaGetLastError());
}

template <typename T, int RPT>
int launch_scan(const DeltaParams& p, cudaStream_t s) {
  using Sh = ScanShape<RPT>;
  if (p.chan_a != nullptr) return launch_scan_channel<T, RPT>(p, s);
  static bool cfg = false, cfg_chunk = false;
  const int chunk_smem = (2 * kC * Sh::kLd + 2 * kC * kGramLd + kChunkThreads) * 4;
  int e = set_smem(delta_chunk_kernel, (2 * kC * ScanShape<16>::kLd + 2 * kC * kGramLd + kChunkThreads) * 4, &cfg_chunk);
  if (e == 0) e = set_smem(delta_scan_kernel<T, RPT, false>, Sh::kSmem, &cfg);
  if (e != 0) return e;
  launch_pdl(delta_chunk_kernel, dim3(chunk_base(p.T, p.B), p.Hk), dim3(kChunkThreads), chunk_smem, s, p,
             static_cast<int>(Sh::kDp));
  e = static_cast<int>(cudaGetLastError());
  if (e != 0) return e;
  launch_pdl(delta_scan_kernel<T, RPT, false>, dim3(p.B, p.H, (p.V + kCols - 1) / kCols), dim3(kScanThreads), Sh::kSmem, s, p);
  return static_cast<int>(cudaGetLastError());
}

template <typename T, int RPL, int CPL>
int launch_step(const DeltaParams& p, cudaStream_t s) {
  constexpr int cols = (kStepThreads / kLanes) * CPL;
  const auto kernel = p.chan_a != nullptr ? delta_step_kernel<T, RPL, CPL, true> : delta_step_kernel<T, RPL, CPL, false>;
  launch_pdl(kernel, dim3(p.B, p.H, (p.V + cols - 1) / cols), dim3(kStepThreads), 0, s, p);
  return static_cast<int>(cudaGetLastError());
}

template <typename T, int RPL>
int launch_step_rows(const DeltaParams& p, cudaStream_t s) {
  // wide accesses once there are states enough to fill the machine with the fewer threads
  const long long groups = static_cast<long long>(p.B) * p.H * ((p.V + 15) / 16);
  constexpr int kMost = RPL <= 16 ? 4 : 2;
  if (groups >= 148 * 32) return launch_step<T, RPL, kMost>(p, s);
  if (groups >= 148 * 8) return launch_step<T, RPL, 2>(p, s);
  return launch_step<T, RPL, 1>(p, s);
}

template <typename T>
int run_delta(const DeltaParams& p, cudaStream_t s) {
  const int wide = p.D > p.V ? p.D : p.V;
  int e;
  if (p.taps <= 4)
    e = wide <= 64 ? launch_prep<T, 2, 4>(p, s) : wide <= 128 ? launch_prep<T, 4, 4>(p, s) : launch_prep<T, 8, 4>(p, s);
  else
    e = wide <= 128 ? launch_prep<T, 4, 16>(p, s) : launch_prep<T, 8, 16>(p, s);
  if (e != 0) return e;
  if (p.cu == nullptr || p.singles) {
    const int r = p.D <= 32 ? launch_step_rows<T, 4>(p, s) : p.D <= 64 ? launch_step_rows<T, 8>(p, s)
                  : p.D <= 128 ? launch_step_rows<T, 16>(p, s) : launch_step_rows<T, 32>(p, s);
    if (r != 0 || p.cu == nullptr || p.singles == p.B) return r;
  }
  if (p.D <= 64) return launch_scan<T, 4>(p, s);
  if (p.D <= 128) return launch_scan<T, 8>(p, s);
  return launch_scan<T, 16>(p, s);
}

}  // namespace
}  // namespace sglb

extern "C" {

// Shapes in DeltaParams, `cols` the eight members of DeltaColumns; T = bf16 or fp32 (`is_f32`) is the type of `proj`, `ba`,
// `conv_w` and `conv_state`.
int sglb_delta_scan(const void* proj, long long ld, const void* ba, long long ba_ld, const int* cols, const void* conv_w,
                    const float* a_log, const float* dt_bias, const void* chan_a, void* conv_state, float* state,
                    const long long* slots, const int* cu, const int* prefix, const int* track_len, const int* track_slot,
                    float* qk, float* v, float* gb, float* coef, float* kq, float* gc, float* o, int B, int T, int H, int Hk,
                    int D, int V, int taps, int singles, int is_f32, cudaStream_t s) {
  using namespace sglb;
  if (B <= 0 || T <= 0) return 0;
  if (cu != nullptr && (prefix == nullptr || (coef == nullptr && singles != B))) return -kBadArgument;
  if (chan_a != nullptr && coef != nullptr && (kq == nullptr || gc == nullptr)) return -kBadArgument;
  if (D < 1 || D > 256 || V < 1 || Hk < 1 || H % Hk != 0 || taps < 1 || taps > 16 || H > 65535) return -kBadArgument;
  const DeltaColumns c{cols[0], cols[1], cols[2], cols[3], cols[4], cols[5], cols[6], cols[7]};
  DeltaParams p{proj, ld, ba, ba_ld, c, conv_w, a_log, dt_bias, chan_a, conv_state, state, slots, cu, prefix,
                track_len, track_slot, qk, v, gb, coef, kq, gc, o, B, T, H, Hk, D, V, taps, singles};
  return is_f32 ? run_delta<float>(p, s) : run_delta<__nv_bfloat16>(p, s);
}

// out [T, H * V] = rmsnorm(o [T, H, V], over V) * w [V] * silu(gate) (or sigmoid(gate)), gate at row stride `ld`, its heads in
// groups of `group` neighbours `step` columns apart.
int sglb_delta_gate(const float* o, const void* gate, long long ld, int group, int step, const void* w, int w_f32, void* out,
                    long long T, int H, int V, float eps, int sigmoid, int is_f32, cudaStream_t s) {
  using namespace sglb;
  if (T <= 0) return 0;
  if (group < 1) return -kBadArgument;
  if (sigmoid)
    return is_f32 ? run_gate<float, true>(o, gate, ld, group, step, w, w_f32, out, T, H, V, eps, s)
                  : run_gate<__nv_bfloat16, true>(o, gate, ld, group, step, w, w_f32, out, T, H, V, eps, s);
  return is_f32 ? run_gate<float, false>(o, gate, ld, group, step, w, w_f32, out, T, H, V, eps, s)
                : run_gate<__nv_bfloat16, false>(o, gate, ld, group, step, w, w_f32, out, T, H, V, eps, s);
}

}  // extern "C"
