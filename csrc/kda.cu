// Kernels of the KDA + latent-MoE model line (Kimi-K3 shape).
//
//  * kda_recurrent: the delta rule with a decay per key channel.  Per token and head,
//      dec[d] = exp(lower * sigmoid(exp(A_log[h]) * (f[d] + dt_bias[h, d])))   (lower < 0, so dec in (e^lower, 1))
//      S      = S * dec (rows of S[Dk, Dv] scaled)        kv = S^T k
//      S     += k (x) ((v - kv) * sigmoid(b))             out = S^T q
//    with q and k L2-normalised (q also times Dk^-0.5).  The gate arithmetic runs inside the kernel, so the
//    step needs no separate gate launch.  The state layout and the thread mapping are those of the scalar-decay
//    rule in gdn.cu: a CTA takes 32 columns of one (sequence, head), four lanes share a column and each keeps a
//    quarter of its Dk elements in registers; a stage of 8 tokens is normalised into shared memory, then
//    walked in order.  A decode step is one pass over the state (read + write).
//    The same kernel runs two more rules (RULE below): the decay in its softplus form, exp(-exp(A_log) softplus(f + dt_bias)),
//    with query / key heads shared by several value heads, plain linear attention with one fixed decay per head
//    (S = decay S + k (x) v, out = S^T q, SiLU on q, k and v), and linear attention with a decay per token and key channel and a
//    bonus for the current token (out = (S + diag(u) k (x) v)^T q in front of S = diag(dec) S + k (x) v, dec = exp(-exp(f + w0))), and
//    state-space duality, one decay per token and head (d = softplus(f + dt_bias), S = exp(-exp(A_log) d) S + d k (x) v, out = S^T q +
//    D v, keys and queries shared by a group of heads).
//    Those take bf16 or f32 rows and any key width up to 256.
//  * attnres_mix: the attention-residual mix.  Every token keeps up to `cap` snapshot rows of its own residual
//    stream; a mix scores each of the first nb snapshots and the current row with
//    dot(x / rms(x), score_w) and returns the softmax-weighted sum of the un-normalised rows.
//
// Functional parity with pegainfer-k3/kernels/tilelang_defs.py:67-139 (attnres_scores / attnres_mix) and
// :304-410 (kda_core) and pegainfer-kernels/csrc/k3/k3_flash_kda.cu (chunked prefill of the same rule).
#include "api.h"
#include "common.cuh"
#include "mma_frag.cuh"
#include "types.cuh"

namespace {

constexpr int KDA_STAGE = 8;
constexpr int KDA_COLS = 32;

// What a token does to the state.  BOUNDED and SOFTPLUS are the delta rule with a decay per key channel and two forms of
// the decay; DECAY is linear attention with a fixed decay per head (no correction term), WKV with a decay per token and key
// channel, read in front of the update with a bonus for the current token, SSD with a decay and a step size per token and head.
enum { RULE_BOUNDED = 0, RULE_SOFTPLUS = 1, RULE_DECAY = 2, RULE_WKV = 3, RULE_SSD = 4 };

template <typename T>
struct RecArgs {
  const T *q, *k, *v;  // token rows of stride ld; q and k [kv_heads * dk], v [heads * dv]
  long long ld;
  const void* f;  // raw decay projection [heads * dk]: T (BOUNDED) or f32 (SOFTPLUS, WKV); SSD: raw step sizes T [heads]
  long long ldf;
  const T* b;  // raw step-size projection [heads]
  long long ldb;
  const float *a_log, *dt_bias, *decay;  // decay [heads]: DECAY; WKV: dt_bias = w0 [heads * dk], decay = the bonus u [heads * dk]; SSD: dt_bias [heads], decay = D [heads]
  float lower;
  float* state;
  T* out;
  const int *q_indptr, *slots;
  int heads, kv_heads, dk, dv, col_groups;
  int skip_len;  // > 0: sequences of at least that many tokens belong to another kernel
};

// XW = false: four adjacent lanes share a state column and reduce with shuffles (prompt chunks: no barrier per token).
// XW = true: a warp owns one quarter of Dk for all 32 columns, so every state load and store of a warp is one 128-byte row
// and the shared-memory reads of k, q and the decays are broadcasts; the four quarters meet through shared memory with two
// barriers per token (decode rows and other steps of a few tokens).
// DK is the key width rounded up to an instantiated size; entries past dk are zero (PAD).
template <typename T, int DK, bool XW, int RULE, bool PAD>
__global__ void __launch_bounds__(128) kda_recurrent_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long ld, const void* __restrict__ f, long long ldf,
                                                            const T* __restrict__ b, long long ldb, const float* __restrict__ a_log, const float* __restrict__ dt_bias, const float* __restrict__ decay,
                                                            float lower, float* __restrict__ state, T* __restrict__ out, const int* __restrict__ q_indptr, const int* __restrict__ slots, int heads,
                                                            int kv_heads, int dk_arg, int dv, int col_groups, int skip_len) {
  constexpr int QK = DK / 4;   // state elements per thread
  constexpr int QS = QK + 4;   // padded quarter stride: the four quarters land in different banks
  constexpr int QL = DK / 32;  // elements per lane when a warp holds one token
  constexpr bool DELTA = RULE == RULE_BOUNDED || RULE == RULE_SOFTPLUS;
  constexpr bool KEYED = RULE != RULE_DECAY && RULE != RULE_SSD;  // a decay per key channel
  __shared__ __align__(16) float sq[KDA_STAGE][4 * QS], sk[KDA_STAGE][4 * QS], sd[KEYED ? KDA_STAGE : 1][4 * QS];
  __shared__ float sv[KDA_STAGE][KDA_COLS], sb[KDA_STAGE], se[RULE == RULE_SSD ? KDA_STAGE : 1];
  __shared__ float red_kv[4][KDA_COLS], red_o[DELTA ? 1 : 2][4][KDA_COLS];
  const int dk = PAD ? dk_arg : DK;
  const int h = blockIdx.x / col_groups, cg = blockIdx.x % col_groups, seq = blockIdx.y;
  const int slot = slots[seq];
  const int q0 = q_indptr[seq], q1 = q_indptr[seq + 1];
  if (q1 == q0 || slot < 0) return;
  if (skip_len > 0 && q1 - q0 >= skip_len) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qtr = XW ? warp : (tid & 3), lc = XW ? lane : (tid >> 2), col = cg * KDA_COLS + lc;
  const bool owner = col < dv;
  float* S = state + (((long long)slot * heads + h) * dk) * dv;  // [dk][dv], v contiguous
  // Shuffle mapping: a thread's own elements sit DK / 4 rows apart, so a warp reads 32-byte pieces of four rows.  Staging
  // the CTA's slice through shared memory instead was measured slower (200 us against 111 us for 32 decode rows of 96
  // heads: the extra 17 KB per CTA costs resident CTAs); the XW mapping reads whole rows without it (86 us).
  float s_col[QK];
#pragma unroll
  for (int i = 0; i < QK; ++i) s_col[i] = owner && (!PAD || qtr * QK + i < dk) ? S[(long long)(qtr * QK + i) * dv + col] : 0.f;
  const int kh = RULE == RULE_SOFTPLUS || RULE == RULE_SSD ? h * kv_heads / heads : h;
  const float q_scale = DELTA ? rsqrtf((float)dk) : 1.f;
  const float a = DELTA || RULE == RULE_SSD ? __expf(a_log[h]) : 0.f;
  const float fixed = RULE == RULE_DECAY || RULE == RULE_SSD ? decay[h] : 0.f;

  for (int t0 = q0; t0 < q1; t0 += KDA_STAGE) {
    const int nt = min(KDA_STAGE, q1 - t0);
    // stage: each warp prepares two tokens' q and k (unit rows, or SiLU of the projections) and their decays
    for (int j = warp; j < nt; j += 4) {
      const long long row = (long long)(t0 + j);
      const T* qp = q + row * ld + (long long)kh * dk;
      const T* kp = k + row * ld + (long long)kh * dk;
      float rq[QL], rk[QL], qs = 0.f, ks = 0.f;
#pragma unroll
      for (int i = 0; i < QL; ++i) {
        const bool in = !PAD || lane + 32 * i < dk;
        rq[i] = in ? to_f32(qp[lane + 32 * i]) : 0.f;
        rk[i] = in ? to_f32(kp[lane + 32 * i]) : 0.f;
        if (DELTA) {
          qs += rq[i] * rq[i];
          ks += rk[i] * rk[i];
        } else if (RULE == RULE_WKV) {
          if (in) qs += rq[i] * rk[i] * decay[h * dk + lane + 32 * i];
        } else if (RULE == RULE_DECAY) {  // the activation's result is what the layer works with, in the activation type
          rq[i] = to_f32(from_f32<T>(rq[i] / (1.f + __expf(-rq[i]))));
          rk[i] = to_f32(from_f32<T>(rk[i] / (1.f + __expf(-rk[i]))));
        }
      }
      float qn = 1.f, kn = 1.f;
      if (DELTA) {
        qs = warp_sum(qs);
        ks = warp_sum(ks);
        qn = rsqrtf(qs + 1e-6f) * q_scale, kn = rsqrtf(ks + 1e-6f);
      }
      if (RULE == RULE_WKV) {  // what the token's own value counts
        qs = warp_sum(qs);
        if (lane == 0) sb[j] = qs;
      }
#pragma unroll
      for (int i = 0; i < QL; ++i) {
        const int e = lane + 32 * i, at = (e / QK) * QS + (e % QK);
        sq[j][at] = rq[i] * qn;
        sk[j][at] = rk[i] * kn;
        if (RULE == RULE_BOUNDED) {
          const float raw = to_f32(((const T*)f)[row * ldf + (long long)h * dk + e]) + dt_bias[h * dk + e];
          sd[j][at] = __expf(lower / (1.f + __expf(-a * raw)));
        } else if (RULE == RULE_SOFTPLUS) {
          float dec = 1.f;
          if (!PAD || e < dk) {
            const float raw = ((const float*)f)[row * ldf + (long long)h * dk + e] + dt_bias[h * dk + e];
            dec = __expf(-a * (raw > 20.f ? raw : log1pf(__expf(raw))));
          }
          sd[j][at] = dec;
        } else if (RULE == RULE_WKV) {
          sd[j][at] = !PAD || e < dk ? __expf(-__expf(((const float*)f)[row * ldf + (long long)h * dk + e] + dt_bias[h * dk + e])) : 1.f;
        }
      }
    }
    for (int idx = tid; idx < nt * KDA_COLS; idx += 128) {
      const int j = idx / KDA_COLS, d = cg * KDA_COLS + idx % KDA_COLS;
      float x = d < dv ? to_f32(v[(long long)(t0 + j) * ld + (long long)h * dv + d]) : 0.f;
      if (RULE == RULE_DECAY) x = to_f32(from_f32<T>(x / (1.f + __expf(-x))));
      sv[j][idx % KDA_COLS] = x;
    }
    if (RULE == RULE_SSD && tid < nt) {
      const float raw = to_f32(((const T*)f)[(long long)(t0 + tid) * ldf + h]) + dt_bias[h], d = raw > 20.f ? raw : log1pf(__expf(raw));
      sb[tid] = d;
      se[tid] = __expf(-a * d);
    }
    if (DELTA && tid < nt) sb[tid] = 1.f / (1.f + __expf(-to_f32(b[(long long)(t0 + tid) * ldb + h])));
    __syncthreads();
    for (int j = 0; j < nt; ++j) {
      const float4* kq = reinterpret_cast<const float4*>(&sk[j][qtr * QS]);
      const float4* qq = reinterpret_cast<const float4*>(&sq[j][qtr * QS]);
      float delta = RULE == RULE_SSD ? sv[j][lc] * sb[j] : sv[j][lc];
      if (DELTA) {
        const float4* dq = reinterpret_cast<const float4*>(&sd[DELTA ? j : 0][qtr * QS]);
        float4 kv4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < QK / 4; ++i) {
          const float4 kk = kq[i], dd = dq[i];
          s_col[4 * i + 0] *= dd.x;
          s_col[4 * i + 1] *= dd.y;
          s_col[4 * i + 2] *= dd.z;
          s_col[4 * i + 3] *= dd.w;
          kv4.x += s_col[4 * i + 0] * kk.x;
          kv4.y += s_col[4 * i + 1] * kk.y;
          kv4.z += s_col[4 * i + 2] * kk.z;
          kv4.w += s_col[4 * i + 3] * kk.w;
        }
        float kv = (kv4.x + kv4.y) + (kv4.z + kv4.w);
        if (XW) {
          red_kv[qtr][lc] = kv;
          __syncthreads();
          kv = (red_kv[0][lc] + red_kv[1][lc]) + (red_kv[2][lc] + red_kv[3][lc]);
        } else {
          kv += __shfl_xor_sync(0xffffffffu, kv, 1);
          kv += __shfl_xor_sync(0xffffffffu, kv, 2);
        }
        delta = (delta - kv) * sb[j];
      }
      float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < QK / 4; ++i) {
        const float4 kk = kq[i], qv = qq[i];
        if (RULE == RULE_WKV) {
          const float4 dd = reinterpret_cast<const float4*>(&sd[KEYED ? j : 0][qtr * QS])[i];
          o4.x += s_col[4 * i + 0] * qv.x;
          o4.y += s_col[4 * i + 1] * qv.y;
          o4.z += s_col[4 * i + 2] * qv.z;
          o4.w += s_col[4 * i + 3] * qv.w;
          s_col[4 * i + 0] = s_col[4 * i + 0] * dd.x + kk.x * delta;
          s_col[4 * i + 1] = s_col[4 * i + 1] * dd.y + kk.y * delta;
          s_col[4 * i + 2] = s_col[4 * i + 2] * dd.z + kk.z * delta;
          s_col[4 * i + 3] = s_col[4 * i + 3] * dd.w + kk.w * delta;
          continue;
        }
        if (!DELTA) {
          const float dec = RULE == RULE_SSD ? se[RULE == RULE_SSD ? j : 0] : fixed;
          s_col[4 * i + 0] *= dec;
          s_col[4 * i + 1] *= dec;
          s_col[4 * i + 2] *= dec;
          s_col[4 * i + 3] *= dec;
        }
        s_col[4 * i + 0] += kk.x * delta;
        s_col[4 * i + 1] += kk.y * delta;
        s_col[4 * i + 2] += kk.z * delta;
        s_col[4 * i + 3] += kk.w * delta;
        o4.x += s_col[4 * i + 0] * qv.x;
        o4.y += s_col[4 * i + 1] * qv.y;
        o4.z += s_col[4 * i + 2] * qv.z;
        o4.w += s_col[4 * i + 3] * qv.w;
      }
      float o = (o4.x + o4.y) + (o4.z + o4.w);
      if (XW) {
        // two buffers: with the delta rule the barrier in front of it orders a token's reads before the next token's
        // writes, without it the next token writes the other buffer and the one after that comes behind its barrier
        red_o[DELTA ? 0 : j & 1][qtr][lc] = o;
        __syncthreads();  // also orders this token's reads of red_kv before the next token's writes
        o = (red_o[DELTA ? 0 : j & 1][0][lc] + red_o[DELTA ? 0 : j & 1][1][lc]) + (red_o[DELTA ? 0 : j & 1][2][lc] + red_o[DELTA ? 0 : j & 1][3][lc]);
      } else {
        o += __shfl_xor_sync(0xffffffffu, o, 1);
        o += __shfl_xor_sync(0xffffffffu, o, 2);
      }
      if (RULE == RULE_WKV) o += sb[j] * delta;
      if (RULE == RULE_SSD) o += fixed * sv[j][lc];
      if (owner && qtr == 0) out[((long long)(t0 + j) * heads + h) * dv + col] = from_f32<T>(o);
    }
    __syncthreads();
  }
  if (owner) {
#pragma unroll
    for (int i = 0; i < QK; ++i)
      if (!PAD || qtr * QK + i < dk) S[(long long)(qtr * QK + i) * dv + col] = s_col[i];
  }
}

template <typename T, int DK, int RULE, bool PAD>
cudaError_t launch_rule(const RecArgs<T>& p, dim3 grid, bool few, cudaStream_t stream) {
  auto kernel = few ? kda_recurrent_kernel<T, DK, true, RULE, PAD> : kda_recurrent_kernel<T, DK, false, RULE, PAD>;
  // launched in plain stream order: a successor that starts early holds CTA slots of this kernel's long-running blocks
  // (prompt of 2048 tokens: 2.5 ms with programmatic launch, 2.1 ms without)
  kernel<<<grid, 128, 0, stream>>>(p.q, p.k, p.v, p.ld, p.f, p.ldf, p.b, p.ldb, p.a_log, p.dt_bias, p.decay, p.lower, p.state, p.out, p.q_indptr, p.slots, p.heads, p.kv_heads, p.dk, p.dv, p.col_groups,
                                   p.skip_len);
  return cudaSuccess;
}
// any key width up to 256, on the next larger instantiated size
template <typename T, int RULE>
cudaError_t launch_padded(const RecArgs<T>& p, dim3 grid, bool few, cudaStream_t stream) {
  if (p.dk == 128) return launch_rule<T, 128, RULE, false>(p, grid, few, stream);
  if (p.dk == 64) return launch_rule<T, 64, RULE, false>(p, grid, few, stream);
  if (p.dk <= 32) return launch_rule<T, 32, RULE, true>(p, grid, few, stream);
  if (p.dk <= 64) return launch_rule<T, 64, RULE, true>(p, grid, few, stream);
  if (p.dk <= 128) return launch_rule<T, 128, RULE, true>(p, grid, few, stream);
  return launch_rule<T, 256, RULE, true>(p, grid, few, stream);
}

template <typename T>
int run_rule(int rule, RecArgs<T> p, int num_seqs, int max_q_len, cudaStream_t stream) {
  p.col_groups = (p.dv + KDA_COLS - 1) / KDA_COLS;
  const dim3 grid(p.heads * p.col_groups, num_seqs);
  const bool few = max_q_len <= 4;  // decode rows and verify steps: the row-coalesced mapping
  PG_CUDA(rule == RULE_SOFTPLUS ? (launch_padded<T, RULE_SOFTPLUS>(p, grid, few, stream))
          : rule == RULE_WKV    ? (launch_padded<T, RULE_WKV>(p, grid, few, stream))
          : rule == RULE_SSD    ? (launch_padded<T, RULE_SSD>(p, grid, few, stream))
                                : (launch_padded<T, RULE_DECAY>(p, grid, few, stream)));
  PG_LAUNCH_CHECK();
  return PG_OK;
}

// ---------------------------------------------------------------------------------
// The delta rule with bounded channel decays, KB_T tokens at a time (prompts, 128-wide keys).  Inside a block
//   kd_t = k_t * P_t, qd_t = q_t * P_t      (P_t: product of the block's decays up to and with token t)
//   kh_t = k_t * (product of the decays behind t),   A_ts = k_t . (k_s * decays of s+1 .. t),   B_ts likewise with q_t
// do not depend on the state, so a warp forms them once per block for all columns of the CTA, and per state column
//   d_t = beta_t (v_t - kd_t . S0 - sum_{s<t} A_ts d_s),   o_t = qd_t . S0 + sum_{s<=t} B_ts d_s,
//   S   = (all decays) * S0 + sum_t kh_t d_t
// Everything stays f32 (products of decays only, no quotients, so nothing can overflow).  Against the token-by-token walk
// this takes 3.25 multiply-adds per state element and token instead of 4, and one reduction, one solve per KB_T tokens.
// A lane holds 16 rows x 4 columns of the state as row pairs for the packed f32x2 instructions; the 8 lanes of a column
// group read 128 contiguous bytes of a vector at a time, which is what the walk, with 32 elements of one column per thread,
// was short of: shared-memory reads (three vectors per 32 elements and token there, 13 per 64 elements and 4 tokens here).
// 3001 tokens in two prompts, 96 heads: 2550 us before, 1145 us now; 16 heads, one prompt of 3000: 1644 and 1099.  Decode rows
// beside a prompt stay on the walk (64 rows and 300 tokens, 96 heads: 398 us with every row in a block of four, 333 now).  What bounds it: FMA issue and shared-memory reads
// (both near half of their rate) by warps that wait for their own sums, few of them where a step has few sequences.
constexpr int KB_T = 4;        // tokens per block
constexpr int KB_BLOCKS = 4;   // blocks per stage: one per warp to prepare
constexpr int KB_COLS = 64;    // state columns per CTA, 16 per warp
constexpr int KB_DK = 128;

struct KdaBlock {
  float kd[KB_T][KB_DK], qd[KB_T][KB_DK], kh[KB_T][KB_DK], dp[KB_DK];
  float v[KB_T][KB_COLS];
  float ab[16];  // A_ts at t (t - 1) / 2 + s, B_ts at 6 + t (t + 1) / 2 + s
  float beta[KB_T];
};
struct KdaBlockSmem {  // 47 KB: no attribute needed
  KdaBlock blk[KB_BLOCKS];
  bf16 raw[KB_BLOCKS][3][KB_T][KB_DK];  // q, k, f rows of the stage after this one
  bf16 raw_v[KB_BLOCKS][KB_T][KB_COLS];
  float u[4][KB_T][16], o[4][KB_T][16];  // per warp: kd . S0, then d; qd . S0
};

static_assert(sizeof(KdaBlockSmem) <= 48 * 1024, "more needs the kernel's attribute, on every device");
__device__ __forceinline__ unsigned long long kb_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long kb_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long kb_pair(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 kb_split(unsigned long long a) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(a));
  return f;
}
// Sum over lanes of N values per lane, scattered: every step halves the values a lane still carries.  Bit `top` of the lane
// picks the upper half first.
template <int N>
__device__ __forceinline__ void kb_reduce_scatter(float* v, int lane, int top) {
#pragma unroll
  for (int n = N / 2, bit = top; n > 0 && bit > 0; n >>= 1, bit >>= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const float send = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
}

__global__ void __launch_bounds__(128, 3)
kda_block_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, long long ld, const bf16* __restrict__ f, long long ldf, const bf16* __restrict__ b, long long ldb,
                 const float* __restrict__ a_log, const float* __restrict__ dt_bias, float lower, float* __restrict__ state, bf16* __restrict__ out, const int* __restrict__ q_indptr,
                 const int* __restrict__ slots, int heads, int dv, int min_len) {
  extern __shared__ __align__(16) uint8_t kb_raw[];
  KdaBlockSmem& sm = *reinterpret_cast<KdaBlockSmem*>(kb_raw);
  const int groups = dv / KB_COLS;
  const int h = blockIdx.x / groups, c0 = blockIdx.x % groups * KB_COLS, seq = blockIdx.y;
  const int slot = slots[seq];
  const int q0 = q_indptr[seq], q1 = q_indptr[seq + 1];
  if (q1 - q0 < min_len || slot < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane & 7, cg = lane >> 3;
  const int col = c0 + warp * 16 + cg * 4;  // the lane's first state column
  float* S = state + ((long long)slot * heads + h) * KB_DK * dv;

  // raw rows of this warp's block of the stage that starts at token t0; rows past the end are zero
  float b_next = 0.f;
  auto fetch = [&](int t0) {
    const int t = t0 + warp * KB_T;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int c = lane + 32 * (i & 1), r = c >> 4, ch = (c & 15) * 8;
      const bool ok = t + r < q1;
      const long long row = ok ? t + r : q0;
      const bf16* src = i < 2 ? q + row * ld : i < 4 ? k + row * ld : f + row * ldf;
      cp_async16(&sm.raw[warp][i >> 1][r][ch], src + (long long)h * KB_DK + ch, ok);
    }
    const int r = lane >> 3, ch = (lane & 7) * 8;
    const bool ok = t + r < q1;
    cp_async16(&sm.raw_v[warp][r][ch], v + (ok ? t + r : q0) * ld + (long long)h * dv + c0 + ch, ok);
    cp_async_commit();
    b_next = lane < KB_T && t + lane < q1 ? to_f32(b[(long long)(t + lane) * ldb + h]) : 0.f;
  };
  fetch(q0);

  unsigned long long s2[4][2][4];  // rows 32 i + 4 rg + {0, 1} and {2, 3}, columns col .. col + 3
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float4 lo = *reinterpret_cast<const float4*>(S + (long long)(32 * i + 4 * rg + 2 * p) * dv + col);
      const float4 hi = *reinterpret_cast<const float4*>(S + (long long)(32 * i + 4 * rg + 2 * p + 1) * dv + col);
      s2[i][p][0] = kb_pair(lo.x, hi.x);
      s2[i][p][1] = kb_pair(lo.y, hi.y);
      s2[i][p][2] = kb_pair(lo.z, hi.z);
      s2[i][p][3] = kb_pair(lo.w, hi.w);
    }
  const float a = __expf(a_log[h]), q_scale = rsqrtf((float)KB_DK);

  for (int t0 = q0; t0 < q1; t0 += KB_T * KB_BLOCKS) {
    // ---- each warp prepares one block; a lane has four key channels of its four tokens ----
    cp_async_wait_all();
    __syncwarp();
    {
      KdaBlock& B = sm.blk[warp];
      const int first = t0 + warp * KB_T;
      float kk[KB_T][4], qq[KB_T][4], dec[KB_T][4];
      const float4 db = *reinterpret_cast<const float4*>(dt_bias + h * KB_DK + lane * 4);
      const float bias[4] = {db.x, db.y, db.z, db.w};
#pragma unroll
      for (int t = 0; t < KB_T; ++t) {
        float x[3][4], qs = 0.f, ks = 0.f;
#pragma unroll
        for (int w = 0; w < 3; ++w) {
          const uint2 raw = *reinterpret_cast<const uint2*>(&sm.raw[warp][w][t][lane * 4]);
          const float2 lo = __bfloat1622float2(*reinterpret_cast<const bf162*>(&raw.x)), hi = __bfloat1622float2(*reinterpret_cast<const bf162*>(&raw.y));
          x[w][0] = lo.x, x[w][1] = lo.y, x[w][2] = hi.x, x[w][3] = hi.y;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          qs += x[0][e] * x[0][e];
          ks += x[1][e] * x[1][e];
        }
        qs = warp_sum(qs);
        ks = warp_sum(ks);
        const float qn = rsqrtf(qs + 1e-6f) * q_scale, kn = rsqrtf(ks + 1e-6f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          qq[t][e] = x[0][e] * qn;
          kk[t][e] = x[1][e] * kn;
          const float raw = x[2][e] + bias[e];
          dec[t][e] = first + t < q1 ? __expf(lower / (1.f + __expf(-a * raw))) : 1.f;
        }
      }
      float ab[16], w[KB_T][4];
#pragma unroll
      for (int s = 0; s < KB_T; ++s) {
#pragma unroll
        for (int e = 0; e < 4; ++e) w[s][e] = kk[s][e];
#pragma unroll
        for (int t = s; t < KB_T; ++t) {  // w[s] = k_s times the decays of s + 1 .. t
          float x = 0.f, y = 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (t > s) w[s][e] *= dec[t][e];
            x += kk[t][e] * w[s][e];
            y += qq[t][e] * w[s][e];
          }
          if (t > s) ab[t * (t - 1) / 2 + s] = x;
          ab[6 + t * (t + 1) / 2 + s] = y;
        }
        *reinterpret_cast<float4*>(&B.kh[s][lane * 4]) = make_float4(w[s][0], w[s][1], w[s][2], w[s][3]);
      }
      float cum[4] = {1.f, 1.f, 1.f, 1.f};
#pragma unroll
      for (int t = 0; t < KB_T; ++t) {
#pragma unroll
        for (int e = 0; e < 4; ++e) cum[e] *= dec[t][e];
        *reinterpret_cast<float4*>(&B.kd[t][lane * 4]) = make_float4(kk[t][0] * cum[0], kk[t][1] * cum[1], kk[t][2] * cum[2], kk[t][3] * cum[3]);
        *reinterpret_cast<float4*>(&B.qd[t][lane * 4]) = make_float4(qq[t][0] * cum[0], qq[t][1] * cum[1], qq[t][2] * cum[2], qq[t][3] * cum[3]);
        const float2 vv = __bfloat1622float2(*reinterpret_cast<const bf162*>(&sm.raw_v[warp][t][lane * 2]));
        *reinterpret_cast<float2*>(&B.v[t][lane * 2]) = vv;
      }
      *reinterpret_cast<float4*>(&B.dp[lane * 4]) = make_float4(cum[0], cum[1], cum[2], cum[3]);
      kb_reduce_scatter<16>(ab, lane, 16);
      ab[0] += __shfl_xor_sync(0xffffffffu, ab[0], 1);
      if (!(lane & 1)) B.ab[lane >> 1] = ab[0];
      if (lane < KB_T) B.beta[lane] = first + lane < q1 ? 1.f / (1.f + __expf(-b_next)) : 0.f;
    }
    __syncthreads();
    if (t0 + KB_T * KB_BLOCKS < q1) fetch(t0 + KB_T * KB_BLOCKS);

    // ---- every warp walks the stage's blocks over its 16 columns ----
    const int blocks = min(KB_BLOCKS, (q1 - t0 + KB_T - 1) / KB_T);
#pragma unroll 1
    for (int n = 0; n < blocks; ++n) {
      const KdaBlock& B = sm.blk[n];
      unsigned long long ak[KB_T][4], aq[KB_T][4];
#pragma unroll
      for (int t = 0; t < KB_T; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) ak[t][c] = aq[t][c] = 0ull;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int t = 0; t < KB_T; ++t) {
          const ulonglong2 x = reinterpret_cast<const ulonglong2*>(B.kd[t])[i * 8 + rg], y = reinterpret_cast<const ulonglong2*>(B.qd[t])[i * 8 + rg];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            ak[t][c] = kb_fma2(s2[i][1][c], x.y, kb_fma2(s2[i][0][c], x.x, ak[t][c]));
            aq[t][c] = kb_fma2(s2[i][1][c], y.y, kb_fma2(s2[i][0][c], y.x, aq[t][c]));
          }
        }
      float sum[32];  // a token's four columns of kd, then of qd
#pragma unroll
      for (int t = 0; t < KB_T; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 x = kb_split(ak[t][c]), y = kb_split(aq[t][c]);
          sum[t * 8 + c] = x.x + x.y;
          sum[t * 8 + 4 + c] = y.x + y.y;
        }
      // over the eight row groups (lane bits 0 .. 2): four columns of one token's kd or qd are left to each lane
      kb_reduce_scatter<32>(sum, lane, 4);
      *reinterpret_cast<float4*>(lane & 1 ? &sm.o[warp][(lane >> 1) & 3][cg * 4] : &sm.u[warp][(lane >> 1) & 3][cg * 4]) = make_float4(sum[0], sum[1], sum[2], sum[3]);
      __syncwarp();
      {
        const int c = lane & 15;  // lanes l and l + 16 solve the same column
        const float4 be = *reinterpret_cast<const float4*>(B.beta);
        float ab[16];
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(ab + i) = *reinterpret_cast<const float4*>(B.ab + i);
        const float d0 = be.x * (B.v[0][warp * 16 + c] - sm.u[warp][0][c]);
        const float d1 = be.y * (B.v[1][warp * 16 + c] - sm.u[warp][1][c] - ab[0] * d0);
        const float d2 = be.z * (B.v[2][warp * 16 + c] - sm.u[warp][2][c] - ab[1] * d0 - ab[2] * d1);
        const float d3 = be.w * (B.v[3][warp * 16 + c] - sm.u[warp][3][c] - ab[3] * d0 - ab[4] * d1 - ab[5] * d2);
        const float o0 = sm.o[warp][0][c] + ab[6] * d0;
        const float o1 = sm.o[warp][1][c] + ab[7] * d0 + ab[8] * d1;
        const float o2 = sm.o[warp][2][c] + ab[9] * d0 + ab[10] * d1 + ab[11] * d2;
        const float o3 = sm.o[warp][3][c] + ab[12] * d0 + ab[13] * d1 + ab[14] * d2 + ab[15] * d3;
        const int t = t0 + n * KB_T + (lane >> 4) * 2;
        bf16* dst = out + ((long long)t * heads + h) * dv + c0 + warp * 16 + c;
        if (t < q1) dst[0] = __float2bfloat16(lane < 16 ? o0 : o2);
        if (t + 1 < q1) dst[(long long)heads * dv] = __float2bfloat16(lane < 16 ? o1 : o3);
        __syncwarp();  // both lanes of a column have read u
        if (lane < 16) {
          sm.u[warp][0][c] = d0;
          sm.u[warp][1][c] = d1;
          sm.u[warp][2][c] = d2;
          sm.u[warp][3][c] = d3;
        }
      }
      __syncwarp();
      unsigned long long d2[KB_T][4];
#pragma unroll
      for (int t = 0; t < KB_T; ++t) {
        const float4 x = *reinterpret_cast<const float4*>(&sm.u[warp][t][cg * 4]);
        d2[t][0] = kb_pair(x.x, x.x);
        d2[t][1] = kb_pair(x.y, x.y);
        d2[t][2] = kb_pair(x.z, x.z);
        d2[t][3] = kb_pair(x.w, x.w);
      }
      __syncwarp();  // d is read; the next block may put its sums there
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 x = reinterpret_cast<const ulonglong2*>(B.dp)[i * 8 + rg];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          s2[i][0][c] = kb_mul2(s2[i][0][c], x.x);
          s2[i][1][c] = kb_mul2(s2[i][1][c], x.y);
        }
#pragma unroll
        for (int t = 0; t < KB_T; ++t) {
          const ulonglong2 y = reinterpret_cast<const ulonglong2*>(B.kh[t])[i * 8 + rg];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            s2[i][0][c] = kb_fma2(y.x, d2[t][c], s2[i][0][c]);
            s2[i][1][c] = kb_fma2(y.y, d2[t][c], s2[i][1][c]);
          }
        }
      }
    }
    __syncthreads();  // the blocks may be written again
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      float2 x[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) x[c] = kb_split(s2[i][p][c]);
      *reinterpret_cast<float4*>(S + (long long)(32 * i + 4 * rg + 2 * p) * dv + col) = make_float4(x[0].x, x[1].x, x[2].x, x[3].x);
      *reinterpret_cast<float4*>(S + (long long)(32 * i + 4 * rg + 2 * p + 1) * dv + col) = make_float4(x[0].y, x[1].y, x[2].y, x[3].y);
    }
}

constexpr int ATTNRES_MAX = 16;  // candidates of one mix (snapshots + the current row)

// One CTA of 256 threads per token.  Pass 1: sum of squares and dot with score_w for every candidate; pass 2: softmax of
// the scores and the weighted sum (the rows come back from L1 / L2).
__global__ void __launch_bounds__(256) attnres_mix_kernel(const bf16* __restrict__ cur, long long ld_cur, const bf16* __restrict__ snaps, long long ld_tok,
                                                           const float* __restrict__ score_w, bf16* __restrict__ out, long long ld_out, int nb, int hidden,
                                                           float eps) {
  PG_PDL_ENTRY();
  __shared__ float red[2][ATTNRES_MAX][8];
  __shared__ float prob[ATTNRES_MAX];
  const long long t = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nvec = hidden / 8;
  const int nc = nb + 1;
  auto row = [&](int c) { return c < nb ? snaps + t * ld_tok + (long long)c * hidden : cur + t * ld_cur; };
  for (int c = 0; c < nc; ++c) {
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(row(c));
    float ss = 0.f, dot = 0.f;
    for (int i = tid; i < nvec; i += 256) {
      float x[8];
      unpack8(xr[i], x);
      const float4 w0 = reinterpret_cast<const float4*>(score_w)[2 * i], w1 = reinterpret_cast<const float4*>(score_w)[2 * i + 1];
      ss += x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3] + x[4] * x[4] + x[5] * x[5] + x[6] * x[6] + x[7] * x[7];
      dot += x[0] * w0.x + x[1] * w0.y + x[2] * w0.z + x[3] * w0.w + x[4] * w1.x + x[5] * w1.y + x[6] * w1.z + x[7] * w1.w;
    }
    ss = warp_sum(ss);
    dot = warp_sum(dot);
    if (lane == 0) red[0][c][warp] = ss, red[1][c][warp] = dot;
  }
  __syncthreads();
  if (tid == 0) {
    float sc[ATTNRES_MAX], mx = -1e30f, den = 0.f;
    for (int c = 0; c < nc; ++c) {
      float ss = 0.f, dot = 0.f;
      for (int w = 0; w < 8; ++w) ss += red[0][c][w], dot += red[1][c][w];
      sc[c] = dot * rsqrtf(ss / (float)hidden + eps);
      mx = fmaxf(mx, sc[c]);
    }
    for (int c = 0; c < nc; ++c) den += (sc[c] = __expf(sc[c] - mx));
    for (int c = 0; c < nc; ++c) prob[c] = sc[c] / den;
  }
  __syncthreads();
  for (int i = tid; i < nvec; i += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < nc; ++c) {
      float x[8];
      unpack8(reinterpret_cast<const bf16x8*>(row(c))[i], x);
      const float p = prob[c];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += p * x[j];
    }
    reinterpret_cast<bf16x8*>(out + t * ld_out)[i] = pack8(acc);
  }
}

}  // namespace

// Sequences of min_len tokens and more go four tokens at a time where rows and state are runs of 16-byte pieces, shorter ones (of
// up to `short_len` tokens; 0: there are none) token by token in a launch of their own, so that a decode row beside a prompt is
// what it is in a step of decode rows.
extern "C" int pg_kda_recurrent(const void* q, const void* k, const void* v, long long ld, const void* f, long long ldf, const void* b, long long ldb,
                                const void* a_log, const void* dt_bias, float lower, void* state, void* out, const void* q_indptr, const void* slots,
                                int num_seqs, int heads, int dk, int dv, int max_q_len, int min_len, int short_len, cudaStream_t stream) {
  PG_REQUIRE(dv <= 128 && lower < 0.f, "kda_recurrent: dv=%d must be <= 128 and the decay lower bound %f negative", dv, (double)lower);
  PG_REQUIRE(min_len >= 1, "kda_recurrent: blocks for sequences of %d tokens", min_len);
  if (num_seqs == 0) return PG_OK;
  RecArgs<bf16> p = {(const bf16*)q, (const bf16*)k, (const bf16*)v, ld, f, ldf, (const bf16*)b, ldb, (const float*)a_log, (const float*)dt_bias, nullptr, lower,
                     (float*)state, (bf16*)out, (const int*)q_indptr, (const int*)slots, heads, heads, dk, dv, (dv + KDA_COLS - 1) / KDA_COLS, 0};
  const bool blocks = max_q_len >= min_len && dk == KB_DK && dv % KB_COLS == 0 && ld % 8 == 0 && ldf % 8 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)f | (uintptr_t)dt_bias | (uintptr_t)state) & 15) == 0;
  if (blocks) {
    kda_block_kernel<<<dim3(heads * (dv / KB_COLS), num_seqs), 128, sizeof(KdaBlockSmem), stream>>>(p.q, p.k, p.v, ld, (const bf16*)f, ldf, p.b, ldb, p.a_log, p.dt_bias, lower, p.state, p.out, p.q_indptr, p.slots,
                                                                                                     heads, dv, min_len);
    PG_LAUNCH_CHECK();
    if (short_len <= 0) return PG_OK;
    p.skip_len = min_len;
  }
  const dim3 grid(heads * p.col_groups, num_seqs);
  const bool few = (blocks ? short_len : max_q_len) <= 4;
  if (dk == 128)
    PG_CUDA((launch_rule<bf16, 128, RULE_BOUNDED, false>(p, grid, few, stream)));
  else if (dk == 64)
    PG_CUDA((launch_rule<bf16, 64, RULE_BOUNDED, false>(p, grid, few, stream)));
  else if (dk == 32)
    PG_CUDA((launch_rule<bf16, 32, RULE_BOUNDED, false>(p, grid, few, stream)));
  else {
    pg_set_error("kda_recurrent: dk=%d not supported (32, 64, 128)", dk);
    return PG_ERR_UNSUPPORTED;
  }
  PG_LAUNCH_CHECK();
  return PG_OK;
}

// The delta rule with the decay exp(-exp(A_log) * softplus(f + dt_bias)), f in f32, and query / key heads that several
// value heads may share.
extern "C" int pg_channel_delta(const void* q, const void* k, const void* v, long long ld, const void* f, long long ldf, const void* b, long long ldb, const void* a_log, const void* dt_bias,
                                void* state, void* out, const void* q_indptr, const void* slots, int num_seqs, int heads, int kv_heads, int dk, int dv, int max_q_len, int skip_len, int is_f32,
                                cudaStream_t stream) {
  PG_REQUIRE(dk >= 1 && dk <= 256 && dv >= 1 && heads % kv_heads == 0, "channel_delta: heads %d / %d, key width %d (at most 256), value width %d", heads, kv_heads, dk, dv);
  PG_REQUIRE(num_seqs <= 65535, "channel_delta: %d sequences", num_seqs);
  if (num_seqs == 0) return PG_OK;
  if (is_f32) {
    RecArgs<float> p = {(const float*)q, (const float*)k, (const float*)v, ld, f, ldf, (const float*)b, ldb, (const float*)a_log, (const float*)dt_bias, nullptr, 0.f,
                        (float*)state, (float*)out, (const int*)q_indptr, (const int*)slots, heads, kv_heads, dk, dv, 0, skip_len};
    return run_rule<float>(RULE_SOFTPLUS, p, num_seqs, max_q_len, stream);
  }
  RecArgs<bf16> p = {(const bf16*)q, (const bf16*)k, (const bf16*)v, ld, f, ldf, (const bf16*)b, ldb, (const float*)a_log, (const float*)dt_bias, nullptr, 0.f,
                     (float*)state, (bf16*)out, (const int*)q_indptr, (const int*)slots, heads, kv_heads, dk, dv, 0, skip_len};
  return run_rule<bf16>(RULE_SOFTPLUS, p, num_seqs, max_q_len, stream);
}

// Linear attention with a fixed decay per head: S <- decay S + k v^T, o = S^T q, with SiLU on q, k and v inside.
extern "C" int pg_decay_recurrent(const void* q, const void* k, const void* v, long long ld, const void* decay, void* state, void* out, const void* q_indptr, const void* slots, int num_seqs,
                                  int heads, int dk, int dv, int max_q_len, int skip_len, int is_f32, cudaStream_t stream) {
  PG_REQUIRE(dk >= 1 && dk <= 256 && dv >= 1, "decay_recurrent: key width %d (at most 256), value width %d", dk, dv);
  PG_REQUIRE(num_seqs <= 65535, "decay_recurrent: %d sequences", num_seqs);
  if (num_seqs == 0) return PG_OK;
  if (is_f32) {
    RecArgs<float> p = {(const float*)q, (const float*)k, (const float*)v, ld, nullptr, 0, nullptr, 0, nullptr, nullptr, (const float*)decay, 0.f,
                        (float*)state, (float*)out, (const int*)q_indptr, (const int*)slots, heads, heads, dk, dv, 0, skip_len};
    return run_rule<float>(RULE_DECAY, p, num_seqs, max_q_len, stream);
  }
  RecArgs<bf16> p = {(const bf16*)q, (const bf16*)k, (const bf16*)v, ld, nullptr, 0, nullptr, 0, nullptr, nullptr, (const float*)decay, 0.f,
                     (float*)state, (bf16*)out, (const int*)q_indptr, (const int*)slots, heads, heads, dk, dv, 0, skip_len};
  return run_rule<bf16>(RULE_DECAY, p, num_seqs, max_q_len, stream);
}

// Linear attention with the decay exp(-exp(f + w0)) per token and key channel (f in f32) and the bonus u [heads, dk] for the
// current token: o = (S + diag(u) k v^T)^T r, then S <- diag(decay) S + k v^T.
extern "C" int pg_wkv_recurrent(const void* r, const void* k, const void* v, long long ld, const void* f, long long ldf, const void* w0, const void* u, void* state, void* out, const void* q_indptr,
                                const void* slots, int num_seqs, int heads, int dk, int dv, int max_q_len, int skip_len, int is_f32, cudaStream_t stream) {
  PG_REQUIRE(dk >= 1 && dk <= 256 && dv >= 1, "wkv_recurrent: key width %d (at most 256), value width %d", dk, dv);
  PG_REQUIRE(num_seqs <= 65535, "wkv_recurrent: %d sequences", num_seqs);
  if (num_seqs == 0) return PG_OK;
  if (is_f32) {
    RecArgs<float> p = {(const float*)r, (const float*)k, (const float*)v, ld, f, ldf, nullptr, 0, nullptr, (const float*)w0, (const float*)u, 0.f,
                        (float*)state, (float*)out, (const int*)q_indptr, (const int*)slots, heads, heads, dk, dv, 0, skip_len};
    return run_rule<float>(RULE_WKV, p, num_seqs, max_q_len, stream);
  }
  RecArgs<bf16> p = {(const bf16*)r, (const bf16*)k, (const bf16*)v, ld, f, ldf, nullptr, 0, nullptr, (const float*)w0, (const float*)u, 0.f,
                     (float*)state, (bf16*)out, (const int*)q_indptr, (const int*)slots, heads, heads, dk, dv, 0, skip_len};
  return run_rule<bf16>(RULE_WKV, p, num_seqs, max_q_len, stream);
}

// State-space duality: x [T, heads, dv] rows of stride ld, B and C [T, groups, n] rows of the same stride, dt [T, heads] raw step sizes of
// stride lddt; d = softplus(dt + dt_bias): S <- exp(-exp(a_log) d) S + d B x^T, out = S^T C + D x.
extern "C" int pg_ssd_recurrent(const void* C, const void* B, const void* x, long long ld, const void* dt, long long lddt, const void* a_log, const void* dt_bias, const void* D, void* state, void* out,
                                const void* q_indptr, const void* slots, int num_seqs, int heads, int groups, int n, int dv, int max_q_len, int skip_len, int is_f32, cudaStream_t stream) {
  PG_REQUIRE(n >= 1 && n <= 256 && dv >= 1 && heads % groups == 0, "ssd_recurrent: heads %d / %d, state width %d (at most 256), value width %d", heads, groups, n, dv);
  PG_REQUIRE(num_seqs <= 65535, "ssd_recurrent: %d sequences", num_seqs);
  if (num_seqs == 0) return PG_OK;
  if (is_f32) {
    RecArgs<float> p = {(const float*)C, (const float*)B, (const float*)x, ld, dt, lddt, nullptr, 0, (const float*)a_log, (const float*)dt_bias, (const float*)D, 0.f,
                        (float*)state, (float*)out, (const int*)q_indptr, (const int*)slots, heads, groups, n, dv, 0, skip_len};
    return run_rule<float>(RULE_SSD, p, num_seqs, max_q_len, stream);
  }
  RecArgs<bf16> p = {(const bf16*)C, (const bf16*)B, (const bf16*)x, ld, dt, lddt, nullptr, 0, (const float*)a_log, (const float*)dt_bias, (const float*)D, 0.f,
                     (float*)state, (bf16*)out, (const int*)q_indptr, (const int*)slots, heads, groups, n, dv, 0, skip_len};
  return run_rule<bf16>(RULE_SSD, p, num_seqs, max_q_len, stream);
}

extern "C" int pg_attnres_mix(const void* cur, long long ld_cur, const void* snaps, long long ld_tok, const void* score_w, void* out, long long ld_out,
                              int tokens, int nb, int hidden, float eps, cudaStream_t stream) {
  PG_REQUIRE(nb >= 0 && nb + 1 <= ATTNRES_MAX && hidden % 8 == 0 && ld_cur % 8 == 0 && ld_tok % 8 == 0 && ld_out % 8 == 0,
             "attnres_mix: %d snapshots (at most %d) and a hidden size %d that is a multiple of 8", nb, ATTNRES_MAX - 1, hidden);
  if (tokens == 0) return PG_OK;
  PG_CUDA(launch_pdl(attnres_mix_kernel, dim3(tokens), dim3(256), (size_t)(0), stream, (const bf16*)cur, ld_cur, (const bf16*)snaps, ld_tok,
                     (const float*)score_w, (bf16*)out, ld_out, nb, hidden, eps));
  PG_LAUNCH_CHECK();
  return PG_OK;
}
