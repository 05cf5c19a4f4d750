// Token selection kernels over logits rows [rows, vocab] (bf16 or f32).
//
//  * argmax: split partial/finalize, ties resolve to the lowest index; writes int32
//    tokens straight into the caller's buffer (the next decode step's input under a
//    CUDA graph).
//  * sample: one thread-block cluster per row (sample_cluster_kernel, below); the one-CTA kernel
//    described here serves vocabularies too large for eight CTAs' shared memory.  Online softmax at the row's temperature, then the
//    keep-set {top-k AND top-p AND min-p} is found as a threshold on the scaled logit
//    by a 4-level byte-radix descent carrying (count, mass) of everything above, and
//    the token is drawn by inverse CDF in vocabulary order from one uniform per row,
//    so a replay with the same uniform is bit-reproducible.
//  * logprob_topk: log-softmax of the picked token plus the k best alternatives.
//
// Functional parity with pegainfer-kernels/csrc/shared/argmax.cu:91-230,
// flashinfer_sampling.cu:69-149 (softmax -> top-k/top-p/min-p sampling) and
// logprob_topk.cu:13-123.
#include <float.h>

#include "api.h"
#include "common.cuh"

namespace {

template <typename T>
__device__ __forceinline__ float ldf(const T* p, long long i);
template <>
__device__ __forceinline__ float ldf<bf16>(const bf16* p, long long i) {
  return __bfloat162float(p[i]);
}
template <>
__device__ __forceinline__ float ldf<float>(const float* p, long long i) {
  return p[i];
}

constexpr int ARG_TILE = 4096;

struct ArgPair {
  float v;
  int i;
};
__device__ __forceinline__ ArgPair arg_better(ArgPair a, ArgPair b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ __forceinline__ ArgPair block_argmax(ArgPair a, ArgPair* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = arg_better(a, b);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = a;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  ArgPair t = lane < nw ? red[lane] : ArgPair{-FLT_MAX, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair b;
    b.v = __shfl_xor_sync(0xffffffffu, t.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, t.i, o);
    t = arg_better(t, b);
  }
  return t;
}

template <typename T>
__global__ void __launch_bounds__(256) argmax_partial_kernel(const T* __restrict__ logits, long long ld, int vocab, ArgPair* __restrict__ partial,
                                                              int tiles) {
  PG_PDL_ENTRY();
  __shared__ ArgPair red[32];
  const int row = blockIdx.y, tile = blockIdx.x;
  const T* r = logits + row * ld;
  ArgPair best{-FLT_MAX, 0x7fffffff};
  const int end = min(vocab, (tile + 1) * ARG_TILE);
  for (int i = tile * ARG_TILE + threadIdx.x; i < end; i += 256) {
    float v = ldf(r, i);
    if (v > best.v) best = ArgPair{v, i};  // ascending i per thread keeps the lowest index on ties
  }
  best = block_argmax(best, red);
  if (threadIdx.x == 0) partial[(long long)row * tiles + tile] = best;
}

__global__ void __launch_bounds__(128) argmax_final_kernel(const ArgPair* __restrict__ partial, int tiles, int* __restrict__ out) {
  PG_PDL_ENTRY();
  __shared__ ArgPair red[32];
  const int row = blockIdx.x;
  ArgPair best{-FLT_MAX, 0x7fffffff};
  for (int i = threadIdx.x; i < tiles; i += 128) best = arg_better(best, partial[(long long)row * tiles + i]);
  best = block_argmax(best, red);
  if (threadIdx.x == 0) out[row] = best.i;
}

// One step of a low-rank Markov head over block-drafted logits: row r scores token v with
// base[(r * block + step) * ld + v] + bias[r * ldb + v] (bias = w2 . w1[previous token]); the best
// token becomes the row's previous token for the next step and entry (r, step) of the drafts.
template <typename T>
__global__ void __launch_bounds__(256) markov_partial_kernel(const T* __restrict__ base, long long ld, int block, int step, const T* __restrict__ bias,
                                                              long long ldb, int vocab, ArgPair* __restrict__ partial, int tiles) {
  PG_PDL_ENTRY();
  __shared__ ArgPair red[32];
  const int row = blockIdx.y, tile = blockIdx.x;
  const T* r = base + ((long long)row * block + step) * ld;
  const T* b = bias + (long long)row * ldb;
  ArgPair best{-FLT_MAX, 0x7fffffff};
  const int end = min(vocab, (tile + 1) * ARG_TILE);
  for (int i = tile * ARG_TILE + threadIdx.x; i < end; i += 256) {
    float v = ldf(r, i) + ldf(b, i);
    if (v > best.v) best = ArgPair{v, i};
  }
  best = block_argmax(best, red);
  if (threadIdx.x == 0) partial[(long long)row * tiles + tile] = best;
}

__global__ void __launch_bounds__(128) markov_final_kernel(const ArgPair* __restrict__ partial, int tiles, int* __restrict__ next, int* __restrict__ drafts,
                                                            int block, int step) {
  PG_PDL_ENTRY();
  __shared__ ArgPair red[32];
  const int row = blockIdx.x;
  ArgPair best{-FLT_MAX, 0x7fffffff};
  for (int i = threadIdx.x; i < tiles; i += 128) best = arg_better(best, partial[(long long)row * tiles + i]);
  best = block_argmax(best, red);
  if (threadIdx.x == 0) {
    next[row] = best.i;
    drafts[(long long)row * block + step] = best.i;
  }
}

// order-preserving float -> uint
__device__ __forceinline__ uint32_t fkey(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int ST = 1024;  // sampler threads

__device__ __forceinline__ float block_sum_f(float v, float* red) { return block_sum(v, red); }
__device__ __forceinline__ float block_max_f(float v, float* red) {
  v = warp_max(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = lane < (int)((blockDim.x + 31) >> 5) ? red[lane] : -FLT_MAX;
  return warp_max(t);
}

template <typename T>
__global__ void __launch_bounds__(ST) sample_kernel(const T* __restrict__ logits, long long ld, int vocab, const float* __restrict__ temperature,
                                                     const int* __restrict__ top_k, const float* __restrict__ top_p,
                                                     const float* __restrict__ min_p, const float* __restrict__ uniform, int* __restrict__ out) {
  PG_PDL_ENTRY();
  __shared__ float red[32];
  __shared__ uint32_t h_cnt[256];
  __shared__ float h_mass[256];
  __shared__ uint32_t s_prefix, s_cnt_above;
  __shared__ float s_mass_above;
  __shared__ float s_scan[ST];
  __shared__ int s_owner;
  const int row = blockIdx.x;
  const T* r = logits + row * ld;
  const float inv_t = 1.f / fmaxf(temperature[row], 1e-6f);
  const int tid = threadIdx.x;

  // pass 1: max and normaliser of the tempered row
  float m = -FLT_MAX;
  for (int i = tid; i < vocab; i += ST) m = fmaxf(m, ldf(r, i) * inv_t);
  m = block_max_f(m, red);
  float z = 0.f;
  for (int i = tid; i < vocab; i += ST) z += __expf(ldf(r, i) * inv_t - m);
  z = block_sum_f(z, red);

  const int kk = top_k[row] > 0 ? min(top_k[row], vocab) : vocab;
  const float p_lim = top_p[row] >= 1.f ? FLT_MAX : top_p[row] * z;
  const float mp = min_p[row];
  const float minp_thr = mp > 0.f ? m + __logf(mp) : -FLT_MAX;

  // radix descent on the key of the scaled logit: find the smallest kept key
  if (tid == 0) {
    s_prefix = 0;
    s_cnt_above = 0;
    s_mass_above = 0.f;
  }
  __syncthreads();
  for (int level = 0; level < 4; ++level) {
    const int shift = 24 - 8 * level;
    const uint32_t hi_mask = level == 0 ? 0u : (0xffffffffu << (shift + 8));
    if (tid < 256) {
      h_cnt[tid] = 0;
      h_mass[tid] = 0.f;
    }
    __syncthreads();
    const uint32_t prefix = s_prefix;
    for (int i = tid; i < vocab; i += ST) {
      const float s = ldf(r, i) * inv_t;
      const uint32_t key = fkey(s);
      if ((key & hi_mask) == prefix) {
        const uint32_t b = (key >> shift) & 255u;
        atomicAdd(&h_cnt[b], 1u);
        atomicAdd(&h_mass[b], __expf(s - m));
      }
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t cnt = s_cnt_above;
      float mass = s_mass_above;
      int chosen = -1;
      uint32_t c_cnt = cnt;
      float c_mass = mass;
      for (int b = 255; b >= 0; --b) {
        if (h_cnt[b] == 0) continue;
        if (cnt < (uint32_t)kk && mass < p_lim) {
          chosen = b;
          c_cnt = cnt;
          c_mass = mass;
        } else {
          break;
        }
        cnt += h_cnt[b];
        mass += h_mass[b];
      }
      if (chosen < 0) chosen = 255;  // cannot happen: the top element is always kept
      s_prefix = prefix | ((uint32_t)chosen << shift);
      s_cnt_above = c_cnt;
      s_mass_above = c_mass;
    }
    __syncthreads();
  }
  const uint32_t thr_key = max(s_prefix, fkey(minp_thr));

  // inverse CDF in vocabulary order over the kept set: contiguous chunk per thread
  const int chunk = (vocab + ST - 1) / ST;
  const int c0 = min(vocab, tid * chunk), c1 = min(vocab, c0 + chunk);
  float local = 0.f;
  for (int i = c0; i < c1; ++i) {
    const float s = ldf(r, i) * inv_t;
    if (fkey(s) >= thr_key) local += __expf(s - m);
  }
  s_scan[tid] = local;
  __syncthreads();
  // inclusive scan (Hillis-Steele over 1024 entries)
  for (int o = 1; o < ST; o <<= 1) {
    float add = tid >= o ? s_scan[tid - o] : 0.f;
    __syncthreads();
    s_scan[tid] += add;
    __syncthreads();
  }
  const float total = s_scan[ST - 1];
  const float target = uniform[row] * total;
  if (tid == 0) s_owner = ST;
  __syncthreads();
  const float before = tid ? s_scan[tid - 1] : 0.f;
  if (local > 0.f && before <= target && target < s_scan[tid]) atomicMin(&s_owner, tid);
  __syncthreads();
  int owner = s_owner;
  __syncthreads();  // every thread has read the owner before anyone may change it below
  if (owner == ST) {  // uniform across the CTA
    // rounding pushed the target past the end: the last thread holding mass owns it
    if (local > 0.f) atomicMax(&s_owner, tid + ST);
    __syncthreads();
    owner = s_owner - ST;
  }
  if (tid == owner) {
    float acc = before;
    int pick = -1, last_kept = -1;
    for (int i = c0; i < c1; ++i) {
      const float s = ldf(r, i) * inv_t;
      if (fkey(s) >= thr_key) {
        last_kept = i;
        acc += __expf(s - m);
        if (acc > target) {
          pick = i;
          break;
        }
      }
    }
    out[row] = pick >= 0 ? pick : last_kept;
  }
}

// ---------------------------------------------------------------------------------
// Cluster sampler: one thread-block cluster per row.  Each CTA of the cluster reads its slice of the row ONCE into shared
// memory and every later pass runs there, with the per-CTA partial results combined across the cluster through distributed
// shared memory.  A token is represented by e = exp(s - max) in [0, 1], whose bit pattern orders the tokens as their logits
// do.  Probability mass is carried as 2^-40 fixed point in 64-bit integers, so every sum is exact and independent of the
// order in which threads add to it: the same (logits, controls, uniform) always pick the same token, and the CDF target
// floor(u * total) is always strictly inside the kept mass (no rounding fallback).
//
// The threshold of the keep-set is found in two steps.  A histogram of counts over 32 bins per factor of two (tokens below
// 2^-40 have no mass and are left out) brackets it: a bin's count times its edges bounds its mass from both sides, and the
// walk from the top with the lower (upper) bounds ends at or below (above) the bin that the exact walk ends in.  Then the
// mass above the bracket is summed exactly and only the tokens inside it, some hundred as a rule, go through a radix
// descent with counts and masses, which ends after its first level where they are all alike (64 rows of 151936 equal logits: 114 us;
// 237 with the four radix levels of all tokens).  Bound by the latency of the passes and of the eight cluster barriers between them, with
// every row of a batch of 64 resident at once (clusters of four).  64 x 151936 bf16, top-k 50, top-p 0.9: 200 us with all tokens
// taking part in each of four radix levels, one warp match per 32 tokens; 61 us with a key formed for every token in every pass, 47 with those
// passed over whose piece of eight has its largest logit below what the pass looks for (1 row: 33 and 28 us).
// ---------------------------------------------------------------------------------
constexpr int SC_THREADS = 512;
constexpr int SC_WARPS = SC_THREADS / 32;
constexpr int SC_MAX_CLUSTER = 8;
constexpr uint32_t SC_ONE = 0x3f800000u;  // key of e = 1, the largest
constexpr uint32_t SC_LOW = (127u - 40u) << 23;  // key of 2^-40: tokens below have no mass
constexpr int SC_BIN_SHIFT = 18;          // 32 coarse bins per factor of two
constexpr int SC_BINS = (int)((SC_ONE - SC_LOW) >> SC_BIN_SHIFT) + 1;  // 1281
constexpr int SC_BINS_PER_THREAD = (SC_BINS + SC_THREADS - 1) / SC_THREADS;
constexpr int SC_LIST = 1024;             // bracketed tokens kept in a list; more of them are found by walking the slice

// (no memory clobber: several of these are in flight together; the cluster barriers around them have one)
__device__ __forceinline__ unsigned long long ld_dsmem_u64(uint32_t cluster_addr) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(cluster_addr));
  return v;
}
__device__ __forceinline__ uint32_t ld_dsmem_u32(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr));
  return v;
}

struct ScLevel {
  unsigned long long mass[256];
  uint32_t cnt[256];
};
struct ScShared {
  // a level's histogram is read by the peers until the next level's barrier, so two take turns; the coarse counts are
  // read for the last time in front of the first level's barrier
  ScLevel even;
  union {
    ScLevel odd;
    uint32_t coarse[SC_BINS_PER_THREAD * SC_THREADS];
  };
  ScLevel merged;  // the cluster's sum (every CTA forms the same)
  uint32_t list[SC_LIST];
  unsigned long long x_u64[4];  // this CTA's contributions to cluster-wide sums: normaliser, mass and count above the bracket, kept mass
  float x_f32;                  // and to the cluster-wide maximum
  uint32_t list_n, prefix, cnt_above;
  uint32_t own_min, own_max, key_min, key_max;  // least and largest key in the bracket, of this CTA and of the cluster
  int bin_lo, bin_hi;
  unsigned long long mass_above;
  unsigned long long warp_tot[SC_WARPS], warp_ub[SC_WARPS];
  uint32_t warp_cnt[SC_WARPS];
};

// floor(e * 2^40) of a token by its bits (2^-40 <= e < 2^24), in integer instructions: a conversion to 64 bits takes several
// times as long as the rest of a token's work
__device__ __forceinline__ unsigned long long sc_fx(uint32_t key) {
  const uint32_t mant = (key & 0x7fffffu) | 0x800000u, hi = mant >> 15, lo = mant << 17;
  const int r = 127 - (int)(key >> 23);  // (hi, lo) = mantissa * 2^17, shifted right by 0 .. 40 (left, where e is 2 and more)
  if (r < 0) return (unsigned long long)mant << (17 - r);
  const uint32_t both = __funnelshift_r(lo, hi, r), high = hi >> (r & 31);
  return r & 32 ? (unsigned long long)high : (unsigned long long)high << 32 | both;
}

// Largest of the logits in 16 bytes; a NaN only where all are.
template <typename T>
__device__ __forceinline__ float sc_max(const uint4& x);
template <>
__device__ __forceinline__ float sc_max<bf16>(const uint4& x) {
  const bf162* p = reinterpret_cast<const bf162*>(&x);
  const bf162 a = __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3]));
  return fmaxf(__low2float(a), __high2float(a));
}
template <>
__device__ __forceinline__ float sc_max<float>(const uint4& x) {
  return fmaxf(fmaxf(__uint_as_float(x.x), __uint_as_float(x.y)), fmaxf(__uint_as_float(x.z), __uint_as_float(x.w)));
}

// Totals of the lanes above this one, of three quantities.
__device__ __forceinline__ void sc_suffix(uint32_t& c, unsigned long long& m, unsigned long long& n, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t cu = __shfl_down_sync(0xffffffffu, c, o);
    const unsigned long long mu = __shfl_down_sync(0xffffffffu, m, o), nu = __shfl_down_sync(0xffffffffu, n, o);
    if (lane + o < 32) {
      c += cu;
      m += mu;
      n += nu;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(SC_THREADS, 2) sample_cluster_kernel(const T* __restrict__ logits, long long ld, int vocab, int slice,
                                                                    const float* __restrict__ temperature, const int* __restrict__ top_k,
                                                                    const float* __restrict__ top_p, const float* __restrict__ min_p,
                                                                    const float* __restrict__ uniform, int* __restrict__ out, int csize) {
  PG_PDL_ENTRY();
  extern __shared__ __align__(16) uint8_t sc_raw[];
  ScShared& sh = *reinterpret_cast<ScShared*>(sc_raw);
  T* vals = reinterpret_cast<T*>(sc_raw + ((sizeof(ScShared) + 15) & ~size_t(15)));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t cr = csize > 1 ? cluster_ctarank() : 0u;
  const int row = blockIdx.x / csize;
  const T* r = logits + row * ld;
  const float inv_t = 1.f / fmaxf(temperature[row], 1e-6f);
  const int i0 = min(vocab, (int)cr * slice), i1 = min(vocab, i0 + slice);
  const int n = i1 - i0;
  __shared__ float red[32];
  auto cluster_barrier = [&]() {
    if (csize > 1) cluster_sync_all(); else __syncthreads();
  };
  // sums over the cluster's CTAs (a lone CTA is a cluster of its own)
  auto sum_u64 = [&](const unsigned long long* at) {
    unsigned long long x[SC_MAX_CLUSTER], t = 0ull;
#pragma unroll
    for (int q = 0; q < SC_MAX_CLUSTER; ++q) x[q] = q < csize ? ld_dsmem_u64(dsmem_addr(smem_u32(at), (uint32_t)q)) : 0ull;
#pragma unroll
    for (int q = 0; q < SC_MAX_CLUSTER; ++q) t += x[q];
    return t;
  };
  auto sum_u32 = [&](const uint32_t* at) {
    uint32_t x[SC_MAX_CLUSTER], t = 0u;
#pragma unroll
    for (int q = 0; q < SC_MAX_CLUSTER; ++q) x[q] = q < csize ? ld_dsmem_u32(dsmem_addr(smem_u32(at), (uint32_t)q)) : 0u;
#pragma unroll
    for (int q = 0; q < SC_MAX_CLUSTER; ++q) t += x[q];
    return t;
  };

  // the slice into shared memory (slices start at multiples of eight tokens); local max
  float raw = -INFINITY;  // (the largest logit is the largest tempered one: a product with one positive factor keeps the order)
  constexpr int VEC = 16 / sizeof(T);
  int done = 0;
  if (((reinterpret_cast<uintptr_t>(r) | (uintptr_t)(i0 * sizeof(T))) & 15) == 0) {
    done = n / VEC * VEC;
#pragma unroll 4
    for (int i = tid; i < n / VEC; i += SC_THREADS) {
      const uint4 x = reinterpret_cast<const uint4*>(r + i0)[i];
      reinterpret_cast<uint4*>(vals)[i] = x;
      raw = fmaxf(raw, sc_max<T>(x));
    }
  }
  for (int i = done + tid; i < n; i += SC_THREADS) {
    const T x = r[i0 + i];
    vals[i] = x;
    raw = fmaxf(raw, ldf(&x, 0));
  }
  float m = block_max_f(fmaxf(raw * inv_t, -FLT_MAX), red);
  if (tid == 0) {
    sh.x_f32 = m;
    sh.list_n = 0u;
    sh.own_min = SC_ONE;
    sh.own_max = 0u;
    sh.bin_lo = SC_BINS;
    sh.bin_hi = SC_BINS;
  }
#pragma unroll
  for (int j = 0; j < SC_BINS_PER_THREAD; ++j) sh.coarse[tid + j * SC_THREADS] = 0u;
  cluster_barrier();
  if (csize > 1) {
    float mm = -FLT_MAX;
    for (int q = 0; q < csize; ++q) mm = fmaxf(mm, ld_dsmem_f32(dsmem_addr(smem_u32(&sh.x_f32), (uint32_t)q)));
    m = mm;
  }
  // bits of a token's e; the maximum (infinite ones too) has e = 1, a NaN has none
  auto key_of = [&](float logit) -> uint32_t {
    const float s = logit * inv_t;
    const float e = s >= m ? 1.f : __expf(s - m);
    return e > 0.f ? min(__float_as_uint(e), SC_ONE) : 0u;
  };
  // f(keys) for the slice's tokens `from` + VEC * first .. `to`, 16 bytes of them at a time, every `step` pieces; all lanes of a
  // warp come together (tokens behind `to` have key 0) unless there is a cut: lanes whose tokens all lie below it stay away.
  // (What is looked for is mostly some hundred tokens; a key takes some 15 instructions, the largest of eight logits four.)
  auto walk = [&](int from, int to, int first, int step, float cut, auto&& f) {
    for (int b = from + (first - lane) * VEC; b < to; b += step * VEC) {
      const int i = b + lane * VEC;
      const uint4 x = i < to ? *reinterpret_cast<const uint4*>(vals + i) : make_uint4(0u, 0u, 0u, 0u);
      if (sc_max<T>(x) * inv_t - m < cut) continue;
      uint32_t key[VEC];
#pragma unroll
      for (int j = 0; j < VEC; ++j) key[j] = i + j < to ? key_of(ldf(reinterpret_cast<const T*>(&x), j)) : 0u;
      f(key);
    }
  };

  // tokens with s - m below it have keys below `key`, however the logarithm and the exponential round, and the product in s: it may be
  // part of a fused multiply-add, exact beside a maximum that is rounded (2^-24 of it, far above 1e-3 at temperatures of 1e-3 and less)
  auto cut_of = [&](uint32_t key) { return __logf(__uint_as_float(key)) - fmaf(fabsf(m), 0x1p-22f, 1e-3f); };
  const uint32_t kk = top_k[row] > 0 ? (uint32_t)min(top_k[row], vocab) : (uint32_t)vocab;
  const float tp = top_p[row];
  const float mp = min_p[row];
  uint32_t thr_key = 0u;
  if (kk < (uint32_t)vocab || tp < 1.f) {  // the same for the whole cluster: every CTA reads the row's controls
    // ---- coarse counts and the normaliser ----
    unsigned long long z = 0ull;
    walk(0, n, tid, SC_THREADS, -INFINITY, [&](const uint32_t (&key)[VEC]) {
      bool same = key[0] >= SC_LOW;  // (equal logits: one atomic for all of a thread's)
#pragma unroll
      for (int j = 1; j < VEC; ++j) same = same && key[j] == key[0];
      if (same) {
        z += VEC * sc_fx(key[0]);
        atomicAdd(&sh.coarse[(key[0] - SC_LOW) >> SC_BIN_SHIFT], (uint32_t)VEC);
        return;
      }
#pragma unroll
      for (int j = 0; j < VEC; ++j)
        if (key[j] >= SC_LOW) {
          z += sc_fx(key[j]);
          atomicAdd(&sh.coarse[(key[j] - SC_LOW) >> SC_BIN_SHIFT], 1u);
        }
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (lane == 0) sh.warp_tot[warp] = z;
    __syncthreads();
    if (tid == 0) {
      unsigned long long t = 0ull;
      for (int w = 0; w < SC_WARPS; ++w) t += sh.warp_tot[w];
      sh.x_u64[0] = t;
    }
    cluster_barrier();
    z = sum_u64(&sh.x_u64[0]);
    const unsigned long long lim = tp >= 1.f ? ~0ull : (unsigned long long)((double)tp * (double)z);
    // thread t owns bins SC_BINS_PER_THREAD * t ..; walking the bins from the top, a bin is kept while (count above < k) and
    // (mass above < top-p limit); both grow as the bin index falls, so the last one kept is the LOWEST non-empty bin that
    // satisfies them
    uint32_t c[SC_BINS_PER_THREAD], csum = 0u;
    unsigned long long lb[SC_BINS_PER_THREAD], ub[SC_BINS_PER_THREAD], lsum = 0ull, usum = 0ull;
#pragma unroll
    for (int j = 0; j < SC_BINS_PER_THREAD; ++j) {
      const int bin = tid * SC_BINS_PER_THREAD + j;
      c[j] = sum_u32(&sh.coarse[bin]);  // (zero behind the last bin)
      lb[j] = c[j] ? c[j] * sc_fx(SC_LOW + ((uint32_t)bin << SC_BIN_SHIFT)) : 0ull;
      ub[j] = c[j] ? c[j] * sc_fx(SC_LOW + ((uint32_t)(bin + 1) << SC_BIN_SHIFT)) : 0ull;
      csum += c[j];
      lsum += lb[j];
      usum += ub[j];
    }
    uint32_t c_hi = csum;
    unsigned long long l_hi = lsum, u_hi = usum;
    sc_suffix(c_hi, l_hi, u_hi, lane);
    __syncthreads();  // warp_tot is read above
    if (lane == 0) {
      sh.warp_cnt[warp] = c_hi;
      sh.warp_tot[warp] = l_hi;
      sh.warp_ub[warp] = u_hi;
    }
    __syncthreads();
    c_hi -= csum;
    l_hi -= lsum;
    u_hi -= usum;
    for (int w = warp + 1; w < SC_WARPS; ++w) {
      c_hi += sh.warp_cnt[w];
      l_hi += sh.warp_tot[w];
      u_hi += sh.warp_ub[w];
    }
    int lo = SC_BINS, hi = SC_BINS;
#pragma unroll
    for (int j = SC_BINS_PER_THREAD - 1; j >= 0; --j) {
      const int bin = tid * SC_BINS_PER_THREAD + j;
      if (c[j] != 0u && c_hi < kk && l_hi < lim) lo = bin;
      if (c[j] != 0u && c_hi < kk && u_hi < lim) hi = bin;
      c_hi += c[j];
      l_hi += lb[j];
      u_hi += ub[j];
    }
    // (a limit of zero mass keeps no bin by these rules: the top element is always kept)
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_min_sync(0xffffffffu, hi);
    if (lane == 0) {
      atomicMin(&sh.bin_lo, lo);
      atomicMin(&sh.bin_hi, hi);
    }
    __syncthreads();
    lo = sh.bin_lo;
    hi = min(sh.bin_hi, SC_BINS - 1);
    if (lo == SC_BINS) {
      thr_key = SC_ONE;
    } else {
      // ---- exact mass above the bracket lo .. hi, and the tokens inside it ----
      const uint32_t k_lo = SC_LOW + ((uint32_t)lo << SC_BIN_SHIFT), k_hi = SC_LOW + ((uint32_t)(hi + 1) << SC_BIN_SHIFT);  // [k_lo, k_hi)
      unsigned long long above = 0ull;
      uint32_t n_above = 0u;
      uint32_t least = SC_ONE, most = 0u;
      walk(0, n, tid, SC_THREADS, cut_of(k_lo), [&](const uint32_t (&key)[VEC]) {
#pragma unroll
        for (int j = 0; j < VEC; ++j)
          if (key[j] >= k_hi) {
            above += sc_fx(key[j]);
            ++n_above;
          } else if (key[j] >= k_lo) {
            least = min(least, key[j]);
            most = max(most, key[j]);
            if (*(volatile uint32_t*)&sh.list_n <= SC_LIST) {  // (a list that is too short takes no more)
              const uint32_t at = atomicAdd(&sh.list_n, 1u);
              if (at < SC_LIST) sh.list[at] = key[j];
            }
          }
      });
      least = __reduce_min_sync(0xffffffffu, least);
      most = __reduce_max_sync(0xffffffffu, most);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        above += __shfl_xor_sync(0xffffffffu, above, o);
        n_above += __shfl_xor_sync(0xffffffffu, n_above, o);
      }
      if (lane == 0) {
        sh.warp_ub[warp] = above;
        sh.warp_cnt[warp] = n_above;
        if (most > 0u) {
          atomicMin(&sh.own_min, least);
          atomicMax(&sh.own_max, most);
        }
      }
      if (tid < 256) {
        sh.even.cnt[tid] = 0u;
        sh.even.mass[tid] = 0ull;
      }
      __syncthreads();
      if (tid == 0) {
        unsigned long long t = 0ull, k = 0ull;
        for (int w = 0; w < SC_WARPS; ++w) {
          t += sh.warp_ub[w];
          k += sh.warp_cnt[w];
        }
        sh.x_u64[1] = t;
        sh.x_u64[2] = k;
      }
      // ---- radix descent over key - k_lo ----
      const int bits = 32 - __clz((int)(k_hi - k_lo - 1u));
      const int levels = (bits + 7) / 8, step = (bits + levels - 1) / levels;
      const uint32_t listed = sh.list_n;
      uint32_t prefix = 0u;  // of key - k_lo
      for (int level = 0; level < levels; ++level) {
        const int shift = max(0, bits - step * (level + 1)), above_shift = bits - step * level;
        ScLevel& h = level & 1 ? sh.odd : sh.even;
        ScLevel& next = level & 1 ? sh.even : sh.odd;
        // all lanes of a warp together.  Tokens of one bin that meet are added up first: 64-bit additions to one shared-memory word are
        // loops that fail but for one lane (64 x 151936 equal logits: 4.9 ms without)
        auto add = [&](uint32_t key, bool in) {
          const uint32_t d = key - k_lo;
          in = in && (level == 0 || (d >> above_shift) == (prefix >> above_shift));
          const int some = __popc(__ballot_sync(0xffffffffu, in));
          if (some == 0) return;
          const uint32_t bin = in ? (d >> shift) & ((1u << (above_shift - shift)) - 1u) : 256u;
          const unsigned long long fx = in ? sc_fx(key) : 0ull;
          if (some <= 4) {
            if (in) {
              atomicAdd(&h.cnt[bin], 1u);
              atomicAdd(&h.mass[bin], fx);
            }
            return;
          }
          const uint32_t peers = __match_any_sync(0xffffffffu, bin);
          const uint32_t low = __reduce_add_sync(peers, (uint32_t)fx & 0xfffffu), high = __reduce_add_sync(peers, (uint32_t)(fx >> 20));
          if (in && lane == __ffs(peers) - 1) {
            atomicAdd(&h.cnt[bin], (uint32_t)__popc(peers));
            atomicAdd(&h.mass[bin], ((unsigned long long)high << 20) + low);
          }
        };
        if (listed <= SC_LIST) {
          for (int b = tid - lane; b < (int)listed; b += SC_THREADS) {
            const uint32_t key = b + lane < (int)listed ? sh.list[b + lane] : 0u;
            add(key, key >= k_lo);
          }
        } else {
          walk(0, n, tid, SC_THREADS, -INFINITY, [&](const uint32_t (&key)[VEC]) {
#pragma unroll
            for (int j = 0; j < VEC; ++j) add(key[j], key[j] >= k_lo && key[j] < k_hi);
          });
        }
        cluster_barrier();
        if (tid < 256) {  // a thread merges one bin
          sh.merged.cnt[tid] = sum_u32(&h.cnt[tid]);
          sh.merged.mass[tid] = sum_u64(&h.mass[tid]);
          if (level == 0 && tid == 0) {
            sh.mass_above = sum_u64(&sh.x_u64[1]);
            sh.cnt_above = (uint32_t)sum_u64(&sh.x_u64[2]);
          }
          if (level == 0 && tid == 32) {
            uint32_t least = SC_ONE, most = 0u;
            for (int q = 0; q < csize; ++q) {
              least = min(least, ld_dsmem_u32(dsmem_addr(smem_u32(&sh.own_min), (uint32_t)q)));
              most = max(most, ld_dsmem_u32(dsmem_addr(smem_u32(&sh.own_max), (uint32_t)q)));
            }
            sh.key_min = least;
            sh.key_max = most;
          }
        } else {
          // the other histogram is free: peers read it (the previous level, or the coarse counts) before they arrived
          next.cnt[tid - 256] = 0u;
          next.mass[tid - 256] = 0ull;
        }
        __syncthreads();
        if (warp == 0) {
          // Lane l owns bins 8l .. 8l + 7; the same walk as over the coarse bins, with exact masses
          uint32_t c8[8], cs = 0u;
          unsigned long long m8[8], ms = 0ull, none = 0ull;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            c8[j] = sh.merged.cnt[lane * 8 + j];
            m8[j] = sh.merged.mass[lane * 8 + j];
            cs += c8[j];
            ms += m8[j];
          }
          const uint32_t cnt0 = sh.cnt_above;
          const unsigned long long mass0 = sh.mass_above;
          __syncwarp();
          uint32_t ch = cs;
          unsigned long long mh = ms;
          sc_suffix(ch, mh, none, lane);
          uint32_t cnt = cnt0 + (ch - cs);
          unsigned long long mass = mass0 + (mh - ms);
          int chosen = 256;
          uint32_t c_cnt = 0u;
          unsigned long long c_mass = 0ull;
#pragma unroll
          for (int j = 7; j >= 0; --j) {
            if (c8[j] != 0u && cnt < kk && mass < lim) {
              chosen = lane * 8 + j;
              c_cnt = cnt;
              c_mass = mass;
            }
            cnt += c8[j];
            mass += m8[j];
          }
          const int best = __reduce_min_sync(0xffffffffu, chosen);
          if (chosen == best && best < 256) {  // exactly one lane owns the chosen bin
            sh.prefix = prefix | ((uint32_t)best << shift);
            sh.cnt_above = c_cnt;
            sh.mass_above = c_mass;
          } else if (best == 256 && lane == 0) {  // cannot happen: the bracket holds the last kept bin
            sh.prefix = prefix;
          }
        }
        __syncthreads();
        prefix = sh.prefix;
        if (sh.key_min == sh.key_max) {  // ties, as many as they are: the bracket has one key
          prefix = sh.key_min - k_lo;
          break;
        }
      }
      thr_key = k_lo + prefix;
    }
  }
  // min-p: e >= min_p (e is relative to the row maximum, whose e is 1)
  if (mp > 0.f) thr_key = max(thr_key, __float_as_uint(fminf(mp, 1.f)));
  thr_key = max(thr_key, SC_LOW);  // tokens below have no mass

  // inverse CDF in vocabulary order over the kept set: a contiguous run of tokens per warp
  const int run = ((n + SC_WARPS - 1) / SC_WARPS + 31) & ~31;  // (a multiple of a 16-byte piece)
  const int c0 = min(n, warp * run), c1 = min(n, c0 + run);
  unsigned long long local = 0ull;
  const float cut = cut_of(thr_key);
  walk(c0, c1, lane, 32, cut, [&](const uint32_t (&key)[VEC]) {
#pragma unroll
    for (int j = 0; j < VEC; ++j)
      if (key[j] >= thr_key) local += sc_fx(key[j]);
  });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  __syncthreads();  // warp_tot is read above
  if (lane == 0) sh.warp_tot[warp] = local;
  __syncthreads();
  unsigned long long before = 0ull, cta_total = 0ull;
  for (int w = 0; w < SC_WARPS; ++w) {
    const unsigned long long t = sh.warp_tot[w];
    if (w < warp) before += t;
    cta_total += t;
  }
  if (tid == 0) sh.x_u64[3] = cta_total;
  cluster_barrier();
  unsigned long long total = 0ull, cta_before = 0ull;
#pragma unroll
  for (int q = 0; q < SC_MAX_CLUSTER; ++q) {
    const unsigned long long t = q < csize ? ld_dsmem_u64(dsmem_addr(smem_u32(&sh.x_u64[3]), (uint32_t)q)) : 0ull;
    if (q < (int)cr) cta_before += t;
    total += t;
  }
  // u < 1, so the target lies strictly inside [0, total)
  const float u = fminf(fmaxf(uniform[row], 0.f), 0.99999994f);
  unsigned long long target = (unsigned long long)((double)u * (double)total);
  if (target >= total && total > 0ull) target = total - 1ull;
  before += cta_before;
  if (local > 0ull && before <= target && target < before + local) {
    for (int b = c0; b < c1; b += 32 * VEC) {  // a lane has the tokens of one piece
      const int i = b + lane * VEC;
      const uint4 x = i < c1 ? *reinterpret_cast<const uint4*>(vals + i) : make_uint4(0u, 0u, 0u, 0u);
      unsigned long long fx[VEC], mine = 0ull;
      const bool none = i >= c1 || sc_max<T>(x) * inv_t - m < cut;
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const uint32_t key = !none && i + j < c1 ? key_of(ldf(reinterpret_cast<const T*>(&x), j)) : 0u;
        fx[j] = key >= thr_key ? sc_fx(key) : 0ull;
        mine += fx[j];
      }
      if (!__any_sync(0xffffffffu, mine > 0ull)) continue;
      unsigned long long incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const uint32_t past = __ballot_sync(0xffffffffu, before + incl > target);
      if (past) {
        if (lane == __ffs(past) - 1) {
          unsigned long long at = before + incl - mine;
          int pick = 0;
          bool found = false;
#pragma unroll
          for (int j = 0; j < VEC; ++j) {
            at += fx[j];
            if (!found && at > target) pick = j, found = true;
          }
          out[row] = i0 + i + pick;
        }
        break;
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
  } else if (total == 0ull && cr == 0u && tid == 0) {
    out[row] = 0;  // no token has mass: nothing but NaN and minus infinity
  }
  // a CTA must not exit while a peer may still read its shared memory
  if (csize > 1) cluster_sync_all();
}

template <typename T>
__global__ void __launch_bounds__(256) logprob_topk_kernel(const T* __restrict__ logits, long long ld, int vocab, const int* __restrict__ picked,
                                                            int k, float* __restrict__ chosen_lp, float* __restrict__ top_lp,
                                                            int* __restrict__ top_idx) {
  PG_PDL_ENTRY();
  __shared__ float red[32];
  __shared__ ArgPair ared[32];
  __shared__ int taken[32];
  const int row = blockIdx.x;
  const T* r = logits + row * ld;
  float m = -FLT_MAX;
  for (int i = threadIdx.x; i < vocab; i += 256) m = fmaxf(m, ldf(r, i));
  m = block_max_f(m, red);
  float z = 0.f;
  for (int i = threadIdx.x; i < vocab; i += 256) z += expf(ldf(r, i) - m);
  z = block_sum_f(z, red);
  const float lse = m + logf(z);
  if (threadIdx.x == 0) {
    int p = picked[row];
    chosen_lp[row] = (p >= 0 && p < vocab) ? ldf(r, p) - lse : -INFINITY;
  }
  for (int round = 0; round < k; ++round) {
    ArgPair best{-FLT_MAX, 0x7fffffff};
    for (int i = threadIdx.x; i < vocab; i += 256) {
      bool skip = false;
      for (int q = 0; q < round; ++q) skip |= (taken[q] == i);
      if (skip) continue;
      float v = ldf(r, i);
      if (v > best.v) best = ArgPair{v, i};
    }
    best = block_argmax(best, ared);
    if (threadIdx.x == 0) {
      taken[round] = best.i;
      top_lp[(long long)row * k + round] = best.v - lse;
      top_idx[(long long)row * k + round] = best.i;
    }
    __syncthreads();
  }
}

}  // namespace

extern "C" long long pg_argmax_scratch_bytes(int rows, int vocab) { return (long long)rows * ceil_div(vocab, ARG_TILE) * (long long)sizeof(ArgPair); }

extern "C" int pg_argmax(const void* logits, int is_f32, int rows, int vocab, long long ld, void* scratch, long long scratch_bytes, void* out,
                         cudaStream_t stream) {
  if (rows == 0) return PG_OK;
  const int tiles = ceil_div(vocab, ARG_TILE);
  PG_REQUIRE(scratch_bytes >= pg_argmax_scratch_bytes(rows, vocab), "argmax: scratch too small");
  dim3 grid(tiles, rows);
  if (is_f32)
    PG_CUDA(launch_pdl(argmax_partial_kernel<float>, dim3(grid), dim3(256), (size_t)(0), stream, (const float*)logits, ld, vocab, (ArgPair*)scratch, tiles));
  else
    PG_CUDA(launch_pdl(argmax_partial_kernel<bf16>, dim3(grid), dim3(256), (size_t)(0), stream, (const bf16*)logits, ld, vocab, (ArgPair*)scratch, tiles));
  PG_LAUNCH_CHECK();
  PG_CUDA(launch_pdl(argmax_final_kernel, dim3(rows), dim3(128), (size_t)(0), stream, (const ArgPair*)scratch, tiles, (int*)out));
  PG_LAUNCH_CHECK();
  return PG_OK;
}

extern "C" int pg_markov_step_argmax(const void* base, int is_f32, int rows, int block, int step, int vocab, long long ld, const void* bias, long long ldb,
                                    void* scratch, long long scratch_bytes, void* next, void* drafts, cudaStream_t stream) {
  if (rows == 0) return PG_OK;
  const int tiles = ceil_div(vocab, ARG_TILE);
  PG_REQUIRE(step >= 0 && step < block, "markov step: step outside the block");
  PG_REQUIRE(scratch_bytes >= pg_argmax_scratch_bytes(rows, vocab), "markov step: scratch too small");
  dim3 grid(tiles, rows);
  if (is_f32)
    PG_CUDA(launch_pdl(markov_partial_kernel<float>, dim3(grid), dim3(256), (size_t)(0), stream, (const float*)base, ld, block, step, (const float*)bias, ldb,
                       vocab, (ArgPair*)scratch, tiles));
  else
    PG_CUDA(launch_pdl(markov_partial_kernel<bf16>, dim3(grid), dim3(256), (size_t)(0), stream, (const bf16*)base, ld, block, step, (const bf16*)bias, ldb, vocab,
                       (ArgPair*)scratch, tiles));
  PG_LAUNCH_CHECK();
  PG_CUDA(launch_pdl(markov_final_kernel, dim3(rows), dim3(128), (size_t)(0), stream, (const ArgPair*)scratch, tiles, (int*)next, (int*)drafts, block, step));
  PG_LAUNCH_CHECK();
  return PG_OK;
}

static int g_force_cluster = 0;
// Test hook: pin the cluster size of the cluster sampler (1, 2, 4 or 8; 0 = chosen from the vocabulary).
extern "C" void pg_sample_force_cluster(int c) { g_force_cluster = c; }

// Cluster size and slice length of the cluster sampler for a vocabulary, or 0 when the row does not fit the shared memory of
// eight CTAs (the one-CTA kernel serves those).  A wave holds so many clusters of 1, 2, 4, 8 CTAs at one or two CTAs an SM
// (74 / 33 / 15 clusters of 2 / 4 / 8 fit the GPCs).  A row takes the time of its slice and of so many thousand tokens more: the
// barriers of its cluster, and the other clusters of a wave that is full.  Us with clusters of 1 / 2 / 4 / 8, top-k 50: 16 rows of
// 4096 15 / 16 / 18 / 30, of 32000 41 / 29 / 23 / 32, of 102400 103 / 61 / 41 / 41; 4 rows of 102400 94 / 58 / 38 / 33; 64 rows of
// 151936 - / 83 / 62 / 102.
static int sampler_cluster_plan(int rows, int vocab, int elem, int max_smem, int* slice_out) {
  const int room = (max_smem - 2048 - (int)sizeof(ScShared) - 64) / elem;  // tokens per CTA (2 KB left for static shared memory)
  static const int per_wave[4] = {148, 74, 33, 15};
  static const double alone[4] = {13.2, 15.8, 17.8, 23.3}, crowded[4] = {5.0, 4.4, 6.7, 14.4};
  int best = 0;
  double least = 0;
  for (int l = 0; l < 4; ++l) {
    const int c = 1 << l, slice = (ceil_div(vocab, c) + 7) & ~7;
    if (slice > room || (g_force_cluster > 0 && c != g_force_cluster)) continue;
    const int wave = per_wave[l] * (2 * (slice * elem + (int)sizeof(ScShared) + 2048) <= max_smem ? 2 : 1);
    const double cost = ceil_div(rows, wave) * (slice / 1000.0 + alone[l] + crowded[l] * (rows < wave ? (double)rows / wave : 1.0));
    if (best == 0 || cost < least) best = c, least = cost, *slice_out = slice;
  }
  return best;
}

template <typename T>
static int launch_sample_cluster(const T* logits, long long ld, int rows, int vocab, int c, int slice, const float* temperature, const int* top_k,
                                 const float* top_p, const float* min_p, const float* uniform, int* out, cudaStream_t stream) {
  const size_t smem = ((sizeof(ScShared) + 15) & ~size_t(15)) + (size_t)slice * sizeof(T);
  static bool attr_done[2] = {false, false};
  const int which = sizeof(T) == 4 ? 1 : 0;
  if (!attr_done[which]) {
    int max_smem = 0, dev = 0;
    PG_CUDA(cudaGetDevice(&dev));
    PG_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PG_CUDA(cudaFuncSetAttribute(sample_cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - 2048));
    attr_done[which] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(rows * c));
  cfg.blockDim = dim3(SC_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  int na = 0;
  if (c > 1) {
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = (unsigned)c;
    at[na].val.clusterDim.y = 1;
    at[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl_enabled()) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = (unsigned)na;
  PG_CUDA(cudaLaunchKernelEx(&cfg, sample_cluster_kernel<T>, logits, ld, vocab, slice, temperature, top_k, top_p, min_p, uniform, out, c));
  PG_LAUNCH_CHECK();
  return PG_OK;
}

extern "C" int pg_sample(const void* logits, int is_f32, int rows, int vocab, long long ld, const void* temperature, const void* top_k,
                         const void* top_p, const void* min_p, const void* uniform, void* out, cudaStream_t stream) {
  if (rows == 0) return PG_OK;
  static int use_cluster = -1, max_smem = 0;
  if (use_cluster < 0) {
    const char* e = getenv("PEGAINFER_SAMPLER_CLUSTER");
    int dev = 0;
    PG_CUDA(cudaGetDevice(&dev));
    PG_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    use_cluster = (e && e[0] == '0') ? 0 : 1;
  }
  int slice = 0;
  const int c = use_cluster ? sampler_cluster_plan(rows, vocab, is_f32 ? 4 : 2, max_smem, &slice) : 0;
  if (c > 0) {
    if (is_f32)
      return launch_sample_cluster<float>((const float*)logits, ld, rows, vocab, c, slice, (const float*)temperature, (const int*)top_k, (const float*)top_p,
                                          (const float*)min_p, (const float*)uniform, (int*)out, stream);
    return launch_sample_cluster<bf16>((const bf16*)logits, ld, rows, vocab, c, slice, (const float*)temperature, (const int*)top_k, (const float*)top_p,
                                       (const float*)min_p, (const float*)uniform, (int*)out, stream);
  }
  if (is_f32)
    PG_CUDA(launch_pdl(sample_kernel<float>, dim3(rows), dim3(ST), (size_t)(0), stream, (const float*)logits, ld, vocab, (const float*)temperature, (const int*)top_k, (const float*)top_p,
                                                  (const float*)min_p, (const float*)uniform, (int*)out));
  else
    PG_CUDA(launch_pdl(sample_kernel<bf16>, dim3(rows), dim3(ST), (size_t)(0), stream, (const bf16*)logits, ld, vocab, (const float*)temperature, (const int*)top_k, (const float*)top_p,
                                                 (const float*)min_p, (const float*)uniform, (int*)out));
  PG_LAUNCH_CHECK();
  return PG_OK;
}

extern "C" int pg_logprob_topk(const void* logits, int is_f32, int rows, int vocab, long long ld, const void* picked, int k, void* chosen_lp,
                               void* top_lp, void* top_idx, cudaStream_t stream) {
  PG_REQUIRE(k >= 0 && k <= 32, "logprob_topk: k=%d out of range [0, 32]", k);
  if (rows == 0) return PG_OK;
  if (is_f32)
    PG_CUDA(launch_pdl(logprob_topk_kernel<float>, dim3(rows), dim3(256), (size_t)(0), stream, (const float*)logits, ld, vocab, (const int*)picked, k, (float*)chosen_lp, (float*)top_lp,
                                                         (int*)top_idx));
  else
    PG_CUDA(launch_pdl(logprob_topk_kernel<bf16>, dim3(rows), dim3(256), (size_t)(0), stream, (const bf16*)logits, ld, vocab, (const int*)picked, k, (float*)chosen_lp, (float*)top_lp,
                                                        (int*)top_idx));
  PG_LAUNCH_CHECK();
  return PG_OK;
}
