// bf16 GEMM  Y[T, M] = X[T, K] * W[M, K]^T  for large T: two SMs work on one tile.
//
// A pair of CTAs (a thread-block cluster of 2) computes a 256 (weight rows) x 256 (tokens)
// tile with tcgen05.mma.cta_group::2.  Each CTA stages only its own half of both operands,
// 128 weight rows and 128 token rows per 64-deep k-block, so a stage is 32 KB per CTA for
// 256 x 256 x 64 multiply-adds of the pair.  The one-CTA kernel in gemm_sm100.cu moves
// 48 KB per CTA for 128 x 256 x 64: per multiply-add this kernel writes and reads a third
// as many shared-memory bytes, which is what limits the one-CTA kernel at large T (TMA
// writes plus operand reads exceed what one SM's shared memory delivers per clock at full
// tensor rate).  The accumulator of each CTA is its 128 rows x 256 columns of the tile in
// its own TMEM, two buffers, so the epilogue of a tile overlaps the main loop of the next.
//
//   CTA rank 0 (leader)                          CTA rank 1
//   warp 0  TMA producer (own halves)            warp 0  TMA producer (own halves)
//   warp 1  TMEM alloc, issues every MMA          warp 1  TMEM alloc / dealloc only
//   warps 2..9 epilogue of rows 0..127            warps 2..9 epilogue of rows 128..255
//
// Barriers: `full[s]` lives in the leader and counts the bytes of BOTH CTAs' loads (each
// CTA's TMA names the leader's barrier); `empty[s]` and `tfull[a]` exist in both CTAs and
// are signalled by tcgen05.commit with a two-CTA multicast mask; `tempty[a]` lives in the
// leader and counts the epilogue warps of the pair.  Every wait is bounded.
//
// Takes the place of the reference's cuBLAS/cuBLASLt layer for prefill-sized problems
// (pegainfer-kernels/csrc/shared/linear.cu:294-596).
#include <stdlib.h>
#include <string.h>

#include <climits>
#include <mutex>

#include "api.h"
#include "common.cuh"

namespace {

constexpr int BM = 128;  // weight rows per CTA (256 per pair)
constexpr int BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int MAX_STAGES = 12;
constexpr int MAX_SPLITS = 4;
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 64 + 32 * EPI_WARPS;
constexpr int RASTER_GROUP = 8;  // weight-row pairs per raster group

struct Gemm2Params {
  bf16* y;
  long long ldy;
  int M, T, K;
  int m_pairs, n_tiles, kblocks;
  int bn;      // token columns of a pair's tile (multiple of 32, <= 256); each CTA stages bn / 2 token rows
  int stages;  // shared-memory ring depth
  uint32_t tmem_cols;
  uint32_t* status;
  int epi;  // 0: y = x W^T; 1: the weight rows alternate (gate_i, up_i) and y [T, M / 2] = bf16(silu(gate)) * up
  const float* xielu;  // epi 0: the two constants of xIELU on every output (nullptr = none)
  int whole;           // tiles that one pair computes over all of K; the `rem` tiles behind them are cut in `splits` ranges of k (1: none are)
  int rem, splits;
  float4* part;        // partial sums [rem][splits][CTA of the pair][bn / 4][128 rows][4]
  uint32_t* counters;  // [rem][CTA of the pair][epilogue warp], zero between launches
};

struct Work {
  int tile, part, kb0, kb1;  // part < 0: a whole tile
};
// The i-th piece of work of a pair: whole tiles in rounds, then at most one range of a cut tile.  Neighbouring pairs take
// neighbouring tiles at the same range of k, so that they share operands through L2.
__device__ __forceinline__ bool work_at(const Gemm2Params& p, int pair, int pairs, int i, Work& w) {
  const int item = pair + i * pairs;
  if (item < p.whole) {
    w = {item, -1, 0, p.kblocks};
    return true;
  }
  const int q = item - p.whole;
  if (q >= p.rem * p.splits) return false;
  const int part = q / p.rem;
  w = {p.whole + q % p.rem, part, part * p.kblocks / p.splits, (part + 1) * p.kblocks / p.splits};
  return true;
}

// Work item -> (weight-row pair, token tile).  Items walk RASTER_GROUP weight-row pairs across
// all token tiles before moving on, so the CTA pairs that run at the same time cover a
// near-square patch of the output and share both operands through L2 (walking all weight
// rows of one token tile first would stream the whole weight matrix once per token tile).
__device__ __forceinline__ void tile_of(const Gemm2Params& p, int item, int& m_pair, int& n_tile) {
  const int per_group = RASTER_GROUP * p.n_tiles;
  const int group = item / per_group;
  const int first = group * RASTER_GROUP;
  const int gsz = min(RASTER_GROUP, p.m_pairs - first);
  const int within = item - group * per_group;
  m_pair = first + within % gsz;
  n_tile = within / gsz;
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A[smem of both CTAs] * B[smem of both CTAs]; one thread of the leader.
__device__ __forceinline__ void umma_bf16_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this shared-memory offset in every CTA of `mask` once all MMAs
// issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(mask)
               : "memory");
}
// Tiled load into this CTA's shared memory; the bytes are counted on `bar_cluster_addr`,
// a barrier that may live in the other CTA of the pair.  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const void* tmap, uint32_t bar_cluster_addr, int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(dst)), "l"(tmap), "r"(bar_cluster_addr), "r"(x), "r"(y), "l"(policy)
      : "memory");
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm2sm_bf16_tn_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const Gemm2Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  uint8_t* tiles = smem_raw + (((base + 1023u) & ~1023u) - base);
  const int bnh = p.bn >> 1;
  const int stage_bytes = A_BYTES + bnh * 128;
  uint64_t* full = reinterpret_cast<uint64_t*>(tiles + p.stages * stage_bytes);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 2 * EPI_WARPS);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, p.tmem_cols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before any remote arrive or multicast commit
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      // both operands are re-read (weights by every token tile, tokens by every weight-row pair)
      const uint64_t pol_w = l2_policy_evict_normal();
      const uint64_t pol_x = l2_policy_evict_normal();
      int stage = 0;
      uint32_t phase = 0;
      uint32_t last_phase[MAX_STAGES];
      bool used[MAX_STAGES];
#pragma unroll
      for (int s = 0; s < MAX_STAGES; ++s) {
        used[s] = false;
        last_phase[s] = 0;
      }
      bool ok = true;
      Work wk;
      for (int i = 0; ok && work_at(p, pair, pairs, i, wk); ++i) {
        int m_pair, n_tile;
        tile_of(p, wk.tile, m_pair, n_tile);
        const int w_row = m_pair * (2 * BM) + (int)rank * BM;
        const int x_row = n_tile * p.bn + (int)rank * bnh;
        for (int kb = wk.kb0; kb < wk.kb1; ++kb) {
          if (!mbar_wait_cluster(&empty[stage], phase ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* a_dst = tiles + stage * stage_bytes;
          const uint32_t bar = dsmem_addr(smem_u32(&full[stage]), 0u);
          if (rank == 0) mbar_expect_tx(&full[stage], 2u * (uint32_t)stage_bytes);
          tma_load_2d_pair(a_dst, &tm_w, bar, kb * BK, w_row, pol_w);
          tma_load_2d_pair(a_dst + A_BYTES, &tm_x, bar, kb * BK, x_row, pol_x);
          used[stage] = true;
          last_phase[stage] = phase;
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      // Drain: the MMAs that read this CTA's stages have completed (so the loads have landed and
      // the leader's multicast arrivals on this CTA's barriers are in) before the CTA may exit.
      for (int s = 0; s < p.stages; ++s) {
        if (!used[s]) continue;
        uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait_cluster(&empty[s], last_phase[s])) {
          if (*abort_flag || globaltimer_ns() - t0 > PG_WAIT_LIMIT_NS) break;
        }
      }
    }
  } else if (warp == 1) {
    // the whole warp walks the loop and one lane issues: what does not depend on the lane stays in uniform registers (a lone
    // thread that forms each descriptor anew takes 60 to 110 cycles a product, near the 128 of the product itself: 1337 rows
    // through four layers of an 8B model 2298 us, 2157 now)
    if (rank == 0) {
      const bool one = elect_one();
      const uint32_t idesc = umma_idesc_bf16_f32(2 * BM, (uint32_t)p.bn);
      const uint64_t a_desc0 = umma_desc_k_sw128(smem_u32(tiles));
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      Work wk;
      for (int i = 0; ok && work_at(p, pair, pairs, i, wk); ++i) {
        if (!mbar_wait_cluster(&tempty[acc], acc_phase ^ 1u, abort_flag)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * p.bn);
        for (int kb = wk.kb0; kb < wk.kb1; ++kb) {
          if (!mbar_wait_cluster(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (one) {
            const uint64_t a = a_desc0 + (uint32_t)(stage * (stage_bytes >> 4));
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) umma_bf16_ss_pair(d_tmem, a + (uint32_t)(k * 2), a + (uint32_t)((A_BYTES >> 4) + k * 2), idesc, (kb > wk.kb0 || k > 0) ? 1u : 0u);
            umma_commit_pair(&empty[stage], (uint16_t)3);
          }
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        if (one) umma_commit_pair(&tfull[acc], (uint16_t)3);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    // epilogue: warp w may touch TMEM lanes 32*(w%4) .. 32*(w%4)+31 of its own CTA; two warps share the lanes, alternating in
    // steps of 32 columns
    const int wq = warp & 3, c0 = ((warp - 2) >> 2) * 32;
    const int r = wq * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    Work wk;
    for (int i = 0; work_at(p, pair, pairs, i, wk); ++i) {
      int m_pair, n_tile;
      tile_of(p, wk.tile, m_pair, n_tile);
      if (!mbar_wait_cluster(&tfull[acc], acc_phase, abort_flag)) break;
      tc_fence_after();
      const int m = m_pair * (2 * BM) + (int)rank * BM + r;
      const int n0 = n_tile * p.bn;
      const uint32_t t_row = tmem_base + ((uint32_t)(wq * 32) << 16) + (uint32_t)(acc * p.bn);
      bf16* yc = p.y + m;
      // A cut tile: every range leaves its sums in scratch, and for each 32 rows the last one to arrive adds them up, in the
      // order of the ranges whoever is last, and stores the output.  Nobody waits.
      const long long part_stride = 2ll * (p.bn / 4) * BM;
      float4* parts = nullptr;
      bool last = true;
      if (wk.part >= 0) {
        const int cut = wk.tile - p.whole;
        parts = p.part + ((long long)cut * p.splits * 2 + rank) * (p.bn / 4) * BM + r;
        float4* mine = parts + wk.part * part_stride;
        for (int c = c0; c < p.bn; c += 64) {
          uint32_t v[2][16];
          tmem_ld16(t_row + c, v[0]);
          tmem_ld16(t_row + c + 16, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t* u = v[q / 4] + q % 4 * 4;
            __stcg(mine + (c / 4 + q) * BM, make_float4(__uint_as_float(u[0]), __uint_as_float(u[1]), __uint_as_float(u[2]), __uint_as_float(u[3])));
          }
        }
        __threadfence();
        __syncwarp();
        uint32_t* counter = p.counters + (cut * 2 + (int)rank) * EPI_WARPS + warp - 2;
        uint32_t before = 0;
        if (lane == 0) before = atomicAdd(counter, 1u);
        last = __shfl_sync(0xFFFFFFFFu, before, 0) == (uint32_t)(p.splits - 1);
        if (last) {
          __threadfence();
          if (lane == 0) *counter = 0u;
        }
      }
      for (int c = c0; last && c < p.bn; c += 64) {
        uint32_t v[2][16];
        tmem_ld16(t_row + c, v[0]);
        tmem_ld16(t_row + c + 16, v[1]);
        if (wk.part < 0) {
          tmem_ld_wait();
        } else {
          // the other ranges, 16 columns at a time (with all 32 in flight the sums spilled, also where no tile is cut: 65 x 1024 x 3072
          // 16.0 us and 14.0 now, 4096 x 4096 x 4096 111 and 109)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            float4 o[MAX_SPLITS - 1][4];
#pragma unroll
            for (int j = 0; j < MAX_SPLITS - 1; ++j)
              if (j < p.splits - 1) {
#pragma unroll
                for (int q = 0; q < 4; ++q) o[j][q] = __ldcg(parts + (j < wk.part ? j : j + 1) * part_stride + (c / 4 + hf * 4 + q) * BM);
              }
            if (hf == 0) tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t* u = v[hf] + q * 4;
              const float4 own = make_float4(__uint_as_float(u[0]), __uint_as_float(u[1]), __uint_as_float(u[2]), __uint_as_float(u[3]));
              float4 sum = wk.part == 0 ? own : o[0][q];
#pragma unroll
              for (int s = 1; s < MAX_SPLITS; ++s)
                if (s < p.splits) {
                  const float4 x = s == wk.part ? own : s < wk.part ? o[min(s, MAX_SPLITS - 2)][q] : o[s - 1][q];
                  sum = make_float4(sum.x + x.x, sum.y + x.y, sum.z + x.z, sum.w + x.w);
                }
              u[0] = __float_as_uint(sum.x);
              u[1] = __float_as_uint(sum.y);
              u[2] = __float_as_uint(sum.z);
              u[3] = __float_as_uint(sum.w);
            }
          }
        }
        if (p.epi != 0) {
          // SwiGLU (1) or its form with tanh-GELU (3): lanes 2 i and 2 i + 1 hold gate and up of output column m / 2 (both rounded to bf16 first, as the
          // separate kernel sees them); the shuffles run on all lanes, the even ones store
          bf16* ys = p.y + (m >> 1);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float mine = __bfloat162float(__float2bfloat16(__uint_as_float(v[h][j])));
              const float other = __shfl_xor_sync(0xFFFFFFFFu, mine, 1);
              const int n = n0 + c + h * 16 + j;
              if (!(lane & 1) && m < p.M && n < p.T) {
                const float a = bf16_round(glu_act(mine, p.epi == 3));
                ys[(long long)n * p.ldy] = __float2bfloat16(a * other);
              }
            }
          }
        } else if (m < p.M) {
          if (p.xielu != nullptr) {
            const float a = p.xielu[0], b = p.xielu[1];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int j = 0; j < 16; ++j) v[h][j] = __float_as_uint(xielu(__uint_as_float(v[h][j]), a, b));
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int n = n0 + c + h * 16 + j;
              if (n < p.T) yc[(long long)n * p.ldy] = __float2bfloat16(__uint_as_float(v[h][j]));
            }
          }
        }
      }
      // this accumulator buffer may be overwritten: tell the leader's MMA thread
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(dsmem_addr(smem_u32(&tempty[acc]), 0u));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA tears down shared memory or TMEM the other may still reach
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, p.tmem_cols);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(p.status, PG_ST_OK, PG_ST_TIMEOUT | (11u << 8));
}

std::mutex g_mu2;
struct Dev2 {
  bool set = false;
  bool usable = false;
  int sms = 0;
  int max_smem = 0;
  int max_pairs = 0;
};
Dev2 g_dev2[64];
int g_enabled = -1;

}  // namespace

static bool gemm2sm_enabled() {
  if (g_enabled < 0) {
    const char* e = getenv("PEGAINFER_GEMM_2SM");
    g_enabled = (e && e[0] == '0') ? 0 : 1;
  }
  return g_enabled == 1;
}

// PEGAINFER_GEMM_2SM_MAXK: longest k of the two-SM kernel; `otherwise` where it is not set
static int gemm2sm_max_k(int otherwise) {
  static const int limit = [] {
    const char* e = getenv("PEGAINFER_GEMM_2SM_MAXK");
    return e ? atoi(e) : 0;
  }();
  return limit > 0 ? limit : otherwise;
}

// 1 if the two-SM kernel takes this problem in a GEMM with bf16 results: above the 64 rows of the decode plans it measured faster
// than the one-CTA kernel at every size.  Us there -> here: T = 65, M x K = 1024 x 1024 20 -> 11, 4096 x 12288 58 -> 34; T = 256,
// 64 x 512 20 -> 9, 5120 x 17408 109 -> 57; T = 1100, 4096 x 12288 144 -> 101; T = 4096, 4096 x 12288 377 -> 280.  At 64 rows and
// below the one-CTA kernel's narrow tiles win (4096 x 4096: 14, here 19).
extern "C" int pg_gemm2sm_takes(int T, int M, int K) { return gemm2sm_enabled() && T > 64 && M >= 64 && K >= 256 && K <= gemm2sm_max_k(INT_MAX) && K % 8 == 0 ? 1 : 0; }

// 1 for the problems whose f32 results callers leave to a bf16 GEMM on this kernel (at least about a round of CTA pairs, k up to
// 8192): a narrower set than pg_gemm2sm_takes, so that no other results lose their 32 bits.
extern "C" int pg_gemm2sm_eligible(int T, int M, int K) {
  if (!gemm2sm_enabled() || T < 256 || M < 1024 || K < 256 || K > gemm2sm_max_k(8192) || K % 8 != 0) return 0;
  return (long long)ceil_div(M, 2 * BM) * ceil_div(T, 256) >= 64 ? 1 : 0;
}

struct Scratch2 {
  void* ws;
  long long ws_bytes;
  void* counters;
  long long counter_bytes;
};
static int gemm2sm_impl(const void* x, const void* w, void* y, int T, int M, int K, long long ldx, long long ldw, long long ldy, const Scratch2& sc, void* status, int epi, cudaStream_t stream,
                        const void* xielu = nullptr, int* plan_out = nullptr);

// How a problem would be launched on the current device with `ws_bytes` of scratch: out = {token-tile width, whole tiles, cut tiles, ranges
// of k of a cut tile}.
extern "C" int pg_gemm2sm_plan(int T, int M, int K, long long ws_bytes, int* out) {
  PG_REQUIRE(out != nullptr, "gemm2sm plan: null output");
  void* fake = reinterpret_cast<void*>(uintptr_t(256));
  return gemm2sm_impl(fake, fake, fake, T, M, K, K, K, M, {fake, ws_bytes, fake, 1ll << 40}, fake, 0, nullptr, nullptr, out);
}

// ws, counters: scratch as for pg_gemm_bf16_tn (null: no tile is cut)
extern "C" int pg_gemm2sm_bf16_tn(const void* x, const void* w, void* y, int T, int M, int K, long long ldx, long long ldw, long long ldy, void* ws, long long ws_bytes, void* counters,
                                  long long counter_bytes, void* status, cudaStream_t stream) {
  return gemm2sm_impl(x, w, y, T, M, K, ldx, ldw, ldy, {ws, ws_bytes, counters, counter_bytes}, status, 0, stream);
}

// The same product with SwiGLU (gelu: tanh-GELU on the gate) in the epilogue: w [M, K] with rows alternating (gate_i, up_i), y [T, M / 2].
extern "C" int pg_gemm2sm_bf16_tn_swiglu(const void* x, const void* w, void* y, int T, int M, int K, long long ldx, long long ldw, long long ldy, int gelu, void* ws, long long ws_bytes, void* counters,
                                         long long counter_bytes, void* status, cudaStream_t stream) {
  PG_REQUIRE(M % 2 == 0, "gemm2sm swiglu: M %d must be even (interleaved gate / up rows)", M);
  return gemm2sm_impl(x, w, y, T, M, K, ldx, ldw, ldy, {ws, ws_bytes, counters, counter_bytes}, status, gelu ? 3 : 1, stream);
}

// The same product with xIELU in the epilogue; act: f32 softplus(p), 1/2 + softplus(q).
extern "C" int pg_gemm2sm_bf16_tn_xielu(const void* x, const void* w, void* y, int T, int M, int K, long long ldx, long long ldw, long long ldy, const void* act, void* ws, long long ws_bytes,
                                        void* counters, long long counter_bytes, void* status, cudaStream_t stream) {
  return gemm2sm_impl(x, w, y, T, M, K, ldx, ldw, ldy, {ws, ws_bytes, counters, counter_bytes}, status, 0, stream, act);
}

static int gemm2sm_impl(const void* x, const void* w, void* y, int T, int M, int K, long long ldx, long long ldw, long long ldy, const Scratch2& sc, void* status, int epi, cudaStream_t stream,
                        const void* xielu, int* plan_out) {
  PG_REQUIRE(T > 0 && M > 0 && K > 0 && K % 8 == 0, "gemm2sm: bad problem %dx%dx%d", T, M, K);
  PG_REQUIRE(status != nullptr, "gemm2sm: a device status word is required");
  if (plan_out == nullptr) pg_gemm_prefetch_next(nullptr, 0);  // a hint was for this GEMM, which has no use for it: it must not outlive the weights it names
  int dev = 0;
  PG_CUDA(cudaGetDevice(&dev));
  Dev2& di = g_dev2[dev & 63];
  const int tail = (2 * MAX_STAGES + 4) * 8 + 64;
  {
    std::lock_guard<std::mutex> lk(g_mu2);
    if (!di.set) {
      PG_CUDA(cudaDeviceGetAttribute(&di.sms, cudaDevAttrMultiProcessorCount, dev));
      PG_CUDA(cudaDeviceGetAttribute(&di.max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
      PG_CUDA(cudaFuncSetAttribute(gemm2sm_bf16_tn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem));
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3((unsigned)(2 * di.sms));
      cfg.blockDim = dim3(NUM_THREADS);
      cfg.dynamicSmemBytes = (size_t)di.max_smem;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm2sm_bf16_tn_kernel, &cfg) == cudaSuccess) di.max_pairs = n;
      else (void)cudaGetLastError();
      di.usable = di.max_pairs > 0;
      di.set = true;
    }
  }
  PG_REQUIRE(di.usable, "gemm2sm: no co-resident CTA pair on this device");
  Gemm2Params p;
  memset(&p, 0, sizeof(p));
  p.y = (bf16*)y;
  p.ldy = ldy;
  p.M = M;
  p.T = T;
  p.K = K;
  p.m_pairs = ceil_div(M, 2 * BM);
  p.kblocks = ceil_div(K, BK);
  // Token-tile width, and ranges of k for the tiles of the last round where it leaves most pairs idle: least time on the busiest
  // pair.  A k-block costs about (width + 256): the MMA time follows the width, the 128 weight rows per CTA and the hand-offs do
  // not.  Cutting tiles costs as much as CUT_KBLOCKS k-blocks (10 us: partial sums out and in again).  A few wide tiles that run alone
  // behind whole rounds take less than a round (T x M x K = 256 x 19456 x 2560, two of 76 tiles: 38 us whole, 42 cut in four; narrow
  // ones, 128 x 19456 x 2560: 35 whole, 31 cut; 842 x 5120 x 5120, 20 k-blocks instead of 80: 55 whole and 51 cut).
  {
    constexpr int CUT_KBLOCKS = 25;
    long long best_cost = -1;
    for (int bn = 256; bn >= 128; bn -= 32) {
      const long long tiles = (long long)p.m_pairs * ceil_div(T, bn), rounds = tiles / di.max_pairs, rem = tiles % di.max_pairs;
      for (int s = 1; s <= MAX_SPLITS; ++s) {
        if (s > 1) {
          if (rem == 0 || rem * s > di.max_pairs || p.kblocks < 8 * s) break;
          if (sc.ws == nullptr || sc.counters == nullptr || (((uintptr_t)sc.ws) & 15) != 0 || rem * s * 2 * bn * BM * 4 > sc.ws_bytes || rem * 2 * EPI_WARPS * 4 > sc.counter_bytes) break;
        }
        const long long whole = rounds > 0 && bn > 192 && 4 * rem <= di.max_pairs ? p.kblocks * 4 / 5 : p.kblocks;
        const long long cost = (rounds * p.kblocks + (rem == 0 ? 0 : s == 1 ? whole : (p.kblocks + s - 1) / s + CUT_KBLOCKS)) * (bn + 256);
        if (best_cost < 0 || cost < best_cost) {
          best_cost = cost;
          p.bn = bn;
          p.splits = s;
        }
      }
    }
  }
  p.n_tiles = ceil_div(T, p.bn);
  const int total = p.m_pairs * p.n_tiles;
  p.rem = p.splits > 1 ? total % di.max_pairs : 0;
  p.whole = total - p.rem;
  if (plan_out != nullptr) {
    plan_out[0] = p.bn, plan_out[1] = p.whole, plan_out[2] = p.rem, plan_out[3] = p.splits;
    return PG_OK;
  }
  p.part = (float4*)sc.ws;
  p.counters = (uint32_t*)sc.counters;
  const int stage_bytes = A_BYTES + (p.bn / 2) * 128;
  p.stages = (di.max_smem - 1024 - tail) / stage_bytes;
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  PG_REQUIRE(p.stages >= 2, "gemm2sm: not enough shared memory");
  p.tmem_cols = 2 * p.bn > 256 ? 512u : 256u;
  p.status = (uint32_t*)status;
  p.epi = epi;
  p.xielu = (const float*)xielu;
  const size_t smem = 1024 + (size_t)p.stages * stage_bytes + tail;
  CUtensorMap tm_w, tm_x;
  int rc = pg_make_tmap_bf16_2d(&tm_w, w, M, K, ldw, BM, BK);
  if (rc) return rc;
  rc = pg_make_tmap_bf16_2d(&tm_x, x, T, K, ldx, p.bn / 2, BK);
  if (rc) return rc;
  const int items = p.whole + p.rem * p.splits;
  const int npairs = items < di.max_pairs ? items : di.max_pairs;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(2 * npairs));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  int na = 0;
  at[na].id = cudaLaunchAttributeClusterDimension;
  at[na].val.clusterDim.x = 2;
  at[na].val.clusterDim.y = 1;
  at[na].val.clusterDim.z = 1;
  ++na;
  if (pdl_enabled()) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = (unsigned)na;
  PG_CUDA(cudaLaunchKernelEx(&cfg, gemm2sm_bf16_tn_kernel, tm_w, tm_x, p));
  PG_LAUNCH_CHECK();
  return PG_OK;
}
