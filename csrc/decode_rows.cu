// Projections of a few token rows (1 .. 4) as streams of weight rows: single GEMMs, and the dependent GEMMs of a decode step
// (the phases of decode_chain.cu) in one persistent kernel.
//
// At so few rows a step is a read of the weights and a chain of latencies.  The tensor-core form pays per phase for a token
// tile through TMA, an accumulator in tensor memory, stream-K partials in global memory and two grid barriers: 27.5 us for the
// four projections of a layer whose 31 MB take 4.8 us (hidden size 1024, one row).  Here every block owns a contiguous range
// of weight rows, its 16 warps split them by rows and by k, and a warp streams pieces of four rows (256 weights of each, 16 bytes
// a lane) through a ring in shared memory that only its own lanes read, by cp.async, against the token rows in shared memory;
// sums over k meet in shared memory, so a phase needs one grid barrier.  The ring is refilled with the next phase's first pieces
// before the barrier, whose latency and that of the token rows remain: 22 us for the four projections.  (The same ring in
// registers streamed 2.4 TB/s: the loads' results were waited for in one group.  In shared memory: 6.6 TB/s.)  Four rows share
// the conversions of the token rows, products are packed pairs (fma.f32x2).
//
// Outputs are those of the chain: bf16 rows, SwiGLU over alternating (gate, up) rows, residual add with the next norm's weight
// and the sums of squares its consumer needs, or per-head QK norm, rotary embedding and KV append (a pass of their own behind
// the last barrier, over f32 rows in scratch).  Sums are f32 in a fixed order.  All waits are bounded.
#include "api.h"
#include "common.cuh"
#include "decode_rows.h"

namespace {

constexpr int DR_WARPS = 16, DR_THREADS = DR_WARPS * 32;
constexpr int DR_PIECE = 256;  // weights of a row per warp and load
constexpr int DR_QUAD = 4;     // rows that share the reads of the token rows
constexpr int DR_RING = 3;     // quads of pieces that a warp has in flight: 96 KB a block

__device__ __forceinline__ uint32_t dr_ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void dr_copy(uint4* dst, const bf16* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); }
__device__ __forceinline__ void dr_pairs(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// acc.xy += w.xy * x.xy
__device__ __forceinline__ void dr_fma2(float2& acc, float2 w, float2 x) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<unsigned long long&>(acc)) : "l"(reinterpret_cast<const unsigned long long&>(w)), "l"(reinterpret_cast<const unsigned long long&>(x)));
}
__device__ __forceinline__ void dr_pairs2(const uint4& v, float2* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}

// Where a warp is in its pieces of a phase: quads of rows from `row` on in steps of `step` rows, pieces 0 .. per_row - 1 of its part of k
struct DrWalk {
  const bf16* base;  // this lane's 16 bytes of the first piece of the block's row 0
  long long ldw;
  int row, step, rows, piece, per_row;
  __device__ __forceinline__ bool done() const { return row >= rows; }
  __device__ __forceinline__ void next() {
    if (++piece == per_row) {
      piece = 0;
      row += step;
    }
  }
};

template <int T>
__device__ __forceinline__ void decode_rows(const DecodeRows& p) {
  extern __shared__ __align__(16) uint8_t dr_raw[];
  __shared__ float red[DR_WARPS][T], s_inv[T];
  __shared__ int s_abort;
  bf16* xs = reinterpret_cast<bf16*>(dr_raw);                      // [T][K] of the phase
  float* part = reinterpret_cast<float*>(dr_raw + p.x_bytes);      // [row of the block][k split][T]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = blockIdx.x;
  if (tid == 0) s_abort = 0;
  pdl_launch_dependents();

  uint4* ring = reinterpret_cast<uint4*>(dr_raw + p.x_bytes + p.part_bytes) + warp * DR_RING * DR_QUAD * 32 + lane;  // [slot][row][lane]: every lane reads what it copied
  DrWalk ld;
  int slot = 0;
  auto enter = [&](const DecodeRowsPhase& P) {
    const int r0 = c * P.rows, split = warp % P.splits;
    DrWalk w;
    w.ldw = P.ldw;
    w.base = P.w + (long long)r0 * P.ldw + split * P.per_row * DR_PIECE + lane * 8;
    w.row = warp / P.splits * DR_QUAD;
    w.step = DR_WARPS / P.splits * DR_QUAD;
    w.rows = min(P.rows, P.M - r0);  // (not positive: a block without rows)
    w.piece = 0;
    w.per_row = P.per_row;
    return w;
  };
  auto fetch = [&](int to) {  // the next pieces of a quad (rows past the last: the last again)
    if (!ld.done()) {
#pragma unroll
      for (int i = 0; i < DR_QUAD; ++i) dr_copy(ring + (to * DR_QUAD + i) * 32, ld.base + min(ld.row + i, ld.rows - 1) * ld.ldw + ld.piece * DR_PIECE);
      ld.next();
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto fill = [&]() {
    slot = 0;
#pragma unroll
    for (int u = 0; u < DR_RING; ++u) fetch(u);
  };
  // waits until every block has finished phase ph (all threads call it)
  auto grid_wait = [&](int ph) {
    if (tid == 0 && dr_ld_acquire(p.counters + ph) < gridDim.x) {
      const uint64_t t0 = globaltimer_ns();
      uint32_t spins = 0;
      while (dr_ld_acquire(p.counters + ph) < gridDim.x) {
        if ((++spins & 31u) == 0u) {
          if (*((volatile uint32_t*)p.status) != PG_ST_OK) s_abort = 1;  // another block gave up
          if (globaltimer_ns() - t0 > PG_WAIT_LIMIT_NS) {
            atomicCAS(p.status, PG_ST_OK, PG_ST_TIMEOUT | (59u << 8));
            s_abort = 1;
          }
          if (s_abort) break;
        }
      }
    }
    __syncthreads();
    return s_abort == 0;
  };
  auto sum_squares = [&](const DecodeRowsPhase& P, int first, int stride) {  // of the residual rows, per tile of 128: units (tile, token)
    for (int u = first; u < P.M / 128 * T; u += stride) {
      const int tile = u / T, t = u % T;
      const uint2 h = __ldcg(reinterpret_cast<const uint2*>(p.residual + t * p.ld_res + tile * 128) + lane);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(&h.x)), b = __bfloat1622float2(*reinterpret_cast<const bf162*>(&h.y));
      const float ss = warp_sum(a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y);
      if (lane == 0) P.out_ssp[t * P.out_ld + tile] = ss;
    }
  };

  ld = enter(p.ph[0]);
  fill();
  pdl_wait();
  bool ok = true;
  for (int ph = 0; ph < p.nphase; ++ph) {
    const DecodeRowsPhase& P = p.ph[ph];
    if (ph > 0) {
      ok = grid_wait(ph - 1);
      if (!ok) break;
    }
    // ---- token rows, and what their deferred norm still owes ----
    for (int t = 0; t < T; ++t)
      for (int i = tid; i < P.K / 8; i += DR_THREADS) reinterpret_cast<uint4*>(xs + (long long)t * P.K)[i] = __ldcg(reinterpret_cast<const uint4*>(P.x + t * P.ldx) + i);
    if (P.in_ssp != nullptr) {
      float ss[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        ss[t] = 0.f;
        if (ph > 0) {  // the sums of squares of the rows that the phase before this one left
          for (int i = tid; i < P.K / 8; i += DR_THREADS) {
            float h[8];
            dr_pairs(__ldcg(reinterpret_cast<const uint4*>(p.residual + t * p.ld_res) + i), h);
#pragma unroll
            for (int j = 0; j < 8; ++j) ss[t] += h[j] * h[j];
          }
        } else {
          for (int i = tid; i < P.in_parts; i += DR_THREADS) ss[t] += __ldcg(P.in_ssp + t * P.in_ld + i);
        }
        ss[t] = warp_sum(ss[t]);
        if (lane == 0) red[warp][t] = ss[t];
      }
      __syncthreads();
      if (tid < T) {
        float s = 0.f;
        for (int w = 0; w < DR_WARPS; ++w) s += red[w][tid];
        s_inv[tid] = rsqrtf(s / (float)P.in_width + P.in_eps);
      }
    } else if (tid < T) {
      s_inv[tid] = 1.f;
    }
    if (ph > 0 && p.ph[ph - 1].epi == DR_RESID_NORM && warp == DR_WARPS - 1) sum_squares(p.ph[ph - 1], c, gridDim.x);
    __syncthreads();
    // ---- this block's weight rows ----
    {
      DrWalk cur = enter(P);
      const bf16* xk = xs + (warp % P.splits) * P.per_row * DR_PIECE + lane * 8;
      constexpr int V = T == 3 ? 16 : DR_QUAD * T;  // sums of a quad, [row][token]
      float2 acc[DR_QUAD][T];
#pragma unroll
      for (int i = 0; i < DR_QUAD; ++i)
#pragma unroll
        for (int t = 0; t < T; ++t) acc[i][t] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (; !cur.done(); cur.next()) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DR_RING - 1) : "memory");
        uint4 raw[DR_QUAD];
#pragma unroll
        for (int i = 0; i < DR_QUAD; ++i) raw[i] = ring[(slot * DR_QUAD + i) * 32];
        fetch(slot);
        slot = slot + 1 == DR_RING ? 0 : slot + 1;
        float2 x[T][4];
#pragma unroll
        for (int t = 0; t < T; ++t) dr_pairs2(*reinterpret_cast<const uint4*>(xk + t * P.K + cur.piece * DR_PIECE), x[t]);
#pragma unroll
        for (int i = 0; i < DR_QUAD; ++i) {
          float2 w[4];
          dr_pairs2(raw[i], w);
#pragma unroll
          for (int t = 0; t < T; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) dr_fma2(acc[i][t], w[j], x[t][j]);
        }
        if (cur.piece == P.per_row - 1) {
          // sums over the lanes, halving the values that a lane holds: lane bits 4, 3, .. name the value, the rest is summed
          float v[V];
#pragma unroll
          for (int i = 0; i < V; ++i) {
            v[i] = i < DR_QUAD * T ? acc[i / T][i % T].x + acc[i / T][i % T].y : 0.f;
            if (i < DR_QUAD * T) acc[i / T][i % T] = make_float2(0.f, 0.f);
          }
          int bit = 16;
#pragma unroll
          for (int n = V / 2; n > 0; n >>= 1, bit >>= 1) {
            const bool up = lane & bit;
#pragma unroll
            for (int i = 0; i < n; ++i) {
              const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
              v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
            }
          }
          const int which = lane / (32 / V);
#pragma unroll
          for (int o = 32 / V / 2; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
          const int q = which / T, t = which % T;
          if (lane % (32 / V) == 0 && which < DR_QUAD * T && cur.row + q < cur.rows) part[((cur.row + q) * P.splits + warp % P.splits) * T + t] = v[0];
        }
      }
    }
    if (ph + 1 < p.nphase) {  // weights do not wait for anyone
      ld = enter(p.ph[ph + 1]);
      fill();
    }
    __syncthreads();
    // ---- sums over the k splits, and the phase's output ----
    const int m0 = c * P.rows, rows = min(P.rows, P.M - m0);
    auto value = [&](int r, int t) {
      float s = 0.f;
      for (int q = 0; q < P.splits; ++q) s += part[(r * P.splits + q) * T + t];
      return s * s_inv[t];
    };
    if (P.epi == DR_SWIGLU) {
      for (int i = tid; i < rows / 2 * T; i += DR_THREADS) {
        const int r = i % (rows / 2), t = i / (rows / 2);
        const float g = bf16_round(value(2 * r, t)), u = bf16_round(value(2 * r + 1, t));
        P.out[t * P.ld_out + (m0 >> 1) + r] = __float2bfloat16(bf16_round(g / (1.f + __expf(-g))) * u);
      }
    } else {
      for (int i = tid; i < rows * T; i += DR_THREADS) {
        const int r = i % rows, t = i / rows, m = m0 + r;
        const float v = value(r, t);
        if (P.epi == DR_RESID_NORM) {
          unsigned short* res = reinterpret_cast<unsigned short*>(p.residual + t * p.ld_res + m);
          const bf16 h = __float2bfloat16(v + __bfloat162float(__ushort_as_bfloat16(__ldcg(res))));
          *res = __bfloat16_as_ushort(h);
          P.out[t * P.ld_out + m] = __float2bfloat16(__bfloat162float(h) * (__bfloat162float(P.norm_w[m]) + (P.norm_offset ? 1.f : 0.f)));
        } else if (P.epi == DR_QKV_ROPE) {
          p.scratch[(long long)t * P.M + m] = bf16_round(v);
        } else if (P.out_f32) {
          reinterpret_cast<float*>(P.out)[t * P.ld_out + m] = v;
        } else {
          P.out[t * P.ld_out + m] = __float2bfloat16(v);
        }
      }
    }
    __syncthreads();
    if (p.barriers && tid == 0) {
      __threadfence();
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.counters + ph) : "memory");
    }
  }
  const DecodeRowsPhase& L = p.ph[p.nphase - 1];
  if (ok && L.epi == DR_RESID_NORM) {
    ok = grid_wait(p.nphase - 1);
    if (ok && warp == 0) sum_squares(L, c, gridDim.x);
  }
  if (ok && L.epi == DR_QKV_ROPE) {
    ok = grid_wait(p.nphase - 1);
    const int heads = L.hq + 2 * L.hkv;
    // warps of different blocks first: few heads are spread over the chip
    for (int u = warp * gridDim.x + c; ok && u < heads * T; u += gridDim.x * DR_WARPS) {
      const int h = u / T, t = u % T;
      const float4 in = __ldcg(reinterpret_cast<const float4*>(p.scratch + (long long)t * L.M + h * 128) + lane);
      float v[4] = {in.x, in.y, in.z, in.w};
      int slot = 0;
      if (h >= L.hq) {
        slot = L.slots[t];
        if (slot < 0 || slot >= L.num_slots) {
          if (lane == 0) atomicCAS(p.status, PG_ST_OK, PG_ST_BOUNDS | (3u << 8));
          continue;
        }
      }
      const long long page = slot / L.page_size, off = slot % L.page_size;
      bf16* dst;
      if (h >= L.hq + L.hkv) {
        dst = L.kv + (((page * 2 + 1) * L.page_size + off) * L.hkv + (h - L.hq - L.hkv)) * 128;
      } else {
        int pos = L.positions[t];
        if (pos < 0 || pos >= L.max_pos) {
          if (lane == 0) atomicCAS(p.status, PG_ST_OK, PG_ST_BOUNDS | (4u << 8));
          pos = pos < 0 ? 0 : L.max_pos - 1;
        }
        if (L.q_w != nullptr) {
          const float inv = rsqrtf(warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]) / 128.f + L.qk_eps);
          const uint2 nw = *reinterpret_cast<const uint2*>((h < L.hq ? L.q_w : L.k_w) + lane * 4);
          const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(&nw.x)), b = __bfloat1622float2(*reinterpret_cast<const bf162*>(&nw.y));
          const float w[4] = {a.x, a.y, b.x, b.y}, add = L.norm_offset ? 1.f : 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = bf16_round(v[j] * inv * (w[j] + add));
        }
        const int half = L.rot >> 1;  // 64 (element i pairs with i +- 64, lane +- 16) or 0
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float other = __shfl_xor_sync(0xffffffffu, v[j], 16);
          if (half > 0) {
            const int i = lane * 4 + j;
            const long long at = (long long)pos * half + (i < half ? i : i - half);
            const float sn = __bfloat162float(L.sin[at]);
            v[j] = v[j] * __bfloat162float(L.cos[at]) + (i < half ? -other : other) * sn;
          }
        }
        dst = h < L.hq ? L.out + ((long long)t * L.hq + h) * 128 : L.kv + (((page * 2 + 0) * L.page_size + off) * L.hkv + (h - L.hq)) * 128;
      }
      const bf162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
      uint2 pk;
      pk.x = *reinterpret_cast<const uint32_t*>(&lo);
      pk.y = *reinterpret_cast<const uint32_t*>(&hi);
      *reinterpret_cast<uint2*>(dst + lane * 4) = pk;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");  // a block that gave up has pieces of the next phase in flight
  // the last block out leaves the counters at zero for the next launch
  if (p.barriers && tid == 0 && atomicAdd(p.counters + DR_MAX_PHASES, 1u) == gridDim.x - 1) {
    for (int i = 0; i <= DR_MAX_PHASES; ++i) p.counters[i] = 0u;
  }
}

// One body, two names: a launch of dependent phases, and a single GEMM
template <int T>
__global__ void __launch_bounds__(DR_THREADS, 1) rows_decode_chain_kernel(const __grid_constant__ DecodeRows p) {
  decode_rows<T>(p);
}
template <int T>
__global__ void __launch_bounds__(DR_THREADS, 1) rows_gemm_bf16_tn_kernel(const __grid_constant__ DecodeRows p) {
  decode_rows<T>(p);
}

struct DrDevice {
  int sms, smem;
};
bool dr_device(DrDevice* d) {
  static DrDevice known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return false;
  if (known[dev].sms == 0) {
    int sms = 0, smem = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return false;
    smem -= 1024;  // static shared memory
    for (auto k : {rows_decode_chain_kernel<1>, rows_decode_chain_kernel<2>, rows_decode_chain_kernel<3>, rows_decode_chain_kernel<4>, rows_gemm_bf16_tn_kernel<1>, rows_gemm_bf16_tn_kernel<2>, rows_gemm_bf16_tn_kernel<3>,
                   rows_gemm_bf16_tn_kernel<4>})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return false;
    known[dev].smem = smem;
    known[dev].sms = sms;
  }
  *d = known[dev];
  return true;
}

}  // namespace

bool decode_rows_plan(DecodeRows& p, int T) {
  DrDevice d;
  if (T < 1 || T > DR_MAX_ROWS || !dr_device(&d)) return false;
  long long x_bytes = 0, part_bytes = 0;
  for (int i = 0; i < p.nphase; ++i) {
    DecodeRowsPhase& P = p.ph[i];
    const int pieces = P.K / DR_PIECE;
    if (P.K % DR_PIECE != 0 || pieces == 0 || P.ldw % 8 != 0 || P.ldx % 8 != 0 || (((uintptr_t)P.w | (uintptr_t)P.x) & 15) != 0 || P.M < 2 || P.M % 2 != 0) return false;
    if (P.epi == DR_RESID_NORM && P.M % 128 != 0) return false;
    // a phase behind RESID_NORM forms the sums of squares of the residual rows that phase left: it must not write them itself (the
    // tile kernel takes such chains), and sums that it takes in must be those
    if (i > 0 && P.epi == DR_RESID_NORM && p.ph[i - 1].epi == DR_RESID_NORM) return false;
    if (i > 0 && P.in_ssp != nullptr && (p.ph[i - 1].epi != DR_RESID_NORM || P.in_ssp != p.ph[i - 1].out_ssp || p.ph[i - 1].M != P.K || P.in_width != P.K || p.ld_res % 8 != 0 || ((uintptr_t)p.residual & 15) != 0)) return false;
    const int unit = P.M >= d.sms * 2 * DR_QUAD ? DR_QUAD : 2;
    P.rows = ceil_div(ceil_div(P.M, d.sms), unit) * unit;
    // warps split k only as far as that evens out the rows: the least work on the busiest warp, where the sums over the lanes that
    // end a quad of rows cost a quarter of a quad of pieces and as much again for every token row
    int best = 0, least = 0;
    for (int s = 1; s <= DR_WARPS; s *= 2) {
      if (pieces % s) break;
      const int steps = ceil_div(ceil_div(P.rows, DR_QUAD), DR_WARPS / s) * (4 * (pieces / s) + 1 + T);
      if ((long long)P.rows * s * T * 4 > 64 * 1024) break;
      if (best == 0 || steps < least) best = s, least = steps;
    }
    if (best == 0) return false;
    P.splits = best;
    P.per_row = pieces / best;
    const long long xb = (long long)T * P.K * 2, pb = (long long)P.rows * best * T * 4;
    x_bytes = xb > x_bytes ? xb : x_bytes;
    part_bytes = pb > part_bytes ? pb : part_bytes;
  }
  part_bytes = (part_bytes + 15) & ~15ll;
  const long long ring_bytes = (long long)DR_THREADS * DR_RING * DR_QUAD * 16;
  if (x_bytes + part_bytes + ring_bytes > d.smem) return false;
  p.x_bytes = (int)x_bytes;
  p.part_bytes = (int)part_bytes;
  p.smem = (int)(x_bytes + part_bytes + ring_bytes);
  p.grid = d.sms;
  return true;
}

int decode_rows_run(const DecodeRows& p, int T, cudaStream_t stream) {
  auto chain = T == 1 ? rows_decode_chain_kernel<1> : T == 2 ? rows_decode_chain_kernel<2> : T == 3 ? rows_decode_chain_kernel<3> : rows_decode_chain_kernel<4>;
  auto gemm = T == 1 ? rows_gemm_bf16_tn_kernel<1> : T == 2 ? rows_gemm_bf16_tn_kernel<2> : T == 3 ? rows_gemm_bf16_tn_kernel<3> : rows_gemm_bf16_tn_kernel<4>;
  auto kernel = p.nphase > 1 ? chain : gemm;
  PG_CUDA(launch_pdl(kernel, dim3((unsigned)p.grid), dim3(DR_THREADS), (size_t)p.smem, stream, p));
  PG_LAUNCH_CHECK();
  return PG_OK;
}
