// Absorbed latent attention of single query rows on tcgen05 (latents of 512 columns with 64 rotated ones or none).
//
// All heads of a row read the same keys, so the heads are the narrow side of both products and everything is transposed:
// with a tile of 64 keys in shared memory, S^T [64 keys, heads] = K Q^T and O^T [512, heads] += V^T P^T, four accumulators of
// 128 value columns x heads in tensor memory.  K is the tile read K-major, V^T the same bytes read MN-major, Q stays in
// shared memory, P^T is written back MN-major (a key's row of heads).  A tile is made of eight boxes of eight keys, each one
// copy of [block of 64 columns][8 keys][128 bytes] (a 16-token page is two of them; boxes of one block and a page's keys are
// 36 copies of 2 KB a tile, which took 1.25 us to issue), and the operand descriptors step from box to box.  Two tiles of
// 72 KB, Q (72 KB at 64 heads) and P fill the shared memory, so a CTA owns an SM.  Up to DT_ROWS rows the CTAs, one an SM, share all tiles
// of the step evenly (dt_shares): a CTA walks pieces of rows one behind the other, copies and queries of the next piece under the
// last tiles of the one before, and a second kernel joins the rows that were cut.  So a row of more than DT_WHOLE tiles is cut where the
// lengths of all rows of the step say, and weights are rounded to bf16 against a reference that starts anew with a piece: its sums
// are those of the step, not of the row alone.  A caller that wants the latter gives no scratch, and a block walks a row.
//
// A product of 64 rows leaves them in the lower half of each warp's tensor-memory lanes: a warp has 16 keys, and a thread
// reads two of them for a quarter of the heads.  Rows are reduced across threads only when it matters: exponentials refer to
// a reference value per head that moves only if some score exceeds it by more than 2^8 (the tile's maxima are formed then, and
// O and the sums rescaled), and each thread sums its own keys' weights, added up once at the end.
//
// Rows of a tile that are no keys are cleared in shared memory, adjacent lanes adjacent bytes (lanes a block of columns apart met in the same
// banks: one row of 8 keys, 16 heads, 25.2 us for the whole operation against 23.4 now; 21.1 on the mma.sync kernel).
//
// Against the mma.sync kernel, in which a CTA of 16 heads exchanges partial scores through shared memory for every 32 keys
// (128 rows x 64 heads x 1150 keys): 284 us; 90 with a
// block a row, 75 with the descriptors of a tile's 52 products in uniform registers, 54 and some 4 for the join with even shares (and an
// output that steps pointers: it took 11 us a piece).  37 rows x 64 heads x 900 keys, the whole operation: 72 us, 50 now.  What bounds it: the
// keys' bytes, 31 us of it at 5.4 TB/s; start, queries and output of 1.9 pieces a block are the rest.
#include "api.h"
#include "attention_tc.cuh"
#include "mla_decode_tc.h"

namespace {

constexpr int DT_KEYS = 64;
constexpr int DT_P = DT_KEYS * 128;      // weights: 64 keys x 64 heads
constexpr int DT_THREADS = 320;          // producer, MMA, four softmax / epilogue warps, four warps that fetch queries
constexpr int DT_ROWS = 512;             // rows whose keys the blocks share
// Rows of up to so many tiles are not cut.  Steps whose longest row the host knows to be no longer get no scratch, no shares and no join (128 rows of
// 100 keys 32 us the whole operation, 36 with them); a captured step, which knows a bound only, has them all the same.
constexpr int DT_WHOLE = 4;
constexpr float DT_NONE = -1e30f;        // reference of a head that has seen no key; also "no keys" among the partial results

template <int HN>
struct DtSync {
  uint64_t full[2], empty[2], cleared, s_full[2], p_ready, o_full, q_full, q_free;
  uint32_t tmem_slot;
  int abort_flag;
  alignas(16) int grew[2][4];          // by tile parity and warp: some score exceeds its reference by too much
  float ref[HN], fac[HN];  // log2 units; factor on what was summed so far, at the end on the output
  float part[4][HN];       // per warp: maxima of a tile, at the end sums of weights
  int from_unit, from_tile, to_unit, to_tile;  // this block's share
};

// A query row's keys, in tiles.
struct DtRow {
  int b, pos, begin, end, tile0, tiles;
};
__device__ __forceinline__ DtRow dt_row(const MlaDecodeTc& p, int t) {
  DtRow r;
  r.b = p.unit_seq[p.first_row + t];
  const int q0 = p.q_indptr[r.b], q1 = p.q_indptr[r.b + 1], kv_len = p.kv_lens[r.b];
  r.pos = kv_len - (q1 - q0) + (p.first_row + t - q0);  // of this query token
  r.end = kv_len == 0 ? 0 : r.pos + 1;
  r.begin = p.window > 0 ? max(0, r.end - p.window) : 0;
  r.tile0 = r.begin / DT_KEYS;
  r.tiles = r.end > 0 ? (r.end + DT_KEYS - 1) / DT_KEYS - r.tile0 : 0;
  return r;
}

// The share of block c, when the blocks share the tiles of all units (row, group of heads), row by row: boundaries at even numbers of
// tiles, moved to the ends of a row that is short or that would lose less than two tiles.  Rows stay whole where there is a block for
// every unit and the longest one takes no more than an even share and three tiles (some 6 us: what the partial results of cut rows and
// their merge cost).  All threads; `n`: DT_ROWS + 2 ints of shared memory that nothing else uses yet.
template <int HN>
__device__ __forceinline__ void dt_shares(const MlaDecodeTc& p, int groups, int* n, DtSync<HN>* sh) {
  for (int t = threadIdx.x; t < p.tokens; t += DT_THREADS) n[t] = dt_row(p, t).tiles;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, each = (p.tokens + 31) / 32, t0 = min(p.tokens, lane * each), t1 = min(p.tokens, t0 + each);
    int sum = 0, longest = 0;
    for (int t = t0; t < t1; ++t) {
      sum += n[t];
      longest = max(longest, n[t]);
    }
    int upto = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    int at = upto - sum;
    for (int t = t0; t < t1; ++t) {  // tiles in front of a row
      const int x = n[t];
      n[t] = at;
      at += x;
    }
    const int all = __shfl_sync(0xffffffffu, upto, 31);
    if (lane == 0) n[p.tokens] = all;
    __syncwarp();
    const int blocks = (int)gridDim.x, units = p.tokens * groups, total = all * groups;
    const int share = max(DT_WHOLE, (total + blocks - 1) / blocks);
    const bool whole = units <= blocks && longest <= share + 3;
    // boundary in front of block c: a unit, and a tile of it
    auto boundary = [&](int c, int& unit, int& tile) {
      if (whole) {
        unit = min(c, units), tile = 0;
        return;
      }
      const long long pos = (long long)c * share;
      unit = tile = 0;
      if (c == 0) return;  // (rows without keys at the front are the first block's)
      if (pos >= total) {
        unit = units, tile = 0;
        return;
      }
      int lo = 0, hi = p.tokens;  // the last row with n[lo] * groups <= pos: one that has tiles
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if ((long long)n[mid] * groups <= pos) lo = mid; else hi = mid;
      }
      const int len = n[lo + 1] - n[lo], off = (int)(pos - (long long)n[lo] * groups);
      unit = lo * groups + off / len;
      tile = off % len;
      if (len <= DT_WHOLE ? 2 * tile < len : tile < 2) {
        tile = 0;
      } else if (len <= DT_WHOLE || len - tile < 2) {
        ++unit;
        tile = 0;
      }
    };
    int u, tile, pieces = 0, last = -1;
    for (int c = (int)blockIdx.x;; c += 31) {  // lane l: the boundary in front of block c + l
      boundary(c + lane, u, tile);
      const int u1 = __shfl_sync(0xffffffffu, u, 1), x1 = __shfl_sync(0xffffffffu, tile, 1);
      if (c == (int)blockIdx.x) {
        if (lane == 0) sh->from_unit = u, sh->from_tile = tile;
        if (lane == 1) sh->to_unit = u, sh->to_tile = tile;
        const int u0 = __shfl_sync(0xffffffffu, u, 0), x0 = __shfl_sync(0xffffffffu, tile, 0);
        if (x1 == 0 || (u0 == u1 && x0 > 0)) break;  // no row that begins here ends elsewhere
        last = u1;
        pieces = 1;
      }
      const uint32_t cut = __ballot_sync(0xffffffffu, lane > 0 && u == last && tile > 0);  // boundaries inside that row
      const int run = __ffs((int)~(cut >> 1)) - 1;
      pieces += run;
      if (run < 31) break;
    }
    if (lane == 0) *reinterpret_cast<int2*>(p.cuts + 2 * blockIdx.x) = make_int2(last, pieces);
  }
  fence_proxy_async_smem();  // the tiles' copies write where `n` was
  __syncthreads();
}

__device__ __forceinline__ void dt_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// 16 lanes x HN columns of tensor memory as mma fragments: r[4 i + e] = lane (lane / 4, + 8 for e >= 2), column 8 i + 2 (lane % 4) + (e & 1).
template <int HN>
__device__ __forceinline__ void dt_ld_frag(uint32_t taddr, uint32_t* r) {
#pragma unroll
  for (int c = 0; c < HN / 16; ++c)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[8 * c]), "=r"(r[8 * c + 1]), "=r"(r[8 * c + 2]), "=r"(r[8 * c + 3]), "=r"(r[8 * c + 4]), "=r"(r[8 * c + 5]), "=r"(r[8 * c + 6]), "=r"(r[8 * c + 7])
                 : "r"(taddr + 16 * c)
                 : "memory");
}
// K-major operand whose groups of eight rows are `sbo` bytes apart
__device__ __forceinline__ uint64_t dt_desc_k(uint32_t smem_addr, uint32_t sbo) {
  return (umma_desc_k_sw128(smem_addr) & ~((uint64_t)0x3FFF << 32)) | (uint64_t)(sbo >> 4) << 32;
}

// Tiles of a piece whose last rows, and whose first rows (in front of a window), are no keys; one of another piece is not in 0 .. tiles - 1.
__device__ __forceinline__ int dt_ragged(const DtRow& r, int first) { return r.end % DT_KEYS ? r.tile0 + r.tiles - 1 - first : -1; }
__device__ __forceinline__ int dt_head(const DtRow& r, int first) { return r.begin % DT_KEYS ? r.tile0 - first : -1; }

// A block takes pieces of units (token row, group of HN heads), tiles of 64 keys in turn.  QKB: 64-column blocks of a key.
template <int HN, int QKB>
__global__ void __launch_bounds__(DT_THREADS, 1) mla_decode_tc_kernel(const __grid_constant__ CUtensorMap tm, const MlaDecodeTc p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  uint8_t* tiles = smem_raw + (((base + 1023u) & ~1023u) - base);
  constexpr int BOX = QKB * 1024, STAGE = DT_KEYS / 8 * BOX, QBLK = HN * 128;
  uint8_t* q_sm = tiles + 2 * STAGE;
  uint8_t* p_sm = q_sm + QKB * QBLK;
  DtSync<HN>* sh = reinterpret_cast<DtSync<HN>*>(p_sm + DT_P);
  constexpr uint32_t TMEM_COLS = HN == 64 ? 512 : HN == 32 ? 256 : 128;  // S twice, O four times
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (p.heads + HN - 1) / HN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
      mbar_init(&sh->s_full[s], 1);
    }
    mbar_init(&sh->cleared, 4);
    mbar_init(&sh->p_ready, 4);
    mbar_init(&sh->o_full, 1);
    mbar_init(&sh->q_full, 128);
    mbar_init(&sh->q_free, 1);
    sh->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm);
  }
  if (warp == 1) {
    tmem_alloc(&sh->tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_slot;
  volatile int* abort_flag = &sh->abort_flag;
  PG_PDL_ENTRY();

  if (p.shared) {
    dt_shares<HN>(p, groups, reinterpret_cast<int*>(tiles), sh);
  } else if (threadIdx.x == 0) {
    sh->from_unit = blockIdx.x, sh->to_unit = blockIdx.x + 1;
    sh->from_tile = sh->to_tile = 0;
  }
  __syncthreads();
  const int from_unit = sh->from_unit, from_tile = sh->from_tile, to_unit = sh->to_unit, to_tile = sh->to_tile;
  // f(row of the step, group of heads, its keys, first tile, tiles, whole): the pieces of this block's share in turn, the same for every role;
  // those of a row without keys have no tiles
  auto pieces = [&](auto&& f) {
    for (int unit = from_unit; unit < to_unit || (unit == to_unit && to_tile > 0); ++unit) {
      const int t = unit / groups;
      const DtRow r = dt_row(p, t);
      const int first = unit == from_unit ? from_tile : 0, end = unit == to_unit ? to_tile : r.tiles;
      f(t, (unit - t * groups) * HN, r, r.tile0 + first, end - first, first == 0 && end == r.tiles);
    }
  };

  if (warp == 0) {
    const uint64_t pol = l2_policy_evict_first();
    bool ok = true;
    int i = 0;  // tiles so far
    pieces([&](int, int, const DtRow& r, int first, int n_tiles, bool) {
      const int* table = p.table + (long long)r.b * p.table_stride;
      for (int j = 0; j < n_tiles && ok; ++j, ++i) {
        const int st = i & 1, key = (first + j) * DT_KEYS + lane * 8;  // of this lane's box
        const int boxes = min(DT_KEYS / 8, (r.end - (first + j) * DT_KEYS + 7) / 8);
        const int page = lane < boxes ? table[min(key / p.page_size, p.table_stride - 1)] : 0;
        if (i >= 2) ok = mbar_wait(&sh->empty[st], (uint32_t)(((i >> 1) - 1) & 1), abort_flag);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&sh->full[st], (uint32_t)(boxes * BOX));
        __syncwarp();
        if (lane < boxes) tma_load_3d(tiles + st * STAGE + lane * BOX, &tm, &sh->full[st], 0, page * p.page_size + key % p.page_size, 0, pol);
      }
    });
  } else if (warp >= 6) {
    // a piece's queries into shared memory while its first tiles are on their way, or the last ones of the piece before are
    // worked on: [block][head][128 B], 128-byte swizzle
    int n = 0;
    bool ok = true;
    pieces([&](int t, int h0, const DtRow& r, int, int n_tiles, bool) {
      if (n_tiles == 0) return;
      ok = ok && (n == 0 || mbar_wait(&sh->q_free, (uint32_t)((n - 1) & 1), abort_flag));
      if (ok)
        for (int i = threadIdx.x - 192; i < HN * QKB * 8; i += 128) {
          const int h = i / (QKB * 8), ch = i % (QKB * 8), head = min(h0 + h, p.heads - 1);  // heads past the last: any row, not stored
          uint4* dst = reinterpret_cast<uint4*>(q_sm + (ch >> 3) * QBLK + h * 128 + (((ch & 7) ^ (h & 7)) << 4));
          const bf16* src = ch < 64 ? p.q_abs + t * p.q_tok + head * p.q_head + ch * 8 : p.q_pe + t * p.pe_tok + head * p.pe_head + (ch - 64) * 8;
          if (ch < 64 || p.cos == nullptr) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
          } else {
            uint4 v = *reinterpret_cast<const uint4*>(src);
            const long long at = (long long)min(max(r.pos, 0), p.max_pos - 1) * 32 + (ch - 64) * 4;
            uint32_t* w = &v.x;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __bfloat1622float2(*reinterpret_cast<const bf162*>(&w[j]));
              const float cs = p.cos[at + j], sn = p.sin[at + j];
              const bf162 x = __floats2bfloat162_rn(f.x * cs - f.y * sn, f.y * cs + f.x * sn);
              w[j] = *reinterpret_cast<const uint32_t*>(&x);
            }
            *dst = v;
          }
        }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
      fence_proxy_async_smem();
      mbar_arrive(&sh->q_full);
      ++n;
    });
  } else if (warp == 1) {
    {
      // The whole warp walks the loop and one lane issues: descriptors are sums of what does not depend on the lane, so they stay in
      // uniform registers (formed anew by a lone thread for each product, they took longer than the product).
      const bool leader = elect_one();
      constexpr uint32_t idesc_s = idesc_bf16(DT_KEYS, HN, 0);
      constexpr uint32_t idesc_o = idesc_bf16(128, HN, 1) | (1u << 15);  // both operands MN-major
      const uint32_t t0 = smem_u32(tiles);
      const uint64_t k_desc = dt_desc_k(t0, BOX), v_desc = umma_desc_mn_sw128(t0, 1024u, BOX), q_desc = umma_desc_k_sw128(smem_u32(q_sm)), p_desc = umma_desc_mn_sw128(smem_u32(p_sm), DT_P, 1024u);
      // Whatever is ready goes first: the product with V as soon as P is there (it frees the tile's memory), the scores of the
      // next tile as soon as it has landed.  (Scores always first left a finished P waiting for a tile that could only be
      // fetched after that product: 3.9 us a tile.)
      int base_i = 0, n = 0, clears = 0;  // tiles and pieces so far, tiles with cleared rows
      bool ok = true;
      pieces([&](int, int, const DtRow& r, int first, int n_tiles, bool) {
        if (n_tiles == 0 || !ok) return;
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(&sh->q_full, (uint32_t)(n & 1), abort_flag));
        ++n;
        const int ragged = dt_ragged(r, first), head = dt_head(r, first);
        int s_next = 0, o_next = 0;
        uint32_t spins = 0;
        uint64_t since = globaltimer_ns();
        while (ok && o_next < n_tiles) {
          const int si = base_i + s_next, oi = base_i + o_next, ss = si & 1, os = oi & 1;
          const bool cleared = s_next == ragged || s_next == head;
          if (s_next > o_next && __all_sync(0xFFFFFFFFu, mbar_try_wait(&sh->p_ready, (uint32_t)(oi & 1)))) {
            tc_fence_after();
            if (leader) {
              const uint64_t v = v_desc + (uint32_t)(os * (STAGE >> 4));
#pragma unroll
              for (int mb = 0; mb < 4; ++mb)
#pragma unroll
                for (int ks = 0; ks < DT_KEYS / 16; ++ks)
                  umma_bf16_ss(tmem + (uint32_t)((2 + mb) * HN), v + (uint32_t)((mb * 2048 + ks * 2 * BOX) >> 4), p_desc + (uint32_t)(ks * 128), idesc_o, (o_next | ks) ? 1u : 0u);
              umma_commit(&sh->o_full);
              umma_commit(&sh->empty[os]);
            }
            ++o_next;
          } else if (s_next < n_tiles && s_next <= o_next + 1 &&
                     __all_sync(0xFFFFFFFFu, mbar_try_wait(&sh->full[ss], (uint32_t)((si >> 1) & 1)) && (!cleared || mbar_try_wait(&sh->cleared, (uint32_t)(clears & 1))))) {
            tc_fence_after();
            clears += cleared;
            if (leader) {
              const uint64_t k = k_desc + (uint32_t)(ss * (STAGE >> 4));
#pragma unroll
              for (int cb = 0; cb < QKB; ++cb)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  umma_bf16_ss(tmem + (uint32_t)(ss * HN), k + (uint32_t)(cb * 64 + i * 2), q_desc + (uint32_t)(cb * (QBLK >> 4) + i * 2), idesc_s, (cb | i) ? 1u : 0u);
              umma_commit(&sh->s_full[ss]);
              if (s_next + 1 == n_tiles) umma_commit(&sh->q_free);
            }
            ++s_next;
          } else {
            if (__any_sync(0xFFFFFFFFu, (++spins & 63u) == 0u && (*abort_flag || globaltimer_ns() - since > PG_WAIT_LIMIT_NS))) {
              *abort_flag = 1;
              ok = false;
            }
            continue;
          }
          since = globaltimer_ns();
        }
        base_i += n_tiles;
      });
    }
  } else {
    const int wq = warp & 3, tid = wq * 32 + lane;  // tensor-memory lanes of this warp: 32 wq ..
    const uint32_t row = tmem + ((uint32_t)(wq * 32) << 16);
    const int key_a = wq * 16 + (lane >> 2), col = 2 * (lane & 3);  // keys key_a and key_a + 8, heads 8 i + col and the next one
    constexpr int HB = HN / 8;
    int base_i = 0;  // tiles so far
    bool ok = true;  // after a wait that ran out the warps go on through the barriers, without work
    pieces([&](int t, int h0, const DtRow& r, int first, int n_tiles, bool whole) {
    const int kv_begin = r.begin, kv_end = r.end, ragged = dt_ragged(r, first), head = dt_head(r, first);
    float l[HB][2], ref[HB][2];
#pragma unroll
    for (int i = 0; i < HB; ++i) l[i][0] = l[i][1] = 0.f, ref[i][0] = ref[i][1] = DT_NONE;
    if (tid < HN) sh->ref[tid] = DT_NONE;
    for (int j = 0; j < n_tiles; ++j) {
      const int ji = base_i + j, st = ji & 1, key0 = (first + j) * DT_KEYS;
      if (j == ragged || j == head) {
        // rows behind the last key or in front of the window may hold anything, and zero weights do not silence a NaN: clear their values
        ok = ok && mbar_wait(&sh->full[st], (uint32_t)((ji >> 1) & 1), abort_flag);
        const int lo = max(0, kv_begin - key0), hi = min(DT_KEYS, kv_end - key0);
        if (ok)
          for (int i = tid; i < (lo + DT_KEYS - hi) * 64; i += 128) {
            const int r = (i >> 6) < lo ? i >> 6 : hi + (i >> 6) - lo;
            *reinterpret_cast<uint4*>(tiles + st * STAGE + (r >> 3) * BOX + ((i >> 3) & 7) * 1024 + (r & 7) * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->cleared);
      }
      float v[HB][4];  // columns col, col + 1 of key_a, then of key_a + 8
      bool grew = false;
      ok = ok && mbar_wait(&sh->s_full[st], (uint32_t)((ji >> 1) & 1), abort_flag);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (ok) {
        tc_fence_after();
        dt_ld_frag<HN>(row + (uint32_t)(st * HN), reinterpret_cast<uint32_t*>(&v[0][0]));
        tmem_ld_wait();
        const int ka = key0 + key_a, kb = ka + 8;
        const bool live_a = ka < kv_end && ka >= kv_begin, live_b = kb < kv_end && kb >= kv_begin;
        float over = -INFINITY;
#pragma unroll
        for (int i = 0; i < HB; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            v[i][e] = (e < 2 ? live_a : live_b) ? v[i][e] * p.scale_log2 : -INFINITY;
            over = fmaxf(over, v[i][e] - ref[i][e & 1]);
          }
        grew = __any_sync(0xFFFFFFFFu, over > RESCALE_LOG2);
      }
      if (lane == 0) sh->grew[st][wq] = grew;
      dt_barrier();
      // the previous product is complete: O may be rescaled, P written again
      if (j > 0) {
        ok = ok && mbar_wait(&sh->o_full, (uint32_t)((ji - 1) & 1), abort_flag);
        ok = __all_sync(0xFFFFFFFFu, ok);
        tc_fence_after();
      }
      const int4 any = *reinterpret_cast<const int4*>(sh->grew[st]);
      if (any.x | any.y | any.z | any.w) {
#pragma unroll
        for (int i = 0; i < HB; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float mx = ok ? fmaxf(v[i][e], v[i][e + 2]) : -INFINITY;
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
            if (lane < 4) sh->part[wq][8 * i + col + e] = mx;
          }
        dt_barrier();
        if (tid < HN) {
          const float old = sh->ref[tid], mx = fmaxf(fmaxf(sh->part[0][tid], sh->part[1][tid]), fmaxf(sh->part[2][tid], sh->part[3][tid]));
          const bool move = mx > old + RESCALE_LOG2;
          sh->fac[tid] = move ? exp2f(old - mx) : 1.f;  // 0 for the first keys
          if (move) sh->ref[tid] = mx;
        }
        dt_barrier();
#pragma unroll
        for (int i = 0; i < HB; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            l[i][e] *= sh->fac[8 * i + col + e];
            ref[i][e] = sh->ref[8 * i + col + e];
          }
        if (j > 0 && ok) {
#pragma unroll 1
          for (int mb = 0; mb < 4; ++mb)
#pragma unroll 1
            for (int c = 0; c < HN; c += 16) {
              uint32_t w[16];
              tmem_ld16(row + (uint32_t)((2 + mb) * HN + c), w);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * sh->fac[c + i]);
              tmem_st16(row + (uint32_t)((2 + mb) * HN + c), w);
            }
          tmem_st_wait();
        }
      }
      if (ok) {
#pragma unroll
        for (int i = 0; i < HB; ++i) {
          const float a0 = ex2_approx(v[i][0] - ref[i][0]), a1 = ex2_approx(v[i][1] - ref[i][1]), b0 = ex2_approx(v[i][2] - ref[i][0]), b1 = ex2_approx(v[i][3] - ref[i][1]);
          l[i][0] += a0 + b0;
          l[i][1] += a1 + b1;
          uint8_t* at = p_sm + key_a * 128 + ((i ^ (key_a & 7)) << 4) + col * 2;  // (key_a + 8 has the same swizzle)
          *reinterpret_cast<bf162*>(at) = __floats2bfloat162_rn(a0, a1);
          *reinterpret_cast<bf162*>(at + 8 * 128) = __floats2bfloat162_rn(b0, b1);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->p_ready);
    }
#pragma unroll
    for (int i = 0; i < HB; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float x = l[i][e];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
        if (lane < 4) sh->part[wq][8 * i + col + e] = x;
      }
    if (n_tiles > 0) {
      ok = ok && mbar_wait(&sh->o_full, (uint32_t)((base_i + n_tiles - 1) & 1), abort_flag);
      ok = __all_sync(0xFFFFFFFFu, ok);
      tc_fence_after();
    }
    dt_barrier();
    const long long slot = 2 * (long long)blockIdx.x + (first == r.tile0 ? 1 : 0);  // of a piece of a row: the first of the block ends a row or lies inside one
    if (tid < HN && h0 + tid < p.heads) {
      const int head = h0 + tid;
      const float m = sh->ref[tid];
      float sum = (sh->part[0][tid] + sh->part[1][tid]) + (sh->part[2][tid] + sh->part[3][tid]), f = 0.f;
      if (!whole) p.part_lse[slot * HN + tid] = sum > 0.f ? m + log2f(sum) : DT_NONE;
      if (sum > 0.f) {
        if (whole && p.sink) sum += exp2f(p.sink[head] * 1.4426950408889634f - m);
        f = 1.f / sum;
        if (whole && p.gate) f /= 1.f + __expf(-__bfloat162float(p.gate[t * p.ld_gate + head]));
      }
      sh->fac[tid] = f;
    }
    dt_barrier();
    if (ok) {
      // (with an address formed per element and a test of its head, the 256 stores of a thread took 11 us)
      bf16* o_at = p.out + t * p.o_tok + h0 * p.o_head + tid;
      float* part_at = p.part_o + slot * HN * 512 + tid;
      const int live = min(HN, p.heads - h0);
#pragma unroll 1
      for (int i = 0; i < HN / 4; ++i) {  // sixteen heads of 128 value columns
        const int c = i % (HN / 16) * 16, mb = i / (HN / 16);
        uint32_t w[16];
        float x[16];
        if (n_tiles > 0) {
          tmem_ld16(row + (uint32_t)((2 + mb) * HN + c), w);
          tmem_ld_wait();
        }
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 f = *reinterpret_cast<const float4*>(&sh->fac[c + j]);
          x[j] = n_tiles > 0 ? __uint_as_float(w[j]) * f.x : 0.f;
          x[j + 1] = n_tiles > 0 ? __uint_as_float(w[j + 1]) * f.y : 0.f;
          x[j + 2] = n_tiles > 0 ? __uint_as_float(w[j + 2]) * f.z : 0.f;
          x[j + 3] = n_tiles > 0 ? __uint_as_float(w[j + 3]) * f.w : 0.f;
        }
        if (!whole) {
          float* d = part_at + c * 512 + mb * 128;
#pragma unroll
          for (int j = 0; j < 16; ++j) d[j * 512] = x[j];  // (a slot has room for all heads of a group)
        } else {
          bf16* d = o_at + c * p.o_head + mb * 128;
          if (c + 16 <= live) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              *d = __float2bfloat16(x[j]);
              d += p.o_head;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (c + j < live) d[j * p.o_head] = __float2bfloat16(x[j]);
          }
        }
      }
    }
    base_i += n_tiles;
    });
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
  if (threadIdx.x == 0 && sh->abort_flag) atomicCAS(p.status, PG_ST_OK, PG_ST_TIMEOUT | (58u << 8));
}

// A row that blocks x, x + 1, .. share, a warp to a head: their results by the sums of their weights.
__global__ void __launch_bounds__(128) mla_decode_join_kernel(const MlaDecodeTc p, int hn) {
  PG_PDL_ENTRY();
  const int2 cut = *reinterpret_cast<const int2*>(p.cuts + 2 * blockIdx.x);
  const int lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (cut.x < 0) return;
  const int groups = (p.heads + hn - 1) / hn, t = cut.x / groups, head = (cut.x - t * groups) * hn + h;
  if (head >= p.heads) return;
  auto at = [&](int i) { return (2 * (long long)(blockIdx.x + i) + (i == 0 ? 1 : 0)) * hn + h; };
  float m = DT_NONE;
  for (int i = 0; i < cut.y; ++i) m = fmaxf(m, p.part_lse[at(i)]);
  float4 acc[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  float sum = 0.f;
  for (int i = 0; i < cut.y; ++i) {
    const float lse = p.part_lse[at(i)], f = lse <= DT_NONE ? 0.f : exp2f(lse - m);
    sum += f;
    const float4* o = reinterpret_cast<const float4*>(p.part_o + at(i) * 512);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 x = o[lane + 32 * j];
      acc[j].x += f * x.x;
      acc[j].y += f * x.y;
      acc[j].z += f * x.z;
      acc[j].w += f * x.w;
    }
  }
  float f = 0.f;
  if (sum > 0.f) {
    if (p.sink) sum += exp2f(p.sink[head] * 1.4426950408889634f - m);
    f = 1.f / sum;
    if (p.gate) f /= 1.f + __expf(-__bfloat162float(p.gate[t * p.ld_gate + head]));
  }
  bf16* dst = p.out + t * p.o_tok + head * p.o_head;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    bf162* d = reinterpret_cast<bf162*>(dst + (lane + 32 * j) * 4);
    d[0] = __floats2bfloat162_rn(acc[j].x * f, acc[j].y * f);
    d[1] = __floats2bfloat162_rn(acc[j].z * f, acc[j].w * f);
  }
}

template <int HN, int QKB>
int launch(const CUtensorMap& tm, MlaDecodeTc p, int sms, void* part, long long part_bytes, cudaStream_t stream) {
  constexpr size_t smem = (size_t)2 * QKB * DT_KEYS * 128 + QKB * HN * 128 + DT_P + sizeof(DtSync<HN>) + 1024;
  static bool set = false;
  if (!set) {
    PG_CUDA(cudaFuncSetAttribute(mla_decode_tc_kernel<HN, QKB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set = true;
  }
  const long long slots = 2ll * sms * HN;
  p.shared = p.tokens <= DT_ROWS && part != nullptr && ((uintptr_t)part & 15) == 0 && part_bytes >= slots * 513 * 4 + 8ll * sms;
  p.part_o = (float*)part;
  p.part_lse = p.part_o + slots * 512;
  p.cuts = (int*)(p.part_lse + slots);
  const unsigned grid = p.shared ? (unsigned)sms : (unsigned)(p.tokens * ((p.heads + HN - 1) / HN));
  PG_CUDA(launch_pdl(mla_decode_tc_kernel<HN, QKB>, dim3(grid), dim3(DT_THREADS), smem, stream, tm, p));
  PG_LAUNCH_CHECK();
  if (p.shared) PG_CUDA(launch_pdl(mla_decode_join_kernel, dim3((unsigned)sms, HN / 4), dim3(128), (size_t)0, stream, p, HN));
  PG_LAUNCH_CHECK();
  return PG_OK;
}

}  // namespace

int mla_decode_tc(MlaDecodeTc p, int r, long long pages, void* part, long long part_bytes, cudaStream_t stream) {
  CUtensorMap tm;
  // eight keys of all blocks of 64 columns per copy
  const cuuint64_t dims[3] = {64u, (cuuint64_t)(pages * p.page_size), (cuuint64_t)((512 + r) / 64)}, strides[2] = {(cuuint64_t)(512 + r) * 2, 128u};
  const cuuint32_t box[3] = {64u, 8u, (cuuint32_t)((512 + r) / 64)};
  if (int rc = make_tmap_bf16(&tm, p.latent, 3, dims, strides, box)) return rc;
  // A block of 64 heads reads a key once for all of them; steps that leave SMs idle get blocks of fewer heads, whose start, first
  // tile and output take less (one row of 64 heads, 100 keys: 45 us for the whole operation with blocks of 64, 37 us with 16).
  static const int sms = [] {
    int dev = 0, n = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? n : 148;
  }();
  int hn = 64;
  while (hn > 16 && (p.heads <= hn / 2 || p.tokens * p.splits * ((p.heads + hn / 2 - 1) / (hn / 2)) <= sms)) hn /= 2;
  switch (hn) {
    case 16: return r ? launch<16, 9>(tm, p, sms, part, part_bytes, stream) : launch<16, 8>(tm, p, sms, part, part_bytes, stream);
    case 32: return r ? launch<32, 9>(tm, p, sms, part, part_bytes, stream) : launch<32, 8>(tm, p, sms, part, part_bytes, stream);
    default: return r ? launch<64, 9>(tm, p, sms, part, part_bytes, stream) : launch<64, 8>(tm, p, sms, part, part_bytes, stream);
  }
}
