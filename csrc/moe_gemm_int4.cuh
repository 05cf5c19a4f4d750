// Grouped GEMM over INT4 expert weights: the dequantised operand goes to the tensor core through tensor memory.
// Part of moe_gemm.cu (inside its anonymous namespace): same parameters, items and epilogue as moe_gemm_kernel.
//
// A thread owns one weight row = one TMEM lane: it reads 32 bytes of its packed row from a 128-byte-swizzled tile without bank
// conflicts, expands them to 64 bf16 in registers and writes these as 32 TMEM columns, from where the MMA reads its A operand.
// Against an A tile in shared memory that saves the 16 KB store and the tensor core's 16 KB load of every k-block, the proxy
// fence, and with one arrival per warp the 64 arrivals on one barrier.  Scales come by TMA beside the weights (read from
// global memory by each thread they were 128 sectors a k-block): 256-deep stages make a row of eight of them the 16 bytes that
// a TMA row needs.
//
// 48 experts of 7168 x 2048, top 8 (routing and both products): 128 tokens 684 us with the A tile in shared memory, 445 now, of
// which 70 by the issue of products from uniform registers (gemm_sm100.cu).  The weights' bytes take 182 us; a product of 128 rows
// and few columns occupies the tensor core for 45 cycles whatever its columns, 165 us of this.
//
// warp 0 TMA producer | warp 1 MMA issuer + TMEM owner | warps 2-5 epilogue | then Q4_GROUPS groups of four dequant warps.
// Group g expands the k-blocks g, g + Q4_GROUPS, .. of the four of a stage into TMEM buffers of two or three stages.
constexpr int Q4_GROUPS = 4;             // divides 4; two groups: 534 us where four take 474 (128 tokens), 688 and 703 (512)
constexpr int Q4_BK = 256;               // weights of a row in one stage: 128 bytes
constexpr int Q4_RAW = BM * Q4_BK / 2;   // packed tile
constexpr int Q4_SC = BM * (Q4_BK / 32) * 2;
constexpr int Q4_STAGES = 8;             // at most
constexpr int Q4_TURNS = 3;              // at most: stages whose A is in tensor memory, four buffers of 32 columns each, behind two accumulators (two: 452 us, three: 445)
constexpr int Q4_BUFS = 4 * Q4_TURNS;
constexpr int Q4_MAX_BN = 128;
constexpr int Q4_THREADS = 192 + Q4_GROUPS * 128;

__global__ void __launch_bounds__(Q4_THREADS, 1)
moe_gemm_int4_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_x, const MoeGemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_tiles[MAX_EXPERTS];
  __shared__ int s_total;
  const uint32_t base = smem_u32(smem_raw);
  uint8_t* tiles = smem_raw + (((base + 1023u) & ~1023u) - base);
  const int x_bytes = p.bn * 128;  // one k-block of the token rows
  const int stage_bytes = Q4_RAW + Q4_SC + 4 * x_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(tiles + p.stages * stage_bytes);
  uint64_t* empty = full + Q4_STAGES;
  uint64_t* aready = empty + Q4_STAGES;
  uint64_t* afree = aready + Q4_BUFS;
  uint64_t* tfull = afree + Q4_BUFS;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < Q4_BUFS; ++b) {
      mbar_init(&aready[b], 4);  // the warps of one group
      mbar_init(&afree[b], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
    if (p.scale_tma) tma_prefetch_desc(&tm_s);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  pdl_wait();
  count_items(p, s_tiles, &s_total);
  pdl_launch_dependents();  // (behind the allocation above: a dependent that takes tensor memory must not be first)
  const uint32_t tmem_base = *tmem_slot;
  const int total = s_total;
  const int turns = min(Q4_TURNS, (512 - 2 * p.bn) / 128);
  const uint32_t a_col = 512u - 128u * (uint32_t)turns;
  const int depth = (p.K + Q4_BK - 1) / Q4_BK;  // stages of an item; TMA fills what lies past K with zeros on every operand
  uint32_t ep_epoch = 0;
  if (p.scatter_src != nullptr) ep_epoch = *((volatile uint32_t*)(p.peer_flags[p.rank] + p.site * 32 + 16));

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t pol_w = l2_policy_evict_first();
      const uint64_t pol_x = l2_policy_evict_last();
      int stage = 0;
      uint32_t phase = 0, used = 0, last = 0;  // a bit per stage: loaded, parity of its last load
      ItemCursor cur;
      Item it;
      bool ok = true;
      for (int item = blockIdx.x; item < total && ok; item += gridDim.x) {
        if (!locate(p, s_tiles, item, cur, it)) break;
        for (int d = 0; d < depth; ++d) {
          if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* st = tiles + stage * stage_bytes;
          mbar_expect_tx(&full[stage], (uint32_t)(stage_bytes - (p.scale_tma ? 0 : Q4_SC)));
          tma_load_3d(st, &tm_w, &full[stage], d * (Q4_BK / 8), it.m_tile * BM, it.e, pol_w);
          if (p.scale_tma) tma_load_3d(st + Q4_RAW, &tm_s, &full[stage], d * (Q4_BK / 32), it.m_tile * BM, it.e, pol_w);
#pragma unroll
          for (int i = 0; i < 4; ++i) tma_load_2d(st + Q4_RAW + Q4_SC + i * x_bytes, &tm_x, &full[stage], d * Q4_BK + i * BK, it.row0, pol_x);
          used |= 1u << stage;
          last = (last & ~(1u << stage)) | (phase << stage);
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      for (int s = 0; s < p.stages; ++s) {
        if (!((used >> s) & 1u)) continue;
        uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&full[s], (last >> s) & 1u)) {
          if (globaltimer_ns() - t0 > PG_WAIT_LIMIT_NS) break;
        }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    {
      const uint32_t idesc = umma_idesc_bf16_f32(BM, (uint32_t)p.bn);
      const uint64_t x_desc0 = umma_desc_k_sw128(smem_u32(tiles) + Q4_RAW + Q4_SC);
      int stage = 0;
      uint32_t phase = 0, a_phase = 0;
      int turn = 0, acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < total && ok; item += gridDim.x) {
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1u, abort_flag)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * p.bn);
        for (int d = 0; d < depth && ok; ++d) {
          if (!mbar_wait(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          const uint64_t x_desc = x_desc0 + (uint32_t)(stage * (stage_bytes >> 4));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int b = turn * 4 + i;
            if (!mbar_wait(&aready[b], a_phase, abort_flag)) {
              ok = false;
              break;
            }
            tc_fence_after();
            if (leader) {
#pragma unroll
              for (int k = 0; k < BK / 16; ++k)
                umma_bf16_ts(d_tmem, tmem_base + a_col + (uint32_t)(b * 32 + k * 8), x_desc + (uint32_t)(i * (x_bytes >> 4) + k * 2), idesc, (d | i | k) ? 1u : 0u);
              umma_commit(&afree[b]);
              if (i == 3) umma_commit(&empty[stage]);
            }
          }
          if (!ok) break;
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
          if (++turn == turns) {
            turn = 0;
            a_phase ^= 1u;
          }
        }
        if (!ok) break;
        if (leader) umma_commit(&tfull[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else if (warp < 6) {
    const int wq = warp & 3;
    const int r = wq * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    ItemCursor cur;
    Item it;
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
      if (!locate(p, s_tiles, item, cur, it)) break;
      bool ok = mbar_wait(&tfull[acc], acc_phase, abort_flag);
      ok = named_bar_all(1, 128, ok);
      if (!ok) break;
      tc_fence_after();
      store_tile(p, it, it.m_tile * BM + r, lane, tmem_base + ((uint32_t)(wq * 32) << 16) + (uint32_t)(acc * p.bn));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    const int wq = warp & 3;  // TMEM lanes of this warp: 32 wq ..
    const int grp = (warp - 6) >> 2;
    const int r = wq * 32 + lane;
    const uint32_t a_row = tmem_base + ((uint32_t)(wq * 32) << 16) + a_col;
    const int groups_per_row = p.K / 32;
    const bf162 bias = __floats2bfloat162_rn(136.f, 136.f);
    uint32_t mask, magic;  // in registers: as two constants of one operation they make it two (474 us where this takes 451)
    asm volatile("mov.b32 %0, 0x000F000F;\n\tmov.b32 %1, 0x43004300;" : "=r"(mask), "=r"(magic));
    int stage = 0, turn = 0;
    uint32_t phase = 0, a_phase = 0;
    ItemCursor cur;
    Item it;
    bool ok = true;
    for (int item = blockIdx.x; item < total && ok; item += gridDim.x) {
      if (!locate(p, s_tiles, item, cur, it)) break;
      const int m = it.m_tile * BM + r;
      const bf16* srow = reinterpret_cast<const bf16*>(p.scales) + ((size_t)it.e * p.M + (m < p.M ? m : 0)) * groups_per_row;
      for (int d = 0; d < depth; ++d) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag));
        if (!ok) break;
        const uint8_t* st = tiles + stage * stage_bytes;
        for (int i = grp; i < 4; i += Q4_GROUPS) {
          const int b = turn * 4 + i;
          uint32_t words[8];
          *reinterpret_cast<uint4*>(words) = *reinterpret_cast<const uint4*>(st + r * 128 + (((2 * i) ^ (r & 7)) << 4));
          *reinterpret_cast<uint4*>(words + 4) = *reinterpret_cast<const uint4*>(st + r * 128 + (((2 * i + 1) ^ (r & 7)) << 4));
          bf162 sc = __floats2bfloat162_rn(0.f, 0.f);
          if (p.scale_tma) {
            sc = *reinterpret_cast<const bf162*>(st + Q4_RAW + r * 16 + i * 4);
          } else if (m < p.M) {
            const int g = d * (Q4_BK / 32) + i * 2;
            if (g < groups_per_row) sc.x = srow[g];
            if (g + 1 < groups_per_row) sc.y = srow[g + 1];
          }
          ok = __all_sync(0xffffffffu, mbar_wait(&afree[b], a_phase ^ 1u, abort_flag));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const bf162 s2 = h ? __halves2bfloat162(sc.y, sc.y) : __halves2bfloat162(sc.x, sc.x);
            uint32_t o[16];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              // pair-interleaved nibbles: (w >> 4j) & 0x000F000F | 0x43004300 = bf16 pair (128 + e[2j], 128 + e[2j+1])
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint32_t tt;
                asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(tt) : "r"(words[h * 4 + c] >> (4 * j)), "r"(mask), "r"(magic));  // (a & b) | c
                bf162 val = *reinterpret_cast<bf162*>(&tt);
                val = __hmul2(__hsub2(val, bias), s2);
                o[c * 4 + j] = *reinterpret_cast<uint32_t*>(&val);
              }
            }
            tmem_st16(a_row + (uint32_t)(b * 32 + h * 16), o);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&aready[b]);
        }
        if (!ok) break;
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
        if (++turn == turns) {
          turn = 0;
          a_phase ^= 1u;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(p.status, PG_ST_OK, PG_ST_TIMEOUT | (5u << 8));
  raise_returned(p, ep_epoch);
}
