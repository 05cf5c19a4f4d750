// Stable counting sort of expert routes inside one CTA (shared by the local MoE path and
// the expert-parallel receive path).
//
// Routes arrive as a flat list of local expert ids (anything outside [0, e_local) means "not for this rank").  Every warp
// owns one contiguous slice of the list and walks it 32 entries at a time: lanes with the same expert find each other by a
// ballot per bit of the id (a warp match takes several times as long), the first of them moves the warp's counter of it.  In
// front of that walk another one counts (atomics on the warp's counters, which need no order), a scan over (expert, warp)
// turns the counts into cursors, and the walk hands out positions, so the order inside an expert is the route order (stable:
// the f32 summation order downstream never depends on scheduling).  Bound by the latency of the walk, n / 512 steps; with
// every warp scanning the whole list for its own experts instead, 10266 routes to 64 experts took 140 us and 1024 routes
// 14 us; 18.8 and 4.9 us with two ordered walks, 12.5 and 3.5 now.  Up to 256 routes to at most 16 experts, a warp per
// expert does scan the list, which it holds in registers (8 experts, 48 routes: 2.0 us, with slices 3.3).
//
// Takes the place of the reference's per-layer host-side routing bookkeeping and of the
// align step of its Marlin MoE path (pegainfer-kernels/csrc/kimi_k2/kimi_marlin_wna16.cu
// callers; pegainfer-deepseek-v2-lite/src/runtime/moe.rs).
#pragma once
#include "common.cuh"

constexpr int ROUTE_SORT_THREADS = 512;
constexpr int ROUTE_SORT_WARPS = ROUTE_SORT_THREADS / 32;
constexpr int ROUTE_SORT_EXPERTS = 512;

struct RouteSortSmem {
  int cursor[ROUTE_SORT_WARPS][ROUTE_SORT_EXPERTS];
  int warp_total[ROUTE_SORT_WARPS];
};

// The sort by slices.  AHEAD: groups of 32 entries whose ids are loaded, and ranked, together; 1 for lists that may leave warps without
// a slice (up to ROUTE_SORT_THREADS entries).
template <int AHEAD, typename Load, typename Emit>
__device__ __forceinline__ void route_sort_sliced(RouteSortSmem& sm, int n, int e_local, int* __restrict__ offsets, Load load, Emit emit) {
  static_assert(ROUTE_SORT_THREADS == ROUTE_SORT_EXPERTS, "the scan gives every expert a thread");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = ((n + ROUTE_SORT_WARPS - 1) / ROUTE_SORT_WARPS + 31) & ~31;
  const int i_begin = min(n, warp * slice), i_end = min(n, i_begin + slice);
  const int used = AHEAD == 1 ? (n + 31) / 32 : ROUTE_SORT_WARPS;  // warps that are looked at
  int* cursor = sm.cursor[warp];
  const int bits = 32 - __clz(e_local - 1);  // of a local expert id (none for a single expert)
  // counts need no order
  auto count = [&]() {
    for (int base = i_begin; base < i_end; base += 32 * AHEAD) {
      int id[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = base + 32 * a + lane;
        id[a] = i < i_end ? load(i) : -1;
      }
#pragma unroll
      for (int a = 0; a < AHEAD; ++a)
        if (id[a] >= 0 && id[a] < e_local) atomicAdd(&cursor[id[a]], 1);
    }
  };
  auto place = [&]() {
    for (int base = i_begin; base < i_end; base += 32 * AHEAD) {
      int id[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = base + 32 * a + lane;
        id[a] = i < i_end ? load(i) : -1;
      }
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = base + 32 * a + lane;
        const bool mine = id[a] >= 0 && id[a] < e_local;
        uint32_t peers = __ballot_sync(0xffffffffu, mine);  // for a lane with a local expert: the lanes that have the same one
#pragma unroll 1
        for (int bit = 0; bit < bits; ++bit) {
          const bool one = id[a] >> bit & 1;
          const uint32_t ones = __ballot_sync(0xffffffffu, one);
          peers &= one ? ones : ~ones;
        }
        const int before = mine ? cursor[id[a]] : 0;
        __syncwarp();
        if (mine && lane == __ffs(peers) - 1) cursor[id[a]] = before + __popc(peers);
        __syncwarp();
        if (i < i_end) emit(i, mine ? before + __popc(peers & ((1u << lane) - 1u)) : -1);
      }
    }
  };
#pragma unroll
  for (int w = 0; w < ROUTE_SORT_WARPS; ++w)
    if (w < used) sm.cursor[w][tid] = 0;
  __syncthreads();
  count();
  __syncthreads();
  int total = 0;  // of expert `tid`
#pragma unroll
  for (int w = 0; w < ROUTE_SORT_WARPS; ++w)
    if (w < used) total += sm.cursor[w][tid];
  int upto = total;  // inclusive scan over the experts
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += x;
  }
  if (lane == 31) sm.warp_total[warp] = upto;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < ROUTE_SORT_WARPS; ++w)
    if (w < warp) upto += sm.warp_total[w];
  int at = upto - total;
  if (tid < e_local) offsets[tid] = at;
  if (tid == e_local - 1) offsets[e_local] = upto;
#pragma unroll
  for (int w = 0; w < ROUTE_SORT_WARPS; ++w)
    if (w < used) {
      const int c = sm.cursor[w][tid];
      sm.cursor[w][tid] = at;
      at += c;
    }
  __syncthreads();
  place();
}

// `load(i)` returns the local expert id of flat entry i (0 <= i < n); `emit(i, pos)` is called
// once per entry with its position in the sorted order, or pos = -1 when the entry is not
// for a local expert.  Writes offsets[0..e_local].  All ROUTE_SORT_THREADS threads call this.
template <typename Load, typename Emit>
__device__ __forceinline__ void route_sort(RouteSortSmem& sm, int n, int e_local, int* __restrict__ offsets, Load load, Emit emit) {
  constexpr int FEW = 8;  // groups of 32 entries that a warp holds
  if (n > ROUTE_SORT_THREADS) {
    route_sort_sliced<4>(sm, n, e_local, offsets, load, emit);
    return;
  }
  if (e_local > ROUTE_SORT_WARPS || n > 32 * FEW) {
    route_sort_sliced<1>(sm, n, e_local, offsets, load, emit);
    return;
  }
  // few routes and experts: a warp per expert, which reads the whole list
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int id[FEW], count = 0;
  uint32_t mine[FEW];
#pragma unroll
  for (int a = 0; a < FEW; ++a) id[a] = 32 * a + lane < n ? load(32 * a + lane) : -1;
#pragma unroll
  for (int a = 0; a < FEW; ++a) {
    mine[a] = __ballot_sync(0xffffffffu, warp < e_local && id[a] == warp);
    count += __popc(mine[a]);
  }
  if (lane == 0) sm.warp_total[warp] = count;
  __syncthreads();
  int at = 0;
#pragma unroll
  for (int w = 0; w < ROUTE_SORT_WARPS; ++w)
    if (w < warp) at += sm.warp_total[w];
  if (lane == 0 && warp < e_local) offsets[warp] = at;
  if (lane == 0 && warp == e_local - 1) offsets[e_local] = at + count;
#pragma unroll
  for (int a = 0; a < FEW; ++a) {
    const int i = 32 * a + lane;
    if (mine[a] >> lane & 1u) emit(i, at + __popc(mine[a] & ((1u << lane) - 1u)));
    if (warp == a && i < n && (id[a] < 0 || id[a] >= e_local)) emit(i, -1);
    at += __popc(mine[a]);
  }
}
