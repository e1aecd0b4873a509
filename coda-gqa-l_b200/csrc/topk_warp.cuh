// The selection of topk_order.h carried out by one warp on a queue in shared memory, with the same result (every
// element ends at the same place, ties included).
//
// What a single thread spends its time on is the partition scans: a shared-memory round trip per element, some
// 40 us for 256 gates.  The outcome of a partition pass does not depend on the order in which it is computed.  Call an
// index a left stopper when its element does not go before the pivot, and a right stopper when the pivot does not
// go before it; the serial pass swaps the k-th left stopper (ascending) with the k-th right stopper (descending) while
// the former lies below the latter.  A warp finds both lists with ballots and prefix counts, 32 elements at a time, and
// swaps all pairs at once.  Median, the at most 3-element tail, heap paths and the sort of more than 16
// elements stay on one lane.
#pragma once
#include "topk_order.h"

namespace topk_order {

// Elements [first, last) around the pivot value `pv`; `ls` / `rs`: scratch of last - first entries each.  All lanes call;
// returns the cut on all lanes.
template <typename It, typename Cmp>
__device__ __forceinline__ int partition_warp(It* q, int first, int last, const It pv, Cmp before, uint16_t* ls, uint16_t* rs) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, n = last - first;
  int nl = 0, nr = 0;
  for (int o = 0; o < n; o += 32) {
    const int i = o + lane, j = n - 1 - i;
    const bool in = i < n;
    const bool sl = in && !before(q[first + i], pv), sr = in && !before(pv, q[first + j]);
    const unsigned bl = __ballot_sync(FULL, sl), br = __ballot_sync(FULL, sr), below = (1u << lane) - 1u;
    if (sl) ls[nl + __popc(bl & below)] = (uint16_t)i;
    if (sr) rs[nr + __popc(br & below)] = (uint16_t)j;
    nl += __popc(bl); nr += __popc(br);
  }
  __syncwarp();
  int swaps = 0;                                   // pairs with left below right form a prefix
  const int np = nl < nr ? nl : nr;
  for (int o = 0; o < np; o += 32) {
    const int k = o + lane;
    bool doit = false;
    int a = 0, b = 0;
    if (k < np) { a = ls[k]; b = rs[k]; doit = a < b; }
    if (doit) swap_items(q, first + a, first + b);
    const unsigned m = __ballot_sync(FULL, doit);
    swaps += __popc(m);
    if (m != FULL) break;
  }
  int cut = swaps < nl ? (int)ls[swaps] : n;       // the next left stopper, or where the last swap left one
  if (swaps > 0 && (int)rs[swaps - 1] < cut) cut = rs[swaps - 1];
  __syncwarp();
  return first + cut;
}

// sort_range of at most 16 elements [0, n): there it is a plain insertion sort, which is stable, so the place of an
// element is the number of elements that go before it or tie with it from the left.  All lanes call.
template <typename It, typename Cmp>
__device__ __forceinline__ void sort_small_warp(It* q, int n, Cmp before) {
  const int lane = threadIdx.x & 31;
  It mine = q[0];
  int place = 0;
  if (lane < n) {
    mine = q[lane];
    for (int j = 0; j < n; ++j) {
      const It o = q[j];
      place += before(o, mine) || (j < lane && !before(mine, o)) ? 1 : 0;
    }
  }
  __syncwarp();
  if (lane < n) q[place] = mine;
  __syncwarp();
}

// topk_queue by one warp; `scratch`: 2 * n uint16.  n < 65536.
template <typename V, bool LARGEST>
__device__ __forceinline__ void topk_queue_warp(Item<V>* q, int n, int k, bool sorted, uint16_t* scratch) {
  if (k <= 0 || n <= 0) return;
  Before<V, LARGEST> before;
  const int lane = threadIdx.x & 31;
  if ((int64_t)k * 64 <= (int64_t)n) {             // heap path: one lane
    if (lane == 0) topk_queue<V, LARGEST>(q, n, k, sorted);
    __syncwarp();
    return;
  }
  int first = 0, last = n;
  const int nth = k - 1;
  if (nth != last) {
    int depth = floor_log2(last - first) * 2;
    bool heap = false;
    while (last - first > 3) {
      if (depth == 0) { heap = true; break; }
      --depth;
      if (lane == 0) median_to_first(q, first, first + 1, first + (last - first) / 2, last - 1, before);
      __syncwarp();
      const Item<V> pv = q[first];
      const int cut = partition_warp(q, first + 1, last, pv, before, scratch, scratch + n);
      if (cut <= nth) first = cut; else last = cut;
    }
    if (lane == 0) {
      if (heap) { heap_select(q, first, nth + 1, last, before); swap_items(q, first, nth); }
      else insertion_sort(q, first, last, before);
      if (sorted && k - 1 > 16) sort_range(q, 0, k - 1, before);
    }
  }
  __syncwarp();
  if (sorted && k - 1 <= 16) sort_small_warp(q, k - 1, before);
}

}  // namespace topk_order
