// The members of a lookup table in one pass: every cell has a bucket of `size`
// slots, an atom takes the next slot of each cell it belongs to, and members
// past the bucket are chained to their cell, so the table is complete whatever
// the bucket's size.  A scan of the counts then places the final lists
// (scan.cuh), and the sort reads bucket and chain and writes them there.
// Enumerating the members twice, to count and to fill, had cost more than the
// bucket's scattered slots do: table stage of 50,000 GBSW atoms 240 -> 220 us,
// of 1,000 40 -> 37, of 6,007 on a grid table 78 -> 60.  (Slots of a number
// side by side, for neighbouring cells' sake, measured the same or worse;
// starts taken inside the sort, by groups of 32 cells, saved the scan's 4 us
// and cost 40 in the sort and 20 in the integrals of 50,000 atoms.)
// The host sizes the buckets from the longest list of the sizing call, with a
// quarter to spare.
// Included by the table translation units; internal linkage in each.
#pragma once

#include "gbx_internal.cuh"

namespace gbx {
namespace {

constexpr int kPutBatch = 4;  // candidates per lane with their slots in flight

// Candidate t of a box of n1 x n2 cells per first index, last index fastest
// (neighbouring lanes on neighbouring cells, whose counters share sectors), by
// FP32 division and a correction either way (at most 2^24 candidates in 2^16
// rows, so the quotient is off by one at most).
struct BoxIndex {
  int n1, n2;
  float inv1, inv2;
  __device__ __forceinline__ BoxIndex(int n1, int n2) : n1(n1), n2(n2), inv1(1.0f / (float)n1), inv2(1.0f / (float)n2) {}
  static __device__ __forceinline__ int div(int t, int n, float inv) {
    int q = (int)(((float)t + 0.5f) * inv);
    q -= q * n > t;
    return q + ((q + 1) * n <= t);
  }
  __device__ __forceinline__ int3 operator()(int t) const {
    const int row = div(t, n2, inv2), i = div(row, n1, inv1);
    return make_int3(i, row - i * n1, t - row * n2);
  }
};

struct Members {
  int* count;   // [cells] members per cell (0 on entry)
  int* slots;   // [cells][size]
  int* chain;   // [cells] 1 + the cell's last chained member (0 on entry)
  int2* node;   // [node_cap] (atom, chain before it)
  int size;
  long long node_cap;
  unsigned* chained;  // members in nodes (0 on entry)
  unsigned* status;
  __device__ __forceinline__ void put(long long cell, int atom) const {
    place(cell, atomicAdd(&count[cell], 1), atom);
  }
  // U cells at once (-1: none): the slots are all on their way before the first
  // is needed, where a warp would wait out an L2 round trip for each (table
  // stage of 50,000 GBSW atoms 218 -> 204 us, of 1,000 36 -> 33.5; 2 or 8 in
  // flight instead of 4: the same at 50,000, slower at 1,000 and 6,007).
  template <int U>
  __device__ __forceinline__ void put(const long long (&cell)[U], int atom) const {
    int slot[U];
#pragma unroll
    for (int u = 0; u < U; ++u) slot[u] = cell[u] >= 0 ? atomicAdd(&count[cell[u]], 1) : 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (cell[u] >= 0) place(cell[u], slot[u], atom);
  }
  __device__ __forceinline__ void place(long long cell, int slot, int atom) const {
    if (slot < size) {
      slots[cell * size + slot] = atom;
      return;
    }
    const unsigned o = atomicAdd(chained, 1u);
    if (o < node_cap) node[o] = make_int2(atom, atomicExch(&chain[cell], (int)o + 1));
    else atomicOr(status, kStatusTableEntries);
  }
  // The members of a cell whose list is longer than its bucket, into out[0 .. cnt):
  // `width` lanes, lane 0 .. width - 1.  (Atom 0 stands for members that found no
  // node; the status then says so.)
  __device__ __forceinline__ void gather(long long cell, int cnt, int* out, int lane, int width) const {
    for (int q = lane; q < size; q += width) out[q] = slots[cell * size + q];
    if (lane != 0) return;
    int k = size;
    for (int o = chain[cell]; o > 0 && k < cnt;) {
      const int2 v = node[o - 1];
      out[k++] = v.x;
      o = v.y;
    }
    while (k < cnt) out[k++] = 0;
  }
};

}  // namespace
}  // namespace gbx
