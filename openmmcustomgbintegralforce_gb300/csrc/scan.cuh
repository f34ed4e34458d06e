// Per-cell counts to list starts in one pass: each block sums its tile and
// takes a contiguous range with one atomic on the running total, so the tiles'
// order in memory is not fixed -- nothing reads it: a cell's list is found by
// its start alone, and its contents do not depend on where it lies.  (A
// three-pass prefix sum took 20 us of a 1,000-atom step, this 4.)
// EVEN rounds each cell's allocation up to an even entry count, so every
// list starts at an even entry (a 32-byte boundary for 16-byte entries) and
// a list's entries can be read in aligned pairs without leaving the table.
// Included by the table translation units; internal linkage in each.
#pragma once

#include "gbx_internal.cuh"

namespace gbx {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;  // two 16-byte loads per thread
constexpr int kScanTile = kScanThreads * kScanItems;

template <bool EVEN>
__device__ __forceinline__ int scan_alloc(int count) {
  return EVEN ? (count + 1) & ~1 : count;
}

// start[c] for the cells of `geom` (none if it has more than cell_cap);
// *total (zero on entry) receives the sum.  Cells past the entry capacity
// raise the status and start at the largest index.  *longest (if wanted)
// receives the largest count above `bucket`.
template <bool EVEN>
__global__ void __launch_bounds__(kScanThreads) scan_kernel(const int* __restrict__ count,
                                                            const TableGeom* gp, int* __restrict__ start,
                                                            long long cell_cap, long long entry_cap,
                                                            unsigned long long* total, int* longest, int bucket,
                                                            unsigned* __restrict__ status) {
  __shared__ int s_warp[kScanThreads / kWarp];
  __shared__ long long s_base;
  const long long ncell = gp->ncell <= cell_cap ? gp->ncell : 0;
  const long long tile = (long long)blockIdx.x * kScanTile;
  if (tile >= ncell) return;
  const int lane = threadIdx.x % kWarp, w = threadIdx.x / kWarp;
  const long long base = tile + (long long)threadIdx.x * kScanItems;
  int v[kScanItems];
  if (base + kScanItems <= ncell) {
    const int4 a = *reinterpret_cast<const int4*>(count + base), b = *reinterpret_cast<const int4*>(count + base + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
    for (int k = 0; k < kScanItems; ++k) v[k] = base + k < ncell ? count[base + k] : 0;
  }
  int sum = 0, most = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    most = max(most, v[k]);
    const int c = scan_alloc<EVEN>(v[k]);
    v[k] = sum;  // exclusive within the thread
    sum += c;
  }
  int incl = sum;
  for (int off = 1; off < kWarp; off <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += u;
  }
  if (lane == kWarp - 1) s_warp[w] = incl;
  if (longest) {
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most > bucket) atomicMax(longest, most);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int k = 0; k < kScanThreads / kWarp; ++k) {
      const int u = s_warp[k];
      s_warp[k] = acc;
      acc += u;
    }
    const long long b = acc > 0 ? (long long)atomicAdd(total, (unsigned long long)acc) : 0;
    if (b + acc > entry_cap) atomicOr(status, kStatusTableEntries);
    s_base = b;
  }
  __syncthreads();
  const long long first = s_base + s_warp[w] + (incl - sum);
  int o[kScanItems];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) o[k] = (int)min(first + v[k], 0x7fffffffLL);
  if (base + kScanItems <= ncell) {
    *reinterpret_cast<int4*>(start + base) = make_int4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<int4*>(start + base + 4) = make_int4(o[4], o[5], o[6], o[7]);
  } else {
    for (int k = 0; k < kScanItems && base + k < ncell; ++k) start[base + k] = o[k];
  }
}

template <bool EVEN = false>
inline void launch_scan(const int* count, const TableGeom* geom, int* start, long long cell_cap, long long entry_cap,
                        unsigned long long* total, int* longest, int bucket, unsigned* status, cudaStream_t st) {
  const long long nb = (cell_cap + kScanTile - 1) / kScanTile;
  scan_kernel<EVEN><<<(int)(nb < 1 ? 1 : nb), kScanThreads, 0, st>>>(count, geom, start, cell_cap, entry_cap, total,
                                                                     longest, bucket, status);
}

}  // namespace
}  // namespace gbx
