// Lookup-table build: bins atoms into per-cell lists that are bit-identical
// to the reference's tables.
//
//   geometry  the grid exactly as the reference derives it (FP64), by the
//             call's first kernel (k_prepare.cu);
//   members   one warp per atom enumerates its candidate cells (or samples)
//             and puts it in the bucket of each it belongs to (buckets.cuh);
//   scan      counts -> list starts;
//   sort      one warp per cell sorts its members, restoring the reference's
//             ascending-atom insertion order, applies the per-cell cap and
//             writes the atoms' positions and parameters inline.
//
// Every FP64 operation that decides membership is written with explicit
// round-to-nearest intrinsics so that no multiply-add is contracted: the
// decisions match the reference's separately rounded C++ arithmetic.
#include <math.h>

#include "bitonic.cuh"
#include "buckets.cuh"
#include "gbx_internal.cuh"
#include "scan.cuh"

namespace gbx {
namespace {

constexpr int kMaxSamples = 96;  // grid values or samples per axis kept in shared memory
constexpr int kMemberThreads = 256;
constexpr int kMemberWarps = kMemberThreads / kWarp;

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// sqrt(3.0)/2.0 as the reference computes it in double.
__device__ __forceinline__ double half_sqrt3() { return ddiv(__dsqrt_rn(3.0), 2.0); }

// --------------------------------------------------------------------------
// Membership enumeration
// --------------------------------------------------------------------------

// CharmmReferenceGBSW.cpp:472-496 (STANDALONE) and CustomGBIntegral.cpp:198-227 (GRID).
// A warp per atom over the grid points of its box, neighbouring lanes on
// neighbouring points (whose counters share sectors).  The offset from the atom
// depends on one axis only, so each axis value's is formed once, in the
// reference's FP64; the membership of a point is decided by the FP32 sum of
// their squares wherever that is clear of the boundary by a margin that covers
// its rounding, and by the reference's FP64 operations otherwise (FP64 for
// every point took 98 us of a pass over 6,007 atoms).  FP64 instructions cost
// the same for three lanes as for 32 and were what bound the pass, so what an
// axis needs of them is done for a block's eight atoms together (24 threads;
// three lanes of each atom's own warp: 78 -> 70 us of that table, and 37 + 49
// -> 28 + 41 us of two passes over 10,000 atoms of the periodic form).
// Five blocks per SM (48 registers): 6 spill; the compiler's own 56 registers
// leave four (table stage of 10,000 GBMV-II atoms with 4, 5, 6: 117, 112, 129 us).
template <int MODE>
__global__ void __launch_bounds__(kMemberThreads, 5) table_members_grid_kernel(const float4* __restrict__ pos, const double* __restrict__ radius, int n,
                                          const TableGeom* __restrict__ gp, double h, double buffer, Members mem,
                                          long long cell_cap) {
  __shared__ double s_d[kMemberWarps][3][kMaxSamples];
  __shared__ float s_sq[kMemberWarps][3][kMaxSamples];
  __shared__ int2 s_range[kMemberWarps][3];  // first grid index and their number
  __shared__ double s_pad[kMemberWarps];
  const int wib = threadIdx.x / kWarp;
  const int lane = threadIdx.x % kWarp;
  const TableGeom& g = *gp;
  if (g.ncell > cell_cap) return;
  const long long ncell = g.ncell;
  const long long sy = g.dims[2], sx = (long long)g.dims[1] * g.dims[2];
  double (*ds)[kMaxSamples] = s_d[wib];
  float (*sq)[kMaxSamples] = s_sq[wib];
  for (int base = blockIdx.x * kMemberWarps; base < n; base += gridDim.x * kMemberWarps) {
    __syncthreads();  // the previous atoms' values are read
    if (threadIdx.x < 3 * kMemberWarps && base + threadIdx.x / 3 < n) {  // an axis of an atom per thread
      const int w = threadIdx.x / 3, k = threadIdx.x % 3;
      double pad;
      if (MODE == GBX_TABLE_STANDALONE) pad = g.pad;
      else pad = dadd(dadd(radius[base + w], dmul(half_sqrt3(), h)), buffer);
      const double c = reinterpret_cast<const float*>(pos + base + w)[k];
      const int first = (int)floor(ddiv(dsub(dsub(c, pad), g.min[k]), h));
      s_range[w][k] = make_int2(first, (int)ceil(ddiv(dsub(dadd(c, pad), g.min[k]), h)) - first + 1);
      if (k == 0) s_pad[w] = pad;
    }
    __syncthreads();
    const int a = base + wib;
    if (a >= n) continue;
    const double pad = s_pad[wib], pad2 = dmul(pad, pad);
    int b[3], nn[3];
    bool ok = true, fits = true;
    for (int k = 0; k < 3; ++k) {
      b[k] = s_range[wib][k].x;
      nn[k] = s_range[wib][k].y;
      ok = ok && nn[k] >= 1 && nn[k] <= 1024;
      fits = fits && nn[k] <= kMaxSamples;
    }
    // non-finite or absurd inputs: skip the atom instead of looping on garbage bounds
    if (!ok) {
      if (lane == 0) atomicOr(mem.status, kStatusTableCells);
      continue;
    }
    // the reference's offset of grid value m of axis k from the atom, and its test of a sum of squares
    auto offset = [&](int k, int m) {
      return dsub(dadd(g.min[k], dmul((double)(s_range[wib][k].x + m), h)),
                  (double)reinterpret_cast<const float*>(pos + a)[k]);
    };
    auto inside = [&](double d0, double d1, double d2) {
      const double s = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
      return MODE == GBX_TABLE_STANDALONE ? __dsqrt_rn(s) < pad : s < pad2;
    };
    if (!fits) {  // a grid finer than a hundredth of the pad: FP64 throughout, a column of points per lane
      for (int col = lane; col < nn[0] * nn[1]; col += kWarp) {
        const int i = col / nn[1], j = col - i * nn[1];
        const double d0 = offset(0, i), d1 = offset(1, j);
        for (int k = 0; k < nn[2]; ++k) {
          const long long cell = (long long)(b[0] + i) * sx + (long long)(b[1] + j) * sy + b[2] + k;
          if (cell >= 0 && cell < ncell && inside(d0, d1, offset(2, k))) mem.put(cell, a);
        }
      }
      continue;
    }
    for (int t = lane; t < nn[0] + nn[1] + nn[2]; t += kWarp) {
      const int k = t < nn[0] ? 0 : (t < nn[0] + nn[1] ? 1 : 2);
      const int m = t - (k == 0 ? 0 : (k == 1 ? nn[0] : nn[0] + nn[1]));
      const double d = offset(k, m);
      ds[k][m] = d;
      sq[k][m] = (float)d * (float)d;
    }
    __syncwarp();
    // FP32 squared distances carry a relative error below 5 2^-24 (three roundings of
    // a square, two of the sums), the rounded bounds 2^-24 more: 1e-6 is 16.8 2^-24
    const float in2 = (float)(pad2 * (1.0 - 1e-6)), out2 = (float)(pad2 * (1.0 + 1e-6));
    const int total = nn[0] * nn[1] * nn[2];
    const BoxIndex box(nn[1], nn[2]);
    for (int t0 = lane; t0 < total; t0 += kPutBatch * kWarp) {
      long long cell[kPutBatch];
#pragma unroll
      for (int u = 0; u < kPutBatch; ++u) {
        const int t = t0 + u * kWarp;
        cell[u] = -1;
        if (t >= total) continue;
        const int3 o = box(t);
        const float r2 = (sq[0][o.x] + sq[1][o.y]) + sq[2][o.z];
        if (!(r2 < in2 || (r2 <= out2 && inside(ds[0][o.x], ds[1][o.y], ds[2][o.z])))) continue;
        const long long c = (long long)(b[0] + o.x) * sx + (long long)(b[1] + o.y) * sy + b[2] + o.z;
        if (c < ncell) cell[u] = c;  // negative: outside, none
      }
      mem.put(cell, a);
    }
  }
}

// CustomGBIntegral.cpp:117-159 (PERIODIC): samples at the grid step, accumulated
// by repeated addition exactly as the reference's for-loops do.  The cell
// index of a sample and the membership test are decided in FP32 wherever the
// FP32 value is clear of the decision's boundary by a margin that covers its
// rounding, and in the reference's FP64 operations otherwise (FP64 runs at a
// small fraction of the FP32 rate on this part).
__global__ void __launch_bounds__(kMemberThreads, 5) table_members_periodic_kernel(const float4* __restrict__ pos, const double* __restrict__ radius,
                                              int n, const TableGeom* __restrict__ gp, double buffer, Members mem,
                                              long long cell_cap, unsigned* __restrict__ status) {
  // per warp and axis: the samples, their cell index (-1 outside) and the
  // squared offset from the atom in FP32 -- each depends on one axis only,
  // so it is computed once per axis value
  __shared__ double s_samp[kMemberWarps][3][kMaxSamples];
  __shared__ float s_sq[kMemberWarps][3][kMaxSamples];
  __shared__ int s_id[kMemberWarps][3][kMaxSamples];
  __shared__ int s_cnt[kMemberWarps][3];
  __shared__ double s_pad2[kMemberWarps];
  __shared__ float s_axis[3][3];  // 1 / box, box, 1 / step
  const int wib = threadIdx.x / kWarp;
  const int lane = threadIdx.x % kWarp;
  const TableGeom& g = *gp;
  if (g.ncell > cell_cap) return;
  const long long ncell = g.ncell;
  double (*samp)[kMaxSamples] = s_samp[wib];
  float (*sq)[kMaxSamples] = s_sq[wib];
  int (*idx)[kMaxSamples] = s_id[wib];
  constexpr float kEpsCell = 1e-4f;  // cell units: far above the FP32 rounding of a sample's position
  if (threadIdx.x < 3) {
    s_axis[0][threadIdx.x] = (float)g.inv_box[threadIdx.x];
    s_axis[1][threadIdx.x] = (float)g.box[threadIdx.x];
    s_axis[2][threadIdx.x] = (float)g.inv_step[threadIdx.x];
  }
  for (int base = blockIdx.x * kMemberWarps; base < n; base += gridDim.x * kMemberWarps) {
    __syncthreads();  // the previous atoms' samples are read
    // an axis of an atom per thread: samples by repeated addition, as the reference
    if (threadIdx.x < 3 * kMemberWarps && base + threadIdx.x / 3 < n) {
      const int w = threadIdx.x / 3, k = threadIdx.x % 3;
      const double c = reinterpret_cast<const float*>(pos + base + w)[k];
      const double L = g.L, step = g.step[k];
      const double pad = dadd(dadd(radius[base + w], dmul(half_sqrt3(), L)), buffer);
      double x = dsub(dsub(c, pad), L);
      const double end = dadd(dadd(c, pad), L);
      // samples certainly below the end, added without a compare: one fewer
      // than fit (half a step covers the additions' rounding many times over)
      const float fit = (float)(end - x) * (float)g.inv_step[k];
      const int sure = fit > 1.0f ? (fit < (float)kMaxSamples ? (int)fit - 1 : kMaxSamples) : 0;
      int m = 0;
      for (; m < sure; ++m) {
        s_samp[w][k][m] = x;
        x = dadd(x, step);
      }
      while (x < end && m <= kMaxSamples) {
        if (m < kMaxSamples) s_samp[w][k][m] = x;
        ++m;
        x = dadd(x, step);
      }
      if (m > kMaxSamples) atomicOr(status, kStatusTableEntries);
      s_cnt[w][k] = m < kMaxSamples ? m : kMaxSamples;
      if (k == 0) s_pad2[w] = dmul(pad, pad);
    }
    __syncthreads();
    const int a = base + wib;
    if (a >= n) continue;
    const float* c = reinterpret_cast<const float*>(pos + a);
    const double pad2 = s_pad2[wib];
    const int cnt[3] = {s_cnt[wib][0], s_cnt[wib][1], s_cnt[wib][2]};
    for (int t = lane; t < cnt[0] + cnt[1] + cnt[2]; t += kWarp) {
      const int k = t < cnt[0] ? 0 : (t < cnt[0] + cnt[1] ? 1 : 2);
      const int m = t - (k == 0 ? 0 : (k == 1 ? cnt[0] : cnt[0] + cnt[1]));
      const double xk = samp[k][m];
      // the sample moved into the box by whole box edges, then its cell
      const float rel = (float)(xk - g.min[k]);
      const float tb = rel * s_axis[0][k];
      const float nb = floorf(tb);
      const float u = fmaf(-nb, s_axis[1][k], rel) * s_axis[2][k];
      const float fu = floorf(u);
      int id;
      if (tb - nb > kEpsCell && tb - nb < 1.0f - kEpsCell && u - fu > kEpsCell && u - fu < 1.0f - kEpsCell) {
        id = (int)fu;
      } else {
        const double d = g.box[k];
        const double x0 = dsub(xk, dmul(d, floor(ddiv(dsub(xk, g.min[k]), d))));
        id = (int)floor(ddiv(dsub(x0, g.min[k]), g.step[k]));
      }
      idx[k][m] = (id < 0 || id >= g.dims[k]) ? -1 : id;
      const float e = (float)(xk - (double)c[k]);
      sq[k][m] = e * e;
    }
    __syncwarp();
    const long long sy = g.dims[2], sx = (long long)g.dims[1] * g.dims[2];
    // the margin of table_members_grid_kernel
    const float in2 = (float)(pad2 * (1.0 - 1e-6)), out2 = (float)(pad2 * (1.0 + 1e-6));
    const int total = cnt[0] * cnt[1] * cnt[2];
    const BoxIndex box(cnt[1], cnt[2]);
    for (int t0 = lane; t0 < total; t0 += kPutBatch * kWarp) {
      long long cell[kPutBatch];
#pragma unroll
      for (int u = 0; u < kPutBatch; ++u) {
        const int t = t0 + u * kWarp;
        cell[u] = -1;
        if (t >= total) continue;
        const int3 o = box(t);
        const float sf = (sq[0][o.x] + sq[1][o.y]) + sq[2][o.z];
        bool member = sf < in2;
        if (!member && sf <= out2) {
          // the reference's FP64 test
          const double e0 = dsub(samp[0][o.x], (double)c[0]), e1 = dsub(samp[1][o.y], (double)c[1]),
                       e2 = dsub(samp[2][o.z], (double)c[2]);
          member = dadd(dadd(dmul(e0, e0), dmul(e1, e1)), dmul(e2, e2)) < pad2;
        }
        const int i0 = idx[0][o.x], i1 = idx[1][o.y], i2 = idx[2][o.z];
        if (!member || i0 < 0 || i1 < 0 || i2 < 0) continue;
        const long long at = (long long)i0 * sx + (long long)i1 * sy + i2;
        if (at < ncell) cell[u] = at;
      }
      mem.put(cell, a);
    }
  }
}

// --------------------------------------------------------------------------
// Per-cell sort (ascending atom index) and cap, and inline copies of each
// listed atom's position and parameters, so the volume kernels stream a
// cell's list without a dependent gather.
// --------------------------------------------------------------------------
constexpr int kSortWarps = 4;

// Inline copies of GBMV lists (ascending, as the list) and GBSW lists (pairs,
// field by field, the likeliest burying atom first: a point's V does not
// depend on the order, and most listed points end at their first entry; the
// integrals of 6,007 atoms: 262 us with ascending single entries, 244 so).
struct Inline {
  const float4* pos;
  const float2* par;
  float4* entry4;
  float2* entry_par;
  int* index;        // GBSW: the atom of each inline entry
  TightCell* first;  // GBSW: each cell's first inline entry and record
  float w;           // GBSW: switching half-width
  __device__ __forceinline__ void put(long long e, int atom) const {
    entry4[e] = __ldg(pos + atom);
    entry_par[e] = __ldg(par + atom);
  }
  __device__ __forceinline__ void put_pair(long long at, const float4 a) const {
    float* p = reinterpret_cast<float*>(entry4) + 8 * (at >> 1) + (at & 1);
    p[0] = a.x;
    p[2] = a.y;
    p[4] = a.z;
    p[6] = -a.w;
  }
  __device__ __forceinline__ void put_gbsw(long long s, int r, int atom, const float4 a, long long cell) const {
    put_pair(s + r, a);
    index[s + r] = atom;
    if (r == 0) first[cell].first = a;
  }
};

// Lists of up to 32 E entries, in registers.
template <bool GBSW, int E>
__device__ __forceinline__ void sort_list(const int* src, int* entries, const Inline& in, const TableGeom& g,
                                          long long c, long long s, int cnt, int kept, int lane) {
  int key[E];
#pragma unroll
  for (int r = 0; r < E; ++r) {
    const int e = lane * E + r;
    key[r] = e < cnt ? src[e] : 0x7fffffff;
  }
  warp_bitonic_sort<E>(key, lane);
#pragma unroll
  for (int r = 0; r < E; ++r) {
    const int e = lane * E + r;
    if (e < cnt) entries[s + e] = key[r];
    if (!GBSW && e < kept) in.put(s + e, key[r]);
  }
  if constexpr (GBSW) {
    // by the distance from the cell's middle to the atom's burying sphere; the
    // low bits carry the list position, which also breaks ties
    constexpr int kMask = kWarp * E - 1;
    const int d12 = g.dims[1] * g.dims[2], ix = (int)c / d12, rem = (int)c - ix * d12, iy = rem / g.dims[2],
              iz = rem - iy * g.dims[2];
    const float mid[3] = {(float)(g.min[0] + (ix + 0.5) * g.step[0]), (float)(g.min[1] + (iy + 0.5) * g.step[1]),
                          (float)(g.min[2] + (iz + 0.5) * g.step[2])};
    int rank[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int e = lane * E + r;
      rank[r] = 0x7fffffff;
      if (e < kept) {
        const float4 a = __ldg(in.pos + key[r]);
        const float dx = a.x - mid[0], dy = a.y - mid[1], dz = a.z - mid[2];
        int b = __float_as_int(sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - (a.w - in.w));
        b ^= (b >> 31) & 0x7fffffff;  // floats in integer order
        rank[r] = (b & ~kMask) | e;
      }
    }
    warp_bitonic_sort<E>(rank, lane);
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int from = rank[r] & kMask;
      int atom = 0;
#pragma unroll
      for (int u = 0; u < E; ++u) {
        const int t = __shfl_sync(0xffffffffu, key[u], from / E);
        if (from % E == u) atom = t;
      }
      if (lane * E + r < kept) in.put_gbsw(s, lane * E + r, atom, __ldg(in.pos + atom), c);
    }
  }
}

template <bool GBSW>
__global__ void __launch_bounds__(kSortWarps * kWarp, 12) sort_cells_kernel(Members mem, const int* __restrict__ start,
                                                                        int* entries, int2* __restrict__ cell,
                                                                        Inline in, const TableGeom* __restrict__ gp,
                                                                        int cap, long long cell_cap,
                                                                        long long entry_cap) {
  const int wib = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const long long ncell = gp->ncell <= cell_cap ? gp->ncell : 0;
  if (gp->total > entry_cap) return;
  for (long long c = (long long)blockIdx.x * kSortWarps + wib; c < ncell; c += (long long)gridDim.x * kSortWarps) {
    int cnt = mem.count[c];
    const int s = start[c];
    if (cnt > kMaxSortSegment) {  // no list: no record may say there is one
      if (lane == 0) atomicOr(mem.status, kStatusSegmentTooLong);
      cnt = 0;
    }
    const int kept = cap > 0 && cnt > cap ? cap : cnt;
    const int* src = mem.slots + c * mem.size;
    if (cnt > mem.size) {
      mem.gather(c, cnt, entries + s, lane, kWarp);
      src = entries + s;
      __syncwarp();
    }
    if (lane == 0) {
      cell[c] = make_int2(kept, s);
      if (GBSW) {
        in.first[c].cs = make_int2(kept, s);
        // after an odd list: pair reads meet a sphere no point is near
        if (kept & 1) in.put_pair((long long)s + kept, make_float4(0.f, 0.f, 0.f, -1e6f));
      }
    }
    if (cnt == 0) continue;
    if (cnt <= kWarp) sort_list<GBSW, 1>(src, entries, in, *gp, c, s, cnt, kept, lane);
    else if (cnt <= 2 * kWarp) sort_list<GBSW, 2>(src, entries, in, *gp, c, s, cnt, kept, lane);
    else if (cnt <= 4 * kWarp) sort_list<GBSW, 4>(src, entries, in, *gp, c, s, cnt, kept, lane);
    else {
      // long list: ranks from global memory, results staged per lane
      int vals[kMaxSortSegment / kWarp], ranks[kMaxSortSegment / kWarp];
      int m = 0;
      for (int p = lane; p < cnt; p += kWarp, ++m) {
        const int v = src[p];
        int r = 0;
        for (int q = 0; q < cnt; ++q) {
          const int u = src[q];
          r += (u < v) || (u == v && q < p);
        }
        vals[m] = v;
        ranks[m] = r;
      }
      __syncwarp();
      for (int k = 0; k < m; ++k) {
        entries[s + ranks[k]] = vals[k];
        if (ranks[k] < kept) {
          if (GBSW) in.put_gbsw(s, ranks[k], vals[k], __ldg(in.pos + vals[k]), c);
          else in.put(s + ranks[k], vals[k]);
        }
      }
    }
    __syncwarp();
    if (lane == 0 && kept < cnt) mem.count[c] = kept;
  }
}

}  // namespace

namespace {

int grid_for(long long work, int per_block) {
  long long b = (work + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > 1048576) b = 1048576;
  return (int)b;
}

}  // namespace

gbx_status launch_table_build(Context* ctx, const float4* pos) {
  const gbx_config& c = ctx->cfg;
  cudaStream_t st = ctx->stream;
  const long long cells = ctx->cell_cap;
  if (cells == 0) return GBX_OK;  // sizing call: the grid alone; the caller reads it back and allocates
  const TableBuckets& bk = ctx->buckets;
  const Members mem{ctx->d_cell_count,     bk.slots, bk.chain, bk.node, bk.size, ctx->entry_cap,
                    &ctx->d_geom->chained, ctx->d_status};
  const int threads = kMemberThreads;
  const int blocks = grid_for((long long)ctx->n * kWarp, threads);
  switch (c.table_mode) {
    case GBX_TABLE_STANDALONE:
      table_members_grid_kernel<GBX_TABLE_STANDALONE>
          <<<blocks, threads, 0, st>>>(pos, ctx->d_radius, ctx->n, ctx->d_geom, c.grid_length, c.table_buffer, mem, cells);
      break;
    case GBX_TABLE_GRID:
      table_members_grid_kernel<GBX_TABLE_GRID>
          <<<blocks, threads, 0, st>>>(pos, ctx->d_radius, ctx->n, ctx->d_geom, c.grid_length, c.table_buffer, mem, cells);
      break;
    default:
      table_members_periodic_kernel<<<blocks, threads, 0, st>>>(pos, ctx->d_radius, ctx->n, ctx->d_geom,
                                                                c.table_buffer, mem, cells, ctx->d_status);
      break;
  }
  ++ctx->launches;
  auto* total = reinterpret_cast<unsigned long long*>(&ctx->d_geom->total);
  if (c.model == GBX_MODEL_GBSW)  // lists in aligned pairs
    launch_scan<true>(ctx->d_cell_count, ctx->d_geom, ctx->d_cell_start, cells, ctx->entry_cap, total,
                      &ctx->d_geom->longest, bk.size, ctx->d_status, st);
  else
    launch_scan<false>(ctx->d_cell_count, ctx->d_geom, ctx->d_cell_start, cells, ctx->entry_cap, total,
                       &ctx->d_geom->longest, bk.size, ctx->d_status, st);
  ++ctx->launches;
  const Inline in{pos,           ctx->d_par, ctx->d_entry4, ctx->d_entry_par, ctx->d_entry_index,
                  ctx->d_rfirst, (float)c.switch_width};
  auto sort = c.model == GBX_MODEL_GBSW ? sort_cells_kernel<true> : sort_cells_kernel<false>;
  sort<<<grid_for(cells, kSortWarps), kSortWarps * kWarp, 0, st>>>(
      mem, ctx->d_cell_start, ctx->d_entries, ctx->d_cell2, in, ctx->d_geom, c.table_cap, cells, ctx->entry_cap);
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("table build launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

}  // namespace gbx
