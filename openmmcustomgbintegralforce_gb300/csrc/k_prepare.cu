// The first kernel of every call: positions staged into the library's layout,
// every accumulator of the call cleared, the atoms' extents reduced and the
// lookup-table grids derived from them -- one launch, where staging, the
// extents, the grid and seven clears each took their own (about 25 us of a
// 1,000-atom step).
//
// Each block reduces the extents of its 256 atoms; the block that finishes
// last (an atomic ticket, no block waits) combines the partial results and
// writes the grid records.  Sums are FP64 in a fixed tree, so the centre of
// geometry is the same bits every call.
#include <math.h>

#include <algorithm>

#include "gbx_internal.cuh"
#include "queries.cuh"

namespace gbx {
namespace {

constexpr int kPrepThreads = 256;
constexpr int kTree = 1024;  // leaves of the tree over the blocks' partial results
constexpr int kMaxClears = 12;

struct GeomPart {
  float mn[3], mx[3];
  float wmax;     // largest main model parameter (GBSW: R')
  float pad;
  double sum[3];  // coordinates (centre of geometry)
  double rmax;    // largest radius
};

struct Clear {
  unsigned* p;
  size_t words;
};

struct PrepareArgs {
  const void* in;
  const int* slot_of;
  const float* wpar;
  const double* radius;
  int n;
  float4* pos;
  ulonglong2* f4;
  GeomPart* parts;
  unsigned* ticket;
  unsigned* status;
  Clear clear[kMaxClears];
  int nclear;
  // the exact table's grid (tight) and the reference's (ref), either may be null
  TableGeom* tight;
  double tight_h, switch_width, extent;
  long long tight_cap;
  TableGeom* ref;
  int mode;
  double h, buffer, box[3], reach;
  long long ref_cap;
  SortGeom* sort;  // the grid of the atoms' spatial order
};

// Internal positions: x, y, z and the model's main per-atom parameter in .w
// (GBSW: R' = (R + 0.03) 0.952, CharmmReferenceGBSW.cpp:625; GBMV-I:
// gamma_j = gamma0 ln(lambda) / R^4, GBMVIntegralTypeI.cpp:168; GBMV-II:
// C_j = 10 P1 R + P2, GBMVIntegralTypeII.cpp:179), from the caller's float4
// or double4 positions (OpenMM's single / double precision posq).  With an
// atom order set, internal atom i is read from the caller's slot slot_of[i].
template <bool DBL>
__device__ __forceinline__ float4 staged(const PrepareArgs& a, int i) {
  const int k = a.slot_of ? a.slot_of[i] : i;
  if (DBL) {
    const double4 p = static_cast<const double4*>(a.in)[k];
    return make_float4((float)p.x, (float)p.y, (float)p.z, a.wpar[i]);
  }
  const float4 p = static_cast<const float4*>(a.in)[k];
  return make_float4(p.x, p.y, p.z, a.wpar[i]);
}

__device__ __forceinline__ float warp_min(float v) {
  for (int off = 16; off > 0; off >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// sqrt(3.0)/2.0 as the reference computes it in double.
__device__ __forceinline__ double half_sqrt3() { return __ddiv_rn(__dsqrt_rn(3.0), 2.0); }

// The exact GBSW table's grid along one axis (k_tight.cu).
__device__ __forceinline__ void tight_axis(const PrepareArgs& a, const GeomPart& e, int k, TableGeom& g,
                                           unsigned& status) {
  const double h = a.tight_h, margin = (double)e.wmax + a.switch_width + h;
  g.min[k] = (double)e.mn[k] - margin;
  g.dims[k] = axis_cells(((double)e.mx[k] - (double)e.mn[k] + 2.0 * margin) / h, status);
  if (g.dims[k] > 65536) {
    status |= kStatusTableCells;
    g.dims[k] = 1;
  }
  g.max[k] = g.min[k] + g.dims[k] * h;
  g.step[k] = h;
  g.box[k] = 0.0;
  g.inv_step[k] = 1.0 / h;
  g.inv_box[k] = 0.0;
}

__device__ __forceinline__ void tight_rest(const PrepareArgs& a, const GeomPart& e, TableGeom& g, unsigned& status) {
  const double margin = (double)e.wmax + a.switch_width + a.tight_h;
  double amax = 0.0;
  for (int k = 0; k < 3; ++k) amax = fmax(amax, fmax(fabs((double)e.mn[k]), fabs((double)e.mx[k])));
  g.mode = -1;
  g.reach = a.reach;
  g.L = a.tight_h;
  // membership margin: FP32 rounding of cell coordinates and distances
  // (extent: a periodic system's longest box edge, by which a point may be moved)
  g.pad = 2e-5 + 4.0 * 1.1920929e-7 * (amax + 2.0 * margin + a.extent);
  g.total = 0;
  g.longest = 0;
  g.chained = 0u;
  g.ncell = grid_cells(g.dims);
  if (g.ncell > a.tight_cap) status |= kStatusTableCells;
}

// The reference's grid along one axis: CharmmReferenceGBSW.cpp:444-466,
// CustomGBIntegral.cpp:53-113,163-193, every operation separately rounded.
__device__ __forceinline__ void ref_axis(const PrepareArgs& a, const GeomPart& e, int k, TableGeom& g,
                                         unsigned& status) {
  const double box = k == 0 ? a.box[0] : (k == 1 ? a.box[1] : a.box[2]);
  g.box[k] = box;  // of a standalone grid read only by a periodic system's wrapped query
  if (a.mode == GBX_TABLE_PERIODIC) {
    const double cog = __ddiv_rn(e.sum[k], (double)a.n), half = __ddiv_rn(box, 2.0);
    g.min[k] = __dsub_rn(cog, half);
    g.max[k] = __dadd_rn(cog, half);
    g.dims[k] = axis_cells(__ddiv_rn(box, a.h), status);
    g.step[k] = __ddiv_rn(box, (double)g.dims[k]);
  } else {
    double pad;
    if (a.mode == GBX_TABLE_STANDALONE)
      pad = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(a.buffer, e.rmax), a.switch_width), __dmul_rn(half_sqrt3(), a.h)),
                      1e-6);
    else
      pad = __dadd_rn(__dadd_rn(0.03, __dmul_rn(half_sqrt3(), a.h)), a.buffer);
    const double lo = __dsub_rn((double)e.mn[k], pad), hi = __dadd_rn((double)e.mx[k], pad);
    const double length = __dsub_rn(hi, lo);
    if (a.mode == GBX_TABLE_GRID && length > 1000.0) {
      status |= kStatusTableCells;
      g.dims[k] = 1;
    } else {
      g.dims[k] = axis_cells(__ddiv_rn(length, a.h), status);
    }
    g.min[k] = lo;
    g.max[k] = __dadd_rn(lo, __dmul_rn((double)(g.dims[k] - 1), a.h));
    g.step[k] = a.h;
    g.pad = pad;  // the same on every axis
  }
  g.inv_step[k] = 1.0 / g.step[k];
  g.inv_box[k] = box > 0.0 ? 1.0 / box : 0.0;
}

__device__ __forceinline__ void ref_rest(const PrepareArgs& a, TableGeom& g, unsigned& status) {
  g.mode = a.mode;
  g.reach = a.reach;
  g.total = 0;
  g.longest = 0;
  g.chained = 0u;
  g.L = a.mode == GBX_TABLE_PERIODIC ? fmax(fmax(g.step[0], g.step[1]), g.step[2]) : a.h;
  if (a.mode == GBX_TABLE_PERIODIC) g.pad = 0.0;
  g.ncell = grid_cells(g.dims);
  if (g.ncell > a.ref_cap) status |= kStatusTableCells;
}

// The grid of the atoms' spatial order: 1 nm cells, grown so that
// there are at most kMaxSortCells.  (One block that read every position for
// its extents took 27 us of a 50,000-atom step.)
__device__ __forceinline__ SortGeom sort_grid(const GeomPart& e) {
  SortGeom g;
  float cell = 1.0f;
  for (;;) {
    long long tot = 1;
    for (int d = 0; d < 3; ++d) {
      const float span = (e.mx[d] - e.mn[d]) / cell;
      // non-finite or huge spans (invalid positions) collapse to one cell row
      g.dims[d] = (span >= 0.0f && span < (float)kMaxSortCells) ? (int)span + 1 : 1;
      tot *= g.dims[d];
    }
    if (tot > kMaxSortCells && cell > 1e6f) {  // absurd extents: one cell
      g.dims[0] = g.dims[1] = g.dims[2] = 1;
      tot = 1;
    }
    if (tot <= kMaxSortCells) {
      for (int d = 0; d < 3; ++d) g.lo[d] = e.mn[d];
      g.inv_cell = 1.0f / cell;
      g.ncell = (int)tot;
      return g;
    }
    cell *= 1.25f;
  }
}

// REF: the reference's grid is wanted (FP64 sums and radii; the exact table's
// grid needs FP32 extents only).
template <bool DBL, bool REF>
__global__ void __launch_bounds__(kPrepThreads) prepare_kernel(const __grid_constant__ PrepareArgs a) {
  constexpr int kWarps = kPrepThreads / kWarp;
  __shared__ float s_f[7][kWarps];
  __shared__ double s_sum[3][REF ? kTree : 1];
  __shared__ double s_r[kWarps];
  __shared__ GeomPart s_all;
  __shared__ TableGeom s_geom[2];
  __shared__ unsigned s_status;
  __shared__ bool s_last;
  const int t = threadIdx.x, lane = t % kWarp, w = t / kWarp;
  // the call's accumulators
  for (int c = 0; c < a.nclear; ++c) {
    const Clear z = a.clear[c];
    uint4* p4 = reinterpret_cast<uint4*>(z.p);  // allocations start on 256-byte boundaries
    const size_t n4 = z.words / 4, stride = (size_t)gridDim.x * kPrepThreads;
    for (size_t k = (size_t)blockIdx.x * kPrepThreads + t; k < n4; k += stride) p4[k] = make_uint4(0u, 0u, 0u, 0u);
    if (blockIdx.x == 0 && t < (int)(z.words - 4 * n4)) z.p[4 * n4 + t] = 0u;
  }
  const int nparts = (a.n + kPrepThreads - 1) / kPrepThreads;
  if ((int)blockIdx.x < nparts) {
    const int i = blockIdx.x * kPrepThreads + t;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    float f[7] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY, 0.f};
    double r = 0.0;
    if (i < a.n) {
      p = staged<DBL>(a, i);
      a.pos[i] = p;
      a.f4[2 * i] = a.f4[2 * i + 1] = make_ulonglong2(0ull, 0ull);  // the chain rule's sums
      f[0] = f[3] = p.x;
      f[1] = f[4] = p.y;
      f[2] = f[5] = p.z;
      f[6] = p.w;
      if (REF) r = a.radius[i];
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      f[k] = k < 3 ? warp_min(f[k]) : warp_max(f[k]);
      if (lane == 0) s_f[k][w] = f[k];
    }
    if (REF) {
      r = warp_max(r);
      if (lane == 0) s_r[w] = r;
      const bool on = i < a.n;
      s_sum[0][t] = on ? (double)p.x : 0.0;
      s_sum[1][t] = on ? (double)p.y : 0.0;
      s_sum[2][t] = on ? (double)p.z : 0.0;
      __syncthreads();
      for (int stride = kPrepThreads / 2; stride > 0; stride >>= 1) {
        if (t < stride)
          for (int k = 0; k < 3; ++k) s_sum[k][t] = __dadd_rn(s_sum[k][t], s_sum[k][t + stride]);
        __syncthreads();
      }
    }
    __syncthreads();
    if (t == 0) {
      GeomPart g;
      for (int k = 0; k < 3; ++k) {
        g.mn[k] = s_f[k][0];
        g.mx[k] = s_f[3 + k][0];
        for (int u = 1; u < kWarps; ++u) {
          g.mn[k] = fminf(g.mn[k], s_f[k][u]);
          g.mx[k] = fmaxf(g.mx[k], s_f[3 + k][u]);
        }
        g.sum[k] = REF ? s_sum[k][0] : 0.0;
      }
      g.wmax = s_f[6][0];
      g.rmax = REF ? s_r[0] : 0.0;
      for (int u = 1; u < kWarps; ++u) {
        g.wmax = fmaxf(g.wmax, s_f[6][u]);
        if (REF) g.rmax = fmax(g.rmax, s_r[u]);
      }
      g.pad = 0.f;
      a.parts[blockIdx.x] = g;
    }
  }
  // the last block to arrive derives the grids
  __threadfence();
  if (t == 0) {
    const unsigned before = atomicAdd(a.ticket, 1u);
    s_last = before == gridDim.x - 1;
    if (s_last) *a.ticket = 0u;  // for the next call
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  float f[7] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY, 0.f};
  double r = 0.0;
  for (int b = t; b < nparts; b += kPrepThreads) {
    const float4 q0 = __ldcg(reinterpret_cast<const float4*>(a.parts + b)),
                 q1 = __ldcg(reinterpret_cast<const float4*>(a.parts + b) + 1);
    f[0] = fminf(f[0], q0.x);
    f[1] = fminf(f[1], q0.y);
    f[2] = fminf(f[2], q0.z);
    f[3] = fmaxf(f[3], q0.w);
    f[4] = fmaxf(f[4], q1.x);
    f[5] = fmaxf(f[5], q1.y);
    f[6] = fmaxf(f[6], q1.z);
    if (REF) r = fmax(r, __ldcg(&a.parts[b].rmax));
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    f[k] = k < 3 ? warp_min(f[k]) : warp_max(f[k]);
    if (lane == 0) s_f[k][w] = f[k];
  }
  if (REF) {
    r = warp_max(r);
    if (lane == 0) s_r[w] = r;
    // leaf v sums blocks v, v + kTree, ... in that order; leaves past the last block are zero
    int leaves = 1;
    while (leaves < nparts && leaves < kTree) leaves <<= 1;
    for (int v = t; v < leaves; v += kPrepThreads)
      for (int k = 0; k < 3; ++k) {
        double s = 0.0;
        for (int b = v; b < nparts; b += kTree) s = __dadd_rn(s, __ldcg(&a.parts[b].sum[k]));
        s_sum[k][v] = s;
      }
    __syncthreads();
    for (int stride = leaves / 2; stride > 0; stride >>= 1) {
      for (int v = t; v < stride; v += kPrepThreads)
        for (int k = 0; k < 3; ++k) s_sum[k][v] = __dadd_rn(s_sum[k][v], s_sum[k][v + stride]);
      __syncthreads();
    }
  }
  __syncthreads();
  if (t == 0) {
    GeomPart g;
    for (int k = 0; k < 3; ++k) {
      g.mn[k] = s_f[k][0];
      g.mx[k] = s_f[3 + k][0];
      for (int u = 1; u < kWarps; ++u) {
        g.mn[k] = fminf(g.mn[k], s_f[k][u]);
        g.mx[k] = fmaxf(g.mx[k], s_f[3 + k][u]);
      }
      g.sum[k] = REF ? s_sum[k][0] : 0.0;
    }
    g.wmax = s_f[6][0];
    g.rmax = REF ? s_r[0] : 0.0;
    for (int u = 1; u < kWarps; ++u) {
      g.wmax = fmaxf(g.wmax, s_f[6][u]);
      if (REF) g.rmax = fmax(g.rmax, s_r[u]);
    }
    s_all = g;
    s_status = 0u;
  }
  __syncthreads();
  // an axis per thread (the FP64 divisions are long chains), one warp per grid
  unsigned status = 0u;
  if (w == 0 && a.tight) {
    if (lane < 3) tight_axis(a, s_all, lane, s_geom[0], status);
    __syncwarp();
    if (lane == 0) tight_rest(a, s_all, s_geom[0], status);
  }
  if (REF && w == 1 && a.ref) {
    if (lane < 3) ref_axis(a, s_all, lane, s_geom[1], status);
    __syncwarp();
    if (lane == 0) ref_rest(a, s_geom[1], status);
  }
  if (a.sort && w == 2 && lane == 0) *a.sort = sort_grid(s_all);
  if (status) atomicOr(&s_status, status);
  __syncthreads();
  if (t == 0) {
    if (a.tight) *a.tight = s_geom[0];
    *a.status = s_status;  // the first word of this call's status
  }
  if (REF && t == 32 && a.ref) *a.ref = s_geom[1];
}

}  // namespace

size_t prepare_scratch_bytes(int n) { return sizeof(GeomPart) * (size_t)((n + kPrepThreads - 1) / kPrepThreads); }

gbx_status launch_prepare(Context* ctx, const void* posq, bool tight, bool reference, bool call) {
  const gbx_config& c = ctx->cfg;
  const int n = ctx->n;
  PrepareArgs a{};
  a.in = posq;
  a.slot_of = ctx->in_permuted ? ctx->d_slot_of : nullptr;
  a.wpar = ctx->d_wpar;
  a.radius = ctx->d_radius;
  a.n = n;
  a.pos = ctx->d_pos;
  a.f4 = reinterpret_cast<ulonglong2*>(ctx->d_f4);
  a.parts = static_cast<GeomPart*>(ctx->d_parts);
  a.ticket = ctx->d_ticket;
  a.status = ctx->d_status;
  size_t words = 0;
  auto clear = [&](void* p, size_t w) {
    if (!p || w == 0) return;
    a.clear[a.nclear++] = Clear{static_cast<unsigned*>(p), w};
    words += w;
  };
  if (call) {
    clear(ctx->d_dEdB_fx, 2 * (size_t)n);
    clear(ctx->d_energy_fx, 2);
    clear(ctx->d_next_item, 1);
    clear(ctx->d_rmax, 1);
  }
  if (call && (pair_in_order(ctx) || items_in_order(ctx))) {
    a.sort = ctx->d_sgeom;
    clear(ctx->d_scount, kMaxSortCells);
  }
  const bool wrapped = tight && c.periodic;  // the standalone grid's edges decide where a point is moved
  if (tight) {
    a.tight = ctx->d_tgeom;
    a.tight_h = ctx->tight_h;
    a.extent = c.periodic ? fmax(c.box[0], fmax(c.box[1], c.box[2])) : 0.0;
    a.tight_cap = ctx->tcell_cap;
    clear(ctx->d_tcount, (size_t)ctx->tcell_cap);
    clear(ctx->d_tburied, (size_t)ctx->tcell_cap);
    clear(ctx->tbuckets.chain, (size_t)ctx->tcell_cap);
  }
  if (reference) {
    clear(ctx->d_cell_count, (size_t)ctx->cell_cap);
    clear(ctx->buckets.chain, (size_t)ctx->cell_cap);
    clear(ctx->d_pcount, (size_t)ctx->cell_cap);
    clear(ctx->d_ptotal, 2);
  }
  a.switch_width = c.switch_width;
  a.ref = reference ? ctx->d_geom : wrapped ? ctx->d_wgeom : nullptr;
  a.mode = wrapped ? GBX_TABLE_STANDALONE : c.table_mode;
  a.h = c.grid_length;
  a.buffer = c.table_buffer;
  a.reach = c.r1;
  for (int k = 0; k < 3; ++k) a.box[k] = c.box[k];
  a.ref_cap = wrapped ? 0x7fffffffffffffffLL : ctx->cell_cap;  // no cell of the wrapping grid is ever indexed
  // a block per 256 atoms; more where the clears are longer than the atoms
  // (4 KB per block and clear), up to four per SM
  const long long atoms = (n + kPrepThreads - 1) / kPrepThreads;
  const long long fill = std::min<long long>((long long)(words / 1024), 4LL * ctx->sms);
  const int grid = (int)std::max(atoms, fill);
  if (a.ref) {
    if (ctx->in_double) prepare_kernel<true, true><<<grid, kPrepThreads, 0, ctx->stream>>>(a);
    else prepare_kernel<false, true><<<grid, kPrepThreads, 0, ctx->stream>>>(a);
  } else {
    if (ctx->in_double) prepare_kernel<true, false><<<grid, kPrepThreads, 0, ctx->stream>>>(a);
    else prepare_kernel<false, false><<<grid, kPrepThreads, 0, ctx->stream>>>(a);
  }
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("prepare launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

}  // namespace gbx
