// GBMV-I / GBMV-II integrals and chain rule, processed cell by cell.
//
// Every quadrature point of the GBMV models reads the whole (capped) list of
// the lookup-table cell it falls in (GBMVIntegralTypeI.cpp:111-173,
// GBMVIntegralTypeII.cpp:116-191), and a cell is shared by a few hundred
// points of many atoms.  Instead of each point gathering its list through
// L1, the points are binned by cell and one warp takes one cell: it stages
// the cell's list in shared memory once, and then every lane evaluates its
// own point against entries that all lanes read at the same address (a
// shared-memory broadcast).
//
//   bin      warp per (atom, quadrature chunk), lanes over points: the
//            point's cell (the reference query, exact near cell faces),
//            a slot in the cell by one atomic per run of a ray's points in
//            one cell, four points per lane in flight; points whose cell has
//            no list get their solvent fraction here
//   scan     points per cell -> each cell's first slot
//   fill     point ids into their cell's slots
//   integral warp per cell: sorts the cell's point ids (the slots were
//            handed out by atomics, in no fixed order) so that every later
//            sum over the cell's points has an order fixed by the input
//            (cells of more than kSortMax points keep the atomic order and
//            the chain rule reduces each of their contributions on its own);
//            per point the list sums in list order, the solvent fraction by
//            point id, and the point's sums by slot for the chain rule
//   reduce   warp per (atom, chunk): J4, J7 over the solvent fractions in
//            quadrature order (the integral pass's partition, so the Born
//            radii are assembled as before)
//   chain    warp per cell over the points whose solvent fraction still
//            varies (the integral pass leaves them first), lanes as 4 points
//            x 8 lanes of entry pairs
//            (packed FP32x2, two entries per instruction; the integral pass
//            likewise evaluates two entries per instruction): each lane
//            keeps the pull of its entries in registers over all of the
//            cell's points (one fixed-point reduction per cell and entry
//            instead of one per point and entry); the point's own pull is
//            summed across its 8 lanes and then over consecutive points of
//            the same atom (the sorted order keeps them together) before one
//            reduction per run
//
// Distances are formed in the cell's frame: entries as x_j - c0 and the
// point as (x_i - c0) + v_q, c0 the cell's corner, so every operand of the
// FP32 difference is within a few tenths of a nanometre of the cell.
#include <math.h>

#include <algorithm>

#include "bitonic.cuh"
#include "gbx_internal.cuh"
#include "queries.cuh"
#include "scan.cuh"

namespace gbx {
namespace {

constexpr int kBinThreads = 128;
constexpr int kCellWarps = 4;           // warps (cells) per block in the cell passes
constexpr int kCellThreads = kCellWarps * kWarp;
constexpr int kMaxList = 64;            // longest list the cell passes stage (the GBMV table cap)
constexpr int kSortMax = 16 * kWarp;    // cells of up to 512 points are sorted in registers
constexpr int kChainPts = 4;            // points per chain sub-step
constexpr int kChainEnt = kWarp / kChainPts;  // entry lanes per point
constexpr int kEntPerLane = kMaxList / kChainEnt;
static_assert(kChainPts * kChainEnt == kWarp && kChainPts == 4, "chain lane split: a point lane per pushed field");

struct CellPoints {
  int* count;   // [cells] points binned into the cell
  int* live;    // [cells] of those, the points the chain rule visits: first in the cell's slots
  int* start;   // [cells + 1] first slot
  int* order;   // [points] point id per slot, sorted within each cell by the integral pass
  int2* at;     // [points] (the point's cell or -1, its slot within the cell in atomic order)
  float* sval;  // [points] solvent fraction by point id
  float* state; // [planes][points] the point's sums by slot (GBMV-I: S; GBMV-II: s1, s2, vx, vy, vz)
  size_t plane;
};

// Point sums of a list for one point (lists in ascending atom order).
struct Sums {
  float s1, s2, vx, vy, vz;
};

// Minimum image for a box-sampled table of a periodic system (CutoffPeriodic:
// GBMVIntegralTypeI.cpp:59-62, TypeII.cpp:64-67); nothing otherwise.
template <bool PER>
struct Image {
  float L[3], iL[3];
  __device__ __forceinline__ void init(const TableGeom& g) {
    if (PER)
      for (int k = 0; k < 3; ++k) {
        L[k] = (float)g.box[k];
        iL[k] = (float)g.inv_box[k];
      }
  }
  __device__ __forceinline__ void apply2(float2& dx, float2& dy, float2& dz) const {
    if (PER) {
      dx = make_float2(fmaf(-L[0], floorf(fmaf(dx.x, iL[0], 0.5f)), dx.x), fmaf(-L[0], floorf(fmaf(dx.y, iL[0], 0.5f)), dx.y));
      dy = make_float2(fmaf(-L[1], floorf(fmaf(dy.x, iL[1], 0.5f)), dy.x), fmaf(-L[1], floorf(fmaf(dy.y, iL[1], 0.5f)), dy.y));
      dz = make_float2(fmaf(-L[2], floorf(fmaf(dz.x, iL[2], 0.5f)), dz.x), fmaf(-L[2], floorf(fmaf(dz.y, iL[2], 0.5f)), dz.y));
    }
  }
  __device__ __forceinline__ float3 apply(float3 d) const {
    if (PER) {
      d.x = fmaf(-L[0], floorf(fmaf(d.x, iL[0], 0.5f)), d.x);
      d.y = fmaf(-L[1], floorf(fmaf(d.y, iL[1], 0.5f)), d.y);
      d.z = fmaf(-L[2], floorf(fmaf(d.z, iL[2], 0.5f)), d.z);
    }
    return d;
  }
};

__device__ __forceinline__ float3 cell_corner(const TableGeom& g, int cell) {
  const int d12 = g.dims[1] * g.dims[2];
  const int ix = cell / d12, r = cell - ix * d12;
  const int iy = r / g.dims[2], iz = r - iy * g.dims[2];
  return make_float3((float)(g.min[0] + ix * g.step[0]), (float)(g.min[1] + iy * g.step[1]),
                     (float)(g.min[2] + iz * g.step[2]));
}

// The solvent fraction of a point whose cell has no list: GBMV-I S = 0;
// GBMV-II an empty list gives V = 0 (GBMVIntegralTypeII.cpp:140).
template <int MODEL>
__device__ __forceinline__ float empty_list_fraction(const ModelConst& m) {
  if (MODEL == GBX_MODEL_GBMV2) return 1.0f;
  float p;
  return logistic_solvent(m.beta, m.lambda, 0.0f, p);
}

// One binned point: its slot in its cell, or (no list) its solvent fraction.
template <int MODEL>
__device__ __forceinline__ void bin_point(const CellPoints& cp, const Entries& tab, const ModelConst& m, size_t p,
                                          long long cell) {
  const int cnt = cell >= 0 ? __ldg(&tab.cell[cell].x) : 0;
  if (cnt > 0) {
    cp.at[p] = make_int2((int)cell, atomicAdd(&cp.count[cell], 1));
  } else {
    cp.at[p].x = -1;
    cp.sval[p] = empty_list_fraction<MODEL>(m);
  }
}

template <int MODEL, class Q>
__global__ void __launch_bounds__(kBinThreads) gbmv_bin_kernel(const float4* __restrict__ pos, int n, Entries tab,
                                                               Quad quad, ModelConst m, int chunk, int n_chunks,
                                                               CellPoints cp) {
  // kBinBatch points per lane per step: their cell queries, list-count loads
  // and slot atomics are issued back to back.  A point within the FP32
  // query's guard band (one in several thousand) needs the FP64 query; those are
  // queued per warp and resolved kBinDefer at a time with every lane busy,
  // instead of stalling the warp for each one (FP64 runs at a small fraction
  // of the FP32 rate on this part, whatever the number of active lanes).
  constexpr int kBinBatch = 4;
  constexpr int kBinDefer = 256;
  static_assert(kBinDefer >= 2 * kBinBatch * kWarp, "deferred queue");
  __shared__ int s_defer[kBinThreads / kWarp][kBinDefer];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp;
  const int wib = threadIdx.x / kWarp;
  if (warp >= n * n_chunks) return;
  const int i = warp % n, c = warp / n;
  const float4 xi = pos[i];
  Q query;
  query.init(tab, xi, quad.qoff);
  const int q0 = c * chunk, q1 = min(m.nq, q0 + chunk);
  const unsigned lt = (1u << lane) - 1u;
  int* defer = s_defer[wib];
  int ndef = 0;  // warp-uniform
  auto flush = [&]() {
    __syncwarp();
    for (int k = lane; k < ndef; k += kWarp) {
      const int q = defer[k];
      bin_point<MODEL>(cp, tab, m, (size_t)i * m.nq + q, query.cell(xi, quad.qv[q], q));
    }
    __syncwarp();
    ndef = 0;
  };
  for (int base = q0; base < q1; base += kBinBatch * kWarp) {
    int cell[kBinBatch];
    int cnt[kBinBatch];
    bool late[kBinBatch];
#pragma unroll
    for (int u = 0; u < kBinBatch; ++u) {
      const int q = base + u * kWarp + lane;
      cell[u] = -1;
      cnt[u] = 0;
      late[u] = false;
      if (q < q1) cell[u] = (int)query.cell_fast(quad.qv[q], late[u]);
      const unsigned dm = __ballot_sync(0xffffffffu, late[u]);
      if (late[u]) defer[ndef + __popc(dm & lt)] = q;
      ndef += __popc(dm);
    }
#pragma unroll
    for (int u = 0; u < kBinBatch; ++u)
      if (cell[u] >= 0) cnt[u] = __ldg(&tab.cell[cell[u]].x);
    // Neighbouring lanes hold neighbouring points of a ray: a run of lanes in one
    // cell takes its slots with one atomic, as consecutive slots
    int slot[kBinBatch];
    int run[kBinBatch];  // the lane that starts this lane's run
#pragma unroll
    for (int u = 0; u < kBinBatch; ++u) {
      const int before = __shfl_up_sync(0xffffffffu, cell[u], 1);
      const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || cell[u] != before);
      run[u] = 31 - __clz((int)(heads & (lt | (1u << lane))));
      const unsigned later = heads & ~(lt | (1u << lane));
      const int len = (later ? __ffs((int)later) - 1 : kWarp) - lane;  // of a run's first lane
      slot[u] = 0;
      if (run[u] == lane && cell[u] >= 0 && cnt[u] > 0) slot[u] = atomicAdd(&cp.count[cell[u]], len);
    }
#pragma unroll
    for (int u = 0; u < kBinBatch; ++u) slot[u] = __shfl_sync(0xffffffffu, slot[u], run[u]) + lane - run[u];
#pragma unroll
    for (int u = 0; u < kBinBatch; ++u) {
      const int q = base + u * kWarp + lane;
      const size_t p = (size_t)i * m.nq + q;
      if (cell[u] >= 0 && cnt[u] > 0) {
        cp.at[p] = make_int2(cell[u], slot[u]);
      } else if (q < q1 && !late[u]) {
        cp.at[p].x = -1;
        cp.sval[p] = empty_list_fraction<MODEL>(m);
      }
    }
    if (ndef > kBinDefer - kBinBatch * kWarp) flush();
  }
  if (ndef > 0) flush();
}

// kFillLoads points in flight per thread; a warp's points are consecutive, so
// a run's slots are written together.
constexpr int kFillLoads = 4;
constexpr int kFillThreads = 256;
__global__ void __launch_bounds__(kFillThreads) gbmv_fill_kernel(long long npts, CellPoints cp) {
  const long long p0 = (long long)blockIdx.x * (kFillThreads * kFillLoads) + threadIdx.x;
  int2 v[kFillLoads];
  int start[kFillLoads];
#pragma unroll
  for (int u = 0; u < kFillLoads; ++u) {
    const long long p = p0 + u * kFillThreads;
    v[u] = p < npts ? __ldcs(cp.at + p) : make_int2(-1, 0);
  }
#pragma unroll
  for (int u = 0; u < kFillLoads; ++u) start[u] = v[u].x >= 0 ? __ldg(cp.start + v[u].x) : 0;
#pragma unroll
  for (int u = 0; u < kFillLoads; ++u)
    if (v[u].x >= 0) cp.order[start[u] + v[u].y] = (int)(p0 + u * kFillThreads);
}

template <int E>
__device__ __forceinline__ void sort_slots(int* __restrict__ order, int P, int lane) {
  int key[E];
#pragma unroll
  for (int r = 0; r < E; ++r) {
    const int e = lane * E + r;
    key[r] = e < P ? order[e] : 0x7fffffff;
  }
  warp_bitonic_sort<E>(key, lane);
#pragma unroll
  for (int r = 0; r < E; ++r) {
    const int e = lane * E + r;
    if (e < P) order[e] = key[r];
  }
}

// Sorts the cell's point ids in place (cells of more than kSortMax points
// keep the atomic order; the chain rule then takes an order-free path).
__device__ __noinline__ void sort_cell(int* order, int P, int lane) {
  if (P <= kWarp) sort_slots<1>(order, P, lane);
  else if (P <= 2 * kWarp) sort_slots<2>(order, P, lane);
  else if (P <= 4 * kWarp) sort_slots<4>(order, P, lane);
  else if (P <= 8 * kWarp) sort_slots<8>(order, P, lane);
  else if (P <= kSortMax) sort_slots<16>(order, P, lane);
}

// Hardware reciprocal (PTX rcp.approx, relative error below 2^-22; the
// denominators here are >= 1 in magnitude, never subnormal).
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 rcp2(float2 t) { return make_float2(rcp_ftz(t.x), rcp_ftz(t.y)); }

// The cell's list staged in shared memory, one array per field, so that four
// consecutive entries load as one float4 (two pairs) and each pair feeds
// packed FP32x2 arithmetic (__ffma2_rn and friends: one instruction for two
// entries, each half rounded as its scalar form).  A list whose length is
// not a multiple of four is padded with entries whose every contribution is
// exactly zero (C = 0 for GBMV-II; T = 100 r^2 + 1 >= 1).
struct __align__(16) CellList {
  float x[kMaxList], y[kMaxList], z[kMaxList];  // x_j - c0
  float w[kMaxList];    // GBMV-II C_j | GBMV-I gamma_j
  float k[kMaxList];    // GBMV-II C_j - 100 R_j^2 | GBMV-I R_j
};

// The chain rule's copy: pairs of entries, read as three 16-byte words per
// pair (five fields and the indices read one by one held the load pipe).
struct __align__(16) ChainPair {
  float2 x, y, z;  // x_j - c0
  float2 w;        // GBMV-II C_j | GBMV-I gamma_j
  float2 k;        // GBMV-II C_j - 100 R_j^2 | GBMV-I's adjoint -4 gamma_j / R_j
  int2 idx;        // atom index
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

template <bool PER>
__device__ __forceinline__ void stage_list(CellList& L, const Entries& tab, int2 cs, int cnt, float3 c0, int lane) {
  const int cnt4 = (cnt + 3) & ~3;
  for (int l = lane; l < cnt4; l += kWarp) {
    if (l < cnt) {
      const float4 a = __ldg(tab.e + cs.y + l);
      const float2 pk = __ldg(tab.par + cs.y + l);
      L.x[l] = a.x - c0.x;
      L.y[l] = a.y - c0.y;
      L.z[l] = a.z - c0.z;
      L.w[l] = a.w;
      L.k[l] = pk.x;
    } else {
      L.x[l] = L.y[l] = L.z[l] = 0.0f;
      L.w[l] = 0.0f;
      L.k[l] = 1.0f;
    }
  }
}

template <int MODEL, bool PER>
__global__ void __launch_bounds__(kCellThreads, 8) gbmv_cell_integral_kernel(const float4* __restrict__ pos, Entries tab,
                                                                          Quad quad, ModelConst m, CellPoints cp) {
  __shared__ CellList s_list[kCellWarps];
  const int w = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const long long cell = (long long)blockIdx.x * kCellWarps + w;
  const TableGeom& G = *tab.geom;
  if (cell >= G.ncell || cell >= tab.cell_cap) return;
  const int P = cp.count[cell];
  if (P == 0) return;
  const int2 cs = __ldg(tab.cell + cell);
  const int cnt = min(cs.x, kMaxList);
  const float3 c0 = cell_corner(G, (int)cell);
  Image<PER> img;
  img.init(G);
  CellList& L = s_list[w];
  stage_list<PER>(L, tab, cs, cnt, c0, lane);
  const int start = cp.start[cell];
  int* order = cp.order + start;
  if (P > 1) sort_cell(order, P, lane);
  __syncwarp();
  // GBMV-II's padding entries add exactly zero; GBMV-I's (e^0 = 1) do not,
  // so its last (cnt mod 4) entries are taken one at a time
  const int nquad = MODEL == GBX_MODEL_GBMV2 ? (cnt + 3) >> 2 : cnt >> 2;
  int kept = 0;  // warp-uniform: points of the cell the chain rule visits
  for (int base = 0; base < P; base += kWarp) {
    const int k = base + lane;
    const bool valid = k < P;
    const int p = valid ? order[k] : 0;
    const int i = m.point_atom(p), q = p - i * m.nq;
    const float4 xi = __ldg(pos + i), v = __ldg(quad.qv + q);
    const float px = (xi.x - c0.x) + v.x, py = (xi.y - c0.y) + v.y, pz = (xi.z - c0.z) + v.z;
    const float2 npx = bc2(-px), npy = bc2(-py), npz = bc2(-pz);
    float2 s1 = bc2(0.f), s2 = bc2(0.f), vx = bc2(0.f), vy = bc2(0.f), vz = bc2(0.f);
    auto pair = [&](float2 ex, float2 ey, float2 ez, float2 ew, float2 ek) {
      float2 dx = __fadd2_rn(ex, npx), dy = __fadd2_rn(ey, npy), dz = __fadd2_rn(ez, npz);
      img.apply2(dx, dy, dz);
      const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
      if (MODEL == GBX_MODEL_GBMV1) {
        const float2 g = __fmul2_rn(ew, __fmul2_rn(r2, r2));
        s1 = __fadd2_rn(s1, make_float2(__expf(g.x), __expf(g.y)));
      } else {
        const float2 T = __ffma2_rn(bc2(100.0f), r2, ek);
        float2 F = __fmul2_rn(ew, rcp2(T));
        F = __fmul2_rn(F, F);
        s1 = __fadd2_rn(s1, F);
        s2 = __ffma2_rn(r2, __fmul2_rn(F, F), s2);
        vx = __ffma2_rn(dx, F, vx);
        vy = __ffma2_rn(dy, F, vy);
        vz = __ffma2_rn(dz, F, vz);
      }
    };
    for (int j = 0; j < nquad; ++j) {
      const int l = 4 * j;
      const float4 X = ld4(L.x + l), Y = ld4(L.y + l), Z = ld4(L.z + l), W = ld4(L.w + l);
      const float4 K4 = MODEL == GBX_MODEL_GBMV2 ? ld4(L.k + l) : make_float4(0.f, 0.f, 0.f, 0.f);
      pair(lo2(X), lo2(Y), lo2(Z), lo2(W), lo2(K4));
      pair(hi2(X), hi2(Y), hi2(Z), hi2(W), hi2(K4));
    }
    Sums s{s1.x + s1.y, s2.x + s2.y, vx.x + vx.y, vy.x + vy.y, vz.x + vz.y};
    if (MODEL == GBX_MODEL_GBMV1) {
      for (int l = 4 * nquad; l < cnt; ++l) {
        const float3 d = img.apply(make_float3(L.x[l] - px, L.y[l] - py, L.z[l] - pz));
        const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
        s.s1 += __expf(L.w[l] * (r2 * r2));
      }
    }
    // Only a point whose solvent fraction still varies pulls on anything (a
    // saturated one, 57 in 100 at 10,000 atoms, has an exactly zero
    // derivative): the chain rule's points and their sums are packed to those,
    // in order, over the slots already read.
    bool live = false;
    if (valid) {
      float pl, S;
      if (MODEL == GBX_MODEL_GBMV1) {
        S = s.s1;
      } else {
        const float s3sq = fmaf(s.vx, s.vx, fmaf(s.vy, s.vy, s.vz * s.vz));
        S = m.s0 * s.s1 * s.s2 / s3sq;
      }
      cp.sval[p] = logistic_solvent(m.beta, m.lambda, S, pl);
      live = logistic_slope(m.beta, pl) != 0.0f;
    }
    const unsigned lm = __ballot_sync(0xffffffffu, live);
    if (live) {
      const int slot = kept + __popc(lm & ((1u << lane) - 1u));
      order[slot] = p;
      float* st = cp.state + start + slot;
      st[0] = s.s1;
      if (MODEL == GBX_MODEL_GBMV2) {
        st[cp.plane] = s.s2;
        st[2 * cp.plane] = s.vx;
        st[3 * cp.plane] = s.vy;
        st[4 * cp.plane] = s.vz;
      }
    }
    kept += __popc(lm);
    __syncwarp();
  }
  if (lane == 0) cp.live[cell] = kept;
}

// J4, J7 per (atom, chunk) over the solvent fractions, in quadrature order.
__global__ void __launch_bounds__(kBinThreads) gbmv_reduce_kernel(int n, Quad quad, int nq, int chunk, int n_chunks,
                                                                  const float* __restrict__ sval,
                                                                  float* __restrict__ Jpart) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp;
  if (warp >= n * n_chunks) return;
  const int i = warp % n, c = warp / n;
  const int q0 = c * chunk, q1 = min(nq, q0 + chunk);
  const float* s = sval + (size_t)i * nq;
  float J4 = 0.0f, J7 = 0.0f;
  for (int q = q0 + lane; q < q1; q += kWarp) {
    const float sf = s[q];
    const float2 w = __ldg(quad.qw + q);
    J4 = fmaf(w.x, sf, J4);
    J7 = fmaf(w.y, sf, J7);
  }
  for (int off = 16; off > 0; off >>= 1) {
    J4 += __shfl_xor_sync(0xffffffffu, J4, off);
    J7 += __shfl_xor_sync(0xffffffffu, J7, off);
  }
  if (lane == 0) {
    Jpart[(size_t)c * n + i] = J4;
    Jpart[((size_t)n_chunks + c) * n + i] = J7;
  }
}

struct CellChainOut {
  unsigned long long* f4;  // per atom: force x, y, z and dE/dR (fixed point)
};

__device__ __forceinline__ void add_fixed3(const CellChainOut& o, int k, float gx, float gy, float gz) {
  const long long fx = float_to_fixed(gx), fy = float_to_fixed(gy), fz = float_to_fixed(gz);
  unsigned long long* f = o.f4 + 4 * (size_t)k;
  if (fx) atomicAdd(f, (unsigned long long)fx);
  if (fy) atomicAdd(f + 1, (unsigned long long)fy);
  if (fz) atomicAdd(f + 2, (unsigned long long)fz);
}

// Field c of atom k (3: dE/dR), one fixed-point reduction (skipped when the value rounds to zero).
__device__ __forceinline__ void add_fixed_one(const CellChainOut& o, int k, int c, float v) {
  const long long r = float_to_fixed(v);
  if (r) atomicAdd(o.f4 + 4 * (size_t)k + c, (unsigned long long)r);
}

// One point's chain-rule factors (the point's own lanes read them from
// shared memory): its position in the cell frame and the factors of the
// gradient with c ds/dS folded in.  GBMV-II: the pull on entry j is
//   g_j = F_j [ (-400 W_j / T_j + B F_j) d_j + V ],  W_j = A + B F_j r_j^2 + V . d_j
// with A = c ds/dS s0 s2 / |v|^2, B = 2 c ds/dS s0 s1 / |v|^2 and
// V = -2 c ds/dS s0 s1 s2 / |v|^4 v (the d s1, d s2 and d |v|^2 factors), and
// c ds/dS dS/dR_j = W_j dF_j/dR_j.  Written this way a pair of entries takes 27
// packed operations, where the expanded gradient took 35.
// GBMV-I: g_j = A e_j r_j^2 d_j with A = 4 c ds/dS, gamma_j folded per entry.
struct __align__(16) PointChain {
  float2 npx, npy, npz;  // minus the point's position in the cell frame, in both halves
  float2 A, B;           // GBMV-I: A only
  float2 Vx, Vy, Vz;
  float cS;
  int i;
};

// One warp (cell) per block: cells differ several-fold in points, and a block of
// four held its registers until its slowest warp was done.  Registers are
// capped where the occupancy measured fastest (10,000 atoms, 24 x 50, with 24,
// 28, 32 blocks per SM: GBMV-II 381, 360, 369 us; GBMV-I 453, 416, 406 us;
// four-warp blocks 405 and 446 us).
constexpr int kChainWarps = 1;
struct ChainShared {
  ChainPair list[kMaxList / 2];
  PointChain pt[kWarp];
  float3 own[kWarp];
};

// One cell: P points, first in its slots, of `binned`.  r: R_j of the pairs (adjoint).
template <int MODEL, bool PER, bool ADJ>
__device__ __forceinline__ void chain_cell(const float4* __restrict__ pos, const Entries& tab, const Quad& quad,
                                           const ModelConst& m, const CellPoints& cp, const float2* __restrict__ dEdJ,
                                           const CellChainOut& out, long long cell, int binned, int P, int lane,
                                           ChainShared& sh, float2* r) {
  const TableGeom& G = *tab.geom;
  const int2 cs = __ldg(tab.cell + cell);
  const int cnt = min(cs.x, kMaxList);
  const float3 c0 = cell_corner(G, (int)cell);
  Image<PER> img;
  img.init(G);
  ChainPair* L = sh.list;
  for (int l = lane; l < ((cnt + 1) & ~1); l += kWarp) {
    float4 a = make_float4(c0.x, c0.y, c0.z, 0.0f);  // padding: every contribution exactly zero
    float2 pk = make_float2(1.0f, 1.0f);
    int k = -1;
    if (l < cnt) {
      a = __ldg(tab.e + cs.y + l);
      pk = __ldg(tab.par + cs.y + l);
      k = __ldg(tab.index + cs.y + l);
    }
    float* f = reinterpret_cast<float*>(L + l / 2) + (l & 1);
    f[0] = a.x - c0.x;
    f[2] = a.y - c0.y;
    f[4] = a.z - c0.z;
    f[6] = a.w;
    // GBMV-I's adjoint: dS/dR_j = -4 gamma_j e_j r^4 / R_j (gamma ~ R^-4), the division once per entry
    f[8] = ADJ && MODEL == GBX_MODEL_GBMV1 ? -4.0f * a.w / pk.x : pk.x;
    f[10] = __int_as_float(k);
    if (ADJ) reinterpret_cast<float*>(r + l / 2)[l & 1] = pk.y;
  }
  __syncwarp();
  const int start = cp.start[cell];
  const int* order = cp.order + start;
  const float* state = cp.state + start;
  // cells too dense to sort keep the atomic slot order: every contribution
  // is then reduced on its own (integer sums, independent of the order)
  const bool sorted = binned <= kSortMax;
  // lane (ps, es): point ps of each group of kChainPts, entry pairs es, es +
  // kChainEnt, ... (entries 2 j and 2 j + 1 of pair j)
  const int ps = lane / kChainEnt, es = lane % kChainEnt;
  constexpr int kPairsPerLane = kEntPerLane / 2;
  float2 acc[kPairsPerLane][3];
  float2 accR[kPairsPerLane];
#pragma unroll
  for (int e = 0; e < kPairsPerLane; ++e) {
    acc[e][0] = acc[e][1] = acc[e][2] = bc2(0.f);
    accR[e] = bc2(0.f);
  }
  PointChain* pts = sh.pt;
  const float Cp = 10.0f * m.p1;
  for (int base = 0; base < P; base += kWarp) {
    // lane t prepares point base + t
    int np;
    {
      const int k = base + lane;
      PointChain pc;
      pc.cS = 0.0f;
      pc.i = -1;
      pc.npx = pc.npy = pc.npz = pc.A = pc.B = bc2(0.f);
      pc.Vx = pc.Vy = pc.Vz = bc2(0.f);
      if (k < P) {
        const int p = order[k];
        const int i = m.point_atom(p), q = p - i * m.nq;
        const float4 xi = __ldg(pos + i), v = __ldg(quad.qv + q);
        const float2 wq = __ldg(quad.qw + q);
        const float2 de = __ldg(dEdJ + i);
        const float cq = fmaf(de.x, wq.x, de.y * wq.y);
        pc.i = i;
        pc.npx = bc2(-((xi.x - c0.x) + v.x));
        pc.npy = bc2(-((xi.y - c0.y) + v.y));
        pc.npz = bc2(-((xi.z - c0.z) + v.z));
        float pl;
        if (MODEL == GBX_MODEL_GBMV1) {
          logistic_solvent(m.beta, m.lambda, state[k], pl);
          pc.cS = cq * logistic_slope(m.beta, pl);
          pc.A = bc2(4.0f * pc.cS);
        } else {
          const float s1 = state[k], s2 = state[k + cp.plane], vx = state[k + 2 * cp.plane],
                      vy = state[k + 3 * cp.plane], vz = state[k + 4 * cp.plane];
          const float s3sq = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
          logistic_solvent(m.beta, m.lambda, m.s0 * s1 * s2 / s3sq, pl);
          pc.cS = cq * logistic_slope(m.beta, pl) * m.s0;
          const float inv3 = 1.0f / s3sq;
          const float A = pc.cS * (s2 * inv3), B = 2.0f * pc.cS * (s1 * inv3),
                      C = 2.0f * pc.cS * (-s1 * s2 * inv3 * inv3);
          pc.A = bc2(A);
          pc.B = bc2(B);
          pc.Vx = bc2(C * vx);
          pc.Vy = bc2(C * vy);
          pc.Vz = bc2(C * vz);
        }
      }
      // a point whose factor came out zero after all (c = 0, an underflow) is
      // left out, the rest keep their order
      const unsigned lm = __ballot_sync(0xffffffffu, pc.cS != 0.0f);
      if (pc.cS != 0.0f) pts[__popc(lm & ((1u << lane) - 1u))] = pc;
      np = __popc(lm);
    }
    __syncwarp();
    for (int sub = 0; sub < np; sub += kChainPts) {
      const int t = sub + ps;
      const PointChain pc = pts[t < np ? t : 0];
      const bool live = t < np;
      float2 ox = bc2(0.f), oy = bc2(0.f), oz = bc2(0.f);
      if (live) {
        const int pi = pc.i;
        // entries l and l + 1 as one pair, accumulated into acc[e]
        auto pair = [&](int e, int l, float2 ex, float2 ey, float2 ez, float2 aw, float2 ek, float2 er, int2 kj) {
          float2 dx = __fadd2_rn(ex, pc.npx), dy = __fadd2_rn(ey, pc.npy), dz = __fadd2_rn(ez, pc.npz);
          img.apply2(dx, dy, dz);
          const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
          // atom i's own entry moves with the point: no force from it (its C or
          // gamma is dropped, or in the adjoint, which needs them, the result)
          if (!ADJ) aw = make_float2(kj.x != pi ? aw.x : 0.0f, kj.y != pi ? aw.y : 0.0f);
          float2 f, hx, hy, hz;  // the pull: f h
          if (MODEL == GBX_MODEL_GBMV1) {
            const float2 r4 = __fmul2_rn(r2, r2);
            const float2 g = __fmul2_rn(aw, r4);
            const float2 ex2 = make_float2(__expf(g.x), __expf(g.y));
            if (ADJ) {
              const float2 dr = __fmul2_rn(__fmul2_rn(__fmul2_rn(bc2(pc.cS), ex2), r4), ek);  // padding: 0
              accR[e] = __fadd2_rn(accR[e], dr);
              if (!sorted) {
                if (l < cnt) add_fixed_one(out, kj.x, 3, dr.x);
                if (l + 1 < cnt) add_fixed_one(out, kj.y, 3, dr.y);
              }
            }
            // dS/d(delta) = 4 gamma e r^2 delta
            f = __fmul2_rn(__fmul2_rn(__fmul2_rn(pc.A, aw), ex2), r2);
            hx = dx;
            hy = dy;
            hz = dz;
          } else {
            const float2 T = __ffma2_rn(bc2(100.0f), r2, ek);
            const float2 rT = rcp2(T);
            const float2 CT = __fmul2_rn(aw, rT);
            const float2 F = __fmul2_rn(CT, CT);
            const float2 W = __ffma2_rn(
                pc.Vx, dx, __ffma2_rn(pc.Vy, dy, __ffma2_rn(pc.Vz, dz, __ffma2_rn(pc.B, __fmul2_rn(F, r2), pc.A))));
            if (ADJ) {
              // dF/dR_j with T = C_j + 100 (r^2 - R_j^2), C_j = 10 p1 R_j + p2 (nm -> A)
              const float2 Tp = __ffma2_rn(bc2(-200.0f), er, bc2(Cp));
              const float2 num = __ffma2_rn(bc2(Cp), T, __fmul2_rn(make_float2(-aw.x, -aw.y), Tp));
              const float2 dFdR = __fmul2_rn(__fmul2_rn(__fmul2_rn(bc2(2.0f), CT), num), __fmul2_rn(rT, rT));
              const float2 dr = __fmul2_rn(dFdR, W);
              accR[e] = __fadd2_rn(accR[e], dr);
              if (!sorted) {
                if (l < cnt) add_fixed_one(out, kj.x, 3, dr.x);
                if (l + 1 < cnt) add_fixed_one(out, kj.y, 3, dr.y);
              }
            }
            const float2 s = __ffma2_rn(__fmul2_rn(bc2(-400.0f), rT), W, __fmul2_rn(pc.B, F));
            f = F;
            hx = __ffma2_rn(s, dx, pc.Vx);
            hy = __ffma2_rn(s, dy, pc.Vy);
            hz = __ffma2_rn(s, dz, pc.Vz);
          }
          if (ADJ) f = make_float2(kj.x != pi ? f.x : 0.0f, kj.y != pi ? f.y : 0.0f);
          if (sorted) {
            acc[e][0] = __ffma2_rn(f, hx, acc[e][0]);
            acc[e][1] = __ffma2_rn(f, hy, acc[e][1]);
            acc[e][2] = __ffma2_rn(f, hz, acc[e][2]);
          } else {
            if (l < cnt && kj.x != pi) add_fixed3(out, kj.x, -f.x * hx.x, -f.x * hy.x, -f.x * hz.x);
            if (l + 1 < cnt && kj.y != pi) add_fixed3(out, kj.y, -f.y * hx.y, -f.y * hy.y, -f.y * hz.y);
          }
          ox = __ffma2_rn(f, hx, ox);
          oy = __ffma2_rn(f, hy, oy);
          oz = __ffma2_rn(f, hz, oz);
        };
#pragma unroll
        for (int e = 0; e < kPairsPerLane; ++e) {
          const int j = es + e * kChainEnt, l = 2 * j;
          if (l < cnt) {
            const ChainPair c = L[j];
            pair(e, l, c.x, c.y, c.z, c.w, c.k, ADJ ? r[j] : bc2(0.f), c.idx);
          }
        }
      }
      // the point's own pull, summed over its entry lanes
      float px_ = ox.x + ox.y, py_ = oy.x + oy.y, pz_ = oz.x + oz.y;
#pragma unroll
      for (int off = 1; off < kChainEnt; off <<= 1) {
        px_ += __shfl_xor_sync(0xffffffffu, px_, off);
        py_ += __shfl_xor_sync(0xffffffffu, py_, off);
        pz_ += __shfl_xor_sync(0xffffffffu, pz_, off);
      }
      if (es == 0 && t < np) sh.own[t] = make_float3(px_, py_, pz_);
    }
    __syncwarp();
    // owner forces of these points: runs of one atom summed, one reduction per run
    {
      float3 o = lane < np ? sh.own[lane] : make_float3(0.f, 0.f, 0.f);
      const int key = lane < np ? pts[lane].i : -1 - lane;
      if (sorted) {
#pragma unroll
        for (int off = 1; off < kWarp; off <<= 1) {
          const float yx = __shfl_up_sync(0xffffffffu, o.x, off);
          const float yy = __shfl_up_sync(0xffffffffu, o.y, off);
          const float yz = __shfl_up_sync(0xffffffffu, o.z, off);
          const int ky = __shfl_up_sync(0xffffffffu, key, off);
          if (lane >= off && ky == key) {
            o.x += yx;
            o.y += yy;
            o.z += yz;
          }
        }
        const int kn = __shfl_down_sync(0xffffffffu, key, 1);
        const bool last = lane < np && (lane == np - 1 || kn != key);  // the run's sum
        if (last) add_fixed3(out, key, o.x, o.y, o.z);
      } else if (lane < np) {
        add_fixed3(out, key, o.x, o.y, o.z);
      }
    }
    __syncwarp();
  }
  if (!sorted) return;
  // the entries' pull over all of the cell's points: summed over the point
  // lanes, one fixed-point reduction per entry
#pragma unroll
  for (int e = 0; e < kPairsPerLane; ++e) {
    if (2 * e * kChainEnt >= cnt) break;
#pragma unroll
    for (int off = kChainEnt; off < kWarp; off <<= 1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        acc[e][c].x += __shfl_xor_sync(0xffffffffu, acc[e][c].x, off);
        acc[e][c].y += __shfl_xor_sync(0xffffffffu, acc[e][c].y, off);
      }
      if (ADJ) {
        accR[e].x += __shfl_xor_sync(0xffffffffu, accR[e].x, off);
        accR[e].y += __shfl_xor_sync(0xffffffffu, accR[e].y, off);
      }
    }
    // lane (ps, es) pushes component ps of the pair's entries: an atom's
    // components leave as neighbouring fields of its sector in one instruction
    const int l = 2 * (es + e * kChainEnt);
    const float2 sum = ps == 0 ? acc[e][0] : ps == 1 ? acc[e][1] : ps == 2 ? acc[e][2] : accR[e];
    if (ps < 3 || ADJ) {
      const float sign = ps < 3 ? -1.0f : 1.0f;
      const int2 k = L[es + e * kChainEnt].idx;
      if (l < cnt) add_fixed_one(out, k.x, ps, sign * sum.x);
      if (l + 1 < cnt) add_fixed_one(out, k.y, ps, sign * sum.y);
    }
  }
}

// SPARSE: a grid of fewer blocks than cells, each warp taking every so manieth
// cell.  A block costs its launch, half a nanosecond of the whole pass, also for
// a cell without points; the loop costs registers (72 to 128 bytes of spills
// where one cell takes 8 to 24).  A molecule in a wide box has mostly empty
// cells: chain rule with a block per cell and with the loop, 300 atoms in 10 nm
// (1,048 cells an atom) 205 and 35 us, 2,000 atoms in 30 nm (4,060) 5,114 and
// 121.  The line, in allocated cells (a quarter more than the box has), 24 x 26
// points, per atom: GBMV-II 10,000 atoms 18 238 and 242, 33 297 and 293, 52 371
// and 252, 2,513 atoms 30 72 and 88, 52 96 and 92, 1,000 atoms 74 49 and 49;
// GBMV-I 10,000 atoms 33 311 and 346, 52 385 and 303.  4,096 to 65,536 blocks:
// the same within a tenth at those sizes, more for 40 atoms (39 us with 65,536, 27
// with 32,768).
constexpr long long kSparseCells = 40;     // allocated cells per atom above which the loop is taken,
constexpr long long kSparseFrom = 65536;   // and in all (41,000 of 1,000 atoms: 41 and 47 us)
constexpr long long kSparseBlocks = 32768; // its grid
template <int MODEL, bool PER, bool ADJ, bool SPARSE>
__global__ void __launch_bounds__(kChainWarps* kWarp, ADJ ? 24 : MODEL == GBX_MODEL_GBMV2 ? 28 : 32)
    gbmv_cell_chain_kernel(const float4* __restrict__ pos, Entries tab, Quad quad, ModelConst m, CellPoints cp,
                           const float2* __restrict__ dEdJ, CellChainOut out) {
  __shared__ ChainShared s_sh[kChainWarps];
  __shared__ float2 s_r[ADJ ? kChainWarps : 1][ADJ ? kMaxList / 2 : 1];
  const int w = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const long long warp = (long long)blockIdx.x * kChainWarps + w;
  const long long ncell = min(tab.geom->ncell, tab.cell_cap);
  if constexpr (!SPARSE) {
    if (warp >= ncell) return;
    const int binned = cp.count[warp];
    if (binned == 0) return;
    const int P = cp.live[warp];
    if (P == 0) return;
    chain_cell<MODEL, PER, ADJ>(pos, tab, quad, m, cp, dEdJ, out, warp, binned, P, lane, s_sh[w], s_r[ADJ ? w : 0]);
  } else {
    // a lane looks at a cell; the warp then does those with points one by one
    const long long warps = (long long)gridDim.x * kChainWarps;
    for (long long first = warp; first < ncell; first += kWarp * warps) {
      const long long mine = first + lane * warps;
      int binned = 0, P = 0;
      if (mine < ncell) binned = cp.count[mine];
      if (binned > 0) P = cp.live[mine];
      for (unsigned todo = __ballot_sync(0xffffffffu, P > 0); todo != 0u; todo &= todo - 1u) {
        const int from = __ffs((int)todo) - 1;
        chain_cell<MODEL, PER, ADJ>(pos, tab, quad, m, cp, dEdJ, out, first + from * warps,
                                    __shfl_sync(0xffffffffu, binned, from), __shfl_sync(0xffffffffu, P, from), lane,
                                    s_sh[w], s_r[ADJ ? w : 0]);
        __syncwarp();  // the next cell takes the same buffers
      }
    }
  }
}

}  // namespace

// The cell passes apply to the GBMV models on a table capped at kMaxList.
bool gbmv_cells_apply(const Context* ctx) {
  const gbx_config& c = ctx->cfg;
  return c.model != GBX_MODEL_GBSW && c.table_cap >= 1 && c.table_cap <= kMaxList && ctx->d_pat != nullptr &&
         ctx->d_pcount != nullptr &&
         (long long)ctx->n * (c.n_radial * c.lebedev_order) < 0x7fffffffLL;
}

namespace {
Entries gbmv_entries(const Context* ctx) {
  return Entries{ctx->d_geom, ctx->d_cell2, ctx->d_entry4, ctx->d_entry_par, ctx->d_entries, ctx->cell_cap, nullptr,
                 ctx->entry_cap};
}
}  // namespace

gbx_status launch_gbmv_cells_bin(Context* ctx, const float4* pos, const ModelConst& m) {
  cudaStream_t st = ctx->stream;
  const Entries t = gbmv_entries(ctx);
  const Quad qd{ctx->d_qv, ctx->d_qw, ctx->d_qoff};
  const int chunk = (m.nq + ctx->n_chunks - 1) / ctx->n_chunks;
  const long long npts = (long long)ctx->n * m.nq;
  const CellPoints cp{ctx->d_pcount, ctx->d_plive, ctx->d_pstart, ctx->d_porder, ctx->d_pat,
                      ctx->d_sval,   ctx->d_pstate, (size_t)npts};
  const long long warps = (long long)ctx->n * ctx->n_chunks;
  const int bin_blocks = (int)((warps * kWarp + kBinThreads - 1) / kBinThreads);
  const long long cells = ctx->cell_cap;
  const bool box = m.table_mode == GBX_TABLE_PERIODIC;  // a point's cell does not depend on minimum images
  if (m.model == GBX_MODEL_GBMV1) {
    if (box) gbmv_bin_kernel<GBX_MODEL_GBMV1, BoxQuery><<<bin_blocks, kBinThreads, 0, st>>>(pos, ctx->n, t, qd, m, chunk, ctx->n_chunks, cp);
    else gbmv_bin_kernel<GBX_MODEL_GBMV1, RefQuery><<<bin_blocks, kBinThreads, 0, st>>>(pos, ctx->n, t, qd, m, chunk, ctx->n_chunks, cp);
  } else {
    if (box) gbmv_bin_kernel<GBX_MODEL_GBMV2, BoxQuery><<<bin_blocks, kBinThreads, 0, st>>>(pos, ctx->n, t, qd, m, chunk, ctx->n_chunks, cp);
    else gbmv_bin_kernel<GBX_MODEL_GBMV2, RefQuery><<<bin_blocks, kBinThreads, 0, st>>>(pos, ctx->n, t, qd, m, chunk, ctx->n_chunks, cp);
  }
  launch_scan(ctx->d_pcount, ctx->d_geom, ctx->d_pstart, cells, 0x7fffffffffffLL, ctx->d_ptotal, nullptr, 0,
              ctx->d_status, st);
  constexpr int per_block = kFillLoads * kFillThreads;
  gbmv_fill_kernel<<<(int)((npts + per_block - 1) / per_block), kFillThreads, 0, st>>>(npts, cp);
  ctx->launches += 3;  // bin, scan, fill
  return GBX_OK;
}

gbx_status launch_gbmv_cells_integral(Context* ctx, const float4* pos, const ModelConst& m) {
  cudaStream_t st = ctx->stream;
  const Entries t = gbmv_entries(ctx);
  const Quad qd{ctx->d_qv, ctx->d_qw, ctx->d_qoff};
  const int chunk = (m.nq + ctx->n_chunks - 1) / ctx->n_chunks;
  const long long npts = (long long)ctx->n * m.nq;
  const CellPoints cp{ctx->d_pcount, ctx->d_plive, ctx->d_pstart, ctx->d_porder, ctx->d_pat,
                      ctx->d_sval,   ctx->d_pstate, (size_t)npts};
  const long long warps = (long long)ctx->n * ctx->n_chunks;
  const int bin_blocks = (int)((warps * kWarp + kBinThreads - 1) / kBinThreads);
  const int cell_blocks = (int)((ctx->cell_cap + kCellWarps - 1) / kCellWarps);
  const bool per = ctx->cfg.periodic != 0;
  if (m.model == GBX_MODEL_GBMV1) {
    if (per) gbmv_cell_integral_kernel<GBX_MODEL_GBMV1, true><<<cell_blocks, kCellThreads, 0, st>>>(pos, t, qd, m, cp);
    else gbmv_cell_integral_kernel<GBX_MODEL_GBMV1, false><<<cell_blocks, kCellThreads, 0, st>>>(pos, t, qd, m, cp);
  } else {
    if (per) gbmv_cell_integral_kernel<GBX_MODEL_GBMV2, true><<<cell_blocks, kCellThreads, 0, st>>>(pos, t, qd, m, cp);
    else gbmv_cell_integral_kernel<GBX_MODEL_GBMV2, false><<<cell_blocks, kCellThreads, 0, st>>>(pos, t, qd, m, cp);
  }
  gbmv_reduce_kernel<<<bin_blocks, kBinThreads, 0, st>>>(ctx->n, qd, m.nq, chunk, ctx->n_chunks, ctx->d_sval,
                                                         ctx->d_J);
  ctx->launches += 2;  // integral, reduce
  return GBX_OK;
}

gbx_status launch_gbmv_cells_chain(Context* ctx, const float4* pos, const ModelConst& m, bool adjoint) {
  cudaStream_t st = ctx->stream;
  const Entries t = gbmv_entries(ctx);
  const Quad qd{ctx->d_qv, ctx->d_qw, ctx->d_qoff};
  const long long npts = (long long)ctx->n * m.nq;
  const CellPoints cp{ctx->d_pcount, ctx->d_plive, ctx->d_pstart, ctx->d_porder, ctx->d_pat,
                      ctx->d_sval,   ctx->d_pstate, (size_t)npts};
  const CellChainOut o{ctx->d_f4};
  const long long cell_blocks = (ctx->cell_cap + kChainWarps - 1) / kChainWarps;
  const bool sparse = ctx->cell_cap > kSparseFrom && ctx->cell_cap > kSparseCells * ctx->n;
  const bool per = ctx->cfg.periodic != 0;
  void (*kernel)(const float4*, Entries, Quad, ModelConst, CellPoints, const float2*, CellChainOut);
  switch ((m.model == GBX_MODEL_GBMV1 ? 0 : 8) + (per ? 4 : 0) + (adjoint ? 2 : 0) + (sparse ? 1 : 0)) {
    case 0: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, false, false, false>; break;
    case 1: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, false, false, true>; break;
    case 2: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, false, true, false>; break;
    case 3: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, false, true, true>; break;
    case 4: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, true, false, false>; break;
    case 5: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, true, false, true>; break;
    case 6: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, true, true, false>; break;
    case 7: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV1, true, true, true>; break;
    case 8: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, false, false, false>; break;
    case 9: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, false, false, true>; break;
    case 10: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, false, true, false>; break;
    case 11: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, false, true, true>; break;
    case 12: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, true, false, false>; break;
    case 13: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, true, false, true>; break;
    case 14: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, true, true, false>; break;
    default: kernel = gbmv_cell_chain_kernel<GBX_MODEL_GBMV2, true, true, true>; break;
  }
  kernel<<<(int)(sparse ? kSparseBlocks : cell_blocks), kChainWarps * kWarp, 0, st>>>(pos, t, qd, m, cp, ctx->d_dEdJ, o);
  ++ctx->launches;
  return GBX_OK;
}

}  // namespace gbx
