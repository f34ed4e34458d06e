// Born-radius integrals and the chain rule through every quadrature point.
//
// Work decomposition: one warp = one atom i x one chunk of quadrature
// points.  GBSW integrals: points classified 128 at a time, those with lists
// queued and walked 32 in step, a lane each; the GBSW chain rule: lanes over
// the shaping entries of recorded points (or of points whose lists it walks);
// GBMV integrals: two lanes per point; the GBMV chain rule: the warp on one
// point at a time, lanes over its list.  The atom is warp-uniform, every per-atom sum is a fixed-shape
// warp reduction (bit-reproducible), the quadrature data is read coalesced,
// and lists are stored inline (x, y, z, model parameter) so there is no
// dependent index -> position gather.
//
// Integrals.  The reference accumulates I_n = sum_q w_q/r_q^(n-2) * (1 - V_q)
// (GBSWIntegral.cpp:142-146) and then forms 1/r0 - I4 and 1/(4 r0^4) - I7,
// which cancel to a few significant digits -- fatal in FP32.  The kernels
// accumulate the complement J_n = sum_q w_q/r_q^(n-2) * s_q, with s_q the
// solvent fraction (GBSW: V_q; GBMV: 1 - V_q = p/(1+p)), all terms >= 0; the
// host supplies the FP64 constants S_n = sum_q w_q/r_q^(n-2), so that
// I_n = S_n - J_n and 1/r0 - I4 = (1/r0 - S4) + J4 without cancellation.
//
// Tables.  GBMV and the integral-class GBSW read the reference's own table,
// whose list contents define the result: the point's cell is computed in
// FP32 and redone in FP64 exactly as the reference does
// (CharmmReferenceGBSW.cpp:539-549, CustomGBIntegral.cpp:284-324) whenever
// the FP32 coordinate lies within a guard band of a cell face.  The
// standalone GBSW model reads the exact table of k_tight.cu instead, in a
// periodic box at the place that the reference moves the point to, with
// minimum-image distances; only a box too narrow for that, or a caller's wish,
// keeps the reference table there, through a query that wraps as the reference
// does.
#include <math.h>

#include <type_traits>

#include "gbx_internal.cuh"
#include "queries.cuh"

namespace gbx {
namespace {

constexpr int kThreads = 128;

// Work counters for roofline accounting: compiled out unless requested.
template <bool ON>
struct Work {
  __device__ __forceinline__ void eval() {}
  __device__ __forceinline__ void shell() {}
};
template <>
struct Work<true> {
  unsigned long long e = 0, s = 0;    // the volume pass: list walk with the first-burying-atom exit
  unsigned long long fe = 0, fs = 0;  // the chain pass: every listed atom of every point
  __device__ __forceinline__ void eval() { ++e; }
  __device__ __forceinline__ void shell() { ++s; }
};

// ---------------------------------------------------------------------------
// Volume models on inline entries.  d = x_j - p comes from the query's
// delta(): (x_j - x_i) - v, so the FP32 difference of nearby atoms is exact,
// and in a periodic system its minimum image.
// ---------------------------------------------------------------------------

// Entry `at` of a list as work counting walks it: a reference table's in the
// reference's order (ascending atoms), the exact table's in its own.
__device__ __forceinline__ float4 counted_entry(const Entries& t, int at) {
  return t.first ? entry_at(t, at) : __ldg(t.e + __ldg(t.index + at));
}

// GBSW, CharmmReferenceGBSW.cpp:616-639 / GBSWIntegral.cpp:187-224: V is the
// product of u_j over the switching shells, 0 once an atom buries the point.
template <class Q, class W>
__device__ __forceinline__ float gbsw_volume(const Q& qy, const ModelConst& m, const Entries& t, int start,
                                             int cnt, const float4 xi, const float4 v, W& wk) {
  float V = 1.0f;
  for (int l = 0; l < cnt; ++l) {
    const float4 a = counted_entry(t, start + l);
    const float3 d = qy.delta(a, xi, v);
    const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
    const float lo = a.w - m.sw, hi = a.w + m.sw;
    wk.eval();
    if (r2 <= lo * lo) return 0.0f;
    if (r2 < hi * hi) {
      wk.shell();
      const float dr = r2 * rsqrtf(r2) - a.w;
      V *= fmaf(dr, fmaf(-m.c3 * dr, dr, m.c1), 0.5f);
    }
  }
  return V;
}

// GBMV-I, GBMVIntegralTypeI.cpp:155-173: S = sum_j exp(gamma_j r^4).
template <class Q, class W>
__device__ __forceinline__ float gbmv1_sum(const Q& qy, const float4* __restrict__ list, int cnt, const float4 xi,
                                           const float4 v, W& wk) {
  float S = 0.0f;
  for (int l = 0; l < cnt; ++l) {
    const float4 a = __ldg(list + l);
    const float3 d = qy.delta(a, xi, v);
    const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
    S += __expf(a.w * (r2 * r2));
    wk.eval();
  }
  return S;
}

struct Gbmv2State {
  float s1, s2, vx, vy, vz;
};

// GBMV-II, GBMVIntegralTypeII.cpp:163-191:
// F_j = (C_j / (C_j + 100 r^2 - 100 R_j^2))^2, sums of F, r^2 F^2 and F d.
template <class Q, class W>
__device__ __forceinline__ Gbmv2State gbmv2_sums(const Q& qy, const float4* __restrict__ list,
                                                 const float2* __restrict__ par,
                                                 int cnt, const float4 xi, const float4 v, W& wk) {
  Gbmv2State s{0.f, 0.f, 0.f, 0.f, 0.f};
  for (int l = 0; l < cnt; ++l) {
    const float4 a = __ldg(list + l);
    const float K = __ldg(&par[l].x);
    const float3 d = qy.delta(a, xi, v);
    const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
    float F = __fdividef(a.w, fmaf(100.0f, r2, K));
    F = F * F;
    s.s1 += F;
    s.s2 = fmaf(r2, F * F, s.s2);
    s.vx = fmaf(d.x, F, s.vx);
    s.vy = fmaf(d.y, F, s.vy);
    s.vz = fmaf(d.z, F, s.vz);
    wk.eval();
  }
  return s;
}

__device__ __forceinline__ float gbmv2_S(const ModelConst& m, const Gbmv2State& s) {
  const float s3sq = fmaf(s.vx, s.vx, fmaf(s.vy, s.vy, s.vz * s.vz));
  return m.s0 * s.s1 * s.s2 / s3sq;
}

// Chain-pass work of one point, counted only for roofline accounting: the
// reference chain kernel (reduceIntegralForce.cu:45-65) visits the whole cell
// list of every point, with the derivative work inside the switching shell.
template <int MODEL, class Q>
__device__ __forceinline__ void count_chain_work(const Q& qy, const ModelConst& m, const Entries& t, long long cell,
                                                 const float4 xi, const float4 v, Work<true>& wk) {
  if (cell < 0) return;
  const int2 cs = __ldg(t.cell + cell);
  if (cs.x <= 0) return;
  wk.fe += cs.x;
  if constexpr (MODEL != GBX_MODEL_GBSW) {
    wk.fs += cs.x;
  } else {
    for (int l = 0; l < cs.x; ++l) {
      const float4 a = counted_entry(t, cs.y + l);
      const float3 d = qy.delta(a, xi, v);
      const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
      const float lo = a.w - m.sw, hi = a.w + m.sw;
      wk.fs += (r2 > lo * lo && r2 < hi * hi) ? 1 : 0;
    }
  }
}

template <int MODEL, class Q, class W>
__device__ __forceinline__ float solvent_fraction(const Q& qy, const ModelConst& m, const Entries& t, long long cell,
                                                  const float4 xi, const float4 v, W& wk) {
  int cnt = 0, s = 0;
  if (cell >= 0) {
    const int2 cs = __ldg(t.cell + cell);
    cnt = cs.x;
    if (cnt < 0) return 0.0f;  // buried cell (exact table)
    s = cs.y;
  }
  if (MODEL == GBX_MODEL_GBSW) return cnt > 0 ? gbsw_volume(qy, m, t, s, cnt, xi, v, wk) : 1.0f;
  float p;
  if (MODEL == GBX_MODEL_GBMV1) return logistic_solvent(m.beta, m.lambda, gbmv1_sum(qy, t.e + s, cnt, xi, v, wk), p);
  if (cnt == 0) return 1.0f;  // empty list: V = 0 (GBMVIntegralTypeII.cpp:140)
  return logistic_solvent(m.beta, m.lambda, gbmv2_S(m, gbmv2_sums(qy, t.e + s, t.par + s, cnt, xi, v, wk)), p);
}

// ---------------------------------------------------------------------------
// Integral kernel: J4 = sum w/r^2 s, J7 = sum w/r^5 s per (atom, chunk).
// ---------------------------------------------------------------------------
// GBMV point state kept for the chain rule (saves it re-summing every list):
// GBMV-I S at state[i Q + q]; GBMV-II s1, s2, vx, vy, vz in five planes of N Q.
template <int MODEL, class Q, class W>
__device__ __forceinline__ float gbmv_fraction_keep(const Q& qy, const ModelConst& m, const Entries& t, long long cell,
                                                    const float4 xi, const float4 v, W& wk, float* state,
                                                    size_t idx, size_t plane) {
  int cnt = 0, s = 0;
  if (cell >= 0) {
    const int2 cs = __ldg(t.cell + cell);
    cnt = cs.x;
    s = cs.y;
  }
  float p;
  if constexpr (MODEL == GBX_MODEL_GBMV1) {
    const float S = gbmv1_sum(qy, t.e + s, cnt, xi, v, wk);
    state[idx] = S;
    return logistic_solvent(m.beta, m.lambda, S, p);
  } else {
    if (cnt == 0) return 1.0f;  // empty list: V = 0 (GBMVIntegralTypeII.cpp:140)
    const Gbmv2State st = gbmv2_sums(qy, t.e + s, t.par + s, cnt, xi, v, wk);
    state[idx] = st.s1;
    state[idx + plane] = st.s2;
    state[idx + 2 * plane] = st.vx;
    state[idx + 3 * plane] = st.vy;
    state[idx + 4 * plane] = st.vz;
    return logistic_solvent(m.beta, m.lambda, gbmv2_S(m, st), p);
  }
}

template <int MODEL, class Q, bool COUNT>
__global__ void __launch_bounds__(kThreads) integral_kernel(const float4* __restrict__ pos, int n, Entries tab,
                                                            Quad quad, ModelConst m, int chunk, int n_chunks,
                                                            float* __restrict__ Jpart,
                                                            unsigned long long* __restrict__ work,
                                                            float* __restrict__ state) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp;
  if (warp >= n * n_chunks) return;
  const int i = warp % n, c = warp / n;
  const float4 xi = pos[i];
  Q query;
  query.init(tab, xi, quad.qoff);
  const int q0 = c * chunk, q1 = min(m.nq, q0 + chunk);
  float J4 = 0.0f, J7 = 0.0f;
  Work<COUNT> wk;
  for (int q = q0 + lane; q < q1; q += kWarp) {
    const float4 v = quad.qv[q];
    const float2 w = quad.qw[q];
    const long long cell = query.cell(xi, v, q);
    float s;
    if constexpr (MODEL != GBX_MODEL_GBSW)
      s = state ? gbmv_fraction_keep<MODEL>(query, m, tab, cell, xi, v, wk, state, (size_t)i * m.nq + q, (size_t)n * m.nq)
                : solvent_fraction<MODEL>(query, m, tab, cell, xi, v, wk);
    else
      s = solvent_fraction<MODEL>(query, m, tab, cell, xi, v, wk);
    if constexpr (COUNT) count_chain_work<MODEL>(query, m, tab, cell, xi, v, wk);
    J4 = fmaf(w.x, s, J4);
    J7 = fmaf(w.y, s, J7);
  }
  for (int off = 16; off > 0; off >>= 1) {
    J4 += __shfl_xor_sync(0xffffffffu, J4, off);
    J7 += __shfl_xor_sync(0xffffffffu, J7, off);
  }
  if (lane == 0) {
    Jpart[(size_t)c * n + i] = J4;
    Jpart[((size_t)n_chunks + c) * n + i] = J7;
  }
  if constexpr (COUNT) {
    unsigned long long e = wk.e, sh = wk.s, fe = wk.fe, fs = wk.fs;
    for (int off = 16; off > 0; off >>= 1) {
      e += __shfl_xor_sync(0xffffffffu, e, off);
      sh += __shfl_xor_sync(0xffffffffu, sh, off);
      fe += __shfl_xor_sync(0xffffffffu, fe, off);
      fs += __shfl_xor_sync(0xffffffffu, fs, off);
    }
    if (lane == 0) {
      atomicAdd(&work[0], e);
      atomicAdd(&work[1], sh);
      atomicAdd(&work[2], fe);
      atomicAdd(&work[3], fs);
    }
  }
}

// GBMV integrals with kGroup lanes per point: the group reads consecutive
// entries of the point's list (kGroup x 16 contiguous bytes per load instead
// of one line per lane), each lane sums every kGroup-th entry and the group
// combines its partial sums by shuffles in a fixed order.  The point's sums
// are kept for the chain rule as in integral_kernel.  Two lanes per point
// measured fastest (GBMV-II, 10k atoms: 1.27 ms against 1.64 ms for one lane,
// 1.47 ms for four and 2.0 ms for eight).
constexpr int kGroup = 2;

template <int MODEL, class Q>
__global__ void __launch_bounds__(kThreads) gbmv_integral_kernel(const float4* __restrict__ pos, int n, Entries tab,
                                                                 Quad quad, ModelConst m, int chunk, int n_chunks,
                                                                 float* __restrict__ Jpart, float* __restrict__ state) {
  constexpr int kPer = kWarp / kGroup;  // points per warp step
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp;
  if (warp >= n * n_chunks) return;
  const int i = warp % n, c = warp / n;
  const int g = lane / kGroup, r = lane % kGroup;
  const float4 xi = pos[i];
  Q query;
  query.init(tab, xi, quad.qoff);
  const int q0 = c * chunk, q1 = min(m.nq, q0 + chunk);
  const size_t plane = (size_t)n * m.nq;
  float J4 = 0.0f, J7 = 0.0f;
  for (int base = q0; base < q1; base += kPer) {
    const int q = base + g;
    int cnt = 0, s = 0;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q < q1) {
      v = quad.qv[q];
      const long long cell = query.cell(xi, v, q);
      if (cell >= 0) {
        const int2 cs = __ldg(tab.cell + cell);
        cnt = cs.x;
        s = cs.y;
      }
    }
    float S1 = 0.f, S2 = 0.f, Vx = 0.f, Vy = 0.f, Vz = 0.f;
    for (int l = r; l < cnt; l += kGroup) {
      const float4 a = __ldg(tab.e + s + l);
      const float3 d = query.delta(a, xi, v);
      const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
      if constexpr (MODEL == GBX_MODEL_GBMV1) {
        S1 += __expf(a.w * (r2 * r2));
      } else {
        float F = __fdividef(a.w, fmaf(100.0f, r2, __ldg(&tab.par[s + l].x)));
        F = F * F;
        S1 += F;
        S2 = fmaf(r2, F * F, S2);
        Vx = fmaf(d.x, F, Vx);
        Vy = fmaf(d.y, F, Vy);
        Vz = fmaf(d.z, F, Vz);
      }
    }
#pragma unroll
    for (int off = 1; off < kGroup; off <<= 1) {
      S1 += __shfl_xor_sync(0xffffffffu, S1, off);
      if constexpr (MODEL != GBX_MODEL_GBMV1) {
        S2 += __shfl_xor_sync(0xffffffffu, S2, off);
        Vx += __shfl_xor_sync(0xffffffffu, Vx, off);
        Vy += __shfl_xor_sync(0xffffffffu, Vy, off);
        Vz += __shfl_xor_sync(0xffffffffu, Vz, off);
      }
    }
    if (r == 0 && q < q1) {
      const size_t idx = (size_t)i * m.nq + q;
      float p, sf;
      if constexpr (MODEL == GBX_MODEL_GBMV1) {
        if (state) state[idx] = S1;
        sf = logistic_solvent(m.beta, m.lambda, S1, p);
      } else if (cnt == 0) {
        sf = 1.0f;  // empty list: V = 0 (GBMVIntegralTypeII.cpp:140)
      } else {
        const Gbmv2State st{S1, S2, Vx, Vy, Vz};
        if (state) {
          state[idx] = st.s1;
          state[idx + plane] = st.s2;
          state[idx + 2 * plane] = st.vx;
          state[idx + 3 * plane] = st.vy;
          state[idx + 4 * plane] = st.vz;
        }
        sf = logistic_solvent(m.beta, m.lambda, gbmv2_S(m, st), p);
      }
      const float2 w = quad.qw[q];
      J4 = fmaf(w.x, sf, J4);
      J7 = fmaf(w.y, sf, J7);
    }
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

// ---------------------------------------------------------------------------
// GBSW integral pass that also records which points the chain rule needs:
// (q, V, mask) for every point with V > 0 shaped by an atom other than i,
// bit l of mask set for each such in-shell list entry l.  The chain rule
// then visits only those entries, with lanes spread over them.  Warp w owns
// records [w R, (w + 1) R), filled in the order points finish; count[w] =
// points recorded, or -1 - needed when they did not fit or a list was longer
// than 64 (the chain rule walks that warp's lists instead).  Records are
// stored evict-first: they are read once, and the lookup table must stay in
// L2.
// ---------------------------------------------------------------------------
struct ShellSink {
  int4* rec;
  int* st;             // the point's list start, beside each record
  int* count;          // [warps]
  unsigned* max_seen;  // largest per-warp need of this call
  int R;               // records per warp
};

__device__ __forceinline__ float shell_g(const ModelConst& m, float V, float dr) {
  const float u = fmaf(dr, fmaf(-m.c3 * dr, dr, m.c1), 0.5f);
  const float du = fmaf(-3.0f * m.c3 * dr, dr, m.c1);
  return __fdividef(V, u) * du;
}

// Signed distance of a point from an atom's sphere, |d| - R'.  A point at an
// atom's own place gives -R' (the tiny term keeps 0 * rsqrt(0) out; it is far
// below the rounding of any other squared distance).
__device__ __forceinline__ float sphere_gap(const float3 d, float Rp) {
  const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, fmaf(d.z, d.z, 1e-30f)));
  return fmaf(r2, rsqrt_ftz(r2), -Rp);
}

// The quadrature points of one (atom, chunk) item.  Radial points well inside
// atom i's own burying sphere (r below R'_i - w by more than FP32 rounding of
// |v|^2 can reach) have V = 0: the exact table lists atom i in every cell they
// fall in, so the walk would end on it at the latest.  V = 0 adds nothing to J
// and records nothing, so the leading `inner` points of every direction are
// left out; the rest, numbered t over all directions, are split into chunks.
struct Points {
  int t0, t1, inner;
  unsigned magic;  // 2^24 / (points kept per direction), rounded up
  template <class Q>
  __device__ __forceinline__ void init(const Quad& quad, const ModelConst& m, const float4 xi, int c, int n_chunks,
                                       int lane) {
    inner = 0;
    if constexpr (IsTight<Q>::value) {
      const float lo = xi.w - m.sw;
      for (int r0 = 0; r0 < m.nrad; r0 += kWarp) {
        const int ir = r0 + lane;
        const bool in = ir < m.nrad && quad.qv[ir].w * (1.0f + 1.0f / 1024.0f) < lo;
        const unsigned out = __ballot_sync(0xffffffffu, !in);
        inner = r0 + (out ? __ffs(out) - 1 : kWarp);
        if (out) break;
      }
      inner = min(inner, m.nrad);
    }
    const int kept = m.nrad - inner;
    const int total = m.nq / m.nrad * kept, chunk = (total + n_chunks - 1) / n_chunks;
    magic = kept > 0 ? ((1u << 24) + kept - 1) / kept : 0u;
    t0 = min(total, c * chunk);
    t1 = min(total, t0 + chunk);
  }
  // the index of point t: exact for the at most 28,160 points of a rule (256 x 110)
  __device__ __forceinline__ int q(int t) const { return t + inner * ((int)__umulhi((unsigned)t << 8, magic) + 1); }
};

// Whether the point lies in atom i's own switching shell.  Without images its
// distance from atom i is |v| (the radial point, to FP32 rounding).
template <class Q>
__device__ __forceinline__ bool in_own_shell(const Q& query, const ModelConst& m, const float4 xi, const float4 v) {
  if (!Q::kImages && fabsf(v.w - xi.w) >= m.sw + 1e-5f) return false;
  return fabsf(sphere_gap(query.delta(xi, xi, v), xi.w)) < m.sw;
}

// GBSW integrals.  A warp classifies kRefill points at a time (empty cell:
// V = 1; buried cell or buried by the list's first entry: V = 0) and queues
// the points that have a list.  Whenever 32 points are pending, the warp walks
// their lists in step, one lane per point, two entries per step: the list
// position is then the same for every lane, so a step is straight-line code
// (no refill, dequeue or record bookkeeping inside the walk: that is paid
// once per 32 points).  Lanes idle from the end of their list to the end of
// the longest, so short and long lists are queued apart.  The walk per point
// is the sequential one of gbsw_volume (same order).  J is summed in an order
// fixed by the input alone, so runs are bit-reproducible.
constexpr int kRefill = 128;       // points classified per refill
constexpr int kQueue = kRefill + kWarp;  // fewer than 32 pending when a refill starts
constexpr int kShortList = 8;      // longest list of the short queue
// What the integral pass records: nothing; the points an atom other than i
// shapes, with those atoms; every shaped point with all its shaping atoms (the
// adjoint, whose dE/dR_i has atom i's own entry).
enum { kEmitNone = 0, kEmitOthers = 1, kEmitAll = 2 };

// Persistent: a grid of resident blocks whose warps take (atom, chunk) items
// from `next_item` one at a time, so a warp that finishes a cheap item (a
// buried or exposed atom) takes the next instead of idling until the slowest
// warp of its block is done.  Each item's results depend on the item alone.
// `order` (or nullptr): the atoms in the order to take them in.
template <class Q, int EMIT>
__global__ void __launch_bounds__(kThreads, 12) gbsw_integral_kernel(const float4* __restrict__ pos, int n, Entries tab,
                                                                 Quad quad, ModelConst m, int n_chunks,
                                                                 float* __restrict__ Jpart, ShellSink sink,
                                                                 unsigned* __restrict__ next_item,
                                                                 const int* __restrict__ order) {
  __shared__ int2 s_queue[kThreads / kWarp][2][kQueue];  // (q | length << 16, list start): short and long lists
  // lists start at even entries and each cell's record sits beside its first
  // entry, so both are read 32 bytes at a time
  const int lane = threadIdx.x % kWarp;
  const int wib = threadIdx.x / kWarp;
  const unsigned lt = (1u << lane) - 1u;
  for (;;) {
    unsigned item = 0;
    if (lane == 0) item = atomicAdd(next_item, 1u);
    const int warp = (int)__shfl_sync(0xffffffffu, item, 0);
    if (warp >= n * n_chunks) return;
    int fill = 0;           // warp-uniform: points recorded so far (may exceed R)
    bool too_long = false;  // a shaping entry beyond list position 63
    const int c = warp / n, k = warp - c * n, i = order ? __ldg(order + k) : k;
    const float4 xi = pos[i];
    Q query;
    query.init(tab, xi, quad.qoff);
    Points pts{};
    pts.init<Q>(quad, m, xi, c, n_chunks, lane);
    float J4 = 0.0f, J7 = 0.0f;
    int pending[2] = {0, 0}, head[2] = {0, 0};  // warp-uniform, per queue
    int next = pts.t0;                          // warp-uniform: first point not yet classified
    for (;;) {
      // a full batch of either queue, else more points, else what is left of both
      int take[2] = {0, 0};
      if (pending[0] >= kWarp) {
        take[0] = kWarp;
      } else if (pending[1] >= kWarp) {
        take[1] = kWarp;
      } else if (next < pts.t1) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // what is pending moves to the front
          int2 e = make_int2(0, 0);
          if (lane < pending[h]) e = s_queue[wib][h][head[h] + lane];
          __syncwarp();
          if (lane < pending[h]) s_queue[wib][h][lane] = e;
          head[h] = 0;
        }
#pragma unroll 4
        for (int k = 0; k < kRefill / kWarp; ++k) {
          const int t = next + k * kWarp + lane;
          const int qc = pts.q(t);
          int2 cs = make_int2(-1, 0);
          if (t < pts.t1) {
            const float4 vc = quad.qv[qc];
            const long long cell = query.cell(xi, vc, qc);
            float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f);
            // the cell's first entry beside its record: one load, not one after the other
            cs = make_int2(0, 0);
            if (cell >= 0) {
              const Float4x2 r = ldg_pair(tab.first + cell);
              a0 = r.a;
              cs = make_int2(__float_as_int(r.b.x), __float_as_int(r.b.y));
            }
            if (cs.x == 0) {
              const float2 wc = quad.qw[qc];
              J4 += wc.x;
              J7 += wc.y;
            } else if (cs.x > 0) {
              // the list's first entry, the likeliest burying atom, buries most
              // listed points: V = 0 adds nothing, the point is not queued
              if (sphere_gap(query.delta(a0, xi, vc), a0.w) <= -m.sw) cs.x = -1;
            }
          }
          const unsigned listed = __ballot_sync(0xffffffffu, cs.x > 0);
          const unsigned longer = __ballot_sync(0xffffffffu, cs.x > kShortList);
          const unsigned shorter = listed & ~longer;
          if (cs.x > 0) {
            const bool h = cs.x > kShortList;
            s_queue[wib][h][h ? pending[1] + __popc(longer & lt) : pending[0] + __popc(shorter & lt)] =
                make_int2(qc | cs.x << 16, cs.y);
          }
          pending[0] += __popc(shorter);
          pending[1] += __popc(longer);
        }
        next += kRefill;
        __syncwarp();
        continue;
      } else {
        take[0] = pending[0];
        take[1] = min(pending[1], kWarp - take[0]);
        if (take[0] + take[1] == 0) break;
      }
      // one point per lane
      int q = 0, s = 0, cnt = 0;
      if (lane < take[0] + take[1]) {
        const bool h = lane >= take[0];
        const int2 e = s_queue[wib][h][h ? head[1] + lane - take[0] : head[0] + lane];
        q = e.x & 0xffff;
        cnt = (unsigned)e.x >> 16;
        s = e.y;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        head[h] += take[h];
        pending[h] -= take[h];
      }
      const bool mine = cnt > 0;
      const float4 v = quad.qv[q];
      float V = mine ? 1.0f : 0.0f;
      unsigned sm_lo = 0u, sm_hi = 0u;  // bit l of (hi:lo): entry l shapes the point
      bool far = false;                 // a shaping entry beyond position 63
      EntryPair pair{};
      auto load = [&](int l) -> EntryPair {
        EntryPair p = pair;
        if (l < cnt) p = ldg_entries(tab.e, s + l);  // an odd list ends in a padding entry no point is near
        return p;
      };
      // entries l and l + 1 of every lane that has them, in packed FP32x2
      // arithmetic (each half rounded as sphere_gap rounds it); bits of the shaping ones
      auto step = [&](const EntryPair& p, int l) -> unsigned {
        const bool on = l < cnt;
        const float2 dx = query.delta2(0, p.x, xi.x, v.x), dy = query.delta2(1, p.y, xi.y, v.y),
                     dz = query.delta2(2, p.z, xi.z, v.z);
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, make_float2(1e-30f, 1e-30f))));
        const float2 g = __ffma2_rn(r2, make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y)), p.nw);
        const float2 u = __ffma2_rn(
            g, __ffma2_rn(__fmul2_rn(make_float2(-m.c3, -m.c3), g), g, make_float2(m.c1, m.c1)), make_float2(0.5f, 0.5f));
        const bool ina = on && fabsf(g.x) < m.sw, inb = on && fabsf(g.y) < m.sw;
        if (ina) V *= u.x;
        if (inb) V *= u.y;
        if (on && fminf(g.x, g.y) <= -m.sw) V = 0.0f;  // buried
        return (ina ? 1u : 0u) | (inb ? 2u : 0u);
      };
      // the first kShortList entries without a test between them, the next pair loaded ahead
      pair = load(0);
#pragma unroll
      for (int l = 0; l < kShortList; l += 2) {
        const EntryPair next_pair = load(l + 2);
        sm_lo |= step(pair, l) << l;
        pair = next_pair;
      }
      for (int l = kShortList; __any_sync(0xffffffffu, l < cnt && V != 0.0f); l += 2) {
        const EntryPair next_pair = load(l + 2);
        const unsigned in = step(pair, l);
        if (l < 32) sm_lo |= in << l;
        else if (l < 64) sm_hi |= in << (l - 32);
        else far = in != 0u || far;
        pair = next_pair;
      }
      if (mine) {
        const float2 w = quad.qw[q];
        J4 = fmaf(w.x, V, J4);
        J7 = fmaf(w.y, V, J7);
      }
      if (EMIT != kEmitNone) {
        if (EMIT == kEmitOthers && (sm_lo | sm_hi) != 0u && V != 0.0f && in_own_shell(query, m, xi, v)) {
          // the point lies in atom i's own shell (one radial shell or two of
          // all): its entry, found by its place and index, is not recorded
          for (unsigned lo = sm_lo, hi = sm_hi; (lo | hi) != 0u;) {
            const int l = lo ? __ffs((int)lo) - 1 : 31 + __ffs((int)hi);
            if (__ldg(tab.index + s + l) == i) {
              if (l < 32) sm_lo &= ~(1u << l);
              else sm_hi &= ~(1u << (l - 32));
            }
            if (lo) lo &= lo - 1;
            else hi &= hi - 1;
          }
        }
        // slots in finishing order (the chain rule's sums do not depend on it)
        const bool emit = (sm_lo | sm_hi) != 0u && V != 0.0f;
        const unsigned em = __ballot_sync(0xffffffffu, emit);
        if (emit) {
          const int slot = fill + __popc(em & lt);
          if (slot < sink.R) {
            __stcs(sink.rec + (size_t)warp * sink.R + slot, make_int4(q, __float_as_int(V), (int)sm_lo, (int)sm_hi));
            __stcs(sink.st + (size_t)warp * sink.R + slot, s);
          }
        }
        fill += __popc(em);
        too_long = __any_sync(0xffffffffu, far && V != 0.0f) || too_long;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      J4 += __shfl_xor_sync(0xffffffffu, J4, off);
      J7 += __shfl_xor_sync(0xffffffffu, J7, off);
    }
    if (lane == 0) {
      Jpart[(size_t)c * n + i] = J4;
      Jpart[((size_t)n_chunks + c) * n + i] = J7;
      if (EMIT != kEmitNone) {
        sink.count[warp] = fill <= sink.R && !too_long ? fill : -1 - fill;
        if (fill > 0) atomicMax(sink.max_seen, (unsigned)fill);
      }
    }
    __syncwarp();  // the queues are reused by the next item
  }
}

// ---------------------------------------------------------------------------
// Chain rule: with c = dE/dJ4_i w/r^2 + dE/dJ7_i w/r^5 for a point of atom i,
// F_k -= c ds/dx_k for every atom k shaping the point and F_i gets the
// opposite (the point moves with atom i) -- GBSWIntegral.cpp:271-314,
// GBMVIntegralTypeI.cpp:195-224, GBMVIntegralTypeII.cpp:221-282, and the
// Born-radius prefactor of CharmmReferenceGBSW.cpp:597-611 folded into
// dE/dJ.  With ADJ also dE/dR_k += c ds/dR_k for every shaping atom
// (atom i's own radius included).
// ---------------------------------------------------------------------------
struct ChainOut {
  // the chain rule's own sums, one 32-byte sector per atom: force x, y, z and
  // dE/dR (fixed point); zeroed by the position staging, added to the
  // caller's buffers by the call's last kernel
  unsigned long long* f4;
  bool quirk;  // drop F_k beyond the cutoff (CharmmReferenceGBSW.cpp:291-292)
  float cutoff2;
};

// Records of the emitting integral pass (count == nullptr: none this call).
struct ChainRecords {
  const int4* rec;  // (q, V, mask low, mask high) per recorded point
  const int* st;    // the point's list start
  const int* count;
  int R;
  const int* order;  // the items' atoms, as the integral pass took them (nullptr: ascending)
};

// A component whose fixed-point value is 0 (|g| < 2^-33, common for distant
// GBMV atoms) changes nothing: its reduction is skipped, the result is the
// same bits.
__device__ __forceinline__ void push3(const ChainOut& o, int k, long long fx, long long fy, long long fz) {
  unsigned long long* f = o.f4 + 4 * (size_t)k;
  if (fx) atomicAdd(f, (unsigned long long)fx);
  if (fy) atomicAdd(f + 1, (unsigned long long)fy);
  if (fz) atomicAdd(f + 2, (unsigned long long)fz);
}
__device__ __forceinline__ void push_force(const ChainOut& o, int k, float gx, float gy, float gz) {
  push3(o, k, float_to_fixed_split(-gx), float_to_fixed_split(-gy), float_to_fixed_split(-gz));
}
__device__ __forceinline__ void push_radius(const ChainOut& o, int k, float v) {
  red_add_fixed(o.f4 + 4 * (size_t)k + 3, v);
}

// A shaping atom's share of one GBSW point: c dV/dR_k and the force on k as
// fixed-point integers.  Atom i gets the negated integers, so the pair's
// momentum balances exactly and one conversion serves both.  The record and
// the list-walk paths share it: the same bits.
template <class Q>
struct Shaping {
  float g;  // (V/u) u'
  long long fx, fy, fz;
  bool push;  // false: the cutoff quirk drops the force on k
  __device__ __forceinline__ Shaping(const Q& query, const ModelConst& m, const ChainOut& out, const float4 a,
                                     const float4 xi, const float4 v, float V, float cq) {
    const float3 d = query.delta(a, xi, v);
    const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, fmaf(d.z, d.z, 1e-30f)));
    const float ir = rsqrt_ftz(r2);
    g = shell_g(m, V, fmaf(r2, ir, -a.w));
    const float gs = cq * g * ir;
    fx = float_to_fixed_split(-(gs * d.x));
    fy = float_to_fixed_split(-(gs * d.y));
    fz = float_to_fixed_split(-(gs * d.z));
    push = true;
    if (out.quirk) {
      const float3 e = query.delta(a, xi, make_float4(0.f, 0.f, 0.f, 0.f));  // x_k - x_i
      push = fmaf(e.x, e.x, fmaf(e.y, e.y, e.z * e.z)) <= out.cutoff2;
    }
  }
};

// dE/dJ of an atom: as a kernel before left it, or formed from dE/dB and dB/dJ
// by the warp that needs it (a launch less: 98.6 -> 97.6 us at 1,000 atoms, and
// no difference from 6,000 up).
struct DEdJ {
  const float2* value;  // nullptr: not formed
  const unsigned long long* dEdB_fx;
  const double* dBdJ;   // [2n]
  __device__ __forceinline__ float2 of(int i, int lane) const {
    if (value) return value[i];
    const float part = (float)(fixed_to_double(dEdB_fx[i]) * dBdJ[2 * i + (lane & 1)]);
    return make_float2(__shfl_sync(0xffffffffu, part, 0), __shfl_sync(0xffffffffu, part, 1));
  }
};

// GBSW chain rule over the recorded points: warp = (atom i, quadrature
// chunk).  Each lane takes one record of a batch of 32 and the warp unrolls
// the shaping-entry masks into a ring of (record, list position) items, from
// which 32 items at a time are evaluated, one per lane, whatever the records'
// entry counts; items left over when a batch ends join the next batch's.
//
// The pushes bound this pass: a warp's 32 shaping atoms are scattered, and an
// L2 reduction costs the same for one 8-byte lane as for a whole 32-byte
// sector.  The warp therefore turns its 32 x (x, y, z) integers through shared
// memory so that an atom's components leave as neighbouring lanes of one
// instruction into the atom's own sector of f4 (with dE/dR the fourth: the
// adjoint's pushes cost no more sectors).  89.6 M random pushes of a triple,
// alone: 2.13 ms as three scattered reductions, 0.65 ms turned.
//
// The entry's position is read as pos[index]: atom i's neighbourhood of
// positions stays in L1, where the 16-byte list entries themselves do not.
template <class Q, bool ADJ>
__global__ void __launch_bounds__(kThreads, 8) gbsw_chain_kernel(const float4* __restrict__ pos, int n, Entries tab,
                                                                 Quad quad, ModelConst m, int n_chunks, DEdJ dEdJ,
                                                                 ChainOut out, ChainRecords rr) {
  constexpr int kComp = ADJ ? 4 : 3;  // integers pushed per item
  constexpr int kWarps = kThreads / kWarp;
  constexpr int kWalkKeep = 4;        // shaping entries remembered by a list walk
  constexpr int kRing = 2 * kWarp;    // fewer than 32 items pending, plus one round of at most 32
  __shared__ float4 s_v[kWarps][kRing];   // (v, V) of two batches' records
  __shared__ float2 s_c[kWarps][kRing];   // (c, list start)
  __shared__ unsigned s_item[kWarps][kRing];  // record slot << 16 | list position
  __shared__ long long s_f[kWarps][kWarp * kComp];
  __shared__ int s_k[kWarps][kWarp];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp, wib = threadIdx.x / kWarp;
  if (warp >= n * n_chunks) return;
  const int c = warp / n, nth = warp - c * n, i = rr.order ? __ldg(rr.order + nth) : nth;
  const float4 xi = pos[i];
  const float2 de = dEdJ.of(i, lane);
  const unsigned lt = (1u << lane) - 1u;
  // F_i as fixed-point integers: every contribution is rounded on its own, so
  // the record and the list-walk paths give the same bits
  long long fix = 0, fiy = 0, fiz = 0;
  // the records need no cell query, and setting one up is FP64 work in every
  // warp: 43 -> 35 us at 6,007 atoms on a grid table, 258 -> 244 in a periodic box
  Q query;
  query.init_images(tab);
  float4* sv = s_v[wib];
  float2* sc = s_c[wib];
  unsigned* items = s_item[wib];
  long long* sf = s_f[wib];
  int* sk = s_k[wib];
  unsigned head = 0, tail = 0;  // warp-uniform ring positions
  // the pending items (at most 32), one per lane
  auto evaluate = [&]() {
    __syncwarp();
    const bool valid = head + lane < tail;
    int k = -1;
    long long f[4] = {0, 0, 0, 0};
    if (valid) {
      const unsigned it = items[(head + lane) & (kRing - 1)];
      const float4 rv = sv[it >> 16];
      const float2 rc = sc[it >> 16];
      k = __ldg(tab.index + __float_as_int(rc.y) + (int)(it & 0xffffu));
      const float4 a = __ldg(pos + k);
      const Shaping<Q> sh(query, m, out, a, xi, rv, rv.w, rc.x);
      if (ADJ) f[3] = float_to_fixed(rc.x * sh.g * (-0.9520f));  // dV/dR_k = -(V/u) u' dR'/dR
      if (k != i) {  // atom i moves with the point
        if (sh.push) {
          f[0] = sh.fx;
          f[1] = sh.fy;
          f[2] = sh.fz;
        }
        fix -= sh.fx;
        fiy -= sh.fy;
        fiz -= sh.fz;
      }
    }
#pragma unroll
    for (int u = 0; u < kComp; ++u) sf[kComp * lane + u] = f[u];
    sk[lane] = k;
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kComp; ++u) {
      const int t = u * kWarp + lane;
      const int e = t / kComp;
      const long long val = sf[t];
      if (val) atomicAdd(out.f4 + 4 * (size_t)sk[e] + (t - kComp * e), (unsigned long long)val);
    }
    head = min(head + kWarp, tail);
  };
  const int npts = rr.count ? rr.count[warp] : -1;
  if (npts >= 0) {
    const int4* region = rr.rec + (size_t)warp * rr.R;
    const int* sregion = rr.st + (size_t)warp * rr.R;
    // the next batch's records and list starts, loaded one batch ahead
    int4 prn = make_int4(0, 0, 0, 0);
    int psn = 0;
    if (lane < npts) {
      prn = __ldcs(region + lane);
      psn = __ldcs(sregion + lane);
    }
    for (int b = 0; b < npts; b += kWarp) {
      const unsigned carried = tail - head;
      const unsigned base = head;
      const int slot = (b & kWarp) + lane;  // two batches' records alternate
      unsigned mlo = 0u, mhi = 0u;
      if (b + lane < npts) {
        mlo = (unsigned)prn.z;
        mhi = (unsigned)prn.w;
        const float4 v = quad.qv[prn.x];
        const float2 w = quad.qw[prn.x];
        sv[slot] = make_float4(v.x, v.y, v.z, __int_as_float(prn.y));
        sc[slot] = make_float2(fmaf(de.x, w.x, de.y * w.y), __int_as_float(psn));
      }
      if (b + kWarp + lane < npts) {
        prn = __ldcs(region + b + kWarp + lane);
        psn = __ldcs(sregion + b + kWarp + lane);
      }
      unsigned have;
      while ((have = __ballot_sync(0xffffffffu, (mlo | mhi) != 0u)) != 0u) {
        if (mlo | mhi) {
          int l;
          if (mlo) {
            l = __ffs((int)mlo) - 1;
            mlo &= mlo - 1;
          } else {
            l = 31 + __ffs((int)mhi);
            mhi &= mhi - 1;
          }
          items[(tail + __popc(have & lt)) & (kRing - 1)] = (unsigned)(slot << 16 | l);
        }
        tail += __popc(have);
        if (tail - head >= kWarp) evaluate();
      }
      // items carried into this batch must not outlive it: the next one takes their records' slots
      if (carried > 0 && head == base) evaluate();
    }
  } else {
    // the list walk, a lane per point: bound by its scattered list reads, so an
    // entry pair is one 32-byte load (a load for each field, and a second walk to
    // find the shaping entries again: 10,000 atoms, 32 x 110, 1,752 us a call
    // where this takes 1,386; lists of 325 entries, 2,000 atoms, 3,109 and 2,006)
    query.init(tab, xi, quad.qoff);
    Points pts{};
    pts.init<Q>(quad, m, xi, c, n_chunks, lane);
    for (int b = pts.t0; b < pts.t1; b += kWarp) {
      const unsigned carried = tail - head;
      const unsigned base = head;
      const int slot = ((b - pts.t0) & kWarp) + lane;
      const int q = pts.q(b + lane);
      int cnt = 0, st = 0;
      int kept[kWalkKeep] = {}, shaping = 0;  // list positions of the first shaping entries, and how many there are
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      float V = 1.0f;
      if (b + lane < pts.t1) {
        v = quad.qv[q];
        const float2 w = quad.qw[q];
        const long long cell = query.cell(xi, v, q);
        if (cell >= 0) {
          const int2 cs = __ldg(tab.cell + cell);
          cnt = cs.x;  // buried or empty: no atom shapes the point
          st = cs.y;
        }
        for (int l = 0; l < cnt; l += 2) {  // an odd list ends in a padding entry no point is near
          const EntryPair p = ldg_entries(tab.e, st + l);
          const float g[2] = {sphere_gap(query.delta(make_float4(p.x.x, p.y.x, p.z.x, 0.f), xi, v), -p.nw.x),
                              sphere_gap(query.delta(make_float4(p.x.y, p.y.y, p.z.y, 0.f), xi, v), -p.nw.y)};
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (g[h] <= -m.sw) {
              V = 0.0f;
              cnt = 0;
            } else if (g[h] < m.sw) {
              V *= fmaf(g[h], fmaf(-m.c3 * g[h], g[h], m.c1), 0.5f);
#pragma unroll
              for (int u = 0; u < kWalkKeep; ++u)
                if (shaping == u) kept[u] = l + h;
              ++shaping;
            }
          }
        }
        if (V == 0.0f) cnt = shaping = 0;
        sv[slot] = make_float4(v.x, v.y, v.z, V);
        sc[slot] = make_float2(fmaf(de.x, w.x, de.y * w.y), __int_as_float(st));
      }
      // the shaping entries: those kept, or where there were more, all looked at again
      const bool few = shaping <= kWalkKeep;
      const int looks = few ? shaping : cnt;
      for (int t = 0; __any_sync(0xffffffffu, t < looks); ++t) {
        bool in = t < looks;
        int l = t;
        if (in && few) {
#pragma unroll
          for (int u = 0; u < kWalkKeep; ++u)
            if (t == u) l = kept[u];
        } else if (in) {
          const float4 a = entry_at(tab, st + l);
          in = fabsf(sphere_gap(query.delta(a, xi, v), a.w)) < m.sw;
        }
        const unsigned have = __ballot_sync(0xffffffffu, in);
        if (in) items[(tail + __popc(have & lt)) & (kRing - 1)] = (unsigned)(slot << 16 | l);
        tail += __popc(have);
        if (tail - head >= kWarp) evaluate();
      }
      if (carried > 0 && head == base) evaluate();
    }
  }
  if (tail != head) evaluate();
  for (int off = 16; off > 0; off >>= 1) {
    fix += __shfl_xor_sync(0xffffffffu, fix, off);
    fiy += __shfl_xor_sync(0xffffffffu, fiy, off);
    fiz += __shfl_xor_sync(0xffffffffu, fiz, off);
  }
  if (lane == 0) push3(out, i, fix, fiy, fiz);
}

// GBMV chain rule with the warp cooperating on one point at a time: the
// point's sums come from the integral pass, lanes read consecutive entries of
// its list (coalesced; GBMV visits whole lists of nearly equal length), push
// their atom's force and accumulate the point's pull on atom i.  Lanes first
// take 32 points' cells together, then the warp walks those points in turn.
template <int MODEL, class Q, bool ADJ>
// Six blocks per SM (at most 80 registers): the occupancy this latency-bound
// kernel was measured fastest at; left to itself the compiler takes 87.
__global__ void __launch_bounds__(kThreads, 6) gbmv_chain_kernel(const float4* __restrict__ pos, int n, Entries tab,
                                                              Quad quad, ModelConst m, int chunk, int n_chunks,
                                                              const float2* __restrict__ dEdJ, ChainOut out,
                                                              const float* __restrict__ state) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp;
  if (warp >= n * n_chunks) return;
  const int i = warp % n, c = warp / n;
  const float4 xi = pos[i];
  const float2 de = dEdJ[i];
  Q query;
  query.init(tab, xi, quad.qoff);
  const int q0 = c * chunk, q1 = min(m.nq, q0 + chunk);
  const size_t plane = (size_t)n * m.nq;
  long long fix = 0, fiy = 0, fiz = 0;
  for (int base = q0; base < q1; base += kWarp) {
    // lane t takes point base + t: its cell, its state (coalesced) and the
    // point's factors of the chain rule, which the warp then broadcasts
    const int qm = base + lane;
    float4 vm = make_float4(0.f, 0.f, 0.f, 0.f);
    int cntm = 0, sm = 0;
    float cSm = 0.0f;                    // c ds/dS (0: nothing to push)
    float t1m = 0.f, t2m = 0.f, t3m = 0.f;  // GBMV-II: d s1, d s2, d s3^2 factors
    float vxm = 0.f, vym = 0.f, vzm = 0.f;
    if (qm < q1) {
      vm = quad.qv[qm];
      const float2 w = quad.qw[qm];
      const float cq = fmaf(de.x, w.x, de.y * w.y);
      const long long cell = query.cell(xi, vm, qm);
      if (cell >= 0) {
        const int2 cs = __ldg(tab.cell + cell);
        cntm = cs.x;
        sm = cs.y;
      }
      if (cntm > 0 && cq != 0.0f) {
        const size_t idx = (size_t)i * m.nq + qm;
        float p;
        if constexpr (MODEL == GBX_MODEL_GBMV1) {
          logistic_solvent(m.beta, m.lambda, state[idx], p);
          cSm = cq * __fdividef(m.beta * p, (1.0f + p) * (1.0f + p));
        } else {
          const Gbmv2State st{state[idx], state[idx + plane], state[idx + 2 * plane], state[idx + 3 * plane],
                              state[idx + 4 * plane]};
          const float s3sq = fmaf(st.vx, st.vx, fmaf(st.vy, st.vy, st.vz * st.vz));
          logistic_solvent(m.beta, m.lambda, m.s0 * st.s1 * st.s2 / s3sq, p);
          cSm = cq * __fdividef(m.beta * p, (1.0f + p) * (1.0f + p)) * m.s0;
          const float inv3 = 1.0f / s3sq;
          t1m = st.s2 * inv3;
          t2m = st.s1 * inv3;
          t3m = -st.s1 * st.s2 * inv3 * inv3;
          vxm = st.vx;
          vym = st.vy;
          vzm = st.vz;
        }
      }
    }
    float px = 0.f, py = 0.f, pz = 0.f;  // this lane's share of the points' pull on atom i
    const int np = min(kWarp, q1 - base);
    for (int t = 0; t < np; ++t) {
      const int cnt = __shfl_sync(0xffffffffu, cntm, t), s = __shfl_sync(0xffffffffu, sm, t);
      const float cS = __shfl_sync(0xffffffffu, cSm, t);
      if (cnt <= 0 || cS == 0.0f) continue;
      const float4 v = make_float4(__shfl_sync(0xffffffffu, vm.x, t), __shfl_sync(0xffffffffu, vm.y, t),
                                   __shfl_sync(0xffffffffu, vm.z, t), 0.f);
      if constexpr (MODEL == GBX_MODEL_GBMV1) {
        for (int l = lane; l < cnt; l += kWarp) {
          const float4 a = __ldg(tab.e + s + l);
          const float3 d = query.delta(a, xi, v);
          const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
          const float r4 = r2 * r2;
          const float e = __expf(a.w * r4);
          const int k = __ldg(tab.index + s + l);
          if (ADJ) push_radius(out, k, cS * e * r4 * (-4.0f * a.w / __ldg(&tab.par[s + l].x)));
          if (k == i) continue;
          const float gs = cS * 4.0f * a.w * e * r2;  // dS/d(delta) = 4 gamma e r^2 delta
          const float gx = gs * d.x, gy = gs * d.y, gz = gs * d.z;
          push_force(out, k, gx, gy, gz);
          px += gx;
          py += gy;
          pz += gz;
        }
      } else {
        const float t1 = __shfl_sync(0xffffffffu, t1m, t), t2 = __shfl_sync(0xffffffffu, t2m, t),
                    t3 = __shfl_sync(0xffffffffu, t3m, t);
        const Gbmv2State st{0.f, 0.f, __shfl_sync(0xffffffffu, vxm, t), __shfl_sync(0xffffffffu, vym, t),
                            __shfl_sync(0xffffffffu, vzm, t)};
        for (int l = lane; l < cnt; l += kWarp) {
          const float4 a = __ldg(tab.e + s + l);
          const float2 pk = __ldg(tab.par + s + l);
          const float3 d = query.delta(a, xi, v);
          const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
          const float T = fmaf(100.0f, r2, pk.x);
          const float CT = __fdividef(a.w, T);
          const float F = CT * CT;
          const float dFf = -400.0f * F * __fdividef(1.0f, T);  // dF/d(delta) = dFf delta
          const float vd = st.vx * d.x + st.vy * d.y + st.vz * d.z;
          const int k = __ldg(tab.index + s + l);
          if (ADJ) {
            const float R = pk.y;
            const float Cp = 10.0f * m.p1, Tp = Cp - 200.0f * R;
            const float dFdR = 2.0f * CT * __fdividef(Cp * T - a.w * Tp, T * T);
            push_radius(out, k, cS * (t1 * dFdR + t2 * (r2 * 2.0f * F * dFdR) + t3 * (2.0f * vd * dFdR)));
          }
          if (k == i) continue;
          const float sc = t1 * dFf + t2 * 2.0f * F * fmaf(dFf, r2, F) + t3 * 2.0f * vd * dFf;
          const float gx = cS * fmaf(sc, d.x, t3 * 2.0f * F * st.vx);
          const float gy = cS * fmaf(sc, d.y, t3 * 2.0f * F * st.vy);
          const float gz = cS * fmaf(sc, d.z, t3 * 2.0f * F * st.vz);
          push_force(out, k, gx, gy, gz);
          px += gx;
          py += gy;
          pz += gz;
        }
      }
    }
    fix += float_to_fixed(px);
    fiy += float_to_fixed(py);
    fiz += float_to_fixed(pz);
  }
  for (int off = 16; off > 0; off >>= 1) {
    fix += __shfl_xor_sync(0xffffffffu, fix, off);
    fiy += __shfl_xor_sync(0xffffffffu, fiy, off);
    fiz += __shfl_xor_sync(0xffffffffu, fiz, off);
  }
  if (lane == 0) push3(out, i, fix, fiy, fiz);
}

Entries entries_of(const Context* ctx) {
  if (ctx->use_tight)
    return Entries{ctx->d_tgeom,     ctx->d_tcell,   ctx->d_tentry,
                   nullptr,          ctx->d_tindex,  ctx->tcell_cap,
                   ctx->d_tfirst,    ctx->tentry_cap, ctx->cfg.periodic ? ctx->d_wgeom : nullptr};
  if (ctx->cfg.model == GBX_MODEL_GBSW)
    return Entries{ctx->d_geom,   ctx->d_cell2, ctx->d_entry4, nullptr, ctx->d_entry_index, ctx->cell_cap,
                   ctx->d_rfirst, ctx->entry_cap};
  return Entries{ctx->d_geom,    ctx->d_cell2,    ctx->d_entry4, ctx->d_entry_par, ctx->d_entries, ctx->cell_cap,
                 nullptr,        ctx->entry_cap};
}

// The same for work counting: a reference GBSW table's lists in ascending atom
// order, through the positions.
Entries counted_entries_of(const Context* ctx, const float4* pos) {
  Entries t = entries_of(ctx);
  if (ctx->cfg.model == GBX_MODEL_GBSW && !ctx->use_tight) {
    t.e = pos;
    t.index = ctx->d_entries;
    t.first = nullptr;
  }
  return t;
}

int volume_blocks(const Context* ctx) {
  const long long warps = (long long)ctx->n * ctx->n_chunks;
  return (int)((warps * kWarp + kThreads - 1) / kThreads);
}

template <int MODEL, class Q>
void launch_integrals_t(Context* ctx, const float4* pos, const ModelConst& m, bool count_work) {
  if (MODEL != GBX_MODEL_GBSW && !count_work && ctx->gbmv_cells) {
    launch_gbmv_cells_integral(ctx, pos, m);
    return;
  }
  const Entries t = entries_of(ctx);
  const Quad qd{ctx->d_qv, ctx->d_qw, ctx->d_qoff};
  const int chunk = (m.nq + ctx->n_chunks - 1) / ctx->n_chunks;
  const ShellSink sink{ctx->d_srec, ctx->d_srec_st, ctx->d_rcount, ctx->d_rmax, ctx->srec_R};
  if (MODEL == GBX_MODEL_GBSW && !count_work) {
    // persistent grid: the resident blocks of every SM (or fewer, for few items)
    if (ctx->integral_grid == 0) {
      int per_sm = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gbsw_integral_kernel<Q, kEmitAll>, kThreads, 0) !=
              cudaSuccess ||
          per_sm < 1)
        per_sm = 1;
      ctx->integral_grid = per_sm * ctx->sms;
    }
    const int grid = std::min(volume_blocks(ctx), ctx->integral_grid);
    auto kernel = !ctx->records       ? gbsw_integral_kernel<Q, kEmitNone>
                  : ctx->records_self ? gbsw_integral_kernel<Q, kEmitAll>
                                      : gbsw_integral_kernel<Q, kEmitOthers>;
    kernel<<<grid, kThreads, 0, ctx->stream>>>(pos, ctx->n, t, qd, m, ctx->n_chunks, ctx->d_J, sink,
                                               ctx->d_next_item, items_in_order(ctx) ? ctx->d_perm_tmp : nullptr);
  }
  else if (count_work)
    integral_kernel<MODEL, Q, true><<<volume_blocks(ctx), kThreads, 0, ctx->stream>>>(
        pos, ctx->n, counted_entries_of(ctx, pos), qd, m, chunk, ctx->n_chunks, ctx->d_J, ctx->d_work, ctx->d_pstate);
  else if constexpr (MODEL != GBX_MODEL_GBSW)
    gbmv_integral_kernel<MODEL, Q><<<volume_blocks(ctx), kThreads, 0, ctx->stream>>>(
        pos, ctx->n, t, qd, m, chunk, ctx->n_chunks, ctx->d_J, ctx->d_pstate);
  ++ctx->launches;
}

template <int MODEL, class Q, bool ADJ>
void launch_chain_t(Context* ctx, const float4* pos, const ModelConst& m) {
  if (MODEL != GBX_MODEL_GBSW && ctx->gbmv_cells) {
    launch_gbmv_cells_chain(ctx, pos, m, ADJ);
    return;
  }
  const Entries t = entries_of(ctx);
  const Quad qd{ctx->d_qv, ctx->d_qw, ctx->d_qoff};
  const int chunk = (m.nq + ctx->n_chunks - 1) / ctx->n_chunks;
  const ChainOut o{ctx->d_f4, m.cutoff_chain_quirk && m.cutoff2 > 0.0f, m.cutoff2};
  const int blocks = volume_blocks(ctx);
  if constexpr (MODEL == GBX_MODEL_GBSW) {
    const ChainRecords rr{ctx->d_srec, ctx->d_srec_st, ctx->records ? ctx->d_rcount : nullptr, ctx->srec_R,
                          items_in_order(ctx) ? ctx->d_perm_tmp : nullptr};
    const DEdJ de{chain_forms_dEdJ(ctx, ADJ) ? nullptr : ctx->d_dEdJ, ctx->d_dEdB_fx, ctx->d_dBdJ};
    gbsw_chain_kernel<Q, ADJ><<<blocks, kThreads, 0, ctx->stream>>>(pos, ctx->n, t, qd, m, ctx->n_chunks, de, o, rr);
  } else {
    gbmv_chain_kernel<MODEL, Q, ADJ><<<blocks, kThreads, 0, ctx->stream>>>(pos, ctx->n, t, qd, m, chunk, ctx->n_chunks,
                                                                           ctx->d_dEdJ, o, ctx->d_pstate);
  }
  ++ctx->launches;
}

gbx_status launch_status(Context* ctx, const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

}  // namespace

gbx_status launch_binning(Context* ctx, const float4* pos, bool count_work) {
  ctx->gbmv_cells = ctx->cfg.model != GBX_MODEL_GBSW && !count_work && gbmv_cells_apply(ctx);
  if (!ctx->gbmv_cells) return GBX_OK;
  launch_gbmv_cells_bin(ctx, pos, make_model_const(ctx));
  return launch_status(ctx, "point binning launch");
}

gbx_status launch_integrals(Context* ctx, const float4* pos, bool count_work) {
  const ModelConst m = make_model_const(ctx);
  if (ctx->use_tight && ctx->cfg.periodic) {
    launch_integrals_t<GBX_MODEL_GBSW, PeriodicTightQuery>(ctx, pos, m, count_work);
  } else if (ctx->use_tight) {
    launch_integrals_t<GBX_MODEL_GBSW, TightQuery>(ctx, pos, m, count_work);
  } else if (ctx->cfg.periodic && ctx->cfg.table_mode == GBX_TABLE_STANDALONE) {
    launch_integrals_t<GBX_MODEL_GBSW, PeriodicQuery>(ctx, pos, m, count_work);
  } else if (ctx->cfg.periodic) {
    switch (ctx->cfg.model) {
      case GBX_MODEL_GBSW: launch_integrals_t<GBX_MODEL_GBSW, MinImageQuery>(ctx, pos, m, count_work); break;
      case GBX_MODEL_GBMV1: launch_integrals_t<GBX_MODEL_GBMV1, MinImageQuery>(ctx, pos, m, count_work); break;
      default: launch_integrals_t<GBX_MODEL_GBMV2, MinImageQuery>(ctx, pos, m, count_work); break;
    }
  } else {
    switch (ctx->cfg.model) {
      case GBX_MODEL_GBSW: launch_integrals_t<GBX_MODEL_GBSW, RefQuery>(ctx, pos, m, count_work); break;
      case GBX_MODEL_GBMV1: launch_integrals_t<GBX_MODEL_GBMV1, RefQuery>(ctx, pos, m, count_work); break;
      default: launch_integrals_t<GBX_MODEL_GBMV2, RefQuery>(ctx, pos, m, count_work); break;
    }
  }
  return launch_status(ctx, "integral launch");
}

gbx_status launch_chain(Context* ctx, const float4* pos, bool adjoint) {
  const ModelConst m = make_model_const(ctx);
  if (ctx->use_tight && ctx->cfg.periodic) {
    if (adjoint) launch_chain_t<GBX_MODEL_GBSW, PeriodicTightQuery, true>(ctx, pos, m);
    else launch_chain_t<GBX_MODEL_GBSW, PeriodicTightQuery, false>(ctx, pos, m);
  } else if (ctx->use_tight) {
    if (adjoint) launch_chain_t<GBX_MODEL_GBSW, TightQuery, true>(ctx, pos, m);
    else launch_chain_t<GBX_MODEL_GBSW, TightQuery, false>(ctx, pos, m);
  } else if (ctx->cfg.periodic && ctx->cfg.table_mode == GBX_TABLE_STANDALONE) {
    if (adjoint) launch_chain_t<GBX_MODEL_GBSW, PeriodicQuery, true>(ctx, pos, m);
    else launch_chain_t<GBX_MODEL_GBSW, PeriodicQuery, false>(ctx, pos, m);
  } else if (ctx->cfg.periodic) {
    switch (ctx->cfg.model * 2 + (adjoint ? 1 : 0)) {
      case 0: launch_chain_t<GBX_MODEL_GBSW, MinImageQuery, false>(ctx, pos, m); break;
      case 1: launch_chain_t<GBX_MODEL_GBSW, MinImageQuery, true>(ctx, pos, m); break;
      case 2: launch_chain_t<GBX_MODEL_GBMV1, MinImageQuery, false>(ctx, pos, m); break;
      case 3: launch_chain_t<GBX_MODEL_GBMV1, MinImageQuery, true>(ctx, pos, m); break;
      case 4: launch_chain_t<GBX_MODEL_GBMV2, MinImageQuery, false>(ctx, pos, m); break;
      default: launch_chain_t<GBX_MODEL_GBMV2, MinImageQuery, true>(ctx, pos, m); break;
    }
  } else {
    switch (ctx->cfg.model * 2 + (adjoint ? 1 : 0)) {
      case 0: launch_chain_t<GBX_MODEL_GBSW, RefQuery, false>(ctx, pos, m); break;
      case 1: launch_chain_t<GBX_MODEL_GBSW, RefQuery, true>(ctx, pos, m); break;
      case 2: launch_chain_t<GBX_MODEL_GBMV1, RefQuery, false>(ctx, pos, m); break;
      case 3: launch_chain_t<GBX_MODEL_GBMV1, RefQuery, true>(ctx, pos, m); break;
      case 4: launch_chain_t<GBX_MODEL_GBMV2, RefQuery, false>(ctx, pos, m); break;
      default: launch_chain_t<GBX_MODEL_GBMV2, RefQuery, true>(ctx, pos, m); break;
    }
  }
  return launch_status(ctx, "chain launch");
}

}  // namespace gbx
