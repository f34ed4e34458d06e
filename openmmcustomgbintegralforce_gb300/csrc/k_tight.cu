// Exact GBSW lookup table.
//
// The GBSW volume of a point is V(p) = 0 if some atom buries it
// (|p - x_j| <= R'_j - w), else the product of u_j over the atoms whose
// switching shell holds it (R'_j - w < |p - x_j| < R'_j + w)
// (CharmmReferenceGBSW.cpp:616-639).  The reference's standalone table pads
// every grid point by buffer + maxR + w + (sqrt3/2) h + 1e-6 (:454-455), more
// than any shell reaches from anywhere in the queried cell, so its lists give
// exactly this V.  This table gives the same V with far shorter lists:
//
//   * cell c (edge h, default 0.1 nm) lists atom j when the distance from
//     x_j to the cell's box is below R'_j + w + eps;
//   * a cell whose farthest corner lies within R'_j - w - eps of some x_j is
//     buried: V = 0 for every point in it, no list is read;
//   * the grid spans the atoms' bounding box plus max(R') + w + h, so a
//     point outside it touches no shell (V = 1).
//
// eps (2e-5 nm plus 4 2^-23 of the largest coordinate, with the grid's margins
// and a periodic system's longest box edge added to it) covers the FP32
// rounding of both the build and the point-to-cell assignment, so every
// atom a point needs is in the list of whichever neighbouring cell its FP32
// coordinates select.  Entries are stored inline (x, y, z, R') and sorted by
// the distance from the cell centre to the atom's burying sphere, so a
// buried point usually stops at its first entry.
#include <math.h>

#include "buckets.cuh"
#include "gbx_internal.cuh"
#include "scan.cuh"

namespace gbx {
namespace {

constexpr int kSortWarps = 4;
constexpr int kSortBuf = 256;
constexpr int kSortLanes = 8;                                   // lanes per short list
constexpr int kSortGroups = kWarp / kSortLanes;
constexpr int kSortSmall = kSortBuf / kSortGroups;              // longest short list (64)

struct TightArgs {
  const float4* pos;  // x, y, z, R'
  int n;
  const TableGeom* geom;
  float w;
  Members mem;
  int* buried;
  long long cell_cap;
};

__global__ void tight_members_kernel(TightArgs a) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x % kWarp;
  const TableGeom& g = *a.geom;
  if (g.ncell > a.cell_cap) return;
  const float h = (float)g.step[0];
  const float inv_h = (float)g.inv_step[0];
  const float eps = (float)g.pad;
  const long long sx = (long long)g.dims[1] * g.dims[2], sy = g.dims[2];
  for (int at = warp; at < a.n; at += (gridDim.x * blockDim.x) / kWarp) {
    const float4 p = a.pos[at];
    // coordinates relative to the grid origin, lane k forming axis k in
    // FP64 (the slow FP64 pipe is then busy for one instruction, not three)
    float xk = 0.0f;
    if (lane < 3) xk = (float)((double)(lane == 0 ? p.x : (lane == 1 ? p.y : p.z)) - g.min[lane]);
    const float x[3] = {__shfl_sync(0xffffffffu, xk, 0), __shfl_sync(0xffffffffu, xk, 1),
                        __shfl_sync(0xffffffffu, xk, 2)};
    const float reach = p.w + a.w + eps;
    const float bury = p.w - a.w - eps;
    int b[3], e[3];
    bool ok = true;
    for (int k = 0; k < 3; ++k) {
      b[k] = max(0, (int)floorf((x[k] - reach) * inv_h));
      e[k] = min(g.dims[k] - 1, (int)floorf((x[k] + reach) * inv_h));
      if (!(e[k] >= b[k] && e[k] - b[k] < 256)) ok = false;
    }
    if (!ok) {
      if (lane == 0) atomicOr(a.mem.status, kStatusTableCells);
      continue;
    }
    // the offsets of cell c's lower and upper face along one axis
    auto faces = [h](int c, float at) {
      const float lo = __fmul_rn((float)c, h);
      return make_float2(__fsub_rn(lo, at), __fsub_rn(__fadd_rn(lo, h), at));
    };
    const int ny = e[1] - b[1] + 1, nz = e[2] - b[2] + 1, total = (e[0] - b[0] + 1) * ny * nz;
    const BoxIndex box(ny, nz);
    for (int t0 = lane; t0 < total; t0 += kPutBatch * kWarp) {
      long long cell[kPutBatch];
#pragma unroll
      for (int u = 0; u < kPutBatch; ++u) {
        const int t = t0 + u * kWarp;
        cell[u] = -1;
        if (t >= total) continue;
        const int3 o = box(t);
        const int c[3] = {b[0] + o.x, b[1] + o.y, b[2] + o.z};
        float near = 0.f, far = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float2 f = faces(c[k], x[k]);
          const float dn = fmaxf(fmaxf(f.x, -f.y), 0.f), df = fmaxf(-f.x, f.y);
          near = fmaf(dn, dn, near);
          far = fmaf(df, df, far);
        }
        if (!(near < reach * reach)) continue;
        cell[u] = c[0] * sx + c[1] * sy + c[2];
        if (bury > 0.f && far <= bury * bury) atomicOr(&a.buried[cell[u]], 1);
      }
      a.mem.put(cell, at);
    }
  }
}

// Sort each list of atom indices, and write the entries (positions and radii)
// in that order: by (distance from the cell centre to the atom's burying
// sphere, atom index) -- a deterministic order whatever the fill order was --
// and mark buried cells with count -1.
__global__ void __launch_bounds__(kSortWarps * kWarp) tight_sort_kernel(const float4* __restrict__ pos,
                                                                        Members mem, const int* __restrict__ start,
                                                                        const int* __restrict__ buried,
                                                                        float4* __restrict__ entry,
                                                                        int* __restrict__ index,
                                                                        int2* __restrict__ cell,
                                                                        TightCell* __restrict__ first,
                                                                        const TableGeom* __restrict__ gp, float w,
                                                                        long long cell_cap, long long entry_cap) {
  // sorted entries, as pairs field by field (EntryPair, queries.cuh)
  auto put = [entry](int at, const float4 e) {
    float* p = reinterpret_cast<float*>(entry) + 8 * (size_t)(at >> 1) + (at & 1);
    p[0] = e.x;
    p[2] = e.y;
    p[4] = e.z;
    p[6] = -e.w;
  };
  // after an odd list: the pair reads of the integral pass meet a sphere no point is near
  const float4 kPadEntry = make_float4(0.f, 0.f, 0.f, -1e6f);
  // keys and atoms only, the positions are read again in sorted order: with them
  // here (24 KB a block) 9 blocks fitted an SM and the table stage took 207 us
  // at 50,000 atoms, 183 without
  __shared__ int s_i[kSortWarps][kSortBuf];
  __shared__ float s_k[kSortWarps][kSortBuf];
  const int wib = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const TableGeom& g = *gp;
  if (g.ncell > cell_cap || g.total > entry_cap) return;
  const long long ncell = g.ncell;
  const int isx = g.dims[1] * g.dims[2];  // fewer than 2^31 cells
  const float cmin[3] = {(float)g.min[0], (float)g.min[1], (float)g.min[2]};
  const float step = (float)g.step[0];
  // eight lanes per cell, four consecutive cells at a time: lists of up to
  // eight entries (most) are ranked in registers, up to kSortSmall in the
  // group's quarter of the warp's buffer; longer lists take the whole warp
  const int grp = lane / kSortLanes, gl = lane % kSortLanes;
  const unsigned gmask = ((1u << kSortLanes) - 1u) << (grp * kSortLanes);
  for (long long c0 = ((long long)blockIdx.x * kSortWarps + wib) * kSortGroups; c0 < ncell;
       c0 += (long long)gridDim.x * kSortWarps * kSortGroups) {
    const long long c = c0 + grp;
    int cnt = 0, s = 0, bur = 0;
    const int* src = index;  // the unsorted members
    if (c < ncell) {
      cnt = mem.count[c];
      s = start[c];
      bur = cnt > 0 ? buried[c] : 0;
      if (cnt > kSortBuf && !bur) {  // no list: no record may say there is one
        if (gl == 0) atomicOr(mem.status, kStatusSegmentTooLong);
        cnt = 0;
      }
      if (cnt > mem.size && !bur) {
        mem.gather(c, cnt, index + s, gl, kSortLanes);
        src = index + s;
      } else {
        src = mem.slots + c * mem.size;
      }
      if (gl == 0) {
        cell[c] = make_int2(bur ? -1 : cnt, s);
        first[c].cs = make_int2(bur ? -1 : cnt, s);
      }
    }
    __syncwarp();
    if (cnt > 0 && !bur && cnt <= kSortSmall) {
      const int cx = (int)c / isx, rem = (int)c - cx * isx, cy = rem / g.dims[2], cz = rem - cy * g.dims[2];
      const float ctr[3] = {cmin[0] + ((float)cx + 0.5f) * step, cmin[1] + ((float)cy + 0.5f) * step,
                            cmin[2] + ((float)cz + 0.5f) * step};
      // key: distance to the cell centre less R' - w (atoms likely to bury
      // the cell's points first); FP32, any fixed order is exact
      auto key = [&](const float4 e) {
        const float dx = e.x - ctr[0], dy = e.y - ctr[1], dz = e.z - ctr[2];
        return sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - (e.w - w);
      };
      if (cnt <= kSortLanes) {
        float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
        int i = 0x7fffffff;
        float k = INFINITY;
        if (gl < cnt) {
          i = src[gl];
          e = __ldg(pos + i);
          k = key(e);
        }
        int r = 0;
#pragma unroll
        for (int o = 0; o < kSortLanes; ++o) {
          const float ko = __shfl_sync(gmask, k, o, kSortLanes);
          const int io = __shfl_sync(gmask, i, o, kSortLanes);
          r += (ko < k) || (ko == k && io < i);
        }
        if (gl < cnt) {
          put(s + r, e);
          index[s + r] = i;
          if (r == 0) first[c].first = e;
        }
      } else {
        int* gi = s_i[wib] + grp * kSortSmall;
        float* gk = s_k[wib] + grp * kSortSmall;
        for (int q = gl; q < cnt; q += kSortLanes) {
          const int i = src[q];
          const float4 e = __ldg(pos + i);
          gi[q] = i;
          gk[q] = key(e);
        }
        __syncwarp(gmask);
        for (int q = gl; q < cnt; q += kSortLanes) {
          const float kq = gk[q];
          const int iq = gi[q];
          int r = 0;
          for (int o = 0; o < cnt; ++o) {
            const float ko = gk[o];
            r += (ko < kq) || (ko == kq && gi[o] < iq);
          }
          const float4 e = __ldg(pos + iq);
          put(s + r, e);
          index[s + r] = iq;
          if (r == 0) first[c].first = e;
        }
      }
      if ((cnt & 1) && gl == 0) put(s + cnt, kPadEntry);
    }
    __syncwarp();
    unsigned todo = __ballot_sync(0xffffffffu, gl == 0 && cnt > kSortSmall && !bur);
    while (todo) {
      const int from = __ffs(todo) - 1;
      todo &= todo - 1;
      const long long cc = c0 + from / kSortLanes;
      const int ccnt = __shfl_sync(0xffffffffu, cnt, from), cs = __shfl_sync(0xffffffffu, s, from);
      const int* csrc = ccnt > mem.size ? index + cs : mem.slots + cc * mem.size;
      const int cx = (int)cc / isx, rem = (int)cc - cx * isx, cy = rem / g.dims[2], cz = rem - cy * g.dims[2];
      const float ctr[3] = {cmin[0] + ((float)cx + 0.5f) * step, cmin[1] + ((float)cy + 0.5f) * step,
                            cmin[2] + ((float)cz + 0.5f) * step};
      for (int q = lane; q < ccnt; q += kWarp) {
        const int i = csrc[q];
        const float4 e = __ldg(pos + i);
        s_i[wib][q] = i;
        const float dx = e.x - ctr[0], dy = e.y - ctr[1], dz = e.z - ctr[2];
        s_k[wib][q] = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - (e.w - w);
      }
      __syncwarp();
      for (int q = lane; q < ccnt; q += kWarp) {
        const float kq = s_k[wib][q];
        const int iq = s_i[wib][q];
        int r = 0;
        for (int o = 0; o < ccnt; ++o) {
          const float ko = s_k[wib][o];
          r += (ko < kq) || (ko == kq && s_i[wib][o] < iq);
        }
        const float4 e = __ldg(pos + iq);
        put(cs + r, e);
        index[cs + r] = iq;
        if (r == 0) first[cc].first = e;
      }
      if ((ccnt & 1) && lane == 0) put(cs + ccnt, kPadEntry);
      __syncwarp();
    }
  }
}

}  // namespace

gbx_status launch_tight_build(Context* ctx, const float4* pos) {
  cudaStream_t st = ctx->stream;
  const long long cells = ctx->tcell_cap;
  if (cells > 0) {
    const TableBuckets& b = ctx->tbuckets;
    const Members mem{ctx->d_tcount, b.slots,         b.chain,
                      b.node,        b.size,          ctx->tentry_cap,
                      &ctx->d_tgeom->chained, ctx->d_status};
    const TightArgs a{pos, ctx->n, ctx->d_tgeom, (float)ctx->cfg.switch_width, mem, ctx->d_tburied, cells};
    const int threads = 256;
    long long blocks = ((long long)ctx->n * kWarp + threads - 1) / threads;
    if (blocks > 65535) blocks = 65535;
    tight_members_kernel<<<(int)blocks, threads, 0, st>>>(a);
    ++ctx->launches;
    launch_scan<true>(ctx->d_tcount, ctx->d_tgeom, ctx->d_tstart, cells, ctx->tentry_cap,
                      reinterpret_cast<unsigned long long*>(&ctx->d_tgeom->total), &ctx->d_tgeom->longest, b.size,
                      ctx->d_status, st);
    ++ctx->launches;
    long long sb = (cells + kSortWarps * kSortGroups - 1) / (kSortWarps * kSortGroups);
    if (sb > (long long)ctx->sms * 64) sb = (long long)ctx->sms * 64;
    tight_sort_kernel<<<(int)sb, kSortWarps * kWarp, 0, st>>>(pos, mem, ctx->d_tstart, ctx->d_tburied, ctx->d_tentry,
                                                              ctx->d_tindex, ctx->d_tcell, ctx->d_tfirst, ctx->d_tgeom,
                                                              (float)ctx->cfg.switch_width, cells, ctx->tentry_cap);
    ++ctx->launches;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("tight table launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

}  // namespace gbx
