// Small per-atom kernels: model constants, FP64 Born-radius
// assembly, dE/dB -> dE/dJ conversion and the deterministic energy reduction.
#include <math.h>

#include "gbx_internal.cuh"

namespace gbx {

ModelConst make_model_const(const Context* ctx) {
  const gbx_config& c = ctx->cfg;
  ModelConst m{};
  m.model = c.model;
  m.table_mode = c.table_mode;
  m.cap = c.table_cap;
  m.skip_empty = c.skip_empty;
  m.nq = c.n_radial * c.lebedev_order;
  m.nrad = c.n_radial;
  int bits = 1;
  while ((1LL << bits) < m.nq) ++bits;
  m.nq_magic = (unsigned)(((1ULL << (31 + bits)) + m.nq - 1) / m.nq);
  m.nq_shift = bits - 1;
  m.cutoff_chain_quirk = c.cutoff_chain_quirk;
  const double w = c.switch_width;
  m.sw = (float)w;
  m.c1 = (float)(3.0 / (4.0 * w));
  m.c3 = (float)(1.0 / (4.0 * w * w * w));
  m.gamma0_lnlambda = (float)(c.gamma0 * log(c.lambda));
  m.beta = (float)c.beta;
  m.lambda = (float)c.lambda;
  m.s0 = (float)c.s0;
  m.p1 = (float)c.p1;
  m.p2 = (float)c.p2;
  m.cutoff2 = c.cutoff > 0 ? (float)(c.cutoff * c.cutoff) : 0.0f;
  m.pref = (float)c.prefactor;
  m.h = c.grid_length;
  m.buffer = c.table_buffer;
  m.cutoff = c.cutoff;
  return m;
}

namespace {

// The caller's outputs of a call that ran on internal buffers: forces added
// to the caller's slots (each slot written by one thread), the energy added
// to a float.
__global__ void finish_outputs_kernel(int n, const int* __restrict__ slot_of,
                                      const unsigned long long* __restrict__ fint, unsigned long long* __restrict__ fout,
                                      int stride, const double* __restrict__ e_int, float* __restrict__ e_float) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && e_float) *e_float += (float)*e_int;
  if (i >= n || !fout) return;
  const int k = slot_of ? slot_of[i] : i;
  for (int c = 0; c < 3; ++c) fout[(size_t)c * stride + k] += fint[(size_t)c * n + i];
}

// The call's device status, published to mapped host memory so that a later
// call can read it without synchronising: counts of table overflows and of
// non-finite results, and the largest table seen (cells, list entries).
__device__ __forceinline__ void publish_status(const unsigned* __restrict__ status, const TableGeom* __restrict__ geom,
                                               unsigned long long* __restrict__ dev, StatusRecord* host) {
  const unsigned st = *status;
  if (st & (kStatusTableCells | kStatusTableEntries | kStatusSegmentTooLong)) ++dev[1];
  if (st & kStatusNonFinite) ++dev[2];
  const unsigned long long c = (unsigned long long)geom->ncell, e = (unsigned long long)geom->total;
  if (c > dev[3]) dev[3] = c;
  if (e > dev[4]) dev[4] = e;
  ++dev[0];
  volatile StatusRecord* h = host;
  h->overflows = dev[1];
  h->nonfinite = dev[2];
  h->max_cells = dev[3];
  h->max_entries = dev[4];
  __threadfence_system();
  h->seq = dev[0];
}

// The call's last kernel.  The chain rule's sums join the force buffer by
// reductions (a caller may have other forces adding to it), the fixed-point
// pair energy joins the energy, one thread publishes the status: one launch
// where the energy and the status took one each.
constexpr int kFinishThreads = 256;
__global__ void __launch_bounds__(kFinishThreads) finish_kernel(
    int n, const ulonglong2* __restrict__ f4, unsigned long long* __restrict__ force, int stride,
    unsigned long long* __restrict__ dEdR, const unsigned long long* __restrict__ energy_fx,
    double* __restrict__ energy, const unsigned* __restrict__ status, const TableGeom* __restrict__ geom,
    unsigned long long* __restrict__ pub, StatusRecord* host) {
  const int i = blockIdx.x * kFinishThreads + threadIdx.x;
  if (i == 0) {
    if (energy) *energy += fixed_to_double(*energy_fx);
    publish_status(status, geom, pub, host);
  }
  if (i >= n || !f4) return;
  const ulonglong2 a = f4[2 * i], b = f4[2 * i + 1];
  atomicAdd(force + i, a.x);
  atomicAdd(force + stride + i, a.y);
  atomicAdd(force + 2 * (size_t)stride + i, b.x);
  if (dEdR) dEdR[i] = b.y;
}

constexpr int kBornThreads = 64;
__global__ void __launch_bounds__(kBornThreads) born_kernel(int n, int n_chunks, const float* __restrict__ J, double S4, double S7, double C4,
                            double C7, double alpha0, double alpha1, double* __restrict__ born,
                            float2* __restrict__ bornf, double* __restrict__ dBdJ, double* __restrict__ dBda,
                            double* __restrict__ integrals, unsigned* __restrict__ status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double J4 = 0.0, J7 = 0.0;
  for (int c = 0; c < n_chunks; ++c) {
    J4 += (double)J[(size_t)c * n + i];
    J7 += (double)J[((size_t)n_chunks + c) * n + i];
  }
  // 1/r0 - I4 = C4 + J4 and 1/(4 r0^4) - I7 = C7 + J7 (CharmmReferenceGBSW.cpp:591-593)
  const double t4 = C4 + J4, t7 = C7 + J7;
  const double q7 = sqrt(sqrt(t7));
  const double inv = alpha0 * t4 + alpha1 * q7;
  const double B = 1.0 / inv;
  born[i] = B;
  bornf[i] = make_float2((float)B, (float)inv);
  const double B2 = B * B;
  dBdJ[2 * i] = -B2 * alpha0;
  dBdJ[2 * i + 1] = -B2 * alpha1 * 0.25 * q7 / t7;  // t7^(-3/4) = t7^(1/4) / t7
  dBda[2 * i] = -B2 * t4;
  dBda[2 * i + 1] = -B2 * q7;
  integrals[i] = S4 - J4;
  integrals[n + i] = S7 - J7;
  if (!isfinite(B) || !(B > 0.0)) atomicOr(status, kStatusNonFinite);
}

__global__ void chain_prep_kernel(int n, const unsigned long long* __restrict__ dEdB_fx,
                                  const double* __restrict__ dBdJ, const double* __restrict__ dBda,
                                  float2* __restrict__ dEdJ, double* __restrict__ alpha_terms) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double g = fixed_to_double(dEdB_fx[i]);
  dEdJ[i] = make_float2((float)(g * dBdJ[2 * i]), (float)(g * dBdJ[2 * i + 1]));
  if (alpha_terms) {
    alpha_terms[2 * i] = g * dBda[2 * i];
    alpha_terms[2 * i + 1] = g * dBda[2 * i + 1];
  }
}

constexpr int kRedThreads = 1024;

// One block; fixed reduction shape, so the result is bit-reproducible.
__global__ void __launch_bounds__(kRedThreads) energy_reduce_kernel(const double* __restrict__ parts, int nparts,
                                                                    const unsigned long long* __restrict__ energy_fx,
                                                                    double* __restrict__ energy,
                                                                    const double* __restrict__ alpha_terms, int n,
                                                                    double* __restrict__ alpha_grad) {
  __shared__ double s[3][kRedThreads];
  double e = 0, a0 = 0, a1 = 0;
  {
    // four independent chains (loads in flight), combined in a fixed order
    double e4[4] = {0, 0, 0, 0};
    int k = threadIdx.x;
    for (; k + 3 * kRedThreads < nparts; k += 4 * kRedThreads)
      for (int u = 0; u < 4; ++u) e4[u] += parts[k + u * kRedThreads];
    for (; k < nparts; k += kRedThreads) e4[0] += parts[k];
    e = (e4[0] + e4[1]) + (e4[2] + e4[3]);
  }
  if (alpha_terms)
    for (int k = threadIdx.x; k < n; k += kRedThreads) {
      a0 += alpha_terms[2 * k];
      a1 += alpha_terms[2 * k + 1];
    }
  s[0][threadIdx.x] = e;
  s[1][threadIdx.x] = a0;
  s[2][threadIdx.x] = a1;
  __syncthreads();
  for (int stride = kRedThreads / 2; stride > 0; stride >>= 1) {
    if (threadIdx.x < stride)
      for (int k = 0; k < 3; ++k) s[k][threadIdx.x] += s[k][threadIdx.x + stride];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (energy) *energy += s[0][0] + (energy_fx ? fixed_to_double(*energy_fx) : 0.0);
    if (alpha_grad) {
      alpha_grad[0] = s[1][0];
      alpha_grad[1] = s[2][0];
    }
  }
}

}  // namespace

gbx_status launch_finish_outputs(Context* ctx, unsigned long long* force, int stride, float* energy_float) {
  const int n = ctx->n;
  finish_outputs_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(
      n, ctx->in_permuted ? ctx->d_slot_of : nullptr, ctx->d_force_fx, force, stride, ctx->d_energy, energy_float);
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("output launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

gbx_status launch_born(Context* ctx) {
  const int n = ctx->n;
  // small blocks: the FP64 chains of a few thousand atoms spread over every SM
  born_kernel<<<(n + kBornThreads - 1) / kBornThreads, kBornThreads, 0, ctx->stream>>>(
      n, ctx->n_chunks, ctx->d_J, ctx->S4, ctx->S7, ctx->C4, ctx->C7, ctx->alpha0, ctx->alpha1, ctx->d_born,
      reinterpret_cast<float2*>(ctx->d_bornf), ctx->d_dBdJ, ctx->d_dBdJ + 2 * (size_t)n, ctx->d_integrals,
      ctx->d_status);
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("born launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

bool chain_forms_dEdJ(const Context* ctx, bool adjoint) {
  return ctx->cfg.model == GBX_MODEL_GBSW && !adjoint && !ctx->custom;
}

gbx_status launch_chain_prep(Context* ctx, bool adjoint) {
  if (chain_forms_dEdJ(ctx, adjoint)) return GBX_OK;
  const int n = ctx->n;
  chain_prep_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(
      n, ctx->d_dEdB_fx, ctx->d_dBdJ, ctx->d_dBdJ + 2 * (size_t)n, ctx->d_dEdJ,
      adjoint ? ctx->d_dBdJ + 4 * (size_t)n : nullptr);
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("chain prep launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

// Device adjoint outputs: fixed-point sums to FP64, forces as [n][3].
__global__ void adjoint_out_kernel(int n, int stride, const unsigned long long* __restrict__ force_fx,
                                   const unsigned long long* __restrict__ dq_fx,
                                   const unsigned long long* __restrict__ dR_fx, const double* __restrict__ e_in,
                                   const double* __restrict__ a_in, double* __restrict__ forces,
                                   double* __restrict__ dEdq, double* __restrict__ dEdR, double* __restrict__ energy,
                                   double* __restrict__ dEdalpha) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    if (energy) *energy = *e_in;
    if (dEdalpha) {
      dEdalpha[0] = a_in[0];
      dEdalpha[1] = a_in[1];
    }
  }
  if (i >= n) return;
  if (forces)
    for (int k = 0; k < 3; ++k) forces[3 * (size_t)i + k] = fixed_to_double(force_fx[(size_t)k * stride + i]);
  if (dEdq) dEdq[i] = fixed_to_double(dq_fx[i]);
  if (dEdR) dEdR[i] = fixed_to_double(dR_fx[i]);
}

gbx_status launch_adjoint_out(Context* ctx, double* energy, double* forces, double* dEdq, double* dEdR,
                              double* dEdalpha) {
  const int n = ctx->n;
  adjoint_out_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(n, n, ctx->d_force_fx, ctx->d_dEdq_fx, ctx->d_dEdR_fx,
                                                               ctx->d_energy, ctx->d_alpha_grad, forces, dEdq, dEdR,
                                                               energy, dEdalpha);
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("adjoint output launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

gbx_status launch_finish(Context* ctx, unsigned long long* force, int stride, double* energy, bool chain, bool adjoint) {
  const int n = ctx->n;
  // per-block energy partials (compiled expressions) and the alpha gradient need their own reduction first
  const bool reduce = ctx->energy_parts > 0 || adjoint;
  if (reduce) {
    energy_reduce_kernel<<<1, kRedThreads, 0, ctx->stream>>>(ctx->d_energy_part, ctx->energy_parts, ctx->d_energy_fx,
                                                             energy, adjoint ? ctx->d_dBdJ + 4 * (size_t)n : nullptr,
                                                             n, adjoint ? ctx->d_alpha_grad : nullptr);
    ++ctx->launches;
  }
  finish_kernel<<<chain ? (n + kFinishThreads - 1) / kFinishThreads : 1, kFinishThreads, 0, ctx->stream>>>(
      n, chain ? reinterpret_cast<const ulonglong2*>(ctx->d_f4) : nullptr, force, stride,
      adjoint ? ctx->d_dEdR_fx : nullptr, ctx->d_energy_fx, reduce ? nullptr : energy, ctx->d_status,
      ctx->use_tight ? ctx->d_tgeom : ctx->d_geom, ctx->d_pub, ctx->h_pub_dev);
  ++ctx->launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->last_error = std::string("finish launch: ") + cudaGetErrorString(e);
    return GBX_ERR_CUDA;
  }
  return GBX_OK;
}

}  // namespace gbx
