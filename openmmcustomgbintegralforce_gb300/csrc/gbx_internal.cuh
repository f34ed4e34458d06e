// Internal types shared by the gbx CUDA translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "gbx.h"
#include "gbx_custom.h"

namespace gbx {

constexpr int kWarp = 32;
constexpr double kFixedScale = 4294967296.0;  // 2^32, OpenMM's force fixed-point scale
constexpr int kMaxSortSegment = 2048;         // longest cell list the sort handles
constexpr int kMaxSortCells = 1 << 17;        // cells of the spatial order

// Device status bits (context->d_status).
enum : unsigned {
  kStatusTableCells = 1u,     // grid has more cells than allocated
  kStatusTableEntries = 2u,   // more list entries than allocated
  kStatusSegmentTooLong = 4u, // a cell list exceeded kMaxSortSegment
  kStatusNonFinite = 8u,      // NaN/Inf Born radius
  kStatusTimeout = 16u,       // bounded device wait expired
};

// Status of the device calls, published by the last kernel of every call
// into mapped host memory (monotone counters; seq written last).
struct StatusRecord {
  unsigned long long seq;          // calls published
  unsigned long long overflows;    // calls whose lookup table outgrew its buffers
  unsigned long long nonfinite;    // calls with a non-finite Born radius
  unsigned long long max_cells;    // largest table geometry seen (cells)
  unsigned long long max_entries;  // largest list-entry total seen
};

// Lookup-table geometry, computed on the device each step.
struct TableGeom {
  double min[3];
  double max[3];
  double step[3];
  double box[3];
  double inv_step[3];  // 1 / step and 1 / box (0 without a box), for the FP32
  double inv_box[3];   // queries: formed once here, not per lane in FP64
  double pad;       // standalone uniform pad
  double L;         // periodic: max(step)
  double reach;     // the quadrature's outer radius: no point is farther from its atom
  int dims[3];
  int mode;
  long long ncell;
  long long total;  // list entries before capping (even per list where lists are read in pairs)
  int longest;       // longest list, where one is longer than its bucket (else 0)
  unsigned chained;  // list members outside their cell's bucket
};

// Grid of the atoms' spatial order (k_pair.cu).
struct SortGeom {
  float lo[3];
  float inv_cell;
  int dims[3];
  int ncell;
};

// Where a table's members are collected (buckets.cuh).
struct TableBuckets {
  int* slots = nullptr;   // [cell_cap][size]
  int size = 0;
  int* chain = nullptr;   // [cell_cap] members past the bucket, as a list of nodes
  int2* node = nullptr;   // [entry_cap]
};

// GBSW tables, per cell: the list's first (sorted) entry and the cell's
// (count or -1 if buried, start) record, read together by one 32-byte load.
struct __align__(32) TightCell {
  float4 first;
  int2 cs;
  int2 pad;
};

// Two consecutive 16-byte entries at a 32-byte aligned address in one
// 256-bit non-coherent load (sm_100 and later).
struct __align__(32) Float4x2 {
  float4 a, b;
};
__device__ __forceinline__ Float4x2 ldg_pair(const void* p) {
  Float4x2 r;
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w)
      : "l"(p));
  return r;
}

// Per-model constants used inside the kernels (FP32 hot path + FP64 exact paths).
struct ModelConst {
  int model;
  int table_mode;
  int cap;
  int skip_empty;
  int nq;
  unsigned nq_magic;         // point_atom: ceil(2^(31 + L) / nq) with 2^(L - 1) < nq <= 2^L
  int nq_shift;              // L - 1
  int nrad;                  // radial points per direction (index = direction * nrad + radial)
  int cutoff_chain_quirk;
  float sw, c1, c3;          // GBSW: u = 1/2 + c1 dr - c3 dr^3, c1 = 3/(4w), c3 = 1/(4w^3)
  float gamma0_lnlambda;     // GBMV-I gamma_j = gamma0 ln(lambda) / R^4
  float beta, lambda, s0;    // GBMV
  float p1, p2;              // GBMV-II
  float cutoff2;             // pair cutoff squared (<= 0: none)
  float pref;                // pair prefactor
  double h, buffer, cutoff;
  // p / nq for a point id below 2^31 (exact: the magic's excess times p stays below 2^(31 + L))
  __device__ __forceinline__ int point_atom(int p) const {
    return nq > 1 ? (int)(__umulhi((unsigned)p, nq_magic) >> nq_shift) : p;
  }
};

// One evaluation context (one force instance).
struct Context {
  gbx_config cfg{};
  int n = 0;
  int device = 0;
  int sms = 0;  // multiprocessors of `device` (grid sizing), read once at creation
  std::string last_error;

  // quadrature (host, FP64) and device copies
  std::vector<double> q_off, q_rad, q_w;  // [Q*3], [Q], [Q]
  double S4 = 0, S7 = 0;                  // sum_q w/r^2, sum_q w/r^5 (FP64)
  double C4 = 0, C7 = 0;                  // 1/r0 - S4, 1/(4 r0^4) - S7
  float4* d_qv = nullptr;                 // (vx, vy, vz, r) FP32
  float2* d_qw = nullptr;                 // (w/r^2, w/r^5) FP32
  double* d_qoff = nullptr;               // FP64 offsets for the exact cell query

  // particle data
  std::vector<double> charge, radius;
  unsigned char* d_params = nullptr;  // one block: the four arrays below
  double* d_radius = nullptr;  // FP64 radii (table geometry)
  float* d_charge = nullptr;
  float2* d_par = nullptr;     // secondary model parameters per atom
  float* d_wpar = nullptr;     // main model parameter (staged into pos.w)
  float alpha0 = 0, alpha1 = 0;

  // table
  TableGeom* d_geom = nullptr;
  long long cell_cap = 0, entry_cap = 0;
  int* d_cell_count = nullptr;   // uncapped count -> final (capped) count
  int* d_cell_start = nullptr;   // [cell_cap+1]
  TableBuckets buckets;
  int2* d_cell2 = nullptr;       // [cell_cap] (capped count, start) for the volume kernels
  int* d_entries = nullptr;      // [entry_cap] atom indices, ascending per cell
  float4* d_entry4 = nullptr;    // [entry_cap] inline copies (x, y, z, main parameter; GBSW: as pairs)
  float2* d_entry_par = nullptr; // GBMV: [entry_cap] inline secondary parameters
  int* d_entry_index = nullptr;  // GBSW: [entry_cap] atom of each inline entry (likeliest burying atom first)
  TightCell* d_rfirst = nullptr; // GBSW: [cell_cap] the cell's first inline entry and record
  void* d_parts = nullptr;       // partial extents of the call's first kernel
  unsigned* d_ticket = nullptr;  // its count of finished blocks (0 between calls)
  bool table_valid = false;

  // exact GBSW table (GBX_TABLE_POLICY_AUTO on a standalone table):
  // count[c] = -1 marks a cell every point of which is buried
  bool use_tight = false;
  bool tight_eligible = false;   // GBSW on a standalone table with the AUTO policy
  double tight_h = 0.1;
  TableGeom* d_tgeom = nullptr;
  TableGeom* d_wgeom = nullptr;  // periodic: the reference's standalone grid (its edges decide the move)
  long long tcell_cap = 0, tentry_cap = 0;
  int* d_tcount = nullptr;
  int* d_tstart = nullptr;
  TableBuckets tbuckets;
  int* d_tburied = nullptr;
  int2* d_tcell = nullptr;       // (count or -1 if buried, start)
  TightCell* d_tfirst = nullptr; // per cell: first entry and (count, start)
  float4* d_tentry = nullptr;    // (x, y, z, R') per list entry; lists start at even entries
  int* d_tindex = nullptr;       // atom index per list entry
  bool tight_valid = false;

  // per-step state
  float4* d_pos = nullptr;       // internal positions (x, y, z, 0)
  int n_chunks = 0;              // quadrature chunks per atom
  float* d_J = nullptr;          // [2][n_chunks][n] FP32 partial integrals
  double* d_born = nullptr;      // [n]
  float* d_bornf = nullptr;      // [n] (B, 1/B interleaved as float2)
  double* d_dBdJ = nullptr;      // [6n]: dB/dJ [2n], dB/dalpha [2n], adjoint alpha terms [2n]
  double* d_integrals = nullptr; // [2n]  I4, I7
  unsigned long long* d_dEdB_fx = nullptr;  // [n] fixed point
  float2* d_dEdJ = nullptr;      // [n]
  double* d_energy_part = nullptr;  // [energy_parts] per-CTA energy partials
  int energy_parts = 0;
  unsigned long long* d_energy_fx = nullptr;  // pair energy, fixed point (2^-32)
  float4* d_tile_box = nullptr;               // cutoff: bounding box of each 32-atom tile
  int* d_perm = nullptr;                      // cutoff: atoms in spatial order, ascending per cell [n]
  int* d_perm_tmp = nullptr;                  // atoms in spatial order, any order within a cell [n]
  int* d_cell_of = nullptr;                   // spatial cell of each atom [n]
  int* d_scount = nullptr;                    // atoms per spatial cell [kMaxSortCells]
  int* d_sstart = nullptr;
  int* d_scursor = nullptr;
  SortGeom* d_sgeom = nullptr;                  // spatial grid geometry
  float* d_pstate = nullptr;                  // GBMV: per-point sums kept for the chain rule
  // GBMV points binned by lookup-table cell (k_gbmv.cu)
  int2* d_pat = nullptr;                      // [n Q] (the point's cell or -1, slot within the cell)
  int* d_porder = nullptr;                    // [n Q] point id per slot
  float* d_sval = nullptr;                    // [n Q] solvent fraction by point id
  int* d_pcount = nullptr;                    // [cell_cap] points per cell
  int* d_plive = nullptr;                     // [cell_cap] of those, the chain rule's
  int* d_pstart = nullptr;                    // [cell_cap + 1] first slot per cell
  unsigned long long* d_ptotal = nullptr;     // [1] points binned
  bool gbmv_cells = false;                    // this call's GBMV passes run by cell
  CustomPlan* custom = nullptr;               // expressions outside the canonical set (gbx_custom.cu)
  unsigned long long* d_force_fx = nullptr;  // internal force buffer [3n] (host path)
  unsigned long long* d_f4 = nullptr;  // [4n] the chain rule's force (x, y, z) and dE/dR per atom
  double* d_energy = nullptr;     // internal energy (host path)
  unsigned long long* d_dEdR_fx = nullptr;  // adjoint [n]
  unsigned long long* d_dEdq_fx = nullptr;  // adjoint [n]
  double* d_alpha_grad = nullptr; // adjoint [2]
  unsigned* d_status = nullptr;
  unsigned long long* d_work = nullptr;  // [4] evaluation counters

  // GBSW chain-rule records (q, V, shaping-entry mask) of the points an atom
  // other than i shapes, written by the integral pass: warp w (atom,
  // quadrature chunk) owns records [w R, (w + 1) R)
  bool records = false;          // this call writes and reads records
  bool records_self = false;     // ... of atom i's own entries too (the adjoint)
  bool srec_manage = false;      // this call may size the regions (automatic, not under capture)
  bool srec_auto = true;         // size R from the largest need seen
  int4* d_srec = nullptr;
  int* d_srec_st = nullptr;      // the recorded point's list start, beside each record
  int srec_R = 0;                // records per warp (0: no buffer)
  long long srec_warps = 0;      // warps the buffer was sized for
  int* d_rcount = nullptr;       // [warps] records written, or -1 - needed
  unsigned* d_rmax = nullptr;    // largest per-warp need of the call
  unsigned* d_next_item = nullptr;  // the GBSW integral pass's (atom, chunk) work counter
  int integral_grid = 0;            // its persistent grid: resident blocks on all SMs
  unsigned* h_rmax = nullptr;    // pinned copy of the last d_rmax
  unsigned* h_status = nullptr;  // pinned: status word of the last host-path call
  double* h_energy = nullptr;    // pinned: energy of the last host-path call
  cudaEvent_t srec_ev = nullptr;
  bool srec_pending = false;     // srec_ev recorded and not yet read
  cudaEvent_t last_ev = nullptr; // the last unchecked call's work (mark_enqueued)
  bool have_result = false;

  long long launches = 0;  // kernels this context has launched

  // CUDA graph of the unchecked device call, replayed while its arguments
  // (buffers, flags, stream) stay the same; dropped by every setter and
  // every reallocation
  cudaGraphExec_t graph = nullptr;
  long long graph_kernels = 0;  // kernels one replay launches
  cudaGraphExec_t host_graph = nullptr;  // the host-buffer call: upload, evaluation, readback
  long long host_graph_kernels = 0;
  int host_graph_forces = -1;            // whether the captured call reads forces back
  unsigned long long epoch = 0; // bumped whenever captured arguments may change
                                // (setters, reallocation): graphs that hold this
                                // context's launches (its own, a batch's) are stale
  struct GraphKey {
    const void* posq = nullptr;
    const void* force = nullptr;
    int stride = 0;
    const void* energy = nullptr;
    int flags = 0;
    cudaStream_t stream = nullptr;
    bool operator==(const GraphKey& o) const {
      return posq == o.posq && force == o.force && stride == o.stride && energy == o.energy && flags == o.flags &&
             stream == o.stream;
    }
  } graph_key;

  // optional per-stage timing (CUDA events on the execute stream)
  bool timing = false;
  static constexpr int kStages = 9;
  cudaEvent_t ev[kStages + 1] = {};

  // caller-facing layout of the device call
  int* d_slot_of = nullptr;       // internal atom i -> the caller's slot (gbx_set_atom_order)
  bool in_permuted = false;       // this call reads and writes through d_slot_of
  bool in_double = false;         // this call's positions are double4

  // status of unchecked device calls, read without synchronising
  unsigned long long* d_pub = nullptr;  // [5] device-side counters of StatusRecord
  StatusRecord* h_pub = nullptr;        // mapped pinned record
  StatusRecord* h_pub_dev = nullptr;    // its device address
  unsigned long long pub_seen_overflows = 0, pub_seen_nonfinite = 0;

  // host staging
  float4* h_pos = nullptr;                 // pinned
  unsigned long long* h_force_fx = nullptr; // pinned
  cudaStream_t own_stream = nullptr;  // created and destroyed by the context
  cudaStream_t stream = nullptr;      // stream of the current call (the caller's or own_stream)
};

// --------------------------------------------------------------------------
// Device helpers
// --------------------------------------------------------------------------

// round(v * 2^32) as a 64-bit integer.  Scaling by a power of two is exact
// in FP32, so converting the float directly gives the same integer as the
// FP64 route without touching the (slow) FP64 pipe.
__device__ __forceinline__ long long float_to_fixed(float v) { return __float2ll_rn(v * 4294967296.0f); }

// Fixed point from two 32-bit conversions (|v| < 2^31): floor(v) 2^32 +
// round((v - floor(v)) 2^32), the fraction formed in FP32.  For v >= 0 and
// v <= -1/2 the fraction is exact and the result is round(v 2^32), the
// integer float_to_fixed gives; for -1/2 < v < 0 the fraction 1 + v is first
// rounded to FP32 (a multiple of 2^-24), so the result can differ from
// round(v 2^32) by up to 2^7 units: an absolute error of at most 2^-25
// (3e-8 in force units) per contribution.  Deterministic; cheaper where
// conversions dominate (the chain rule's force pushes: an exact form on |v|
// measured 13 % slower in the GBMV chain).
__device__ __forceinline__ long long float_to_fixed_split(float v) {
  const float hf = floorf(v);
  const unsigned lo = __float2uint_rn((v - hf) * 4294967296.0f);
  return (long long)(((unsigned long long)(long long)__float2int_rz(hf) << 32) + lo);
}

// Hardware 1/sqrt(x) (PTX rsqrt.approx, relative error below 2^-22;
// subnormal inputs flush to zero).
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void red_add_fixed(unsigned long long* addr, float v) {
  atomicAdd(addr, (unsigned long long)float_to_fixed(v));
}

__device__ __forceinline__ void red_add_fixed_d(unsigned long long* addr, double v) {
  long long q = __double2ll_rn(v * kFixedScale);
  atomicAdd(addr, (unsigned long long)q);
}

__host__ __device__ __forceinline__ double fixed_to_double(unsigned long long v) {
  return (double)(long long)v / kFixedScale;
}

// --------------------------------------------------------------------------
// Launchers (implemented in the k_*.cu files); all enqueue on ctx->stream.
// --------------------------------------------------------------------------

// Whole evaluation on ctx->stream (gbx_api.cu); used by the batch.
gbx_status pipeline(Context* ctx, const float4* posq, unsigned long long* force, int stride, double* energy, bool check,
                    bool adjoint, bool count_work, bool forces);
gbx_status set_chunks(Context* ctx, int chunks);
// For a call whose first, unchecked run outgrew its table (status st, read back)
// and that evaluates again: what that run published is settled within the call,
// so that no later call reports it.  What calls before it published stays due.
void settle_published(Context* ctx, unsigned st);
gbx_status fix_chain_records(Context* ctx);
// Whether the exact GBSW table serves this context's configuration and
// parameters (a periodic one needs the standalone grid's reach below half
// the shortest box edge); switching drops graphs and tables.
void choose_table(Context* ctx);

// The call's first kernel: positions staged, the accumulators cleared, the
// grids of the exact and / or the reference table.  call: false builds a
// table alone, outside an evaluation (the last call's results stay).
gbx_status launch_prepare(Context* ctx, const void* posq, bool tight, bool reference, bool call);
size_t prepare_scratch_bytes(int n);
gbx_status launch_finish_outputs(Context* ctx, unsigned long long* force, int stride, float* energy_float);
// The call's last kernel: the chain rule's sums added to the force buffer
// (and dE/dR), the energy, the published status.
gbx_status launch_finish(Context* ctx, unsigned long long* force, int stride, double* energy, bool chain, bool adjoint);
gbx_status launch_table_build(Context* ctx, const float4* pos);
gbx_status launch_tight_build(Context* ctx, const float4* pos);
// GBMV on a table the cell passes serve: bins the quadrature points by
// cell (the cell passes' data layout); nothing otherwise.
gbx_status launch_binning(Context* ctx, const float4* pos, bool count_work);
gbx_status launch_integrals(Context* ctx, const float4* pos, bool count_work);
gbx_status launch_born(Context* ctx);
gbx_status launch_pair(Context* ctx, const float4* pos, unsigned long long* force, int stride, bool adjoint);
int pair_energy_parts(int n, int segments);
int pair_segments(int n, int sms);
ModelConst make_model_const(const Context* ctx);
// The atoms in spatial order: for the cutoff pair term's tiles (d_perm, sorted
// within a cell), and for the GBSW integrals and chain rule (d_perm_tmp, any
// order within a cell), whose running warps then share a part of the table.
// That pays once the table (some 2.6 KB an atom) crowds the 129 MB L2, or where
// the pair term needs the order anyway.  Forming it takes 17 us; whole calls
// without and with it, all pairs: 20,000 atoms, 32 x 110 points 1,385 and 1,400
// us, 30,000 2,201 and 2,195, 40,000 3,160 and 3,084, 50,000 4,242 and 4,061 (24 x
// 38 points 1,093 and 1,109 at 30,000, 1,629 and 1,630 at 40,000, 2,265 and 2,239
// at 50,000); 1.5 nm cutoff, 10,000 atoms 342 and 338, 50,000 1,515 and 1,466.
constexpr int kOrderAtoms = 40000;
inline bool pair_in_order(const Context* ctx) { return ctx->cfg.cutoff > 0 && !ctx->cfg.periodic && !ctx->custom; }
inline bool items_in_order(const Context* ctx) {
  return ctx->cfg.model == GBX_MODEL_GBSW && (ctx->n >= kOrderAtoms || pair_in_order(ctx));
}
gbx_status launch_spatial_order(Context* ctx, const float4* pos);

// The GBSW chain rule forms dE/dJ itself: no launch_chain_prep (compiled
// expressions and the adjoint, which needs more from it, go through memory).
bool chain_forms_dEdJ(const Context* ctx, bool adjoint);
gbx_status launch_chain_prep(Context* ctx, bool adjoint);
gbx_status launch_chain(Context* ctx, const float4* pos, bool adjoint);
bool gbmv_cells_apply(const Context* ctx);
gbx_status launch_gbmv_cells_bin(Context* ctx, const float4* pos, const ModelConst& m);
gbx_status launch_gbmv_cells_integral(Context* ctx, const float4* pos, const ModelConst& m);
gbx_status launch_gbmv_cells_chain(Context* ctx, const float4* pos, const ModelConst& m, bool adjoint);
gbx_status launch_adjoint_out(Context* ctx, double* energy, double* forces, double* dEdq, double* dEdR,
                              double* dEdalpha);

}  // namespace gbx
