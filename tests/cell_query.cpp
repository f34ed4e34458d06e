// The reference table's cell query on the CPU, for the tests that compare it
// with its FP64 form and with the cells that are allocated.
#include "device_on_host.h"

#include "queries.cuh"

// Cells of `n` quadrature points (offsets off [3 n], FP64) of an atom at x in a
// grid of the given geometry, of which `cell_cap` cells and `entry_cap` entries
// are allocated and `total` entries needed: the query's, and the FP64 form's.
extern "C" void query_cells(int mode, const double* lo, const double* step, const int* dims, double reach,
                            long long cell_cap, long long entry_cap, long long total, const float* x,
                            const double* off, int n, long long* cell, long long* exact) {
  gbx::TableGeom g{};
  for (int k = 0; k < 3; ++k) {
    g.min[k] = lo[k];
    g.step[k] = step[k];
    g.dims[k] = dims[k];
    g.max[k] = lo[k] + (mode == GBX_TABLE_PERIODIC ? dims[k] : dims[k] - 1) * step[k];
    g.box[k] = mode == GBX_TABLE_PERIODIC ? dims[k] * step[k] : 0.0;
    g.inv_step[k] = 1.0 / step[k];
    g.inv_box[k] = g.box[k] > 0.0 ? 1.0 / g.box[k] : 0.0;
  }
  g.mode = mode;
  g.reach = reach;
  g.ncell = (long long)dims[0] * dims[1] * dims[2];
  g.total = total;
  gbx::Entries t{};
  t.geom = &g;
  t.cell_cap = cell_cap;
  t.entry_cap = entry_cap;
  const float4 xi = make_float4(x[0], x[1], x[2], 0.f);
  gbx::RefQuery query;
  query.init(t, xi, off);
  for (int q = 0; q < n; ++q) {
    const float4 v = make_float4((float)off[3 * q], (float)off[3 * q + 1], (float)off[3 * q + 2], 0.f);
    cell[q] = query.cell(xi, v, q);
    exact[q] = gbx::query_exact(g, xi, off, q);
  }
}

// The grid of three axes of `steps` grid steps: its dims, its cells, the status.
extern "C" long long grid_of(const double* steps, int* dims, unsigned* status) {
  *status = 0u;
  for (int k = 0; k < 3; ++k) dims[k] = gbx::axis_cells(steps[k], *status);
  return gbx::grid_cells(dims);
}
