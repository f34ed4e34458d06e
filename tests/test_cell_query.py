"""The reference table's cell query (csrc/queries.cuh), compiled for the CPU:
the FP32 form gives the FP64 form's cell, and a table that outgrew its
buffers, in cells or in entries, gives none, in each table mode and however
far the points lie."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300.spec import TABLE_GRID, TABLE_PERIODIC, TABLE_STANDALONE

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(NVCC))), "include")

MODES = {"standalone": TABLE_STANDALONE, "grid": TABLE_GRID, "periodic": TABLE_PERIODIC}


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cells") / "cell_query.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-frounding-math", "-ffp-contract=off", "-fPIC", "-shared", "-w",
                    "-I", CUDA_INCLUDE, "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(REPO, "openmmcustomgbintegralforce_gb300", "csrc"),
                    os.path.join(HERE, "cell_query.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.grid_of.restype = ctypes.c_longlong
    return lib


def query(lib, mode, lo, step, dims, x, off, cells=None, entries=0, total=0, reach=2.0):
    """(FP32 query's cells, FP64 query's cells); by default every cell is allocated."""
    a = lambda v, t: np.ascontiguousarray(v, dtype=t)  # noqa: E731
    lo, step, off, x = a(lo, np.float64), a(step, np.float64), a(off, np.float64), a(x, np.float32)
    dims = a(dims, np.int32)
    n = len(off)
    got, exact = np.zeros(n, np.int64), np.zeros(n, np.int64)
    p = lambda v: v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    ll = ctypes.c_longlong
    lib.query_cells(mode, p(lo), p(step), p(dims), ctypes.c_double(reach),
                    ll(int(np.prod(dims.astype(np.int64))) if cells is None else cells), ll(entries), ll(total), p(x),
                    p(off), n, p(got), p(exact))
    return got, exact


def points(rng, n, reach=2.0):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True) * rng.uniform(0.05, reach, (n, 1))


@pytest.mark.parametrize("mode", list(MODES))
def test_the_fp32_query_gives_the_fp64_query_s_cell(lib, mode):
    rng = np.random.default_rng(3)
    inside = 0
    for _ in range(200):
        dims = rng.integers(1, 60, 3)
        lo, step = rng.uniform(-5, 5, 3), np.full(3, 0.15)
        x = lo + rng.uniform(-0.2, 1.2, 3) * dims * step  # atoms on and off the grid
        off = points(rng, 400)
        # some points exactly on cell faces and grid edges
        face = lo + rng.integers(0, dims + 1, (100, 3)) * step
        off[:100] = face - x.astype(np.float32).astype(np.float64)
        got, exact = query(lib, MODES[mode], lo, step, dims, x, off, reach=float(np.abs(off).max()) * 2)
        assert np.array_equal(np.maximum(got, -1), np.maximum(exact, -1))
        inside += int((exact >= 0).sum())
    assert inside > 1000


@pytest.mark.parametrize("short", ["cells", "entries"])
@pytest.mark.parametrize("mode", list(MODES))
def test_an_outgrown_table_gives_no_cell(lib, mode, short):
    rng = np.random.default_rng(5)
    for dims in [(30, 31, 32), (20, 20, 7000), (1, 1, 1)]:
        ncell = int(np.prod(dims))
        lo, step = np.array([-1.0, 0.5, 2.0]), np.full(3, 0.15)
        for z in (0.01, 0.5, 0.99, -0.3, 1.3):
            x = lo + np.array([0.4, 0.6, z]) * dims * step
            room = dict(cells=ncell - 1) if short == "cells" else dict(entries=99, total=100)
            got, _ = query(lib, MODES[mode], lo, step, dims, x, points(rng, 300), **room)
            assert (got < 0).all(), (dims, z)



def grid_of(lib, steps):
    dims, status = (ctypes.c_int * 3)(), ctypes.c_uint()
    ncell = lib.grid_of((ctypes.c_double * 3)(*steps), dims, ctypes.byref(status))
    return list(dims), ncell, status.value


TABLE_CELLS = 1  # status: the grid has more cells than are allocated


# lengths in grid steps, with the largest that an index still holds
@pytest.mark.parametrize("steps", [(0.0, 0.4, 1.0), (19.99, 20.0, 20.01), (1.0, 2147483646.0, 3.5), (2.0 ** 30,) * 3])
def test_grids_that_exist(lib, steps):
    dims, ncell, status = grid_of(lib, steps)
    assert dims == [int(np.ceil(s)) + 1 for s in steps] and status == 0
    assert ncell == min(int(np.prod([int(d) for d in dims], dtype=object)), 2 ** 62)


# no grid: atoms out of any range, or nowhere
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 2147483646.5, 1e20, 1e300, -1.0])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_grids_that_do_not_exist(lib, axis, bad):
    steps = [20.0, 21.0, 22.0]
    steps[axis] = bad
    dims, ncell, status = grid_of(lib, steps)
    assert status == TABLE_CELLS and min(dims) == 1 and ncell == np.prod(dims)
