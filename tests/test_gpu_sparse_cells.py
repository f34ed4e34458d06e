"""GBMV on grids with many more cells than atoms, whose chain rule takes the
cells in a loop: a context that was sized in a wide box keeps its buffers in a
narrow one and so runs the loop on the table that a context of its own runs a
block per cell on, with the same bits; and wide boxes against the oracle."""
import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300._lib import Context
from openmmcustomgbintegralforce_gb300.globule import make_globule
from openmmcustomgbintegralforce_gb300.spec import GBModel, box_for
from oracle import oracle as O

pytestmark = pytest.mark.gpu

E_TOL, F_TOL, I_TOL = 2e-5, 1e-4, 1e-5  # as everywhere in this suite
GRADS = ("forces", "dEdq", "dEdR", "dEdalpha")


def rel_rms(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def context(m, g):
    ctx = Context(m, g.n)
    ctx.set_particle_parameters(g.charge, g.radius)
    return ctx


# the loop is taken above 65,536 allocated cells and 40 an atom; a box of 12 nm
# has 531,441 cells
@pytest.mark.parametrize("kw", [{}, dict(cutoff=1.0, periodic=True)], ids=["plain", "periodic"])
@pytest.mark.parametrize("n", [2, 33, 600, 1500])
@pytest.mark.parametrize("name", ["gbmv1", "gbmv2"])
def test_the_loop_gives_the_bits_of_a_block_per_cell(name, n, kw):
    g = make_globule(n, seed=n)
    narrow = box_for(g.positions)
    a, b = context(getattr(GBModel, name)(box=(12.0,) * 3, **kw), g), context(getattr(GBModel, name)(box=narrow, **kw), g)
    a.execute_host(g.positions)
    a.adjoint(g.positions)
    a.set_box(narrow)
    for _ in range(2):
        Ea, Fa = a.execute_host(g.positions)
        Eb, Fb = b.execute_host(g.positions)
        assert Ea == Eb and np.array_equal(Fa, Fb)
    x, y = a.adjoint(g.positions), b.adjoint(g.positions)
    assert x["energy"] == y["energy"]
    for k in GRADS:
        assert np.array_equal(x[k], y[k]), k
    a.close()
    b.close()


# in 10 nm a warp has nine or ten of the 314,432 cells to look at, in 30 nm 248
@pytest.mark.parametrize("n,side", [(2, 10.0), (2, 30.0), (120, 10.0), (120, 30.0)])
@pytest.mark.parametrize("name", ["gbmv1", "gbmv2"])
def test_wide_boxes(name, n, side):
    g = make_globule(n, seed=7)
    pos = g.positions.astype(np.float32).astype(np.float64)
    m = getattr(GBModel, name)(box=(side,) * 3)
    ctx = context(m, g)
    ref = O.Oracle(m).energy_forces(pos, g.charge, g.radius, adjoint=True)
    E, F = ctx.execute_host(pos)
    out = ctx.adjoint(pos)
    assert np.abs(ctx.integrals() - ref["integrals"]).max() < I_TOL * np.abs(ref["integrals"]).max()
    assert abs(E / ref["energy"] - 1) < E_TOL and abs(out["energy"] / ref["energy"] - 1) < E_TOL
    assert rel_rms(F, ref["forces"]) < F_TOL
    for k in ("forces", "dEdq", "dEdR"):
        assert rel_rms(out[k], ref[k]) < F_TOL, k
    ctx.close()
