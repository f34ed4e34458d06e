"""The GBSW chain rule by list walk against the same by records: every
contribution is rounded the same way on both, so the bits are equal whatever
the number of shaping entries of a point (the walk remembers four), the
parity of a list's length, the table, and the order that atoms are taken in
(spatial from 40,000 atoms on); and the ordered integrals there against the
counting pass, which takes the atoms as they come."""
import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300._lib import Context
from openmmcustomgbintegralforce_gb300.globule import make_globule
from openmmcustomgbintegralforce_gb300.quadrature import tensor_quadrature
from openmmcustomgbintegralforce_gb300.spec import TABLE_PERIODIC, GBModel, box_for
from oracle import oracle as O

pytestmark = pytest.mark.gpu

F_TOL, I_TOL = 1e-4, 1e-5  # as everywhere in this suite
GRADS = ("forces", "dEdq", "dEdR", "dEdalpha")
SMALL = dict(n_radial=8, lebedev=6)


def rel_rms(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def context(m, q, r, records=True):
    ctx = Context(m, len(q))
    ctx.set_particle_parameters(q, r)
    if not records:
        ctx.set_chain_records(0)
    return ctx


def assert_same(m, pos, q, r):
    a, b = context(m, q, r), context(m, q, r, records=False)
    for _ in range(2):
        Ea, Fa = a.execute_host(pos)
        Eb, Fb = b.execute_host(pos)
        assert Ea == Eb and np.array_equal(Fa, Fb)
        x, y = a.adjoint(pos), b.adjoint(pos)
        assert x["energy"] == y["energy"]
        for k in GRADS:
            assert np.array_equal(x[k], y[k]), k
    assert a.chain_records()["written"] > 0 and b.chain_records()["written"] == -1
    a.close()
    b.close()
    return x


def shaping_counts(m, pos, r):
    """Per quadrature point that no atom buries: the atoms whose shell holds it."""
    v = tensor_quadrature(m.n_radial, m.lebedev, m.r0, m.r1)[0]
    Rp = (r + 0.03) * 0.952
    out = []
    for x in pos:
        gap = np.linalg.norm((x + v)[:, None, :] - pos[None, :, :], axis=2) - Rp
        out.append(np.where((gap <= -m.sw).any(axis=1), 0, (np.abs(gap) < m.sw).sum(axis=1)))
    return np.concatenate(out)


# atoms crowded into one cube: points of one to more than eight shaping atoms
@pytest.mark.parametrize("n", [1, 2, 7, 40, 63])
@pytest.mark.parametrize("name", ["exact", "standalone", "grid"])
def test_crowded_atoms(n, name):
    rng = np.random.default_rng(n)
    pos = rng.uniform(1.0, 1.12, (n, 3)).astype(np.float32).astype(np.float64)
    q, r = rng.normal(size=n), rng.uniform(0.15, 0.17, n)
    m = {"exact": GBModel.charmm_gbsw(), "standalone": GBModel.charmm_gbsw(reference_table=True),
         "grid": GBModel.gbsw_integral()}[name]
    counts = shaping_counts(m, pos, r)
    assert counts.max() >= min(n, 9) and (n == 1 or (counts == 1).any())
    out = assert_same(m, pos, q, r)
    if n > 1:
        ref = O.Oracle(m).energy_forces(pos, q, r, adjoint=True)
        for k in ("forces", "dEdq", "dEdR"):
            assert rel_rms(out[k], ref[k]) < F_TOL, k


@pytest.mark.parametrize("name", ["grid", "grid_cutoff", "minimum_image", "periodic_reference"])
def test_tables_and_images(name):
    g = make_globule(700, seed=19)
    box = box_for(g.positions)
    m = {"grid": GBModel.gbsw_integral(), "grid_cutoff": GBModel.gbsw_integral(cutoff=1.2),
         "minimum_image": GBModel.gbsw_integral(table_mode=TABLE_PERIODIC, box=box, cutoff=1.2, periodic=True),
         "periodic_reference": GBModel.charmm_gbsw(reference_table=True, box=box, cutoff=1.2, periodic=True)}[name]
    assert_same(m, g.positions, g.charge, g.radius)


@pytest.mark.parametrize("n", [39999, 40003])
@pytest.mark.parametrize("name", ["exact", "standalone", "grid"])
def test_items_in_spatial_order(n, name):
    g = make_globule(n, seed=3)
    m = {"exact": GBModel.charmm_gbsw(**SMALL), "standalone": GBModel.charmm_gbsw(reference_table=True, **SMALL),
         "grid": GBModel.gbsw_integral(**SMALL)}[name]
    assert_same(m, g.positions, g.charge, g.radius)
    ctx = context(m, g.charge, g.radius)
    ctx.execute_host(g.positions)
    ctx.execute_host(g.positions)
    I, B = ctx.integrals(), ctx.born_radii()
    ctx.execute_host(g.positions, count_work=True)
    assert np.abs(I - ctx.integrals()).max() < I_TOL * np.abs(I).max()
    assert np.abs(B / ctx.born_radii() - 1).max() < I_TOL
    ctx.close()
