"""Calls whose lookup table outgrew its buffers, on the reference's tables:
an unchecked call lacks the volume terms (every point is solvent) and the next
one reports it, a host call and a checked adjoint evaluate again, and both then
give a fresh context's bits."""
import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300._lib import (EXEC_CHECK, EXEC_ENERGY, EXEC_FORCES, Batch, Context,
                                                     CustomContext, GBXError)
from openmmcustomgbintegralforce_gb300.expression_sets import MODIFIED
from openmmcustomgbintegralforce_gb300.globule import make_globule
from openmmcustomgbintegralforce_gb300.spec import TABLE_GRID, GBModel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BOTH = EXEC_FORCES | EXEC_ENERGY
NONFINITE, TOO_LARGE, STALE = 5, 6, 10
MODELS = {"grid": GBModel.gbsw_integral(), "standalone": GBModel.charmm_gbsw(reference_table=True),
          "gbmv1": GBModel.gbmv1(table_mode=TABLE_GRID), "gbmv2": GBModel.gbmv2(table_mode=TABLE_GRID)}


def context(m, g):
    ctx = Context(m, g.n)
    ctx.set_particle_parameters(g.charge, g.radius)
    return ctx


def device_call(ctx, pos, flags=BOTH):
    """(energy, forces, status) of a call on the current stream's buffers."""
    n = ctx.n
    posq = torch.zeros((n, 4), dtype=torch.float32, device="cuda:0")
    posq[:, :3] = torch.from_numpy(pos).to(posq)
    force = torch.zeros((3, n), dtype=torch.int64, device="cuda:0")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    status = 0
    try:
        ctx.execute_device(posq.data_ptr(), force.data_ptr(), n, energy.data_ptr(), flags, 0)
    except GBXError as e:
        status = e.status
    torch.cuda.synchronize()
    return float(energy), force.T.cpu().numpy() / 2.0 ** 32, status


def spread(g):
    """The atoms 1.6 times as far apart: some four times the cells."""
    c = g.positions.mean(axis=0)
    return c + 1.6 * (g.positions - c)


def far(g):
    """One atom 60 nm away along z: few more atoms per cell, far longer an axis."""
    x = g.positions.copy()
    x[7, 2] += 60.0
    return x


@pytest.mark.parametrize("moved", [spread, far])
@pytest.mark.parametrize("name", list(MODELS))
def test_unchecked_call_lacks_the_volume_terms(name, moved):
    g = make_globule(400, seed=13)
    m = MODELS[name]
    ctx, fresh = context(m, g), context(m, g)
    assert device_call(ctx, g.positions, BOTH | EXEC_CHECK)[2] == 0
    inside = ctx.integrals()
    assert device_call(ctx, g.positions)[2] == 0
    x = moved(g)
    assert device_call(ctx, x)[2] == 0
    # no cell: V = 0 at every point (GBMV-I: 1 / (1 + e^10), from its empty sum), so an
    # integral is that fraction of the quadrature's own sum, to the rounding of
    # 624 to 912 FP32 terms added 32 apart (30 additions of 2^-24: 2e-6 of it);
    # the sums are 1/r0 - 1/r1 and (1/r0^4 - 1/r1^4) / 4, far above any error of the rule
    got = ctx.integrals()
    S = np.array([1 / m.r0 - 1 / m.r1, 0.25 * (m.r0 ** -4 - m.r1 ** -4)])
    covered = 1 / (1 + np.exp(10.0)) if name == "gbmv1" else 0.0
    assert (np.abs(got) < (2e-6 + 1.1 * covered) * S[:, None]).all()
    assert (np.abs(inside).max(axis=1) > 100 * np.abs(got).max(axis=1)).all()
    E, F, status = device_call(ctx, x)  # reported, evaluated checked
    assert status == STALE
    Ef, Ff, _ = device_call(fresh, x, BOTH | EXEC_CHECK)
    assert E == Ef and np.array_equal(F, Ff)
    E, F, status = device_call(ctx, x)
    assert status == 0 and E == Ef and np.array_equal(F, Ff)
    ctx.close()
    fresh.close()


@pytest.mark.parametrize("moved", [spread, far])
@pytest.mark.parametrize("name", list(MODELS))
def test_host_call_and_adjoint_evaluate_again(name, moved):
    g = make_globule(400, seed=14)
    a, b, fresh = (context(MODELS[name], g) for _ in range(3))
    x = moved(g)
    for _ in range(2):
        a.execute_host(g.positions)
        b.adjoint(g.positions)
    n = g.n
    posq = torch.zeros((n, 4), dtype=torch.float32, device="cuda:0")
    posq[:, :3] = torch.from_numpy(x).to(posq)
    out = torch.zeros(3 + 5 * n, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    at = out.data_ptr()
    b.adjoint_device(posq.data_ptr(), at, at + 8, at + 8 * (1 + 3 * n), at + 8 * (1 + 4 * n), at + 8 * (1 + 5 * n),
                     EXEC_CHECK, 0)
    torch.cuda.synchronize()
    want = fresh.adjoint(x)
    got = out.cpu().numpy()
    assert got[0] == want["energy"]
    assert np.array_equal(got[1:], np.concatenate([want[k].reshape(-1) for k in ("forces", "dEdq", "dEdR", "dEdalpha")]))
    E, F = a.execute_host(x)
    Ef, Ff = fresh.execute_host(x)
    assert E == Ef and np.array_equal(F, Ff)
    for c in (a, b, fresh):
        c.close()


# the same table under a user's expressions
def test_compiled_expressions_on_the_grid_table():
    g = make_globule(400, seed=15)
    params = np.stack([g.charge, g.radius, np.ones(g.n)], axis=1)
    x = far(g)

    def make():
        c = CustomContext(MODELS["grid"], g.n, MODIFIED)
        c.set_custom_parameters(params)
        return c

    ctx, fresh = make(), make()
    assert device_call(ctx, g.positions, BOTH | EXEC_CHECK)[2] == 0
    assert device_call(ctx, g.positions)[2] == 0
    assert device_call(ctx, x)[2] == 0
    E, F, status = device_call(ctx, x)
    assert status == STALE
    Ef, Ff, _ = device_call(fresh, x, BOTH | EXEC_CHECK)
    assert E == Ef and np.array_equal(F, Ff)
    ctx.close()
    fresh.close()


# atoms nowhere, or so far away that no grid has an index for them: an error,
# no cell of such a grid is read, and the context goes on
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e20, -1e20])
@pytest.mark.parametrize("which", ["one", "all"])
@pytest.mark.parametrize("name", ["grid", "standalone", "gbmv1", "gbmv2"])
def test_positions_without_a_grid(name, which, bad):
    g = make_globule(200, seed=16)
    ctx = context(MODELS[name], g)
    E, F, status = device_call(ctx, g.positions, BOTH | EXEC_CHECK)
    assert status == 0
    x = g.positions.copy()
    if which == "one":
        x[3, 1] = bad
    else:
        x[:] = bad
    # the extents leave out one position that is not a number, and atoms all at
    # one place have a grid wherever that is
    grid = np.isnan(bad) if which == "one" else np.isfinite(bad)
    for _ in range(2):
        assert device_call(ctx, x, BOTH | EXEC_CHECK)[2] in ((0, NONFINITE) if grid else (TOO_LARGE,))
        device_call(ctx, x)  # unchecked: reported by the next call
    # nor may such atoms size a table (a grid of one cell is not taken for one then)
    fresh = context(MODELS[name], g)
    assert device_call(fresh, x)[2] in ((0, NONFINITE, TOO_LARGE) if grid else (TOO_LARGE,))
    assert device_call(fresh, g.positions)[1].shape == F.shape
    fresh.close()
    device_call(ctx, g.positions, BOTH | EXEC_CHECK)
    E2, F2, status = device_call(ctx, g.positions, BOTH | EXEC_CHECK)
    assert status == 0 and E2 == E and np.array_equal(F2, F)
    ctx.close()


# a call that evaluates again has dealt with its table: the next call has
# nothing to report, unless an unchecked one before was not reported yet
@pytest.mark.parametrize("due", [False, True])
@pytest.mark.parametrize("entry", ["host", "adjoint", "batch", "batch_adjoint"])
@pytest.mark.parametrize("name", ["exact", "grid", "gbmv2"])
def test_a_call_that_evaluated_again_leaves_nothing_to_report(name, entry, due):
    g = make_globule(400, seed=18)
    m = MODELS.get(name, GBModel.charmm_gbsw())
    fresh = context(m, g)
    batch = Batch([m, m], [g.n, g.n]) if entry.startswith("batch") else None
    ctx = batch.molecules[1] if batch else Context(m, g.n)
    for c in batch.molecules if batch else [ctx]:
        c.set_particle_parameters(g.charge, g.radius)

    def call(pos):
        if batch:
            x = np.concatenate([g.positions, pos])
            batch.adjoint_host(x) if entry == "batch_adjoint" else batch.execute_host(x)
        elif entry == "host":
            ctx.execute_host(pos)
        else:
            n = g.n
            posq = torch.zeros((n, 4), dtype=torch.float32, device="cuda:0")
            posq[:, :3] = torch.from_numpy(pos).to(posq)
            out = torch.zeros(1, dtype=torch.float64, device="cuda:0")
            torch.cuda.synchronize()
            ctx.adjoint_device(posq.data_ptr(), out.data_ptr(), 0, 0, 0, 0, EXEC_CHECK, 0)

    for _ in range(2):
        call(g.positions)
    assert device_call(ctx, g.positions)[2] == 0
    if due:
        # in between in size, so that the call below outgrows the same buffers
        assert device_call(ctx, spread(g))[2] == 0
    call(spread(g))
    E, F, status = device_call(ctx, g.positions)
    assert status == (STALE if due else 0)
    Ef, Ff, _ = device_call(fresh, g.positions, BOTH | EXEC_CHECK)
    assert E == Ef and np.array_equal(F, Ff)
    assert device_call(ctx, spread(g))[2] == 0
    (batch or ctx).close()
    fresh.close()


def blown(g):
    """Some 10^27 cells."""
    return g.positions * 1e8


# an outgrown table has no lists to return, however many cells it wanted
@pytest.mark.parametrize("name,moved", [(k, f) for k in ("grid", "standalone", "gbmv2") for f in (spread, far, blown)
                                        if k == "standalone" or f is not blown])
def test_no_table_where_it_outgrew_its_buffers(name, moved):
    g = make_globule(400, seed=20)
    ctx = context(MODELS[name], g)
    assert device_call(ctx, g.positions, BOTH | EXEC_CHECK)[2] == 0
    assert device_call(ctx, moved(g))[2] == 0
    with pytest.raises(GBXError) as e:
        ctx.lookup_table()
    assert e.value.status == STALE
    assert device_call(ctx, g.positions)[2] == STALE
    assert ctx.lookup_table()["counts"].sum() > 0
    ctx.close()
