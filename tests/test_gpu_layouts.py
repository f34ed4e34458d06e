"""Sizes and shapes at which the table, pair, quadrature and adjoint kernels
change path: list lengths around the register sorts, grids too fine for the
shared-memory axis values, partial and single pair tiles, odd quadrature
rules, points that leave the box, the adjoint on records and on lists, inside
a captured graph and after its table outgrew the buffers."""
import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300._lib import EXEC_CHECK, Context
from openmmcustomgbintegralforce_gb300.globule import jitter, make_globule
from openmmcustomgbintegralforce_gb300.spec import GBModel, box_for
from oracle import oracle as O

pytestmark = pytest.mark.gpu

E_TOL = 2e-5  # FP32 terms of an energy, forces and integrals against FP64,
F_TOL = 1e-4  # as everywhere in this suite
I_TOL = 1e-5
GRADS = ("forces", "dEdq", "dEdR", "dEdalpha")


def rel_rms(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def context(model, g_or_qr):
    q, r = g_or_qr if isinstance(g_or_qr, tuple) else (g_or_qr.charge, g_or_qr.radius)
    ctx = Context(model, len(q))
    ctx.set_particle_parameters(q, r)
    return ctx


def assert_table(ctx, model, pos, radius):
    t, ref = ctx.lookup_table(), O.Oracle(model).table(pos, radius)
    assert np.array_equal(t["dims"], ref["dims"])
    assert np.array_equal(t["counts"], ref["counts"])
    assert np.array_equal(t["atoms"], ref["atoms"])
    return ref["counts"]


# atoms crowded into one cube of 0.3 nm: lists of up to `n` entries, on both
# sides of the register sorts'
# 32, 64 and 128, and past the 64-entry cap of the integral classes
@pytest.mark.parametrize("n", [31, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("name", ["standalone", "grid", "periodic"])
def test_list_lengths(n, name):
    rng = np.random.default_rng(n)
    pos = rng.uniform(1.0, 1.3, (n, 3))
    pos = pos.astype(np.float32).astype(np.float64)
    r = rng.uniform(0.12, 0.2, n)
    q = rng.normal(size=n)
    m = {"standalone": GBModel.charmm_gbsw(reference_table=True), "grid": GBModel.gbsw_integral(),
         "periodic": GBModel.gbmv2(box=(3.0, 3.0, 3.0))}[name]
    ctx = context(m, (q, r))
    ctx.execute_host(pos)
    assert assert_table(ctx, m, pos, r).max() >= min(n, m.cap or n) * 0.9
    ref = O.Oracle(m).integrals(pos, r)[0]
    assert np.abs(ctx.integrals() - ref).max() < I_TOL * np.abs(ref).max()
    ctx.close()


# 96 grid values per axis are kept in shared memory; a step of 0.009 nm needs
# about 94 of them, 0.008 about 105
@pytest.mark.parametrize("h", [0.009, 0.008])
def test_fine_grids(h):
    pos = np.array([[0.0, 0.0, 0.0], [0.1, 0.03, 0.2], [0.25, 0.1, 0.0]], np.float32).astype(np.float64)
    q, r = np.array([0.5, -0.3, 0.2]), np.array([0.2, 0.15, 0.17])
    m = GBModel.charmm_gbsw(h=h, reference_table=True)
    ctx = context(m, (q, r))
    E, F = ctx.execute_host(pos)
    assert_table(ctx, m, pos, r)
    ref = O.Oracle(m).energy_forces(pos, q, r)
    assert abs(E / ref["energy"] - 1) < E_TOL and rel_rms(F, ref["forces"]) < F_TOL
    ctx.close()


# tiles of 32 atoms, i-blocks of 128; units of one j tile below 2,048 tile
# visits (n = 4,000 is below, 4,200 above).  No pair lies within 3e-7 of its
# distance of the cutoff (7e-5 with images), where FP32 and FP64 could disagree.
@pytest.mark.parametrize("n,kind", [(n, k) for n in (31, 32, 127, 128, 129, 161, 4000, 4200)
                                    for k in ("all", "cutoff", "periodic") if k != "periodic" or n < 4000])
def test_pair_tiles(n, kind):
    g = make_globule(n, seed=n)
    pos = (g.positions - g.positions.min(axis=0)).astype(np.float32).astype(np.float64)
    m = GBModel.charmm_gbsw(**{"all": {}, "cutoff": dict(cutoff=0.972),
                               "periodic": dict(cutoff=1.311, periodic=True, box=(2.8, 2.8, 2.8))}[kind])
    ctx = context(m, g)
    ref = O.Oracle(m).energy_forces(pos, g.charge, g.radius, adjoint=True)
    E, F = ctx.execute_host(pos)
    out = ctx.adjoint(pos)
    assert abs(E / ref["energy"] - 1) < E_TOL and rel_rms(F, ref["forces"]) < F_TOL
    assert abs(out["energy"] / ref["energy"] - 1) < E_TOL
    for k in ("forces", "dEdq", "dEdR"):
        assert rel_rms(out[k], ref[k]) < F_TOL, k
    ctx.close()


# the radial points of a direction are numbered together, and the leading ones
# inside the atom's own sphere left out on the exact table
@pytest.mark.parametrize("n_radial,lebedev", [(1, 6), (5, 14), (31, 26), (33, 6), (64, 110)])
@pytest.mark.parametrize("name", ["gbsw", "gbsw_integral", "gbmv1", "gbmv2"])
def test_quadrature_rules(n_radial, lebedev, name):
    g = make_globule(130, seed=3)
    kw = dict(n_radial=n_radial, lebedev=lebedev)
    box = box_for(g.positions)
    m = {"gbsw": GBModel.charmm_gbsw(**kw), "gbsw_integral": GBModel.gbsw_integral(**kw),
         "gbmv1": GBModel.gbmv1(box=box, **kw), "gbmv2": GBModel.gbmv2(box=box, **kw)}[name]
    pos = g.positions.astype(np.float32).astype(np.float64)
    ctx = context(m, g)
    ctx.execute_host(pos, forces=False)
    ref = O.Oracle(m).integrals(pos, g.radius)[0]
    assert np.abs(ctx.integrals() - ref).max() < I_TOL * np.abs(ref).max()
    ctx.close()


# a box smaller than the points' reach, and the molecule across its faces
@pytest.mark.parametrize("name", ["gbmv1", "gbmv2"])
@pytest.mark.parametrize("shift", [0.0, 1.7, -4.4])
def test_points_and_atoms_leave_the_box(name, shift):
    g = make_globule(200, seed=8)
    pos = (g.positions - g.positions.min(axis=0) + shift).astype(np.float32).astype(np.float64)
    m = getattr(GBModel, name)(box=(2.4, 2.4, 2.55))
    ctx = context(m, g)
    E, F = ctx.execute_host(pos)
    ref = O.Oracle(m).energy_forces(pos, g.charge, g.radius)
    assert np.abs(ctx.integrals() - ref["integrals"]).max() < I_TOL * np.abs(ref["integrals"]).max()
    assert abs(E / ref["energy"] - 1) < E_TOL and rel_rms(F, ref["forces"]) < F_TOL
    ctx.close()


@pytest.mark.parametrize("kw", [{}, dict(cutoff=1.2), dict(reference_table=True),
                                dict(cutoff=1.3, periodic=True, box=(4.0, 4.0, 4.2))],
                         ids=["all", "cutoff", "reference_table", "periodic"])
def test_adjoint_on_records_and_on_lists(kw):
    """Every contribution is rounded the same way on both: the same bits."""
    g = make_globule(700, seed=19)
    m = GBModel.charmm_gbsw(**kw)
    a, b = context(m, g), context(m, g)
    b.set_chain_records(0)
    for _ in range(2):
        x, y = a.adjoint(g.positions), b.adjoint(g.positions)
        assert x["energy"] == y["energy"]
        for k in GRADS:
            assert np.array_equal(x[k], y[k]), k
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["gbsw", "gbmv2"])
def test_adjoint_in_a_captured_graph_and_after_its_table_grew(name):
    torch = pytest.importorskip("torch")
    g = make_globule(900, seed=29)
    wide = g.positions * 1.6
    m = GBModel.charmm_gbsw() if name == "gbsw" else GBModel.gbmv2(box=box_for(wide))
    ctx, fresh = context(m, g), context(m, g)
    dev = torch.device("cuda:0")
    n = g.n
    posq = torch.zeros((n, 4), dtype=torch.float32, device=dev)
    out = torch.zeros(3 + 5 * n, dtype=torch.float64, device=dev)
    at = out.data_ptr()

    def call(flags, stream):
        ctx.adjoint_device(posq.data_ptr(), at, at + 8, at + 8 * (1 + 3 * n), at + 8 * (1 + 4 * n),
                           at + 8 * (1 + 5 * n), flags, stream)

    def same(pos):
        want = fresh.adjoint(pos)
        got = out.cpu().numpy()
        assert got[0] == want["energy"]
        assert np.array_equal(got[1:], np.concatenate([want[k].reshape(-1) for k in GRADS]))

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        posq[:, :3] = torch.from_numpy(g.positions.astype(np.float32)).to(dev)
        call(EXEC_CHECK, s.cuda_stream)
    s.synchronize()
    same(g.positions)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call(0, s.cuda_stream)
    near = jitter(g.positions, 0.001, np.random.default_rng(1))
    posq[:, :3] = torch.from_numpy(near.astype(np.float32)).to(dev)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    same(near)
    del graph
    # a checked call whose table needs more room than the first one's
    with torch.cuda.stream(s):
        posq[:, :3] = torch.from_numpy(wide.astype(np.float32)).to(dev)
        call(EXEC_CHECK, s.cuda_stream)
    s.synchronize()
    same(wide)
    ctx.close()
    fresh.close()


@pytest.mark.parametrize("dtypes", [("float64",) * 4, ("float32",) * 4, ("float32", "float64", "float32", "float64")])
def test_autograd_types_and_streams(dtypes):
    torch = pytest.importorskip("torch")
    from openmmcustomgbintegralforce_gb300.autograd import GBEnergy

    g = make_globule(300, seed=6)
    m = GBModel.charmm_gbsw()
    mod = GBEnergy(m, g.n)
    values = [g.positions, g.charge, g.radius, np.array([m.alpha0, m.alpha1])]

    def run(add):
        ts = [torch.tensor(v, dtype=getattr(torch, d), device="cuda:0", requires_grad=True)
              for v, d in zip(values, dtypes)]
        E = mod(*ts)
        value = E.detach().clone()
        if add:
            E += 1.0  # the caller's own tensor
        E.backward()
        torch.cuda.synchronize()
        assert E.dtype == ts[0].dtype and all(t.grad.dtype == t.dtype and t.grad.shape == t.shape for t in ts)
        return [value] + [t.grad for t in ts]

    plain = run(False)
    with torch.cuda.stream(torch.cuda.Stream()):
        side = run(True)
    for x, y in zip(plain, side):
        assert torch.equal(x, y)
    exact = [torch.tensor(v).to(getattr(torch, d)).double().numpy() for v, d in zip(values, dtypes)]
    ref = O.Oracle(m.replace(alpha0=exact[3][0], alpha1=exact[3][1])).energy_forces(
        exact[0].astype(np.float32).astype(np.float64), exact[1], exact[2], adjoint=True)
    assert abs(float(plain[0]) / ref["energy"] - 1) < E_TOL
    for t, k in zip(plain[1:], GRADS):
        want = -ref[k] if k == "forces" else ref[k]
        assert rel_rms(t.double().cpu().numpy(), want) < F_TOL, k


# a table sized on spread-out atoms keeps buckets for short lists: crowded, the
# same atoms have lists far longer than their buckets and as many entries
@pytest.mark.parametrize("n", [40, 250])
@pytest.mark.parametrize("name", ["exact", "standalone", "grid", "gbmv1", "gbmv2"])
def test_lists_longer_than_their_buckets(n, name):
    rng = np.random.default_rng(n)
    k = int(np.ceil(n ** (1 / 3)))
    lattice = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    sparse = 0.6 * lattice.astype(np.float64)
    dense = (rng.uniform(1.0, 1.3, (n, 3))).astype(np.float32).astype(np.float64)
    r = rng.uniform(0.12, 0.2, n)
    q = rng.normal(size=n)
    box = box_for(sparse)
    m = {"exact": GBModel.charmm_gbsw(), "standalone": GBModel.charmm_gbsw(reference_table=True),
         "grid": GBModel.gbsw_integral(), "gbmv1": GBModel.gbmv1(box=box), "gbmv2": GBModel.gbmv2(box=box)}[name]
    a, b = context(m, (q, r)), context(m, (q, r))
    a.execute_host(sparse)
    for _ in range(2):
        Ea, Fa = a.execute_host(dense)
        Eb, Fb = b.execute_host(dense)
        assert Ea == Eb and np.array_equal(Fa, Fb)
        assert np.array_equal(a.integrals(), b.integrals())
    assert_table(a, m, dense, r)
    ref = O.Oracle(m).integrals(dense, r)[0]
    assert np.abs(a.integrals() - ref).max() < I_TOL * np.abs(ref).max()
    a.close()
    b.close()


# the work counters follow the reference's walk (ascending lists, first burying
# atom ends it), whatever order the integrals read; a point within rounding of
# a sphere may count differently in FP32, fewer than one in 10,000
@pytest.mark.parametrize("name", ["standalone", "grid"])
def test_counted_work_is_the_reference_walk(name):
    g = make_globule(300, seed=12)
    pos = g.positions.astype(np.float32).astype(np.float64)
    m = GBModel.charmm_gbsw(reference_table=True) if name == "standalone" else GBModel.gbsw_integral()
    ctx = context(m, g)
    ctx.execute_host(pos, count_work=True)
    got, ref = ctx.work(), O.Oracle(m).integrals(pos, g.radius)[1]
    for k in ("volume_evals", "shell_evals"):
        assert abs(got[k] / ref[k] - 1) < 1e-4, k
    ctx.close()


# with a cutoff the integrals take the atoms in spatial order, without (below
# 40,000 atoms) as they come; neither changes a volume
@pytest.mark.parametrize("n", [1, 33, 700])
@pytest.mark.parametrize("kw", [{}, dict(reference_table=True)], ids=["exact", "reference"])
def test_integrals_do_not_depend_on_the_order(n, kw):
    g = make_globule(n, seed=14)
    a, b = context(GBModel.charmm_gbsw(**kw), g), context(GBModel.charmm_gbsw(cutoff=1.2, **kw), g)
    for _ in range(2):
        a.execute_host(g.positions)
        b.execute_host(g.positions)
        assert np.array_equal(a.integrals(), b.integrals()) and np.array_equal(a.born_radii(), b.born_radii())
    a.adjoint(g.positions)
    b.adjoint(g.positions)
    assert np.array_equal(a.integrals(), b.integrals())
    a.close()
    b.close()
