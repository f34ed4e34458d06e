"""gbx_get_lookup_table returns the table of the last call's positions, also
where that call replayed a graph and an earlier one's table was asked for."""
import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300._lib import EXEC_ENERGY, EXEC_FORCES, Batch, Context
from openmmcustomgbintegralforce_gb300.globule import jitter, make_globule
from openmmcustomgbintegralforce_gb300.spec import GBModel, box_for
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("entry", ["host", "device", "batch"])
@pytest.mark.parametrize("name", ["exact", "standalone", "grid", "gbmv2"])
def test_table_of_the_last_call(name, entry):
    g = make_globule(200, seed=31)
    m = {"exact": GBModel.charmm_gbsw(), "standalone": GBModel.charmm_gbsw(reference_table=True),
         "grid": GBModel.gbsw_integral(), "gbmv2": GBModel.gbmv2(box=box_for(g.positions))}[name]
    batch = Batch([m, m], [g.n, g.n]) if entry == "batch" else None
    ctx = batch.molecules[1] if batch else Context(m, g.n)
    for c in batch.molecules if batch else [ctx]:
        c.set_particle_parameters(g.charge, g.radius)
    posq = torch.zeros((g.n, 4), dtype=torch.float32, device="cuda:0")
    force = torch.zeros((3, g.n), dtype=torch.int64, device="cuda:0")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda:0")
    rng = np.random.default_rng(2)
    x = g.positions.astype(np.float32).astype(np.float64)
    for _ in range(5):
        if batch:
            batch.execute_host(np.concatenate([x, x]))
        elif entry == "host":
            ctx.execute_host(x)
        else:
            posq[:, :3] = torch.from_numpy(x).to(posq)
            torch.cuda.synchronize()
            ctx.execute_device(posq.data_ptr(), force.data_ptr(), g.n, energy.data_ptr(), EXEC_FORCES | EXEC_ENERGY, 0)
        t, ref = ctx.lookup_table(), O.Oracle(m).table(x, g.radius)
        assert np.array_equal(t["dims"], ref["dims"])
        assert np.array_equal(t["counts"], ref["counts"]) and np.array_equal(t["atoms"], ref["atoms"])
        x = jitter(x, 0.02, rng).astype(np.float32).astype(np.float64)
    (batch or ctx).close()
