"""New parameters set while an unchecked call is still running: that call's
result is the one of the parameters it was issued with, the next call's the
one of the new."""
import numpy as np
import pytest

from openmmcustomgbintegralforce_gb300._lib import EXEC_CHECK, EXEC_ENERGY, EXEC_FORCES, Context, CustomContext
from openmmcustomgbintegralforce_gb300.expression_sets import MODIFIED
from openmmcustomgbintegralforce_gb300.globule import make_globule
from openmmcustomgbintegralforce_gb300.spec import GBModel, box_for

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BOTH = EXEC_FORCES | EXEC_ENERGY


@pytest.fixture(scope="module")
def glob():
    return make_globule(8000, seed=23)


def make(name, g):
    if name == "custom":
        return CustomContext(GBModel.gbmv2(box=box_for(g.positions)), g.n, MODIFIED)
    return Context(GBModel.charmm_gbsw() if name == "gbsw" else GBModel.gbmv2(box=box_for(g.positions)), g.n)


def set_parameters(ctx, q, R):
    if isinstance(ctx, CustomContext):
        ctx.set_custom_parameters(np.stack([q, R, np.ones(len(q))], axis=1))
    else:
        ctx.set_particle_parameters(q, R)


@pytest.mark.parametrize("how", ["call", "graph"])
@pytest.mark.parametrize("entry", ["gbsw-execute", "gbmv2-execute", "custom-execute", "gbsw-adjoint", "gbmv2-adjoint"])
def test_parameters_set_while_a_call_runs(glob, entry, how):
    g = glob
    name, what = entry.split("-")
    ctx, fresh = make(name, g), make(name, g)
    rng = np.random.default_rng(4)
    sets = [(rng.normal(0.0, 0.35, g.n), g.radius * s) for s in (1.0, 0.9, 1.0)]
    n = g.n
    posq = torch.zeros((n, 4), dtype=torch.float32, device="cuda:0")
    posq[:, :3] = torch.from_numpy(g.positions).to(posq)
    outs = [torch.zeros(3 + 5 * n, dtype=torch.float64, device="cuda:0") for _ in sets]
    stage = torch.zeros(3 + 5 * n, dtype=torch.float64, device="cuda:0")

    def call(c, flags, s):
        at = stage.data_ptr()
        if what == "adjoint":
            c.adjoint_device(posq.data_ptr(), at, at + 8, at + 8 * (1 + 3 * n), at + 8 * (1 + 4 * n),
                             at + 8 * (1 + 5 * n), flags, s.cuda_stream)
        else:
            stage.zero_()
            c.execute_device(posq.data_ptr(), at + 8, n, at, BOTH | flags, s.cuda_stream)

    want = []
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for q, R in sets:
            set_parameters(fresh, q, R)
            call(fresh, EXEC_CHECK, s)
            s.synchronize()
            want.append(stage.clone())
        # buffers sized and record regions settled
        set_parameters(ctx, *sets[0])
        for flags in (EXEC_CHECK, EXEC_CHECK, 0):
            call(ctx, flags, s)
            s.synchronize()
        graph = None
        if how == "graph":
            set_parameters(ctx, *sets[0])  # the context's own graph of the call would be launched, not captured
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                call(ctx, 0, s)
        # nothing waits between a call and the next parameters
        for (q, R), out in zip(sets, outs):
            set_parameters(ctx, q, R)
            graph.replay() if graph else call(ctx, 0, s)
            out.copy_(stage)
        s.synchronize()
    torch.cuda.synchronize()
    for out, w in zip(outs, want):
        assert torch.equal(out.view(torch.int64), w.view(torch.int64))  # a force buffer holds integers
    del graph
    ctx.close()
    fresh.close()
