"""Performance cases: what a program has this library evaluate, through its
public entry points.

A case is one force instance on one synthetic globule (``globule.py``; a
batch: several), re-oriented and jittered by the seed as a frame of a
trajectory would be, with charges of its own.  ``run`` is one pass: an MD
step's energy and forces on device buffers, a host-array call, a
differentiable evaluation with its backward, or a batch of molecules.

The arithmetic of every entry point is FP32 with fixed-point and FP64 sums,
so the passes hand energies and forces on in single precision, as an
integrator in OpenMM's single or mixed precision reads them (force buffer x
2^-32).

``exact`` evaluates the same models in 64 bits with plain torch: its own
quadrature rules, lookup tables, volume functions and chain rule.
"""
from __future__ import annotations

import functools
import math
from types import SimpleNamespace

import numpy as np
import torch

from openmmcustomgbintegralforce_gb300._lib import EXEC_ENERGY, EXEC_FORCES, Batch, Context, CustomContext
from openmmcustomgbintegralforce_gb300.autograd import GBEnergy
from openmmcustomgbintegralforce_gb300.expression_sets import MODIFIED
from openmmcustomgbintegralforce_gb300.globule import make_globule
from openmmcustomgbintegralforce_gb300.spec import GBModel, box_for

DEVICE = "cuda"
NATIVE = (24, 26)   # the integral classes' own quadrature: 24 radial x 26 angular points
STANDARD = (24, 38)   # CharmmGBSWForce's own
MEDIUM = (24, 50)
FINE = (32, 110)


def _case(entry, model, atoms, quad, cutoff=0.0, periodic=False, molecules=1, **name):
    return {**name, "entry": entry, "model": model, "atoms": atoms, "n_radial": quad[0], "lebedev": quad[1],
            "cutoff": cutoff, "periodic": periodic, "molecules": molecules}


def listed():
    return [
        # one MD step of a small protein: latency and launches
        _case("device", "gbsw", 1000, STANDARD, name="gbsw_1k"),
        # one MD step of a large assembly, all pairs: the headline workload
        _case("device", "gbsw", 50000, FINE, name="gbsw_50k"),
        # the same size as large systems are usually run, with a pair cutoff
        _case("device", "gbsw", 50000, FINE, cutoff=2.0, name="gbsw_50k_cutoff"),
        # CutoffPeriodic: minimum images and wrapped table queries
        _case("device", "gbsw", 9973, FINE, cutoff=1.5, periodic=True, name="gbsw_10k_periodic"),
        # CharmmGBMVForce on the GBSW integral class: capped per-cell lists
        _case("device", "gbsw_integral", 6007, NATIVE, name="gbsw_integral_6k"),
        # MD steps of a mid-sized protein with either GBMV volume
        _case("device", "gbmv1", 10000, MEDIUM, name="gbmv1_10k"),
        _case("device", "gbmv2", 10000, MEDIUM, name="gbmv2_10k"),
        # host arrays in and out, the Reference-platform style of call
        _case("host", "gbmv2", 2513, NATIVE, name="gbmv2_host_2k"),
        # parameter fitting: forward and backward through torch.autograd
        _case("grad", "gbsw", 5000, STANDARD, name="gbsw_grad_5k"),
        _case("grad", "gbmv2", 3001, MEDIUM, name="gbmv2_grad_3k"),
        # conformations of uneven sizes, GBSW and GBMV-II mixed, in one call
        _case("batch", "mixed", 500, MEDIUM, molecules=12, name="batch_mixed_12"),
        # a user's own expressions, compiled for the device
        _case("custom", "gbmv2", 4001, NATIVE, name="custom_gbmv2_4k"),
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    quad = rng.choice([NATIVE, STANDARD, MEDIUM])
    kind = rng.choice(["gbsw", "gbsw", "cutoff", "periodic", "integral", "gbmv", "gbmv", "host", "grad", "batch",
                       "custom"])
    gbmv = rng.choice(["gbmv1", "gbmv2"])
    if kind == "gbsw":
        return _case("device", "gbsw", size(500, 45000), rng.choice([quad, FINE]))
    if kind == "cutoff":
        return _case("device", "gbsw", size(2000, 45000), rng.choice([quad, FINE]), cutoff=rng.choice([1.2, 1.6, 2.0]))
    if kind == "periodic":
        return _case("device", "gbsw", size(2000, 20000), rng.choice([quad, FINE]), cutoff=rng.choice([1.2, 1.5]),
                     periodic=True)
    if kind == "integral":
        return _case("device", "gbsw_integral", size(500, 12000), quad)
    if kind == "gbmv":
        return _case("device", gbmv, size(500, 12000), quad)
    if kind == "host":
        return _case("host", rng.choice(["gbsw", "gbmv1", "gbmv2"]), size(500, 8000), quad)
    if kind == "grad":
        return _case("grad", rng.choice(["gbsw", "gbmv1", "gbmv2"]), size(500, 6000), quad)
    if kind == "batch":
        return _case("batch", "mixed", size(500, 900), quad, molecules=rng.randrange(4, 13))
    return _case("custom", gbmv, size(500, 6000), quad)


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------

@functools.lru_cache(maxsize=32)
def _globule(n):
    return make_globule(n, seed=n)


def _frame(n, seed):
    """Positions [n, 3] (nm, float32 values), charges and radii of one frame:
    the globule turned at random, N(0, 0.05 A) off its places, its charges
    N(0, 0.35 e) shifted to a net charge of zero."""
    g = _globule(n)
    rng = np.random.default_rng([seed, n])
    turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    x = (g.positions - g.positions.mean(0)) @ turn + rng.normal(0.0, 0.005, size=(n, 3)) + rng.uniform(-1, 1, 3)
    q = rng.normal(0.0, 0.35, size=n)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    return SimpleNamespace(n=n, x=f32(x), q=f32(q - q.mean()), R=g.radius)


def _frames(case, seed):
    """The case's molecules; a batch's sizes rise from `atoms` to about 16 times that."""
    m = case["molecules"]
    return [_frame(int(case["atoms"] * 16 ** (k / m)), seed + 7919 * k) for k in range(m)]


def _model_name(case, k):
    return case["model"] if case["model"] != "mixed" else ("gbsw", "gbmv2")[k % 2]


def _model(case, f, k=0):
    quad = dict(n_radial=case["n_radial"], lebedev=case["lebedev"])
    name = _model_name(case, k)
    if name == "gbsw":
        if case["periodic"]:
            return GBModel.charmm_gbsw(cutoff=case["cutoff"], periodic=True, box=box_for(f.x, margin=0.5), **quad)
        return GBModel.charmm_gbsw(cutoff=case["cutoff"], **quad)
    if name == "gbsw_integral":
        return GBModel.gbsw_integral(**quad)
    return getattr(GBModel, name)(box=box_for(f.x, margin=1.0), **quad)


def _custom_params(f, seed):
    return np.stack([f.q, f.R, 0.9 + 0.2 * np.random.default_rng([seed, 1]).random(f.n)], axis=1)


@functools.lru_cache(maxsize=1)
def _stream():
    """The program's one stream: steps follow one another."""
    return torch.cuda.Stream()


def prepare(case, seed):
    frames = _frames(case, seed)
    f = frames[0]
    models = [_model(case, g, k) for k, g in enumerate(frames)]
    s = SimpleNamespace(entry=case["entry"], n=f.n)
    if s.entry == "batch":
        s.gb = Batch(models, [g.n for g in frames])
        for c, g in zip(s.gb.molecules, frames):
            c.set_particle_parameters(g.q, g.R)
        s.x = np.concatenate([g.x for g in frames])
        return s
    s.stream = _stream()
    if s.entry == "grad":
        s.gb = GBEnergy(models[0], f.n)
        s.leaves = [torch.tensor(v, dtype=torch.float32, device=DEVICE).requires_grad_()
                    for v in (f.x, f.q, f.R, [models[0].alpha0, models[0].alpha1])]
        return s
    if s.entry == "custom":
        s.gb = CustomContext(models[0], f.n, MODIFIED)
        s.gb.set_custom_parameters(_custom_params(f, seed))
    else:
        s.gb = Context(models[0], f.n)
        s.gb.set_particle_parameters(f.q, f.R)
    if s.entry == "host":
        s.x = f.x
        return s
    s.stride = (f.n + 31) // 32 * 32
    s.posq = torch.zeros((f.n, 4), dtype=torch.float32, device=DEVICE)
    s.posq[:, :3] = torch.tensor(f.x, dtype=torch.float32, device=DEVICE)
    s.force = torch.zeros((3, s.stride), dtype=torch.int64, device=DEVICE)
    s.energy = torch.zeros(1, dtype=torch.float64, device=DEVICE)
    return s


def run(s):
    if s.entry in ("host", "batch"):
        energy, forces = s.gb.execute_host(s.x)
        return {"energy": np.float32(energy), "forces": forces.astype(np.float32)}
    with torch.cuda.stream(s.stream):
        if s.entry == "grad":
            energy = s.gb(*s.leaves)
            dx, dq, dR, dalpha = torch.autograd.grad(energy, s.leaves)
            return {"energy": energy.detach(), "dx": dx, "dq": dq, "dR": dR, "dalpha": dalpha}
        # the engine clears its buffers, every force adds to them, the integrator reads them
        s.force.zero_()
        s.energy.zero_()
        s.gb.execute_device(s.posq.data_ptr(), s.force.data_ptr(), s.stride, s.energy.data_ptr(),
                            EXEC_FORCES | EXEC_ENERGY, s.stream.cuda_stream)
        return {"energy": s.energy.to(torch.float32), "forces": s.force[:, :s.n].to(torch.float32) * 2.0 ** -32}


def work(case):
    """Operations per pass (multiply-add = 2): every pair within the cutoff,
    every quadrature point, and of the points inside the globule (about 60 in
    100) the atoms that the model makes them read: GBSW those whose switching
    shell or burying sphere can hold the point, GBMV its cell's list."""
    nbytes = flops = 0.0
    for k in range(case["molecules"]):
        n = int(case["atoms"] * 16 ** (k / case["molecules"]))
        reach = n if case["cutoff"] <= 0 else min(n, 100.0 * 4.19 * case["cutoff"] ** 3)
        per_point = {"gbsw": 4 * 10 + 2 * 22, "gbsw_integral": 4 * 10 + 2 * 22, "gbmv1": 50 * (11 + 24),
                     "gbmv2": 50 * (21 + 46)}[_model_name(case, k)]
        flops += 39.0 * n * reach / 2 + n * case["n_radial"] * case["lebedev"] * (2 * 13 + 0.6 * per_point)
        nbytes += n * (12 + 4 + 4) + n * (20 if case["entry"] == "grad" else 12) + 4
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------------
# The same in 64 bits
# --------------------------------------------------------------------------

def _orbit(kind, w, a=0.0, b=0.0):
    """Points of one octahedral orbit (all sign changes and permutations) and their weight."""
    v = {"a1": (1, 0, 0), "a2": (0, 0.5 ** 0.5, 0.5 ** 0.5), "a3": (3 ** -0.5,) * 3, "llm": (a, a, b),
         "pq0": (a, b, 0.0)}[kind]
    pts = {(s0 * v[i], s1 * v[j], s2 * v[k]) for i, j, k in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))
           for s0 in (1, -1) for s1 in (1, -1) for s2 in (1, -1)}
    pts = {tuple(x + 0.0 for x in p) for p in pts}  # -0.0 and 0.0 are one point
    return [(*p, w) for p in sorted(pts)]


def _sphere(order):
    """Lebedev's octahedral rules (Zh. Vychisl. Mat. Mat. Fiz. 15, 48 (1975) and 16, 293 (1976))."""
    def llm(a, w):
        return _orbit("llm", w, a, math.sqrt(1 - 2 * a * a))

    def pq0(a, w):
        return _orbit("pq0", w, a, math.sqrt(1 - a * a))

    if order == 26:
        pts = _orbit("a1", 1 / 21) + _orbit("a2", 4 / 105) + _orbit("a3", 9 / 280)
    elif order == 38:
        pts = _orbit("a1", 1 / 105) + _orbit("a3", 9 / 280) + pq0(math.sqrt((1 - 3 ** -0.5) / 2), 1 / 35)
    elif order == 50:
        pts = (_orbit("a1", 4 / 315) + _orbit("a2", 64 / 2835) + _orbit("a3", 27 / 1280)
               + llm(11 ** -0.5, 14641 / 725760))
    else:
        pts = (_orbit("a1", 0.3828270494937162e-2) + _orbit("a3", 0.9793737512487512e-2)
               + llm(0.1851156353447362, 0.8211737283191111e-2) + llm(0.6904210483822922, 0.9942814891178103e-2)
               + llm(0.3956894730559419, 0.9595471336070963e-2) + pq0(0.4783690288121502, 0.9694996361663028e-2))
    assert len(pts) == order
    return np.array(pts)


def _quadrature(m):
    """Offsets [Q, 3] and the two integrals' weights w / r^2 and w / r^5, [Q] each."""
    t, w = np.polynomial.legendre.leggauss(m.n_radial)
    r, w = 0.5 * (m.r1 - m.r0) * t + 0.5 * (m.r1 + m.r0), 0.5 * (m.r1 - m.r0) * w
    s = _sphere(m.lebedev)
    off = (r[:, None, None] * s[None, :, :3]).reshape(-1, 3)
    w = (w[:, None] * s[None, :, 3]).reshape(-1)
    rr = np.repeat(r, m.lebedev)
    return [torch.tensor(v, dtype=torch.float64, device=DEVICE) for v in (off, w / rr ** 2, w / rr ** 5)]


def _lists(cell, atom, ncell, cap):
    """Each cell's atoms in ascending order, at most `cap` (0: all): [ncell, K], -1 where there is none."""
    order = torch.argsort(cell * (int(atom.max()) + 1) + atom)
    cell, atom = cell[order], atom[order]
    count = torch.bincount(cell, minlength=ncell)
    rank = torch.arange(len(cell), device=DEVICE) - (torch.cumsum(count, 0) - count)[cell]
    k = int(count.max()) if cap <= 0 else min(cap, int(count.max()))
    table = torch.full((ncell, k), -1, dtype=torch.int64, device=DEVICE)
    keep = rank < k
    table[cell[keep], rank[keep]] = atom[keep]
    return table


def _table(m, x, R):
    """The atoms that a point reads: the lists and the function from points to their row (-1: none).
    Standalone GBSW: every atom near enough to matter.  The integral classes: the model's own capped lists."""
    n, h = len(x), m.h
    ids = torch.arange(n, device=DEVICE)

    def flat(c, dims):
        return (c[..., 0] * dims[1] + c[..., 1]) * dims[2] + c[..., 2]

    if m.table_mode == 0:
        h = 0.25  # above the largest switching shell's outer radius: 27 cells around a point hold all it reads
        lo = x.amin(0) - 2 * h
        dims = ((x.amax(0) + 2 * h - lo) / h).ceil().long()
        own = ((x - lo) / h).floor().long()
        near = torch.cartesian_prod(*[torch.arange(-1, 2, device=DEVICE)] * 3)
        table = _lists(flat(own[:, None] + near, dims).reshape(-1), ids.repeat_interleave(27), int(dims.prod()), 0)
        glo, ghi = None, None
        if m.periodic:  # the reference's grid: a point off it is moved by one box edge
            pad = m.buffer + R.max() + m.sw + math.sqrt(3.0) / 2 * m.h + 1e-6
            glo = x.amin(0) - pad
            ghi = glo + ((x.amax(0) + pad - glo) / m.h).ceil() * m.h
            box = torch.tensor(m.box, dtype=torch.float64, device=DEVICE)

        def find(p):
            if glo is not None:
                p = torch.where(p < glo, p + box, p)
                p = torch.where(p > ghi, p - box, p)
            c = ((p - lo) / h).floor().long()
            return torch.where(((c >= 0) & (c < dims)).all(-1), flat(c, dims), -1), p

        return table, find
    if m.table_mode == 1:  # grid points, an atom's pad around each
        pad0 = 0.03 + math.sqrt(3.0) / 2 * h + m.buffer
        lo = x.amin(0) - pad0
        dims = ((x.amax(0) + pad0 - lo) / h).ceil().long() + 1
        hi = lo + (dims - 1) * h
        pad = R + math.sqrt(3.0) / 2 * h + m.buffer
        first = ((x - pad[:, None] - lo) / h).floor().long()
        span = int(2 * float(pad.max()) / h) + 3
        c = first[:, None] + torch.cartesian_prod(*[torch.arange(span, device=DEVICE)] * 3)
        member = (((lo + c * h) - x[:, None]) ** 2).sum(-1) < (pad ** 2)[:, None]
        cell = flat(c, dims)
        member &= (cell >= 0) & (cell < dims.prod())
        table = _lists(cell[member], ids[:, None].expand_as(cell)[member], int(dims.prod()), m.cap)

        def find(p):
            c = ((p - lo) / h).floor().long()
            return torch.where(((p >= lo) & (p <= hi)).all(-1), flat(c, dims), -1), p

        return table, find
    # a grid over the box around the centre of geometry, membership decided at samples around each atom
    box = torch.tensor(m.box, dtype=torch.float64, device=DEVICE)
    lo = x.mean(0) - box / 2
    dims = (box / h).ceil().long() + 1
    step = box / dims
    pad = R + math.sqrt(3.0) / 2 * step.max() + m.buffer
    start = x - pad[:, None] - step.max()
    span = int((2 * (pad.max() + step.max()) / step.min()).ceil()) + 1
    sample = start[:, None] + torch.cartesian_prod(*[torch.arange(span, device=DEVICE)] * 3) * step

    def cell_of(p):
        inside = p - torch.floor((p - lo) / box) * box
        c = ((inside - lo) / step).floor().long()
        return torch.where(((c >= 0) & (c < dims)).all(-1), flat(c, dims), -1)

    cell = cell_of(sample)
    member = (((sample - x[:, None]) ** 2).sum(-1) < (pad ** 2)[:, None]) & (cell >= 0)
    table = _lists(cell[member], ids[:, None].expand_as(cell)[member], int(dims.prod()), m.cap)
    return table, lambda p: (cell_of(p), p)


def _solvent(m, d, R, listed_):
    """Solvent fraction of each point from its listed atoms: d [P, K, 3] = x_j - p, R [P, K]."""
    r2 = (d * d).sum(-1)
    if m.model == 0:
        r = torch.sqrt(r2)
        dr = r - (R + 0.03) * 0.9520
        u = 0.5 + 0.75 * dr / m.sw - 0.25 * (dr / m.sw) ** 3
        u = torch.where(dr >= m.sw, 1.0, torch.where(dr <= -m.sw, 0.0, u))
        return torch.where(listed_, u, 1.0).prod(-1)
    if m.model == 1:
        e = torch.exp(m.gamma0 * math.log(m.lam) / R ** 4 * r2 ** 2)
        S = torch.where(listed_, e, 0.0).sum(-1)
    else:
        C = 10.0 * m.p1 * R + m.p2
        F = torch.where(listed_, (C / (C + 100.0 * r2 - 100.0 * R ** 2)) ** 2, 0.0)
        v = (d * F[..., None]).sum(1)
        S = m.s0 * F.sum(-1) * (r2 * F * F).sum(-1) / (v * v).sum(-1)
    return torch.sigmoid(m.beta * (S - m.lam))


def _chunks(m, x, off, table, find):
    """Points that read any atom, a piece at a time: (atom, quadrature index, listed atoms, mask, x_j - p)."""
    Q, K = len(off), table.shape[1]
    rows = max(1, 12_000_000 // (Q * K))
    for a in range(0, len(x), rows):
        p = (x[a:a + rows, None] + off).reshape(-1, 3)
        cell, moved = find(p)
        some = (cell >= 0) & (table[cell.clamp(min=0)] >= 0).any(-1)
        at = torch.nonzero(some).squeeze(-1)
        j = table[cell[at]]
        yield a + at // Q, at % Q, j.clamp(min=0), j >= 0, x[j.clamp(min=0)] - moved[at][:, None]


def _minimum_image(m, d):
    if m.periodic:
        box = torch.tensor(m.box, dtype=torch.float64, device=DEVICE)
        d = d - box * torch.floor(d / box + 0.5)
    return d


def _energy(m, x, q, R, B, custom):
    """Pair and single-particle terms, a block of rows at a time, each with its backward: returns the energy."""
    scale, pref = B, m.pref
    total = 0.0
    if custom is not None:
        pref = -138.935456 * (1.0 - 1.0 / 78.5)
        scale = custom * B
    own = (0.5 * pref * q * q / scale).sum()
    if custom is not None:
        own = own + (0.54 * 4 * 3.14159265 * (R + 0.14) ** 2 * (R / scale) ** 6).sum()
    own.backward(retain_graph=True)
    total += own.item()
    sleaf = scale.detach().requires_grad_()
    rows = max(1, 12_000_000 // len(x))
    for a in range(0, len(x), rows):
        d = _minimum_image(m, x - x[a:a + rows, None])
        r2 = (d * d).sum(-1)
        BB = sleaf[a:a + rows, None] * sleaf
        e = 0.5 * pref * q[a:a + rows, None] * q / torch.sqrt(r2 + BB * torch.exp(-r2 / (4 * BB)))
        skip = torch.eye(len(x), dtype=torch.bool, device=DEVICE)[a:a + rows] if len(x) <= 4096 else \
            torch.arange(len(x), device=DEVICE) == torch.arange(a, a + len(e), device=DEVICE)[:, None]
        if m.cutoff > 0:
            skip = skip | (r2 > m.cutoff ** 2)
        e = torch.where(skip, 0.0, e).sum()
        e.backward()
        total += e.item()
    scale.backward(sleaf.grad)
    return total


def _evaluate(m, f, alpha=None, custom=None):
    def t(v):
        return torch.tensor(v, dtype=torch.float64, device=DEVICE)

    x, q, R = t(f.x), t(f.q), t(f.R)
    alpha = t([m.alpha0, m.alpha1] if alpha is None else alpha)
    off, w4, w7 = _quadrature(m)
    table, find = _table(m, x, R)
    # a point that reads no atom is solvent; GBMV-I evaluates its empty sum
    empty = 1.0 if m.model != 1 else 1.0 / (1.0 + math.exp(m.beta * m.lam))
    s = torch.full((f.n, len(off)), empty, dtype=torch.float64, device=DEVICE)
    with torch.no_grad():
        for i, k, j, ok, d in _chunks(m, x, off, table, find):
            s[i, k] = _solvent(m, d, R[j], ok)
    I4, I7 = ((1 - s) @ w4).requires_grad_(), ((1 - s) @ w7).requires_grad_()
    for v in (x, q, R, alpha):
        v.requires_grad_()
    B = 1 / (alpha[0] * (1 / m.r0 - I4) + alpha[1] * (1 / (4 * m.r0 ** 4) - I7) ** 0.25)
    E = _energy(m, x, q, R, B, custom)
    dx, dR = x.grad.clone(), torch.zeros_like(R) if R.grad is None else R.grad.clone()
    xx, RR = x.detach(), R.detach()
    for i, k, j, ok, d in _chunks(m, xx, off, table, find):
        d.requires_grad_()
        r = RR[j].requires_grad_()
        weight = -(I4.grad[i] * w4[k] + I7.grad[i] * w7[k])  # dE/ds
        _solvent(m, d, r, ok).backward(weight)
        gd, gr = torch.nan_to_num(d.grad), torch.nan_to_num(r.grad)  # 0 at an atom's own place
        moves = (j != i[:, None]) & ok
        gd = gd * moves[..., None]
        dx.index_add_(0, i, -gd.sum(1))
        if m.cutoff > 0 and m.cutoff_chain_quirk:  # the reference drops the pull on atoms beyond the cutoff
            apart = _minimum_image(m, xx[j] - xx[i][:, None])
            gd = gd * ((apart * apart).sum(-1) <= m.cutoff ** 2)[..., None]
        hit = (gd != 0).any(-1) | (gr != 0)
        dx.index_add_(0, j[hit], gd[hit])
        dR.index_add_(0, j[hit], gr[hit])
    return SimpleNamespace(E=E, dx=dx, dq=q.grad, dR=dR, dalpha=alpha.grad)


def exact(case, seed):
    frames = _frames(case, seed)
    f, m = frames[0], _model(case, frames[0])
    if case["entry"] == "batch":
        got = [_evaluate(_model(case, g, k), g) for k, g in enumerate(frames)]
        return {"energy": torch.tensor([g.E for g in got], dtype=torch.float64),
                "forces": torch.cat([-g.dx for g in got])}
    if case["entry"] == "grad":
        g = _evaluate(m, f, alpha=[float(np.float32(m.alpha0)), float(np.float32(m.alpha1))])
        return {"energy": torch.tensor(g.E, dtype=torch.float64), "dx": g.dx, "dq": g.dq, "dR": g.dR,
                "dalpha": g.dalpha}
    custom = None
    if case["entry"] == "custom":
        custom = torch.tensor(_custom_params(f, seed)[:, 2], dtype=torch.float64, device=DEVICE)
    g = _evaluate(m, f, custom=custom)
    if case["entry"] == "host":
        return {"energy": torch.tensor(g.E, dtype=torch.float64), "forces": -g.dx}
    return {"energy": torch.tensor([g.E], dtype=torch.float64), "forces": (-g.dx).T}
