"""Differentiable GB energy for parameter fitting: a torch.autograd.Function
over the device adjoint (``gbx_adjoint``).

One forward call runs the whole pipeline once in adjoint mode -- table,
integrals, Born radii, pair term, chain rule with dE/dR and dE/dq -- and
keeps the gradients with respect to positions, charges, input radii and the
two Born-radius coefficients (alpha0, alpha1) for the backward, which only
scales them by the incoming gradient.  Beside the table the context holds a
record per point that some atom's shell holds (GBSW) or the sums of every
point (GBMV); none of them is kept for the backward.

The reference exposes the same gradients through its reference platform
(CharmmReferenceGBSW.cpp:597-674 for dB/dx, CharmmReferenceGBMV.cpp:349-443
for the chain rule and the parameter derivatives); here they come from the
GPU path.  Positions are in nm, energies in kJ/mol.
"""
from __future__ import annotations

import torch

from ._lib import EXEC_CHECK, Context
from .spec import GBModel

_LEGACY_STREAM = 1  # cudaStreamLegacy: torch's default stream


class GBEnergyFunction(torch.autograd.Function):
    """E = GB(positions [n,3], charges [n], radii [n], alpha [2]) on one context."""

    @staticmethod
    def forward(ctx, positions, charges, radii, alpha, gb: Context, check: bool = True):
        if not positions.is_cuda:
            raise ValueError("GBEnergyFunction: positions must be a CUDA tensor")
        n = gb.n
        if positions.shape != (n, 3) or charges.shape != (n,) or radii.shape != (n,) or alpha.shape != (2,):
            raise ValueError("GBEnergyFunction: expected positions [n,3], charges [n], radii [n], alpha [2]")
        # one transfer for the three parameter tensors, one allocation for every
        # output: the call's host work is torch operations, each of them 5 to 30 us
        parts = [t.detach() for t in (charges, radii, alpha)]
        if len({(t.dtype, t.device) for t in parts}) > 1:
            parts = [t.to(positions.device, torch.float64) for t in parts]
        p = torch.cat(parts).to("cpu", torch.float64).numpy()
        gb.set_particle_parameters(p[:n], p[n:2 * n])
        gb.set_global_parameters(float(p[2 * n]), float(p[2 * n + 1]))
        dev = positions.device
        posq = torch.empty((n, 4), dtype=torch.float32, device=dev)  # w is not read
        posq[:, :3] = positions.detach()
        # energy | forces [n, 3] | dE/dq [n] | dE/dR [n] | dE/dalpha [2]
        out = torch.empty(3 + 5 * n, dtype=torch.float64, device=dev)
        at = out.data_ptr()
        # the default stream by its own handle: 0 would be the context's stream,
        # which nothing orders after the copy into posq
        stream = torch.cuda.current_stream(dev).cuda_stream or _LEGACY_STREAM
        gb.adjoint_device(posq.data_ptr(), at, at + 8, at + 8 * (1 + 3 * n), at + 8 * (1 + 4 * n),
                          at + 8 * (1 + 5 * n), EXEC_CHECK if check else 0, stream)
        ctx.save_for_backward(out)
        ctx.n = n
        ctx.dtypes = (positions.dtype, charges.dtype, radii.dtype, alpha.dtype)
        return out[0].to(positions.dtype, copy=True)  # its own memory: a caller may write to it before backward

    @staticmethod
    def backward(ctx, grad):
        (out,) = ctx.saved_tensors
        n = ctx.n
        g = out[1:] * grad  # FP64, as the saved gradients: `grad` is one number
        tp, tq, tr, ta = ctx.dtypes
        if tp == tq == tr == ta:
            g = g.to(tp)
        # copies, none a view of the product: a caller may write to one, or keep
        # it, whatever becomes of the others
        dx, dq, dR, da = torch.split_with_sizes_copy(g, (3 * n, n, n, 2))
        return dx.view(n, 3).neg().to(tp), dq.to(tq), dR.to(tr), da.to(ta), None, None


class GBEnergy(torch.nn.Module):
    """Module form: owns the CUDA context; charges, radii and alpha may be
    nn.Parameters (the fitting use case)."""

    def __init__(self, model: GBModel, n_atoms: int):
        super().__init__()
        self.model = model
        self.gb = Context(model, n_atoms)

    def forward(self, positions, charges, radii, alpha=None):
        if alpha is None:
            alpha = torch.tensor([self.model.alpha0, self.model.alpha1], dtype=torch.float64,
                                 device=positions.device)
        return GBEnergyFunction.apply(positions, charges, radii, alpha, self.gb)


def gb_energy(positions, charges, radii, alpha, gb: Context):
    """Functional form of GBEnergyFunction."""
    return GBEnergyFunction.apply(positions, charges, radii, alpha, gb)


__all__ = ["GBEnergyFunction", "GBEnergy", "gb_energy"]
