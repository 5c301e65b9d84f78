"""torch.autograd face of the engine's hand-written adjoint.

``FreeEnergy.apply(delta, a, b_ext, ctx, w_omega, beta_j)`` returns
L = w_omega * Omega + sum(beta_j * j) for the complex order parameter
``delta`` [Nc][N0][N0] (complex128), the induced vector potential ``a``
[2][N0][N0] (internal units, float64) and the external field ``b_ext``
(0-d float64, B0 units), evaluated on the engine context ``ctx`` with its
incoming boundary values held fixed (one frozen-boundary pass of the
self-consistency map, ComputeFreeEnergy.h:281-414, ComputeCurrent.h:175-222).
``backward`` runs the adjoint sweep and
returns dL/dDelta, dL/dA and dL/dB_ext in PyTorch's convention for complex
inputs (dL/dRe + i dL/dIm).

``edge_current_weights`` builds beta_j for the total azimuthal current of a
ring of sites near the grain's edge.
"""
from __future__ import annotations

import numpy as np
import torch


def _on_gpu(t: torch.Tensor, dtype, size: int, what: str) -> torch.Tensor:
    """``t`` on the engine's GPU (the current device, where its kernels run)."""
    if t.numel() != size:
        raise ValueError(f"FreeEnergy: {what} has {t.numel()} values, the context takes {size}")
    return t.detach().to(torch.device("cuda", torch.cuda.current_device()), dtype)


def _planar(delta: torch.Tensor, ctx) -> torch.Tensor:
    """[Nc][N0][N0] complex as the engine's [Nc][2][N0][N0], a tensor of its own."""
    d = ctx.dims
    z = _on_gpu(delta, torch.complex128, d.n_comp * d.n0 * d.n0, "delta").resolve_conj()
    z = z.reshape(d.n_comp, d.n0, d.n0)
    return torch.stack([z.real, z.imag], dim=1).contiguous()


class FreeEnergy(torch.autograd.Function):
    """State and gradients stay on the GPU.  The engine works on a stream of
    its own: this stream is waited for before the engine reads a tensor, and
    every engine call here that hands values back is complete when it returns."""

    @staticmethod
    def forward(fctx, delta, a, b_ext, ctx, w_omega=1.0, beta_j=None):
        d = _planar(delta, ctx)
        n0 = ctx.dims.n0
        av = _on_gpu(a, torch.float64, 2 * n0 * n0, "a").resolve_neg().reshape(2, n0, n0).clone(
            memory_format=torch.contiguous_format)
        b = float(b_ext.detach().cpu())
        # In C order whatever the weight's own: backward hands its address on.
        beta = None if beta_j is None else torch.from_numpy(
            np.array(beta_j, np.float64, order="C")).to(d.device)
        torch.cuda.current_stream().synchronize()
        ctx.set_state_device(d.data_ptr(), av.data_ptr())
        ctx.set_external_field(b)
        fe = ctx.evaluate()
        if beta is None:
            loss = torch.tensor(w_omega * fe, dtype=torch.float64, device=delta.device)
        else:
            j = torch.empty(2, n0, n0, dtype=torch.float64, device=d.device)
            ctx.results_device(j_ptr=j.data_ptr())
            loss = (torch.sum(beta * j) + w_omega * fe).to(delta.device)
        fctx.engine = ctx
        fctx.args = (d, av, b, w_omega, beta)
        fctx.devices = (delta.device, a.device, b_ext.device)
        return loss

    @staticmethod
    def backward(fctx, grad_out):
        ctx = fctx.engine
        d, av, b, w_omega, beta = fctx.args
        n0 = ctx.dims.n0
        if beta is not None:
            beta = beta.reshape(2, n0, n0)
        gd, ga = torch.empty_like(d), torch.empty_like(av)
        gb = torch.empty((), dtype=torch.float64, device=d.device)
        torch.cuda.current_stream().synchronize()
        ctx.set_state_device(d.data_ptr(), av.data_ptr())
        ctx.set_external_field(b)
        ctx.adjoint_device(w_omega, None if beta is None else beta.data_ptr(), gd.data_ptr(), ga.data_ptr(),
                           gb.data_ptr())
        g = grad_out.detach().to(d.device, torch.float64)
        gdel = torch.complex(gd[:, 0], gd[:, 1]) * g
        return (gdel.to(fctx.devices[0]), (ga * g).to(fctx.devices[1]), (gb * g).to(fctx.devices[2]), None, None,
                None)


def edge_current_weights(domain: np.ndarray, h: float, width: float) -> np.ndarray:
    """beta [2][N0][N0] with sum(beta * j) the azimuthal current (z x r_hat) . j
    summed over the grain sites within ``width`` (in xi0) of the grain's
    outermost radius, measured from the lattice centre."""
    n0 = domain.shape[0]
    yy, xx = np.mgrid[0:n0, 0:n0].astype(np.float64)
    c = 0.5 * (n0 - 1)
    x, y = (xx - c) * h, (yy - c) * h
    r = np.hypot(x, y)
    inside = domain > 0
    rmax = r[inside].max()
    ring = inside & (r > rmax - width)
    rs = np.where(r > 0, r, 1.0)
    beta = np.zeros((2, n0, n0))
    beta[0] = np.where(ring, -y / rs, 0.0)
    beta[1] = np.where(ring, x / rs, 0.0)
    return beta
