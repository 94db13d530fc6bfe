"""Differentiation of the interpolant behind ``torch.autograd``.

``interpolate(ip, x, nodal_values)`` evaluates the mixed-precision form of a
built interpolant and registers a hand-written backward:

* dL/dx      -- G = g C^T on the tensor cores, then a reverse pass through the
                basis products per point (``smx_tensor_vjp_x``);
* dL/dvalues -- dL/dC = A(x)^T g on the tensor cores, the adjoint of the FP64
                coefficient transform (``smx_spectral_coefficients_adjoint``)
                and the chain rule through the plan's rows
                F[r] = zeta_s (fu[umap r] - fu[u0]) and its constant term.

The reference has no derivative with respect to the nodal values; its
derivative with respect to x is the dense Jacobian of ``gradient``
(interpolation.py:306-345), which the FP64 path reproduces.
"""
from __future__ import annotations

import torch

from . import _capi as capi


def _value_runs(umap, n):
    """Rows by nodal value in runs of at most 64 rows of one value: (value_run
    [n + 1], run_begin [runs + 1], rows)."""
    zero = torch.zeros(1, dtype=torch.int64, device=umap.device)
    count = torch.bincount(umap, minlength=n)
    runs = (count + 63) // 64
    value_run = torch.cat([zero, runs.cumsum(0)])
    value = torch.repeat_interleave(torch.arange(n, device=umap.device), runs)
    first = torch.cat([zero, count.cumsum(0)])  # the first row of each value
    begin = first[value] + 64 * (torch.arange(value.numel(), device=umap.device) - value_run[value])
    return value_run, torch.cat([begin, first[n:]]), torch.argsort(umap, stable=True)


def _row_factors(keep):
    """The plan's constants of the chain rule, laid out with its first gradient:
    zeta of every row, the rows of each nodal value, the first row's value and the
    factor of the constant term (reading them back costs a synchronisation each,
    which a backward does not repeat)."""
    if "row_factors" not in keep:
        eoff, umap = keep["sum_eoff"], keep["umap"]
        zrow = torch.repeat_interleave(keep["sum_zeta"].double(), (eoff[1:] - eoff[:-1]))
        runs = _value_runs(umap, int(keep["fu"].shape[0]))
        factor = float(keep["sum_zeta"].sum().item()) + float(keep["zeta0"])
        keep["row_factors"] = (zrow, runs, int(umap[0].item()), factor)
    return keep["row_factors"]


def _fu_gradient(ip, Fbar, dC_root):
    """Chain rule from dL/dF (plan rows) and dL/d(constant term) to dL/dfu:
    F = zeta (fu[umap] - c), offset = zeta0 fu[u0] + c sum(zeta), c = fu[u0]."""
    P = ip._plan
    keep = P.keep
    fu = keep["fu"]
    if P.c.n_entries == 0:
        return torch.zeros_like(fu)
    zrow, (value_run, begin, rows), u0, factor = _row_factors(keep)
    dfu = torch.empty_like(fu)
    n, n_runs, d_out = int(fu.shape[0]), int(begin.numel()) - 1, int(fu.shape[1])
    nws = capi.size("smx_nodal_adjoint_workspace", n, n_runs, d_out)
    ws = torch.empty(nws, dtype=torch.uint8, device=fu.device)
    ptr = capi.ptr
    capi.call("smx_nodal_adjoint", ptr(Fbar), ptr(zrow), n, n_runs, d_out, ptr(value_run), ptr(begin), ptr(rows),
              ptr(dC_root), factor, u0, ptr(dfu), ptr(ws), nws, capi.stream_ptr(torch.cuda.current_stream()))
    return dfu


class _SmolyakFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, fu, ip):
        ctx.ip = ip
        ctx.save_for_backward(x)
        return ip(x, precision="fp32")

    @staticmethod
    def backward(ctx, g):
        (x,) = ctx.saved_tensors
        ip = ctx.ip
        sp = ip.spectral_plan()
        need_x, need_fu = ctx.needs_input_grad[0], ctx.needs_input_grad[1]
        # the error flag is read once everything is queued
        dx, dC = sp.vjp(x.contiguous(), g.contiguous(), need_x=need_x, need_coef=need_fu, check=False)
        dfu = None
        if need_fu:
            Fbar = sp.coefficient_adjoint(dC)
            dfu = _fu_gradient(ip, Fbar, dC[0])
        dx = dx.to(x.dtype) if dx is not None else None
        sp.check_vjp()
        return dx, dfu, None


def interpolate(ip, x, nodal_values=None):
    """y = I[f](x) (FP32 orthogonal form) with gradients w.r.t. x and the nodal values.

    ``nodal_values`` defaults to ``ip.nodal_values``; pass a tensor with
    ``requires_grad=True`` to receive dL/d(nodal values).  A tensor with other
    values than the interpolant's is loaded with ``ip.set_nodal_values``."""
    fu = ip.nodal_values if nodal_values is None else nodal_values
    if fu is not ip.nodal_values and not torch.equal(fu.detach(), ip.nodal_values):
        ip.set_nodal_values(fu.detach())
    if not isinstance(x, torch.Tensor):
        x = torch.as_tensor(x)
    x = x.to(device=fu.device, dtype=torch.float64)
    return _SmolyakFunction.apply(x, fu, ip)
