"""FP64 Jacobian of the orthogonal form (``csrc/jacobian64.cu``) against the
combination sum's (``smx_jacobian``), at the edges of its tiles: 4 points per
thread, 16 to 512 points per block, 32 outputs and 32 dimensions per tile; with
points on interpolation nodes (NaN in that dimension alone) and non-finite
coordinates.

Bound: the combination sum's terms are up to ~1e4 times the derivative, so
its FP64 rounding leaves up to ~1e4 * 2^-53 * sqrt(summands) ~ 1e-10 of the
largest component; that is the bound between the two."""
import numpy as np
import pytest

import functions as fns

pytestmark = pytest.mark.gpu


def _combination(ip, x):
    import torch

    from smolyax_gb300 import _capi as capi

    pl = ip._plan
    J = torch.empty(x.shape[0], ip.d_out, ip.d_in, dtype=torch.float64, device=x.device)
    ws = torch.empty(capi.size("smx_jacobian_workspace", pl.ref(), x.shape[0]), dtype=torch.uint8, device=x.device)
    capi.call("smx_jacobian", pl.ref(), capi.ptr(x), x.shape[0], ip.d_in, capi.ptr(J), capi.ptr(ws), ws.numel(),
              capi.stream_ptr(torch.cuda.current_stream()))
    return J.cpu().numpy()


@pytest.mark.parametrize("kind,d,t,d_out,P", [("leja", 1, 6.0, 1, 5), ("gh", 1, 6.0, 3, 4), ("leja", 10, 7.5, 1, 513),
                                              ("gh", 33, 6.5, 5, 17), ("leja", 40, 6.5, 32, 16),
                                              ("gh", 31, 6.0, 33, 1), ("leja", 64, 6.0, 70, 19), ("gh", 3, 13.0, 2, 9)])
def test_matches_the_combination_sum(kind, d, t, d_out, P):
    import torch

    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    gen = nodes.Leja(dim=d) if kind == "leja" else nodes.GaussHermite(dim=d)
    f = fns.rational_vec(d, d_out, seed=3) if kind == "leja" else fns.exponential(d, d_out, seed=3)
    ip = SmolyakBarycentricInterpolator(node_gen=gen, k=k, t=t, d_out=d_out, f=f)
    rng = np.random.default_rng(P)
    x = rng.uniform(-1, 1, (P, d)) if kind == "leja" else rng.normal(size=(P, d)) / np.sqrt(2)
    x[0, 0] = gen[0](int(ip._maxdeg[0]))[-1]  # a node of the finest rule of dimension 0
    if P > 4:
        x[3, min(1, d - 1)], x[4, 0] = np.inf, np.nan
    xd = torch.as_tensor(x, device="cuda")
    J = ip.gradient(xd).cpu().numpy()
    assert ip._jacobian_plan() is not None
    ref = _combination(ip, xd)
    assert np.array_equal(np.isnan(J), np.isnan(ref))
    assert np.all(np.isnan(J[0, :, 0])) and (d == 1 or np.all(np.isfinite(J[0, :, 1:])))
    ok = np.isfinite(ref)
    if ok.any():
        assert np.max(np.abs(J[ok] - ref[ok])) <= 1e-10 * np.max(np.abs(ref[ok]))
    # chunks of points (a small memory limit) give the same values
    ip._memory_limit = 1e-4
    np.testing.assert_array_equal(ip.gradient(xd).cpu().numpy(), J)
