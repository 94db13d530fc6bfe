"""The combination sum in FP64 (``csrc/eval64.cu`` contract_kernel) against the
orthogonal form of the same plan (independent tables and kernels) at 1e-10 of the
scale: every width of a block's outputs and more than one pass of them, point
counts around a block's 32, plans of 1 to 8 blocks per cluster, summands of more
pairs than are nested, basis values beyond shared memory; a point's value does not
depend on its batch."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu

PLANS = [(3, 2.5, "Leja"), (6, 10.0, "Leja"), (10, 6.5, "GaussHermite"), (30, 6.0, "Leja"), (100, 6.6, "GaussHermite"),
         (1000, 6.9, "Leja")]


def _ip(d, t, rule, d_out):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    return SmolyakBarycentricInterpolator(node_gen=getattr(nodes, rule)(dim=d), k=k, t=t, d_out=d_out,
                                          f=fns.rational_vec(d, d_out, seed=3), precision="fp64")


def _check(ip, P):
    x = torch.as_tensor(np.random.default_rng(P).uniform(-1, 1, (P, ip.d_in)), device="cuda")
    y = ip(x, precision="fp64_barycentric").reshape(P, -1)
    ref = ip(x, precision="fp64").reshape(P, -1)
    assert float((y - ref).abs().max()) <= 1e-10 * float(ref.abs().max())
    last = ip(x[P - 1 :], precision="fp64_barycentric").reshape(1, -1)
    assert torch.equal(last[0], y[P - 1])


@pytest.mark.parametrize("d,t,rule", PLANS)
@pytest.mark.parametrize("d_out", [1, 3, 8])
def test_plans(d, t, rule, d_out):
    ip = _ip(d, t, rule, d_out)
    for P in (1, 31, 33, 300):
        _check(ip, P)


@pytest.mark.parametrize("d_out", [2, 4, 5, 6, 7, 9, 16, 17])
def test_output_widths(d_out):
    _check(_ip(20, 6.0, "Leja", d_out), 65)
