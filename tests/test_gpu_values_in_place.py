"""Nodal values that a program updates in place, as optimizers do: the interpolant follows
every update, and what it was set from does not change with the program's tensor."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d_out", [1, 20])
def test_updates_in_place_are_seen(d_out):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes
    from smolyax_gb300.autograd import interpolate

    d = 10
    k = np.log((2 + np.arange(d)) / np.log(2))
    ip = SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=5.0, d_out=d_out,
                                        f=fns.rational_vec(d, d_out, seed=3))
    x = torch.as_tensor(np.random.default_rng(0).uniform(-1, 1, (50, d)), device="cuda")
    values = ip.nodal_values.clone().requires_grad_(True)
    first = interpolate(ip, x, values).detach()
    for step in range(1, 4):  # the interpolant is linear in its values
        with torch.no_grad():
            values += 1.0
        y = interpolate(ip, x, values).detach()
        assert float((y - first - step).abs().max()) <= 1e-5 * (step + 1)
    kept = ip(x, precision="fp64")
    with torch.no_grad():
        values.zero_()
    ip.spectral_plan()
    assert torch.equal(ip(x, precision="fp64"), kept) and float(ip.nodal_values.abs().min()) > 0
