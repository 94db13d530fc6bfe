"""More points in one call than the contraction's grid has row tiles for (65535 * 128),
on a plan whose panel takes few bytes a point."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def test_more_points_than_row_tiles():
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    d, P = 3, 65535 * 128 + 1000
    k = np.log((2 + np.arange(d)) / np.log(2))
    f = fns.rational_vec(d, 16, seed=3)
    ip = SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=5.0, d_out=16, f=f)
    assert ip.spectral_plan().tc is not None and ip.spectral_plan().tc["K"] <= 64
    x = torch.rand(P, d, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    y = ip(x, precision="fp32")
    for part in (slice(0, 300), slice(65535 * 128 - 150, 65535 * 128 + 150), slice(P - 300, P)):
        assert torch.equal(y[part], ip(x[part].contiguous(), precision="fp32"))
