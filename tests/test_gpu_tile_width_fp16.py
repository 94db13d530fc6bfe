"""The tile width does not change a value of the scaled FP16 product either (row scale per
64 products, column scale, K slices, D in blocks of 32 columns for the adjoints): points of
batches for which the rule (``csrc/tile_rule.h``) takes 64, 128 and 256 columns are equal
bit for bit."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def _width(rows, cols, slices=1):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cost = {bn: -(-(-(-rows // 128) * slices * -(-cols // bn)) // sms) * w for bn, w in ((256, 177), (128, 100), (64, 94))}
    return min(cost, key=cost.get)


def _plan(d, n, d_out):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, indices, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    t = indices.find_approximate_threshold(k, n, nested=True, accuracy=0.05)
    f = fns.rational_vec(d, d_out, seed=3)
    f.vectorized = True
    return SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=t, d_out=d_out, f=f).spectral_plan()


@pytest.mark.parametrize("n,d_out", [(900, 150), (900, 301), (6000, 150)])
def test_values(n, d_out):
    sp = _plan(40, n, d_out)
    assert (sp.tc_splits() > 1) == (n > 2500)
    sizes = [next(P for P in range(101, 20000, 100) if _width(P, d_out, sp.tc_splits()) == w) for w in (64, 128, 256)]
    x = torch.rand(max(sizes), 40, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    y = [sp.evaluate(x[:P].contiguous(), torch.empty(P, d_out, dtype=torch.float32, device="cuda")) for P in sizes]
    for a in y:
        for b in y:
            n_both = min(a.shape[0], b.shape[0])
            assert torch.equal(a[:n_both], b[:n_both])


def test_adjoints():
    sp = _plan(200, 5000, 130)
    rows = sp._backward_ops()["walk"][1].n_rows
    sizes = (1, 1000, 4000)
    assert [_width(rows, P) for P in sizes] == [64, 128, 256]
    gen = torch.Generator("cuda").manual_seed(0)
    x = torch.rand(4000, 200, dtype=torch.float64, device="cuda", generator=gen)
    g = torch.randn(4000, 130, device="cuda", generator=gen)
    dx = [sp.vjp(x[:P].contiguous(), g[:P].contiguous(), need_coef=False)[0] for P in sizes]
    assert torch.equal(dx[0], dx[2][:1]) and torch.equal(dx[1], dx[2][:1000])
