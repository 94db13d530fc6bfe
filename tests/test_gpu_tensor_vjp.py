"""dL/dx by the chunked gradient walk (``csrc/tensor_vjp.cu``) against the FP64
Jacobian contracted with the cotangent, at 1e-5 of the scale (the FP32 form's
bound): output counts around the 64-output slices, point counts around a block's
32 points and the GEMM's 128, one-entry plans up to plans of several chunks, both
families; a point's result does not depend on its batch, and a point that is not
finite leaves the others alone."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def _plan(d, d_out, n, rule="Leja"):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, indices, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    t = indices.find_approximate_threshold(k, n, nested=rule == "Leja", accuracy=0.05)
    ip = SmolyakBarycentricInterpolator(node_gen=getattr(nodes, rule)(dim=d), k=k, t=t, d_out=d_out,
                                        f=fns.rational_vec(d, d_out, seed=3))
    return ip, ip.spectral_plan()


@pytest.mark.parametrize("d,d_out,n,rule", [(1, 1, 4, "Leja"), (5, 2, 120, "Leja"), (40, 63, 900, "Leja"),
                                            (40, 64, 900, "GaussHermite"), (90, 65, 2500, "Leja"),
                                            (200, 130, 5000, "Leja")])
@pytest.mark.parametrize("P", [1, 31, 33, 129, 1000])
def test_walk_matches_jacobian(d, d_out, n, rule, P):
    ip, sp = _plan(d, d_out, n, rule)
    assert sp._backward_ops()["walk"] is not None
    rng = np.random.default_rng(P)
    x = torch.as_tensor(rng.uniform(-1, 1, (P, d)), device="cuda")
    g = torch.as_tensor(rng.normal(size=(P, d_out)).astype(np.float32), device="cuda")
    g[P // 2] *= 1e-20  # a point's cotangent has its own scale
    dx, _ = sp.vjp(x, g, need_x=True, need_coef=False)
    ref = torch.einsum("po,poi->pi", g.double(), ip.gradient(x))
    for got, want in ((dx, ref), (dx[P // 2], ref[P // 2])):
        assert float((got - want).abs().max()) < 1e-5 * float(want.abs().max())
    one = sp.vjp(x[P - 1 :].contiguous(), g[P - 1 :].contiguous(), need_x=True, need_coef=False)[0]
    assert torch.equal(one[0], dx[P - 1])


def test_non_finite_points_stay_alone():
    ip, sp = _plan(40, 5, 900)
    x = torch.rand(70, 40, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    g = torch.ones(70, 5, device="cuda")
    clean = sp.vjp(x, g, need_x=True, need_coef=False)[0]
    x[3, 0], g[40, 2], g[41, 1] = float("nan"), float("inf"), float("nan")
    dx = sp.vjp(x, g, need_x=True, need_coef=False)[0]
    keep = [i for i in range(70) if i not in (3, 40, 41)]
    assert torch.equal(dx[keep], clean[keep])
    assert not torch.isfinite(dx[[3, 40, 41]]).all(dim=1).any()


def test_plans_outside_the_walk_keep_their_path():
    ip, sp = _plan(1000, 2, 12000)
    assert sp._backward_ops()["walk"] is None  # the rows of 32 points do not fit in shared memory
    x = torch.rand(33, 1000, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(0)) * 2 - 1
    g = torch.ones(33, 2, device="cuda")
    ref = torch.einsum("po,poi->pi", g.double(), ip.gradient(x))
    dx = sp.vjp(x, g, need_x=True, need_coef=False)[0]
    assert float((dx - ref).abs().max()) < 1e-5 * float(ref.abs().max())
