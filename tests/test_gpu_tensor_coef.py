"""dL/d(coefficients) by the sliced FP16 panel (``csrc/tensor_vjp.cu``
smx_tensor_vjp_coef) against the FP64 sum over the points, at 1e-5 of the scale
(the FP32 form's bound): point counts around a slice of 64 points, output counts
around the 64-output tiles, one entry up to plans with one block per SM, several
passes, both families, and a cotangent whose points and outputs have very
different sizes."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def _plan(d, d_out, n, rule="Leja", **kw):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, indices, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    t = indices.find_approximate_threshold(k, n, nested=rule == "Leja", accuracy=0.05)
    ip = SmolyakBarycentricInterpolator(node_gen=getattr(nodes, rule)(dim=d), k=k, t=t, d_out=d_out,
                                        f=fns.rational_vec(d, d_out, seed=3), **kw)
    return ip, ip.spectral_plan()


def _direct(sp, x, g):
    from smolyax_gb300.spectral import _phi_table

    tr, _, maxdeg, fam, fa, fb = sp._fwd_args[:6]
    A = np.ones((tr["parent"].size, x.shape[0]))
    table = {j: _phi_table(int(fam[j]), fa[j] * x[:, j] + fb[j], int(maxdeg[j])) for j in np.nonzero(maxdeg)[0]}
    for e in range(1, A.shape[0]):
        A[e] = A[tr["parent"][e]] * table[int(tr["dim"][e])][int(tr["deg"][e])]
    return A @ g


@pytest.mark.parametrize("d,d_out,n,rule", [(1, 1, 4, "Leja"), (5, 2, 120, "Leja"), (40, 63, 900, "Leja"),
                                            (40, 64, 900, "GaussHermite"), (90, 65, 2500, "Leja"),
                                            (200, 200, 5000, "Leja"), (500, 3, 3000, "Leja")])
@pytest.mark.parametrize("P", [1, 63, 65, 128, 1000])
def test_matches_direct_sum(d, d_out, n, rule, P):
    ip, sp = _plan(d, d_out, n, rule)
    assert sp._backward_ops()["coef"] is not None
    rng = np.random.default_rng(P)
    x = rng.uniform(-1, 1, (P, d))
    g = rng.normal(size=(P, d_out)).astype(np.float32)
    g[:, d_out // 2] *= np.float32(1e-20)  # an output has its own scale
    _, dC = sp.vjp(torch.as_tensor(x, device="cuda"), torch.as_tensor(g, device="cuda"), need_x=False)
    ref = _direct(sp, x, g.astype(np.float64))
    got = dC.cpu().numpy()
    for a, b in ((got, ref), (got[:, d_out // 2], ref[:, d_out // 2])):
        assert np.abs(a - b).max() < 1e-5 * np.abs(b).max()


def test_several_passes_add_up():
    ip, sp = _plan(40, 5, 900)
    rng = np.random.default_rng(0)
    x = torch.as_tensor(rng.uniform(-1, 1, (1000, 40)), device="cuda")
    g = torch.as_tensor(rng.normal(size=(1000, 5)).astype(np.float32), device="cuda")
    g[500:] *= 1e-3
    one = sp.vjp(x, g, need_x=False)[1]
    t, _ = sp._backward_ops()["coef"]
    t.chunk = 128
    many = sp.vjp(x, g, need_x=False)[1]
    assert float((one - many).abs().max()) < 1e-5 * float(one.abs().max())


def test_plans_with_many_slots_keep_their_path():
    ip, sp = _plan(1000, 2, 5000)
    assert sp._backward_ops()["coef"] is None  # the basis rows of 64 points do not fit in shared memory
    rng = np.random.default_rng(0)
    x, g = rng.uniform(-1, 1, (70, 1000)), rng.normal(size=(70, 2)).astype(np.float32)
    dC = sp.vjp(torch.as_tensor(x, device="cuda"), torch.as_tensor(g, device="cuda"), need_x=False)[1].cpu().numpy()
    ref = _direct(sp, x, g.astype(np.float64))
    assert np.abs(dC - ref).max() < 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("P", [1, 129, 700])
def test_basis_rows_of_the_walk_are_shared(P):
    """dL/dx and dL/dC together (one set of basis rows) are what they are alone."""
    ip, sp = _plan(40, 5, 900)
    rng = np.random.default_rng(P)
    x = torch.as_tensor(rng.uniform(-1, 1, (P, 40)), device="cuda")
    g = torch.as_tensor(rng.normal(size=(P, 5)).astype(np.float32), device="cuda")
    dx, dC = sp.vjp(x, g)
    assert torch.equal(dx, sp.vjp(x, g, need_coef=False)[0]) and torch.equal(dC, sp.vjp(x, g, need_x=False)[1])
    sp._backward_ops()["walk"][1].chunk = 128  # several passes of the walk: its rows are of the last
    many = sp.vjp(x, g)
    assert torch.equal(many[0], dx) and torch.equal(many[1], dC)
