"""Range of the scaled FP16 pairs (``csrc/tensor_eval.cu``, ``csrc/tensor_vjp.cu``):
outputs, entries and points of very different sizes side by side, against FP64.

Bound: 1e-5 of the scale for gradients, 1e-6 for values (the FP32 form's bounds)."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def _plan(d, n, d_out, f, rule="Leja", **kw):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, indices, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    t = indices.find_approximate_threshold(k, n, nested=rule == "Leja", accuracy=0.05)
    return SmolyakBarycentricInterpolator(node_gen=getattr(nodes, rule)(dim=d), k=k, t=t, d_out=d_out, f=f, **kw)


def _x(P, d, seed=0):
    return torch.as_tensor(np.random.default_rng(seed).uniform(-1, 1, (P, d)), device="cuda")


@pytest.mark.parametrize("size", [1e-6, 1e-9, 1e-14])
@pytest.mark.parametrize("d_out", [2, 64, 130])
def test_a_constant_output_does_not_hide_small_ones(d_out, size):
    """dL/dx beside an output that f keeps constant (no coefficients)."""
    h = fns.rational_vec(40, d_out - 1, seed=3)
    ip = _plan(40, 900, d_out, lambda x: np.concatenate([[1.0], size * h(x)]))
    sp = ip.spectral_plan()
    assert sp._backward_ops()["walk"] is not None
    assert float(sp.C64[1:, 0].abs().max()) == 0.0
    x = _x(100, 40)
    g = torch.as_tensor(np.random.default_rng(1).normal(size=(100, d_out)).astype(np.float32), device="cuda")
    dx, _ = sp.vjp(x, g, need_coef=False)
    ref = torch.einsum("po,poi->pi", g.double(), ip.gradient(x))
    assert float((dx - ref).abs().max()) < 1e-5 * float(ref.abs().max())
