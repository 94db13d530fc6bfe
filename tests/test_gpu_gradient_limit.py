"""``gradient`` keeps to the memory limit: where the orthogonal form's coefficients would
take more scratch than the limit, the combination sum computes the Jacobian, as it does
for the other rules; coefficients that are there already are used."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def _ip(limit):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    d, d_out = 40, 64
    k = np.log((2 + np.arange(d)) / np.log(2))
    f = fns.rational_vec(d, d_out, seed=3)
    f.vectorized = True
    return SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=7.0, d_out=d_out, f=f,
                                          memory_limit=limit)


def test_a_jacobian_stays_within_the_limit():
    x = torch.as_tensor(np.random.default_rng(0).uniform(-1, 1, (3, 40)), device="cuda")
    ref = _ip(4.0).gradient(x)
    limit = 2.0**-9  # 2 MB
    ip = _ip(limit)
    rows = 8 * ip.d_out * int(ip._plan.c.n_entries)
    assert rows > limit * 1024**3
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    J = ip.gradient(x)
    used = torch.cuda.max_memory_allocated() - before - J.numel() * 8
    assert used <= 1.1 * limit * 1024**3 + 4096
    assert float((J - ref).abs().max()) <= 1e-10 * float(ref.abs().max())
    ip.spectral_plan()  # an evaluation needs the coefficients all the same
    assert torch.equal(ip.gradient(x), ref)


@pytest.mark.parametrize("d_out", [1, 64])
def test_the_coefficients_take_what_is_counted(d_out):
    """The bytes that the limit is compared with cover what building them allocates."""
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    d = 40
    k = np.log((2 + np.arange(d)) / np.log(2))
    f = fns.rational_vec(d, d_out, seed=3)
    f.vectorized = True
    ip = SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=7.0, d_out=d_out, f=f)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    ip._coefficients()
    assert torch.cuda.max_memory_allocated() - before <= 1.1 * ip._coefficient_bytes() + (1 << 18)
