"""A plan lays out the operands that its backward reads, and no others: the TF32 rows of
the coefficients are for plans outside the gradient walk's limits."""
import numpy as np
import pytest

import functions as fns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,walk", [(40, 900, True), (1000, 12000, False)])
def test_operands_of_the_path_that_runs(d, n, walk):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, indices, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    t = indices.find_approximate_threshold(k, n, nested=True, accuracy=0.05)
    ip = SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=t, d_out=2, f=fns.rational_vec(d, 2, seed=3))
    ops = ip.spectral_plan()._backward_ops()
    assert (ops["walk"] is not None) == walk
    assert ("Rh" in ops) == ("Rl" in ops) == (not walk)
