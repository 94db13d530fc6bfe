"""Operands that are built on first use, first used inside a graph capture: their
construction is only recorded there, so the plan does not keep them, and evaluations
outside the graph are right before it has run, while it runs and after it is gone."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def test_bf16_operands_first_used_under_capture():
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    d, d_out, P = 30, 20, 200
    k = np.log((2 + np.arange(d)) / np.log(2))

    def make():
        return SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=6.0, d_out=d_out,
                                              f=fns.rational_vec(d, d_out, seed=3), precision="fp64")

    x = torch.as_tensor(np.random.default_rng(0).uniform(-1, 1, (P, d)), device="cuda")
    want = make()(x, precision="bf16x3")  # the kernels are loaded
    sp = make().spectral_plan()
    out = [torch.zeros(P, d_out, dtype=torch.float32, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sp.evaluate(x, out[0], mode="bf16x3")
        sp.evaluate(x, out[1], mode="bf16x3")
    assert "bf16" not in sp.tc  # what a graph has only recorded is not the plan's
    sp.evaluate(x, out[2], mode="bf16x3")
    assert torch.equal(out[2], want)
    for _ in range(2):
        out[0].zero_(), out[1].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want) and torch.equal(out[1], want)
    del graph
    sp.evaluate(x, out[3], mode="bf16x3")
    assert torch.equal(out[3], want)
