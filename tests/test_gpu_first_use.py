"""Operands that a plan lays out belong to the plan, not to the stream or the
capture that first evaluates it: a plan whose first evaluation is captured into a
graph evaluates rightly before the graph has run, and the graph rightly when it
runs; a plan first used on one stream is right on another at once, in evaluation
and in the backward."""
import numpy as np
import pytest
import torch

import functions as fns

pytestmark = pytest.mark.gpu


def _ip(d_out, seed=3):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    d = 30
    k = np.log((2 + np.arange(d)) / np.log(2))
    return SmolyakBarycentricInterpolator(node_gen=nodes.Leja(dim=d), k=k, t=6.0, d_out=d_out,
                                          f=fns.rational_vec(d, d_out, seed=seed), precision="fp64")


def _x(P):
    return torch.as_tensor(np.random.default_rng(0).uniform(-1, 1, (P, 30)), device="cuda")


def _close(y, ref):
    return float((y.double() - ref).abs().max()) <= 1e-6 * float(ref.abs().max())


def test_first_evaluation_captured():
    x = _x(200)
    _ip(20)(x, precision="fp32")  # the kernels are loaded
    ip = _ip(20)
    ref = ip(x, precision="fp64")
    sp = ip.spectral_plan()
    y = torch.zeros(200, 20, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sp.evaluate(x, y)
    assert _close(ip(x, precision="fp32"), ref)  # nothing of the graph has run yet
    graph.replay()
    torch.cuda.synchronize()
    assert _close(y, ref)


@pytest.mark.parametrize("call", ["fp32", "bf16x3", "vjp", "gradient"])
def test_first_use_on_another_stream(call):
    x = _x(3000)
    g = torch.ones(3000, 20, device="cuda")
    ip = _ip(20)
    sp = ip.spectral_plan()

    def run():
        if call == "vjp":
            dx, dC = sp.vjp(x, g, check=False)
            return torch.cat([dx.flatten(), dC.flatten()])
        return ip.gradient(x[:300]) if call == "gradient" else ip(x, precision=call)

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(20_000_000)  # the first stream is ~10 ms behind
        first = run()
    with torch.cuda.stream(b):
        second = run()
    torch.cuda.synchronize()
    assert torch.equal(first, second) and bool(torch.isfinite(second).all()) and float(second.abs().max()) > 0
