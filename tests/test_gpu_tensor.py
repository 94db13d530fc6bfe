"""Tensor-core evaluation with scaled FP16 pairs (``csrc/tensor_eval.cu``) at the
edges of its tiles: 32 points and 64 columns per panel tile, 128 points and 128
or 256 outputs per contraction tile, K slices, chunks of points, and the three
homes of the basis rows (shared memory with 16 or 8 warps, global memory).

Bounds: 22 significant bits per operand and FP32 sums in 64-product pieces give
the accuracy of the 3xTF32 product, whose bound here is 1e-6 of the point's
largest output (norm-wise) against the FP64 evaluation."""
import ctypes

import numpy as np
import pytest

import functions as fns

pytestmark = pytest.mark.gpu


def _ip(kind, d, t, d_out, **kw):
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    k = np.log((2 + np.arange(d)) / np.log(2))
    gen = nodes.Leja(dim=d) if kind == "leja" else nodes.GaussHermite(dim=d)
    f = fns.rational_vec(d, d_out, seed=3) if kind == "leja" else fns.exponential(d, d_out, seed=3)
    f.vectorized = True
    return SmolyakBarycentricInterpolator(node_gen=gen, k=k, t=t, d_out=d_out, f=f, **kw)


@pytest.mark.parametrize("kind,d,t,d_out,P", [("leja", 1, 6.0, 16, 1), ("leja", 3, 5.0, 17, 33),
                                              ("gh", 10, 6.0, 128, 31), ("leja", 30, 6.5, 129, 127),
                                              ("gh", 40, 6.5, 257, 129), ("leja", 200, 7.5, 16, 1000),
                                              ("leja", 1000, 7.2, 16, 40), ("leja", 1400, 7.3, 18, 70)])
def test_matches_fp64_and_does_not_depend_on_the_batch(kind, d, t, d_out, P):
    import torch

    ip = _ip(kind, d, t, d_out)
    sp = ip.spectral_plan()
    assert sp.tc is not None
    rng = np.random.default_rng(P)
    x = rng.uniform(-1, 1, (P, d)) if kind == "leja" else rng.normal(size=(P, d)) / np.sqrt(2)
    x = torch.as_tensor(x, device="cuda")
    y = ip(x, precision="fp32").cpu().numpy()
    ref = ip(x, precision="fp64_barycentric").cpu().numpy()
    err = float(np.max(np.max(np.abs(y - ref), axis=1) / np.max(np.abs(ref), axis=1)))
    print("%s d=%d d_out=%d P=%d K=%d slots=%d splits=%d: %.2e" % (kind, d, d_out, P, sp.tc["K"], sp.tc["n_slots"],
                                                                  sp.tc_splits(), err))
    assert err <= 1e-6
    np.testing.assert_array_equal(ip(x[P // 2 :], precision="fp32").cpu().numpy(), y[P // 2 :])
    s = type(sp._tc_struct()).from_buffer_copy(sp._tc_struct())
    s.chunk = 128  # several passes
    from smolyax_gb300 import _capi as capi

    got = torch.empty(P, d_out, dtype=torch.float32, device="cuda")
    nws = capi.size("smx_tensor_workspace", ctypes.byref(s), P)
    ws = torch.empty(nws, dtype=torch.uint8, device="cuda")
    capi.call("smx_tensor_eval", ctypes.byref(s), capi.ptr(x), P, d, capi.ptr(got), capi.ptr(ws), nws,
              capi.stream_ptr(torch.cuda.current_stream()))
    np.testing.assert_array_equal(got.cpu().numpy(), y)


def test_scales_cover_the_exponent_range():
    """Outputs 2^-90 .. 2^90 apart are each as accurate as alone (the output
    scales are exact powers of two: the values scale bit for bit), and points far
    outside the box keep the accuracy relative to
    sum |terms|."""
    import torch

    from test_gpu_spectral import term_relative_error

    ip = _ip("leja", 20, 6.5, 24)
    x = torch.as_tensor(np.random.default_rng(0).uniform(-1, 1, (300, 20)), device="cuda")
    x[200:] *= 20.0
    y = ip(x, precision="fp32").cpu().numpy()
    y64 = ip(x, precision="fp64").cpu().numpy()
    assert np.all(np.isfinite(y))
    assert term_relative_error(ip, x.cpu().numpy(), y, y64) <= 1e-6
    p = (np.arange(24) - 12) * 8
    ip.set_nodal_values(ip.nodal_values * torch.as_tensor(2.0 ** p, device="cuda")[None, :])
    np.testing.assert_array_equal(ip(x, precision="fp32").cpu().numpy(), y * (2.0 ** p).astype(np.float32)[None, :])
