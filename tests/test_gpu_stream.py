"""Stream evaluator (``csrc/stream_eval.cuh``) against the general tables of the
same plan (the struct with ``stream.pass = 0``), at the edges of its tiles (128
points and 4 outputs per pass or 96 and 8 in FP32, 32 points and 1 or 4 outputs
in FP64), with tiles split over clusters of 2, 4 and 8 blocks, non-finite
coordinates and strided rows.

Bounds, relative to the largest output: FP32 1e-6 (the bound of every FP32
evaluator here; both sides are within half of it), FP64 1e-13 (sums of ~1e4
terms of the size of the result)."""
import ctypes

import numpy as np
import pytest

import functions as fns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,d,t,d_out,P", [("leja", 1, 5.0, 2, 1), ("gh", 4, 9.0, 4, 127), ("leja", 30, 7.0, 5, 128),
                                              ("gh", 60, 6.5, 8, 129), ("leja", 200, 6.5, 9, 300),
                                              ("gh", 20, 7.0, 15, 1000), ("leja", 10, 8.0, 1, 33),
                                              ("gh", 100, 7.0, 1, 4900), ("leja", 300, 6.0, 3, 31),
                                              ("leja", 20, 7.0, 6, 15000), ("gh", 12, 8.0, 1, 9900)])
def test_stream_matches_the_general_tables(kind, d, t, d_out, P):
    import torch

    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes
    from smolyax_gb300 import _capi as capi

    k = np.log((2 + np.arange(d)) / np.log(2))
    gen = nodes.Leja(domains=[(-1.0, 1.0 + 0.1 * (j % 2)) for j in range(d)]) if kind == "leja" else \
        nodes.GaussHermite(dim=d)
    f = fns.rational_vec(d, d_out, seed=3) if kind == "leja" else fns.exponential(d, d_out, seed=3)
    ip = SmolyakBarycentricInterpolator(node_gen=gen, k=k, t=t, d_out=d_out, f=f)
    sp = ip.spectral_plan()
    rng = np.random.default_rng(P)
    wide = torch.as_tensor(rng.uniform(-1, 1, (P, d + 3)) if kind == "leja" else rng.normal(size=(P, d + 3)) * 0.7,
                           device="cuda")
    if P > 40:
        wide[37, 0], wide[5, d - 1 if ip._maxdeg[d - 1] else 0] = float("inf"), float("nan")
    st = capi.stream_ptr(torch.cuda.current_stream())

    def run(struct, fn, dtype):
        y = torch.full((P, d_out), -1.0, dtype=dtype, device="cuda")
        capi.call(fn, ctypes.byref(struct), capi.ptr(wide), P, d + 3, capi.ptr(y), st)
        return y.cpu().numpy()

    forms = [(sp.fp64_form()[0], "smx_spectral_eval64", torch.float64, 1e-13)]
    if d_out > 1:
        forms.append((sp.c, "smx_spectral_eval", torch.float32, 1e-6))
    for struct, fn, dtype, bound in forms:
        assert struct.stream.pass_ > 0
        plain = type(struct).from_buffer_copy(struct)
        plain.stream.pass_ = 0
        got, ref = run(struct, fn, dtype), run(plain, fn, dtype)
        assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.isnan(got).any() == (P > 40)
        err = np.nanmax(np.abs(got - ref)) / np.nanmax(np.abs(ref))
        print("%s d=%d d_out=%d P=%d: %.2e" % (fn, d, d_out, P, err))
        assert err <= bound
        # a point's value does not depend on its batch (nor on how its tile is split)
        for n in {1, min(P, 400), min(P, 1500), min(P, 3000)}:
            tail = torch.full((n, d_out), -1.0, dtype=dtype, device="cuda")
            capi.call(fn, ctypes.byref(struct), capi.ptr(wide[P - n :]), n, d + 3, capi.ptr(tail), st)
            np.testing.assert_array_equal(tail.cpu().numpy(), got[P - n :])
