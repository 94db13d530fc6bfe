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


def _products(sp, x):
    """A [P, entries] in FP64, from the index set and the recurrences alone."""
    from smolyax_gb300.spectral import _phi_table

    tr, _, maxdeg, fam, fa, fb = sp._fwd_args[:6]
    A = np.ones((tr["parent"].size, x.shape[0]))
    table = {j: _phi_table(int(fam[j]), fa[j] * x[:, j] + fb[j], int(maxdeg[j])) for j in np.nonzero(maxdeg)[0]}
    for e in range(1, A.shape[0]):
        A[e] = A[tr["parent"][e]] * table[int(tr["dim"][e])][int(tr["deg"][e])]
    return A.T


def _set_coefficients(sp, C):
    """The plan's tensor-core operands from other coefficients (row 0 stays)."""
    tc = sp.tc
    tc["Bd"][:, : tc["K"]] = torch.as_tensor(C[tc["ent_h"][::-1]].T.astype(np.float32), device="cuda")
    tc.pop("f16")


def _term_error(sp, C, x):
    """Per output: largest error over the points, relative to sum |terms|."""
    y = torch.empty(x.shape[0], C.shape[1], dtype=torch.float32, device="cuda")
    sp.evaluate(torch.as_tensor(x, device="cuda"), y)
    A, C32 = _products(sp, x), C.astype(np.float32).astype(float)
    return np.max(np.abs(y.cpu().numpy() - A @ C32) / (np.abs(A) @ np.abs(C32)), axis=0)


@pytest.mark.parametrize("far", [1.0, 30.0, 3000.0])
@pytest.mark.parametrize("j", [0, 2, 8])
def test_entries_without_coefficients_do_not_hide_the_others(j, far):
    """Values where the target ignores a coordinate that lies far outside its box:
    the entries of that coordinate have no coefficients, whatever their products."""
    d = 20
    ip = _plan(d, 900, 24, fns.rational_vec(d, 24, seed=3))
    sp = ip.spectral_plan()
    tr = sp._fwd_args[0]
    uses = np.zeros(tr["parent"].size, dtype=bool)
    for e in range(1, uses.size):
        uses[e] = uses[tr["parent"][e]] or tr["dim"][e] == j
    C = np.where(uses[:, None], 0.0, sp.C64.cpu().numpy())
    _set_coefficients(sp, C)
    x = np.random.default_rng(0).uniform(-1, 1, (200, d))
    x[:, j] = far
    assert _term_error(sp, C, x).max() <= 1e-6


@pytest.mark.parametrize("j,far", [(0, 1.0), (0, 30.0), (2, 1e3), (2, 1e4), (8, 1e5)])
def test_small_terms_beside_large_ones(j, far):
    """Values of outputs without a coordinate beside outputs of that coordinate alone,
    whose terms are up to 1e16 times larger."""
    d = 20
    ip = _plan(d, 900, 24, fns.rational_vec(d, 24, seed=3))
    sp = ip.spectral_plan()
    tr = sp._fwd_args[0]
    uses = np.zeros(tr["parent"].size, dtype=bool)
    for e in range(1, uses.size):
        uses[e] = uses[tr["parent"][e]] or tr["dim"][e] == j
    C = sp.C64.cpu().numpy().copy()
    C[1:, 0::2][uses[1:]] = 0.0
    C[1:, 1::2][~uses[1:]] = 0.0
    _set_coefficients(sp, C)
    x = np.random.default_rng(0).uniform(-1, 1, (200, d))
    x[:, j] = far
    assert _term_error(sp, C, x).max() <= 1e-6


@pytest.mark.parametrize("size", [1.0, 1e-4, 1e-6, 1e-8])
@pytest.mark.parametrize("d_out", [2, 130])
def test_derivatives_of_small_outputs_in_their_own_inputs(d_out, size):
    """dL/dx in the inputs that only the small outputs use, beside large outputs of
    other inputs, relative to their own size."""
    d, half = 20, d_out // 2
    h = fns.rational_vec(10, d_out, seed=3)

    def f(x):
        return np.concatenate([h(x[0::2])[:half], size * h(x[1::2])[half:]])

    ip = _plan(d, 400, d_out, f)
    sp = ip.spectral_plan()
    assert sp._backward_ops()["walk"] is not None
    x = _x(100, d)
    g = torch.as_tensor(np.random.default_rng(1).normal(size=(100, d_out)).astype(np.float32), device="cuda")
    dx, _ = sp.vjp(x, g, need_coef=False)
    ref = torch.einsum("po,poi->pi", g.double(), ip.gradient(x))
    for i in (0, 1):
        assert float((dx - ref)[:, i::2].abs().max()) < 1e-5 * float(ref[:, i::2].abs().max())


def _coef_error(sp, x, g):
    """Largest error of dL/dC relative to sum |A g| of the entry and output."""
    _, dC = sp.vjp(torch.as_tensor(x, device="cuda"), torch.as_tensor(g, device="cuda"), need_x=False)
    A, g = _products(sp, x).T, g.astype(float)
    return np.max(np.abs(dC.cpu().numpy() - A @ g) / np.maximum(np.abs(A) @ np.abs(g), 1e-300))


@pytest.mark.parametrize("spread", [1.0, 2.0**20, 2.0**30, 2.0**45])
@pytest.mark.parametrize("d_out", [3, 70])
def test_products_and_cotangents_of_opposite_spread(d_out, spread):
    """dL/dC over points whose products grow as their cotangents fall."""
    ip = _plan(20, 900, d_out, fns.rational_vec(20, d_out, seed=3))
    sp = ip.spectral_plan()
    assert sp._backward_ops()["coef"] is not None
    rng = np.random.default_rng(0)
    P, deg = 200, int(np.max(ip._maxdeg))
    x = rng.uniform(-1, 1, (P, 20))
    w = spread ** rng.uniform(0, 1, P)  # the largest products of the points, about
    x[:, 0] = np.maximum(w ** (1 / deg), np.abs(x[:, 0]))
    g = (rng.normal(size=(P, d_out)) / w[:, None]).astype(np.float32)
    assert _coef_error(sp, x, g) <= 1e-5


def test_points_without_a_cotangent_weigh_nothing():
    """dL/dC where points far outside the box are masked out by a zero cotangent."""
    ip = _plan(20, 900, 5, fns.rational_vec(20, 5, seed=3))
    sp = ip.spectral_plan()
    rng = np.random.default_rng(0)
    x = rng.uniform(-1, 1, (200, 20))
    g = rng.normal(size=(200, 5)).astype(np.float32)
    x[::7] *= 1e4
    g[::7] = 0.0
    assert _coef_error(sp, x, g) <= 1e-5


@pytest.mark.parametrize("n,d_out", [(900, 24), (900, 130), (900, 300), (3000, 17), (3000, 70)])
def test_far_points_among_others(n, d_out):
    """Points far outside the box between points inside, with one slice of K and several:
    term-relative errors, and every value the same in other batches and passes."""
    from smolyax_gb300 import _capi as capi

    import ctypes

    d, P = 20, 333
    ip = _plan(d, n, d_out, fns.rational_vec(d, d_out, seed=3))
    sp = ip.spectral_plan()
    assert (sp.tc_splits() > 1) == (n > 2048)
    C = sp.C64.cpu().numpy()
    x = np.random.default_rng(0).uniform(-1, 1, (P, d))
    x[::5, 1] = 1e3
    x[7::50] *= 1e2
    assert _term_error(sp, C, x).max() <= 1e-6
    xd = torch.as_tensor(x, device="cuda")
    y, got = (torch.empty(P, d_out, dtype=torch.float32, device="cuda") for _ in range(2))
    sp.evaluate(xd, y)
    for part in (slice(5, 6), slice(100, 201), slice(330, 333)):
        alone = torch.empty(xd[part].shape[0], d_out, dtype=torch.float32, device="cuda")
        assert torch.equal(sp.evaluate(xd[part].contiguous(), alone), y[part])
    s = type(sp._tc_struct()).from_buffer_copy(sp._tc_struct())
    s.chunk = 128
    nws = capi.size("smx_tensor_workspace", ctypes.byref(s), P)
    ws = torch.empty(nws, dtype=torch.uint8, device="cuda")
    capi.call("smx_tensor_eval", ctypes.byref(s), capi.ptr(xd), P, d, capi.ptr(got), capi.ptr(ws), nws,
              capi.stream_ptr(torch.cuda.current_stream()))
    assert torch.equal(got, y)


def test_far_points_of_the_c_plan():
    """The C plan carries the FP32 coefficients and column paths too: the same values."""
    from smolyax_gb300 import _capi as capi
    from test_gpu_capi_fp32 import _fp32_plan

    d, P, d_out = 20, 100, 24
    ip = _plan(d, 900, d_out, fns.rational_vec(d, d_out, seed=3))
    sp = ip.spectral_plan()
    x = np.random.default_rng(0).uniform(-1, 1, (P, d))
    x[::5, 1] = 1e3
    xd = torch.as_tensor(x, device="cuda")
    want, got = (torch.empty(P, d_out, dtype=torch.float32, device="cuda") for _ in range(2))
    sp.evaluate(xd, want)
    lib, h = _fp32_plan(ip)
    try:
        nws = lib.smx_fp32_workspace(h, P)
        ws = torch.empty(nws, dtype=torch.uint8, device="cuda")
        capi.call("smx_fp32_eval", h, capi.ptr(xd), P, d, capi.ptr(got), capi.ptr(ws), nws,
                  capi.stream_ptr(torch.cuda.current_stream()))
        torch.cuda.synchronize()
        assert torch.equal(got, want) and _term_error(sp, sp.C64.cpu().numpy(), x).max() <= 1e-6
    finally:
        lib.smx_fp32_plan_destroy(h)
