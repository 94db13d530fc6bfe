"""dL/d(nodal values) from dL/dF (``csrc/tensor_vjp.cu`` smx_nodal_adjoint) against
the sums in numpy, at the FP64 rounding of a sum of all rows (2^-50 of the sum of
the terms' sizes): one value, values without rows, counts around the blocks of 512
rows and widths around the 256 columns of a block."""
import numpy as np
import pytest
import torch

from smolyax_gb300 import _capi as capi
from smolyax_gb300.autograd import _value_runs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rows,d_out", [(1, 1, 1), (3, 0, 2), (5, 17, 3), (511, 700, 64), (513, 2000, 65),
                                          (1025, 1025, 256), (700, 3000, 300)])
def test_matches_direct_sum(n, rows, d_out):
    rng = np.random.default_rng(n + rows)
    u = np.where(rng.random(rows) < 0.5, 0, rng.integers(0, n, rows))  # one value in half of the rows
    F, zeta, root = rng.normal(size=(max(rows, 1), d_out)), rng.integers(-9, 9, max(rows, 1)).astype(float), rng.normal(size=d_out)
    first, factor = n // 2, 2.5
    ref = np.zeros((n, d_out))
    terms = zeta[:rows, None] * F[:rows]
    np.add.at(ref, u, terms)
    ref[first] += factor * root - terms.sum(0)
    T = lambda a: torch.as_tensor(a, device="cuda")
    value_run, begin, order = _value_runs(T(u.astype(np.int64)), n)
    assert int((begin[1:] - begin[:-1]).max()) <= 64 if rows else begin.numel() == 1
    F_d, zeta_d, root_d = T(F), T(zeta), T(root)
    row = order if rows else torch.zeros(1, dtype=torch.int64, device="cuda")
    out = torch.full((n, d_out), 7.0, dtype=torch.float64, device="cuda")
    n_runs = begin.numel() - 1
    nws = capi.size("smx_nodal_adjoint_workspace", n, n_runs, d_out)
    ws = torch.empty(nws, dtype=torch.uint8, device="cuda")
    capi.call("smx_nodal_adjoint", capi.ptr(F_d), capi.ptr(zeta_d), n, n_runs, d_out, capi.ptr(value_run),
              capi.ptr(begin), capi.ptr(row), capi.ptr(root_d), factor, first, capi.ptr(out), capi.ptr(ws), nws, None)
    torch.cuda.synchronize()
    bound = 2.0**-50 * (np.abs(terms).sum(0) + factor * np.abs(root)) + 1e-300
    assert np.all(np.abs(out.cpu().numpy() - ref) <= bound)
