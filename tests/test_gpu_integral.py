"""The integral kernel (``smx_integral``, ``csrc/eval64.cu``) at the edges of its
row chunks and output lanes, against the same FP64 sum on the host."""
import numpy as np
import pytest

import functions as fns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d_out,t", [(1, 4.0), (3, 6.5), (32, 5.0), (33, 6.0)])
def test_integral_lanes_and_chunks(d_out, t):
    """The integral's row chunks (512) and output lanes against the same sum in
    FP64 on the host: rounding only, 1e-13 of sum |term|."""
    from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes

    d = 20
    k = np.log((2 + np.arange(d)) / np.log(2))
    ip = SmolyakBarycentricInterpolator(node_gen=nodes.GaussHermite(dim=d), k=k, t=t, d_out=d_out,
                                        f=fns.exponential(d, d_out, seed=3))
    q = ip.integral().cpu().numpy()
    keep = {key: v.cpu().numpy() for key, v in ip._plan.keep.items() if hasattr(v, "cpu")}
    F = keep["F64"].reshape(-1, d_out)
    total, size = keep["offset"].copy(), np.abs(keep["offset"])
    for s in range(ip._plan.c.n_summands):
        w = np.ones(1)
        for u in keep["sum_pairs"][keep["sum_poff"][s] : keep["sum_poff"][s + 1]]:
            o, g = keep["pair_voff"][u], keep["pair_deg"][u]
            w = np.outer(w, keep["qnode"][o : o + g + 1]).ravel()
        rows = F[keep["sum_eoff"][s] : keep["sum_eoff"][s + 1]]
        total += w @ rows
        size += np.abs(w) @ np.abs(rows)
    assert np.max(np.abs(q - total) / size) <= 1e-13
