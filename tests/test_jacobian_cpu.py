"""Tables of the FP64 Jacobian (``smolyax_gb300/jacobian.py``), no GPU needed:
a host replay of the kernels' sums over the tables against central formulas of
the same polynomial, entry by entry."""
import numpy as np
import pytest

from smolyax_gb300.jacobian import UNIT, jacobian_terms
from test_layout_cpu import python_tree


def _phi(fam, z, n):
    p, d = [np.ones_like(z)], [np.zeros_like(z)]
    pm1 = dm1 = np.zeros_like(z)
    for m in range(n):
        al, be = ((2 * m + 1) / (m + 1), m / (m + 1)) if fam == 0 else (np.sqrt(2 / (m + 1)), np.sqrt(m / (m + 1)))
        pn, dn = al * z * p[-1] - be * pm1, al * (p[-1] + z * d[-1]) - be * dm1
        pm1, dm1 = p[-1], d[-1]
        p.append(pn)
        d.append(dn)
    return p, d


@pytest.mark.parametrize("d,t,fam", [(1, 6.0, 0), (2, 9.0, 1), (5, 6.0, 0), (12, 6.0, 1), (60, 5.8, 0), (4, 14.0, 0)])
def test_tables_replay_the_derivative(d, t, fam):
    tr = python_tree(list(np.log((2 + np.arange(d)) / np.log(2))), t)
    n = tr["parent"].size
    maxdeg = np.zeros(d, np.int64)
    np.maximum.at(maxdeg, tr["dim"][1:], tr["deg"][1:])
    host = jacobian_terms(tr["parent"], tr["dim"], tr["deg"], tr["level"], maxdeg)
    rng = np.random.default_rng(d)
    x, C = rng.uniform(-1, 1, (7, d)), rng.normal(size=(n, 2))
    tab = [_phi(fam, x[:, j], int(maxdeg[j])) for j in range(d)]
    slots = [(j, g) for j in host["dim"] for g in range(1, maxdeg[j] + 1)]
    assert len(slots) == host["n_slots"]
    phi = np.stack([tab[j][0][g] for j, g in slots])
    dphi = np.stack([tab[j][1][g] for j, g in slots])
    rows = np.stack([np.prod(phi[host["row_slot"][host["row_off"][r] : host["row_off"][r + 1]]], axis=0)
                     for r in range(host["n_rows"])])
    J = np.zeros((7, 2, d))
    seen = 0
    for h, j in enumerate(host["dim"]):
        for u in range(host["unit_off"][h], host["unit_off"][h + 1]):
            t0, t1, slot, uh = host["unit"][u]
            assert uh == h and 0 < t1 - t0 <= UNIT and slots[slot][0] == j
            seen += t1 - t0
            terms = host["term"][t0:t1]
            J[:, :, j] += dphi[slot][:, None] * (rows[terms[:, 0]].T @ C[terms[:, 1]])
    assert seen == tr["level"].sum() == host["term"].shape[0]
    ref = np.zeros_like(J)
    for e in range(1, n):
        path, q = [], e
        while q > 0:
            path.append((tr["dim"][q], tr["deg"][q]))
            q = tr["parent"][q]
        for i, (j, g) in enumerate(path):
            v = tab[j][1][g].copy()
            for i2, (j2, g2) in enumerate(path):
                if i2 != i:
                    v *= tab[j2][0][g2]
            ref[:, :, j] += v[:, None] * C[e][None, :]
    np.testing.assert_allclose(J, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())
