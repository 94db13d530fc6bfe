"""Tables of the gradient walk (``smx_layout_build`` kind SMX_LAYOUT_WALK,
``csrc/layout.cu``), no GPU needed: the tables are decoded and walked on the host
in FP64, as ``vjp_walk_kernel`` of ``csrc/tensor_vjp.cu`` does, and compared with
the sum over the index set of cotangent, coefficient and differentiated factor."""
import numpy as np
import pytest

from smolyax_gb300 import _capi as capi
from smolyax_gb300.spectral import WALK_SCALARS, WALK_TABLES
from test_layout_cpu import python_tree


def _tree(d, t):
    tr = python_tree(list(np.log((2 + np.arange(d)) / np.log(2))), t)
    maxdeg = np.zeros(d, np.int64)
    np.maximum.at(maxdeg, tr["dim"][1:], tr["deg"][1:])
    return tr, maxdeg


@pytest.mark.parametrize("d,t", [(1, 1.1), (1, 5.0), (3, 4.5), (6, 5.0), (12, 6.0), (40, 5.5), (60, 5.8), (200, 6.5)])
def test_walk_matches_direct_derivative(d, t):
    tr, maxdeg = _tree(d, t)
    n = tr["parent"].size
    lay = capi.host_layout("walk", tr, None, 1, maxdeg, np.zeros(d, np.int32), np.ones(d), np.zeros(d),
                           i32=WALK_TABLES, scalars=WALK_SCALARS)
    nn, nc, E, most = (int(lay[s]) for s in WALK_SCALARS)
    rng = np.random.default_rng(d)
    active = np.nonzero(maxdeg)[0]
    first = dict(zip(active, np.cumsum(maxdeg[active]) - maxdeg[active]))  # slots by dimension, then degree
    ns = int(maxdeg.sum())
    phi = rng.normal(size=ns)
    G = rng.normal(size=n)
    value, factors = np.ones(n), [[] for _ in range(n)]
    for e in range(1, n):
        s = first[tr["dim"][e]] + tr["deg"][e] - 1
        factors[e] = factors[tr["parent"][e]] + [s]
        value[e] = value[tr["parent"][e]] * phi[s]
    ref = np.zeros(ns)
    for e in range(1, n):
        for i, s in enumerate(factors[e]):
            ref[s] += G[e] * np.prod([phi[q] for j, q in enumerate(factors[e]) if j != i])

    def product(packed):
        s = np.ascontiguousarray(packed).view(np.uint16)
        return np.prod(phi[s[s != 0xFFFF]])

    perm = lay["w_perm"]
    assert perm.size == nc * E and sorted(perm[perm >= 0]) == list(range(1, n))
    rows = np.zeros(2 * (ns + nn) + 1)
    assert rows.size * 128 + 3 * (E * 128 + most * 8) + 256 <= 226 * 1024
    rows[:ns] = phi
    for i, v in enumerate(lay["w_node_path"].reshape(-1, 4)[:nn]):
        rows[ns + i] = product(v)
    off, term = lay["w_off"].reshape(nc, 33), lay["w_term"].reshape(-1, 2)
    assert np.all(off % 2 == 0) and (off[:, 32] - off[:, 0]).max() == most and not np.any(term[:, 1] % 128)
    owner = {}
    for c in range(nc):
        for w in range(32):
            for i in range(off[c, w], off[c, w + 1], 2):
                a, b = ((v & 0xFFFF, v >> 16, at // 128) for v, at in term[i : i + 2].tolist())
                assert a[1] != b[1]  # a pair is added without order
                for src, dst, at in (a, b):
                    if dst == rows.size - 1:
                        continue  # padding
                    assert ns + nn <= dst and owner.setdefault(dst, w) == w  # one warp owns a row
                    rows[dst] += rows[src] * G[perm[c * E + at]]
    bar, seen = np.zeros(ns), []
    slots, warp = lay["w_slot"].reshape(-1, 4), lay["w_warp"]
    assert warp[32] == slots.shape[0] == ns
    for w in range(32):
        for s, begin, end, _ in slots[warp[w] : warp[w + 1]]:
            seen.append(s)
            bar[s] = rows[ns + nn + s]
            for q in range(begin, end):
                bar[s] += rows[lay["w_row"][q]] * product(lay["w_other"].reshape(-1, 4)[q])
    assert sorted(seen) == list(range(ns))
    np.testing.assert_allclose(bar, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


def test_walk_is_refused_where_rows_do_not_fit():
    tr, maxdeg = _tree(1000, 8.3)
    d = maxdeg.size
    assert capi.host_layout("walk", tr, None, 1, maxdeg, np.zeros(d, np.int32), np.ones(d), np.zeros(d),
                            i32=WALK_TABLES, scalars=WALK_SCALARS) is None
