"""Stream tables (``smx_layout_build`` kind SMX_LAYOUT_STREAM, ``csrc/layout.cu``),
no GPU needed: the tables are decoded and summed on the host in FP64, as the
kernel of ``csrc/stream_eval.cuh`` does, and compared with the direct sum over
the index set."""
import numpy as np
import pytest

from smolyax_gb300 import _capi as capi
from smolyax_gb300.spectral import STREAM_TABLES, _phi_table
from test_layout_cpu import direct, python_tree


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("d,t,d_out,fam_id", [(1, 5.0, 2, 0), (3, 4.5, 1, 0), (6, 5.0, 2, 1), (12, 6.0, 5, 0),
                                               (40, 5.5, 9, 0), (60, 5.8, 1, 1), (200, 6.5, 4, 0)])
def test_stream_matches_direct_sum(d, t, d_out, fam_id, fp64):
    k = list(np.log((2 + np.arange(d)) / np.log(2)))
    tr = python_tree(k, t)
    n = tr["parent"].size
    rng = np.random.default_rng(d + d_out)
    maxdeg = np.zeros(d, np.int64)
    np.maximum.at(maxdeg, tr["dim"][1:], tr["deg"][1:])
    C = rng.normal(size=(n, d_out)).astype(np.float64 if fp64 else np.float32)
    fam = np.full(d, fam_id, np.int32)
    fa, fb = np.where(np.arange(d) % 3 == 0, 1.0, 0.75), np.where(np.arange(d) % 3 == 0, 0.0, 0.125)
    lay = capi.host_layout("stream", tr, C, d_out, maxdeg, fam, fa, fb, fp64=fp64, **STREAM_TABLES)
    x = rng.uniform(-1, 1, (5, d))
    w, ps = (8 if fp64 else 4), int(lay["st_pass"])
    assert ps == (1 if d_out == 1 else 8 if d_out > 4 and not fp64 else 4)
    n_hb, n_rows, n_chunks = (int(lay["st_" + s]) for s in ("n_hb", "n_rows", "n_chunks"))
    hot = lay["st_hot"].reshape(-1, 8)
    rows = np.zeros((n_rows, 5))
    for h in hot:
        a, b = np.ascontiguousarray(h[4:]).view(np.float64)
        rows[h[2] : h[2] + h[1]] = _phi_table(int(h[3]), a * x[:, h[0]] + b, int(h[1]))[1:]
    for r, v in enumerate(lay["st_vp"].reshape(-1, 4)):
        s = np.ascontiguousarray(v).view(np.uint16)
        s = s[s != 0xFFFF]
        rows[n_hb + r] = np.prod(rows[s], axis=0) if s.size else 1.0
    chunk = np.frombuffer(lay["st_chunk"].tobytes(), np.uint8).reshape(-1, n_chunks, 64 + 16 * ps * w)
    assert chunk.shape[0] == -(-d_out // ps)
    warp, desc = lay["st_warp"], lay["st_desc"].reshape(-1, 8)
    assert warp[16] == desc.shape[0] and warp[33] == n_chunks and np.all(np.diff(warp[:17]) >= 0)
    y = np.tile(C[0].astype(float), (5, 1))
    for p in range(chunk.shape[0]):
        for q in range(16):
            item, s, run = int(warp[q]), None, 0
            for c in range(warp[17 + q], warp[18 + q]):
                slot = chunk[p, c, :64].view(np.int32)
                cf = chunk[p, c, 64:].view(np.float64 if fp64 else np.float32).reshape(16, ps).astype(float)
                for i in range(16):
                    if item == warp[q + 1]:
                        assert not np.any(cf[i:])  # padding
                        break
                    if s is None:
                        s = np.full((5, ps), 0.0 if desc[item][0] & 256 else desc[item][2:4].copy().view(np.float64)[0])
                    s += rows[slot[i] // int(lay["st_row_bytes"])][:, None] * cf[i][None, :]
                    run += 1
                    if slot[i] & 1:
                        assert run <= (64 if fp64 else 32) and (fp64 or run % 4 == 0)
                        de = desc[item]
                        if de[0] & 256:
                            a, b = np.ascontiguousarray(de[4:]).view(np.float64)
                            g = int(de[0]) >> 16
                            assert bool(de[0] & 2048) == (a == 1.0 and b == 0.0 and g == 1 and fam_id == 0)
                            v = _phi_table((int(de[0]) >> 9) & 1, a * x[:, de[1]] + b, g)[g]
                        else:
                            f = np.ascontiguousarray(de[4:]).view(np.uint16)[: de[0] & 255]
                            v = np.prod(rows[f], axis=0) if f.size else np.ones(5)
                        hi = min(d_out, (p + 1) * ps)
                        y[:, p * ps : hi] += (v[:, None] * s)[:, : hi - p * ps]
                        item, s, run = item + 1, None, 0
            assert item == warp[q + 1] and s is None
    ref = direct(tr, C.astype(float), x, fam, fa, fb)
    np.testing.assert_allclose(y, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())
