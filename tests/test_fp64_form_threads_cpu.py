"""The FP64 tables of a plan are built once, under the plan's lock: a thread that asks
while another builds them waits and gets the same tables (and not "no FP64 form")."""
import threading
import types

import numpy as np
import torch

from smolyax_gb300 import spectral


def test_a_second_thread_waits_for_the_tables(monkeypatch):
    building, go, built = threading.Event(), threading.Event(), []

    def host_layout(kind, *args, **kw):
        built.append(kind)
        building.set()
        assert go.wait(20)
        i32 = ("node_seg", "cold_seg", "hot_dim", "hot_deg", "hot_soff", "node", "cold", "run")
        lay = {name: np.zeros(5, np.int32) for name in i32}
        lay.update({name: np.zeros(4) for name in ("node_c", "cold_ab", "terms", "coef")})
        lay.update({name: 1 for name in ("d_out", "dstride", "row", "n_hb", "n_vp", "n_hot_dims", "n_nodes",
                                         "n_cold_groups", "max_depth", "n_terms")})
        return lay

    monkeypatch.setattr(spectral.capi, "host_layout", host_layout)
    monkeypatch.setattr(spectral, "stream_tables", lambda *args: torch.zeros(1))
    monkeypatch.setattr(spectral, "finish_build", lambda: True)
    sp = spectral.SpectralPlan.__new__(spectral.SpectralPlan)
    sp._lock, sp._f64, sp.c = threading.RLock(), None, types.SimpleNamespace(d_in=1)
    sp.C64 = torch.zeros(1, 1, dtype=torch.float64)
    sp.fa64 = sp.fb64 = torch.zeros(1, dtype=torch.float64)
    sp.fam = torch.zeros(1, dtype=torch.int32)
    T = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a), dtype=dt)
    sp._fwd_args = ({}, None, np.ones(1), np.zeros(1), np.ones(1), np.zeros(1), T, None)
    got = [None, None]

    def ask(i):
        got[i] = sp.fp64_form()

    first = threading.Thread(target=ask, args=(0,))
    first.start()
    assert building.wait(20)
    second = threading.Thread(target=ask, args=(1,))
    second.start()
    second.join(0.5)  # (long enough for an answer that does not wait)
    go.set()
    first.join(20), second.join(20)
    assert built == ["perpoint"]
    assert got[0] is not None and got[1] is got[0]
