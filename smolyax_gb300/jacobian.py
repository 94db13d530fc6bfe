"""Tables of the FP64 Jacobian of the orthogonal form (``csrc/jacobian64.cu``).

The derivative in dimension j sums, over the entries e with e_j > 0, the
product of e's other factors times the entry's coefficients; "e without j" is
an entry again, so the products are shared (``interpolation.py:306-345`` is
the reference's Jacobian, the same derivative of the combination sum).
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _capi as capi
from ._capi import call, ptr

UNIT = 128  # terms per unit, at most (csrc/jacobian64.cu)
MAX_DEGREE = 24  # degrees below this use the on-device basis change
MAX_POINTS = 1 << 19  # points per call


def jacobian_terms(parent, dim, deg, level, maxdeg):
    """Slots, rows, terms and units of an index-set tree (host arrays; entry 0 is
    the root, children follow their parents): the tables of
    ``struct smx_jacobian64`` that depend on the index set alone."""
    parent, dim, deg, level = (np.asarray(a, dtype=np.int64) for a in (parent, dim, deg, level))
    maxdeg = np.asarray(maxdeg, dtype=np.int64)
    dims = np.nonzero(maxdeg > 0)[0]
    soff = np.concatenate([[0], np.cumsum(maxdeg[dims])[:-1]]).astype(np.int64)
    dim_index = np.full(maxdeg.size, -1, dtype=np.int64)
    dim_index[dims] = np.arange(dims.size)
    n_slots = int(maxdeg.sum())
    n = parent.size
    slot = np.zeros(n, dtype=np.int64)
    slot[1:] = soff[dim_index[dim[1:]]] + deg[1:] - 1
    # child lookup: (parent, slot) -> entry
    key = parent[1:] * n_slots + slot[1:]
    order = np.argsort(key)
    key_sorted = key[order]

    def child(p, s):
        return order[np.searchsorted(key_sorted, p * n_slots + s)] + 1

    # per level: the slots of every entry's path and the entry without each of them
    place = np.zeros(n, dtype=np.int64)
    paths, rests = [np.zeros((1, 0), np.int64)], [np.zeros((1, 0), np.int64)]
    t_slot, t_row, t_ent = [], [], []
    path_of = {0: (np.zeros(1, np.int64), paths[0])}
    for lv in range(1, int(level.max(initial=0)) + 1):
        e = np.nonzero(level == lv)[0]
        place[e] = np.arange(e.size)
        up, s = parent[e], slot[e]
        path = np.concatenate([paths[-1][place[up]], s[:, None]], axis=1)
        rest = np.concatenate([child(rests[-1][place[up]], s[:, None]) if lv > 1 else np.zeros((e.size, 0), np.int64),
                               up[:, None]], axis=1)
        paths.append(path)
        rests.append(rest)
        path_of[lv] = (e, path)
        t_slot.append(path.ravel())
        t_row.append(rest.ravel())
        t_ent.append(np.repeat(e, lv))
    t_slot, t_row, t_ent = (np.concatenate(a) if a else np.zeros(0, np.int64) for a in (t_slot, t_row, t_ent))
    by = np.lexsort((t_ent, t_slot))
    t_slot, t_row, t_ent = t_slot[by], t_row[by], t_ent[by]
    rows, t_row = np.unique(t_row, return_inverse=True)
    row_len = level[rows]
    row_off = np.concatenate([[0], np.cumsum(row_len)])
    row_slot = np.zeros(max(int(row_off[-1]), 1), dtype=np.int64)
    for lv, (e, path) in path_of.items():
        at = np.nonzero(row_len == lv)[0]
        if lv and at.size:
            row_slot[row_off[at][:, None] + np.arange(lv)[None, :]] = path[place[rows[at]]]
    # units: runs of one slot, at most UNIT terms
    start = np.searchsorted(t_slot, np.arange(n_slots))
    end = np.searchsorted(t_slot, np.arange(n_slots), side="right")
    per = -(-(end - start) // UNIT)
    u_slot = np.repeat(np.arange(n_slots), per)
    u_t0 = start[u_slot] + UNIT * (np.arange(u_slot.size) - np.repeat(np.cumsum(per) - per, per))
    u_t1 = np.minimum(u_t0 + UNIT, end[u_slot])
    u_h = np.repeat(np.arange(dims.size), maxdeg[dims])[u_slot]
    unit_off = np.searchsorted(u_h, np.arange(dims.size + 1))
    return dict(dim=dims, deg=maxdeg[dims], soff=soff, dim_index=dim_index, n_slots=n_slots, row_off=row_off,
                row_slot=row_slot, n_rows=int(rows.size), unit=np.stack([u_t0, u_t1, u_slot, u_h], axis=1),
                unit_off=unit_off, term=np.stack([t_row, t_ent], axis=1), rows=rows)


class JacobianPlan:
    """Device tables of one interpolant's index set, and the evaluation."""

    def __init__(self, ip):
        tree, pl = ip._tree, ip._plan
        dev = tree.rem.device
        host = jacobian_terms(tree.parent.cpu().numpy(), tree.dim.cpu().numpy(), tree.deg.cpu().numpy(),
                              tree.level_of().cpu().numpy(), ip._maxdeg)
        # nodes of the summands' pairs by dimension: the barycentric derivative is NaN at each
        pdim, pdeg, pvoff, node = (pl.keep[key].cpu().numpy() for key in ("pair_dim", "pair_deg", "pair_voff", "node"))
        n_used = int(pl.keep["sum_poff"][-1].item())
        used = np.unique(pl.keep["sum_pairs"][:n_used].cpu().numpy())
        nodes = [[] for _ in range(ip.d_in)]
        for u in used:
            nodes[pdim[u]].append(node[pvoff[u] : pvoff[u] + pdeg[u] + 1])
        nodes = [np.unique(np.concatenate(nodes[j])) if nodes[j] else np.zeros(0) for j in host["dim"]]
        node_off = np.concatenate([[0], np.cumsum([a.size for a in nodes])])
        max_deg = int(host["deg"].max())
        m = np.arange(max_deg)
        rec = np.stack([np.stack([(2 * m + 1) / (m + 1), m / (m + 1)], axis=1),
                        np.stack([np.sqrt(2.0 / (m + 1)), np.sqrt(m / (m + 1))], axis=1)])
        self.keep = {key: torch.as_tensor(np.ascontiguousarray(host[key]), dtype=torch.int32, device=dev)
                     for key in ("dim", "deg", "soff", "dim_index", "row_off", "row_slot", "unit", "unit_off", "term")}
        self.keep["node_off"] = torch.as_tensor(node_off, dtype=torch.int32, device=dev)
        self.keep["node"] = torch.as_tensor(np.concatenate(nodes + [np.zeros(1)]), device=dev)
        self.keep["rec"] = torch.as_tensor(np.ascontiguousarray(rec), device=dev)
        s = self.c = capi.SmxJacobian64()
        s.d_in, s.d_out = ip.d_in, ip.d_out
        s.n_dims, s.n_slots, s.n_rows = int(host["dim"].size), host["n_slots"], host["n_rows"]
        s.n_units, s.max_deg = int(host["unit"].shape[0]), max_deg
        for key, t in self.keep.items():
            setattr(s, key, t.data_ptr())

    def evaluate(self, co, x, J, st, budget):
        """J [P, d_out, d_in] at x [P, d_in] (contiguous FP64), in chunks of points
        whose workspace is at most `budget` bytes; co: the interpolant's Coefficients."""
        s = capi.SmxJacobian64.from_buffer_copy(self.c)  # a copy per call: several threads may share the plan
        s.C, s.fam_a, s.fam_b, s.fam = (t.data_ptr() for t in (co.C64, co.fa64, co.fb64, co.fam))
        ref = ctypes.byref(s)
        P, d = x.shape
        step = max(1, min(MAX_POINTS, int(budget * 4 // max(1, capi.size("smx_jacobian64_workspace", ref, 4)))))
        nws = capi.size("smx_jacobian64_workspace", ref, min(step, P))
        ws = torch.empty(nws, dtype=torch.uint8, device=x.device)
        for p0 in range(0, P, step):
            p1 = min(P, p0 + step)
            call("smx_jacobian64_eval", ref, ptr(x[p0:p1]), p1 - p0, d, ptr(J[p0:p1]), ptr(ws), nws, st)
        return J
