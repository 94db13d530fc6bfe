"""Points per pass of the tensor-core evaluation (``smx_tensor_chunk``): whole tiles of
128 points, the panel within the memory limit, and no more row tiles than a grid's
second dimension has (65535), however few bytes a point takes."""
import ctypes

import pytest

from smolyax_gb300 import _capi as capi


def _chunk(K, limit, n_slots=1, d_out=16):
    t = capi.SmxTensor()
    t.d_in, t.d_out, t.K, t.n_slots, t.splits = 10, d_out, K, n_slots, 1
    t.n_groups = (K + 63) // 64
    t.ldb = max(64, 64 * t.n_groups)
    return capi.size("smx_tensor_chunk", ctypes.byref(t), limit), t


@pytest.mark.parametrize("limit", [1e-6, 0.5, 4.0, 64.0, 1000.0])
@pytest.mark.parametrize("K", [0, 1, 64, 65, 127, 128, 1000, 20010, 100000])
def test_chunk_is_a_launchable_pass(K, limit):
    n, t = _chunk(K, limit)
    assert n >= 128 and n % 128 == 0 and n // 128 <= 65535
    assert n == 128 or n * 4 * t.ldb <= limit * 1024**3


@pytest.mark.parametrize("K,n_slots", [(64, 64), (400, 400), (1400, 1400), (5000, 600), (20010, 500)])
@pytest.mark.parametrize("d_out", [16, 300])
def test_all_scratch_stays_near_the_limit(K, n_slots, d_out):
    """Basis rows, scales and partial sums count too: plans with a slot per entry have
    rows as large as half their panel."""
    limit = 0.25
    t = _chunk(K, limit, n_slots, d_out)[1]
    t.splits = capi.size("smx_tensor_splits", d_out, K)
    t.chunk = capi.size("smx_tensor_chunk", ctypes.byref(t), limit)
    used = capi.size("smx_tensor_workspace", ctypes.byref(t), 1 << 30)
    assert t.chunk >= 128 and used <= 1.13 * limit * 1024**3
