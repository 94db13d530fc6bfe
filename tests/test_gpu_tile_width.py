"""The products' tile width (``csrc/gemm_tc.cu``: 64, 128 or 256 columns by rounds of
tiles on the SMs) does not change a value: columns of a wide product are, bit for
bit, those of the narrower products of the same columns, at widths around the tiles
and row counts that make the rule choose differently."""
import pytest
import torch

from smolyax_gb300 import _capi as capi
from smolyax_gb300._capi import call, ptr

pytestmark = pytest.mark.gpu


def _product(A, B, M, N, K, entry):
    D = torch.empty(M, N, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    call(entry, ptr(A[0]), ptr(A[1]), K, ptr(B[0]), ptr(B[1]), K, M, N, K, ptr(D), N, None, 0, ptr(err),
         capi.stream_ptr(torch.cuda.current_stream()))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return D


@pytest.mark.parametrize("entry", ["smx_gemm_bf16x3", "smx_gemm_tf32x3"])
@pytest.mark.parametrize("M,N", [(1, 1), (129, 63), (128, 65), (3001, 300), (19457, 129), (20001, 257), (700, 520)])
def test_columns_do_not_depend_on_the_width(entry, M, N):
    K = 320
    gen = torch.Generator("cuda").manual_seed(M + N)
    draw = lambda n, scale: torch.randn(n, K, device="cuda", generator=gen) * scale
    parts = []
    for n in (M, N):
        hi = draw(n, 1.0).bfloat16()  # exact in TF32 too
        lo = draw(n, 2.0**-9).bfloat16()
        parts.append((hi, lo) if entry.endswith("bf16x3") else (hi.float(), lo.float()))
    A, B = parts
    whole = _product(A, B, M, N, K, entry)
    for n0, n1 in ((0, min(N, 64)), (max(0, N - 64), N), (0, min(N, 130)), (N // 2, N // 2 + 1)):
        part = _product(A, tuple(b[n0:n1].contiguous() for b in B), M, n1 - n0, K, entry)
        assert torch.equal(part, whole[:, n0:n1])
    ref = sum(a.double() @ b.double().T for a, b in ((A[0], B[0]), (A[0], B[1]), (A[1], B[0])))
    assert float((whole.double() - ref).abs().max()) <= 2e-6 * float((A[0].double().abs() @ B[0].double().abs().T).max())
