"""The clean-up of the kernels that copy through a ring of buffers
(``csrc/tc_util.cuh`` for_pending_copies: gradient walk, adjoint product, GEMM), by a
host model of the barriers' phases."""
import os
import subprocess

from smolyax_gb300 import build


def test_every_copy_in_flight_is_waited_for(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "pending")
    subprocess.run([build._nvcc(), "-std=c++17", "-I", build.CSRC, "-o", exe,
                    os.path.join(here, "cuda", "pending_copies.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
