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


def test_pipelines_give_nothing_up_before_all_roles_have_stopped():
    """The product kernels look at the abort flag for their last copies and MMAs behind a
    block barrier that follows all roles, not in the middle of one."""
    for name, free in (("gemm_tc.cu", '"tcgen05.dealloc'), ("tensor_vjp.cu", '"tcgen05.dealloc')):
        with open(os.path.join(build.CSRC, name)) as fh:
            code = fh.read()
        end = code.index(free)
        tail = code[code.rindex("tcgen05.fence::before_thread_sync", 0, end) : end]
        barrier, look = tail.index("__syncthreads();"), tail.index("if (*abort_flag)")
        assert barrier < look < tail.index("for_pending_copies") < tail.rindex("__syncthreads();")
        assert look < tail.index("mma_commit(flush)") < tail.rindex("__syncthreads();")
        assert code[:end].count("for_pending_copies") == tail.count("for_pending_copies")
