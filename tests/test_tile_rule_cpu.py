"""The slices of dL/dC's contraction are chosen for the tile width that the product takes
(``csrc/tile_rule.h``): by both rules no count of slices is more than 2 % better."""
import os
import subprocess

from smolyax_gb300 import build


def test_slices_fit_the_width(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "rule")
    subprocess.run([build._nvcc(), "-std=c++17", "-I", build.CSRC, "-o", exe, os.path.join(here, "cuda", "tile_rule.cu")],
                   check=True, capture_output=True)
    sizes = [(M, N) for M in (64, 700, 5056, 20032, 64000) for N in (1, 63, 64, 65, 128, 129, 160, 192, 193, 300, 2048)]
    out = subprocess.run([exe, *[str(v) for s in sizes for v in s]], check=True, capture_output=True, text=True).stdout
    for (M, N), line in zip(sizes, out.splitlines()):
        width, slices, *cost = line.split()
        cost = [float(c) for c in cost]
        assert cost[int(slices) - 1] <= min(cost) / 0.98, (M, N)
        # the width is the one with the least rounds x weight, from the definition
        rounds = {bn: -(-(-(-M // 128) * -(-N // bn)) // 152) * w for bn, w in ((64, 94), (128, 100), (256, 177))}
        assert rounds[int(width)] == min(rounds.values()), (M, N)
    for name, use in (("gemm_tc.cu", "choose_tile("), ("tensor_vjp.cu", "choose_slices(")):
        with open(os.path.join(build.CSRC, name)) as fh:
            assert use in fh.read()
