"""The combination sum (``csrc/eval64.cu``) serves any device of a process: it keeps no
flag or attribute of the process for what belongs to a device."""
import os
import re

from smolyax_gb300 import build


def test_combination_sum_keeps_no_process_state():
    with open(os.path.join(build.CSRC, "eval64.cu")) as fh:
        code = re.sub(r"//[^\n]*", "", fh.read())
    assert not re.search(r"\bstatic\s+(?!__|inline|constexpr)\w+", code)
    for call in re.finditer(r"cudaFuncSetAttribute", code):
        assert "static" not in code[max(0, call.start() - 200) : call.start()]
