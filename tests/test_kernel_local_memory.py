"""The loop kernels and the FP64 parallel operator keep everything in registers
and shared memory: a stack frame costs them traffic in the loop, and the first
pass after a program's other kernels tens of milliseconds.  Read from what ptxas
reports for each kernel."""
import os
import re
import subprocess

import pytest

from imgrecsrc_b200 import build


@pytest.mark.parametrize("source, kernel", [("tv.cu", "k_tv_loop"), ("wavelet.cu", "k_admm_loop"), ("parprj.cu", "k_par_")])
def test_no_stack_frame(source, kernel, tmp_path):
    r = subprocess.run([build.nvcc()] + build.ARCH + build.FLAGS + ["-Xptxas", "-v", "-c", os.path.join(build.CSRC, source), "-o",
                        str(tmp_path / "a.o")], capture_output=True, text=True, check=True)
    frames = re.findall(r"Function properties for (\S*%s\S*)\n\s*(\d+) bytes stack frame" % kernel, r.stdout + r.stderr)
    assert frames and all(int(size) == 0 for _, size in frames), frames
