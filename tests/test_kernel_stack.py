"""Kernels that index a pointer set from their parameters at run time must not copy it to the stack (every thread would
write and read it: the prolongation to level 6 took three times as long). Read off the compiler's resource report."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("source,kernels", [("transfer.cu", ["prolongate_kernel", "restrict_kernel"])])
def test_no_stack(tmp_path, source, kernels):
    csrc = os.path.join(ROOT, "terra-ng_b200", "csrc")
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler",
                        "-ffp-contract=off", "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"), "-I" + csrc,
                        "-Xptxas", "-v", "-c", os.path.join(csrc, source), "-o", str(tmp_path / "k.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    frames = re.findall(r"Function properties for (\S+)\s+(\d+) bytes stack frame", r.stderr)
    for k in kernels:
        mine = [int(b) for name, b in frames if k in name]
        assert mine and not any(mine), (k, frames)
