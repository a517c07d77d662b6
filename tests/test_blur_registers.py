"""The fused blur keeps its sums in registers: an array that a rolled loop indexes is a stack frame of its size. Compiles
csrc/fg_kernels.cu for its resource use (nvcc, no GPU)."""
import os
import re
import shutil
import subprocess

import build
import pytest

CSRC = os.path.join(build.HERE, "csrc")


@pytest.mark.skipif(not (os.path.exists(build.NVCC) or shutil.which("nvcc")), reason="no nvcc")
def test_fused_blur_sums_are_not_on_the_stack(tmp_path):
    nvcc = build.NVCC if os.path.exists(build.NVCC) else "nvcc"
    flags = [f for f in build.FLAGS if f != "-shared"]
    r = subprocess.run([nvcc] + flags + ["-cubin", "-Xptxas", "-v", "-o", str(tmp_path / "k.cubin"), os.path.join(CSRC, "fg_kernels.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    frames = re.findall(r"Function properties for \S*k_synth_blur_t\S*\n\s+(\d+) bytes stack frame", r.stderr)
    assert len(frames) == 2   # with and without the overlay's rejection
    assert all(int(f) < 8 * 3 * 4 for f in frames), frames   # 8 rows x 3 channels of sums
