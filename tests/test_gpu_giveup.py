"""Bounded waits that give up are reported (needs a B200 and nvcc).

The axis passes of a caller's field have no error word to set: when a load
never completes the kernel leaves, and the lines it gave up must not look like
a result.  tests/giveup.cu runs the ring-fed kernels on one 256 x 256 plane
with the copies of one tile left out and a short spin limit.
"""

import os
import subprocess

import pytest

from ifdm_code_b200.build import ARCH, CSRC, INC

pytestmark = pytest.mark.gpu


def test_given_up_lines_are_nan_or_set_the_error_word(tmp_path):
    exe = os.path.join(tmp_path, "giveup")
    src = os.path.join(os.path.dirname(__file__), "giveup.cu")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, *ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-DIFDM_MAX_SPINS=8192u", "-I" + CSRC,
                    "-I" + INC, src, "-o", exe], check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    lines = out.stdout.split("\n")
    assert lines[-2] == "done" and len(lines) == 14, out.stdout
    for line in lines[:12]:
        name, word, err, differ, nan, lost = line.split()
        # every element outside the given-up tiles is that of the full transform
        assert int(differ) == int(lost), line
        assert (int(err), int(nan)) == ((2, 0) if word == "1" else (0, int(lost))), line
