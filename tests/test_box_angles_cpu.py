"""Sines and cosines of the box kernels' kick angles against 80-bit libm, over
magnitudes from 1e-12 to 1e9 (the device functions compiled for the host).

sincos_pi keeps the argument to well below its last bit (the product with 1/pi
carries its rounding error along), so its error is that of sincospi and of two
roundings: 4e-16 = 3.6 roundings of one.  The full series (to z^15 and z^16, 5e-17
left at pi/4) keeps its argument the same way and rounds it twice and its sum
once: 4e-16 too.  The short one stops at z^11 and z^12 ((pi/4)^13/13! = 6.9e-12
left) with an argument that one product rounds: 2^-53 of it, and of the
multiplication by pi, 7e-12 + 2.5e-16 |p|.
"""

import os
import subprocess

from ifdm_code_b200.build import ARCH, CSRC, _cuda_home


def test_angles_against_long_double(tmp_path):
    exe = os.path.join(tmp_path, "angles")
    src = os.path.join(os.path.dirname(__file__), "angles.cu")
    subprocess.run([os.path.join(_cuda_home(), "bin", "nvcc"), *ARCH, "-O2", "-std=c++17", "-I" + CSRC, src, "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout.split("\n")[:-1]
    assert len(out) == 22
    for line in out:
        dec, e_pi, e_full, e_short = line.split()
        assert float(e_pi) <= 4e-16 and float(e_full) <= 4e-16, line
        assert float(e_short) <= 7e-12 + 2.5e-16 * 10.0 ** int(dec), line
