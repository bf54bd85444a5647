"""softfp.cuh's integer square roots and quotients equal the host's FP64
operations bit for bit: random operands of ordinary and extreme exponents, zeros,
subnormals, infinities, NaNs, squares and their neighbours, exact quotients, with
the Newton seeds perturbed by up to 2^-21 (softfp_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_soft_roots_and_quotients_round_as_fp64(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "softfp_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "softfp_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, "4000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
