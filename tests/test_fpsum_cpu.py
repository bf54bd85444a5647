"""fpsum.cuh: sums of FP32 values on the FP32 pipe equal the FP64 sums rounded to
FP32, bit for bit (random magnitudes, cancellation, ties, overflow on the way,
infinities, NaNs, zeros, subnormals; one value to more than the pair takes), and
sums of 152 FP32 pairs as triples are no further from the sum in 113 bits than
FP64 sums of the same pairs, and within 2^-53 of the magnitudes added."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_sums_round_as_fp64(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "fpsum_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "fpsum_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, "4000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
