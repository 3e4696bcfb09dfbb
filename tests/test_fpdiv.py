"""The integer FP64 division (csrc/fpdiv.cuh) built for the host against the `/` operator: the
correctly rounded quotient is one value, so every bit must agree, whatever reciprocal the
device's approximate instruction returns within its error (one float ulp; two are tried)."""
import subprocess
from pathlib import Path

import pytest

TESTS = Path(__file__).resolve().parent


@pytest.mark.parametrize("ulps", [-2, 0, 2])
def test_quotients_are_correctly_rounded(tmp_path, ulps):
    exe = tmp_path / "fpdiv"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DFPDIV_SEED_ULPS={ulps}", "-o", str(exe),
                    str(TESTS / "fpdiv_harness.cpp")], check=True)
    r = subprocess.run([str(exe), "20000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
