"""The error bounds that ag_tf64.cuh states for the native functions, against
113-bit arithmetic (tests/emu_host/n64_ulp.cpp): 0.52 ulp; 0.76 for sine and
cosine beside multiples of pi/2, where the reduced argument is known to 2^-77
and no smaller than 2^-22, a quarter ulp of the result; and the normal draw's
8 x 2^-53 of the reference's steps, abs + rel. A NaN where the result is finite counts as
an infinite error, whatever follows it. The wide ranges include arguments that
take the function out of line, rounded from exact here."""

import json
import math
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_within_the_stated_bounds(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path / "n64_ulp")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "emu_host", "n64_ulp.cpp"), "-lquadmath"], capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in r.stderr:
        pytest.skip("no libquadmath")
    assert r.returncode == 0, r.stderr
    report = json.loads(subprocess.check_output([exe]).decode().replace("inf", "Infinity"))
    assert len(report) == 21
    for name, worst in report.items():
        bound = 8.0 if name == "normal" else 0.76 if name.endswith("multiples") else 0.52
        assert math.isfinite(worst) and worst <= bound, (name, worst)
