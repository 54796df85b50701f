"""How near the triple-float sqrt, reciprocal and quotient of the native double
functions are to the exact values (tests/emu_host/n64_margin.cpp): ag::n64 rounds
them itself unless they lie within 2^-12 of an ulp of a rounding boundary, so
half of that is the bound here."""
import json
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_half_the_margin_is_not_reached(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path / "n64_margin")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "emu_host", "n64_margin.cpp"), "-lquadmath"], capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in r.stderr:
        pytest.skip("no libquadmath")
    assert r.returncode == 0, r.stderr
    far = json.loads(subprocess.check_output([exe]))
    assert set(far) == {"sqrt", "recip", "div"}
    assert max(far.values()) <= 2.0 ** -13, far
