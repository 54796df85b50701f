"""The native functions over every exponent of a double and on special values
(tests/emu_host/n64_wide.cpp): sqrt, rsqrt and div equal the correctly rounded
host operations, signed zeros, overflow and subnormals included; exp, log, log1p
and, to 2^22, sin and cos stay within the stated 0.52 ulp (a subnormal result, rounded twice at
most, within 1); and arguments outside the triple-float range no longer go to
the FP64 functions, one in a hundred apart."""

import json
import math
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("n64w") / "n64_wide")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "emu_host", "n64_wide.cpp"), "-lquadmath"], capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in r.stderr:
        pytest.skip("no libquadmath")
    assert r.returncode == 0, r.stderr
    return json.loads(subprocess.check_output([exe]).decode().replace("inf", "Infinity"))


def test_results(report):
    assert len(report) == 23
    for name, r in report.items():
        assert r["differ"] == 0, (name, r)
        bound = 1.0 if "subnormal" in name or "special" in name else 0.52
        assert math.isfinite(r["max_ulp"]) and r["max_ulp"] <= bound, (name, r)


def test_few_reach_the_fp64_functions(report):
    for name in ("sqrt", "rsqrt", "exp", "exp_tiny", "log", "log1p", "log1p_tiny", "sin", "cos"):
        assert report[name]["slow"] <= 0.01 * report[name]["n"], (name, report[name])
    # every other pair of draws has a quotient outside the doubles or near their ends
    assert report["div"]["slow"] <= 0.3 * report["div"]["n"], report["div"]
