"""Host check of the reassembly of triple-floats into doubles (out_double of
ag_tf64.cuh; tests/emu_host/tf_out_check.cpp) after sums that cancel by 2^2 to
2^52, after single operations, on ties, whole numbers, heads next to powers of
two and at the edges of the range.

Bounds, derived: the rest in units of the double's last place is rounded from a
float below 2^10 units, 2^-14 of one at most, so a result lies within
0.5 + 2^-13 ulp of the exact sum of the three floats and differs from the FP64
sum only where that sum is as close to a tie, one value in 2^12. Differences of
doubles, ties and whole numbers are exact in these units: none may differ."""

import json
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("tfo") / "tf_out_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "emu_host", "tf_out_check.cpp"), "-lquadmath"], capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in r.stderr:
        pytest.skip("no libquadmath")
    assert r.returncode == 0, r.stderr
    return json.loads(subprocess.check_output([exe]))


def test_rounded_once(report):
    for name, r in report.items():
        assert r["max_ulp"] <= 0.5 + 2.0 ** -13, (name, r)
        # log(1 + d) is d - d^2/2, beside a tie wherever d ends in half a unit of it
        assert name == "near_0" or r["differ"] <= r["n"] * 2.0 ** -12, (name, r)


def test_few_leave_for_the_native_lane(report):
    # renormalised, only what falls below 2^-75 does: differences of doubles above
    # 2^-30 that cancel by 2^44 and more, and log x - log x
    for name, r in report.items():
        kind, k = name.split("_")
        if kind in ("ties", "whole", "heads", "op", "near") or (kind in ("difference", "products", "logarithms") and int(k) <= 40):
            assert r["native"] <= 1e-3 * r["n"], (name, r)


def test_exact_values(report):
    for name, r in report.items():
        if name.split("_")[0] in ("difference", "ties", "whole"):
            assert r["differ"] == 0, (name, r)
