"""Host check of the double functions native plans call (ag::n64 of
ag_tf64.cuh and ag_tf64_trig.cuh; tests/emu_host/n64_check.cpp) against
113-bit arithmetic: sqrt, rsqrt and div equal the correctly rounded host
operations everywhere, the others stay under CUDA's documented 1 ulp.

Bounds, derived: the triple-float kernels are held to 0.25 x 2^-53 of the
result (0.5 near multiples of pi/2, tests/test_tf64_host.py), at most a quarter
(half) of an ulp beside the half ulp of the final rounding."""

import json
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

EXACT = ["sqrt", "sqrt_edge", "sqrt_square", "rsqrt", "rsqrt_edge", "div", "div_edge", "div_pairs",
         "reassemble", "pairs"]
BOUNDS = {"exp": 0.75, "exp_small": 0.75, "log": 0.75, "log_near_1": 0.75, "log1p": 0.75, "log1p_neg": 0.75,
          "log1p_neg_small": 0.75, "sin": 0.75, "sin_unit": 0.75, "sin_small": 0.75, "sin_multiples": 1.0, "cos": 0.75,
          "cos_unit": 0.75, "cos_small": 0.75, "cos_multiples": 1.0}


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("n64") / "n64_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "emu_host", "n64_check.cpp"), "-lquadmath"], capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in r.stderr:
        pytest.skip("no libquadmath")
    assert r.returncode == 0, r.stderr
    return json.loads(subprocess.check_output([exe]))


@pytest.mark.parametrize("name", EXACT)
def test_correctly_rounded(report, name):
    assert report[name]["differ"] == 0, report[name]


@pytest.mark.parametrize("name", sorted(BOUNDS))
def test_ulps(report, name):
    assert report[name]["max_ulp"] <= BOUNDS[name], report[name]


def test_fast_path_serves_ordinary_arguments(report):
    for name in ("sqrt_square", "log_near_1", "sin_unit", "cos_unit", "normal"):
        assert report[name]["slow"] <= 0.02 * report[name]["n"], (name, report[name])


def test_normal_follows_the_reference_steps(report):
    # each of log, sqrt and sin rounded within 0.75 ulp where the reference's
    # value is rounded within 0.5, and the product: 8 x 2^-53 abs + rel is the
    # native draw's own bound
    assert report["normal"]["max_ulp"] <= 8.0, report["normal"]
