"""Host check of the reassembly of double-floats into doubles (out_double of
ag_emu64.cuh; tests/emu_host/df_out_check.cpp): the FP64 sum of the two floats
bit for bit at every exponent of the head, powers of two with an opposing rest,
zeros and NaN among them; heads in [2^-90, 2^126) are never left to the native
lane. No tolerance: both round hi + lo once."""

import json
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_equals_the_fp64_sum(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path / "df_out_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "emu_host", "df_out_check.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    report = json.loads(subprocess.check_output([exe]))
    assert len(report) == 254
    assert {k: v for k, v in report.items() if v["differ"]} == {}
    assert {k: v for k, v in report.items() if v["native"] and (k == "special" or -90 <= int(k) < 126)} == {}
