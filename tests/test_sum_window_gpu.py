"""The integer window of a sum plan's threads: terms above, inside and below
it, windows that move, signs that cancel, subnormals, zeros and non-finite
terms, against math.fsum.

Tolerance, derived: one rounding of hi + comp (1 ulp), and for the terms and
partial sums that the compensated pair carries, n additions to comp rounded at
2^-53 of at most n 2^-53 sum|x|."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag


def _terms(kind, n, rng):
    m = rng.uniform(1, 2, n) * np.where(rng.random(n) < 0.5, -1.0, 1.0)
    if kind == "wide":
        return m * 2.0 ** rng.integers(-300, 300, n)
    if kind == "edges":   # exponents around the window's two ends
        return m * 2.0 ** rng.choice([0, -1, 3, 4, 5, -53, -54, -55, -58, -59, -60, 58, 59], n)
    if kind == "rising":
        return m * 2.0 ** (np.arange(n) * 900 // n - 450)
    if kind == "falling":
        return m * 2.0 ** (450 - np.arange(n) * 900 // n)
    if kind == "cancel":
        x = m[: n // 2] * 2.0 ** rng.integers(-20, 40, n // 2)
        t = np.concatenate([x, -x, np.full(n - 2 * (n // 2), 2.0 ** -40)])
        rng.shuffle(t)
        return t
    if kind == "small":
        return np.where(rng.random(n) < 0.5, 0.0, rng.integers(-1000, 1000, n) * 5e-324)
    if kind == "sparse":
        return np.where(rng.random(n) < 0.999, 0.0, m * 1e5)
    return m


@pytest.mark.parametrize("kind", ["wide", "edges", "rising", "falling", "cancel", "small", "sparse", "plain"])
@pytest.mark.parametrize("n", [1, 33, 700, 100001, 3000000])
def test_against_fsum(kind, n):
    x = _terms(kind, n, np.random.default_rng(n))
    a = ag.Array("f64", (1,), n)
    a.upload(x[None, :])
    exact = math.fsum(x.tolist())
    got = [ag.global_sum(a.view().sum(), n).cpu().numpy() for _ in range(2)]
    assert np.array_equal(got[0], got[1])
    tol = float(np.spacing(abs(exact))) + n * n * 2.0 ** -106 * float(np.abs(x).sum())
    assert abs((float(got[0][0]) + float(got[0][1])) - exact) <= tol


@pytest.mark.parametrize("special", [np.inf, -np.inf, np.nan])
def test_non_finite_terms(special):
    n = 50000
    x = np.random.default_rng(2).uniform(-1, 1, n)
    x[n // 3] = special
    a = ag.Array("f64", (1,), n)
    a.upload(x[None, :])
    got = ag.global_sum(a.view().sum(), n).cpu().numpy()
    assert np.isnan(got[0]) if np.isnan(special) else got[0] == special
    assert got[1] == 0.0 or np.isnan(got[1])
