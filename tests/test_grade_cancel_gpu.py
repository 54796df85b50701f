"""FP64-grade outputs that cancel: a - b of nearby doubles equals the device's
own difference bit for bit (its triple-float is exact), as an assignment, a
+= and -=, a sum and a batch item, from the kernel that holds two samples and
from the one that holds one (unaligned planes); a b - c d stays within
the lowering's stated bound of the exact value."""

import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag
from aether_gb300 import accuracy

N = 26 * 1500 + 7


def _near(seed):
    """Doubles and neighbours 2^-2 to 2^-52 away, equal ones among them."""
    r = np.random.default_rng(seed)
    a = r.choice([-1.0, 1.0], N) * 2.0 ** r.uniform(-8, 40, N)
    k = 2.0 + 2.0 * (np.arange(N) % 26)
    b = a * (1.0 + r.choice([-1.0, 1.0], N) * r.uniform(0.5, 2.0, N) * 2.0 ** -k)
    b[::101] = a[::101]
    return a, b


def _plane(x, shift):
    """x in a plane that starts `shift` doubles off a 16-byte boundary."""
    t = torch.zeros((1, N + 2), dtype=torch.float64, device="cuda")[:, shift:shift + N]
    t.copy_(torch.from_numpy(x))
    return t


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("op", ["set", "add", "sub", "setsum", "sum", "batch"])
def test_difference_is_exact(op, shift):
    if op == "batch" and shift:
        pytest.skip("batch items are aligned")
    x, y = _near(3)
    a, b = _plane(x, shift), _plane(y, shift)
    d = _plane(np.random.default_rng(4).uniform(-1, 1, N), shift)
    want = {"add": d + (a - b), "sub": d - (a - b)}.get(op, a - b)
    wrap = lambda t: ag.Array.wrap(t, n=N)
    e = wrap(a).view() - wrap(b).view()
    if op in ("sum", "setsum"):
        red = torch.zeros(2, dtype=torch.float64, device="cuda")
        if op == "sum":
            red = ag.global_sum(e.sum(), N, math=3)
        else:
            ag.assign(wrap(d), e, op="setsum", reduce_out=red, math=3)
            assert torch.equal(d, want)
        hi, lo = red.cpu().tolist()
        exact = math.fsum((x - y).tolist())
        assert abs(hi + lo - exact) <= np.spacing(abs(exact)) + N * N * 2.0 ** -106 * float(np.abs(x - y).sum())
        return
    if op == "batch":
        f = _plane(x, 0)
        ag.Batch([ag.prepare(wrap(d), e, math=3), ag.prepare(wrap(f), e, math=3)]).launch()
        assert torch.equal(f, want)
    else:
        ag.assign(wrap(d), e, op=op, math=3)
    assert torch.equal(d, want)


@pytest.mark.parametrize("odd", [0, 1])
def test_three_components_and_products(odd):
    n = 2001
    cap = n + odd if odd else 2016
    r = np.random.default_rng(9)
    p, q, s = (r.choice([-1.0, 1.0], (3, n)) * 2.0 ** r.uniform(-4, 4, (3, n)) for _ in range(3))
    t = p * q / s * (1.0 + r.uniform(0.5, 2.0, (3, n)) * 2.0 ** -(2.0 + 2.0 * (np.arange(n) % 26)))
    buf = [torch.zeros((3, cap), dtype=torch.float64, device="cuda") for _ in range(5)]
    for b, v in zip(buf, (p, q, s, t)):
        b[:, :n] = torch.from_numpy(v)
    v = [ag.Array.wrap(b, n=n).view() for b in buf[:4]]
    ag.assign(ag.Array.wrap(buf[4], n=n), v[0] * v[1] - v[2] * v[3], math=3)
    got = buf[4][:, :n].cpu().numpy()
    for c in range(3):
        for i in range(n):
            x, y = Fraction(p[c, i]) * Fraction(q[c, i]), Fraction(s[c, i]) * Fraction(t[c, i])
            bound = accuracy.FP64_GRADE_EXACT_ULPS * np.spacing(float(max(abs(x), abs(y))))
            assert abs(Fraction(got[c, i]) - (x - y)) <= Fraction(bound), (c, i)
