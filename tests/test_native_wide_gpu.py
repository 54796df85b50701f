"""Native functions on the device over every exponent: sqrt, 1/sqrt and a/b bit
for bit as the device's correctly rounded operations give them; exp, log, log1p,
sin and cos against the host's, each within 0.52 ulp of exact (1 ulp the host's,
taken as 1.52 together, 3 units where a binade ends between them)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag

SPECIAL = [0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1022, 1.7976931348623157e308, 1.0, -1.0, 2.0 ** -40, 2.0 ** -41, 2.0 ** 60, 2.0 ** 61,
           np.inf, -np.inf, np.nan, 709.78, 709.79, -745.2, 1024.0, 2.0 ** 22]


def _arrays(x, odd):
    n = len(x)
    t = torch.zeros((2, n + odd if odd else (n + 31) // 32 * 32), dtype=torch.float64, device="cuda")
    t[:, :n] = torch.from_numpy(x).cuda()
    return ag.Array.wrap(t, n=n), ag.Array.wrap(torch.zeros_like(t), n=n)


def _wide(seed, n, lo=-1022, hi=1024):
    r = np.random.default_rng(seed)
    x = np.ldexp(r.uniform(1, 2, n), r.integers(lo, hi, n)) * r.choice([-1.0, 1.0], n)
    x[:len(SPECIAL)] = SPECIAL
    return x


def _same(a, b):
    return torch.equal(a.view(torch.int64)[~torch.isnan(a)], b.view(torch.int64)[~torch.isnan(b)]) and \
        torch.equal(torch.isnan(a), torch.isnan(b))


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("name", ["sqrt", "rsqrt", "div"])
def test_correctly_rounded(name, odd):
    n = 400002 + odd
    x = _wide(1, n)
    a, d = _arrays(x, odd)
    y = _wide(2, n)
    y[1::2] = x[1::2] * np.ldexp(np.random.default_rng(3).uniform(1, 2, n), np.random.default_rng(4).integers(-60, 60, n))[1::2]
    b, _ = _arrays(np.roll(y, 7) if odd else y, odd)
    e = {"sqrt": lambda: ag.cwiseSqrt(a.view()), "rsqrt": lambda: ag.cwiseRsqrt(a.view()),
         "div": lambda: ag.cwiseDiv(a.view(), b.view())}[name]()
    ag.assign(d, e)
    s, t = a.data[:, :n], b.data[:, :n]
    want = {"sqrt": lambda: torch.sqrt(s), "rsqrt": lambda: 1.0 / torch.sqrt(s), "div": lambda: s / t}[name]()
    assert _same(d.data[:, :n], want)


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("name,lo,hi", [("exp", -60, 10), ("log", -1022, 1024), ("log1p", -1022, 1024), ("sin", -60, 25),
                                        ("cos", -60, 25)])
def test_functions(name, lo, hi, odd):
    n = 200002 + odd
    x = _wide(5, n, lo, hi)
    a, d = _arrays(x, odd)
    fn = {"exp": ag.cwiseExp, "log": ag.cwiseLog, "log1p": ag.cwiseLog1p, "sin": ag.cwiseSin, "cos": ag.cwiseCos}[name]
    ag.assign(d, fn(a.view()))
    got = d.data[0, :n].cpu().numpy()
    assert np.array_equal(got, d.data[1, :n].cpu().numpy(), equal_nan=True)
    with np.errstate(all="ignore"):
        want = getattr(np, name)(x)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf])
    ok = np.isfinite(want)
    assert np.array_equal(np.signbit(got[ok]), np.signbit(want[ok]))
    assert np.all(np.abs(got[ok] - want[ok]) <= 3 * np.spacing(np.abs(want[ok])))
