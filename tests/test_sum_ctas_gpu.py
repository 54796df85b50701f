"""Sum plans whose CTAs keep one (hi, comp) pair per thread over many chunks:
sizes at the edges of a lane group, a chunk and a whole grid of chunks, against
math.fsum; and the two-operation residual of an accumulation plane against
Knuth's five-operation one, bit for bit, special values included.

Tolerance of the sums, derived: hi + comp is rounded once (1 ulp covers it);
each of the n additions to comp rounds at 2^-53 of a comp that is at most n
2^-53 of sum|x|, so the pair itself is off by at most n^2 2^-106 sum|x|."""

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

CHUNK = 512            # 256 threads x 2 f64 samples
FULL = 152 * 8         # CTAs of a full grid at most


@pytest.mark.parametrize("store,math_", [("f64", 0), ("f64", 1), ("f32", 2)])
@pytest.mark.parametrize("n", [1, 2, CHUNK - 1, CHUNK, CHUNK + 1, FULL * CHUNK - 1, FULL * CHUNK + 1,
                               5 * FULL * CHUNK + 777])
def test_sum_sizes(store, math_, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-3.0, 5.0, n).astype(np.float64 if store == "f64" else np.float32)
    a = ag.Array(store, (1,), n)
    a.upload(x[None, :])
    exact = math.fsum(x.astype(np.float64).tolist())
    tol = float(np.spacing(abs(exact))) + n * n * 2.0 ** -106 * float(np.abs(x).sum(dtype=np.float64))
    if math_ == 1:   # each term enters as a float pair, 2^-47 of itself
        tol += 2.0 ** -47 * float(np.abs(x).sum())
    if math_ == 2:   # at most 4 samples a chunk in float-float, each addition within 3 2^-48
        tol += 12 * 2.0 ** -48 * float(np.abs(x).sum(dtype=np.float64))
    got = [ag.global_sum(a.view().sum(), n, dtype=store, math=math_).cpu().numpy() for _ in range(2)]
    assert np.array_equal(got[0], got[1])
    assert abs((got[0][0] + got[0][1]) - exact) <= tol


def _knuth(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def test_residual_is_knuths():
    big = np.finfo(np.float64).max
    special = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-310, 2.0 ** -1022, 1.0, -1.0, np.nextafter(1.0, 2.0),
                        np.nextafter(1.0, 0.0), 1.5, 2.0 ** 53, 2.0 ** 53 + 2, -2.0 ** 54, 1e300, -1e300, big, -big,
                        np.inf, -np.inf, np.nan])
    rng = np.random.default_rng(4)
    r = rng.uniform(-1, 1, 4096) * 2.0 ** rng.integers(-60, 60, 4096)
    v = np.concatenate([np.repeat(special, special.size), r, r])
    t = np.concatenate([np.tile(special, special.size), rng.permutation(r), -r * (1 + 2.0 ** -30)])
    n = v.size
    plane, x = ag.AccumPlane((1,), n), ag.Array("f64", (1,), n)
    plane.data[0, :n] = torch.from_numpy(v)
    x.upload(t[None, :])
    plane.add(x.view())
    with np.errstate(all="ignore"):
        s, e = _knuth(v, t)
    got = plane.data[:, :n].cpu().numpy()
    assert np.array_equal(got[0], s, equal_nan=True)
    assert np.array_equal(got[1], 0.0 + e, equal_nan=True)
