"""Emulated, precision-form and FP64-grade assignments whose destination is one
of their operands, with samples that the fast path hands to the native lane
among ordinary ones: the same bits as into a buffer of its own, in place and
one plane further along, at the edges of a lane group and a chunk."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag

SPECIAL = {"f64": [0.0, -0.0, 1e-30, -1e30, 5e-324, 1e200, np.inf, np.nan, -2.0 ** -61],
           "f32": [0.0, -0.0, 1e-30, -1e30, 1e-44, 3e38, np.inf, np.nan, -2.0 ** -61]}


def _plain(v):
    return v * v + v


def _heavy(v):
    return ag.cwiseSin(v) * ag.cwiseExp(v) + v


@pytest.mark.parametrize("form", [_plain, _heavy])
@pytest.mark.parametrize("math,dt", [(1, "f64"), (3, "f64"), (2, "f32")])
@pytest.mark.parametrize("low", [{}, {"ipt": 2}, {"vec": 1}])
def test_in_place(form, math, dt, low):
    for n in (1, 2, 5, 513, 40001):
        for cap in ((n + 31) // 32 * 32, n | 1):
            r = np.random.default_rng(n)
            x = r.uniform(0.5, 1.5, (4, cap))
            special = r.random((4, cap)) < 0.2
            x[special] = r.choice(SPECIAL[dt], special.sum())
            buf = torch.from_numpy(x.astype(np.float64 if dt == "f64" else np.float32)).cuda()
            want = torch.full((3, cap), 7.0, dtype=buf.dtype, device="cuda")
            src = ag.Array.wrap(buf[:3].clone(), n=n)
            ag.assign(ag.Array(dt, (3,), n, data=want), form(src.view()), math=math, **low)
            # in place
            own = ag.Array.wrap(buf[:3].clone(), n=n)
            ag.assign(own, form(own.view()), math=math, **low)
            same = lambda a, b: torch.equal(torch.nan_to_num(a, nan=12345.0), torch.nan_to_num(b, nan=12345.0))
            assert same(own.data[:, :n], want[:, :n]), (n, cap)
            assert same(own.data[:, n:], buf[:3, n:])
            # one plane further along
            s = ag.Array.wrap(buf[:3], n=n)
            ag.assign(ag.Array.wrap(buf[1:], n=n), form(s.view()), math=math, **low)
            assert same(buf[1:, :n], want[:, :n]), (n, cap)
