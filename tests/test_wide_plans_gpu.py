"""Plans of many components whose caller names no block: they keep the
registers they need, and give the bits of the plan compiled for 256 threads."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag


def _fused(v):
    return v[0] + v[1] * v[2] + ag.cwiseSin(v[0]) * ag.cwiseExp((v[2] * v[2]) * (-1.0))


def _products(v):
    return v[0] * v[1] - v[2] * v[2]


@pytest.mark.parametrize("form", [_fused, _products])
@pytest.mark.parametrize("math,dt", [(0, "f64"), (1, "f64"), (2, "f32"), (3, "f64")])
@pytest.mark.parametrize("comps", [4, 6, 9])
def test_wide_trees(form, math, dt, comps):
    for n in (1, 700, 300001):
        a = [ag.Array(dt, (comps,), n) for _ in range(3)]
        for x in a:
            x.data.uniform_(-1, 1)
        d, e = ag.Array(dt, (comps,), n), ag.Array(dt, (comps,), n)
        own = ag.prepare(d, form([x.view() for x in a]), math=math)
        ref = ag.prepare(e, form([x.view() for x in a]), math=math, block=256)
        own()
        ref()
        assert torch.equal(d.data[:, :n], e.data[:, :n])
    # a thread of the widest kernels needs more than the 80 registers that
    # 768 threads leave it
    if comps == 9 and math:
        assert own.plan.info().registers > 80, (own.plan.info().registers, own.plan.info().block)
