"""Launches that run the one-sample kernel for their size: the bits of the
vector kernel (the same plan with its block named) at the sizes where the choice
turns and at the smallest ones, in an assignment and under capture."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag


def _light(a, b):
    return a * b - b


def _heavy(a, b):
    return ag.cwiseExp(a) * ag.cwiseSin(b) + ag.cwiseDiv(a, b)


@pytest.mark.parametrize("form", [_light, _heavy])
@pytest.mark.parametrize("math,dt", [(0, "f64"), (1, "f64"), (2, "f32"), (3, "f64")])
def test_same_bits_around_the_limits(form, math, dt):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (1, 2, 3, 65, 512 * sms - 1, 512 * sms, 512 * sms + 1, 2048 * sms - 1, 2048 * sms, 2048 * sms + 1):
        a, b, d, e = (ag.Array(dt, (2,), n) for _ in range(4))
        a.data.uniform_(-2, 2)
        b.data.uniform_(0.5, 2)
        L = ag.prepare(d, form(a.view(), b.view()), math=math)
        L()
        ag.assign(e, form(a.view(), b.view()), math=math, block=256)
        assert torch.equal(d.data[:, :n], e.data[:, :n]), n
        if n < 100:
            d.data.zero_()
            s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.current_stream())
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                L()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(d.data[:, :n], e.data[:, :n]), n
