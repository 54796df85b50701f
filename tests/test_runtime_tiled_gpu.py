"""The runtime evaluator's tiled kernel: permuted, sliced, broadcast and
gap-strided views at the edges of its tiles (32 x 32 with a turned input, 8 x
128 and 1 x 1024 without), against torch, bit for bit (each operation rounds
once), and with everything outside the output view left alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


from aether_gb300 import RuntimeOp, runtime_eval


def _view(rng, shape, order, pad, dtype, zero=None):
    """`shape` over a buffer whose axes lie in `order` (outermost first), `pad`
    spare elements on each."""
    strides, acc = [0] * len(shape), 1
    for k in reversed(order):
        strides[k] = acc * (2 if pad and k == order[-1] else 1)
        acc = strides[k] * (shape[k] + pad)
    if zero is not None:
        strides[zero] = 0
    base = torch.from_numpy(rng.uniform(-4, 4, acc + 9)).to(dtype).cuda()
    return base, base.as_strided(shape, strides, 5)


SHAPES = [(33, 65), (16, 16), (1, 31, 33), (32, 32, 32), (5, 129, 17), (3, 1, 1023), (2, 1025), (7, 2, 127, 18),
          (2, 3, 4, 5, 40), (1030,), (300, 15), (3, 5, 64)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_views(shape, dtype):
    rng = np.random.default_rng(len(shape) * 1000 + shape[-1])
    rank = len(shape)
    for _ in range(6):
        pick = [rng.permutation(rank).tolist() for _ in range(3)]
        pads = rng.integers(0, 2, 3)
        zero = int(rng.integers(rank)) if rng.random() < 0.3 else None
        _, a = _view(rng, shape, pick[0], int(pads[0]), dtype, zero)
        _, b = _view(rng, shape, pick[1], int(pads[1]), dtype)
        base, o = _view(rng, shape, pick[2], int(pads[2]), dtype)
        before = base.clone()
        runtime_eval(RuntimeOp.AddScaled, a, b, o, 0.75)
        want = a + b * 0.75   # the product is rounded, then the sum
        assert torch.equal(o, want)
        touched = torch.zeros(base.numel(), dtype=torch.bool, device="cuda")
        touched.as_strided(shape, o.stride(), 5).fill_(True)
        assert torch.equal(base[~touched], before[~touched])
        other = torch.float32 if dtype == torch.float64 else torch.float64
        _, c = _view(rng, shape, pick[2], int(pads[2]), other)
        runtime_eval(RuntimeOp.Assign, a, None, c)
        assert torch.equal(c, a.to(other))


def test_in_place():
    x = torch.rand((64, 70, 80), dtype=torch.float64, device="cuda").permute(2, 0, 1)
    want = x + x * 0.5
    runtime_eval(RuntimeOp.AddScaled, x, x, x, 0.5)
    assert torch.equal(x, want)
