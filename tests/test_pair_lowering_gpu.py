"""Kernels that hold two samples in a register pair and take one component of
a componentwise tree at a time, against the one-sample kernel of the same plan
(planes at an odd pitch): the same bits at the edges of a lane group, a chunk
and a grid, for every lowering; and a destination that lies one plane further
along its own operand."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag


def _fused(a, b, c):
    return a + b * c + ag.cwiseSin(a) * ag.cwiseExp((c * c) * (-1.0))


def _stream(a, b, c):
    return ag.cwiseSqrt(a * a + b * b) * ag.cwiseLog1p(ag.cwiseAbs(c)) + ag.cwiseRsqrt(ag.constant(1.0, (3,)) + c * c)


def _select(a, b, c):
    return ag.select(a > b, ag.cwiseCos(c), ag.clamp(ag.cwiseDiv(a, c), -2.0, 2.0)) + ag.Generator(3).normal(3, 0.0, 1.0)


def _mixed(a, b, c):   # not componentwise
    return a.cross(b) * ag.cwiseExp(c).norm() + c.unitVector()


@pytest.mark.parametrize("form", [_fused, _stream, _select, _mixed])
@pytest.mark.parametrize("store,out,math", [("f64", "f64", 0), ("f64", "f64", 1), ("f64", "f64", 3), ("f32", "ff", 2),
                                            ("f32", "f32", 2)])
def test_same_bits_as_one_sample_at_a_time(form, store, out, math):
    for n in (1, 2, 3, 511, 512, 513, 1025, 200003):
        g = torch.Generator(device="cuda").manual_seed(n)
        dt = torch.float64 if store == "f64" else torch.float32
        planes = 6 if out == "ff" else 3
        res = []
        src = [torch.rand((3, n), generator=g, device="cuda", dtype=dt) * 4 - 2 for _ in range(3)]
        for cap in ((n + 31) // 32 * 32, n | 1):
            ins = []
            for s in src:
                t = torch.zeros((3, cap), dtype=dt, device="cuda")
                t[:, :n] = s
                ins.append(ag.Array.wrap(t, n=n).view())
            buf = torch.full((planes, cap), 7.0, dtype=torch.float64 if out == "f64" else torch.float32, device="cuda")
            ag.assign(ag.Array(out, (3,), n, data=buf), form(*ins), math=math)
            assert torch.all(buf[:, n:] == 7.0)
            res.append(buf[:, :n])
        assert torch.equal(res[0], res[1]), (form.__name__, n)


@pytest.mark.parametrize("math", [0, 1, 3])
def test_destination_shifted_by_a_plane(math):
    n, cap = 40000, 40000
    buf = torch.rand((4, cap), dtype=torch.float64, device="cuda") + 0.5
    a = ag.Array.wrap(buf[:3].clone(), n=n)
    want = ag.Array("f64", (3,), n)
    ag.assign(want, ag.cwiseSin(a.view()) * ag.cwiseExp(a.view()), math=math)
    src, dst = ag.Array.wrap(buf[:3], n=n), ag.Array.wrap(buf[1:], n=n)
    ag.assign(dst, ag.cwiseSin(src.view()) * ag.cwiseExp(src.view()), math=math)
    assert torch.equal(buf[1:, :n], want.data[:, :n])
    # in place, component by component
    ag.assign(a, ag.cwiseSin(a.view()) * ag.cwiseExp(a.view()), math=math)
    assert torch.equal(a.data[:, :n], want.data[:, :n])
