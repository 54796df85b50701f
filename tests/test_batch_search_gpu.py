"""The work-list search of a batched launch: item counts at the edges of the
32 probes of a step and far beyond them, items of one tile, of many and of
none, each item's result bit for bit that of its own samples."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag


@pytest.mark.parametrize("count,longest", [(1, 700), (2, 5000), (32, 3), (33, 3), (34, 60000), (1025, 1100), (1057, 1),
                                           (21000, 40), (600, 20000)])
def test_items_of_every_size(count, longest):
    rng = np.random.default_rng(count + longest)
    sizes = np.maximum(1, np.exp(rng.uniform(0, np.log(longest + 1), count)).astype(int) - 1)
    sizes[rng.random(count) < 0.1] = 0 if count > 2 else 1
    caps = [ag.quantized_capacity(max(1, int(n))) for n in sizes]
    offs = np.concatenate([[0], np.cumsum(caps)])
    x = torch.rand((3, int(offs[-1])), dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    launches = []
    for o, n in zip(offs[:-1].tolist(), sizes.tolist()):
        a = ag.Array.wrap(x[:, o:o + max(n, 1)], n=n)
        d = ag.Array.wrap(y[:, o:o + max(n, 1)], n=n)
        launches.append(ag.prepare(d, a.view() + a.view()))
    ag.Batch(launches).launch()
    live = torch.zeros(int(offs[-1]), dtype=torch.float64)
    for o, n in zip(offs[:-1].tolist(), sizes.tolist()):
        live[o:o + n] = 1.0
    assert torch.equal(y, (x + x) * live.cuda())
