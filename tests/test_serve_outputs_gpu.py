"""Where a served request's output may go: pageable memory, mapped pinned memory
(written by the kernel up to 8 MiB, copied above), the same off a 16-byte
boundary, and outputs also kept on the device. The same samples everywhere, and
nothing written outside the output's planes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


import aether_gb300 as ag
from aether_gb300 import serve

GUARD = 64


@pytest.fixture(scope="module")
def shapes():
    return serve.standard_shapes()


@pytest.fixture(scope="module")
def pools():
    return serve.HostPools(f64_bytes=64 << 20, f32_bytes=32 << 20, seed=4)


# 349525 planes of three doubles: 8 MiB less 8 bytes before padding
@pytest.mark.parametrize("n", [1, 31, 4097, 349504, 349536, 500001])
@pytest.mark.parametrize("mode", ["batched", "plain"])
def test_outputs(shapes, pools, n, mode):
    k = [s.name for s in shapes].index("cross_f64")
    sh, cap = shapes[k], serve.capacity(n)
    ids = [701, 702]
    hosts = [pools.window(dt, i, sh.operand_bytes(j, n)) for j, ((dt, _), i) in enumerate(zip(sh.operands, ids))]
    size = sh.out_comps * cap
    kinds = [("pageable", False, 0, False), ("pinned", True, 0, False), ("unaligned", True, 1, False),
             ("pageable unaligned", False, 1, False), ("kept", True, 0, True)]
    bufs = [torch.full((size + 2 * GUARD,), 7.0, dtype=torch.float64, pin_memory=pin) for _, pin, _, _ in kinds]
    outs = [b[GUARD + off:GUARD + off + size] for b, (_, _, off, _) in zip(bufs, kinds)]
    with serve.Server(shapes, 1 << 30, mode=mode) as srv:
        for together in (False, True):
            for b in bufs:
                b.fill_(7.0)
            reqs = [srv.request(k, n, ids, hosts, host_out=o, keep=keep) for o, (_, _, _, keep) in zip(outs, kinds)]
            sts = srv.wait_all(srv.feed(reqs)) if together else [srv.wait(srv.submit(r)) for r in reqs]
            assert all(s["state"] == "done" for s in sts)
            want = outs[0].reshape(-1, cap)[:, :n]
            for (name, _, off, _), b, o in zip(kinds, bufs, outs):
                assert torch.equal(o.reshape(-1, cap)[:, :n], want), name
                assert torch.all(b[:GUARD + off] == 7.0) and torch.all(b[GUARD + off + size:] == 7.0), name
            a, c = (pools.array("f64", i, 3, n) for i in ids)
            np.testing.assert_allclose(want.numpy(), np.cross(a.T, c.T).T, rtol=0, atol=2.0 ** -44)
