"""The work that performance is measured on.

Each case is one call, or one small group of calls, that a program makes
through the package's public entry points: a fused assignment (every lowering,
plain and wrapped buffers), Philox fills, compensated reductions, an uneven
batch in one launch, the runtime-typed evaluator and a serving loop. Sizes and
distributions are those of the benchmark's configurations and of the tests,
with ragged ones beside them.

`listed()` are the standing cases, `draw(rng)` gives one more from the same
ranges, `prepare` makes a case's inputs and the plans a program keeps,
`run` is one pass, `work` the bytes and operations a pass cannot do without,
and `exact` its outputs in 64 bits without this package.
"""

import math

import numpy as np
import torch

import aether_gb300 as ag
from aether_gb300 import serve as ag_serve

MASK64 = (1 << 64) - 1
TORCH = {"f64": torch.float64, "f32": torch.float32, "ff": torch.float32}
SIZE = {"f64": 8, "f32": 4, "ff": 8}


def listed():
    return [
        # the plain fused expression on a few thousand samples, written as one
        # statement in an interactive program or an outer loop: latency counts
        {"name": "assign_small", "kind": "expr", "form": "fused", "store": "f64", "out": "f64", "math": 0, "n": 4099,
         "call": "assign", "memory": "array"},
        # the same expression on config 1's 2^20 samples in the default lowering
        {"name": "fused_f64", "kind": "expr", "form": "fused", "store": "f64", "out": "f64", "math": 0, "n": 1 << 20,
         "call": "prepared", "memory": "array"},
        # the large streaming expression of the benchmark, double-float
        {"name": "stream_emulated", "kind": "expr", "form": "stream", "store": "f64", "out": "f64", "math": 1,
         "n": 1 << 26, "call": "prepared", "memory": "array"},
        # the same at FP64 grade, a ragged size
        {"name": "stream_grade", "kind": "expr", "form": "stream", "store": "f64", "out": "f64", "math": 3,
         "n": (1 << 24) + 37, "call": "prepared", "memory": "array"},
        # quaternion rotation of f32 vectors held in another library's
        # unpadded tensors (odd pitch), the plain lowering
        {"name": "rotate_f32", "kind": "expr", "form": "rotate", "store": "f32", "out": "f32", "math": 0,
         "n": 10000003, "call": "prepared", "memory": "wrapped"},
        # Monte Carlo inputs in the default lowering: uniform vectors and N(0, 1) draws
        {"name": "fill_f64", "kind": "fill", "store": "f64", "math": 0, "n": 10000019},
        # the benchmark's normal fill, double-float
        {"name": "normal_emulated", "kind": "normal", "store": "f64", "math": 1, "n": 1 << 28},
        # the precision form: per-sample dot products and their global sum
        {"name": "dot_sum_f32", "kind": "sum", "store": "f32", "math": 2, "comps": 8, "n": 1 << 26, "keep": True},
        # a compensated global sum of f64 dot products, ragged
        {"name": "sum_f64", "kind": "sum", "store": "f64", "math": 0, "comps": 3, "n": (1 << 25) + 11, "keep": False},
        # uneven arrays of three kinds in one persistent launch
        {"name": "batch_uneven", "kind": "batch", "items": 2048, "median": 4096, "math": 1},
        # a + s b over transposed and sliced tensors of a runtime-typed caller
        {"name": "runtime_strided", "kind": "runtime", "op": "AddScaled", "store": "f64", "view": "transposed",
         "d0": 96, "d1": 509, "d2": 515},
        # requests of mixed shapes on resident operands, results back to the host
        {"name": "serve_mixed", "kind": "serve", "requests": 48, "median": 16384},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["expr", "expr", "expr", "fill", "normal", "sum", "sum", "accumulate", "batch", "runtime",
                       "runtime", "serve"])
    if kind == "expr":
        form = rng.choice(["fused", "stream", "rotate", "arith", "inverse"])
        store = rng.choice(["f64", "f64", "f32"])
        lower = rng.choice([0, 0, 1, 3]) if store == "f64" else rng.choice([0, 2])
        out = "ff" if lower == 2 and form in ("fused", "stream") and rng.random() < 0.5 else store
        top = (1 << 25) if lower or form in ("rotate", "arith") else (1 << 23)
        return {"kind": kind, "form": form, "store": store, "out": out, "math": lower, "n": _log_int(rng, 300, top),
                "call": rng.choice(["assign", "prepared"]), "memory": rng.choice(["array", "array", "wrapped"])}
    if kind == "fill":
        store = rng.choice(["f64", "f64", "f32"])
        return {"kind": kind, "store": store, "math": rng.choice([0, 1]) if store == "f64" else 0,
                "n": _log_int(rng, 1000, 1 << 24)}
    if kind == "normal":
        return {"kind": kind, "store": "f64", "math": rng.choice([0, 1, 3]), "n": _log_int(rng, 1000, 1 << 25)}
    if kind == "sum":
        store = rng.choice(["f64", "f32"])
        return {"kind": kind, "store": store, "math": rng.choice([0, 1]) if store == "f64" else rng.choice([0, 2]),
                "comps": rng.choice([1, 3, 8]), "n": _log_int(rng, 500, 1 << 25), "keep": rng.random() < 0.5}
    if kind == "accumulate":
        return {"kind": kind, "comps": rng.choice([1, 3]), "n": _log_int(rng, 1000, 1 << 24)}
    if kind == "batch":
        return {"kind": kind, "items": _log_int(rng, 16, 2048), "median": _log_int(rng, 256, 4096),
                "math": rng.choice([0, 1, 3])}
    if kind == "runtime":
        return {"kind": kind, "op": rng.choice(["Assign", "Add", "AddScaled", "SubScaled", "Scale"]),
                "store": rng.choice(["f64", "f32"]), "view": rng.choice(["contiguous", "transposed", "sliced"]),
                "d0": _log_int(rng, 3, 96), "d1": _log_int(rng, 17, 512), "d2": _log_int(rng, 33, 512)}
    return {"kind": kind, "requests": _log_int(rng, 4, 60), "median": _log_int(rng, 1024, 32768)}


# ---------------------------------------------------------------------------
# Inputs, from the seed alone.
# ---------------------------------------------------------------------------
# form -> (components and value range of each operand, output components)
FORMS = {
    "fused": ([(3, -1.0, 1.0)] * 3, 3),       # config 1
    "stream": ([(3, -4.0, 4.0)] * 4, 3),      # config 2
    "rotate": ([(4, -1.0, 1.0), (3, -1.0, 1.0)], 3),
    "arith": ([(3, -1.0, 1.0)] * 3, 3),
    "inverse": ([(9, -1.0, 1.0)], 9),
}


def _planes(comps, n, dtype, memory):
    """A (comps, pitch) device buffer: the package's own padded planes, or the
    gapless rows of another library's tensor."""
    if memory == "wrapped":
        return torch.zeros((comps, n), dtype=dtype, device="cuda")
    return torch.zeros((comps, ag.quantized_capacity(n)), dtype=dtype, device="cuda")


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _operands(case, seed):
    g = _gen(seed)
    out = []
    for comps, lo, hi in FORMS[case["form"]][0]:
        t = _planes(comps, case["n"], TORCH[case["store"]], case["memory"])
        t.uniform_(lo, hi, generator=g)
        if case["form"] == "inverse":
            t[0::4] += 2.5   # matrices away from singular
        out.append(t)
    return out


def _expression(form, v):
    if form == "fused":
        a, b, c = v
        return a + b * c + ag.cwiseSin(a) * ag.cwiseExp((c * c) * (-1.0))
    if form == "stream":
        a, b, c, d = v
        return ag.cwiseSqrt(a * a + b * b) * ag.cwiseLog1p(ag.cwiseAbs(c)) + ag.cwiseRsqrt(ag.constant(1.0, (3,)) + d * d)
    if form == "rotate":
        return v[0].quatRotate(v[1])
    if form == "arith":
        a, b, c = v
        return a + b * c
    m = v[0]
    return ag.select(ag.cwiseAbs(m.det()) > 1e-300, m.inverse(), ag.constant(0.0, (3, 3)))


def _elementwise(form, v, lib):
    """The same in torch or numpy (`lib`), on (comps, n) values."""
    if form == "fused":
        a, b, c = v
        return a + b * c + lib.sin(a) * lib.exp(-(c * c))
    if form == "stream":
        a, b, c, d = v
        return lib.sqrt(a * a + b * b) * lib.log1p(abs(c)) + 1 / lib.sqrt(1 + d * d)
    if form == "arith":
        a, b, c = v
        return a + b * c
    if form == "cross":
        a, b = v
        return lib.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])
    if form == "rotate":
        q, p = v
        t = [2 * (q[2] * p[2] - q[3] * p[1]), 2 * (q[3] * p[0] - q[1] * p[2]), 2 * (q[1] * p[1] - q[2] * p[0])]
        return lib.stack([p[0] + q[0] * t[0] + (q[2] * t[2] - q[3] * t[1]),
                          p[1] + q[0] * t[1] + (q[3] * t[0] - q[1] * t[2]),
                          p[2] + q[0] * t[2] + (q[1] * t[1] - q[2] * t[0])])
    m = v[0]
    cof = [m[4] * m[8] - m[5] * m[7], m[2] * m[7] - m[1] * m[8], m[1] * m[5] - m[2] * m[4],
           m[5] * m[6] - m[3] * m[8], m[0] * m[8] - m[2] * m[6], m[2] * m[3] - m[0] * m[5],
           m[3] * m[7] - m[4] * m[6], m[1] * m[6] - m[0] * m[7], m[0] * m[4] - m[1] * m[3]]
    det = m[0] * cof[0] + m[1] * cof[3] + m[2] * cof[6]
    return lib.stack([c / det for c in cof])


def _shape(comps):
    return (3, 3) if comps == 9 else (comps,)


def _launch(state, dst, expr, case, **kw):
    """Keep a bound launch, or the statement itself for a program that writes
    `assign` where it needs it."""
    if case.get("call") == "assign":
        state["statement"] = (dst, expr, dict(kw, math=case["math"]))
    else:
        state["launches"] = [ag.prepare(dst, expr, math=case["math"], **kw)]


# ---------------------------------------------------------------------------
# Philox4x32-10 in torch, for exact(): the generator's published algorithm and
# the package's documented keying and word conversions.
# ---------------------------------------------------------------------------
UNIFORM_SALT, NORMAL_SALT = 0x243F6A8885A308D3, 0x13198A2E03707344


def _splitmix64(x):
    x = (x + 0x9E3779B97F4A7C15) & MASK64
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & MASK64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & MASK64
    return x ^ (x >> 31)


def _key(seed, sub):
    key = _splitmix64(seed ^ _splitmix64(0))
    return _splitmix64(key ^ _splitmix64(sub ^ 0x2545F4914F6CDD1D))


def _philox(key, n, counter):
    low = 0xFFFFFFFF
    kx, ky = key & low, key >> 32
    z = torch.zeros(n, dtype=torch.int64, device="cuda")
    c = [z + counter, z, torch.arange(n, dtype=torch.int64, device="cuda"), z]
    for r in range(10):
        if r:
            kx, ky = (kx + 0x9E3779B9) & low, (ky + 0xBB67AE85) & low
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & low) ^ c[1] ^ kx, p1 & low, ((p0 >> 32) & low) ^ c[3] ^ ky, p0 & low]
    return c


def _uniform(key, n, comps, lo, hi, store):
    out = []
    for k in range(comps):
        w = _philox(key ^ UNIFORM_SALT, n, k)[0]
        if store == "f32":
            u = (((w >> 9) << 1) | 1).double() * float(np.float32(5.9604645e-8))
        else:
            u = w.double() * 2.0 ** -32 + 2.0 ** -33
        out.append(lo + (hi - lo) * u)
    return torch.stack(out)


def _normal(key, n, store):
    x = _philox(key ^ NORMAL_SALT, n, 0)
    if store == "f32":
        k = np.float32(2.3283064e-10) * np.float32(6.2831855)
        u = (((x[0] >> 9) << 1) | 1).float() * np.float32(5.9604645e-8).item()
        v = x[1].float() * k.item() + (k / np.float32(2)).item()
        u, v = u.double(), v.double()
    else:
        u = (x[0] ^ (x[1] << 21)).double() * 2.0 ** -53 + 2.0 ** -54
        v = ((x[2] ^ (x[3] << 21)).double() * 2.0 ** -52 + 2.0 ** -53) * math.pi
    if n > 1 << 24:
        return torch.sqrt(-2.0 * torch.log(u)) * torch.sin(v)
    u, v = u.cpu().numpy(), v.cpu().numpy()
    return torch.from_numpy(np.sqrt(-2.0 * np.log(u)) * np.sin(v))


# ---------------------------------------------------------------------------
# Batches: arrays carved from a few pools, as a program with its own arena holds them.
# ---------------------------------------------------------------------------
KINDS = [("cross", [3, 3], 3), ("rotate", [4, 3], 3), ("inverse", [9], 9)]


def _batch_sizes(case):
    r = np.random.default_rng(case["items"] * 1000003 + case["median"])
    return np.clip(np.round(r.lognormal(math.log(case["median"]), 1.5, case["items"])), 64, 1 << 21).astype(int).tolist()


def _batch_layout(case):
    """Per kind: [(offset, n)], and the pool's samples."""
    spots, total = [[], [], []], [0, 0, 0]
    for i, n in enumerate(_batch_sizes(case)):
        spots[i % 3].append((total[i % 3], n))
        total[i % 3] += ag.quantized_capacity(n)
    return spots, [max(t, 32) for t in total]


def _batch_pools(case, seed):
    g = _gen(seed)
    spots, total = _batch_layout(case)
    pools = []
    for (form, comps, _), t in zip(KINDS, total):
        ins = []
        for c in comps:
            x = torch.zeros((c, t), dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)
            if form == "inverse":
                x[0::4] += 2.5
            ins.append(x)
        pools.append(ins)
    return spots, total, pools


# ---------------------------------------------------------------------------
# Runtime-typed views.
# ---------------------------------------------------------------------------
def _runtime_views(case, seed):
    """Tensors (a, b, out) of one logical shape: gapless, permuted axes, or a
    window of a larger tensor with every other plane."""
    g = _gen(seed)
    dt = TORCH[case["store"]]
    d = (case["d0"], case["d1"], case["d2"])

    def make(k):
        if case["view"] == "transposed" and k == 1:
            t = torch.empty((d[2], d[0], d[1]), dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=g)
            return t.permute(1, 2, 0)
        if case["view"] == "sliced":
            t = torch.empty((2 * d[0], d[1] + 3, d[2] + 5), dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=g)
            return t[::2, 1:d[1] + 1, 2:d[2] + 2]
        return torch.empty(d, dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=g)

    return make(0), make(1), make(2)


RUNTIME_B = ("Add", "AddScaled", "SubScaled")


# ---------------------------------------------------------------------------
# Serving: requests over the standard shapes.
# ---------------------------------------------------------------------------
SERVE_FORMS = ["fused", "fused", "stream", "stream", "dot8", "cross", "rotate", "inverse"]


def _serve_trace(case, seed):
    r = np.random.default_rng(case["requests"] * 65537 + case["median"])
    sizes = np.clip(np.round(r.lognormal(math.log(case["median"]), 1.0, case["requests"])), 1024, 1 << 18).astype(int)
    values = np.random.default_rng(seed)
    trace = []
    for i, n in enumerate(sizes.tolist()):
        k = i % 8
        trace.append((k, n, values.integers(1 << 60)))
    return trace


def _serve_values(shapes, k, n, seed):
    """Host operand planes of one request (capacity pitch)."""
    r = np.random.default_rng(int(seed))
    out = []
    for dt, sh in shapes[k].operands:
        comps = int(np.prod(sh)) if sh else 1
        x = r.random((comps, ag_serve.capacity(n)), dtype=np.float64 if dt == "f64" else np.float32) * 2 - 1
        if SERVE_FORMS[k] == "inverse":
            x[0::4] += 2.5
        out.append(x)
    return out


class _Shape:
    """What exact() needs of a served shape."""

    def __init__(self, operands):
        self.operands = operands


_V3, _V4, _V8, _M9 = (3,), (4,), (8,), (3, 3)
SERVE_OPERANDS = [_Shape(o) for o in (
    [("f64", _V3)] * 3, [("f32", _V3)] * 3, [("f64", _V3)] * 4, [("f32", _V3)] * 4, [("f32", _V8)] * 2,
    [("f64", _V3)] * 2, [("f64", _V4), ("f64", _V3)], [("f64", _M9)])]


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "expr":
        ins = _operands(case, seed)
        comps = FORMS[case["form"]][1]
        planes = comps * (2 if case["out"] == "ff" else 1)
        buf = _planes(planes, case["n"], TORCH[case["out"]], case["memory"])
        views = [ag.Array.wrap(t, shape=_shape(t.shape[0]), n=case["n"]).view() for t in ins]
        dst = ag.Array(case["out"], _shape(comps), case["n"], data=buf)
        state["outputs"] = [buf]
        _launch(state, dst, _expression(case["form"], views), case)
    elif kind in ("fill", "normal"):
        n, g = case["n"], ag.Generator(seed)
        z = ag.Array(case["store"], (1,), n)
        state["launches"] = [ag.prepare(z, g.substream(1).normal(1, 0.0, 1.0), math=case["math"])]
        state["outputs"] = [z.data]
        if kind == "fill":
            u = ag.Array(case["store"], (3,), n)
            state["launches"].insert(0, ag.prepare(u, g.substream(0).uniform(3, -1.0, 1.0), math=case["math"]))
            state["outputs"].insert(0, u.data)
    elif kind == "sum":
        n = case["n"]
        x, y = _sum_inputs(case, seed)
        e = x.view().dot(y.view())
        total = torch.zeros(2, dtype=torch.float64, device="cuda")
        state["total"] = total
        state["outputs"] = []
        if case["keep"]:
            d = ag.Array(case["store"], (1,), n)
            state["launches"] = [ag.prepare(d, e, op="setsum", reduce_out=total, math=case["math"])]
            state["outputs"].append(d.data)
        else:
            state["launches"] = [ag.prepare((case["store"], ()), e, op="sum", n=n, reduce_out=total, math=case["math"])]
    elif kind == "accumulate":
        n, c = case["n"], case["comps"]
        plane = ag.AccumPlane((c,), n)
        x, y = (ag.Array("f64", (c,), n) for _ in range(2))
        g = _gen(seed)
        plane.data[:c].uniform_(-1e3, 1e3, generator=g)
        for t in (x, y):
            t.data.uniform_(-1.0, 1.0, generator=g)
        state["launches"] = [ag.prepare(plane, x.view() * y.view(), op="acc")]
        state["outputs"] = [plane.data]
        state["hold"] = (x, y)
    elif kind == "batch":
        spots, total, pools = _batch_pools(case, seed)
        launches, outs = [], [torch.zeros((c, t), dtype=torch.float64, device="cuda") for (_, _, c), t in zip(KINDS, total)]
        for k, (form, _, comps) in enumerate(KINDS):
            for off, n in spots[k]:
                views = [ag.Array.wrap(p[:, off:off + n], shape=_shape(p.shape[0]), n=n).view() for p in pools[k]]
                dst = ag.Array.wrap(outs[k][:, off:off + n], shape=_shape(comps), n=n)
                e = views[0].cross(views[1]) if form == "cross" else _expression(form, views)
                launches.append(ag.prepare(dst, e, math=case["math"]))
        state["batch"] = ag.Batch(launches)
        state["outputs"] = outs
        state["hold"] = pools
    elif kind == "runtime":
        a, b, out = _runtime_views(case, seed)
        state.update(op=getattr(ag.RuntimeOp, case["op"]), a=a, b=b if case["op"] in RUNTIME_B else None, out=out)
    else:
        shapes = ag_serve.standard_shapes()
        server = ag_serve.Server(shapes, 2 << 30)
        requests, outputs, hold = [], [], []
        for i, (k, n, vs) in enumerate(_serve_trace(case, seed)):
            hosts = [torch.from_numpy(x).pin_memory() for x in _serve_values(shapes, k, n, vs)]
            dt = TORCH[shapes[k].out_dtype]
            out = torch.zeros((shapes[k].out_comps, ag_serve.capacity(n)), dtype=dt, pin_memory=True)
            ids = [1 + 8 * i + j for j in range(len(hosts))]
            requests.append(server.request(k, n, ids, [h.data_ptr() for h in hosts], host_out=out))
            outputs.append(out[:, :n])   # the planes' spare samples are not written
            hold.append(hosts)
        state.update(server=server, requests=requests, outputs=outputs, hold=hold)
    return state


def _sum_inputs(case, seed):
    """Log-uniform magnitudes of random sign, 1e-3..1e3 (config 3's form)."""
    g = _gen(seed)
    out = []
    for _ in range(2):
        a = ag.Array(case["store"], (case["comps"],), case["n"])
        a.data.uniform_(-3.0, 3.0, generator=g)
        a.data.mul_(math.log(10.0)).exp_()
        for p in a.data:   # random signs, one plane at a time
            p.mul_(torch.randint(0, 2, p.shape, generator=g, device="cuda", dtype=torch.int8).mul_(2).sub_(1))
        out.append(a)
    return out


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].launch()
    elif kind == "runtime":
        ag.runtime_eval(state["op"], state["a"], state["b"], state["out"], scalar=0.375)
        return state["out"]
    elif kind == "serve":
        server = state["server"]
        server.wait_all([server.submit(r) for r in state["requests"]])
    elif "statement" in state:
        dst, expr, kw = state["statement"]
        ag.assign(dst, expr, **kw)
    else:
        for launch in state["launches"]:
            launch()
        if kind == "sum":   # the pair (hi, comp) stands for one number, its sum
            return [state["total"].sum()] + state["outputs"]
    return state["outputs"]


def work(case):
    kind = case["kind"]
    if kind == "expr":
        ins, out = FORMS[case["form"]]
        n = case["n"]
        ops = {"fused": 24, "stream": 30, "rotate": 33, "arith": 6, "inverse": 50}[case["form"]]
        return {"bytes": n * (sum(c for c, _, _ in ins) * SIZE[case["store"]] + out * SIZE[case["out"]]), "flops": n * ops}
    if kind == "normal":
        return {"bytes": case["n"] * SIZE[case["store"]], "flops": case["n"] * 8}
    if kind == "fill":
        return {"bytes": case["n"] * 4 * SIZE[case["store"]], "flops": case["n"] * 14}
    if kind == "sum":
        planes = 2 * case["comps"] + (1 if case["keep"] else 0)
        return {"bytes": case["n"] * planes * SIZE[case["store"]] + 16, "flops": case["n"] * (2 * case["comps"] + 1)}
    if kind == "accumulate":
        return {"bytes": case["n"] * case["comps"] * 8 * 6, "flops": case["n"] * case["comps"] * 9}
    if kind == "batch":
        spots, _ = _batch_layout(case)
        nbytes = flops = 0
        for (form, comps, out), sp in zip(KINDS, spots):
            n = sum(s[1] for s in sp)
            nbytes += n * 8 * (sum(comps) + out)
            flops += n * {"cross": 9, "rotate": 33, "inverse": 50}[form]
        return {"bytes": nbytes, "flops": flops}
    if kind == "runtime":
        n = case["d0"] * case["d1"] * case["d2"]
        return {"bytes": n * SIZE[case["store"]] * (3 if case["op"] in RUNTIME_B else 2), "flops": 2 * n}
    nbytes = flops = 0
    outs = [24, 12, 24, 12, 4, 24, 24, 72]
    for k, n, _ in _serve_trace(case, 0):
        nbytes += n * (sum(int(np.prod(sh)) * SIZE[dt] for dt, sh in SERVE_OPERANDS[k].operands) + outs[k])
        flops += n * 30
    return {"bytes": nbytes, "flops": flops}


def _pad(values, width):
    """(comps, n) values in planes of `width` samples, zero beyond n."""
    out = torch.zeros((values.shape[0], width), dtype=torch.float64, device=values.device)
    out[:, : values.shape[1]] = values
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "expr":
        n = case["n"]
        ins = [t[:, :n] for t in _operands(case, seed)]
        width = n if case["memory"] == "wrapped" else ag_serve.capacity(n)
        if n <= 1 << 20 and case["form"] in ("fused", "stream"):
            # wide enough that what is left is the result's own rounding
            v = [t.cpu().numpy().astype(np.longdouble) for t in ins]
            y = _elementwise(case["form"], v, np)
            hi = torch.from_numpy(y.astype(np.float64))
        else:
            hi = _elementwise(case["form"], [t.double() for t in ins], torch)
        if case["out"] == "ff":   # the value as a pair of floats
            head = hi.float().double()
            hi = torch.cat([head, (hi - head).float().double()])
        return [_pad(hi, width)]
    if kind in ("fill", "normal"):
        n = case["n"]
        width = ag_serve.capacity(n)
        out = [_pad(_normal(_key(seed, 1), n, case["store"]).reshape(1, n), width)]
        if kind == "fill":
            out.insert(0, _pad(_uniform(_key(seed, 0), n, 3, -1.0, 1.0, case["store"]), width))
        return out
    if kind == "sum":
        n = case["n"]
        x, y = (a.data[:, :n] for a in _sum_inputs(case, seed))
        d = torch.zeros(n, dtype=torch.float64, device="cuda")
        for p, q in zip(x, y):
            d += p.double() * q.double()
        rows = d[: n // 64 * 64].reshape(64, -1)
        total = math.fsum([math.fsum(r.sum(dim=0).reshape(1).tolist()) for r in rows] + d[n // 64 * 64:].tolist())
        out = [torch.tensor(total, dtype=torch.float64)]
        if case["keep"]:
            out.append(_pad(d.reshape(1, n), ag_serve.capacity(n)))
        return out
    if kind == "accumulate":
        return None   # the compensation planes are the residuals of the value planes' own roundings
    if kind == "batch":
        spots, total, pools = _batch_pools(case, seed)
        out = []
        for k, (form, _, _) in enumerate(KINDS):
            y = _elementwise(form, pools[k], torch)
            live = torch.zeros(total[k], dtype=torch.float64, device="cuda")
            for off, n in spots[k]:
                live[off:off + n] = 1.0
            out.append(y * live)
        return out
    if kind == "runtime":
        a, b, out = _runtime_views(case, seed)
        a, b, s = a.double(), b.double(), 0.375
        return {"Assign": lambda: a, "Add": lambda: a + b, "AddScaled": lambda: a + s * b,
                "SubScaled": lambda: a - s * b, "Scale": lambda: s * a}[case["op"]]()
    out = []
    for k, n, vs in _serve_trace(case, seed):
        v = [torch.from_numpy(x[:, :n]).cuda().double() for x in _serve_values(SERVE_OPERANDS, k, n, vs)]
        y = (v[0] * v[1]).sum(dim=0, keepdim=True) if SERVE_FORMS[k] == "dot8" else _elementwise(SERVE_FORMS[k], v, torch)
        out.append(y)
    return out
