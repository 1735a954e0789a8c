"""The native side of the frequent calls against the general way: same results, and what is out of the ordinary
goes the general way with the errors that it has."""
import numpy as np
import pytest
import torch

from ccbench_b200 import CcbError, Communicator
from ccbench_b200 import _lib
from ccbench_b200.comm import launch_count
from ccbench_b200.ops import lossless, standalone, sz
from ccbench_b200.parallel import moe

pytestmark = pytest.mark.gpu


def _general(monkeypatch):
    for module in (standalone, sz, _lib):
        monkeypatch.setattr(module, "calls", lambda: None)


def _everything(comm, n):
    g = torch.Generator(device="cuda").manual_seed(1)
    v = lambda *s: torch.randn(*s, generator=g, device="cuda")
    xs, es = [v(3000) for _ in range(n)], [torch.zeros(3000, device="cuda") for _ in range(n)]
    ys, zs, ws = [torch.empty_like(x) for x in xs], [torch.empty(3000 // n, device="cuda") for _ in xs], [torch.empty(3000 * n, device="cuda") for _ in xs]
    comm.all_reduce(xs, ys, codec="int8", error_feedback=es)
    comm.reduce_scatter(tuple(xs), zs, codec="fp8")
    comm.all_gather(xs, ws, codec="int4")
    rows = [v(40, 512).bfloat16() for _ in range(n)]
    routes = [moe.plan_route(torch.randint(0, n, (40, 2), generator=g, device="cuda"), v(40, 2), n) for _ in range(n)]
    counts = [r.send_counts.tolist() for r in routes]
    recv, out = [torch.zeros(80 * n, 512, dtype=torch.bfloat16, device="cuda") for _ in rows], [torch.empty_like(r) for r in rows]
    moe.dispatch(comm, rows, recv, routes, counts)
    moe.combine(comm, recv, out, routes, counts)
    wires = [standalone.encode(x, "int8") for x in xs]
    field = v(17, 9, 70)
    packed, used = sz.compress(field, 1e-2)
    blob = sz.to_container(packed, field.shape, 1e-2)
    again, shape, eb = sz.from_container(blob)
    half = xs[0].half()
    return [*ys, *es, *zs, *ws, *recv, *out, *[standalone.decode(w, "int8", 3000, torch.float32) for w in wires], standalone.decode(standalone.reduce_recode(wires, "int8", 3000), "int8", 3000, torch.float16), used, blob, again,
            torch.tensor([*shape, eb]), sz.decompress(again, shape, eb), lossless.decode(lossless.encode(half), 3000, torch.float16)]


@pytest.mark.parametrize("n", [2, 4])
def test_both_ways_give_the_same(n, monkeypatch):
    comm = Communicator.local(n, arena_bytes=32 << 20)
    assert comm._calls is not None and _lib.calls() is not None
    before = launch_count()
    got = _everything(comm, n)
    launched = launch_count() - before
    _general(monkeypatch)
    comm._calls = None
    want = _everything(comm, n)
    assert launch_count() - before == 2 * launched
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape and a.device == b.device
        if a.dtype == torch.uint8 and a.numel() > 1 << 16:   # slots of a compressed field: used prefixes apart, anything
            continue
        assert torch.equal(a, b)
    comm.close()


def test_what_is_out_of_the_ordinary_goes_the_general_way():
    comm = Communicator.local(2, arena_bytes=16 << 20)
    x, y = torch.ones(512, device="cuda"), torch.empty(512, device="cuda")
    with pytest.raises(ValueError):
        comm.all_reduce([x], [y])
    with pytest.raises(ValueError):
        comm.all_reduce([x, torch.ones(1024, device="cuda")[::2]], [y, y.clone()])
    with pytest.raises(ValueError):
        comm.all_reduce([x, x.cpu()], [y, y.clone()])
    with pytest.raises(TypeError):
        comm.all_reduce([x.double(), x.double()], [y, y.clone()])
    with pytest.raises(KeyError):
        comm.all_reduce([x, x], [y, y.clone()], codec="int3")
    with pytest.raises(ValueError):
        comm.all_reduce([x, x], [y, y.clone()], error_feedback=[y, y[:100]])
    with pytest.raises(ValueError):
        comm.all_gather([x, x], [y, y])
    with pytest.raises(RuntimeError):
        torch.vmap(lambda v: comm.all_reduce([v, v], [v, v])[0])(torch.ones(3, 512, device="cuda"))
    with pytest.raises(CcbError):
        standalone.reduce_recode([standalone.encode(x, "int8")] * 17, "int8", 512)
    p = torch.nn.Parameter(x.clone())
    assert torch.equal(standalone.decode(standalone.encode(p, "fp8"), "fp8", np.int64(512), torch.float32), x)
    assert torch.equal(sz.decompress(sz.compress(x.view(1, 8, 64), 1)[0], [1, 8, 64], 1), x.view(1, 8, 64) * 0 + sz.decompress(sz.compress(x.view(1, 8, 64), 1.0)[0], (1, 8, 64), 1.0))
    comm.all_reduce(iter([x, x]), [y, y.clone()], codec="none")
    assert torch.equal(y, 2 * x)
    comm.close()
    with pytest.raises(CcbError):
        comm.all_reduce([x, x], [y, y.clone()])
