"""Exchanges of ranks of one GPU at odd offsets, in runs of one to eight units a warp: the sectors where runs
meet, blocks in place, and rows of experts in groups of units that do not divide them. Against the kernels of
ranks on several GPUs: same inputs, same bits."""
import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.parallel import moe

pytestmark = pytest.mark.gpu


def _values(count, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(count, generator=g, device="cuda").to(dtype)
    x[::97] *= 100
    return x


def _both(comm, call):
    got = call()
    comm.set_trace(True)
    want = call()
    comm.set_trace(False)
    torch.cuda.synchronize()
    assert comm.status()[0] == 0
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.parametrize("dtype,codec", [(torch.bfloat16, "fp8"), (torch.float16, "int4"), (torch.float32, "int8")])
@pytest.mark.parametrize("n,count", [(2, 400_001), (8, 600_003), (8, 1_000_007), (4, 3_700_001)])
@pytest.mark.parametrize("in_place", [False, True])
def test_all_gather_of_odd_blocks(dtype, codec, n, count, in_place):
    comm = Communicator.local(n, arena_bytes=160 << 20)
    xs = [_values(count, dtype, r) for r in range(n)]

    def call():
        out = [torch.full((n * count + 3,), 7.0, dtype=dtype, device="cuda")[1:-2] for _ in range(n)]
        if in_place:
            for r in range(n):
                out[r][r * count:(r + 1) * count] = xs[r]
        comm.all_gather([o[r * count:(r + 1) * count] for r, o in enumerate(out)] if in_place else xs, out, codec=codec)
        return out

    _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("codec", ["none", "int8", "int4"])
@pytest.mark.parametrize("topk", [1, 2, 3, 5, 9])   # beyond four (fp32: two) the rows of a token take several turns
@pytest.mark.parametrize("hidden", [512, 1536, 3584])
def test_rows_in_groups_of_units(dtype, codec, topk, hidden):
    n, tokens = 3, 61
    comm = Communicator.local(n, arena_bytes=96 << 20)
    g = torch.Generator().manual_seed(topk)
    xs = [_values(tokens * hidden, dtype, r).view(tokens, hidden) for r in range(n)]
    routes, counts = [], []
    for r in range(n):
        ids = torch.randint(0, n, (tokens, topk), generator=g).cuda()
        routes.append(moe.plan_route(ids, torch.rand(tokens, topk, generator=g).cuda(), n))
        counts.append(routes[r].send_counts.tolist())
    pairs = torch.arange(0, tokens * topk, 7, device="cuda")
    for r in range(n):
        routes[r].pos[pairs] = -1   # dropped on the way back
    rows_in = [sum(counts[s][d] for s in range(n)) for d in range(n)]

    def call():
        recv = [torch.zeros(max(k, 1), hidden, dtype=dtype, device="cuda") for k in rows_in]
        out = [torch.full_like(x, 3.0) for x in xs]
        moe.dispatch(comm, xs, recv, routes, counts, codec=codec)
        moe.combine(comm, recv, out, routes, counts, codec=codec)
        return recv + out

    _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hidden", [512, 1536, 4096])
def test_a_token_of_no_rows_is_zero(dtype, hidden):
    n, tokens = 2, 37
    comm = Communicator.local(n, arena_bytes=32 << 20)
    routes = [moe.plan_route(torch.empty(tokens, 0, dtype=torch.int64, device="cuda"), torch.empty(tokens, 0, device="cuda"), n) for _ in range(n)]
    counts = [r.send_counts.tolist() for r in routes]

    def call():
        xs, recv, out = ([torch.full((rows, hidden), 3.0, dtype=dtype, device="cuda") for _ in range(n)] for rows in (tokens, 1, tokens))
        moe.dispatch(comm, xs, recv, routes, counts)
        moe.combine(comm, recv, out, routes, counts)
        assert all(bool((o == 0).all()) for o in out) and all(bool((r == 3).all()) for r in recv)
        return out

    _both(comm, call)
    comm.close()
