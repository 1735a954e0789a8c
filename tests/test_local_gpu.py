"""Ranks that share one GPU reduce and exchange in registers; with a phase trace they take the
kernels of ranks on several GPUs. Same inputs, same bits, by both ways: every algorithm, codec and
type, sizes round the 512-element unit and the shards, residuals, operators, buffers off the 32-byte
boundaries, in place, special values. (Bits and no tolerance: both ways round at the same places and
add in the same order.)"""
import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.comm import launch_count
from ccbench_b200.parallel import moe

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16, torch.float16]
CODECS = ["none", "int8", "int8_g256", "fp8", "int4"]


def _bits(t):
    return t.view(torch.int32 if t.element_size() == 4 else torch.int16)


def _values(count, dtype, seed, shift=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(count + shift, generator=g, device="cuda").to(dtype)[shift:]
    x[::97] *= 100
    x[5::311] = 0
    return x


def _both(comm, call):
    """call() through the registers and through the arena; the outputs of each as lists of tensors."""
    got = call()
    comm.set_trace(True)
    want = call()
    comm.set_trace(False)
    torch.cuda.synchronize()
    assert comm.status()[0] == 0
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert torch.equal(_bits(a), _bits(b)), (a[_bits(a) != _bits(b)][:4], b[_bits(a) != _bits(b)][:4], int((_bits(a) != _bits(b)).sum()))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("codec", CODECS)
@pytest.mark.parametrize("algo", ["oneshot", "twoshot", "ring", "tree"])
@pytest.mark.parametrize("n", [2, 3, 5, 8])
def test_all_reduce(dtype, codec, algo, n):
    comm = Communicator.local(n, arena_bytes=64 << 20)
    for count in (1, 511, 512 * n, 512 * n + 1, 4096 * n + 700, 150_003):
        for ef in (False, True):
            xs = [_values(count, dtype, 10 * r + n) for r in range(n)]

            def call():
                res = [torch.linspace(-1, 1, count, device="cuda") * (r + 1) for r in range(n)] if ef else None
                out = [torch.empty_like(x) for x in xs]
                for _ in range(2):
                    comm.all_reduce(xs, out, codec=codec, algo=algo, error_feedback=res)
                return out + (res or [])

            _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shift", [0, 1, 8])
@pytest.mark.parametrize("algo", ["oneshot", "twoshot", "ring", "tree"])
def test_all_reduce_off_the_boundaries_and_in_place(dtype, shift, algo):
    n, count = 4, 512 * 9 + 33
    comm = Communicator.local(n, arena_bytes=16 << 20)
    for op in ("sum", "prod", "max", "min"):
        for codec in ("none", "int8") if op == "sum" else ("none",):

            def call():
                xs = [_values(count, dtype, r, shift) for r in range(n)]
                out = [torch.zeros(count + 24, dtype=dtype, device="cuda")[24 - shift:][:count] for _ in range(n)]
                comm.all_reduce(xs, out, codec=codec, algo=algo, op=op)
                comm.all_reduce(xs, codec=codec, algo=algo, op=op)   # in place
                return out + xs

            _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("codec", CODECS)
@pytest.mark.parametrize("n", [2, 3, 8])
def test_reduce_scatter_and_reduce(dtype, codec, n):
    comm = Communicator.local(n, arena_bytes=64 << 20)
    for count in (1, 15, 512, 513, 2048 + 16, 20_001, 40_960):
        for ef in (False, True):
            xs = [_values(count * n, dtype, r + n) for r in range(n)]

            def call():
                res = [torch.linspace(-1, 1, count * n, device="cuda") for _ in range(n)] if ef else None
                out = [torch.empty(count, dtype=dtype, device="cuda") for _ in range(n)]
                for _ in range(2):
                    comm.reduce_scatter(xs, out, codec=codec, error_feedback=res)
                return out + (res or [])

            _both(comm, call)

        def rooted():
            out = [torch.zeros_like(x) for x in xs]
            comm.reduce(xs, out, root=n - 1, codec=codec)
            return out

        _both(comm, rooted)

        def in_place():
            bufs = [x.clone() for x in xs]
            comm.reduce_scatter(bufs, [b[r * count:(r + 1) * count] for r, b in enumerate(bufs)], codec=codec)
            return bufs

        _both(comm, in_place)
    comm.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("codec", CODECS)
@pytest.mark.parametrize("n", [2, 3, 8])
def test_exchanges(dtype, codec, n):
    comm = Communicator.local(n, arena_bytes=128 << 20)
    for count in (1, 15, 512, 513, 3 * 512 + 16, 8 * 512 * 3 + 5, 9 * 512 * 3 + 511, 300_007):
        xs = [_values(count, dtype, r) for r in range(n)]
        many = [_values(count * n, dtype, r) for r in range(n)]
        wide = lambda: [torch.full((count * n,), 7.0, dtype=dtype, device="cuda") for _ in range(n)]
        same = lambda: [torch.full((count,), 7.0, dtype=dtype, device="cuda") for _ in range(n)]

        def call():
            ag, a2a, bc, ga, sc, ip = wide(), wide(), same(), wide(), same(), wide()
            comm.all_gather(xs, ag, codec=codec)
            comm.all_to_all(many, a2a, codec=codec)
            comm.broadcast(xs, bc, root=n - 1, codec=codec)
            comm.gather(xs, ga, root=1, codec=codec)
            comm.scatter(many, sc, root=0, codec=codec)
            for r in range(n):
                ip[r][r * count:(r + 1) * count] = xs[r]
            comm.all_gather([b[r * count:(r + 1) * count] for r, b in enumerate(ip)], ip, codec=codec)
            return ag + a2a + bc + ga + sc + ip

        _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("codec", ["none", "int8"])
def test_long_runs_at_every_offset(dtype, codec):
    """All-gathers large enough for runs of eight units, at every offset of the destinations on their
    32-byte sectors (alike on all ranks, and not), with guards around each block."""
    n, count = 2, 148 * 24 * 8 * 512 // 2 + 512 * 3 + 77   # 16 runs' worth a warp slot over the ranks
    per = 32 // torch.empty((), dtype=dtype).element_size()
    comm = Communicator.local(n, arena_bytes=256 << 20)
    xs = [_values(count, dtype, r) for r in range(n)]
    for shift in list(range(1, per)) + [0]:
        for skew in (0, 1):
            recv_off = [[shift + r * skew + q * (count + 3 + per) for q in range(n)] for r in range(n)]

            def call():
                out = [torch.full((n * (count + 8 + per) + 64,), 7.0, dtype=dtype, device="cuda") for _ in range(n)]
                comm.exchange(xs, out, [[count] * n] * n, [[0] * n] * n, recv_off, codec=codec)
                return out

            _both(comm, call)
    comm.close()


@pytest.mark.parametrize("codec", CODECS)
@pytest.mark.parametrize("algo", ["oneshot", "twoshot", "ring", "tree"])
def test_special_values(codec, algo):
    n, count = 3, 512 * 7 + 9
    comm = Communicator.local(n, arena_bytes=16 << 20)
    xs = [_values(count, torch.float32, r) for r in range(n)]
    for r, v in enumerate((float("inf"), float("nan"), -float("inf"))):
        xs[r][40 * r::701] = v
    xs[0][1300] = torch.finfo(torch.float32).max
    xs[1][1500:1700] = 1e-40   # subnormal

    def call():
        out = [torch.empty_like(x) for x in xs]
        comm.all_reduce(xs, out, codec=codec, algo=algo)
        return out

    _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("codec", CODECS)
@pytest.mark.parametrize("n,tokens,hidden,topk", [(2, 1, 512, 1), (3, 67, 1536, 2), (8, 300, 1024, 4), (4, 1100, 512, 2)])
def test_moe(dtype, codec, n, tokens, hidden, topk):
    comm = Communicator.local(n, arena_bytes=256 << 20)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    xs = [_values(tokens * hidden, dtype, r).view(tokens, hidden) for r in range(n)]
    routes = []
    for r in range(n):
        p = torch.softmax(torch.rand(tokens, 8, generator=g, device="cuda") + (torch.arange(8, device="cuda") == 2), -1)
        w, ids = torch.topk(p, topk, -1)
        routes.append(moe.plan_route(ids, w, n))
    counts = [r.send_counts.tolist() for r in routes]
    rows = [sum(counts[q][d] for q in range(n)) for d in range(n)]

    def call():
        recv = [torch.full((rows[d] + 1, hidden), 7.0, dtype=dtype, device="cuda") for d in range(n)]
        out = [torch.full((tokens, hidden), 7.0, dtype=dtype, device="cuda") for _ in range(n)]
        moe.dispatch(comm, xs, recv, routes, counts, codec=codec)
        moe.combine(comm, recv, out, routes, counts, codec=codec)
        return recv + out

    _both(comm, call)
    if rows[0] >= tokens:   # results on the rows that they come from

        def onto():
            recv = [torch.zeros(max(rows[d], 1), hidden, dtype=dtype, device="cuda") for d in range(n)]
            moe.dispatch(comm, xs, recv, routes, counts, codec=codec)
            out = [recv[0][:tokens]] + [torch.empty(tokens, hidden, dtype=dtype, device="cuda") for _ in range(n - 1)]
            moe.combine(comm, recv, out, routes, counts, codec=codec)
            return out

        _both(comm, onto)
    comm.close()


@pytest.mark.parametrize("codec", ["none", "fp8", "int4"])
@pytest.mark.parametrize("n,tokens,hidden,topk", [(2, 33, 512, 1), (4, 130, 1536, 2)])
def test_moe_with_dropped_pairs(codec, n, tokens, hidden, topk):
    """Experts that take so many pairs of each rank and no more: what is beyond is left out of perm and
    counts, and marked in pos or dest_rank."""
    keep = tokens * topk // n // 2 + 1
    comm = Communicator.local(n, arena_bytes=64 << 20)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    xs = [_values(tokens * hidden, torch.bfloat16, r).view(tokens, hidden) for r in range(n)]
    routes, counts, gates = [], [], []
    for r in range(n):
        w, ids = torch.topk(torch.softmax(torch.rand(tokens, 8, generator=g, device="cuda"), -1), topk, -1)
        full = moe.plan_route(ids, w, n)
        sent = full.send_counts.tolist()
        kept = [min(c, keep) for c in sent]
        perm = torch.cat([full.perm[sum(sent[:d]):][:kept[d]] for d in range(n)])
        dropped = full.pos >= keep
        assert dropped.any()
        pos = torch.where(dropped, torch.full_like(full.pos, -1 if r % 2 else keep), full.pos)
        dest = torch.where(dropped & (torch.arange(tokens * topk, device="cuda") % 3 == 0), torch.full_like(full.dest_rank, -1 if r % 2 else n), full.dest_rank)
        routes.append(moe.Route(perm.contiguous(), dest, pos, full.gate, torch.tensor(kept), topk))
        counts.append(kept)
        gates.append(torch.where(dropped, torch.zeros_like(full.gate), full.gate).view(tokens, topk).sum(1, keepdim=True))
    rows = [sum(counts[q][d] for q in range(n)) for d in range(n)]

    def call():
        recv = [torch.full((rows[d] + 1, hidden), 7.0, dtype=torch.bfloat16, device="cuda") for d in range(n)]
        out = [torch.full((tokens, hidden), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(n)]
        moe.dispatch(comm, xs, recv, routes, counts, codec=codec)
        moe.combine(comm, recv, out, routes, counts, codec=codec)
        if codec == "none":   # every kept copy of a token is the token; topk products and sums in fp32, one rounding to bf16
            for o, x, gate in zip(out, xs, gates):
                assert ((o.float() - x.float() * gate).abs() <= 2.0 ** -8 * (x.float() * gate).abs() + 1e-30).all()
        return recv + out

    _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("codec", ["none", "int8", "int4"])
@pytest.mark.parametrize("algo", ["oneshot", "twoshot", "ring", "tree"])
@pytest.mark.parametrize("ef", [False, True])
def test_messages_cut_to_a_small_arena(dtype, codec, algo, ef):
    """Several launches a call: the halves of the arena and the flag rows taken in turn, residuals and
    results at the slices' places. (An arena of 4 MiB, half of it for a call; these messages would need 2.8 MB and more.)"""
    n, count = 3, 4_000_003
    comm = Communicator.local(n, arena_bytes=4 << 20)
    xs = [_values(count, dtype, r + n) for r in range(n)]

    def call():
        before = launch_count()
        res = [torch.linspace(-1, 1, count, device="cuda") * (r + 1) for r in range(n)] if ef else None
        out = [torch.empty_like(x) for x in xs]
        for _ in range(2):
            comm.all_reduce(xs, out, codec=codec, algo=algo, error_feedback=res)
        assert launch_count() - before >= 4
        return out + (res or [])

    _both(comm, call)
    comm.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [2, 5])
@pytest.mark.parametrize("overlap", [False, True])
def test_one_shot_that_reads_its_own_values_again(dtype, n, overlap):
    """From 8 MiB over the ranks played a rank's own uncompressed values are read from `send` and not
    from its arena, unless another rank's result lies there."""
    count = (8 << 20) // n // torch.empty((), dtype=dtype).element_size() + 700
    comm = Communicator.local(n, arena_bytes=160 << 20)
    xs = [_values(count, dtype, r + n) for r in range(n)]

    def call():
        bufs = [x.clone() for x in xs]
        out = bufs[1:] + bufs[:1] if overlap else [torch.empty_like(x) for x in xs]
        comm.all_reduce(bufs, out, codec="none", algo="oneshot")
        return out + bufs

    _both(comm, call)
    comm.close()
