"""Ranks of one process whose buffers lie in one another: a result received into another rank's
send buffer. What a rank sends is read before its flag, what it receives is written after the
flags of the others, so these calls have one right answer."""
import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.ops import codecs as C

pytestmark = pytest.mark.gpu

COUNTS = [700, 3 * 16 * 512 + 40, 148 * 2 * 8 * 512 + 9]   # one CTA, a few, several tiles a CTA


def _inputs(n, count, dtype):
    return [torch.randn(count, generator=torch.Generator().manual_seed(r + count)).to(dtype) for r in range(n)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count", COUNTS)
@pytest.mark.parametrize("codec,algo", [("none", "oneshot"), ("int8", "oneshot"), ("none", "twoshot"), ("int8", "twoshot")])
def test_every_result_in_the_first_ranks_buffer(dtype, count, codec, algo):
    n = 3
    comm = Communicator.local(n, arena_bytes=64 << 20)
    xs = _inputs(n, count, dtype)
    want = C.simulate_all_reduce(xs, codec, algo, dtype)
    for _ in range(4):
        xg = [x.cuda() for x in xs]
        comm.all_reduce(xg, [xg[0]] * n, codec=codec, algo=algo)
        torch.cuda.synchronize()
        assert torch.equal(xg[0].float().cpu(), want)
        assert all(torch.equal(a.cpu(), b) for a, b in zip(xg[1:], xs[1:]))
    comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count", COUNTS)
@pytest.mark.parametrize("codec", ["none", "fp8"])
def test_all_to_all_into_the_next_ranks_buffer(dtype, count, codec):
    n = 4
    comm = Communicator.local(n, arena_bytes=64 << 20)
    xs = _inputs(n, n * count, dtype)
    for _ in range(4):
        xg = [x.cuda() for x in xs]
        out = xg[1:] + xg[:1]
        comm.all_to_all(xg, out, codec=codec)
        torch.cuda.synchronize()
        for d in range(n):
            want = torch.cat([C.roundtrip(x[d * count:(d + 1) * count].float(), codec, dtype).to(dtype) for x in xs])
            assert torch.equal(out[d].cpu(), want), d
    comm.close()


def test_gathered_blocks_shared_and_moved():
    n, count = 2, 5 * 512 + 3
    comm = Communicator.local(n, arena_bytes=32 << 20)
    xs = _inputs(n, count, torch.float32)
    whole = torch.zeros(n * count, device="cuda")
    for r in range(n):
        whole[r * count:(r + 1) * count] = xs[r].cuda()
    parts = list(whole.split(count))
    comm.all_gather(parts, [whole] * n, codec="int8")   # every rank gathers into the one buffer that holds the parts
    torch.cuda.synchronize()
    assert torch.equal(whole.cpu(), torch.cat([C.roundtrip(x, "int8") for x in xs]))
    # one CTA, the own block of rank 0 moved within its buffer
    buf = [torch.arange(64.0, device="cuda"), torch.arange(64.0, device="cuda") + 100]
    comm.exchange(buf, [buf[0], torch.empty(64, device="cuda")], [[32, 0], [0, 0]], [[0, 0], [0, 0]], [[16, 0], [0, 0]], codec="none")
    torch.cuda.synchronize()
    assert torch.equal(buf[0].cpu(), torch.cat([torch.arange(16.0), torch.arange(32.0), torch.arange(48.0, 64.0)]))
    comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("codec", ["int8", "fp8"])
@pytest.mark.parametrize("count", [700, 148 * 24 * 512 + 9])   # one CTA; more units than warps at once
def test_block_in_place_whose_start_is_sent_too(dtype, codec, count):
    """Every rank's own block stays where it is and goes through the codec there; the others get the
    first part of it as it was before, its last group by itself."""
    n, part = 3, count - 70
    comm = Communicator.local(n, arena_bytes=128 << 20)
    xs = _inputs(n, count, dtype)
    counts = [[count if p == r else part for p in range(n)] for r in range(n)]
    recv_off = [[0 if q == r else count + ((q - r - 1) % n) * part for q in range(n)] for r in range(n)]
    trip = lambda x: C.roundtrip(x.float(), codec, dtype).to(dtype)
    for _ in range(4):
        bufs = [torch.cat([x, torch.zeros((n - 1) * part, dtype=dtype)]).cuda() for x in xs]
        comm.exchange(bufs, bufs, counts, [[0] * n] * n, recv_off, codec=codec)
        torch.cuda.synchronize()
        for r in range(n):
            want = torch.cat([trip(xs[r])] + [trip(xs[(r + 1 + j) % n][:part]) for j in range(n - 1)])
            assert torch.equal(bufs[r].cpu(), want), r
    comm.close()
