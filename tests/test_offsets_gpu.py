"""Blocks at odd offsets of a buffer, and the packed container by kernels: the addresses at
which the 32-byte accesses have to shift, rotate or give way."""
import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.ops import codecs as C
from ccbench_b200.ops import sz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("codec", ["none", "int8", "fp8"])
def test_exchange_at_every_offset_in_a_32_byte_line(dtype, codec):
    n, count = 2, 2 * 512 + 37      # two whole units, which are rotated, and a partial one
    per_line = 32 // torch.empty((), dtype=dtype).element_size()
    comm = Communicator.local(n, arena_bytes=16 << 20)
    stride = count + per_line
    xs = [torch.randn(stride * n, generator=torch.Generator().manual_seed(r)).to(dtype) for r in range(n)]
    xg = [x.cuda() for x in xs]
    for shift in range(per_line):
        send_off = [[shift + d * (count + 1) for d in range(n)] for _ in range(n)]
        recv_off = [[(per_line - shift) + s * (count + 3) for s in range(n)] for _ in range(n)]
        out = [torch.full((2 * stride + 64,), 7.0, dtype=dtype, device="cuda") for _ in range(n)]
        comm.exchange(xg, out, [[count] * n for _ in range(n)], send_off, recv_off, codec=codec)
        torch.cuda.synchronize()
        for d in range(n):
            want = torch.full((2 * stride + 64,), 7.0, dtype=dtype)
            for s in range(n):
                block = xs[s][send_off[s][d]:send_off[s][d] + count]
                want[recv_off[d][s]:recv_off[d][s] + count] = C.roundtrip(block.float(), codec, dtype).to(dtype)
            assert torch.equal(out[d].cpu(), want), (shift, d)
    comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("codec", ["none", "int8", "int4"])
@pytest.mark.parametrize("ctas", [1, 2])
def test_exchange_at_odd_offsets_over_several_tiles_a_cta(dtype, codec, ctas):
    """One or two CTAs a rank: the tile ahead is requested, shifted and stored several times, in
    blocks that differ (an all-to-all) and in one block for all (an all-gather)."""
    n, count = 3, 4 * 16 * 512 * ctas + 3 * 512 + 11
    comm = Communicator.local(n, arena_bytes=32 << 20)
    comm.set_max_ctas(ctas)
    xs = [torch.randn(n * (count + 3), generator=torch.Generator().manual_seed(r)).to(dtype) for r in range(n)]
    xg = [x.cuda() for x in xs]
    through = lambda v: C.roundtrip(v.float(), codec, dtype).to(dtype)
    for shift in (1, 3, 6):
        send_off = [[shift + d * (count + 1) for d in range(n)] for _ in range(n)]
        recv_off = [[5 - shift % 2 + s * (count + 3) for s in range(n)] for _ in range(n)]
        for off in (send_off, [[o[0]] * n for o in send_off]):
            out = [torch.full((n * (count + 3) + 16,), 7.0, dtype=dtype, device="cuda") for _ in range(n)]
            comm.exchange(xg, out, [[count] * n for _ in range(n)], off, recv_off, codec=codec)
            torch.cuda.synchronize()
            for d in range(n):
                want = torch.full(out[d].shape, 7.0, dtype=dtype)
                for s in range(n):
                    want[recv_off[d][s]:recv_off[d][s] + count] = through(xs[s][off[s][d]:off[s][d] + count])
                assert torch.equal(out[d].cpu(), want), (shift, d)
    comm.close()


def test_exchange_in_place_all_to_all_of_odd_blocks():
    n, count = 4, 3 * 512 + 1
    comm = Communicator.local(n, arena_bytes=16 << 20)
    xs = [torch.randn(n * count, generator=torch.Generator().manual_seed(r)) for r in range(n)]
    bufs = [x.cuda() for x in xs]
    comm.all_to_all(bufs, bufs, codec="none")
    torch.cuda.synchronize()
    for d in range(n):
        assert torch.equal(bufs[d].cpu(), torch.cat([x[d * count:(d + 1) * count] for x in xs]))
    comm.close()


@pytest.mark.parametrize("shape", [(1, 1, 1), (9, 7, 33), (17, 40, 130), (64, 64, 72)])
@pytest.mark.parametrize("shift", [0, 4, 8, 12])
def test_container_by_kernel_is_the_container_of_the_host_codec(shape, shift):
    g = torch.Generator().manual_seed(sum(shape))
    f = torch.randn(shape, generator=g).cumsum(2)
    eb = 1e-3
    buf, _ = sz.compress(f.cuda(), eb)
    blob = sz.to_container(buf, shape, eb)
    assert torch.equal(blob.cpu(), torch.from_numpy(sz.encode_cpu(f.numpy(), eb)))
    # a container that starts at another alignment (part of a larger message), and one on the host
    room = torch.zeros(blob.numel() + 16, dtype=torch.uint8, device="cuda")
    room[shift:shift + blob.numel()] = blob
    for view in (room[shift:shift + blob.numel()], blob.cpu()):
        again, s2, e2 = sz.from_container(view)
        assert tuple(s2) == shape and e2 == torch.tensor(eb, dtype=torch.float32).item()
        slots = buf.view(-1, sz.GROUP_STRIDE).cpu()
        for got, had in zip(again.view(-1, sz.GROUP_STRIDE).cpu(), slots):
            used = int(had[:32].view(torch.int32).sum()) + 32
            assert torch.equal(got[:used], had[:used]) and not got[used:].any()
    bad = blob.clone()
    bad[sz.HEADER_BYTES:sz.HEADER_BYTES + 4].view(torch.int32).add_(16)
    with pytest.raises(ValueError):
        sz.from_container(bad)
