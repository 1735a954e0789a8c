"""Launches that are got ready while the kernel before them runs: a chain in which every kernel reads what the one
before it wrote, ours and torch's in turn, on the default stream, on another, and as a graph."""
import ctypes

import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.ops import lossless, standalone, sz

pytestmark = pytest.mark.gpu


def _chain(comm, x, wait):
    out = []
    for k in range(6):
        x = standalone.decode(standalone.encode(x, ("int8", "fp8", "int4")[k % 3]), ("int8", "fp8", "int4")[k % 3], x.numel(), x.dtype)
        wait()
        ys = [torch.empty_like(x) for _ in range(2)]
        comm.all_reduce([x, x.flip(0)], ys, codec="int8")
        wait()
        x = ys[1] * 0.5
        wait()
        x = lossless.decode(lossless.encode(x), x.numel(), x.dtype)
        wait()
        f = x[:x.numel() // 2048 * 2048].view(-1, 32, 64)
        packed, used = sz.compress(f, 1e-3)
        wait()
        f = sz.decompress(packed, f.shape, 1e-3)
        wait()
        x = torch.cat([f.reshape(-1), x[f.numel():]])
        out += [x, used]
    return out


@pytest.mark.parametrize("count", [5_000, 300_001, 6_000_003])
def test_a_chain_waits_for_what_it_reads(count):
    comm = Communicator.local(2, arena_bytes=64 << 20)
    x = torch.randn(count, generator=torch.Generator(device="cuda").manual_seed(count), device="cuda")
    want = _chain(comm, x, torch.cuda.synchronize)
    side = torch.cuda.Stream()
    for _ in range(5):
        for stream in (torch.cuda.current_stream(), side):
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                got = _chain(comm, x, lambda: None)
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _chain(comm, x, lambda: None)
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    del graph
    comm.close()


def test_a_call_behind_a_capped_one_leaves_the_other_sms_free():
    """What is launched behind a collective of a few CTAs does not wait on the SMs that the cap leaves to other streams."""
    comm, behind = Communicator.local(2, arena_bytes=1 << 30), Communicator.local(2, arena_bytes=32 << 20)
    comm.set_pipeline(2)
    comm.set_max_ctas(4)
    xs = [torch.randn(48 << 20, device="cuda").bfloat16() for _ in range(2)]
    ys, zs = [torch.empty_like(x) for x in xs], [torch.empty_like(x) for x in xs]
    small = torch.zeros(1 << 16, device="cuda")
    other = torch.cuda.Stream()
    for _ in range(3):   # once to load the kernels
        torch.cuda.synchronize()
        start, done, end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        start.record()
        comm.all_reduce(xs, ys)
        behind.all_reduce(xs, zs)   # more CTAs than fit
        with torch.cuda.stream(other):
            small += 1
            done.record()
        end.record()
        torch.cuda.synchronize()
    assert start.elapsed_time(end) > 1.0
    assert start.elapsed_time(done) < 0.5 * start.elapsed_time(end)
    comm.close()
    behind.close()


@pytest.mark.parametrize("blocking", [False, True])
def test_a_launch_waits_for_other_streams_that_its_own_waits_for(blocking):
    """A kernel of ours, a long one of another stream behind it, and ours again, which reads what that wrote: ordered by an
    event, or by the default stream's own rule for streams that block."""
    stream, other = torch.cuda.current_stream(), torch.cuda.Stream()
    if blocking:   # torch's own do not
        made = ctypes.c_void_p()
        assert ctypes.CDLL("libcudart.so.12").cudaStreamCreate(ctypes.byref(made)) == 0
        other = torch.cuda.ExternalStream(made.value)
    x = torch.zeros(1 << 20, device="cuda")
    want = standalone.encode(torch.full_like(x, 7.0), "int8")
    for _ in range(3):
        x.zero_()
        before = standalone.encode(x, "int8")
        if not blocking:
            other.wait_stream(stream)
        with torch.cuda.stream(other):
            torch.cuda._sleep(20_000_000)   # some 10 ms
            x.fill_(7.0)
        if not blocking:
            stream.wait_stream(other)
        got = standalone.encode(x, "int8")
        torch.cuda.synchronize()
        assert torch.equal(got, want) and not torch.equal(before, want)
