"""An all-reduce of one rank (its own kernel) against the restated algorithms: partial and whole
units, more units than resident warps, views at odd offsets, with and without error feedback."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.ops import codecs as C

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    c = Communicator.create(0, 1, f"solo{os.getpid()}", arena_bytes=32 << 20)
    yield c
    c.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("codec", ["int8", "int8_g256", "fp8", "int4", "none"])
@pytest.mark.parametrize("count", [1, 511, 512, 4096 + 17, 148 * 5 * 8 * 512 + 512 * 3 + 5])
def test_one_rank_matches_the_restatement(comm, dtype, codec, count):
    x = (torch.randn(count + 3, generator=torch.Generator().manual_seed(count)) * 3).to(dtype)
    xg = x.cuda()
    for algo, shift in (("twoshot", 0), ("oneshot", 1), ("ring", 0), ("tree", 3)):
        send = xg[shift:shift + count]
        out = torch.zeros(count + 2, dtype=dtype, device="cuda")
        comm.all_reduce(send, out[1:1 + count], codec=codec, algo=algo)
        torch.cuda.synchronize()
        want = C.simulate_all_reduce([x[shift:shift + count]], codec, algo, dtype)
        assert torch.equal(out[1:1 + count].float().cpu(), want), (algo, shift)
        assert out[0] == 0 and out[-1] == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("codec", ["int8", "fp8"])
def test_one_rank_error_feedback_in_place(comm, dtype, codec):
    count = 3 * 512 + 40
    x = torch.randn(count, generator=torch.Generator().manual_seed(5)).to(dtype)
    buf, ef = x.cuda(), torch.zeros(count, device="cuda")
    want_ef = [torch.zeros(count)]
    for _ in range(3):
        buf.copy_(x)
        comm.all_reduce(buf, codec=codec, error_feedback=ef)
        want = C.simulate_all_reduce([x], codec, "twoshot", dtype, ef=want_ef)
        torch.cuda.synchronize()
        assert torch.equal(buf.float().cpu(), want)
        assert torch.equal(ef.cpu(), want_ef[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("codec", ["int8", "fp8", "none"])
@pytest.mark.parametrize("cap", [1, 3, 148, 149])
@pytest.mark.parametrize("with_ef", [False, True])
def test_one_rank_under_a_grid_cap(comm, dtype, codec, cap, with_ef):
    """Several turns of the look-ahead loop in both CTA sizes (512 threads up to a CTA an SM, else
    256), in place, the last unit partial."""
    count = (3 if cap < 100 else 2) * cap * 16 * 512 + 5 * 512 + 21
    x = (torch.randn(count, generator=torch.Generator().manual_seed(cap)) * 3).to(dtype)
    ef = torch.zeros(count, device="cuda") if with_ef else None
    want_ef = [torch.zeros(count)] if with_ef else None
    buf = torch.zeros(count + 1, dtype=dtype, device="cuda")[1:]
    comm.set_max_ctas(cap)
    try:
        for _ in range(2 if with_ef else 1):
            buf.copy_(x)
            comm.all_reduce(buf, codec=codec, algo="twoshot", error_feedback=ef)
            torch.cuda.synchronize()
            assert torch.equal(buf.float().cpu(), C.simulate_all_reduce([x], codec, "twoshot", dtype, ef=want_ef))
            assert not with_ef or torch.equal(ef.cpu(), want_ef[0])
    finally:
        comm.set_max_ctas(0)


@pytest.mark.parametrize("algo", ["auto", "twoshot"])
@pytest.mark.parametrize("count,ef", [(100, False), (8 << 20, False), (8 << 20, True)])
def test_one_rank_trace(comm, algo, count, ef):
    x = torch.randn(count, device="cuda")
    res = torch.zeros(count, device="cuda") if ef else None
    comm.set_trace(True)
    try:
        comm.all_reduce(x, torch.empty_like(x), codec="int8", algo=algo, error_feedback=res)
        torch.cuda.synchronize()
        tr = comm.read_trace(1024)
    finally:
        comm.set_trace(False)
    tr = tr[tr[:, 0] > 0]
    assert 1 <= tr.shape[0] <= -(-count // 4096)
    assert (tr[:, 0] <= tr[:, 1]).all()
    assert (tr[:, 1] <= tr[:, 2]).all() and (tr[:, 2] <= tr[:, 3]).all() and (tr[:, 3] <= tr[:, 4]).all()
    assert int(tr[:, 4].max() - tr[:, 0].min()) < 1_000_000_000


def test_phase_timeline_of_one_rank():
    env = {k: v for k, v in os.environ.items() if k not in ("WORLD_SIZE", "RANK", "LOCAL_RANK")}
    out = subprocess.run([sys.executable, "-m", "ccbench_b200.bench.phases", "--what", "allreduce"], capture_output=True, text=True, timeout=300,
                         env=env, cwd=Path(__file__).resolve().parent.parent)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.count("mark 4") == 3
