"""MoE dispatch / combine: routed token exchange with per-destination compression,
all ranks played on one GPU, against a plain torch restatement."""
import pytest
import torch

from ccbench_b200 import Communicator
from ccbench_b200.models.workloads import moe_routing
from ccbench_b200.ops import codecs as C
from ccbench_b200.parallel import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("codec", ["fp8", "none", "int8"])
@pytest.mark.parametrize("n,T,H", [(4, 300, 1024), (8, 256, 512), (2, 77, 2048)])
def test_dispatch_then_combine(codec, n, T, H):
    comm = Communicator.local(n, arena_bytes=64 << 20)
    try:
        dt = torch.bfloat16
        xs = [torch.randn(T, H, generator=torch.Generator().manual_seed(r)).to(dt) for r in range(n)]
        routes_cpu = []
        for r in range(n):
            ids, gates = moe_routing(T, n, 2, seed=r)
            routes_cpu.append(moe.plan_route(ids, gates, n))
        cm = [rt.send_counts.tolist() for rt in routes_cpu]
        to_dev = lambda rt: moe.Route(rt.perm.cuda(), rt.dest_rank.cuda(), rt.pos.cuda(), rt.gate.cuda(), rt.send_counts, rt.topk)
        routes = [to_dev(rt) for rt in routes_cpu]
        xg = [x.cuda() for x in xs]
        rows_in = [sum(cm[s][d] for s in range(n)) for d in range(n)]
        recv = [torch.zeros(max(rows_in[d], 1), H, dtype=dt, device="cuda") for d in range(n)]
        for _ in range(2):
            moe.dispatch(comm, xg, recv, routes, cm, codec=codec)
        torch.cuda.synchronize()
        assert comm.status()[0] == 0
        rt_ = lambda v: C.roundtrip(v.float(), codec, dt).to(dt)
        for d in range(n):
            want = []
            for s in range(n):
                rtc = routes_cpu[s]
                start = sum(cm[s][:d])
                rows = rtc.perm[start:start + cm[s][d]].long()
                want.append(rt_(xs[s][rows]).reshape(-1, H))
            want = torch.cat(want) if want else torch.zeros(0, H, dtype=dt)
            assert torch.equal(recv[d][:rows_in[d]].cpu(), want)
        # experts scale their inputs; combine brings them back gate-weighted
        ys = [(recv[d].float() * (d + 1)).to(dt) for d in range(n)]
        out = [torch.zeros(T, H, dtype=dt, device="cuda") for _ in range(n)]
        moe.combine(comm, ys, out, routes, cm, codec=codec)
        torch.cuda.synchronize()
        assert comm.status()[0] == 0
        for s in range(n):
            rtc = routes_cpu[s]
            acc = torch.zeros(T, H)
            for pair in range(T * 2):
                t, d, j = pair // 2, int(rtc.dest_rank[pair]), int(rtc.pos[pair])
                row0 = sum(cm[q][d] for q in range(s))
                acc[t] += rtc.gate[pair] * rt_(ys[d][row0 + j].cpu()).float()
            got = out[s].float().cpu()
            assert (got - acc).abs().max().item() <= 2.0 ** -7 * acc.abs().max().item() + 1e-6
    finally:
        comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("codec", ["none", "int8", "fp8", "int4"])
@pytest.mark.parametrize("topk,ctas", [(1, 1), (3, 2), (4, 0)])
def test_every_topk_over_several_turns(dtype, codec, topk, ctas):
    """One or two CTAs a rank: the loops that request a unit ahead go round many times."""
    n, T, H = 4, 150, 1536
    comm = Communicator.local(n, arena_bytes=48 << 20)
    try:
        if ctas:
            comm.set_max_ctas(ctas)
        xs = [(torch.randn(T, H, generator=torch.Generator().manual_seed(r)) * 2).to(dtype) for r in range(n)]
        cpu = [moe.plan_route(*moe_routing(T, n, topk, seed=10 + r), n) for r in range(n)]
        cm = [rt.send_counts.tolist() for rt in cpu]
        routes = [moe.Route(rt.perm.cuda(), rt.dest_rank.cuda(), rt.pos.cuda(), rt.gate.cuda(), rt.send_counts, rt.topk) for rt in cpu]
        rows_in = [sum(cm[s][d] for s in range(n)) for d in range(n)]
        recv = [torch.zeros(max(k, 1), H, dtype=dtype, device="cuda") for k in rows_in]
        moe.dispatch(comm, [x.cuda() for x in xs], recv, routes, cm, codec=codec)
        torch.cuda.synchronize()
        through = lambda v: C.roundtrip(v.float(), codec, dtype).reshape(-1, H)
        for d in range(n):
            want = [through(xs[s][cpu[s].perm[sum(cm[s][:d]):sum(cm[s][:d + 1])].long()]) for s in range(n)]
            assert torch.equal(recv[d][:rows_in[d]].cpu(), torch.cat(want).to(dtype)), d
        out = [torch.zeros(T, H, dtype=dtype, device="cuda") for _ in range(n)]
        moe.combine(comm, recv, out, routes, cm, codec=codec)
        torch.cuda.synchronize()
        assert comm.status()[0] == 0
        wire = [through(recv[d].cpu()).double() for d in range(n)]
        half_ulp = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
        for s in range(n):
            acc, size = torch.zeros(T, H, dtype=torch.float64), torch.zeros(T, H, dtype=torch.float64)
            row = torch.tensor([sum(cm[q][d] for q in range(s)) for d in range(n)])[cpu[s].dest_rank.long()] + cpu[s].pos.long()
            for k in range(topk):
                pair = torch.arange(T) * topk + k
                d = torch.stack([wire[int(cpu[s].dest_rank[i])][int(row[i])] for i in pair]) * cpu[s].gate[pair].double().unsqueeze(1)
                acc += d
                size += d.abs()
            # one rounding of fp32 for each of the topk sums, then one to the output's type (fp16: or to its smallest step)
            bound = (topk + 1) * 2.0 ** -24 * size + half_ulp * acc.abs() * 1.001 + 2.0 ** -25
            assert ((out[s].cpu().double() - acc).abs() <= bound).all()
    finally:
        comm.close()
