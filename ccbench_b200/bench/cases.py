"""Small single-GPU cases of the hot kernels, sized for a profiler capture: inputs
larger than L2 (126 MB) but well under a few GB, a few launches, no multi-rank
process. `python -m ccbench_b200.bench.cases --case NAME [--launches 3] [--arena]`.
Ranks of one GPU run in registers; --arena asks for the kernels of ranks on several GPUs
(a phase trace does). With each case the kernel that it launches, without and with --arena:

  allreduce_int8_1rank         local_solo_kernel / solo_kernel, 128 Mi bf16
  allreduce_int8_8ranks        local_reduce_kernel (two-shot) / reduce_kernel, 16 Mi bf16 each
  allreduce_ef_int8_4ranks     local_reduce_kernel with residuals / reduce_kernel or pipe_kernel, 12.5 Mi bf16 each
  allreduce_ring_int8_8ranks   local_reduce_kernel (ring) / ring_kernel, 16 Mi bf16 each
  allreduce_pipe_int8_4ranks   pipe_kernel (warp-specialised two-shot, 1024 threads), 16 Mi bf16 each
  reducescatter_int8_8ranks    local_reduce_kernel (reduce-scatter) / reduce_kernel, 16 Mi bf16 each
  allgather_fp8_8ranks         local_exchange_kernel / exchange_kernel, 4 Mi bf16 each
  allgather_fp8_odd_8ranks     the same at odd offsets, 1,638,401 bf16 each
  moe_dispatch_fp8             moe_local_dispatch_kernel / moe_kernel, 4096 tokens x 4096 hidden bf16, 4 ranks
  moe_combine_fp8              moe_local_combine_kernel / moe_kernel, the same
  sz_compress / sz_decompress  sz_pack_kernel / sz_unpack_kernel, 384^3 fp32 field (226 MB)
  lossless_encode / lossless_decode   lossless_encode_kernel / lossless_decode_kernel, 128 Mi bf16 (256 MB)

A pattern for the profiler's -k is best anchored (regex:^reduce_kernel): local_reduce_kernel
and local_exchange_kernel hold the other kernels' names.
"""
from __future__ import annotations

import argparse
import os

import torch

from .. import Communicator
from ..models.workloads import gradient_like, moe_routing, normal, smooth_field
from ..ops import sz
from ..parallel import moe


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--case", required=True)
    ap.add_argument("--launches", type=int, default=3)
    ap.add_argument("--arena", action="store_true", help="the kernels of ranks on several GPUs, for ranks of one GPU too")
    a = ap.parse_args(argv)
    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)

    def local(n, arena_bytes):
        comm = Communicator.local(n, arena_bytes=arena_bytes)
        comm.set_trace(a.arena)
        return comm

    if a.case == "allreduce_int8_1rank":
        comm = Communicator.create(0, 1, f"case{os.getpid()}", arena_bytes=640 << 20)
        comm.set_trace(a.arena)
        x = gradient_like(128 << 20, torch.bfloat16, device=dev)
        y = torch.empty_like(x)
        for _ in range(a.launches):
            comm.all_reduce(x, y, codec="int8", algo="twoshot")
    elif a.case == "allreduce_int8_8ranks":
        n = 8
        comm = local(n, 96 << 20)
        xs = [gradient_like(16 << 20, torch.bfloat16, seed=r, device=dev) for r in range(n)]
        ys = [torch.empty_like(x) for x in xs]
        for _ in range(a.launches):
            comm.all_reduce(xs, ys, codec="int8", algo="twoshot")
    elif a.case == "allreduce_ef_int8_4ranks":
        n = 4
        comm = local(n, 96 << 20)
        xs = [gradient_like(25 << 19, torch.bfloat16, seed=r, device=dev) for r in range(n)]
        ys, es = [torch.empty_like(x) for x in xs], [torch.zeros(25 << 19, device=dev) for _ in range(n)]
        for _ in range(a.launches):
            comm.all_reduce(xs, ys, codec="int8", algo="twoshot", error_feedback=es)
    elif a.case == "reducescatter_int8_8ranks":
        n = 8
        comm = local(n, 96 << 20)
        xs = [gradient_like(16 << 20, torch.bfloat16, seed=r, device=dev) for r in range(n)]
        ys = [torch.empty(2 << 20, dtype=torch.bfloat16, device=dev) for _ in range(n)]
        for _ in range(a.launches):
            comm.reduce_scatter(xs, ys, codec="int8")
    elif a.case == "allreduce_ring_int8_8ranks":
        n = 8
        comm = local(n, 96 << 20)
        xs = [gradient_like(16 << 20, torch.bfloat16, seed=r, device=dev) for r in range(n)]
        ys = [torch.empty_like(x) for x in xs]
        for _ in range(a.launches):
            comm.all_reduce(xs, ys, codec="int8", algo="ring")
    elif a.case == "allreduce_pipe_int8_4ranks":
        n = 4
        comm = local(n, 96 << 20)
        comm.set_pipeline(2)
        xs = [gradient_like(16 << 20, torch.bfloat16, seed=r, device=dev) for r in range(n)]
        ys = [torch.empty_like(x) for x in xs]
        for _ in range(a.launches):
            comm.all_reduce(xs, ys, codec="int8", algo="twoshot")
    elif a.case in ("lossless_encode", "lossless_decode"):
        from ..ops import lossless

        x = gradient_like(128 << 20, torch.bfloat16, device=dev)
        comp = lossless.encode(x)
        out = torch.empty_like(x)
        for _ in range(a.launches):
            if a.case == "lossless_encode":
                lossless.encode(x)
            else:
                lossless.decode(comp, x.numel(), x.dtype, out=out)
    elif a.case in ("allgather_fp8_8ranks", "allgather_fp8_odd_8ranks"):
        n, count = 8, 1638401 if "odd" in a.case else 4 << 20
        comm = local(n, 96 << 20)
        xs = [normal(count, torch.bfloat16, seed=r, device=dev) for r in range(n)]
        ys = [torch.empty(n * count, dtype=torch.bfloat16, device=dev) for _ in range(n)]
        for _ in range(a.launches):
            comm.all_gather(xs, ys, codec="fp8")
    elif a.case in ("sz_compress", "sz_decompress"):
        f = smooth_field(384, device=dev)
        eb = 1e-4 * (f.max() - f.min()).item()
        buf, _ = sz.compress(f, eb)
        for _ in range(a.launches):
            if a.case == "sz_compress":
                sz.compress(f, eb)
            else:
                sz.decompress(buf, f.shape, eb)
    elif a.case in ("moe_dispatch_fp8", "moe_combine_fp8"):
        n, T, H = 4, 4096, 4096
        comm = local(n, 192 << 20)
        xs = [normal(T * H, torch.bfloat16, seed=r, device=dev).view(T, H) for r in range(n)]
        routes = [moe.plan_route(*moe_routing(T, n, 2, seed=r, device=dev), n) for r in range(n)]
        cm = [rt.send_counts.tolist() for rt in routes]
        recv = [torch.zeros(sum(cm[s][d] for s in range(n)), H, dtype=torch.bfloat16, device=dev) for d in range(n)]
        out = [torch.empty_like(x) for x in xs]
        for _ in range(a.launches):
            if a.case == "moe_dispatch_fp8":
                moe.dispatch(comm, xs, recv, routes, cm, codec="fp8")
            else:
                moe.combine(comm, recv, out, routes, cm, codec="fp8")
    else:
        raise SystemExit(f"unknown case {a.case}")
    torch.cuda.synchronize()
    print("case", a.case, "done")


if __name__ == "__main__":
    main()
