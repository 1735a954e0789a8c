"""The work that programs have this framework do on one GPU, as a list of timed cases.

A case names a kind of call, its sizes and its options; `prepare` makes what the calling
program holds (buffers, a communicator, a routing plan), `run` is one pass through the
package's public entry points, and `exact` says in 64-bit torch what the pass approximates.
Collectives run with all their ranks on the one GPU (`Communicator.local`), or with a single
rank (`Communicator.create`), which is what a one-GPU box offers.
"""
import math
import uuid

import torch

from ccbench_b200 import Communicator
from ccbench_b200.ops import lossless, standalone, sz
from ccbench_b200.parallel import moe

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
MiB = 1 << 20


# ------------------------------------------------------------------------------- cases --
def listed():
    return [
        # A small all-reduce (norms, loss scalars, a last short bucket): latency and launches.
        {"name": "ar_small", "kind": "all_reduce", "ranks": 8, "count": 4096, "dtype": "bf16", "codec": "int8", "algo": "auto", "ef": False},
        # The benchmark's default message, 256 MiB of bf16 gradients, as a one-rank job runs it.
        {"name": "ar_256MiB_one_rank", "kind": "all_reduce", "ranks": 1, "count": 128 * MiB, "dtype": "bf16", "codec": "int8", "algo": "twoshot", "ef": False},
        # One 25 MiB gradient bucket of data-parallel training with error feedback: the comm hook's call.
        {"name": "ar_bucket_ef", "kind": "all_reduce", "ranks": 4, "count": 25 * MiB // 2, "dtype": "bf16", "codec": "int8", "algo": "auto", "ef": True},
        # The ring with per-hop fp8 requantisation, on gradients of 64 MiB a rank.
        {"name": "ar_ring_fp8", "kind": "all_reduce", "ranks": 4, "count": 32 * MiB, "dtype": "bf16", "codec": "fp8", "algo": "ring", "ef": False},
        # The uncompressed baseline on fp32 data, of an odd element count.
        {"name": "ar_plain_f32_odd", "kind": "all_reduce", "ranks": 2, "count": 5000011, "dtype": "f32", "codec": "none", "algo": "auto", "ef": False},
        # ZeRO: a 25 MiB gradient bucket reduced to its owners.
        {"name": "rs_bucket", "kind": "reduce_scatter", "ranks": 8, "count": 25 * MiB // 2 // 8, "dtype": "bf16", "codec": "int8"},
        # FSDP / ZeRO-3: updated parameter shards gathered in fp8; a shard that is no multiple of a tile.
        {"name": "ag_params_fp8", "kind": "all_gather", "ranks": 8, "count": 1638401, "dtype": "bf16", "codec": "fp8"},
        # Expert parallelism: top-2 of 8 experts, 8192 tokens of 4096 a rank, fp8 rows out and back.
        {"name": "moe_8192x4096", "kind": "moe", "ranks": 8, "tokens": 8192, "hidden": 4096, "topk": 2, "dtype": "bf16", "codec": "fp8"},
        # The compression hooks' sequence on a chunk of fp32 values from three ranks:
        # compress each, decode + add + re-encode, decompress.
        {"name": "hooks_f32_int8", "kind": "hooks", "inputs": 3, "count": 3000001, "dtype": "f32", "codec": "int8"},
        # A 512^3 simulation field through the error-bounded codec and back.
        {"name": "sz_512", "kind": "sz", "nz": 512, "ny": 512, "nx": 512, "rel_eb": 1e-4},
        # A smaller field of ragged extents through the container that is stored or sent, and back.
        {"name": "sz_store_ragged", "kind": "sz_store", "nz": 130, "ny": 201, "nx": 258, "rel_eb": 1e-4},
        # Gradients through the lossless float codec and back, 64 MiB of bf16.
        {"name": "lossless_bf16", "kind": "lossless", "count": 32 * MiB, "dtype": "bf16"},
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    how = rng.random()   # half of the sizes as they come, the rest on the boundaries that programs pad to
    return n if how < 0.5 else max(lo, n // 512 * 512) if how < 0.8 else max(lo, n // 16 * 16)


def draw(rng):
    kind = rng.choice(["all_reduce", "all_reduce", "all_reduce", "reduce_scatter", "all_gather", "moe", "hooks", "sz", "sz_store", "lossless"])
    codec = rng.choice(["int8", "int8", "fp8", "none", "int8_g256", "int4"])
    dtype = rng.choice(["bf16", "bf16", "f32", "f16"])
    ranks = rng.choice([2, 4, 8])
    if kind == "all_reduce":
        ranks = rng.choice([1, 2, 3, 4, 8])
        algo = rng.choice(["auto", "auto", "twoshot", "ring", "tree"])
        return {"kind": kind, "ranks": ranks, "count": _size(rng, 512, 64 * MiB // ranks), "dtype": dtype, "codec": codec, "algo": algo,
                "ef": codec != "none" and rng.random() < 0.4}
    if kind in ("reduce_scatter", "all_gather"):
        return {"kind": kind, "ranks": ranks, "count": _size(rng, 256, 64 * MiB // ranks // ranks), "dtype": dtype, "codec": codec}
    if kind == "moe":
        return {"kind": kind, "ranks": ranks, "tokens": _size(rng, 16, 4096), "hidden": 512 * rng.randint(1, 8), "topk": rng.choice([1, 2, 2, 4]),
                "dtype": dtype, "codec": codec}
    if kind == "hooks":
        return {"kind": kind, "inputs": rng.randint(2, 8), "count": _size(rng, 1024, 16 * MiB), "dtype": "f32", "codec": rng.choice(["int8", "int8_g256", "fp8", "int4"])}
    if kind == "sz":
        return {"kind": kind, "nz": _size(rng, 8, 400), "ny": _size(rng, 16, 400), "nx": _size(rng, 32, 400), "rel_eb": rng.choice([1e-4, 1e-4, 1e-3, 1e-2, 1e-5])}
    if kind == "sz_store":
        return {"kind": kind, "nz": _size(rng, 8, 200), "ny": _size(rng, 16, 250), "nx": _size(rng, 32, 250), "rel_eb": rng.choice([1e-4, 1e-3])}
    return {"kind": kind, "count": _size(rng, 1024, 32 * MiB), "dtype": dtype}


# ------------------------------------------------------------------------------ inputs --
def _gen(seed, k):
    return torch.Generator(device="cuda").manual_seed(1000003 * (int(seed) + 1) + k)


def _gradients(count, dtype, g):
    """Laplace(0, 1e-3) values, one in a thousand of them a hundred times larger."""
    out = torch.empty(count, dtype=DTYPES[dtype], device="cuda")
    step = 1 << 25
    for lo in range(0, count, step):
        n = min(step, count - lo)
        u = torch.rand(n, generator=g, device="cuda") - 0.5
        v = -1e-3 * torch.sign(u) * torch.log1p(-2 * u.abs().clamp_(max=0.4999999))
        far = torch.rand(n, generator=g, device="cuda") < 1e-3
        out[lo:lo + n] = torch.where(far, v * 100, v).to(out.dtype)
    return out


def _field(case, seed):
    """64 Gaussian bumps (widths 8 to 64 in 512 of an axis, amplitudes N(0, 1)) and white noise of 1e-3."""
    g = _gen(seed, 7)
    r = torch.rand(64, 4, generator=g, device="cuda")
    amp = torch.randn(64, generator=g, device="cuda")
    line = []
    for i, n in enumerate((case["nz"], case["ny"], case["nx"])):
        at = torch.arange(n, device="cuda", dtype=torch.float32)
        line.append(torch.exp(-0.5 * ((at[None] / n - r[:, i:i + 1]) * 512 / (8 + 56 * r[:, 3:])) ** 2))
    plane = (amp[:, None, None] * line[0][:, :, None] * line[1][:, None, :]).reshape(64, -1)
    f = (plane.T @ line[2]).reshape(case["nz"], case["ny"], case["nx"])
    f += 1e-3 * torch.randn(f.shape, generator=g, device="cuda")
    return f.contiguous()


def _inputs(case, seed):
    kind = case["kind"]
    if kind in ("all_reduce", "reduce_scatter", "all_gather"):
        n = case["ranks"]
        count = case["count"] * (n if kind == "reduce_scatter" else 1)
        return [_gradients(count, case["dtype"], _gen(seed, r)) for r in range(n)]
    if kind == "hooks":
        return [_gradients(case["count"], "f32", _gen(seed, r)) for r in range(case["inputs"])]
    if kind == "lossless":
        return _gradients(case["count"], case["dtype"], _gen(seed, 0))
    if kind in ("sz", "sz_store"):
        return _field(case, seed)
    x, ids, gates = [], [], []
    for r in range(case["ranks"]):
        g = _gen(seed, r)
        x.append(torch.randn(case["tokens"], case["hidden"], generator=g, device="cuda").to(DTYPES[case["dtype"]]))
        p = torch.softmax(torch.rand(case["tokens"], 8, generator=g, device="cuda"), dim=-1)
        w, i = torch.topk(p, case["topk"], dim=-1)
        ids.append(i)
        gates.append((w / w.sum(-1, keepdim=True)).float())
    return x, ids, gates


def _error_bound(case, field):
    return case["rel_eb"] * float(field.max() - field.min())


def _communicator(case, half_bytes):
    """A communicator whose arenas hold two staging halves of `half_bytes`."""
    arena = 2 * int(half_bytes) + 16 * MiB
    if case["ranks"] == 1:
        return Communicator.create(0, 1, uuid.uuid4().hex[:16], arena_bytes=arena)
    return Communicator.local(case["ranks"], arena_bytes=arena)


def _capacity(case):
    """Rows that an expert's receive buffer holds: the mean and eight standard deviations. The rows beyond those sent stay zero."""
    mean = case["tokens"] * case["topk"]
    return int(mean + 8 * math.sqrt(mean) + 64)


def prepare(case, seed):
    kind, data = case["kind"], _inputs(case, seed)
    s = {"case": case, "in": data}
    if kind == "all_reduce":
        n, esz = case["ranks"], data[0].element_size()
        # the tree keeps a slot of the whole message for each level, the others a shard for each rank and phase
        s["comm"] = _communicator(case, (case["count"] + 1024 * n) * esz * 1.1 * 5 + MiB)
        s["out"] = [torch.empty_like(x) for x in data]
        s["ef"] = [torch.zeros(case["count"], device="cuda") for _ in data] if case["ef"] else None
    elif kind == "reduce_scatter":
        s["comm"] = _communicator(case, (case["count"] + 1024) * case["ranks"] * data[0].element_size() * 1.1 + MiB)
        s["out"] = [torch.empty(case["count"], dtype=x.dtype, device="cuda") for x in data]
    elif kind == "all_gather":
        s["comm"] = _communicator(case, (case["count"] + 1024) * case["ranks"] * data[0].element_size() * 1.1 + MiB)
        s["out"] = [torch.empty(case["count"] * case["ranks"], dtype=x.dtype, device="cuda") for x in data]
    elif kind == "moe":
        x, ids, gates = data
        n, h, dt = case["ranks"], case["hidden"], x[0].dtype
        s["routes"] = [moe.plan_route(ids[r], gates[r], n) for r in range(n)]
        s["counts"] = [r.send_counts.tolist() for r in s["routes"]]
        most = max(max(row) for row in s["counts"])
        s["comm"] = _communicator(case, (most + 2) * h * x[0].element_size() * 1.1 * n + MiB)
        s["rows"] = [torch.zeros(_capacity(case), h, dtype=dt, device="cuda") for _ in range(n)]
        assert all(sum(s["counts"][q][d] for q in range(n)) <= _capacity(case) for d in range(n))
        s["out"] = [torch.empty_like(t) for t in x]
    elif kind in ("sz", "sz_store"):
        s["eb"] = _error_bound(case, data)
    return s


def run(s):
    case, data = s["case"], s["in"]
    kind = case["kind"]
    if kind == "all_reduce":
        one = case["ranks"] == 1
        s["comm"].all_reduce(data[0] if one else data, s["out"][0] if one else s["out"], codec=case["codec"], algo=case["algo"], error_feedback=s["ef"])
        return {"out": s["out"], "ef": s["ef"]} if case["ef"] else {"out": s["out"]}
    if kind == "reduce_scatter":
        return {"out": s["comm"].reduce_scatter(data, s["out"], codec=case["codec"])}
    if kind == "all_gather":
        return {"out": s["comm"].all_gather(data, s["out"], codec=case["codec"])}
    if kind == "moe":
        moe.dispatch(s["comm"], data[0], s["rows"], s["routes"], s["counts"], codec=case["codec"])
        moe.combine(s["comm"], s["rows"], s["out"], s["routes"], s["counts"], codec=case["codec"])
        return {"rows": s["rows"], "out": s["out"]}
    if kind == "hooks":
        wires = [standalone.encode(x, case["codec"]) for x in data]
        total = standalone.reduce_recode(wires, case["codec"], case["count"])
        return {"out": standalone.decode(total, case["codec"], case["count"], data[0].dtype)}
    if kind == "sz":
        packed, used = sz.compress(data, s["eb"])
        return {"used": used, "out": sz.decompress(packed, data.shape, s["eb"])}
    if kind == "sz_store":
        packed, _ = sz.compress(data, s["eb"])
        blob = sz.to_container(packed, data.shape, s["eb"])
        packed, shape, eb = sz.from_container(blob)
        return {"bytes": blob.numel(), "out": sz.decompress(packed, shape, eb)}
    return {"out": lossless.decode(lossless.encode(data), case["count"], data.dtype)}


# ------------------------------------------------------------------------- what it costs --
def work(case):
    """Each input read once and each output written once; what travels compressed counts as
    written and read once at its wire size where the caller receives it between two calls."""
    kind = case["kind"]
    esz = torch.empty((), dtype=DTYPES[case.get("dtype", "f32")]).element_size()
    wire = {"none": esz, "int8": 1 + 4 / 128, "int8_g256": 1 + 4 / 256, "fp8": 1 + 1 / 32, "int4": 0.5 + 4 / 128}.get(case.get("codec"), 0)
    if kind == "all_reduce":
        each = case["count"] * case["ranks"]
        return {"bytes": each * (2 * esz + (8 if case["ef"] else 0)), "flops": each}
    if kind in ("reduce_scatter", "all_gather"):
        small, n = case["count"] * case["ranks"], case["ranks"]
        return {"bytes": (small + small * n) * esz, "flops": small * n}
    if kind == "moe":
        rows = case["ranks"] * case["tokens"] * case["hidden"]
        return {"bytes": rows * esz * (2 + 2 * case["topk"]), "flops": rows * 2 * case["topk"]}
    if kind == "hooks":
        n = case["inputs"]
        return {"bytes": case["count"] * (n * (esz + 2 * wire) + 2 * wire + esz), "flops": case["count"] * n}
    if kind in ("sz", "sz_store"):
        values = case["nz"] * case["ny"] * case["nx"]
        # a byte a value is what the packed field comes to at these bounds, more or less; it is
        # written and read once, and copied once into and once out of a container
        return {"bytes": values * (4 + 1 + (5 if kind == "sz" else 7)), "flops": values * 8}
    packed = {2: 1.5, 4: 3.5}[esz]
    return {"bytes": case["count"] * 2 * (esz + packed), "flops": case["count"]}


def tolerance(case):
    """Bytes and codes that are written down by rule are the same everywhere. A sum over ranks
    taken in another order, or with a fused multiply-add, moves a value across a rounding
    boundary now and then, by one step of its codec or type. Measured against 64-bit sums
    between the roundings, two to eight ranks: int8 up to 1.1e-4, fp8 up to 1.1e-4, int4 up to
    2.6e-4, uncompressed fp32 1.7e-7, uncompressed 16-bit types (the ring rounds at each hop)
    1.3e-4. An all-gather has no sums, only the decoder's product; a combine has two to four."""
    kind = case["kind"]
    if kind in ("sz", "sz_store", "lossless"):
        return "exact"
    if kind == "all_gather":
        return {"rel": 1e-6}
    if kind == "moe":
        return {"rel": 1e-4}
    if case["codec"] == "none":
        return {"rel": 1e-6 if case["dtype"] == "f32" else 5e-4}
    return {"rel": 1e-3 if case["codec"] == "int4" else 4e-4}


def exact(case, seed):
    kind, data = case["kind"], _inputs(case, seed)
    if kind == "all_reduce":
        total = data[0].double()
        for x in data[1:]:
            total += x
        out = {"out": [total] * case["ranks"]}
        if case["ef"]:
            out["ef"] = [None] * case["ranks"]   # the quantisation error itself
        return out
    if kind == "reduce_scatter":
        total = data[0].double()
        for x in data[1:]:
            total += x
        return {"out": list(total.split(case["count"]))}
    if kind == "all_gather":
        return {"out": [torch.cat([x.double() for x in data])] * case["ranks"]}
    if kind == "moe":
        x, ids, gates = data
        n = case["ranks"]
        rows = [[] for _ in range(n)]
        for r in range(n):
            dest = ids[r].reshape(-1) % n
            for d in range(n):
                rows[d].append(x[r][(dest == d).nonzero().reshape(-1) // case["topk"]])
        rows = [torch.cat(v).double() for v in rows]
        rows = [torch.cat([v, v.new_zeros(_capacity(case) - v.shape[0], v.shape[1])]) for v in rows]
        return {"rows": rows, "out": [t.double() * g.double().sum(1, keepdim=True) for t, g in zip(x, gates)]}
    if kind == "hooks":
        return {"out": sum(x.double() for x in data)}
    if kind == "lossless":
        return {"out": data.double()}
    return {"used" if kind == "sz" else "bytes": None, "out": data.double()}
