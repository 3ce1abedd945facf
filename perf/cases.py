"""The work that users of this package have it do, as cases whose time can be measured.

Two kinds of program use the package.  One keeps a `HierarchicalEngine` and calls its
collectives; on a single GPU the rank is its own network peer, so every byte goes
device -> pinned staging -> loopback sockets -> rx page pool -> fused unpack kernel.
The other receives into a page pool of its own and calls the unpack kernels (`ops`)
on scatter lists.  Sizes are those of the benchmark, the sweeps, the DDP harness and
the tests: 1 KiB to 256 MiB per collective, one 1 MiB network request to 64 MiB per
kernel launch, odd element counts and ragged last fragments among them.
"""
import numpy as np
import torch

from nccl_plugin_gpudirecttcpx_b200 import ops
from nccl_plugin_gpudirecttcpx_b200.ops import unpack as U
from nccl_plugin_gpudirecttcpx_b200.parallel import engine as E

KIB, MIB = 1 << 10, 1 << 20
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
COLLECTIVES = ("all_reduce", "all_reduce_async", "all_gather", "reduce_scatter")


def listed():
    return [
        # the smallest collective of the sweeps (a norm, a flag, a loss value): nothing but latency
        {"name": "all_reduce_1k", "op": "all_reduce", "dtype": "bf16", "numel": 512},
        # a mid-sized gradient whose element count is odd: off the native granularity, so the binding pads it
        {"name": "all_reduce_4m_odd", "op": "all_reduce", "dtype": "bf16", "numel": (2 << 20) + 3},
        # the headline benchmark: 256 MiB of bf16 per GPU
        {"name": "all_reduce_256m", "op": "all_reduce", "dtype": "bf16", "numel": 128 << 20},
        # data-parallel training: four 25 MB fp32 gradient buckets queued in place while backward runs, then averaged
        {"name": "ddp_buckets_4x25m", "op": "all_reduce_async", "dtype": "f32", "numel": 25 * MIB // 4, "buckets": 4},
        # sharded parameters gathered before use: 16 MiB of bf16 per rank
        {"name": "all_gather_16m", "op": "all_gather", "dtype": "bf16", "numel": 8 << 20},
        # gradients of sharded parameters, fp32, an odd element count: parts off the 16-byte granularity
        {"name": "reduce_scatter_1m_odd", "op": "reduce_scatter", "dtype": "f32", "numel": (256 << 10) + 1},
        # a 64 MiB message from 4 KiB rx pages at permuted pool offsets, the last one ragged
        {"name": "unpack_copy_64m", "op": "unpack_copy", "bytes": 64 * MIB - 4096 + 2222, "frag": 4096, "pool": "hbm",
         "ctas": 0, "early": False},
        # a 4 MiB message from a NIC with standard Ethernet frames: one 1448-byte payload at the start of every page,
        # so that all but every second destination is off the 16-byte phase of its source
        {"name": "unpack_copy_4m_frames", "op": "unpack_copy", "bytes": 4 * MIB, "frag": 1448, "pool": "hbm", "ctas": 0,
         "early": False},
        # the same 64 MiB summed into a bf16 partial sum, launches chained with early start
        {"name": "unpack_reduce_64m", "op": "unpack_reduce", "dtype": "bf16", "bytes": 64 * MIB - 4096 + 2222, "frag": 4096,
         "pool": "hbm", "ctas": 0, "early": True},
        # one network request as the engine runs it: 1 MiB of fp32 out of the pinned host pool, 16 CTAs
        {"name": "unpack_reduce_1m_request", "op": "unpack_reduce", "dtype": "f32", "bytes": MIB, "frag": 4096, "pool": "host",
         "ctas": 16, "early": False},
        # the last step of a hierarchical all_reduce: 16 MiB summed and stored to three more buffers of the node
        {"name": "reduce_fanout_16m", "op": "reduce_fanout", "dtype": "bf16", "bytes": 16 * MIB, "frag": 4096, "pool": "hbm",
         "ctas": 0, "early": False, "peers": 3},
        # its first step: one GPU's shard of the work buffers of a node of four
        {"name": "peer_reduce_4x16m", "op": "peer_reduce", "dtype": "bf16", "bytes": 16 * MIB, "srcs": 4},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(("all_reduce", "all_reduce", "all_reduce_async", "all_gather", "reduce_scatter", "unpack_copy", "unpack_copy",
                     "unpack_reduce", "unpack_reduce", "reduce_fanout", "peer_reduce"))
    dtype = rng.choice(("bf16", "f32"))
    size = DTYPES[dtype].itemsize
    if op == "all_reduce_async":
        # native granularity only (32 bytes), as its contract says
        return {"op": op, "dtype": dtype, "numel": _log(rng, 64 * KIB, 25 * MIB) // 32 * 32 // size, "buckets": rng.randint(1, 4)}
    if op in COLLECTIVES:
        top = {"all_reduce": 256, "all_gather": 64, "reduce_scatter": 64}[op] * MIB
        n = _log(rng, KIB, top) // size
        return {"op": op, "dtype": dtype, "numel": n if rng.random() < 0.4 else n // 16 * 16}
    if op == "peer_reduce":
        return {"op": op, "dtype": dtype, "bytes": _log(rng, 64 * KIB, 64 * MIB) // 16 * 16, "srcs": rng.randint(2, 8)}
    pool = "host" if op == "unpack_reduce" and rng.random() < 0.4 else "hbm"
    frag = 4096 if rng.random() < 0.6 else rng.choice((1448, 2048, 3000, 4088))
    top = {"unpack_copy": 64 if frag == 4096 else 16, "unpack_reduce": 64 if frag == 4096 else 16, "reduce_fanout": 16}[op] * MIB
    if pool == "host":
        top = 4 * MIB
    c = {"op": op, "bytes": _log(rng, 64 * KIB, top), "frag": frag, "pool": pool, "ctas": 16 if pool == "host" else 0,
         "early": rng.random() < 0.3}
    if op != "unpack_copy":
        c.update(dtype=dtype, bytes=c["bytes"] // size * size)
    if op == "reduce_fanout":
        c["peers"] = rng.randint(1, 7)
    return c


_engine = None


def _the_engine():
    """One engine per process, as a program keeps it: connections and page pool are set up once."""
    global _engine
    if _engine is None:
        E.default_transport_env()
        _engine = E.HierarchicalEngine(gpus_per_node=1)
    return _engine


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    op = case["op"]
    dt = DTYPES.get(case.get("dtype"), torch.uint8)

    def normal(numel):
        return torch.randn(numel, device=dev, generator=g).to(dt)

    s = {"op": op, "buckets": case.get("buckets", 1)}
    if op in COLLECTIVES:
        s["engine"] = _the_engine()
        s["x"] = [normal(case["numel"]) for _ in range(s["buckets"])]
        s["out"] = torch.empty_like(s["x"][0]) if op == "all_reduce" else None
        return s
    total = case["bytes"]
    numel = total // dt.itemsize
    if op == "peer_reduce":
        # the shard of GPU 1: the second of `srcs` equal parts of every work buffer
        s["srcs"] = [normal(2 * numel) for _ in range(case["srcs"])]
        s["out"] = torch.empty(numel, dtype=dt, device=dev)
        s["shard_off"] = total
        return s
    # fragments of `frag` bytes, each at the start of a pool page of its own, pages in random order
    frag = case["frag"]
    n = (total + frag - 1) // frag
    pages = max(4 * n, 1024) if case["pool"] == "hbm" else 4 * n
    rng = np.random.default_rng(seed)
    lens = np.full(n, frag, dtype=np.uint64)
    lens[-1] = total - (n - 1) * frag
    descs = U.make_descriptors(rng.permutation(pages)[:n].astype(np.uint64) * 4096, lens, np.arange(n, dtype=np.uint64) * frag)
    if dt == torch.uint8:
        s["pool"] = torch.randint(0, 256, (pages * 4096,), dtype=torch.uint8, device=dev, generator=g)
    else:
        s["pool"] = normal(pages * 4096 // dt.itemsize)
    if case["pool"] == "host":
        s["pool"] = s["pool"].cpu().pin_memory()
    s["descs"] = U.descriptors_to_device(descs)
    s["dst"] = torch.empty(numel, dtype=dt, device=dev)
    s["acc"] = normal(numel) if op != "unpack_copy" else None
    s["peers"] = [torch.empty_like(s["dst"]) for _ in range(case.get("peers", 0))]
    s["status"] = U.status_buffer()
    s["opts"] = {"max_ctas": case["ctas"], "early_launch": case["early"]}
    return s


def run(s):
    op = s["op"]
    if op == "all_reduce":
        return s["engine"].all_reduce(s["x"][0], s["out"])
    if op == "all_gather":
        return s["engine"].all_gather(s["x"][0])
    if op == "reduce_scatter":
        return s["engine"].reduce_scatter(s["x"][0])
    if op == "all_reduce_async":
        # as the DDP hook does it: every bucket is queued in place, then joined and averaged over the two ranks
        works = [s["engine"].all_reduce_async(x, out=x) for x in s["x"]]
        return [w.wait().mul_(0.5) for w in works]
    if op == "peer_reduce":
        ops.peer_reduce(s["out"], s["srcs"], shard_off=s["shard_off"])
        return s["out"]
    if op == "unpack_copy":
        ops.unpack_copy(s["pool"], s["dst"], s["descs"], status=s["status"], **s["opts"])
    elif op == "unpack_reduce":
        ops.unpack_reduce(s["pool"], s["acc"], s["descs"], out=s["dst"], status=s["status"], **s["opts"])
    else:
        ops.unpack_reduce_fanout(s["pool"], s["acc"], s["dst"], s["peers"], s["descs"], status=s["status"], **s["opts"])
    return [s["dst"], s["status"]] + s["peers"]


def work(case):
    """Bytes read and written once each (scatter records included), and one add per summed element."""
    op = case["op"]
    size = DTYPES[case["dtype"]].itemsize if "dtype" in case else 1
    if op in COLLECTIVES:
        n = case["numel"] * case.get("buckets", 1)
        return {"bytes": (3 if op == "all_gather" else 2) * n * size, "flops": 0 if op == "all_gather" else n}
    if op == "peer_reduce":
        return {"bytes": (case["srcs"] + 1) * case["bytes"], "flops": (case["srcs"] - 1) * case["bytes"] // size}
    records = 16 * ((case["bytes"] + case["frag"] - 1) // case["frag"])
    copies = {"unpack_copy": 2, "unpack_reduce": 3, "reduce_fanout": 3 + case.get("peers", 0)}[op]
    return {"bytes": copies * case["bytes"] + records, "flops": 0 if op == "unpack_copy" else case["bytes"] // size}


def tolerance(case):
    """Bytes that are only moved stay the same.  A sum of two values has one correctly rounded result, so every
    implementation gives the same one.  More sources can be added in another order: one rounding of bf16 (2^-9 relative
    at most) may fall the other way, and fp32 sums differ in their last bits."""
    if case["op"] != "peer_reduce" or case["srcs"] == 2:
        return "exact"
    return {"rel": 2.0 ** -9} if case["dtype"] == "bf16" else {"rel": 1e-6}
