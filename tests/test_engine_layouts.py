"""Tensors the native calls cannot take as they are (strides, an output of another type, too small, or overlapping the
input) at sizes that are whole multiples of every granularity, where no padding hides them.  Stand-in device, gloo ranks."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from conftest import free_port

HERE = Path(__file__).resolve().parent

WORKER = r"""
import os, sys
sys.path[:0] = [sys.argv[1], os.path.dirname(sys.argv[1])]
import torch
import torch.distributed as dist
world, G = int(os.environ.get("WORLD_SIZE", "1")), int(sys.argv[2])
if world > 1:
    dist.init_process_group("gloo")
rank = dist.get_rank() if world > 1 else 0
from nccl_plugin_gpudirecttcpx_b200.parallel.engine import default_transport_env
from standin_engine import StandinEngine
default_transport_env(nics=2, nthreads=2, pool_mb=64)
eng = StandinEngine(gpus_per_node=G, request_bytes=256 << 10, buffer_bytes=1 << 22 if G > 1 else 0, plain_mode=len(sys.argv) > 3)
ranks = max(2, world)
rows = 12  # divides into the parts of every layout here
for cols in (16, 1024):
    ins = [torch.randint(-64, 64, (rows, cols), generator=torch.Generator().manual_seed(s)).float() for s in range(ranks if world > 1 else 1)]
    ins = ins if world > 1 else ins * 2  # a single rank is its own twin
    total = sum(ins)
    a = ins[rank]
    strided = a.t().contiguous().t()  # the same values in another memory order
    assert not strided.is_contiguous()
    mine = a if rank % 2 else strided  # ranks differ in their layouts
    assert torch.equal(eng.all_reduce(mine), total)
    wide = torch.empty(rows, cols, dtype=torch.float64)
    assert eng.all_reduce(mine, wide) is wide and torch.equal(wide, total.double())
    across = torch.zeros(cols, rows).t()
    assert eng.all_reduce(a, across) is across and torch.equal(across, total)
    base = torch.zeros(2 * rows * cols)
    x, shifted = base[:rows * cols], base[16:16 + rows * cols]
    x.copy_(a.reshape(-1))
    assert eng.all_reduce(x, shifted) is shifted and torch.equal(shifted, total.reshape(-1))
    flat = torch.full((rows * cols + 32,), 7.0)  # another shape and room to spare: filled in memory order, as ever
    assert eng.all_reduce(a, flat) is flat and torch.equal(flat[:rows * cols], total.reshape(-1)) and (flat[rows * cols:] == 7).all()
    room = torch.full((rows * cols,), 7.0)
    try:
        eng.all_reduce(a, room[:rows * cols // 2])
        raise SystemExit("an output that is too small was taken")
    except RuntimeError:
        assert (room == 7).all(), "written past the end of the output"
    try:
        eng.all_reduce_async(a, room[:rows * cols // 2]).wait()
        raise SystemExit("an output that is too small was taken")
    except ValueError:
        assert (room == 7).all(), "written past the end of the output"
    assert torch.equal(eng.all_gather(mine), torch.cat([t.reshape(-1) for t in ins]))
    parts = ranks if world > 1 else 1
    assert torch.equal(eng.reduce_scatter(mine), total.reshape(parts, -1)[rank])
    if G > 1:
        # a strided view of the symmetric buffer itself
        w = eng.work_view(rows * cols, torch.float32).view(cols, rows)
        w.copy_(a.t())
        assert torch.equal(eng.all_reduce(w.t()), total)
        w.copy_(a.t())
        assert torch.equal(eng.reduce_scatter(w.t()), total.reshape(parts, -1)[rank])
if world > 1:
    dist.barrier()
eng.close()
print("layouts ok", flush=True)
"""


@pytest.mark.parametrize("nproc,gpn,plain", [(1, 1, False), (2, 1, False), (2, 1, True), (3, 1, False), (4, 2, False)])
def test_whole_sizes(tmp_path, nproc, gpn, plain):
    worker = tmp_path / "worker.py"
    worker.write_text(WORKER)
    env = dict(os.environ, OMP_NUM_THREADS="1", TCPXB_FAKE_GPU="1")
    launch = [sys.executable] if nproc == 1 else [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={nproc}",
                                                  "--master-addr", "127.0.0.1", "--master-port", str(free_port())]
    r = subprocess.run(launch + [str(worker), str(HERE), str(gpn)] + (["plain"] if plain else []), env=env, capture_output=True,
                       text=True, timeout=200)
    assert r.returncode == 0 and r.stdout.count("layouts ok") == nproc, r.stdout[-2000:] + r.stderr[-3000:]
