"""Two ranks whose tensors of an odd size are laid out differently: one contiguous, the other strided, with an output of
another type.  What goes over the wire may depend on the size only.  Runs on the stand-in device (gloo ranks)."""
import os
import subprocess
import sys
from pathlib import Path

from conftest import free_port

HERE = Path(__file__).resolve().parent

WORKER = r"""
import os, sys
sys.path[:0] = [sys.argv[1], os.path.dirname(sys.argv[1])]
import torch
import torch.distributed as dist
dist.init_process_group("gloo")
rank = dist.get_rank()
from nccl_plugin_gpudirecttcpx_b200.parallel.engine import default_transport_env
from standin_engine import StandinEngine
default_transport_env(nics=2, nthreads=2, pool_mb=64)
eng = StandinEngine(gpus_per_node=1, request_bytes=256 << 10)
for cols in (1, 501, 100001):
    a, b = (torch.randn(2, cols, generator=torch.Generator().manual_seed(s)) for s in (1, 2))
    mine = a if rank == 0 else b.t().contiguous().t()  # the same values in another memory order
    assert rank == 0 or cols == 1 or not mine.is_contiguous()
    out = None if rank == 0 else torch.empty(2, cols, dtype=torch.float64)
    assert torch.equal(eng.all_reduce(mine, out).float(), a + b)
    assert torch.equal(eng.all_gather(mine), torch.cat([a.reshape(-1), b.reshape(-1)]))
    assert torch.equal(eng.reduce_scatter(mine), (a + b)[rank])
dist.barrier()
eng.close()
print("mixed layouts ok", flush=True)
"""


def test_wire_size_does_not_depend_on_the_layout(tmp_path):
    worker = tmp_path / "worker.py"
    worker.write_text(WORKER)
    env = dict(os.environ, OMP_NUM_THREADS="1", TCPXB_FAKE_GPU="1")
    r = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
                        "--master-port", str(free_port()), str(worker), str(HERE)], env=env, capture_output=True, text=True, timeout=200)
    assert r.returncode == 0 and r.stdout.count("mixed layouts ok") == 2, r.stdout[-2000:] + r.stderr[-3000:]
