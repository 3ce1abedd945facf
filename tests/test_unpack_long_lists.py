"""Scatter lists around the length at which the unpack kernels change (one record per warp of the ring
kernel), with fragments in every phase, against the PyTorch oracle: byte for byte, since a copy moves bytes
and the sum of two values has one correctly rounded result."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from nccl_plugin_gpudirecttcpx_b200.ops import unpack as U

RING_WARPS = 12


def _list(count, frag, es, seed):
    """`count` fragments of up to `frag` bytes at mixed phases: whole ones, ragged ones, short ones, one empty."""
    rng = np.random.default_rng(seed)
    lens = np.full(count, frag // es * es, dtype=np.int64)
    ragged = rng.random(count) < 0.3
    lens[ragged] = rng.integers(1, frag // es + 1, ragged.sum()) * es
    lens[7] = 0
    step = (frag + 63) // 32 * 32
    src = rng.permutation(count).astype(np.int64) * step + rng.integers(0, 32 // es, count) * es * (rng.random(count) < 0.5)
    dst = np.arange(count, dtype=np.int64) * step + rng.integers(0, 32 // es, count) * es * (rng.random(count) < 0.5)
    return U.make_descriptors(src, lens, dst), count * step + 64


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("frag", [48, 1448, 4096, 9000])
@pytest.mark.parametrize("over", [-1, 0, 1, 700])
def test_long_lists(dtype, frag, over):
    count = torch.cuda.get_device_properties(0).multi_processor_count * RING_WARPS + over
    descs, nbytes = _list(count, frag, dtype.itemsize, seed=frag + over)
    g = torch.Generator().manual_seed(frag)
    if dtype == torch.uint8:
        pool, acc = torch.randint(0, 256, (nbytes,), dtype=dtype, generator=g), None
    else:
        pool, acc = (torch.randn(nbytes // dtype.itemsize, generator=g).to(dtype) for _ in range(2))
    out = torch.full((nbytes // dtype.itemsize,), 3, dtype=dtype)
    d_out, st = out.cuda(), U.status_buffer()
    bad = descs.copy()
    bad[count // 2]["src_off"] = nbytes  # past the end: skipped and reported, the rest still runs
    for lst, status in ((bad, U.ST_BOUNDS), (descs, U.ST_OK)):
        st.zero_()
        if acc is None:
            U.unpack_copy(pool.cuda(), d_out, U.descriptors_to_device(lst), status=st)
        else:
            U.unpack_reduce(pool.cuda(), acc.cuda(), U.descriptors_to_device(lst), out=d_out, status=st)
        torch.cuda.synchronize()
        want = U.reference_unpack(pool, out, lst, acc=acc)
        assert torch.equal(d_out.cpu().view(torch.uint8), want.view(torch.uint8))
        s = st.tolist()
        assert s[0] == status and (status == U.ST_OK or (s[1] == count // 2 and s[2] == 1))


def test_accumulator_in_another_phase_than_the_output():
    count = torch.cuda.get_device_properties(0).multi_processor_count * RING_WARPS + 5
    descs, nbytes = _list(count, 1448, 2, seed=3)
    n = nbytes // 2
    g = torch.Generator().manual_seed(5)
    pool, acc = (torch.randn(n, generator=g).to(torch.bfloat16) for _ in range(2))
    d_acc = torch.empty(n + 8, dtype=torch.bfloat16, device="cuda")[3:3 + n]
    d_acc.copy_(acc)
    out = torch.zeros(n, dtype=torch.bfloat16)
    d_out = out.cuda()
    U.unpack_reduce(pool.cuda(), d_acc, U.descriptors_to_device(descs), out=d_out)
    torch.cuda.synchronize()
    want = U.reference_unpack(pool, out, descs, acc=acc)
    assert torch.equal(d_out.cpu().view(torch.uint8), want.view(torch.uint8))
