"""peer_reduce where its variants change: few and many sources, odd vector counts, spans off the 32-byte phase, edges
of a CTA.  The sum runs over the sources in order from zero with one rounding, so the oracle's bits are the kernel's."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from nccl_plugin_gpudirecttcpx_b200 import ops


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nsrcs", [1, 4, 5, 8])
@pytest.mark.parametrize("vecs", [1, 2, 3, 255, 256, 257, 511, 512, 513, 5001])
@pytest.mark.parametrize("off", [0, 16])
def test_edges(dtype, nsrcs, vecs, off):
    per = 16 // dtype.itemsize
    n, lead = vecs * per, 32 // dtype.itemsize
    g = torch.Generator().manual_seed(vecs + nsrcs)
    srcs = [torch.randn(lead + n + 2 * per, generator=g).to(dtype) for _ in range(nsrcs)]
    srcs[-1][lead + off // dtype.itemsize] = float("inf")
    shard_off = 32 + off
    first = shard_off // dtype.itemsize
    whole = torch.full((n + 3 * per,), 5.0, dtype=dtype, device="cuda")
    out = whole[per if off else 0:][:n]
    ops.peer_reduce(out, [s.cuda() for s in srcs], shard_off=shard_off)
    torch.cuda.synchronize()
    want = torch.zeros(n)
    for s in srcs:
        want = want + s[first:first + n].float()
    assert torch.equal(out.cpu(), want.to(dtype))
    behind = whole[(per if off else 0) + n:]
    assert (behind == 5.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nsrcs", range(1, 10))
@pytest.mark.parametrize("vecs", [3, 514])
def test_every_number_of_sources(dtype, nsrcs, vecs):
    """One kernel each; an odd last vector and whole 32-byte pairs, on and off the 32-byte phase."""
    per = 16 // dtype.itemsize
    g = torch.Generator().manual_seed(nsrcs)
    srcs = [torch.randn((vecs + 2) * per, generator=g).to(dtype) for _ in range(nsrcs)]
    for off in (0, 1):
        out = torch.empty(vecs * per, dtype=dtype, device="cuda")
        ops.peer_reduce(out, [s.cuda() for s in srcs], shard_off=off * 16)
        want = torch.zeros(vecs * per)
        for s in srcs:
            want = want + s[off * per:off * per + vecs * per].float()
        assert torch.equal(out.cpu(), want.to(dtype))
