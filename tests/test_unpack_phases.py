"""Fragments whose source, destination and accumulator lie at any phase of a 16-byte vector, around the sizes where the ring
kernel's vector stores begin and end, for every product: byte for byte against the oracle, guard bytes included."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from nccl_plugin_gpudirecttcpx_b200.ops import unpack as U

LENGTHS = [1, 2, 3, 4, 8, 15, 16, 17, 28, 31, 32, 33, 47, 64, 500, 512, 528, 1448, 4080, 4092, 4095, 4096]


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("npeers", [0, 1, 3])
@pytest.mark.parametrize("lead", [0, 4, 12])
@pytest.mark.parametrize("ctas", [0, 2])
def test_every_phase(dtype, npeers, lead, ctas):
    es = dtype.itemsize
    lens = np.array([n // es * es for n in LENGTHS for _ in range(16) if n // es])
    phase = np.tile(np.arange(16), len(lens) // 16) // es * es
    idx = np.arange(len(lens))
    step = 4160
    src, dst = idx[::-1] * step + phase, idx * step + (phase * 5 + idx // 16 * es) % 16 // es * es
    descs, nbytes = U.make_descriptors(src, lens, dst), len(lens) * step + 32
    g = torch.Generator().manual_seed(es)
    make = lambda: torch.randint(0, 256, (nbytes,), dtype=dtype, generator=g) if es == 1 else torch.randn(nbytes // es, generator=g).to(dtype)
    pool, acc, out = make(), make(), make()
    room = torch.zeros(nbytes + 64, dtype=torch.uint8, device="cuda")
    d_acc = room[lead:lead + nbytes].view(dtype)  # in a phase of its own, apart from the output's
    d_acc.copy_(acc)
    outs = [out.cuda() for _ in range(1 + npeers)]
    st, d_descs, opts = U.status_buffer(), U.descriptors_to_device(descs), {"max_ctas": ctas}
    if npeers == 0:
        if es == 1:
            U.unpack_copy(pool.cuda(), outs[0], d_descs, status=st, **opts)
        else:
            U.unpack_reduce(pool.cuda(), d_acc, d_descs, out=outs[0], status=st, **opts)
    elif es == 1:
        U.unpack_fanout(pool.cuda(), outs[0], outs[1:], d_descs, status=st, **opts)
    else:
        U.unpack_reduce_fanout(pool.cuda(), d_acc, outs[0], outs[1:], d_descs, status=st, **opts)
    torch.cuda.synchronize()
    want = U.reference_unpack(pool, out, descs, acc=None if es == 1 else acc).view(torch.uint8)
    assert st.tolist()[0] == U.ST_OK
    for o in outs:
        assert torch.equal(o.cpu().view(torch.uint8), want)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("l2", [False, True])
@pytest.mark.parametrize("npeers", [0, 2])
def test_fragments_that_take_plain_loads_and_stores(dtype, l2, npeers):
    """Longer than a slot, and (added at the destination) off the phase: lengths around whole batches of the warp's loop."""
    es = dtype.itemsize
    if es == 1 and l2:
        pytest.skip("copies have one form")
    lens = [n // es * es for n in (4100, 4352, 6144, 8192, 8196, 9000)] + [n * es for n in (1, 31, 32, 33, 127, 128, 129, 255, 257, 1000)]
    lens = np.array([n for n in lens for _ in range(4)])
    idx = np.arange(len(lens))
    step = 9088
    src, dst = idx[::-1] * step + idx % 4 * 4, idx * step + idx % 3 * 4
    descs, nbytes = U.make_descriptors(src, lens, dst), len(lens) * step + 32
    g = torch.Generator().manual_seed(es + npeers)
    make = lambda: torch.randint(0, 256, (nbytes,), dtype=dtype, generator=g) if es == 1 else torch.randn(nbytes // es, generator=g).to(dtype)
    pool, acc = make(), make()
    hosts = [acc if l2 else make()] + [make() for _ in range(npeers)]
    outs = [h.cuda() for h in hosts]
    st, d_descs = U.status_buffer(), U.descriptors_to_device(descs)
    impl = U.REDUCE_L2 if l2 else U.REDUCE_SM
    if es == 1 and npeers:
        U.unpack_fanout(pool.cuda(), outs[0], outs[1:], d_descs, status=st)
    elif es == 1:
        U.unpack_copy(pool.cuda(), outs[0], d_descs, status=st)
    elif npeers:
        U.unpack_reduce_fanout(pool.cuda(), None if l2 else acc.cuda(), outs[0], outs[1:], d_descs, impl=impl, status=st)
    else:
        U.unpack_reduce(pool.cuda(), outs[0] if l2 else acc.cuda(), d_descs, out=outs[0], impl=impl, status=st)
    torch.cuda.synchronize()
    assert st.tolist()[0] == U.ST_OK
    for h, o in zip(hosts, outs):
        # added at the destination, every buffer takes the fragment on top of its own value
        want = U.reference_unpack(pool, h, descs, acc=None if es == 1 else h if l2 else acc)
        assert torch.equal(o.cpu().view(torch.uint8), want.view(torch.uint8))
