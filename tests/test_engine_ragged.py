"""Collectives of sizes that are no multiple of 16 bytes, on the buffers themselves: one GPU per node, the rank as its
own network peer.  A sum of a value and itself is exact, and a gather moves bytes, so results are compared bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from nccl_plugin_gpudirecttcpx_b200.parallel.engine import HierarchicalEngine, default_transport_env
    default_transport_env(nics=2, nthreads=2, nsocks_per_thread=1, pool_mb=256)
    e = HierarchicalEngine(gpus_per_node=1, request_bytes=1 << 20)
    yield e
    e.close()


SIZES = [1, 3, 9, 1025, 32767, 32769, (1 << 19) + 1, (2 << 20) + 3]


def _values(numel, dtype, lead):
    """Random values `lead` elements into an allocation, so that the data starts off the 16-byte phase."""
    g = torch.Generator("cuda").manual_seed(numel)
    return torch.randn(numel + lead, device="cuda", generator=g).to(dtype)[lead:]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lead", [0, 1])
@pytest.mark.parametrize("numel", SIZES)
def test_all_reduce(engine, dtype, lead, numel):
    x = _values(numel, dtype, lead)
    want = x * 2
    guard = torch.full((numel + 17,), 5.0, dtype=dtype, device="cuda")
    out = guard[1:1 + numel]
    assert engine.all_reduce(x, out) is out
    torch.cuda.synchronize()
    assert torch.equal(out, want) and guard[0] == 5 and (guard[1 + numel:] == 5).all()
    assert torch.equal(engine.all_reduce(x), want)
    y = x.clone()
    assert engine.all_reduce(y, y) is y and torch.equal(y, want)  # in place
    assert engine.device_status()[0] == 0


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lead", [0, 1])
@pytest.mark.parametrize("numel", SIZES)
def test_all_gather_and_reduce_scatter(engine, dtype, lead, numel):
    x = _values(numel, torch.float32, lead).mul(50).to(torch.uint8) if dtype == torch.uint8 else _values(numel, dtype, lead)
    assert torch.equal(engine.all_gather(x), torch.cat([x, x]))
    if dtype != torch.uint8:
        assert torch.equal(engine.reduce_scatter(x), x * 2)
    assert engine.device_status()[0] == 0


def test_layouts_that_are_put_right_by_copies(engine):
    """Strides, a partial overlap and an output of another type gave right results through padded copies and still do."""
    base = torch.randn(2 * 1001, device="cuda")
    strided = base.view(2, 1001).t()
    assert torch.equal(engine.all_reduce(strided), strided * 2)
    assert torch.equal(engine.all_gather(strided), torch.cat([strided, strided]).reshape(-1))
    want = base[:1001] * 2
    wide = torch.empty(1001, dtype=torch.float64, device="cuda")
    assert engine.all_reduce(base[:1001], wide) is wide and torch.equal(wide, want.double())
    shifted = base[4:1005]
    assert engine.all_reduce(base[:1001], shifted) is shifted and torch.equal(shifted, want)
    on_host = torch.empty(1001)
    assert engine.all_reduce(base[:1001].copy_(want), on_host) is on_host and torch.equal(on_host, want.cpu() * 2)


def test_native_sizes_stay_checked(engine):
    """A caller of the C entry point that did not ask for ragged sizes is told so, as before."""
    x, y = torch.zeros(8, device="cuda"), torch.zeros(8, device="cuda")
    assert engine._api.tcpxb_engine_set_ragged(engine._h, 0) == 0
    try:
        assert engine._api.tcpxb_engine_all_reduce(engine._h, x.data_ptr(), y.data_ptr(), 20, 2, None) != 0
        assert engine._api.tcpxb_engine_all_gather(engine._h, x.data_ptr(), y.data_ptr(), 12, None) != 0
        assert engine._api.tcpxb_engine_reduce_scatter(engine._h, x.data_ptr(), y.data_ptr(), 12, 2, None) != 0
    finally:
        engine._api.tcpxb_engine_set_ragged(engine._h, 1)


def test_layouts_at_whole_sizes(engine):
    """The same at sizes that need no padding, and an output of the wrong size is refused before anything is written."""
    base = torch.randint(-64, 64, (2 * 1008,), device="cuda").float()
    strided = base.view(2, 1008).t()
    assert torch.equal(engine.all_reduce(strided), strided * 2)
    assert torch.equal(engine.all_gather(strided), torch.cat([strided, strided]).reshape(-1))
    assert torch.equal(engine.reduce_scatter(strided), (strided * 2).reshape(-1))
    want = base[:1008] * 2
    wide = torch.empty(1008, dtype=torch.float64, device="cuda")
    assert engine.all_reduce(base[:1008], wide) is wide and torch.equal(wide, want.double())
    on_host = torch.empty(1008)
    assert engine.all_reduce(base[:1008], on_host) is on_host and torch.equal(on_host, want.cpu())
    assert torch.equal(engine.all_reduce(base[:1008].cpu()), want.cpu())
    room = torch.full((1008,), 7.0, device="cuda")
    with pytest.raises(RuntimeError):
        engine.all_reduce(base[:1008], room[:512])
    assert (room == 7).all()
    shifted = base[16:1024]
    assert engine.all_reduce(base[:1008], shifted) is shifted and torch.equal(shifted, want)
    assert engine.device_status()[0] == 0
