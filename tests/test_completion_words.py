"""Kernels that tell a polling host that they are done: the unpack kernels' completion word and the staging
kernel of small sends.  Both are compared byte for byte: one moves bytes, the other sums two values."""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

from nccl_plugin_gpudirecttcpx_b200.ops import unpack as U


def _word():
    w = torch.zeros(16, dtype=torch.int32).pin_memory()
    return w, (ctypes.c_uint32 * 16).from_address(w.data_ptr())


def _wait(view, value):
    t = time.perf_counter()
    while view[0] != value and time.perf_counter() - t < 5:
        pass
    assert view[0] == value


def _request():
    f = U._k().tcpxb_unpack_request
    vp, u64, u32, ci = ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint32, ctypes.c_int
    f.argtypes = [vp, u64, vp, vp, vp, u64, vp, ci, vp, vp, u32, ci, ci, vp, vp, vp, u32, vp]
    return f


@pytest.mark.parametrize("nbytes", [1, 15, 16, 17, 1000, 4096, 16384, 16400, 65535, 65536])
@pytest.mark.parametrize("off", [0, 3, 16])
def test_stage_out(nbytes, off):
    lib = U._k()
    lib.tcpxb_stage_out.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p]
    src = torch.randint(0, 256, (nbytes + 32,), dtype=torch.uint8, device="cuda")
    host = torch.full((nbytes + 64,), 7, dtype=torch.uint8).pin_memory()
    word, view = _word()
    torch.cuda.synchronize()
    assert lib.tcpxb_stage_out(src.data_ptr() + off, host.data_ptr() + 16, nbytes, word.data_ptr(), 41, None) == 0
    _wait(view, 41)
    got = host.clone()  # before any synchronize: the word alone says that the bytes are there
    assert torch.equal(got[16:16 + nbytes], src[off:off + nbytes].cpu())
    assert (got[:16] == 7).all() and (got[16 + nbytes:] == 7).all()
    torch.cuda.synchronize()


@pytest.mark.parametrize("count,ctas", [(1, 16), (15, 16), (17, 16), (256, 16), (2000, 0)])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16])
@pytest.mark.parametrize("bad", [False, True])
def test_done_word(count, ctas, dtype, bad):
    total = count * 4096 - 96
    pool = torch.randint(0, 256, (count * 8192,), dtype=torch.uint8)
    if dtype != torch.uint8:
        pool = torch.randn(count * 4096).to(dtype)
    descs = U.permuted_fragments(total, count * 8192, seed=count)
    if bad:
        descs[count // 2]["src_off"] = count * 8192  # refused; the word is written all the same, the fan-out flag is not
    acc = None if dtype == torch.uint8 else torch.randn(total // 2).to(dtype)
    out = torch.zeros(total // dtype.itemsize, dtype=dtype)
    d_out, d_pool, d_descs = out.cuda(), pool.cuda(), U.descriptors_to_device(descs)
    word, view = _word()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    ticket, st = torch.zeros(1, dtype=torch.int32, device="cuda"), U.status_buffer()
    opts = U._Opts()
    opts.max_ctas, opts.ticket = ctas, ticket.data_ptr()
    opts.flag_value, opts.peer_flags[0] = 9, flag.data_ptr()
    d_acc = None if acc is None else acc.cuda()
    torch.cuda.synchronize()
    for turn in (1, 2):
        rc = _request()(d_pool.data_ptr(), U._nbytes(d_pool), U._ptr(d_acc), d_out.data_ptr(), None, total, None, 0, d_descs.data_ptr(), None,
                        count, U.DTYPE_BF16, U.REDUCE_SM, st.data_ptr(), ctypes.byref(opts), word.data_ptr(), turn, None)
        assert rc == 0
        _wait(view, turn)
    torch.cuda.synchronize()
    want = U.reference_unpack(pool, out, descs, acc=acc)
    assert torch.equal(d_out.cpu().view(torch.uint8), want.view(torch.uint8))
    assert ticket.item() == 0 and flag.item() == (0 if bad else 9)
    assert st.tolist()[0] == (U.ST_BOUNDS if bad else U.ST_OK)


def test_done_word_needs_a_ticket():
    opts = U._Opts()
    x = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    d = U.descriptors_to_device(U.make_descriptors([0], [16], [0]))
    word, view = _word()
    assert _request()(x.data_ptr(), 4096, None, x.data_ptr(), None, 4096, None, 0, d.data_ptr(), None, 1, 0, 0, None, ctypes.byref(opts),
                      word.data_ptr(), 1, None) != 0
    assert view[0] == 0


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("count", [1, 2, 7, 8, 9])
@pytest.mark.parametrize("frag,phase", [(1, 0), (20, 12), (1448, 0), (4096, 0), (4096, 4), (9000, 4)])
@pytest.mark.parametrize("bad", [False, True])
def test_short_lists_travel_with_the_launch(dtype, count, frag, phase, bad):
    """Up to eight records out of pinned memory; the list on the device is poisoned where it must not be read."""
    es = dtype.itemsize
    frag = max(frag // es, 1) * es
    step = frag + 64 - frag % 32
    nbytes = count * step + 64
    g = torch.Generator().manual_seed(frag + count)
    pool = torch.randint(0, 256, (nbytes,), dtype=torch.uint8, generator=g) if es == 1 else torch.randn(nbytes // es, generator=g).to(dtype)
    pool = pool.pin_memory()
    acc = None if es == 1 else torch.randn(nbytes // es, generator=g).to(dtype)
    idx = torch.arange(count).numpy()
    descs = U.make_descriptors(idx[::-1] * step + phase, [frag] * (count - 1) + [max(frag // 2 // es, 1) * es], idx * step + 8)
    if bad:
        descs[count // 2]["src_off"] = nbytes
    out = torch.full((nbytes // es,), 3, dtype=dtype)
    d_out, d_acc, st = out.cuda(), None if acc is None else acc.cuda(), U.status_buffer()
    d_descs = U.descriptors_to_device(descs) if count > 8 else torch.zeros(16 * count, dtype=torch.uint8, device="cuda")
    word, view = _word()
    opts, ticket = U._Opts(), torch.zeros(1, dtype=torch.int32, device="cuda")
    opts.max_ctas, opts.ticket = 16, ticket.data_ptr()
    torch.cuda.synchronize()
    code = {1: U.DTYPE_U8, 2: U.DTYPE_BF16, 4: U.DTYPE_F32}[es]
    assert _request()(pool.data_ptr(), U._nbytes(pool), U._ptr(d_acc), d_out.data_ptr(), None, U._nbytes(out), None, 0, d_descs.data_ptr(),
                      descs.ctypes.data, count, code, U.REDUCE_SM, st.data_ptr(), ctypes.byref(opts), word.data_ptr(), 3, None) == 0
    _wait(view, 3)
    torch.cuda.synchronize()
    want = U.reference_unpack(pool, out, descs, acc=acc)
    assert torch.equal(d_out.cpu().view(torch.uint8), want.view(torch.uint8))
    assert st.tolist()[:2] == ([U.ST_BOUNDS, count // 2] if bad else [U.ST_OK, 0]) and ticket.item() == 0
