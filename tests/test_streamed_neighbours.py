"""A streamed unpack waits for its producer while more launches are queued behind it.  They must not come in and take the
registers that work on other streams, the producer among it, needs.  The host is the producer here, and the kernel on the
other stream waits for nothing."""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

from nccl_plugin_gpudirecttcpx_b200.ops import unpack as U


@pytest.mark.parametrize("max_ctas,early", [(0, False), (0, True), (16, True)])
def test_launches_behind_a_streamed_one_stay_out(max_ctas, early):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, page = 12 * sms + 200, 4096
    pool = torch.randint(0, 256, (2 * n * page,), dtype=torch.uint8, device="cuda")
    host = U.permuted_fragments(n * page, 2 * n * page, seed=7)
    descs = U.descriptors_to_device(host)
    dst, behind = torch.zeros(n * page, dtype=torch.uint8, device="cuda"), torch.zeros(n * page, dtype=torch.uint8, device="cuda")
    sums = [torch.zeros(n * page // 4, device="cuda") for _ in range(2)]
    ready, word = torch.zeros(1, dtype=torch.int32).pin_memory(), torch.zeros(1, dtype=torch.int32).pin_memory()
    landed = (ctypes.c_uint32 * 1).from_address(word.data_ptr())
    src, staged = torch.ones(1 << 16, dtype=torch.uint8, device="cuda"), torch.zeros(1 << 16, dtype=torch.uint8).pin_memory()
    st = U.status_buffer()
    lib = U._k()
    lib.tcpxb_stage_out.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    # every kernel once, so that none is loaded while another one waits
    U.unpack_copy(pool, behind, descs)
    U.unpack_copy(pool, dst, descs, ready_count=torch.full((1,), n, dtype=torch.int32, device="cuda"))
    U.peer_reduce(sums[0], sums, 0)
    assert lib.tcpxb_stage_out(src.data_ptr(), staged.data_ptr(), 1 << 16, word.data_ptr(), 1, None) == 0
    torch.cuda.synchronize()
    dst.zero_(), behind.zero_(), staged.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        U.unpack_copy(pool, dst, descs, status=st, ready_count=ready.data_ptr(), wait_ns=5_000_000_000, max_ctas=max_ctas, early_launch=early)
        U.unpack_copy(pool, behind, descs, status=st)  # two register kernels, which fit beside the waiting one
        U.peer_reduce(sums[0], sums, 0)
    time.sleep(0.05)
    assert lib.tcpxb_stage_out(src.data_ptr(), staged.data_ptr(), 1 << 16, word.data_ptr(), 2, b.cuda_stream) == 0  # CTAs of 1024 threads
    t = time.perf_counter()
    while landed[0] != 2 and time.perf_counter() - t < 1.0:
        pass
    seen = landed[0]
    ready[0] = n  # whatever came of that, let the streamed launch finish
    torch.cuda.synchronize()
    assert seen == 2, "the other stream's kernel did not run while the streamed launch waited"
    want = U.reference_unpack(pool, torch.zeros(n * page, dtype=torch.uint8), host)
    assert st.tolist()[0] == U.ST_OK and torch.equal(dst.cpu(), want) and torch.equal(behind.cpu(), want)
