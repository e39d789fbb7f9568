"""The library's memory pool: idle memory is bounded, given back on request,
and reused safely between streams and threads."""
import threading

import numpy as np
import pytest

import benchsp_b200 as bsp
from benchsp_b200 import _lib

pytestmark = pytest.mark.gpu
SLACK = 64 << 20    # pool granularity and other small allocations


def _held(base):
    import torch
    torch.cuda.synchronize()
    return base - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("copies", [1, 12])
def test_idle_memory_is_bounded_and_given_back(cuda, copies):
    import torch
    A = bsp.gen_stencil27(40, 4, 5)
    rp, ci, va = A.to_device()
    _lib.check(_lib.lib().bsp_pool_trim())
    torch.cuda.synchronize()
    base, total = torch.cuda.mem_get_info()
    live = [bsp.csr2bsr(rp, ci, va, rows=A.rows, cols=A.cols, bs=8) for _ in range(copies)]
    size = _held(base)
    assert size >= copies * live[0].blc_num * 512
    for M in live:
        M.free()
    assert _held(base) <= min(size, total // 64) + SLACK
    _lib.check(_lib.lib().bsp_pool_trim())
    assert _held(base) <= SLACK


def test_streams_and_threads_share_the_pool(cuda):
    import torch
    A = bsp.gen_stencil27(24, 4, 6)
    rp, ci, va = A.to_device()
    x = torch.from_numpy(bsp.gen_uniform(A.cols, 7)).to(cuda)
    want = bsp.csr2bsr(rp, ci, va, rows=A.rows, cols=A.cols).spmv(x).cpu().numpy()
    torch.cuda.synchronize()
    bad = []

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                M = bsp.csr2bsr(rp, ci, va, rows=A.rows, cols=A.cols)
                y = M.spmv(x)
                s.synchronize()
                if not np.array_equal(y.cpu().numpy(), want):
                    bad.append(1)
                M.free()

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_threads_leave_no_more_than_the_bound(cuda):
    """Matrices made and freed by several threads, the frees on other streams than
    the allocations: what the pool keeps at the end is bounded as for one thread."""
    import torch
    A = bsp.gen_stencil27(40, 4, 5)
    rp, ci, va = A.to_device()
    _lib.check(_lib.lib().bsp_pool_trim())
    torch.cuda.synchronize()
    base, total = torch.cuda.mem_get_info()
    made, lock = [], threading.Lock()
    start = threading.Barrier(4)

    def work():
        s = torch.cuda.Stream()
        start.wait()
        with torch.cuda.stream(s):
            for k in range(24):
                M = bsp.csr2bsr(rp, ci, va, rows=A.rows, cols=A.cols, bs=8 if k % 2 else 4)
                s.synchronize()
                with lock:
                    made.append(M)
                    M = made.pop(0) if len(made) > 12 else None
                if M:
                    M.free()

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    rest = [threading.Thread(target=M.free) for M in made]
    for t in rest:
        t.start()
    for t in rest:
        t.join()
    assert _held(base) <= total // 64 + SLACK
    _lib.check(_lib.lib().bsp_pool_trim())
    assert _held(base) <= SLACK


@pytest.mark.parametrize("call", ["csr2bsr", "csr2bcsr"])
def test_a_refused_conversion_keeps_no_memory(cuda, call):
    """33,554,432 blocks of 8x8 (four entries each, in one of the block's rows) are one
    more than int32 indexing holds: refused, and nothing of the attempt stays."""
    import torch
    k = torch.arange(4, dtype=torch.int32, device=cuda)
    row = torch.arange(8, device=cuda, dtype=torch.int32)[:, None, None]
    blk = torch.arange(8, device=cuda, dtype=torch.int32)[None, :, None] * 8
    ci = ((blk + row) * 8 + k).reshape(-1).repeat(1 << 19)   # row r of a block-row: blocks r, 8 + r, ..., 56 + r
    rp = torch.arange(0, ci.numel() + 1, 32, dtype=torch.int32, device=cuda)
    va = torch.zeros(ci.numel(), dtype=torch.float64, device=cuda)
    f = {"csr2bsr": lambda: bsp.csr2bsr(rp, ci, va, rows=1 << 22, cols=512, bs=8),
         "csr2bcsr": lambda: bsp.csr2bcsr(rp, ci, va, rows=1 << 22, cols=512, tile_m=8, tile_k=8)}[call]
    _lib.check(_lib.lib().bsp_pool_trim())
    torch.cuda.synchronize()
    base = torch.cuda.mem_get_info()[0]
    for _ in range(40):                        # 2 MB of block pointers each
        with pytest.raises(bsp.BspError) as e:
            f()
        assert e.value.status == bsp._lib.BSP_ERR_UNSUPPORTED
    torch.cuda.synchronize()
    _lib.check(_lib.lib().bsp_pool_trim())
    assert _held(base) < 32 << 20
