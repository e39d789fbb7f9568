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
