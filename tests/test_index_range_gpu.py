"""Matrices whose last nonzero stands at the end of the int32 range: positions
that a kernel steps to behind the last row stay above its end."""
import numpy as np
import pytest

import benchsp_b200 as bsp

pytestmark = pytest.mark.gpu
NNZ = 2 ** 31 - 1


def _row_pointers(kind):
    """Rows of one length up to NNZ, or rows of 64 and a last one of 3000."""
    if kind == "long last":
        rp = np.append(np.arange(0, NNZ - 3000, 64), [NNZ - 3000, NNZ])
    else:
        rp = np.minimum(np.arange(0, NNZ + kind, kind), NNZ)
    return rp.astype(np.int32)


@pytest.fixture(scope="module")
def ones():
    """Columns 0 and FP16 values 1, NNZ of each (13 GB)."""
    import torch
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    return torch.zeros(NNZ, dtype=torch.int32, device="cuda"), torch.ones(NNZ, dtype=torch.float16, device="cuda")


@pytest.mark.parametrize("kind", [2048, 512, 128, "long last"])
def test_csr_spmv_up_to_the_last_index(cuda, ones, kind):
    import torch
    rp = _row_pointers(kind)
    y = bsp.csr_spmv(torch.from_numpy(rp).to(cuda), *ones, torch.ones(1, dtype=torch.float16, device=cuda))
    assert np.array_equal(y.float().cpu().numpy(), np.diff(rp).astype(np.float32))   # exact up to 2048, even above


@pytest.mark.parametrize("kind", [2048, 128, "long last"])
def test_spmm_plan_up_to_the_last_index(cuda, ones, kind):
    import torch
    rp = _row_pointers(kind)
    P = bsp.SpmmPlan(torch.from_numpy(rp).to(cuda), *ones, cols=1)
    C = P.spmm(torch.ones(1, 8, dtype=torch.float16, device=cuda))
    P.free()
    assert torch.equal(C, torch.from_numpy(np.diff(rp)).to(cuda).float()[:, None].expand(-1, 8))


@pytest.mark.parametrize("bs", [4, 8])
def test_conversion_up_to_the_last_index(cuda, bs):
    """Whole blocks but for the last entry: their 2^31 values are one more than
    the index range holds, which is refused once the blocks are counted."""
    import torch
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of device memory")
    rp = torch.from_numpy(_row_pointers(512)).to(cuda)
    ci = torch.arange(512, dtype=torch.int32, device=cuda).repeat(1 << 22)[:NNZ]
    va = torch.empty(NNZ, dtype=torch.float64, device=cuda)
    with pytest.raises(bsp.BspError) as e:
        bsp.csr2bsr(rp, ci, va, rows=rp.numel() - 1, cols=512, bs=bs)
    assert e.value.status == bsp._lib.BSP_ERR_UNSUPPORTED
