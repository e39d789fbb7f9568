"""CG on the GPU: FP64 and mixed precision (FP32 / per-group-scaled FP16 and
BF16 storage, FP64 refinement) reach ||b - A x|| / ||b|| <= 1e-10, checked
with the CPU oracle's FP64 SpMV, and agree with the CPU FP64 CG oracle."""
import numpy as np
import pytest

import benchsp_b200 as bsp
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _dev(cuda, *arrs):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in arrs]


def _permuted_laplace(nx, seed):
    """A symmetric permutation of a 2-D Laplacian: SPD, and with nx*nx > 32768
    rows some |col - row| exceed the int16 offset range."""
    import scipy.sparse as sp
    A = bsp.gen_laplace2d(nx, nx)
    M = sp.csr_matrix((A.values, A.colidx, A.rowptr), shape=(A.rows, A.rows))
    perm = np.random.default_rng(seed).permutation(A.rows)
    M = M[perm][:, perm].tocsr()
    M.sort_indices()
    return bsp.HostCSR(A.rows, A.rows, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.copy())


def _ragged_laplace(nx):
    """2-D Laplacian plus symmetric couplings (-0.1) from every 97th row to
    the rows 100, 200, ..., 1000 after it, diagonal raised to keep it
    diagonally dominant: SPD, offsets within int16, and SELL-32 slices of
    uneven length (padding all to the longest would cost far more than 1/32
    extra storage, so the low-precision copy keeps per-slice lengths)."""
    import scipy.sparse as sp
    A = bsp.gen_laplace2d(nx, nx)
    n = A.rows
    M = sp.csr_matrix((A.values, A.colidx, A.rowptr), shape=(n, n)).tolil()
    for i in range(0, n, 97):
        for d in range(100, 1001, 100):
            if i + d < n:
                M[i, i + d] = M[i + d, i] = -0.1
                M[i, i] += 0.1
                M[i + d, i + d] += 0.1
    M = M.tocsr()
    M.sort_indices()
    return bsp.HostCSR(n, n, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.copy())


@pytest.mark.parametrize("mode", ["f32", "f16", "bf16"])
def test_cg_mixed_uneven_slices(cuda, mode):
    A = _ragged_laplace(120)
    lens = np.zeros(-(-A.rows // 32) * 32, np.int64)
    lens[:A.rows] = np.diff(A.rowptr)
    sl = lens.reshape(-1, 32).max(axis=1)
    assert sl.size * 32 * sl.max() > 32 * sl.sum() * 33 // 32      # per-slice lengths are kept
    b = bsp.gen_uniform(A.rows, 12)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    x, res = S.solve(bb)
    S.close()
    x = x.cpu().numpy()
    assert res["converged"] == 1 and res["delta16"] == 1
    assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x) <= 2e-10
    xr, _ = pyoracle.cg(A.rowptr, A.colidx, A.values, b, 1e-12)
    assert np.linalg.norm(x - xr) / np.linalg.norm(xr) < 1e-7


@pytest.mark.parametrize("mode", ["fp64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("kind", ["poisson24", "permuted_laplace"])
def test_cg_reaches_1e10(cuda, mode, kind):
    A = bsp.gen_poisson3d(24) if kind == "poisson24" else _permuted_laplace(200, 4)
    b = bsp.gen_uniform(A.rows, 11)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    x, res = S.solve(bb)
    x = x.cpu().numpy()
    assert res["converged"] == 1 and res["rel_residual"] <= 1e-10
    assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x) <= 2e-10
    if mode != "fp64":
        assert res["reliable_updates"] >= 2
        assert res["delta16"] == (1 if kind == "poisson24" else 0)
    xr, _ = pyoracle.cg(A.rowptr, A.colidx, A.values, b, 1e-12)
    assert np.linalg.norm(x - xr) / np.linalg.norm(xr) < 1e-7


def test_cg_repeated_solves_and_initial_guess(cuda):
    import torch
    A = bsp.gen_poisson3d(16)
    rp, ci, va = _dev(cuda, A.rowptr, A.colidx, A.values)
    S = bsp.CgSolver(rp, ci, va, mode="f16")
    for seed in (1, 2):
        b = bsp.gen_uniform(A.rows, seed)
        x, res = S.solve(_dev(cuda, b)[0])
        assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x.cpu().numpy()) <= 2e-10
    # starting from the solution: no iterations needed
    x2, res2 = S.solve(_dev(cuda, b)[0], x.clone())
    assert res2["iterations"] == 0 and res2["converged"] == 1


def test_cg_not_converged_is_reported(cuda):
    A = bsp.gen_poisson3d(16)
    b = bsp.gen_uniform(A.rows, 5)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode="fp64", max_iters=4, check_every=2)
    with pytest.raises(bsp.BspError):
        S.solve(bb)
    x, res = S.solve(bb, raise_on_stall=False)
    assert res["converged"] == 0 and res["rel_residual"] > 1e-10


def test_cg_without_graphs_matches(cuda):
    A = bsp.gen_poisson3d(12)
    b = bsp.gen_uniform(A.rows, 9)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    x1, r1 = bsp.CgSolver(rp, ci, va, mode="f16", use_graphs=True).solve(bb)
    x2, r2 = bsp.CgSolver(rp, ci, va, mode="f16", use_graphs=False).solve(bb)
    assert r1["iterations"] == r2["iterations"]
    assert np.array_equal(x1.cpu().numpy(), x2.cpu().numpy())


def _banded(n, diags, seed):
    """SPD: symmetric bands at +-diags with varying negative values (every 50th
    entry missing), diagonally dominant."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    M = sp.csr_matrix((n, n))
    for d in diags:
        if d < n:
            v = -rng.uniform(0.5, 1.0, n - d)
            v[::50] = 0.0
            M = M + sp.diags([v, v], [d, -d], shape=(n, n), format="csr")
    M.eliminate_zeros()
    M = (M + sp.diags(np.asarray(abs(M).sum(1)).ravel() + 0.5, format="csr")).tocsr()
    M.sort_indices()
    return bsp.HostCSR(n, n, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64))


# the fused iteration (at most 8 diagonals, vectors in shared memory): one row,
# a part of a slice, one CTA and several, 1, 3, 5 and 7 diagonals, neighbours in
# the next CTA and several CTAs away, a ragged last slice, the last size that
# fits 148 SMs in FP32 and the first that does not; 9 diagonals take two kernels
@pytest.mark.parametrize("n,diags", [
    (1, []), (31, [1]), (33, [1]), (1000, []), (1025, [1, 7]), (5000, [1, 70]), (70001, [1, 33, 1024]),
    (200003, [2, 450, 45000]), (20000, [1, 50, 700, 3000]), (2150144, [1, 1466]), (2160000, [1, 1466])])
@pytest.mark.parametrize("mode", ["fp64", "f32", "f16", "bf16"])
def test_cg_fused_edges(cuda, n, diags, mode):
    A = _banded(n, diags, n)
    b = bsp.gen_uniform(n, 15)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    for start in (None, bb * 0.5):
        x, res = S.solve(bb, None if start is None else start.clone())
        assert res["converged"] == 1
        assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x.cpu().numpy()) <= 2e-10
    S.close()


def test_cg_fused_on_several_streams(cuda):
    """Solves on streams of their own, all at once: the same bits as alone."""
    import threading

    import torch
    A = bsp.gen_poisson3d(64)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, bsp.gen_uniform(A.rows, 16))
    modes = ["f16", "f32", "bf16", "f16"]
    want = {}
    for m in set(modes):
        S = bsp.CgSolver(rp, ci, va, mode=m, tol=1e-10)
        want[m] = S.solve(bb)[0]
        S.close()
    torch.cuda.synchronize()
    same = [False] * len(modes)

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            S = bsp.CgSolver(rp, ci, va, mode=modes[k], tol=1e-10)
            xs = [S.solve(bb)[0] for _ in range(3)]
            s.synchronize()
            same[k] = all(torch.equal(x, want[modes[k]]) for x in xs)
            S.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(modes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(same)


def _rewritten(A, kind):
    """A's entries stored another way: "repeated" splits every diagonal entry in
    two equal halves (as reading a symmetric file entry by entry gives it),
    "descending" reverses each row."""
    rp, ci, va = [0], [], []
    for i in range(A.rows):
        s = slice(A.rowptr[i], A.rowptr[i + 1])
        c, v = A.colidx[s], A.values[s]
        if kind == "repeated":
            k = 1 + (c == i)
            c, v = np.repeat(c, k), np.repeat(v / k, k)
        else:
            c, v = c[::-1], v[::-1]
        ci.append(c)
        va.append(v)
        rp.append(rp[-1] + len(c))
    return bsp.HostCSR(A.rows, A.rows, np.asarray(rp, np.int32), np.concatenate(ci), np.concatenate(va))


# a copy by 5 or 7 diagonals has no free place for a repeated entry, by 3 it has
@pytest.mark.parametrize("diags", [[1], [1, 70], [1, 33, 1024]])
@pytest.mark.parametrize("kind", ["repeated", "descending"])
@pytest.mark.parametrize("mode", ["fp64", "f16"])
def test_cg_rows_with_repeated_or_unsorted_columns(cuda, diags, kind, mode):
    A = _banded(3000, diags, 7)
    R = _rewritten(A, kind)
    b = bsp.gen_uniform(A.rows, 8)
    rp, ci, va, bb = _dev(cuda, R.rowptr, R.colidx, R.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    x, res = S.solve(bb)
    S.close()
    assert res["converged"] == 1
    assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x.cpu().numpy()) <= 2e-10


@pytest.mark.parametrize("mode", ["fp64", "f16"])
def test_cg_fused_wait_that_runs_out(cuda, mode):
    """With one read per wait the fused launch gives up: the solve returns the
    status, leaves x alone, and the plan solves again to the same bits."""
    import torch
    A = bsp.gen_poisson3d(64)
    rp, ci, va, b = _dev(cuda, A.rowptr, A.colidx, A.values, bsp.gen_uniform(A.rows, 17))
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    assert S.fused_ctas > 1
    want, _ = S.solve(b)
    for _ in range(2):
        S.set_wait_limit(1)
        x = torch.full_like(b, 0.25)
        with pytest.raises(bsp.BspError) as e:
            S.solve(b, x)
        assert e.value.status == bsp._lib.BSP_ERR_TIMEOUT
        assert torch.all(x == 0.25)
        S.set_wait_limit(1 << 23)
        got, res = S.solve(b)
        assert res["converged"] == 1 and torch.equal(got, want)
    with pytest.raises(bsp.BspError):
        S.set_wait_limit(0)
    S.close()


@pytest.mark.parametrize("mode", ["fp64", "f16"])
def test_cg_two_kernels_without_graphs_match(cuda, mode):
    """use_graphs changes nothing in the two-kernel iteration (9 diagonals)."""
    A = _banded(20000, [1, 50, 700, 3000], 3)
    rp, ci, va, b = _dev(cuda, A.rowptr, A.colidx, A.values, bsp.gen_uniform(A.rows, 18))
    out = []
    for graphs in (True, False):
        S = bsp.CgSolver(rp, ci, va, mode=mode, use_graphs=graphs)
        assert S.fused_ctas == 0
        x, res = S.solve(b)
        out.append((x.cpu().numpy(), res["iterations"]))
        S.close()
    assert out[0][1] == out[1][1] and np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("mode,value,vector", [("fp64", 8, 8), ("f32", 4, 4), ("f16", 2, 4)])
def test_cg_fused_bytes_leave_out_what_stays_on_the_sms(cuda, mode, value, vector):
    """bytes_moved of a fused solve: per iteration 8 diagonals, an exponent per row
    in FP16, and p published with its tag, written and read; per chunk x, r and p in
    and out; per FP64 residual the CSR matrix and three vectors."""
    A = bsp.gen_poisson3d(16)
    n = A.rows
    rp, ci, va, b = _dev(cuda, A.rowptr, A.colidx, A.values, bsp.gen_uniform(n, 19))
    S = bsp.CgSolver(rp, ci, va, mode=mode, check_every=8)
    assert S.fused_ctas > 0
    _, r = S.solve(b)
    S.close()
    per_iter = n * (8 * value + (value == 2) + 4 * vector)
    residuals = r["reliable_updates"] + 2
    assert r["bytes_moved"] == r["iterations"] * per_iter + r["iterations"] // 8 * 6 * vector * n + \
        residuals * (12 * A.nnz + 4 * (n + 1) + 24 * n)


# the last size whose vectors fit 148 SMs next to the kernel's own shared memory (453
# slices of 512 bytes per CTA in the mixed modes, 226 of 1024 in FP64), with the last
# slice ragged, and the first size past it; the iterates of both forms agree
@pytest.mark.parametrize("mode,n", [("f32", 2145408), ("f16", 2145408), ("bf16", 2145395), ("f32", 2145409),
                                    ("fp64", 1070336), ("fp64", 1070325), ("fp64", 1070337)])
def test_cg_fused_up_to_the_last_size(cuda, mode, n):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes of 148 SMs")
    A = _banded(n, [1, 1466], n)
    b = bsp.gen_uniform(n, 15)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    assert S.fused_ctas == (0 if n in (2145409, 1070337) else 148)
    x, res = S.solve(bb)
    S.close()
    assert res["converged"] == 1
    assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x.cpu().numpy()) <= 2e-10
    if n not in (2145409, 1070337):            # the other form: 8192 rows more, uncoupled from the rest
        R = bsp.HostCSR(n + 8192, n + 8192, np.append(A.rowptr, A.rowptr[-1] + np.arange(1, 8193)).astype(np.int32),
                        np.append(A.colidx, np.arange(n, n + 8192)).astype(np.int32),
                        np.append(A.values, np.ones(8192)))
        rp, ci, va, b2 = _dev(cuda, R.rowptr, R.colidx, R.values, np.append(b, np.zeros(8192)))
        S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
        assert S.fused_ctas == 0
        y, res2 = S.solve(b2)
        S.close()
        assert res2["iterations"] == res["iterations"] and torch.all(y[n:] == 0)
        # two residuals of 1e-10, eigenvalues between 0.5 and 2 * 4 + 0.5
        assert float((y[:n] - x).norm() / x.norm()) <= 2e-10 * 17


@pytest.mark.parametrize("n,diags,fused", [(31, [1], True), (5000, [1, 70], True), (200003, [2, 450, 45000], True),
                                           (20000, [1, 50, 700, 3000], False)])
def test_cg_form_that_runs(cuda, n, diags, fused):
    """Which matrices the fused iteration takes, and none with a preconditioner."""
    A = _banded(n, diags, n)
    rp, ci, va = _dev(cuda, A.rowptr, A.colidx, A.values)
    for mode in ("fp64", "f32", "f16", "bf16"):
        S = bsp.CgSolver(rp, ci, va, mode=mode)
        assert (S.fused_ctas > 0) == fused
        S.close()
    S = bsp.CgSolver(rp, ci, va, mode="f16", precond="jacobi")
    assert S.fused_ctas == 0
    S.close()


@pytest.mark.parametrize("mode,n,fused", [("fp64", 18000, True), ("fp64", 18001, False), ("fp64", 179999, False),
                                          ("fp64", 180000, True), ("f32", 36000, True), ("f32", 36001, False),
                                          ("f32", 119999, False), ("f32", 120000, True), ("f16", 64000, True)])
def test_cg_two_kernels_between_the_sizes(cuda, mode, n, fused):
    """The middle sizes iterate with two kernels, and both forms solve."""
    A = _banded(n, [1, 50], n)
    b = bsp.gen_uniform(n, 15)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    assert (S.fused_ctas > 0) == fused
    x, res = S.solve(bb)
    S.close()
    assert res["converged"] == 1
    assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x.cpu().numpy()) <= 2e-10


@pytest.mark.parametrize("mode", ["fp64", "f16"])
def test_cg_on_a_stream_of_fewer_sms(cuda, mode):
    """A stream confined to 16 SMs has no room for the fused launch: the plan goes over
    to two kernels and solves."""
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]

    A = bsp.gen_poisson3d(64)
    b = bsp.gen_uniform(A.rows, 21)
    rp, ci, va, bb = _dev(cuda, A.rowptr, A.colidx, A.values, b)
    S = bsp.CgSolver(rp, ci, va, mode=mode, tol=1e-10)
    assert S.fused_ctas > 16
    dev = ok(drv.cuDeviceGet(0))
    sms = ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    part = ok(drv.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    ctx = ok(drv.cuGreenCtxCreate(ok(drv.cuDevResourceGenerateDesc([part[0]], 1)), dev,
                                  drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    raw = ok(drv.cuGreenCtxStreamCreate(ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    stream = torch.cuda.ExternalStream(int(raw))
    torch.cuda.synchronize()
    x, res = S.solve(bb, torch.zeros_like(bb), stream=stream)
    stream.synchronize()
    assert res["converged"] == 1 and S.fused_ctas == 0
    assert pyoracle.rel_residual(A.rowptr, A.colidx, A.values, b, x.cpu().numpy()) <= 2e-10
    _, again = S.solve(bb)                     # the whole device: two kernels too
    assert again["converged"] == 1
    S.close()
    torch.cuda.synchronize()
    ok(drv.cuStreamDestroy(raw) + (None,))
    ok(drv.cuGreenCtxDestroy(ctx) + (None,))


@pytest.mark.parametrize("n,every,fused", [(599999, 1, False), (599999, 4, True), (600000, 2, True)])
def test_cg_form_by_check_every(cuda, n, every, fused):
    A = _banded(n, [1, 50], n)
    rp, ci, va, b = _dev(cuda, A.rowptr, A.colidx, A.values, bsp.gen_uniform(n, 15))
    S = bsp.CgSolver(rp, ci, va, mode="f16", check_every=every)
    assert (S.fused_ctas > 0) == fused
    assert S.solve(b)[1]["converged"] == 1
    S.close()
