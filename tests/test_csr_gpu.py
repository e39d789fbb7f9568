"""CSR SpMV kernels on the GPU against the oracle (src/ref.cpp restated) and
the reference's own outputs in tests/golden."""
import glob
from pathlib import Path

import numpy as np
import pytest

import benchsp_b200 as bsp
from oracle import pyoracle

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"
SPMV = sorted(Path(p).name for p in glob.glob(str(GOLDEN / "spmv_*.npz")))


def _dev(cuda, *arrs):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in arrs]


def _within(y, ref, tol):
    err = np.abs(y - ref)
    assert np.all(err <= tol), f"max excess {np.max(err - tol)} at {int(np.argmax(err - tol))}"


@pytest.mark.parametrize("name", SPMV)
def test_scalar_fp64_is_bit_exact_with_reference(cuda, golden, name):
    g = golden(name)
    rp, ci, va, x = _dev(cuda, g["rowptr"], g["colidx"], g["values"], g["x"])
    y = bsp.csr_spmv(rp, ci, va, x, algo="scalar").cpu().numpy()
    assert np.array_equal(y.view(np.uint64), g["y_fp64"].view(np.uint64))


@pytest.mark.parametrize("name", SPMV)
def test_stream_is_bit_exact_with_reference(cuda, golden, name):
    """The warp-per-32-rows stream kernel sums each row left to right with
    separately rounded multiply and add: the reference's own results, bit for
    bit, in FP64, FP32 and FP16."""
    import torch
    g = golden(name)
    rp, ci, va, x = _dev(cuda, g["rowptr"], g["colidx"], g["values"], g["x"])
    y = bsp.csr_spmv(rp, ci, va, x, algo="stream").cpu().numpy()
    assert np.array_equal(y.view(np.uint64), g["y_fp64"].view(np.uint64))
    v32 = torch.from_numpy(g["values"].astype(np.float32)).to(cuda)
    x32 = torch.from_numpy(g["x"].astype(np.float32)).to(cuda)
    y32 = bsp.csr_spmv(rp, ci, v32, x32, algo="stream").cpu().numpy()
    assert np.array_equal(y32.view(np.uint32), g["y_fp32"].view(np.uint32))
    y16 = bsp.csr_spmv(rp, ci, v32.half(), x32.half(), algo="stream").float().cpu().numpy()
    assert np.array_equal(y16.view(np.uint32), g["y_fp16"].view(np.uint32))


def test_stream_long_rows_bit_exact(cuda):
    """Rows far longer than a 256-entry piece (and warps whose 32 rows span
    many pieces) give the scalar kernel's results exactly."""
    A = bsp.gen_powerlaw(200000, 1.6, 100000, 12)
    assert np.diff(A.rowptr).max() > 10000
    x = bsp.gen_uniform(A.cols, 13)
    ref = pyoracle.spmv_f64(A.rowptr, A.colidx, A.values, x)
    rp, ci, va, xx = _dev(cuda, A.rowptr, A.colidx, A.values, x)
    y = bsp.csr_spmv(rp, ci, va, xx, algo="stream").cpu().numpy()
    assert np.array_equal(y, ref)
    ys = bsp.csr_spmv(rp, ci, va, xx, algo="scalar").cpu().numpy()
    assert np.array_equal(y, ys)


@pytest.mark.parametrize("rows", [1, 31, 33, 1000])
def test_stream_ragged_tail_warp(cuda, rows):
    """Row counts that leave the last warp partly empty."""
    rng = np.random.default_rng(rows)
    lens = rng.integers(0, 40, rows)
    rp = np.zeros(rows + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    cols = 500
    ci = np.concatenate([np.sort(rng.choice(cols, l, replace=False)) for l in lens]).astype(np.int32)
    va = rng.standard_normal(ci.size)
    x = rng.uniform(-1, 1, cols)
    ref = pyoracle.spmv_f64(rp, ci, va, x)
    d = _dev(cuda, rp, ci, va, x)
    y = bsp.csr_spmv(*d, algo="stream").cpu().numpy()
    assert np.array_equal(y, ref)


@pytest.mark.parametrize("name", SPMV)
@pytest.mark.parametrize("algo,lanes", [("vector", 0), ("vector", 1), ("vector", 4), ("vector", 32),
                                        ("merge", 0)])
def test_fp64_kernels_within_rounding_bound(cuda, golden, name, algo, lanes):
    g = golden(name)
    rp, ci, va, x = _dev(cuda, g["rowptr"], g["colidx"], g["values"], g["x"])
    y = bsp.csr_spmv(rp, ci, va, x, algo=algo, lanes=lanes).cpu().numpy()
    tol = pyoracle.spmv_tolerance(g["rowptr"], g["colidx"], g["values"], g["x"])
    _within(y, g["y_fp64"], tol)


@pytest.mark.parametrize("name", SPMV)
def test_scalar_fp32_and_fp16_bit_exact_with_reference(cuda, golden, name):
    import torch
    g = golden(name)
    rp, ci = _dev(cuda, g["rowptr"], g["colidx"])
    v32 = torch.from_numpy(g["values"].astype(np.float32)).to(cuda)
    x32 = torch.from_numpy(g["x"].astype(np.float32)).to(cuda)
    y32 = bsp.csr_spmv(rp, ci, v32, x32, algo="scalar").cpu().numpy()
    assert np.array_equal(y32.view(np.uint32), g["y_fp32"].view(np.uint32))
    y16 = bsp.csr_spmv(rp, ci, v32.half(), x32.half(), algo="scalar").float().cpu().numpy()
    assert np.array_equal(y16.view(np.uint32), g["y_fp16"].view(np.uint32))


@pytest.mark.parametrize("dt", ["float32", "float16", "bfloat16"])
def test_reduced_precision_vector_kernels(cuda, dt):
    import torch
    A = bsp.gen_powerlaw(50000, 2.0, 2000, 5)
    x = bsp.gen_uniform(A.cols, 6)
    ref = pyoracle.spmv_f64(A.rowptr, A.colidx, A.values, x)
    tdt = getattr(torch, dt)
    rp, ci = _dev(cuda, A.rowptr, A.colidx)
    v = torch.from_numpy(A.values).to(cuda).to(tdt)
    xx = torch.from_numpy(x).to(cuda).to(tdt)
    y = bsp.csr_spmv(rp, ci, v, xx).double().cpu().numpy()
    # storage rounding of values and x (2 * unit) plus FP32 accumulation
    unit = {"float32": 2.0 ** -24, "float16": 2.0 ** -11, "bfloat16": 2.0 ** -8}[dt]
    scale = pyoracle.abs_rowsum(A.rowptr, A.colidx, A.values, x)
    out_round = unit * np.abs(ref)
    tol = (3 * unit + 2 * np.diff(A.rowptr) * 2.0 ** -24) * scale + out_round + 1e-30
    _within(y, ref, tol * 1.01)


@pytest.mark.parametrize("algo", ["vector", "merge", "scalar", "stream"])
def test_laplace_512_config(cuda, algo):
    A = bsp.gen_laplace2d(512, 512)
    x = bsp.gen_uniform(A.cols, 20261203)
    ref = pyoracle.spmv_f64(A.rowptr, A.colidx, A.values, x)
    rp, ci, va, xx = _dev(cuda, A.rowptr, A.colidx, A.values, x)
    y = bsp.csr_spmv(rp, ci, va, xx, algo=algo).cpu().numpy()
    if algo in ("scalar", "stream"):
        assert np.array_equal(y, ref)
    else:
        _within(y, ref, pyoracle.spmv_tolerance(A.rowptr, A.colidx, A.values, x))


def test_merge_path_power_law_long_rows(cuda):
    A = bsp.gen_powerlaw(200000, 1.6, 100000, 12)
    assert np.diff(A.rowptr).max() > 10000
    x = bsp.gen_uniform(A.cols, 13)
    ref = pyoracle.spmv_f64(A.rowptr, A.colidx, A.values, x)
    rp, ci, va, xx = _dev(cuda, A.rowptr, A.colidx, A.values, x)
    tol = pyoracle.spmv_tolerance(A.rowptr, A.colidx, A.values, x)
    _within(bsp.csr_spmv_merge(rp, ci, va, xx).cpu().numpy(), ref, tol)
    # lanes 1 / 4 / auto: rows above 64 entries per lane go to the whole warp
    for lanes in (32, 4, 1, 0):
        _within(bsp.csr_spmv(rp, ci, va, xx, algo="vector", lanes=lanes).cpu().numpy(), ref, tol)


@pytest.mark.parametrize("lanes", [1, 2, 8])
def test_vector_warp_rows_alpha_beta(cuda, lanes):
    """Rows just above and below the whole-warp threshold (64 entries per
    lane), with alpha and beta, in every position of a warp's row group."""
    import torch
    rng = np.random.default_rng(lanes)
    n, cols = 700, 5000
    lens = rng.integers(0, 8, n)
    thr = 64 * lanes
    lens[rng.choice(n, 60, replace=False)] = rng.choice([thr - 1, thr, thr + 1, 3 * thr + 7], 60)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    ci = np.concatenate([np.sort(rng.choice(cols, l, replace=False)) for l in lens]).astype(np.int32)
    va = rng.standard_normal(ci.size)
    x = rng.uniform(-1, 1, cols)
    y0 = rng.uniform(-1, 1, n)
    ref = 1.5 * pyoracle.spmv_f64(rp, ci, va, x) + 0.25 * y0
    d = _dev(cuda, rp, ci, va, x)
    y = torch.from_numpy(y0.copy()).to(cuda)
    bsp.csr_spmv(*d, y=y, alpha=1.5, beta=0.25, algo="vector", lanes=lanes)
    tol = 1.5 * pyoracle.spmv_tolerance(rp, ci, va, x) + 4 * 2.0 ** -53 * (np.abs(ref) + 1)
    _within(y.cpu().numpy(), ref, tol)


@pytest.mark.parametrize("algo", ["vector", "merge", "scalar", "stream"])
def test_alpha_beta_and_empty_rows(cuda, algo):
    import torch
    rng = np.random.default_rng(0)
    n = 1000
    lens = rng.integers(0, 4, n)
    lens[:50] = 0
    lens[-50:] = 0
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    ci = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in lens]).astype(np.int32)
    va = rng.standard_normal(ci.size)
    x = rng.uniform(-1, 1, n)
    y0 = rng.uniform(-1, 1, n)
    ref = 2.5 * pyoracle.spmv_f64(rp, ci, va, x) - 0.5 * y0
    d = _dev(cuda, rp, ci, va, x)
    y = torch.from_numpy(y0.copy()).to(cuda)
    bsp.csr_spmv(*d, y=y, alpha=2.5, beta=-0.5, algo=algo)
    tol = 2.5 * pyoracle.spmv_tolerance(rp, ci, va, x) + 4 * 2.0 ** -53 * (np.abs(ref) + 1)
    _within(y.cpu().numpy(), ref, tol)


def test_empty_matrix(cuda):
    import torch
    rp = torch.zeros(101, dtype=torch.int32, device=cuda)
    ci = torch.zeros(0, dtype=torch.int32, device=cuda)
    va = torch.zeros(0, dtype=torch.float64, device=cuda)
    x = torch.ones(100, dtype=torch.float64, device=cuda)
    for algo in ("vector", "merge", "scalar", "stream"):
        y = torch.full((100,), 7.0, dtype=torch.float64, device=cuda)
        bsp.csr_spmv(rp, ci, va, x, y=y, algo=algo)
        assert torch.all(y == 0)


def test_merge_workspace_too_small_is_rejected(cuda):
    import torch
    A = bsp.gen_laplace2d(32, 32)
    d = _dev(cuda, A.rowptr, A.colidx, A.values, np.ones(A.cols))
    ws = torch.empty(8, dtype=torch.uint8, device=cuda)
    with pytest.raises(bsp.BspError):
        bsp.csr_spmv_merge(*d, workspace=ws)


# rows at the lengths where a row changes hands: 8 entries per lane, 16 per lane
# (the lanes' own / a warp), 512 (a warp / the CTA), several rounds of the CTA,
# more long rows in one CTA than its list holds, a ragged last CTA
@pytest.mark.parametrize("rows,cols,lens", [
    (1, 3000, [2500]), (300, 600, [16, 17, 8, 9, 0]), (257, 5000, [0, 1, 511, 512, 513, 3]), (520, 300, [33]),
    (700, 9000, [2, 0, 4097, 1, 1, 1, 600, 129]), (64, 4000, [257, 256, 2049])])
@pytest.mark.parametrize("lanes", [0, 1, 2, 8, 32])
@pytest.mark.parametrize("dt", ["float64", "float32", "float16", "bfloat16"])
def test_vector_long_rows(cuda, rows, cols, lens, lanes, dt):
    import torch
    rng = np.random.default_rng(rows + cols)
    lens = np.resize(np.array(lens), rows)
    rp = np.zeros(rows + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    ci = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in lens]).astype(np.int32)
    tdt = getattr(torch, dt)
    v, x, y0 = (torch.from_numpy(a).to(tdt) for a in (rng.standard_normal(ci.size), rng.uniform(-1, 1, cols),
                                                      rng.uniform(-1, 1, rows)))
    vh, xh, yh = (t.double().numpy() for t in (v, x, y0))
    ax = pyoracle.spmv_f64(rp, ci, vh, xh)
    d_rp, d_ci = _dev(cuda, rp, ci)
    y = y0.to(cuda)
    bsp.csr_spmv(d_rp, d_ci, v.to(cuda), x.to(cuda), y, alpha=0.5, beta=-2.0, lanes=lanes)
    got = y.double().cpu().numpy()
    # the accumulation bound of A x, three roundings of alpha * (A x) + beta * y, one of the output
    unit = 2.0 ** -53 if dt == "float64" else 2.0 ** -24
    out = {"float64": 0.0, "float32": 0.0, "float16": 2.0 ** -11, "bfloat16": 2.0 ** -8}[dt]
    ref = 0.5 * ax - 2.0 * yh
    tol = 0.5 * pyoracle.spmv_tolerance(rp, ci, vh, xh, unit=unit) + \
        3 * unit * (np.abs(0.5 * ax) + np.abs(2.0 * yh)) + 1.01 * out * np.abs(ref) + 2.0 ** -24 * (dt == "float16")
    _within(got, ref, tol)


# few long rows among rows of 0 to 3, so that the bound for a long row is 16
# entries per lane: rows at it, at the CTA's bound (512, with 8 and 16 lanes 128 per
# lane) and one past each, several rounds of the CTA, and more of them in one CTA
# than its list holds
@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("dt", ["float64", "float32", "float16"])
def test_vector_few_long_rows(cuda, lanes, dt):
    import torch
    rng = np.random.default_rng(lanes)
    bound, cta = 16 * lanes, 128 * max(lanes, 4)
    lens = np.resize([0, 3, 1, 2], 8000)
    lens[[0, 5, 9, 300, 301, 302, lens.size - 1]] = [bound, bound + 1, cta, cta + 1, 4097, 9000, cta + 1]
    lens[512:512 + 70] = bound + 1
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    assert 4 * rp[-1] // lens.size <= bound
    cols = 9500
    ci = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in lens]).astype(np.int32)
    v, x = (torch.from_numpy(a).to(getattr(torch, dt)) for a in (rng.standard_normal(ci.size), rng.uniform(-1, 1, cols)))
    vh, xh = (t.double().numpy() for t in (v, x))
    d_rp, d_ci = _dev(cuda, rp, ci)
    got = bsp.csr_spmv(d_rp, d_ci, v.to(cuda), x.to(cuda), lanes=lanes).double().cpu().numpy()
    ref = pyoracle.spmv_f64(rp, ci, vh, xh)
    unit = 2.0 ** -53 if dt == "float64" else 2.0 ** -24
    tol = pyoracle.spmv_tolerance(rp, ci, vh, xh, unit=unit) + \
        (1.01 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24 if dt == "float16" else 0.0)
    _within(got, ref, tol)


def _us_per_million(cuda, rows, length, dt):
    """Best time of csr_spmv per million nonzeros: `rows` rows of `length`
    consecutive columns around the diagonal."""
    import torch
    rp = torch.arange(0, rows * length + 1, length, dtype=torch.int32, device=cuda)
    start = torch.arange(rows, dtype=torch.int32, device=cuda).clamp(max=rows - length)
    ci = (start[:, None] + torch.arange(length, dtype=torch.int32, device=cuda)).reshape(-1)
    va = torch.ones(ci.numel(), dtype=dt, device=cuda)
    x, y = (torch.ones(rows, dtype=dt, device=cuda) for _ in range(2))
    best = float("inf")
    for _ in range(5):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        e[0].record()
        for _ in range(10):
            bsp.csr_spmv(rp, ci, va, x, y)
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best * 100 / (ci.numel() / 1e6)


@pytest.mark.parametrize("dt", ["float64", "float16"])
def test_rows_all_long_cost_no_more_per_entry(cuda, dt):
    """A nonzero of a matrix whose rows are all long takes no longer than one of
    rows of 200 (with every row left to the CTA it took 1.5x to 1.9x)."""
    import torch
    dt = getattr(torch, dt)
    assert _us_per_million(cuda, 60000, 600, dt) <= 1.25 * _us_per_million(cuda, 200000, 200, dt)


def test_lanes_out_of_range_are_refused(cuda):
    A = bsp.gen_laplace2d(8, 8)
    d = _dev(cuda, A.rowptr, A.colidx, A.values, np.ones(A.cols))
    for lanes in (3, 64, 512):
        with pytest.raises(bsp.BspError):
            bsp.csr_spmv(*d, lanes=lanes)


def _few_long(kind, lanes, sms):
    """Row lengths: "own": rows above 16 entries in CTAs of 256 rows with none, one and
    only rows above 64; "short": rows far below the lanes' 8 entries each, some at and
    past 4 per lane; "queue": more rows than the warps of one launch, and rows past 512
    among them, several of one CTA."""
    if kind == "own":
        n = np.resize([2, 0, 1, 3], 1100)
        n[[3, 17, 255]] = [17, 64, 33]
        n[[256, 300, 511]] = [17, 65, 64]
        n[[600, 700]] = [600, 70]
        n[1099] = 64
    elif kind == "short":
        n = np.resize([lanes, 0, 2 * lanes, 1], 3000)
        n[[0, 7, 8, 2999]] = [4 * lanes, 4 * lanes + 1, 12 * lanes, 5 * lanes - 1]
    else:
        warps = sms * 64 * 8
        n = np.resize([1, 0, 2], 2 * warps + 13)
        n[[0, 1, 8, warps, warps + 1, 2 * warps, n.size - 1]] = [513, 512, 9000, 600, 3, 2000, 513]
    return n


@pytest.mark.parametrize("kind,lanes", [("own", 1), ("short", 2), ("short", 4), ("short", 8), ("short", 16),
                                        ("short", 32), ("queue", 32)])
@pytest.mark.parametrize("dt", ["float64", "float32", "float16"])
def test_vector_rows_by_length(cuda, kind, lanes, dt):
    import torch
    rng = np.random.default_rng(lanes)
    lens = _few_long(kind, lanes, torch.cuda.get_device_properties(0).multi_processor_count)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = 9500
    ci = rng.integers(0, cols, rp[-1]).astype(np.int32)
    v, x = (torch.from_numpy(a).to(getattr(torch, dt)) for a in (rng.standard_normal(ci.size), rng.uniform(-1, 1, cols)))
    vh, xh = (t.double().numpy() for t in (v, x))
    d_rp, d_ci = _dev(cuda, rp, ci)
    y = torch.full((lens.size,), float("nan"), dtype=v.dtype, device=cuda)
    got = bsp.csr_spmv(d_rp, d_ci, v.to(cuda), x.to(cuda), y, lanes=lanes).double().cpu().numpy()
    ref = pyoracle.spmv_f64(rp, ci, vh, xh)
    unit = 2.0 ** -53 if dt == "float64" else 2.0 ** -24
    tol = pyoracle.spmv_tolerance(rp, ci, vh, xh, unit=unit) + \
        (1.01 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24 if dt == "float16" else 0.0)
    _within(got, ref, tol)


def _best_us(f):
    import torch
    best = float("inf")
    for _ in range(6):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        e[0].record()
        for _ in range(10):
            f()
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best * 100


def _rows_on_device(cuda, lens, cols, dt):
    """Rows of the given lengths, their columns spread evenly."""
    import torch
    lens = lens.to(cuda)
    rp = torch.zeros(lens.numel() + 1, dtype=torch.int64, device=cuda)
    rp[1:] = lens.cumsum(0)
    r = torch.repeat_interleave(torch.arange(lens.numel(), device=cuda), lens)
    k = torch.arange(int(rp[-1]), device=cuda) - rp[r]
    ci = (k * (cols // lens.clamp(min=1))[r] + r % 61).clamp(max=cols - 1)
    va, x, y = (torch.ones(n, dtype=dt, device=cuda) for n in (ci.numel(), cols, lens.numel()))
    return rp.int(), ci.int(), va, x, y


@pytest.mark.parametrize("dt", ["float64", "float16"])
def test_a_few_rows_above_16_do_not_go_to_the_list(cuda, dt):
    """2M rows, a tenth of them of 20 entries and the others empty: a nonzero takes
    no more than 1.6 times as long as one of rows of 16 (with the rows of 20 summed by a
    warp each after the pass 1.7 to 2.2 times)."""
    import torch
    dt = getattr(torch, dt)

    def per_nonzero(k):
        lens = torch.zeros(2000000, dtype=torch.int64)
        lens[::10] = k
        a = _rows_on_device(cuda, lens, 2000000, dt)
        return _best_us(lambda: bsp.csr_spmv(*a)) / a[1].numel()

    assert per_nonzero(20) <= 1.6 * per_nonzero(16)


def test_long_rows_among_long_rows_leave_their_warp(cuda):
    """200,000 rows of 130 on average, the longest 20,000 (FP64): at most 1.25 times the
    merge path, which splits such rows (with every row left to its warp 1.7 times)."""
    import torch
    g = torch.Generator().manual_seed(1)
    u = torch.rand(200000, generator=g, dtype=torch.float64).clamp(min=1e-9)
    a = _rows_on_device(cuda, (u ** (-1.0 / 0.6)).clamp(max=20000.0).long(), 200000, torch.float64)
    assert a[1].numel() > 128 * 200000
    assert _best_us(lambda: bsp.csr_spmv(*a)) <= 1.25 * _best_us(lambda: bsp.csr_spmv(*a, algo="merge"))


@pytest.mark.parametrize("dt,length", [("float32", 16), ("float32", 32), ("float32", 130), ("float16", 130)])
def test_lanes_from_the_mean_are_near_the_best(cuda, dt, length):
    """Rows of one length: no other number of lanes takes less than 0.87 of the time."""
    import torch
    dt = getattr(torch, dt)
    rows = 8000000 // length
    rp = torch.arange(0, rows * length + 1, length, dtype=torch.int32, device=cuda)
    start = torch.arange(rows, dtype=torch.int32, device=cuda).clamp(max=rows - length)
    ci = (start[:, None] + torch.arange(length, dtype=torch.int32, device=cuda)).reshape(-1)
    va = torch.ones(ci.numel(), dtype=dt, device=cuda)
    x, y = (torch.ones(rows, dtype=dt, device=cuda) for _ in range(2))
    auto = _best_us(lambda: bsp.csr_spmv(rp, ci, va, x, y))
    best = min(_best_us(lambda: bsp.csr_spmv(rp, ci, va, x, y, lanes=1 << k)) for k in range(6))
    assert best >= 0.87 * auto


def test_one_lane_on_long_rows_leaves_them_to_a_warp(cuda):
    """100,000 rows of 200, FP64, by 1 lane: at most 1.85 times the time of 32 (with rows of
    200 left to their lane 1.94 times)."""
    import torch
    a = _rows_on_device(cuda, torch.full((100000,), 200), 200000, torch.float64)
    one, all32 = (_best_us(lambda: bsp.csr_spmv(*a, lanes=k)) for k in (1, 32))
    assert one <= 1.85 * all32
