"""Performance cases of the public entry points, over the sizes they are used at.

Every case is one call (or the call pair) a user's program repeats: CSR SpMV
from a few thousand rows to tens of millions of nonzeros, BSR SpMV, CSR ->
BSR / DASP conversion, DASP SpMV, SpMM on power-law graphs and on 16x16
tiles, the batched launch, and a whole CG solve.  The matrices are the ones
bench.py and the tests use (grid stencils, Zipf row lengths, random tiles),
built here on the GPU from the seed.

listed() names twelve of them, draw() gives further ones of the same ranges,
prepare() builds what a program holds before the call (inputs and plans),
run() is one pass, work() the bytes and operations a pass cannot do without
and exact() its result in FP64 from plain torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import benchsp_b200 as bsp

DTYPES = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
VALUE_BYTES = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}
ZIPF_CAP = 10000        # longest row of the power-law matrices
GRAPH_DEGREE = 32.0     # mean out-degree of the SpMM graph
BATCH_ROWS = (1000, 65536)


def listed() -> list:
    return [
        # a small implicit step or a coarse multigrid level: launch latency
        {"name": "csr_laplace_64x64_f64", "kind": "csr", "matrix": "laplace2d", "nx": 64, "ny": 64, "dtype": "f64",
         "alpha": 1.0, "beta": 0.0},
        # the plain CSR configuration: 5-point Laplacian on a 512 x 512 grid
        {"name": "csr_laplace_512x512_f64", "kind": "csr", "matrix": "laplace2d", "nx": 512, "ny": 512,
         "dtype": "f64", "alpha": 1.0, "beta": 0.0},
        # web / social matrices: a few long rows among many short ones
        {"name": "csr_powerlaw_1M_f64", "kind": "csr", "matrix": "powerlaw", "n": 1 << 20, "dtype": "f64",
         "alpha": 1.0, "beta": 0.0},
        # half-precision CSR inside an iteration (y = alpha A x + beta y)
        {"name": "csr_stencil27_128_f16", "kind": "csr", "matrix": "stencil27", "n": 128, "dtype": "f16",
         "alpha": 0.5, "beta": 0.25},
        # finite elements with 4 unknowns per node: the headline BSR matrix
        {"name": "bsr4_stencil27_64_f64", "kind": "bsr", "n": 64, "bs": 4, "store": "f64"},
        # the same matrix after reassembly: CSR -> BSR on the device
        {"name": "convert_bsr4_stencil27_64", "kind": "convert", "to": "bsr4", "n": 64},
        # DASP on the power-law configuration (2M rows)
        {"name": "dasp_powerlaw_2M_f64", "kind": "dasp", "n": 1 << 21},
        # graph propagation: adjacency times a block of 128 features
        {"name": "spmm_graph_1M_N128_f16", "kind": "spmm", "n": 1 << 20, "N": 128, "dtype": "f16"},
        # block-sparse layer: 16x16 tiles times 64 columns
        {"name": "smat_tiles_512k_N64_f16", "kind": "smat", "block_rows": 32768, "per_row": 8, "fill": 1.0, "N": 64,
         "dtype": "f16"},
        # 512 independent matrices in one launch, one vector each
        {"name": "batch_512_f64", "kind": "batch", "count": 512, "dtype": "f64", "nrhs": 1},
        # the same with 8 right-hand sides in single precision
        {"name": "batch_512_f32_8rhs", "kind": "batch", "count": 512, "dtype": "f32", "nrhs": 8},
        # a whole solve to 1e-10: FP16 matrix, FP64 refinement
        {"name": "cg_poisson_128_f16", "kind": "cg", "n": 128, "mode": "f16"},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["csr", "csr", "csr", "bsr", "convert", "dasp", "spmm", "smat", "batch", "cg"])
    if kind == "csr":
        case = {"kind": "csr", "matrix": rng.choice(["laplace2d", "powerlaw", "stencil27"]),
                "dtype": rng.choice(["f64", "f64", "f32", "f16", "bf16"])}
        if case["matrix"] == "laplace2d":
            case.update(nx=_log_int(rng, 24, 1500), ny=_log_int(rng, 24, 1500))
        elif case["matrix"] == "powerlaw":
            case.update(n=_log_int(rng, 1 << 12, 1 << 21))
        else:
            case.update(n=_log_int(rng, 10, 128))
        case.update(zip(("alpha", "beta"), rng.choice([(1.0, 0.0), (1.0, 0.0), (0.5, 0.25)])))
        return case
    if kind == "bsr":
        return {"kind": "bsr", "n": _log_int(rng, 10, 64), "bs": rng.choice([4, 4, 8]),
                "store": rng.choice(["f64", "f64", "f16", "bf16"])}
    if kind == "convert":
        to = rng.choice(["bsr4", "bsr8", "dasp"])
        return {"kind": "convert", "to": to,
                "n": _log_int(rng, 1 << 13, 1 << 21) if to == "dasp" else _log_int(rng, 10, 62)}
    if kind == "dasp":
        return {"kind": "dasp", "n": _log_int(rng, 1 << 13, (1 << 21) - 1)}
    if kind == "spmm":
        return {"kind": "spmm", "n": _log_int(rng, 1 << 13, 1 << 20), "N": rng.choice([32, 64, 96, 128]),
                "dtype": rng.choice(["f16", "bf16"])}
    if kind == "smat":
        return {"kind": "smat", "block_rows": _log_int(rng, 1000, 32768), "per_row": rng.randint(2, 8),
                "fill": round(rng.uniform(0.3, 1.0), 3), "N": rng.choice([32, 64, 128, 256]),
                "dtype": rng.choice(["f16", "bf16"])}
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 30, 511), "dtype": rng.choice(["f64", "f32"]),
                "nrhs": rng.choice([1, 8])}
    return {"kind": "cg", "n": _log_int(rng, 24, 104), "mode": rng.choice(["fp64", "f32", "f16", "bf16"])}


# ---------------------------------------------------------------------------
# Matrices, built on the GPU: (rowptr int32, colidx int32) plus sizes.

def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rowptr(counts: torch.Tensor) -> torch.Tensor:
    rp = torch.zeros(counts.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=rp[1:])
    return rp.int()


def _grid(dims: tuple, offsets: list, dof: int = 1) -> tuple:
    """CSR structure of a grid stencil (`offsets` ascending, one coordinate
    per dimension) with `dof` unknowns per node, all coupled."""
    shape = torch.meshgrid(*[torch.arange(d, device="cuda") for d in dims], indexing="ij")
    cols, ok = [], []
    for off in offsets:
        c = torch.zeros_like(shape[0])
        inside = torch.ones_like(shape[0], dtype=torch.bool)
        for x, d, o in zip(shape, dims, off):
            c = c * d + (x + o)
            inside &= (x + o >= 0) & (x + o < d)
        cols.append(c.reshape(-1))
        ok.append(inside.reshape(-1))
    col, mask = torch.stack(cols, 1).int(), torch.stack(ok, 1)
    counts = mask.sum(1) * dof
    if dof > 1:
        nodes, k = col.shape
        d = torch.arange(dof, dtype=torch.int32, device="cuda")
        col = (col * dof)[:, None, :, None] + d[None, None, None, :]
        col = col.expand(nodes, dof, k, dof)
        mask = mask[:, None, :, None].expand(nodes, dof, k, dof)
        counts = counts.repeat_interleave(dof)
    return _rowptr(counts), col[mask].contiguous()


def _box(dims: int) -> list:
    offs = [()]
    for _ in range(dims):
        offs = [o + (d,) for o in offs for d in (-1, 0, 1)]
    return offs


def _star(dims: int) -> list:
    return [o for o in _box(dims) if sum(abs(d) for d in o) <= 1]


def _zipf_cdf(alpha: float, cap: int) -> np.ndarray:
    return np.cumsum(np.arange(1, cap + 1, dtype=np.float64) ** -alpha)


def _zipf_mean(alpha: float, cap: int) -> float:
    k = np.arange(1, cap + 1, dtype=np.float64)
    return float((k ** (1 - alpha)).sum() / (k ** -alpha).sum())


def _zipf_lengths(n: int, alpha: float, cap: int, g: torch.Generator) -> torch.Tensor:
    cdf = torch.from_numpy(_zipf_cdf(alpha, cap)).cuda()
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * cdf[-1]
    return (torch.searchsorted(cdf, u) + 1).clamp_(max=cap)


def _random_rows(lengths: torch.Tensor, cols, g: torch.Generator) -> tuple:
    """CSR with `lengths` uniform columns per row (repeats merged), ascending.
    `cols`: the column count, one number or one per row."""
    n = lengths.numel()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lengths)
    u = torch.rand(row.numel(), dtype=torch.float64, device="cuda", generator=g)
    limit = cols[row] if torch.is_tensor(cols) else cols
    key = torch.unique(row * (1 << 21) + (u * limit).long())
    return _rowptr(torch.bincount(key >> 21, minlength=n)), (key & ((1 << 21) - 1)).int()


def _graph_cap(n: int, alpha: float, mean: float) -> int:
    """Longest row that gives Zipf(alpha) lengths this mean."""
    k = np.arange(1, n + 1, dtype=np.float64)
    means = np.cumsum(k ** (1 - alpha)) / np.cumsum(k ** -alpha)
    return int(min(n, np.searchsorted(means, mean) + 1))


def _structure(case: dict, g: torch.Generator) -> tuple:
    m = case.get("matrix") or {"bsr": "stencil27x4", "dasp": "powerlaw", "cg": "poisson3d"}[case["kind"]]
    if m == "laplace2d":
        return _grid((case["ny"], case["nx"]), _star(2))
    if m == "poisson3d":
        return _grid((case["n"],) * 3, _star(3))
    if m == "stencil27":
        return _grid((case["n"],) * 3, _box(3))
    if m == "stencil27x4":
        return _grid((case["n"],) * 3, _box(3), 4)
    return _random_rows(_zipf_lengths(case["n"], 2.0, min(ZIPF_CAP, case["n"]), g), case["n"], g)


def _laplace_values(rp: torch.Tensor, ci: torch.Tensor, diag: float) -> torch.Tensor:
    return torch.where(_row_ids(rp) == ci, diag, -1.0).double()


def _row_ids(rp: torch.Tensor) -> torch.Tensor:
    return torch.repeat_interleave(torch.arange(rp.numel() - 1, device="cuda"), rp.diff())


def _uniform(shape, dtype: torch.dtype, g: torch.Generator) -> torch.Tensor:
    return (torch.rand(shape, device="cuda", generator=g, dtype=torch.float64) * 2 - 1).to(dtype)


def _normal(n: int, dtype: torch.dtype, g: torch.Generator) -> torch.Tensor:
    return torch.randn(n, device="cuda", generator=g, dtype=torch.float64).to(dtype)


def _tiles(case: dict, g: torch.Generator) -> tuple:
    """Rows of 16x16 tiles at random block columns (repeats merged), each tile
    filled to `fill`."""
    nb, k = case["block_rows"], case["per_row"]
    b = torch.randint(nb, (nb, k), device="cuda", generator=g).sort(1).values
    keep = torch.ones_like(b, dtype=torch.bool)
    keep[:, 1:] = b[:, 1:] != b[:, :-1]
    d = torch.arange(16, dtype=torch.int32, device="cuda")
    col = (b.int() * 16)[:, None, :, None] + d
    mask = keep[:, None, :, None].expand(nb, 16, k, 16)
    if case["fill"] < 1.0:
        mask = mask & (torch.rand((nb, 16, k, 16), device="cuda", generator=g) < case["fill"])
    counts = mask.sum((2, 3)).reshape(-1)
    return _rowptr(counts), col.expand(nb, 16, k, 16)[mask].contiguous()


def _batch(case: dict, g: torch.Generator) -> dict:
    """Half banded (width 3..27), half Zipf(2.2) row lengths capped at n, sizes
    log-uniform (the same for every seed: a program's batch keeps its shape);
    every array of the batch in one buffer, each matrix's part 16-entry
    aligned."""
    rng = random.Random(case["count"])
    n = [_log_int(rng, *BATCH_ROWS) for _ in range(case["count"])]
    width = [rng.randint(3, 27) if i % 2 == 0 else 0 for i in range(case["count"])]
    first = np.concatenate([[0], np.cumsum([(v + 15) // 16 * 16 for v in n])])
    dev = lambda v: torch.tensor(v, device="cuda")  # noqa: E731
    sizes = dev(n)
    mat = torch.repeat_interleave(torch.arange(len(n), device="cuda"), sizes)
    local = torch.arange(mat.numel(), device="cuda") - torch.repeat_interleave(sizes.cumsum(0) - sizes, sizes)
    w, cap = dev(width)[mat], sizes[mat]
    lo = (local - (w - 1) // 2).clamp_(min=0)
    band = torch.minimum(cap - 1, local + w // 2) - lo + 1
    cdf = torch.from_numpy(_zipf_cdf(2.2, BATCH_ROWS[1])).cuda()
    u = torch.rand(mat.numel(), dtype=torch.float64, device="cuda", generator=g) * cdf[cap - 1]
    length = torch.where(w > 0, band, torch.minimum(torch.searchsorted(cdf, u) + 1, cap))
    row = torch.repeat_interleave(torch.arange(mat.numel(), device="cuda"), length)
    k = torch.arange(row.numel(), device="cuda") - torch.repeat_interleave(length.cumsum(0) - length, length)
    u = torch.rand(row.numel(), dtype=torch.float64, device="cuda", generator=g)
    col = torch.where(w[row] > 0, lo[row] + k, (u * cap[row]).long())
    key = torch.unique(row * (1 << 17) + col)
    rp = torch.zeros(mat.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(key >> 17, minlength=mat.numel()), 0, out=rp[1:])
    dt = DTYPES[case["dtype"]]
    rhs = (case["nrhs"],) if case["nrhs"] > 1 else ()
    return {"n": n, "first": first, "mat": mat, "local": local, "rp": rp, "row": key >> 17,
            "ci": (key & ((1 << 17) - 1)).int(), "va": _normal(key.numel(), dt, g),
            "x": _uniform((int(first[-1]),) + rhs, dt, g), "dt": dt, "rhs": rhs}


# ---------------------------------------------------------------------------

def _inputs(case: dict, seed: int) -> dict:
    """The matrix and vectors of a case, from the seed alone."""
    g, kind = _gen(seed), case["kind"]
    if kind == "batch":
        return _batch(case, g)
    if kind == "smat":
        rp, ci = _tiles(case, g)
        dt = DTYPES[case["dtype"]]
        return {"rp": rp, "ci": ci, "va": _normal(ci.numel(), dt, g).double(),
                "B": _uniform((rp.numel() - 1, case["N"]), dt, g), "cols": rp.numel() - 1}
    if kind == "spmm":
        n, dt = case["n"], DTYPES[case["dtype"]]
        rp, ci = _random_rows(_zipf_lengths(n, 1.8, _graph_cap(n, 1.8, GRAPH_DEGREE), g), n, g)
        degree = rp.diff().double()
        return {"rp": rp, "ci": ci, "va": (1.0 / degree)[_row_ids(rp)].to(dt), "B": _uniform((n, case["N"]), dt, g),
                "cols": n}
    if kind == "convert":
        # reassembly: the same structure, the seed's values
        rp, ci = _structure(dict(case, matrix="powerlaw" if case["to"] == "dasp" else "stencil27x4"), _gen(case["n"]))
        return {"rp": rp, "ci": ci, "va": _normal(ci.numel(), torch.float64, g), "cols": rp.numel() - 1}
    rp, ci = _structure(case, g)
    n = rp.numel() - 1
    dt = DTYPES[case["dtype"]] if kind == "csr" else torch.float64
    if case.get("matrix") == "laplace2d":
        va = _laplace_values(rp, ci, 4.0).to(dt)
    elif kind == "cg":
        va = _laplace_values(rp, ci, 6.0)
    else:
        va = _normal(ci.numel(), dt, g)
    s = {"rp": rp, "ci": ci, "va": va, "x": _uniform(n, dt, g), "cols": n}
    if kind == "csr":
        s["y"] = _uniform(n, dt, g)
    return s


def prepare(case: dict, seed: int) -> dict:
    s = _inputs(case, seed)
    s["case"], kind = case, case["kind"]
    if kind == "batch":
        starts = s["rp"][torch.tensor(np.cumsum([0] + s["n"]), device="cuda")].tolist()
        s["y"] = torch.zeros_like(s["x"])
        mats, r0 = [], 0
        for i, n in enumerate(s["n"]):
            a, b, f = starts[i], starts[i + 1], int(s["first"][i])
            rp = (s["rp"][r0:r0 + n + 1] - a).int()
            mats.append((rp, s["ci"][a:b].clone(), s["va"][a:b].clone(), s["x"][f:f + n], s["y"][f:f + n]))
            r0 += n
        s["plan"] = bsp.BatchPlan(mats, nrhs=case["nrhs"])
        return {k: s[k] for k in ("case", "plan", "x", "y")}
    if kind == "bsr":
        s["M"] = bsp.csr2bsr(s["rp"], s["ci"], s["va"], rows=s["cols"], cols=s["cols"], bs=case["bs"])
        if case["store"] != "f64":
            s["M"] = s["M"].scaled(case["store"])
        return {"case": case, "M": s["M"], "x": s["x"], "y": torch.empty_like(s["x"])}
    if kind == "dasp":
        M = bsp.csr2dasp(s["rp"], s["ci"], s["va"], rows=s["cols"], cols=s["cols"])
        return {"case": case, "M": M, "x": s["x"], "y": torch.empty_like(s["x"])}
    if kind == "spmm":
        s["plan"] = bsp.SpmmPlan(s["rp"], s["ci"], s["va"], cols=s["cols"])
        s["C"] = torch.empty(s["cols"], case["N"], dtype=torch.float32, device="cuda")
    if kind == "smat":
        M = bsp.SmatMatrix(s["rp"], s["ci"], s["va"], rows=s["cols"], cols=s["cols"], dtype=case["dtype"])
        C = torch.empty(s["cols"], case["N"], dtype=torch.float32, device="cuda")
        return {"case": case, "M": M, "B": s["B"], "C": C}
    if kind == "cg":
        s["solver"] = bsp.CgSolver(s["rp"], s["ci"], s["va"], mode=case["mode"], tol=1e-10)
    return s


class _DeviceArray:
    """A matrix's device array for torch.as_tensor (no copy; the matrix lives
    as long as the tensor does)."""

    def __init__(self, owner, ptr: int, count: int, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(owner, ptr: int, count: int, typestr: str) -> torch.Tensor:
    if count == 0:
        return torch.empty(0, dtype=torch.float64 if typestr == "<f8" else torch.int32, device="cuda")
    return torch.as_tensor(_DeviceArray(owner, ptr, count, typestr), device="cuda")


def _converted(M, to: str) -> list:
    if to == "dasp":
        parts = [(M.long_val, M.fill0_nnz_long, "<f8"), (M.long_cid, M.fill0_nnz_long, "<i4"),
                 (M.reg_val, M.fill0_nnz_reg, "<f8"), (M.reg_cid, M.fill0_nnz_reg, "<i4"),
                 (M.block_ptr, M.blocknum + 1, "<i4"), (M.irreg_val, M.nnz_irreg, "<f8"),
                 (M.irreg_cid, M.nnz_irreg, "<i4"), (M.irreg_rpt, M.row_block + 1, "<i4"),
                 (M.short_val, M.fill0_nnz_short, "<f8"), (M.short_cid, M.fill0_nnz_short, "<i4"),
                 (M.order_rid, M.rows, "<i4")]
    else:
        parts = [(M.blcPtr, M.blc_row + 1, "<i4"), (M.blcIdx, M.blc_num, "<i4"),
                 (M.blcVal, M.blc_num * M.bs * M.bs, "<f8"), (M.blcMap, M.blc_num, "<i2" if M.bs == 4 else "<i8"),
                 (M.rowPtrbyWarp, M.blc_row + 1, "<i4"), (M.rowIdxbyWarp, M.warpnum, "<i4")]
    return [_view(M, *p) for p in parts]


def run(s: dict):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "csr":
        return bsp.csr_spmv(s["rp"], s["ci"], s["va"], s["x"], s["y"], alpha=case["alpha"], beta=case["beta"])
    if kind in ("bsr", "dasp"):
        return s["M"].spmv(s["x"], s["y"])
    if kind == "convert":
        s.pop("M", None)     # the previous assembly's matrix is released first
        if case["to"] == "dasp":
            s["M"] = bsp.csr2dasp(s["rp"], s["ci"], s["va"], rows=s["cols"], cols=s["cols"])
        else:
            s["M"] = bsp.csr2bsr(s["rp"], s["ci"], s["va"], rows=s["cols"], cols=s["cols"], bs=int(case["to"][3:]))
        return _converted(s["M"], case["to"])
    if kind == "spmm":
        return s["plan"].spmm(s["B"], s["C"])
    if kind == "smat":
        return s["M"].spmm(s["B"], s["C"])
    if kind == "batch":
        s["plan"].run()
        return s["y"]
    return s["solver"].solve(s["x"])[0]


# ---------------------------------------------------------------------------

def _stencil_nnz(case: dict) -> tuple:
    n = case.get("n", 0)
    if case.get("matrix") == "laplace2d":
        nx, ny = case["nx"], case["ny"]
        return nx * ny, 5 * nx * ny - 2 * (nx + ny)
    if case.get("matrix") == "powerlaw" or case["kind"] == "dasp" or case.get("to") == "dasp":
        return n, int(n * _zipf_mean(2.0, min(ZIPF_CAP, n)))
    if case.get("matrix") == "stencil27":
        return n ** 3, (3 * n - 2) ** 3
    return 4 * n ** 3, 16 * (3 * n - 2) ** 3     # stencil27 with 4 unknowns per node


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "csr":
        rows, nnz = _stencil_nnz(case)
        v = VALUE_BYTES[case["dtype"]]
        return {"bytes": nnz * (v + 4) + 4 * (rows + 1) + rows * v * (3 if case["beta"] else 2), "flops": 2 * nnz}
    if kind in ("bsr", "convert") and case.get("to") != "dasp":
        rows, nnz = _stencil_nnz(case)
        n, bs = case["n"], case["bs"] if kind == "bsr" else int(case["to"][3:])
        blocks = (3 * n - 2) ** 3 if bs == 4 else max(1, 3 * n // 2 - 2) * (3 * n - 2) ** 2
        per_block = bs * bs * (2 if case.get("store", "f64") != "f64" else 8) + 4
        stored = blocks * per_block + 4 * (rows // bs + 1)
        if kind == "bsr":
            return {"bytes": stored + 16 * rows, "flops": 2 * nnz}
        return {"bytes": 12 * nnz + 4 * (rows + 1) + stored + blocks * (2 if bs == 4 else 8), "flops": 0}
    if kind in ("dasp", "convert"):
        rows, nnz = _stencil_nnz(case)
        csr = 12 * nnz + 4 * (rows + 1)
        return {"bytes": 2 * csr if kind == "convert" else csr + 16 * rows, "flops": 0 if kind == "convert" else 2 * nnz}
    if kind == "spmm":
        n, N = case["n"], case["N"]
        nnz = int(n * GRAPH_DEGREE)
        return {"bytes": 6 * nnz + 4 * (n + 1) + 6 * n * N, "flops": 2 * nnz * N}
    if kind == "smat":
        rows, tiles = 16 * case["block_rows"], case["block_rows"] * case["per_row"]
        return {"bytes": 516 * tiles + 6 * rows * case["N"], "flops": 2 * 256 * tiles * case["fill"] * case["N"]}
    if kind == "batch":
        lo, hi = BATCH_ROWS
        rows = (hi - lo) / math.log(hi / lo) * case["count"]
        nnz = rows * (0.5 * 15 + 0.5 * _zipf_mean(2.2, hi))
        v, k = VALUE_BYTES[case["dtype"]], case["nrhs"]
        return {"bytes": nnz * (v + 4) + 4 * rows + 2 * rows * v * k, "flops": 2 * nnz * k}
    n = case["n"]
    rows, nnz, steps = n ** 3, 7 * n ** 3 - 6 * n * n, 4.25 * n      # CG steps to 1e-10 grow with the grid's width
    v = 8 if case["mode"] == "fp64" else 4
    entry = {"fp64": 10, "f32": 6}.get(case["mode"], 4)
    return {"bytes": steps * (nnz * entry + 8 * rows * v), "flops": steps * (2 * nnz + 10 * rows)}


def _spmv_exact(rp, ci, va, x) -> torch.Tensor:
    y = torch.zeros((rp.numel() - 1,), dtype=torch.float64, device="cuda")
    return y.index_add_(0, _row_ids(rp), va.double() * x.double()[ci.long()])


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "convert":
        return None      # the arrays are copies of the inputs: compared as they are
    s = _inputs(case, seed)
    if kind == "batch":
        first = torch.from_numpy(s["first"]).cuda()[s["mat"]]
        src = s["x"].double()[first[s["row"]] + s["ci"].long()]
        va = s["va"].double()
        y = torch.zeros_like(s["x"], dtype=torch.float64)
        return y.index_add_(0, (first + s["local"])[s["row"]], src * (va[:, None] if s["rhs"] else va))
    if kind in ("spmm", "smat"):
        A = torch.sparse_csr_tensor(s["rp"].long(), s["ci"].long(), s["va"].double(),
                                    size=(s["rp"].numel() - 1, s["cols"]))
        return A @ s["B"].double()
    if kind == "cg":
        # A is diagonal in the sine basis of each direction
        n = case["n"]
        k = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
        S = torch.sin(torch.pi / (n + 1) * k[:, None] * k[None, :]) * math.sqrt(2.0 / (n + 1))
        lam = 2.0 - 2.0 * torch.cos(torch.pi / (n + 1) * k)

        def sines(t):
            for _ in range(3):      # one direction at a time, the axes in turn
                t = torch.einsum("ai,ijk->jka", S, t)
            return t

        t = sines(s["x"].reshape(n, n, n)) / (lam[:, None, None] + lam[None, :, None] + lam[None, None, :])
        return sines(t).reshape(-1)
    y = _spmv_exact(s["rp"], s["ci"], s["va"], s["x"])
    if kind == "csr":
        y = case["alpha"] * y + (case["beta"] * s["y"].double() if case["beta"] else 0.0)
    return y
