"""Performance cases of the engine: what a program that uses it has it do.

Each case is one call through the public entry points on seeded inputs:
  spmv     y = A x on a device-resident handle (DeviceMatrix.spmv), any format
  host     y = A x with page-locked host vectors (DeviceMatrix.spmv_host)
  batch    one product over a set of uneven matrices (Batch.spmv)
  convert  a format conversion on the device (convert.csr_from_coo, coo_from_csr, ell_from_csr, hybrid_from_csr)
over the matrix families of the engine's benchmark and tests: the 2-D 5-point
Laplacian, Zipf(2) power-law rows with uniform columns, the 27-point stencil,
a random band (32 of 129 columns per row) and rows of 4 to 64 uniform columns.
Matrices are built on the GPU with torch from the seed; values and x are
U[-1, 1].
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

DEVICE = "cuda"
HALF_BAND, PER_ROW = 64, 32
ZIPF_CLIP = 50_000
SPMV_FORMATS = ("csr", "csr_vector", "csr_adaptive", "ell", "coo", "scoo", "hybrid")
TORCH_DTYPE = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.float32, "f16": torch.float32}


# ---- the cases ---------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # a solver's inner product on a small grid: launch latency and host overhead
        {"name": "laplacian_128_csr_f32", "op": "spmv", "matrix": "laplacian", "n": 128, "format": "csr", "dtype": "f32"},
        # a small graph in FP64 through the format with the most launches; odd row count
        {"name": "power_law_100k_hybrid_f64", "op": "spmv", "matrix": "power_law", "n": 100_003, "format": "hybrid",
         "dtype": "f64"},
        # the benchmark's headline matrix in its fastest format
        {"name": "power_law_4M_coo_f32", "op": "spmv", "matrix": "power_law", "n": 4_194_304, "format": "coo",
         "dtype": "f32"},
        # the same matrix through the format the reference recommends for uneven rows
        {"name": "power_law_4M_csr_adaptive_f32", "op": "spmv", "matrix": "power_law", "n": 4_194_304,
         "format": "csr_adaptive", "dtype": "f32"},
        # a middle-sized graph in FP64, sliced COO, odd row count
        {"name": "power_law_1M_scoo_f64", "op": "spmv", "matrix": "power_law", "n": 1_048_583, "format": "scoo",
         "dtype": "f64"},
        # the reference operator's own contract: host x in, host y out
        {"name": "power_law_4M_hybrid_host_f32", "op": "host", "matrix": "power_law", "n": 4_194_304,
         "format": "hybrid", "dtype": "f32"},
        # a PDE stencil in the format made for it
        {"name": "stencil_128_ell_f32", "op": "spmv", "matrix": "stencil", "n": 128, "format": "ell", "dtype": "f32"},
        # the same operator in FP64 CSR on a grid of odd side
        {"name": "stencil_101_csr_vector_f64", "op": "spmv", "matrix": "stencil", "n": 101, "format": "csr_vector",
         "dtype": "f64"},
        # the largest matrix of the benchmark in the default format
        {"name": "banded_8M_csr_f32", "op": "spmv", "matrix": "banded", "n": 8_388_608, "format": "csr", "dtype": "f32"},
        # reduced-precision values and 16-bit column offsets
        {"name": "banded_1M_ell_bf16", "op": "spmv", "matrix": "banded", "n": 1_048_576, "format": "ell_lowp",
         "dtype": "bf16"},
        # many uneven matrices in one call
        {"name": "batch_64_f32", "op": "batch", "count": 64, "mix": 0, "dtype": "f32"},
        # what a Matrix Market reader hands over: triplets in any order into CSR
        {"name": "power_law_2M_triplets_to_csr_f32", "op": "convert", "matrix": "power_law", "n": 2_000_003, "to": "csr",
         "dtype": "f32"},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng: random.Random, kinds) -> dict:
    kind = rng.choice(kinds)
    if kind == "laplacian":
        n = _log_int(rng, 64, 1400)
    elif kind == "power_law":
        n = _log_int(rng, 20_000, 4_194_304)
    elif kind == "stencil":
        n = _log_int(rng, 24, 140)
    elif kind == "banded":
        n = _log_int(rng, 20_000, 8_388_608)
    else:
        n = _log_int(rng, 10_000, 2_000_000)
    return {"matrix": kind, "n": n}


def draw(rng: random.Random) -> dict:
    p = rng.random()
    if p < 0.64:
        c = {"op": "spmv", **_draw_matrix(rng, ("laplacian", "power_law", "power_law", "stencil", "banded", "uniform"))}
        formats = [f for f in SPMV_FORMATS if f != "ell" or c["matrix"] != "power_law"]
        c.update(format=rng.choice(formats), dtype=rng.choice(("f32", "f32", "f64")))
        if c["matrix"] == "banded" and c["dtype"] == "f64":
            c["n"] = min(c["n"], 5_000_000)
        return c
    if p < 0.76:
        kind = rng.choice(("stencil", "banded"))
        n = _log_int(rng, 24, 110) if kind == "stencil" else _log_int(rng, 20_000, 1_048_576)
        return {"op": "spmv", "matrix": kind, "n": n, "format": rng.choice(("ell_lowp", "csr_lowp")),
                "dtype": rng.choice(("bf16", "f16"))}
    if p < 0.82:
        c = {"op": "host", **_draw_matrix(rng, ("laplacian", "power_law", "stencil"))}
        formats = [f for f in SPMV_FORMATS if f != "ell" or c["matrix"] != "power_law"]
        return {**c, "format": rng.choice(formats), "dtype": rng.choice(("f32", "f64"))}
    if p < 0.89:
        return {"op": "batch", "count": _log_int(rng, 12, 64), "mix": rng.randrange(1, 1000),
                "dtype": rng.choice(("f32", "f64"))}
    to = rng.choice(("csr", "csr", "coo", "ell", "hybrid"))
    kinds = ("stencil", "laplacian") if to == "ell" else ("power_law", "stencil", "uniform")
    c = {"op": "convert", **_draw_matrix(rng, kinds)}
    if to == "csr" and c["matrix"] == "power_law":
        c["n"] = min(c["n"], 2_000_000)
    elif to == "csr" and c["matrix"] == "uniform":
        c["n"] = min(c["n"], 440_000)
    elif to == "csr":
        c["n"] = min(c["n"], 80)
    return {**c, "to": to, "dtype": rng.choice(("f32", "f32", "f64"))}


# ---- matrices (CSR on the GPU: row_ptr, columns, values in FP64) --------------
def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _uniform_values(n: int, g: torch.Generator) -> torch.Tensor:
    return torch.rand(n, generator=g, device=DEVICE, dtype=torch.float64) * 2.0 - 1.0


def _row_ptr(lengths: torch.Tensor) -> torch.Tensor:
    rp = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device=DEVICE)
    torch.cumsum(lengths, 0, out=rp[1:])
    return rp.to(torch.int32)


def _zipf_cdf(alpha: float, clip: int) -> torch.Tensor:
    """P(length <= k) of a Zipf(alpha) law on k >= 1 clipped to [1, clip]."""
    k = torch.arange(1, clip, dtype=torch.float64, device=DEVICE)
    zeta = float((torch.arange(1, 2_000_001, dtype=torch.float64, device=DEVICE) ** -alpha).sum())
    zeta += 2_000_000.0 ** (1.0 - alpha) / (alpha - 1.0)
    return torch.cumsum(k ** -alpha / zeta, 0)  # the remaining mass is the clip itself


def _from_lengths(rows: int, cols: int, lengths: torch.Tensor, g: torch.Generator):
    """Rows of the given lengths (in an order drawn here) with distinct, sorted, scattered columns:
    element j of a row of L takes a uniform column of the j-th of L equal parts."""
    lengths = lengths[torch.randperm(rows, generator=g, device=DEVICE)]
    rp = _row_ptr(lengths)
    row_length = torch.repeat_interleave(lengths, lengths)
    j = torch.arange(row_length.numel(), device=DEVICE) - torch.repeat_interleave(rp[:-1].long(), lengths)
    first = j * cols // row_length
    part = (j + 1) * cols // row_length - first
    u = torch.rand(part.numel(), generator=g, device=DEVICE, dtype=torch.float64)
    columns = first + torch.minimum((u * part).long(), part - 1)
    return rp, columns.to(torch.int32), _uniform_values(part.numel(), g)


def _power_law(rows: int, g: torch.Generator, alpha: float = 2.0, clip: int = ZIPF_CLIP):
    u = (torch.arange(rows, dtype=torch.float64, device=DEVICE) + 0.5) / rows  # the law's quantiles
    lengths = torch.searchsorted(_zipf_cdf(alpha, min(clip, rows)), u) + 1
    return _from_lengths(rows, rows, lengths, g)


def _uniform(rows: int, g: torch.Generator, lo: int = 4, hi: int = 64):
    lengths = lo + torch.arange(rows, device=DEVICE) % (hi - lo + 1)
    return _from_lengths(rows, rows, lengths, g)


def _grid(n: int, offsets, g: torch.Generator):
    """Neighbours `offsets` (lexicographic, so columns ascend) on an n^d grid."""
    d = len(offsets[0])
    rows = n ** d
    i = torch.arange(rows, device=DEVICE)
    coord = [(i // n ** (d - 1 - k)) % n for k in range(d)]
    keep, col = [], []
    for off in offsets:
        ok = torch.ones(rows, dtype=torch.bool, device=DEVICE)
        c = i.clone()
        for k, o in enumerate(off):
            t = coord[k] + o
            ok &= (t >= 0) & (t < n)
            c += o * n ** (d - 1 - k)
        keep.append(ok)
        col.append(c.to(torch.int32))
    keep, col = torch.stack(keep, 1), torch.stack(col, 1)
    columns = col[keep]
    return _row_ptr(keep.sum(1)), columns, _uniform_values(columns.numel(), g)


def _laplacian(n: int, g: torch.Generator):
    rp, ci, _ = _grid(n, [(-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)], g)
    rows = n * n
    r = torch.repeat_interleave(torch.arange(rows, device=DEVICE), (rp[1:] - rp[:-1]).long())
    return rp, ci, torch.where(ci == r, 4.0, -1.0).to(torch.float64)


def _stencil(n: int, g: torch.Generator):
    return _grid(n, [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)], g)


def _banded(rows: int, g: torch.Generator):
    width = 2 * HALF_BAND + 1
    columns = torch.empty((rows, PER_ROW), dtype=torch.int32, device=DEVICE)
    for r0 in range(0, rows, 1 << 20):
        r = torch.arange(r0, min(rows, r0 + (1 << 20)), device=DEVICE)
        pick = torch.rand((r.numel(), width), generator=g, device=DEVICE).topk(PER_ROW, dim=1, sorted=False).indices
        first = (r - HALF_BAND).clamp(0, rows - width)
        columns[r0:r0 + r.numel()] = (first[:, None] + pick.sort(dim=1).values).to(torch.int32)
    lengths = torch.full((rows,), PER_ROW, dtype=torch.int64, device=DEVICE)
    return _row_ptr(lengths), columns.view(-1), _uniform_values(rows * PER_ROW, g)


def _blocks(rows: int, g: torch.Generator, b: int = 32):
    r = torch.arange(rows, device=DEVICE)
    first = r // b * b
    lengths = torch.minimum(first + b, torch.tensor(rows, device=DEVICE)) - first
    rp = _row_ptr(lengths)
    row = torch.repeat_interleave(r, lengths)
    ci = first[row] + torch.arange(row.numel(), device=DEVICE) - rp[row].long()
    return rp, ci.to(torch.int32), _uniform_values(row.numel(), g)


def _tridiagonal(rows: int, g: torch.Generator):
    return _grid(rows, [(-1,), (0,), (1,)], g)


def _matrix(case: dict, g: torch.Generator):
    n = case["n"]
    make = {"laplacian": _laplacian, "power_law": _power_law, "stencil": _stencil, "banded": _banded,
            "uniform": _uniform}[case["matrix"]]
    rp, ci, v = make(n, g)
    return rp, ci, v.to(TORCH_DTYPE[case["dtype"]])


def _batch_rows(case: dict) -> list[tuple[int, int]]:
    """(family, rows) per matrix: rows log-uniform in [1,000, 200,000]."""
    rng = random.Random(7919 * case["mix"] + case["count"])
    return [(rng.randrange(4), _log_int(rng, 1_000, 200_000)) for _ in range(case["count"])]


def _batch_matrices(case: dict, g: torch.Generator):
    out = []
    for family, rows in _batch_rows(case):
        make = (_uniform, lambda n, gen: _power_law(n, gen, 1.8, n), _tridiagonal, _blocks)[family]
        rp, ci, v = make(rows, g)
        out.append((rows, rp, ci, v.to(TORCH_DTYPE[case["dtype"]])))
    return out


def _vector(n: int, case: dict, g: torch.Generator) -> torch.Tensor:
    return _uniform_values(n, g).to(TORCH_DTYPE[case["dtype"]])


def _quantile_width(rp: torch.Tensor) -> int:
    """The hybrid's ELL width: the 2/3-quantile of the row lengths."""
    lengths = (rp[1:] - rp[:-1]).sort().values
    return int(lengths[min(lengths.numel() - 1, int(2 * lengths.numel() / 3))])


def _host(t: torch.Tensor, dtype=None) -> np.ndarray:
    a = t.cpu().numpy()
    return a if dtype is None else a.view(dtype)


# ---- inputs and calls ----------------------------------------------------------
def _handle(case: dict, rp, ci, v):
    from matrix_format_performance_b200 import device
    from matrix_format_performance_b200.formats import csr_matrix_class
    rows = rp.numel() - 1
    if case["format"] in ("ell_lowp", "csr_lowp"):
        m = csr_matrix_class.from_arrays(rows, rows, _host(rp, np.uint32), _host(ci, np.uint32), _host(v))
        vt = device.BF16 if case["dtype"] == "bf16" else device.F16
        build = device.DeviceMatrix.from_ell_lowp if case["format"] == "ell_lowp" else device.DeviceMatrix.from_csr_lowp
        return build(m, vt, True)
    width = _quantile_width(rp) if case["format"] == "hybrid" else None
    return device.DeviceMatrix.from_device_csr(rp, ci, v, rows, device.FORMAT_NAMES[case["format"]], ell_width=width)


def _triplets(rp, ci, v, g):
    row = torch.repeat_interleave(torch.arange(rp.numel() - 1, device=DEVICE, dtype=torch.int32), (rp[1:] - rp[:-1]).long())
    order = torch.randperm(ci.numel(), generator=g, device=DEVICE)
    return row[order], ci[order], v[order].to(torch.float64)


def prepare(case: dict, seed: int) -> dict:
    g = _generator(seed)
    s = {"case": case}
    if case["op"] == "batch":
        from matrix_format_performance_b200.batch import Batch
        from matrix_format_performance_b200.formats import csr_matrix_class
        mats = _batch_matrices(case, g)
        total = sum(m[0] for m in mats)
        s["batch"] = Batch([csr_matrix_class.from_arrays(rows, rows, _host(rp, np.uint32), _host(ci, np.uint32), _host(v))
                            for rows, rp, ci, v in mats])
        s["x"] = _vector(total, case, g)
        s["y"] = torch.empty(total, dtype=s["x"].dtype, device=DEVICE)
        return s
    rp, ci, v = _matrix(case, g)
    rows = rp.numel() - 1
    if case["op"] == "convert":
        s["rows"] = rows
        s["in"] = _triplets(rp, ci, v, g) if case["to"] == "csr" else (rp, ci, v)
        s["dtype"] = v.dtype
        s["width"] = _quantile_width(rp)
        return s
    s["handle"] = _handle(case, rp, ci, v)
    x = _vector(rows, case, g)
    if case["op"] == "host":
        s["keep"] = x.cpu().pin_memory(), torch.empty(rows, dtype=x.dtype).pin_memory()
        s["x"], s["y"] = (t.numpy() for t in s["keep"])
    else:
        s["x"], s["y"] = x, torch.empty(rows, dtype=x.dtype, device=DEVICE)
    return s


def run(s: dict):
    op = s["case"]["op"]
    if op == "spmv":
        s["handle"].spmv(s["x"], s["y"])
        return s["y"]
    if op == "host":
        s["handle"].spmv_host(s["x"], s["y"])
        return s["y"]
    if op == "batch":
        s["batch"].spmv(s["x"], s["y"])
        return s["y"]
    from matrix_format_performance_b200 import convert
    to = s["case"]["to"]
    if to == "csr":
        return convert.csr_from_coo(s["rows"], s["rows"], *s["in"], dtype=s["dtype"])
    if to == "coo":
        return convert.coo_from_csr(*s["in"])
    if to == "ell":
        return convert.ell_from_csr(*s["in"])
    (ed, ec), (cd, cc, cr) = convert.hybrid_from_csr(*s["in"], s["width"])
    return ed, ec, cd, cc, cr


# ---- work and exact results ------------------------------------------------------
def _zipf_mean(alpha: float, clip: int) -> float:
    zeta = sum(k ** -alpha for k in range(1, 200_001)) + 200_000.0 ** (1.0 - alpha) / (alpha - 1.0)
    k = np.arange(1, clip, dtype=np.float64)
    p = k ** -alpha / zeta
    return float((k * p).sum() + clip * (1.0 - p.sum()))


def _size(kind: str, n: int) -> tuple[int, int]:
    """(rows, expected nonzeros)."""
    if kind == "laplacian":
        return n * n, 5 * n * n - 4 * n
    if kind == "stencil":
        return n ** 3, (3 * n - 2) ** 3
    if kind == "banded":
        return n, n * PER_ROW
    if kind == "uniform":
        return n, n * 34
    return n, int(n * _zipf_mean(2.0, min(ZIPF_CLIP, n)))


def work(case: dict) -> dict:
    val = {"f32": 4, "f64": 8, "bf16": 2, "f16": 2}[case["dtype"]]
    vec = 8 if case["dtype"] == "f64" else 4
    if case["op"] == "batch":
        rows = nnz = 0
        for family, r in _batch_rows(case):
            rows += r
            nnz += (34 * r, int(r * _zipf_mean(1.8, r)), 3 * r, 32 * r)[family]
        return {"bytes": nnz * (val + 4) + rows * (4 + 2 * vec), "flops": 2 * nnz}
    rows, nnz = _size(case["matrix"], case["n"])
    if case["op"] == "convert":
        if case["to"] == "csr":
            return {"bytes": nnz * (16 + 4 + val) + 4 * rows, "flops": 0}
        extra = {"coo": 4, "ell": 0, "hybrid": 2}[case["to"]]  # row ids of the COO part
        return {"bytes": nnz * (2 * (4 + val) + extra) + 4 * rows, "flops": 0}
    if case["op"] == "host":  # the handle's arrays, and x in and y out over the host link too
        return {"bytes": nnz * (val + 4) + rows * (4 + 4 * vec), "flops": 2 * nnz}
    if case["format"] in ("ell_lowp", "csr_lowp"):  # 16-bit values and offsets, an FP32 scale per row
        return {"bytes": nnz * 4 + rows * 12, "flops": 2 * nnz}
    return {"bytes": nnz * (val + 4) + rows * (4 + 2 * vec), "flops": 2 * nnz}


def _product(rp, ci, v, x) -> torch.Tensor:
    rows = rp.numel() - 1
    r = torch.repeat_interleave(torch.arange(rows, device=DEVICE), (rp[1:] - rp[:-1]).long())
    y = torch.zeros(rows, dtype=torch.float64, device=DEVICE)
    return y.index_add_(0, r, v.double() * x.double()[ci.long()])


def _rounded_values(case: dict, rp, v):
    """What the 16-bit layouts store: a / scale rounded to FP32, then to 16 bits, times the row's scale."""
    rows = rp.numel() - 1
    r = torch.repeat_interleave(torch.arange(rows, device=DEVICE), (rp[1:] - rp[:-1]).long())
    a = v.double()
    scale = torch.zeros(rows, dtype=torch.float64, device=DEVICE).scatter_reduce_(0, r, a.abs(), "amax")
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))[r]
    q = (a / scale).float().to(torch.bfloat16 if case["dtype"] == "bf16" else torch.float16)
    return q.double() * scale


def exact(case: dict, seed: int):
    if case["op"] == "convert":  # index arrays and copied values: nothing is computed
        return None
    g = _generator(seed)
    if case["op"] == "batch":
        mats = _batch_matrices(case, g)
        x = _vector(sum(m[0] for m in mats), case, g)
        out, at = [], 0
        for rows, rp, ci, v in mats:
            out.append(_product(rp, ci, v, x[at:at + rows]))
            at += rows
        return torch.cat(out)
    rp, ci, v = _matrix(case, g)
    x = _vector(rp.numel() - 1, case, g)
    if case["format"] in ("ell_lowp", "csr_lowp"):
        v = _rounded_values(case, rp, v)
    return _product(rp, ci, v, x)
