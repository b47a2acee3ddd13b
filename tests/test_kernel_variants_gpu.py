"""Kernel variants chosen by a matrix's sizes and structure, at the sizes where
they can go wrong: remainders, tile and slice edges, the ends of their ranges."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import formats as F  # noqa: E402
from matrix_format_performance_b200 import synth  # noqa: E402
from matrix_format_performance_b200._capi import call  # noqa: E402
from matrix_format_performance_b200.device import SCOO, DeviceMatrix  # noqa: E402

TOL = {np.float32: 1e-5, np.float64: 1e-12}  # per row, of sum |a_ij x_j|


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def p(t):
    return C.c_void_p(t.data_ptr())


def check(oracle_lib, m, x, y, what):
    ys, ab = oracle_lib.csr_spmv_exact(m.rows, m.row_ptr, m.columns, m.data, x)
    bad = ~(np.abs(y.astype(np.float64) - ys) <= TOL[m.dtype.type] * ab)
    assert not bad.any(), f"{what}: {int(bad.sum())} rows, first {int(np.argmax(bad))}"


def csr(lens, cols, dtype, seed=3):
    """Random columns (repeats allowed), values U[-1, 1]."""
    rng = np.random.default_rng(seed)
    rp = np.zeros(len(lens) + 1, np.int64)
    rp[1:] = np.cumsum(lens)
    row = np.repeat(np.arange(len(lens)), lens)
    c = rng.integers(0, cols, int(rp[-1]))
    c = c[np.lexsort((c, row))].astype(np.uint32)
    return F.csr_matrix_class.from_arrays(len(lens), cols, rp.astype(np.uint32), c, rng.uniform(-1, 1, len(c)), dtype)


def spmv(dm, m, x):
    xt, y = dev(x), torch.full((m.rows,), float("nan"), dtype=dev(x).dtype, device="cuda")
    dm.spmv(xt, y)
    torch.cuda.synchronize()
    return y.cpu().numpy()


def uneven_lengths(case):
    rng = np.random.default_rng(8)
    lens = rng.integers(0, 13, 3000)
    if case == "long_rows":     # crossing chains of 250, 36 and 2 tiles, one of them ending a slice
        lens[700], lens[1500], lens[2099] = 64_000, 9_001, 400
    elif case == "holes":       # empty slices (21 rows each) at the start, inside and at the end
        lens[:63], lens[1008:1050], lens[2900:] = 0, 0, 0
        lens[1700] = 20_011
    else:                       # one row holds almost everything
        lens[:] = 0
        lens[[5, 2999]] = 50_003, 1
    return lens


@pytest.mark.parametrize("case", ["long_rows", "holes", "one_row"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_scoo_tiles_give_the_bits_of_one_cta_per_slice(oracle_lib, case, dtype):
    """Uneven SCOO slices run as independent warp tiles; the raw entry point
    keeps one CTA per slice.  Same tiles, same order of a crossing row's
    partial sums: the same bits."""
    m = csr(uneven_lengths(case), 5_000, dtype)
    x = synth.vector(4, m.cols).astype(dtype)
    s = F.scoo_matrix_class(148, 49152, m)
    dm = DeviceMatrix.build(m, SCOO)
    assert dm.info().kernel_launches == 2  # tiles and fix-up
    y = spmv(dm, m, x)
    dm.close()
    keep = [dev(a) for a in (s.values, s.c_index.view(np.int32), s.r_index.view(np.int32), s.slices_ptr.view(np.int32), x)]
    raw = torch.full((m.rows,), float("nan"), dtype=keep[0].dtype, device="cuda")
    v, ci, ri, sp, xt = (p(t) for t in keep)
    call(f"mfp_scoo_spmv_{'f32' if dtype == np.float32 else 'f64'}", m.rows, m.cols, s.slices_count, s.slice_size, v, ci,
         ri, sp, None, 0, None, xt, p(raw), None)
    torch.cuda.synchronize()
    check(oracle_lib, m, x, y, case)
    assert np.array_equal(raw.cpu().numpy().view(np.uint8), y.view(np.uint8))


def test_scoo_tiles_on_two_streams_and_in_a_graph():
    """One handle used from two streams at once and from a captured graph:
    each call has its own carries."""
    m = csr(uneven_lengths("long_rows"), 5_000, np.float32)
    dm = DeviceMatrix.build(m, SCOO)
    xs = [dev(synth.vector(k, m.cols).astype(np.float32)) for k in range(3)]
    want = [spmv(dm, m, x.cpu().numpy()) for x in xs]
    ys = [torch.zeros(m.rows, device="cuda") for _ in xs]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        dm.spmv(xs[2], ys[2])
    for _ in range(20):
        for s, x, y in zip(streams, xs, ys):
            dm.spmv(x, y, s)
        graph.replay()
    torch.cuda.synchronize()
    del graph
    dm.close()
    for w, y in zip(want, ys):
        assert np.array_equal(w.view(np.uint32), y.cpu().numpy().view(np.uint32))


TILE = 6144  # keys per tile of the triplet sort


@pytest.mark.parametrize("n", [1, 31, 33, TILE - 1, TILE, TILE + 1, 40 * TILE + 17])
@pytest.mark.parametrize("rows, cols", [(2, 1), (1, 200), (3, 300), (500, 509), (70_000, 65_537), (1 << 20, 1 << 12),
                                        (1 << 24, 0xFFFFFFFF)])
def test_triplet_sort_digits_and_tiles(n, rows, cols):
    """CSR from triplets equals a stable host sort: element counts around the
    sort's tiles, key widths of 1 to 56 bits (1 to 7 digits of 8 or 9 bits,
    digits that straddle the key's halves), repeated entries in input order."""
    from matrix_format_performance_b200 import convert
    rng = np.random.default_rng(n + rows)
    r = rng.integers(0, rows, n).astype(np.uint32)
    c = rng.integers(0, cols, n, dtype=np.uint64).astype(np.uint32)
    r[n // 2:] = r[: n - n // 2]  # repeats
    c[n // 2:] = c[: n - n // 2]
    v = np.arange(n, dtype=np.float64)
    rp, co, d = convert.csr_from_coo(rows, cols, dev(r.view(np.int32)), dev(c.view(np.int32)), dev(v), dtype=torch.float64)
    order = np.lexsort((np.arange(n), c, r))
    want = np.zeros(rows + 1, np.int64)
    np.add.at(want, r.astype(np.int64) + 1, 1)
    assert np.array_equal(rp.cpu().numpy(), np.cumsum(want))
    assert np.array_equal(co.cpu().numpy().view(np.uint32), c[order])
    assert np.array_equal(d.cpu().numpy(), v[order])


NEVER = 0xFFFFFFFF


def short_lengths(case):
    rng = np.random.default_rng(21)
    if case == "two_lanes":       # 0 to 9 elements: 2 lanes per row
        return rng.integers(0, 10, 1001)
    if case == "sixteen_lanes":   # up to 64 elements, several passes; a last block of one row
        return np.concatenate([rng.integers(40, 65, 512), [64]])
    if case == "growing":         # every lane count, the last row ends the array inside a quad
        return np.concatenate([np.arange(65).repeat(40), [3]])
    lens = rng.integers(20, 40, 20 * 4096)  # mixed: blocks with longer rows between blocks without
    lens[300], lens[301], lens[1500], lens[3000:3010], lens[-1] = 65, 4_097, 20_000, 3_000, 66
    return lens


@pytest.mark.parametrize("case", ["two_lanes", "sixteen_lanes", "growing", "mixed"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_csr_short_rows_straight_from_memory(oracle_lib, case, dtype):
    """CSR plans without a configuration read row blocks of short rows straight
    from global memory.  CSR scalar keeps the bits of the exact-order setting
    (one thread per row) on rows up to 64 elements; every algorithm is within
    tolerance, also on arrays that are not 16-byte aligned."""
    from matrix_format_performance_b200.device import CSR_ADAPTIVE, CSR_SCALAR, CSR_VECTOR
    m = csr(short_lengths(case), 3_000, dtype)
    x = synth.vector(6, m.cols).astype(dtype)
    exact = DeviceMatrix.from_csr(m, CSR_SCALAR, {"long_row_threshold": NEVER, "assist_threshold": NEVER})
    want = spmv(exact, m, x)
    exact.close()
    short = np.diff(m.row_ptr.astype(np.int64)) <= 64
    sfx = "f32" if dtype == np.float32 else "f64"
    for fmt in (CSR_SCALAR, CSR_VECTOR, CSR_ADAPTIVE):
        dm = DeviceMatrix.from_csr(m, fmt)
        assert dm.info().kernel_launches == (2 if case == "mixed" else 1)
        y = spmv(dm, m, x)
        assert np.array_equal(y.view(np.uint8), spmv(dm, m, x).view(np.uint8))
        dm.close()
        check(oracle_lib, m, x, y, f"{case} {fmt}")
        if fmt == CSR_SCALAR:
            assert np.array_equal(y[short].view(np.uint8), want[short].view(np.uint8))
        plan = C.c_void_p()
        rp_host = np.ascontiguousarray(m.row_ptr)
        call("mfp_csr_plan_create", m.rows, m.cols, m.nnz, C.c_void_p(rp_host.ctypes.data), fmt, None, C.byref(plan))
        v = torch.zeros(m.nnz + 1, dtype=dev(m.data).dtype, device="cuda")
        c = torch.zeros(m.nnz + 1, dtype=torch.int32, device="cuda")
        v[1:], c[1:] = dev(m.data), dev(m.columns.view(np.int32))
        rp, xt = dev(m.row_ptr.view(np.int32)), dev(x)
        yt = torch.full((m.rows,), float("nan"), dtype=v.dtype, device="cuda")
        call(f"mfp_csr_spmv_{sfx}", plan, p(v[1:]), p(c[1:]), p(rp), p(xt), p(yt), None)
        torch.cuda.synchronize()
        call("mfp_csr_plan_destroy", plan)
        check(oracle_lib, m, x, yt.cpu().numpy(), f"unaligned {case} {fmt}")


@pytest.mark.parametrize("width", [1, 2, 3, 7, 8, 9, 15, 64])
@pytest.mark.parametrize("rows", [1, 255, 4_001, 600_000, 600_004])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_ell_widths_and_row_counts(width, rows, dtype):
    """ELL on both sides of the row count from which a thread takes four rows,
    at widths around the slots in flight: the bits of the slot loop in order,
    padding included."""
    from matrix_format_performance_b200.device import DeviceMatrix as D
    if rows > 10_000 and width > 9:
        rows = 600_000 // 4
    rng = np.random.default_rng(width + rows)
    cols = 777
    e = F.ell_matrix_class.__new__(F.ell_matrix_class)
    e.rows, e.cols, e.dtype, e.elements_in_rows = rows, cols, np.dtype(dtype), width
    e.columns = rng.integers(0, cols, rows * width).astype(np.uint32)
    e.data = rng.uniform(-1, 1, rows * width).astype(dtype)
    e.data[rng.random(rows * width) < 0.1] = 0
    x = rng.uniform(-1, 1, cols).astype(dtype)
    dm = D.from_ell(e)
    y = spmv(dm, e, x)
    dm.close()
    want = np.zeros(rows, dtype)
    for k in range(width):
        s = slice(k * rows, (k + 1) * rows)
        want = want + e.data[s] * x[e.columns[s]]
    assert np.array_equal(y.view(np.uint8), want.astype(dtype).view(np.uint8))


@pytest.mark.parametrize("rows, width", [(1, 3), (199_999, 9), (200_000, 8), (200_002, 7), (200_001, 12), (1_750_000, 5),
                                         (1_750_004, 4)])
@pytest.mark.parametrize("index16", [False, True])
@pytest.mark.parametrize("vt", [2, 3])
def test_lowp_ell_rows_per_thread(rows, width, index16, vt):
    """16-bit ELL on both sides of the row counts where a thread takes 1, 2 or 8
    rows, at widths around the slots in flight: the same bits whether the
    arrays' alignment lets a thread take several rows or not, and y within FP32
    rounding of the 64-bit product."""
    rng = np.random.default_rng(rows + width)
    cols = rows + 500
    n = rows * width
    off = rng.integers(-200, 200, n)
    off[rng.random(n) < 0.5] = 3  # runs of equal offsets
    row = np.tile(np.arange(rows), width)
    col = np.clip(row + off, 0, cols - 1)
    bits = torch.from_numpy(rng.uniform(-1, 1, n).astype(np.float32)).to(torch.bfloat16 if vt == 2 else torch.float16)
    scale = rng.uniform(0.5, 2, rows).astype(np.float32)
    x = rng.uniform(-1, 1, cols).astype(np.float32)
    idx = (col - row + 32768).astype(np.uint16) if index16 else col.astype(np.uint32)
    outs = []
    for shift in (0, 1):  # elements past an aligned start
        q = torch.zeros(n + 8, dtype=torch.int16, device="cuda")
        q[shift:shift + n] = bits.view(torch.int16).cuda()
        ix = torch.zeros(n + 8, dtype=torch.int16 if index16 else torch.int32, device="cuda")
        ix[shift:shift + n] = dev(idx.view(np.int16 if index16 else np.int32))
        sc, xt = dev(scale), dev(x)
        y = torch.full((rows,), float("nan"), device="cuda")
        call("mfp_lowp_ell_spmv", vt, rows, cols, width, p(q[shift:]), p(sc), None if index16 else p(ix[shift:]),
             p(ix[shift:]) if index16 else None, p(xt), p(y), None)
        torch.cuda.synchronize()
        outs.append(y.cpu().numpy())
    assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
    prod = bits.double().numpy() * x[col].astype(np.float64)
    want = prod.reshape(width, rows).sum(0) * scale
    bound = (width + 1) * 2.0 ** -23 * np.abs(prod).reshape(width, rows).sum(0) * scale
    assert np.all(np.abs(outs[0] - want) <= bound + 1e-30)
