"""SCOO handles whose slices run as warp tiles, against one CTA per slice."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import formats as F  # noqa: E402
from matrix_format_performance_b200._capi import MfpError, ScooParams, call  # noqa: E402
from matrix_format_performance_b200.device import SCOO, DeviceMatrix  # noqa: E402


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def raw_scoo(s, m, x):
    """y from the raw entry point, which keeps one CTA per slice."""
    keep = [dev(a) for a in (s.values, s.c_index.view(np.int32), s.r_index.view(np.int32), s.slices_ptr.view(np.int32), x)]
    y = torch.full((m.rows,), float("nan"), dtype=keep[0].dtype, device="cuda")
    v, ci, ri, sp, xt = (C.c_void_p(t.data_ptr()) for t in keep)
    call(f"mfp_scoo_spmv_{'f32' if m.dtype == np.float32 else 'f64'}", m.rows, m.cols, s.slices_count, s.slice_size, v, ci,
         ri, sp, None, 0, None, xt, C.c_void_p(y.data_ptr()), None)
    torch.cuda.synchronize()
    return y.cpu().numpy()


def handle_spmv(dm, m, x):
    xt, y = dev(x), torch.full((m.rows,), float("nan"), dtype=dev(x).dtype, device="cuda")
    dm.spmv(xt, y)
    torch.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_rows_of_negative_zero_products(dtype):
    """Rows whose products are all -0 (one, several, a whole tile and more of
    them) have the sign that one CTA per slice gives them."""
    rng = np.random.default_rng(12)
    lens = rng.integers(0, 9, 3000)
    lens[700] = 20_000  # uneven slices: the handle runs tiles
    lens[[40, 1400, 2999]] = 300, 700, 1
    lens[[10, 11, 12]] = 1, 2, 8
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    n, cols = int(rp[-1]), 500
    v = rng.uniform(0.5, 1, n)
    row = np.repeat(np.arange(3000), lens)
    zero_rows = np.isin(row, [10, 11, 12, 40, 1400, 2999]) | (row % 5 == 0)
    v[zero_rows] = -0.0
    m = F.csr_matrix_class.from_arrays(3000, cols, rp, rng.integers(0, cols, n).astype(np.uint32), v, dtype)
    x = rng.uniform(0.5, 1, cols).astype(dtype)
    dm = DeviceMatrix.build(m, SCOO)
    assert dm.info().kernel_launches == 2  # tiles and fix-up
    y = handle_spmv(dm, m, x)
    dm.close()
    assert np.array_equal(y.view(np.uint8), raw_scoo(F.scoo_matrix_class(148, 49152, m), m, x).view(np.uint8))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_slices_beyond_shared_memory_are_refused(dtype):
    """A slice whose rows do not fit one CTA's shared memory is refused, whether or
    not its handle could run warp tiles."""
    rng = np.random.default_rng(4)
    rows = 60_000
    lens = rng.integers(0, 40, rows)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    m = F.csr_matrix_class.from_arrays(rows, 100, rp, rng.integers(0, 100, int(rp[-1])).astype(np.uint32),
                                       rng.uniform(-1, 1, int(rp[-1])), dtype)
    prm = ScooParams()
    prm.slices_count, prm.slice_size, prm.lane_size = 1, rows, 1
    dm = DeviceMatrix.from_device_csr(dev(m.row_ptr.view(np.int32)), dev(m.columns.view(np.int32)), dev(m.data), 100, SCOO,
                                      scoo=prm)
    with pytest.raises(MfpError, match="too large for shared memory"):
        handle_spmv(dm, m, np.ones(100, dtype))
    dm.close()


def pinned(n, dtype):
    return torch.full((n,), float("nan"), dtype=torch.float32 if dtype == np.float32 else torch.float64).pin_memory()


@pytest.mark.parametrize("longest", [64, 20_000])  # many rows and even slices; few rows and a heavy slice
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_host_vectors(oracle_lib, longest, dtype):
    """A tiled handle's product with host vectors, y page-locked or not, has the
    bits of the device call, whichever kernel stores it."""
    rng = np.random.default_rng(longest)
    rows = 400_000 if longest == 64 else 3_000
    lens = rng.integers(0, 6, rows)
    lens[rows // 2] = longest
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    m = F.csr_matrix_class.from_arrays(rows, rows, rp, rng.integers(0, rows, int(rp[-1])).astype(np.uint32),
                                       rng.uniform(-1, 1, int(rp[-1])), dtype)
    dm = DeviceMatrix.build(m, SCOO)
    assert dm.info().kernel_launches == 2  # tiles and fix-up
    x = rng.uniform(-1, 1, rows).astype(dtype)
    want = handle_spmv(dm, m, x)
    ys, ab = oracle_lib.csr_spmv_exact(m.rows, m.row_ptr, m.columns, m.data, x)
    assert np.all(np.abs(want.astype(np.float64) - ys) <= {np.float32: 1e-5, np.float64: 1e-12}[dtype] * ab)
    for y in (pinned(rows, dtype).numpy(), np.full(rows, np.nan, dtype)):
        dm.spmv_host(x, y)
        assert np.array_equal(y.view(np.uint8), want.view(np.uint8))
    dm.close()
