"""ELL on both sides of the row count from which an FP32 thread takes four rows,
with row counts that are no multiple of four and widths past the slots in flight."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import formats as F  # noqa: E402
from matrix_format_performance_b200.device import DeviceMatrix  # noqa: E402


@pytest.mark.parametrize("rows", [599_996, 600_000, 600_001, 600_002, 600_003])
@pytest.mark.parametrize("width", [15, 21])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_four_rows_per_thread(rows, width, dtype):
    """The bits of the slot loop in order, padding included."""
    rng = np.random.default_rng(rows + width)
    cols = 4_321
    e = F.ell_matrix_class.__new__(F.ell_matrix_class)
    e.rows, e.cols, e.dtype, e.elements_in_rows = rows, cols, np.dtype(dtype), width
    e.columns = rng.integers(0, cols, rows * width, dtype=np.uint32)
    e.data = rng.uniform(-1, 1, rows * width).astype(dtype)
    x = rng.uniform(-1, 1, cols).astype(dtype)
    dm = DeviceMatrix.from_ell(e)
    y = torch.full((rows,), float("nan"), dtype=torch.float32 if dtype == np.float32 else torch.float64, device="cuda")
    dm.spmv(torch.from_numpy(x).cuda(), y)
    torch.cuda.synchronize()
    dm.close()
    want = np.zeros(rows, dtype)
    for k in range(width):
        s = slice(k * rows, (k + 1) * rows)
        want = want + e.data[s] * x[e.columns[s]]
    assert np.array_equal(y.cpu().numpy().view(np.uint8), want.view(np.uint8))
