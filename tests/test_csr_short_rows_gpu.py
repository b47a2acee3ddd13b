"""CSR row blocks read straight from global memory: every number of CTAs a block
is split into, and large matrices of which only part is such blocks."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import formats as F  # noqa: E402
from matrix_format_performance_b200 import synth  # noqa: E402
from matrix_format_performance_b200.device import CSR_ADAPTIVE, CSR_SCALAR, CSR_VECTOR, DeviceMatrix  # noqa: E402

TOL = {np.float32: 1e-5, np.float64: 1e-12}  # per row, of sum |a_ij x_j|
NEVER = 0xFFFFFFFF


def csr(lens, cols, dtype, seed=3):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    c = rng.integers(0, cols, int(rp[-1])).astype(np.uint32)
    return F.csr_matrix_class.from_arrays(len(lens), cols, rp, c, rng.uniform(-1, 1, len(c)), dtype)


def spmv(m, fmt, x, launches, config=None):
    dm = DeviceMatrix.from_csr(m, fmt, config)
    if launches:
        assert dm.info().kernel_launches == launches
    xt = torch.from_numpy(x).cuda()
    y = torch.full((m.rows,), float("nan"), dtype=xt.dtype, device="cuda")
    dm.spmv(xt, y)
    torch.cuda.synchronize()
    dm.close()
    return y.cpu().numpy()


def check(oracle_lib, m, x, launches):
    """All three algorithms within tolerance; CSR scalar with the bits of one
    thread per row on rows up to 64 elements."""
    ys, ab = oracle_lib.csr_spmv_exact(m.rows, m.row_ptr, m.columns, m.data, x)
    want = spmv(m, CSR_SCALAR, x, None, {"long_row_threshold": NEVER, "assist_threshold": NEVER})
    short = np.diff(m.row_ptr.astype(np.int64)) <= 64
    for fmt in (CSR_SCALAR, CSR_VECTOR, CSR_ADAPTIVE):
        y = spmv(m, fmt, x, launches)
        assert np.all(np.abs(y.astype(np.float64) - ys) <= TOL[m.dtype.type] * ab), fmt
        if fmt == CSR_SCALAR:
            assert np.array_equal(y[short].view(np.uint8), want[short].view(np.uint8))


# row blocks of 256 rows; 148 x 8 (FP32) or 148 x 6 (FP64) CTAs fit the chip at once
@pytest.mark.parametrize("blocks", [1, 100, 200, 400, 700, 888, 889, 1184, 1185, 1300, 2000, 2400])
@pytest.mark.parametrize("lo, hi", [(0, 4), (3, 30)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_every_split_of_a_row_block(oracle_lib, blocks, lo, hi, dtype):
    rng = np.random.default_rng(blocks)
    m = csr(rng.integers(lo, hi + 1, blocks * 256 - 17), 2_000, dtype)
    check(oracle_lib, m, synth.vector(1, m.cols).astype(dtype), 1)


def part_short(blocks, rng):
    """Rows of 20 to 49 elements; 30% of the row blocks hold a longer one too."""
    lens = rng.integers(20, 50, blocks * 256)
    for b in rng.choice(blocks, blocks * 3 // 10, replace=False):
        lens[b * 256 + rng.integers(0, 256)] = rng.choice([65, 300, 3_000])
    lens[1234 * 256] = 20_000
    return lens


def test_large_matrix_with_part_of_its_elements_in_short_row_blocks(oracle_lib):
    """FP32 from 64M elements on: half of them in such blocks are enough, the other
    blocks are a launch beside them."""
    m = csr(part_short(7_600, np.random.default_rng(77)), 50_000, np.float32)
    assert m.nnz >= 64 << 20
    check(oracle_lib, m, synth.vector(2, m.cols).astype(np.float32), 2)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_middle_sized_matrix_with_part_of_its_elements_in_short_row_blocks(oracle_lib, dtype):
    """Below that, and in FP64: one kernel for all blocks (vector: two passes)."""
    m = csr(part_short(2_000, np.random.default_rng(78)), 50_000, dtype)
    x = synth.vector(2, m.cols).astype(dtype)
    check(oracle_lib, m, x, None)
    for fmt, launches in ((CSR_SCALAR, 1), (CSR_VECTOR, 2), (CSR_ADAPTIVE, 1)):
        spmv(m, fmt, x, launches)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_short_rows_alone_in_a_bin(oracle_lib, dtype):
    """Rows of up to 64 elements between two that fill a bin each."""
    rng = np.random.default_rng(79)
    lens = rng.integers(20, 50, 1000 * 256)
    for b in range(0, 1000, 50):
        lens[b * 256:b * 256 + 7] = [rng.integers(30, 65), 2_500, 64, 4_000, 1, 2_300, 40]
    m = csr(lens, 50_000, dtype)
    check(oracle_lib, m, synth.vector(2, m.cols).astype(dtype), 2)
