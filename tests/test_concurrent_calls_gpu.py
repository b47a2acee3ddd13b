"""One handle, plan or batch used by several streams, threads and captured graphs
at once: each call's scratch is its own, so every result has the bits of a lone
call."""
import ctypes as C
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import formats as F  # noqa: E402
from matrix_format_performance_b200 import synth  # noqa: E402
from matrix_format_performance_b200._capi import call  # noqa: E402
from matrix_format_performance_b200.batch import Batch  # noqa: E402
from matrix_format_performance_b200.device import CSR_ADAPTIVE, CSR_SCALAR, SCOO, DeviceMatrix  # noqa: E402

TOL = {np.float32: 1e-5, np.float64: 1e-12}  # per row, of sum |a_ij x_j|


def long_rows(dtype, rows=3000, cols=70_000, seed=31):
    """Short rows and rows of 5,000 to 60,000 elements, which are several pieces each."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 80, rows)
    lens[rng.choice(rows, 12, replace=False)] = np.linspace(5_000, 60_000, 12).astype(int)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    c = rng.integers(0, cols, int(rp[-1])).astype(np.uint32)
    return F.csr_matrix_class.from_arrays(rows, cols, rp, c, rng.uniform(-1, 1, len(c)), dtype)


def vectors(m, n):
    return [torch.from_numpy(synth.vector(k, m.cols).astype(m.dtype)).cuda() for k in range(n)]


def same(a, b):
    return np.array_equal(a.cpu().numpy().view(np.uint8), b.cpu().numpy().view(np.uint8))


def check_all(product, xs, rows, streams=20, threads=4):
    """product(x, y, stream) on `streams` streams, from threads that share a stream, and in
    two graphs, all at once, against lone calls."""
    want = []
    for x in xs:
        y = torch.empty(rows, dtype=x.dtype, device="cuda")
        product(x, y, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(y)
    ss = [torch.cuda.Stream() for _ in range(streams)]
    shared = torch.cuda.Stream()
    graphs = []
    for k in range(2):
        y = torch.empty_like(want[0])
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            product(xs[k], y, torch.cuda.current_stream())
        graphs.append((g, k, y, torch.cuda.Stream()))
    got = [[torch.empty_like(want[0]) for _ in range(5)] for _ in ss]
    thread_got = [[torch.empty_like(want[0]) for _ in range(5)] for _ in range(threads)]
    torch.cuda.synchronize()

    def work(t):
        for i, y in enumerate(thread_got[t]):
            product(xs[(t + i) % len(xs)], y, shared)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in ts:
        t.start()
    for i in range(5):
        for k, s in enumerate(ss):
            product(xs[(k + i) % len(xs)], got[k][i], s)
        for g, _, _, s in graphs:
            with torch.cuda.stream(s):
                g.replay()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for k in range(len(ss)):
        for i in range(5):
            assert same(got[k][i], want[(k + i) % len(xs)]), (k, i)
    for t in range(threads):
        for i in range(5):
            assert same(thread_got[t][i], want[(t + i) % len(xs)]), (t, i)
    for _, k, y, _ in graphs:
        assert same(y, want[k])
    del graphs
    # a lone call afterwards finds its scratch as the first one did
    y = torch.empty_like(want[0])
    product(xs[0], y, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert same(y, want[0])


@pytest.mark.parametrize("fmt", [CSR_SCALAR, CSR_ADAPTIVE])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_csr_rows_of_several_pieces(fmt, dtype):
    m = long_rows(dtype)
    dm = DeviceMatrix.from_csr(m, fmt)
    check_all(lambda x, y, s: dm.spmv(x, y, s), vectors(m, 3), m.rows)
    dm.close()


def test_batch_rows_of_several_pieces():
    ms = [long_rows(np.float32, rows=800, seed=k) for k in range(3)]
    b = Batch(ms)
    rows = sum(m.rows for m in ms)
    cols = sum(m.cols for m in ms)
    xs = [torch.from_numpy(synth.vector(k, cols).astype(np.float32)).cuda() for k in range(3)]
    check_all(lambda x, y, s: b.spmv(x, y, s), xs, rows)
    b.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_scoo_tiles(dtype):
    m = long_rows(dtype)
    dm = DeviceMatrix.build(m, SCOO)
    assert dm.info().kernel_launches == 2  # tiles and fix-up
    check_all(lambda x, y, s: dm.spmv(x, y, s), vectors(m, 3), m.rows)
    dm.close()


@pytest.mark.parametrize("fmt", [CSR_ADAPTIVE, SCOO])
def test_captured_calls_allocate_nothing_in_the_graph(fmt):
    """A captured call is kernel launches only, so its graph can be cloned, be a
    child graph and be instantiated again."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    m = long_rows(np.float32)
    dm = DeviceMatrix.build(m, fmt)
    x = vectors(m, 1)[0]
    y, want = (torch.empty(m.rows, device="cuda") for _ in range(2))
    dm.spmv(x, want)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        dm.spmv(x, y)
    raw = rt.cudaGraph_t(g.raw_cuda_graph())
    _, _, n = rt.cudaGraphGetNodes(raw, 0)
    _, nodes, n = rt.cudaGraphGetNodes(raw, n)
    kinds = [rt.cudaGraphNodeGetType(v)[1] for v in nodes[:n]]
    assert kinds and all(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)
    g.instantiate()
    g.replay()
    torch.cuda.synchronize()
    assert same(y, want)
    del g
    dm.close()


@pytest.fixture
def no_device_memory():
    """take(stream): allocates all device memory that is left."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    held = []

    def take(stream):
        torch.cuda.empty_cache()
        size = 1 << 36
        while size >= 1 << 20:
            err, p = rt.cudaMalloc(size)
            if int(err):
                rt.cudaGetLastError()
                size >>= 1
            else:
                held.append(p)
        assert int(rt.cudaMallocAsync(1, stream.cuda_stream)[0])
        rt.cudaGetLastError()

    yield take
    for p in held:
        rt.cudaFree(p)


@pytest.mark.parametrize("fmt", [CSR_ADAPTIVE, CSR_SCALAR, SCOO])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_calls_without_memory_for_their_scratch(oracle_lib, no_device_memory, fmt, dtype):
    """With no memory left, a second stream's call runs without
    scratch: SCOO one CTA per slice, CSR one CTA per long row."""
    m = long_rows(dtype)
    dm = DeviceMatrix.build(m, fmt)
    x = vectors(m, 1)[0]
    first, second = (torch.full((m.rows,), float("nan"), dtype=x.dtype, device="cuda") for _ in range(2))
    if fmt == SCOO:  # its kernel is loaded while there is memory
        s = F.scoo_matrix_class(148, 49152, m)
        keep = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
                (s.values, s.c_index.view(np.int32), s.r_index.view(np.int32), s.slices_ptr.view(np.int32))]
        v, ci, ri, sp, xp, yp = (C.c_void_p(t.data_ptr()) for t in (*keep, x, first))
        call(f"mfp_scoo_spmv_{'f32' if dtype == np.float32 else 'f64'}", m.rows, m.cols, s.slices_count, s.slice_size, v,
             ci, ri, sp, None, 0, None, xp, yp, None)
        torch.cuda.synchronize()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    dm.spmv(x, first, one)  # its stream takes the handle's own block
    torch.cuda.synchronize()
    no_device_memory(two)
    dm.spmv(x, second, two)
    torch.cuda.synchronize()
    ys, ab = oracle_lib.csr_spmv_exact(m.rows, m.row_ptr, m.columns, m.data, x.cpu().numpy())
    for y in (first, second):
        assert np.all(np.abs(y.cpu().numpy().astype(np.float64) - ys) <= TOL[dtype] * ab)
    dm.close()
