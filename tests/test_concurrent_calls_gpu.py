"""One handle, plan or batch used by several streams, threads and captured graphs
at once: each call's scratch is its own, so every result has the bits of a lone
call."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import formats as F  # noqa: E402
from matrix_format_performance_b200 import synth  # noqa: E402
from matrix_format_performance_b200.batch import Batch  # noqa: E402
from matrix_format_performance_b200.device import CSR_ADAPTIVE, CSR_SCALAR, DeviceMatrix  # noqa: E402


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


def test_captured_calls_allocate_nothing_in_the_graph():
    """A captured call is kernel launches only, so its graph can be cloned, be a
    child graph and be instantiated again."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    m = long_rows(np.float32)
    dm = DeviceMatrix.from_csr(m, CSR_ADAPTIVE)
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
