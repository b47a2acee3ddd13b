"""Edges of the device triplets -> CSR conversion: waits that run out,
outputs in the inputs' memory."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from matrix_format_performance_b200 import convert  # noqa: E402
from matrix_format_performance_b200._capi import MfpError, call  # noqa: E402

TILE = 6144  # keys per tile of the triplet sort
DEVICE_WAIT = 6
GUARD = 4096  # words before and after each output


def triplets(rows, cols, n, seed=5):
    rng = np.random.default_rng(seed)
    r = rng.integers(0, rows, n).astype(np.int32)
    c = rng.integers(0, cols, n).astype(np.int32)
    return r, c, rng.uniform(-1, 1, n)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("rows, cols", [(3, 200), (70_000, 65_537)])  # one digit, four digits
@pytest.mark.parametrize("vt, dtype", [(0, torch.float32), (1, torch.float64)])
def test_a_wait_that_runs_out_is_an_error_and_writes_nothing_outside(rows, cols, vt, dtype):
    """With a limit of 0 every tile but the first gives up: the status says so,
    nothing beyond the outputs is written, and the next conversion is right."""
    n = 300 * TILE + 11
    r, c, v = triplets(rows, cols, n)
    tr, tc, tv = dev(r), dev(c), dev(v)

    def guarded(count, dt):
        t = torch.full((count + 2 * GUARD,), 77, dtype=dt, device="cuda")
        return t, t[GUARD:GUARD + count]

    outs = [guarded(rows + 1, torch.int32), guarded(n, torch.int32), guarded(n, dtype)]
    with pytest.raises(MfpError) as e:
        call("mfp_dev_csr_from_coo_limited", vt, rows, cols, n, p(tr), p(tc), p(tv), *[p(o) for _, o in outs], 0, None)
    assert e.value.status == DEVICE_WAIT
    torch.cuda.synchronize()
    for t, o in outs:
        assert bool((t[:GUARD] == 77).all()) and bool((t[GUARD + o.numel():] == 77).all())
    rp, co, d = convert.csr_from_coo(rows, cols, tr, tc, tv, dtype=dtype)
    order = np.lexsort((np.arange(n), c, r))
    assert np.array_equal(rp.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(r, minlength=rows))]))
    assert np.array_equal(co.cpu().numpy(), c[order])
    assert np.array_equal(d.cpu().numpy(), v[order].astype(d.cpu().numpy().dtype))


def test_one_tile_never_waits():
    r, c, v = triplets(500, 509, TILE)
    outs = [torch.empty(501, dtype=torch.int32, device="cuda"), torch.empty(TILE, dtype=torch.int32, device="cuda"),
            torch.empty(TILE, dtype=torch.float64, device="cuda")]
    tr, tc, tv = dev(r), dev(c), dev(v)
    call("mfp_dev_csr_from_coo_limited", 1, 500, 509, TILE, p(tr), p(tc), p(tv), *[p(o) for o in outs], 0, None)
    order = np.lexsort((np.arange(TILE), c, r))
    assert np.array_equal(outs[1].cpu().numpy(), c[order])
    assert np.array_equal(outs[2].cpu().numpy(), v[order])


@pytest.mark.parametrize("order", ["sorted", "shuffled"])
@pytest.mark.parametrize("rows, cols", [(3, 200), (70_000, 65_537)])  # one digit (one pass), four digits
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_outputs_in_the_inputs_memory(order, rows, cols, dtype):
    """columns = col_ids, data = values and row_ptr = row_ids give what separate
    outputs give."""
    n = 100 * TILE + 5
    r, c, v = triplets(rows, cols, n, seed=9)
    if order == "sorted":
        k = np.lexsort((c, r))
        r, c, v = r[k], c[k], v[k]
    want = [t.cpu().numpy() for t in convert.csr_from_coo(rows, cols, dev(r), dev(c), dev(v), dtype=dtype)]
    tr, tc, tv = dev(r), dev(c), dev(v)
    call("mfp_dev_csr_from_coo", int(dtype == torch.float64), rows, cols, n, p(tr), p(tc), p(tv), p(tr), p(tc), p(tv),
         None)
    got = tr[:rows + 1], tc, tv.view(dtype)[:n]
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)
