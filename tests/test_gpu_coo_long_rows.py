"""COO -> CSR on the device where rows are longer than a block sorts well (from 16384 entries, where
there are fewer such rows than SMs, the whole device sorts all long rows): both lines, one such row,
several, others beside them."""
import statistics
import time

import numpy as np
import pytest

from pava_b200 import matrices as M

pytestmark = pytest.mark.gpu

CASES = {
    "below": [16383, 3, 300],
    "at": [16384],
    "at_and_others": [5, 257, 16384, 0, 256, 300, 1],
    "one": [0, 100_003, 0],
    "several": [70_001, 16_385, 0, 40_000, 20_000, 2],
    "many_listed": [300] * 600 + [30_000] + [257] * 600,
    "a_row_per_sm": [16_384] * 148,
    "fewer": [16_384] * 147 + [16_383],
}


@pytest.mark.parametrize("order", ["row", "random"])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n", [7, 60_000])            # few columns: mostly duplicates
@pytest.mark.parametrize("name", list(CASES))
def test_sorted(cuda, name, n, symmetric, order):
    torch = cuda
    lens = np.array(CASES[name])
    rng = np.random.default_rng(5)
    m = len(lens)
    if symmetric:
        n = m = max(m, n)
    r = np.repeat(np.arange(len(lens)), lens)
    c = rng.integers(0, n, len(r))
    v = rng.normal(size=len(r))
    at = np.lexsort((c, r)) if order == "row" else rng.permutation(len(r))
    r, c, v = r[at], c[at], v[at]
    dev = [torch.from_numpy(a).cuda() for a in (r.astype(np.int32), c.astype(np.int32), v)]
    rp, ci, vv = (t.cpu().numpy() for t in M.coo_to_csr_device(m, n, *dev, symmetric=symmetric))
    if symmetric:
        off = r != c
        r, c, v = np.concatenate([r, c[off]]), np.concatenate([c, r[off]]), np.concatenate([v, v[off]])
    want = np.argsort(r * np.int64(n) + c, kind="stable")
    assert np.array_equal(rp, np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]))
    assert np.array_equal(ci, c[want])
    assert np.array_equal(vv, v[want])


def _seconds(torch, fn):
    times = []
    for _ in range(7):
        torch.cuda.synchronize()
        start = time.perf_counter()
        fn()
        torch.cuda.synchronize()
        times.append(time.perf_counter() - start)
    return statistics.median(times[2:])


@pytest.mark.parametrize("rows", [1, 2])
def test_one_row_takes_no_more_than_many(cuda, rows):
    """The same bytes and the same passes, whatever the rows: 3 M entries in one row or in rows of
    300.  Sorted by one block the single row took 43 times as long; 8 leaves room for the clock."""
    torch = cuda
    nnz, n = 3_000_000, 5_000_000
    c = torch.randint(0, n, (nnz,), dtype=torch.int32, device="cuda")
    v = torch.randn(nnz, dtype=torch.float64, device="cuda")
    k = torch.arange(nnz, dtype=torch.int32, device="cuda")
    many, few = k // 300, k // ((nnz + rows - 1) // rows)
    base = _seconds(torch, lambda: M.coo_to_csr_device(10_000, n, many, c, v))
    assert _seconds(torch, lambda: M.coo_to_csr_device(10_000, n, few, c, v)) < 8 * base
