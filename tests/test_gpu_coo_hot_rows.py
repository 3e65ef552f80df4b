"""COO -> CSR on the device where a few rows hold much of a shuffled input: counting and scattering
take one atomic per row and warp there, with lanes of other rows and absent lanes between."""
import statistics
import time

import numpy as np
import pytest

from pava_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _rows(name, nnz, m, rng):
    spread = rng.integers(0, m, nnz)
    if name == "two":
        return np.arange(nnz) % 2
    if name == "nine":
        return rng.integers(0, 9, nnz)
    if name == "blocks":           # runs of five: a hot row's runs and others alternate
        return np.where(np.arange(nnz) // 5 % 2, 3, spread)
    return np.where(rng.random(nnz) < float(name), 7, spread)


@pytest.mark.parametrize("name", ["two", "nine", "blocks", "0.1", "0.5", "0.95"])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("nnz", [17, 31, 33, 4_099, 100_001])
def test_sorted(cuda, name, symmetric, nnz):
    torch = cuda
    rng = np.random.default_rng(nnz)
    m = n = 700
    r = _rows(name, nnz, m, rng)
    c = _rows("0.5", nnz, n, rng)          # a hot column too: mirrored, a hot row
    v = rng.normal(size=nnz)
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


def test_shuffled_hot_row(cuda):
    """Half of 20 M entries in one row, shuffled or in row order.  With an atomic for nearly each
    entry the shuffled order took 4.5 times as long; the scattered records are read and written in
    sectors of 32 bytes for 16 either way, so 3 is above what the order itself costs."""
    torch = cuda
    nnz, m = 20_000_000, 1_000_000
    rows = torch.randint(0, m, (nnz,), dtype=torch.int32, device="cuda")
    rows[torch.rand(nnz, device="cuda") < 0.5] = 0
    c = torch.randint(0, m, (nnz,), dtype=torch.int32, device="cuda")
    v = torch.randn(nnz, dtype=torch.float64, device="cuda")
    ordered = rows.sort()[0]
    base = _seconds(torch, lambda: M.coo_to_csr_device(m, m, ordered, c, v))
    assert _seconds(torch, lambda: M.coo_to_csr_device(m, m, rows, c, v)) < 3 * base
