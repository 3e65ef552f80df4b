"""COO -> CSR on the device at the row lengths where its sorting changes: batches of 512 entries,
rows of up to 256 entries and longer ones, duplicates, hypersparse rows, each input order."""
import numpy as np
import pytest

from pava_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _cases():
    yield "edges", np.array([0, 1, 255, 256, 257, 0, 0, 511, 512, 513, 3, 256, 256, 1, 0, 5000]), 6000
    yield "batches", np.full(1000, 16), 900      # 32 rows are one batch exactly
    yield "batches_odd", np.full(1000, 17), 900
    lens = np.zeros(200_000, np.int64)
    lens[::3001] = 40
    yield "hypersparse", lens, 300_000
    yield "all_long", np.full(70, 300), 2000


@pytest.mark.parametrize("order", ["row", "column", "random"])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("name,lens,n", list(_cases()), ids=[c[0] for c in _cases()])
def test_rows(cuda, name, lens, n, symmetric, order):
    torch = cuda
    rng = np.random.default_rng(11)
    m = len(lens)
    n = m = max(m, n) if symmetric else n
    m = m if symmetric else len(lens)
    r = np.repeat(np.arange(len(lens)), lens)
    c = rng.integers(0, n, len(r))
    c[::5] = c[::5] // 7 * 7                     # duplicates
    v = rng.normal(size=len(r))
    at = {"row": np.lexsort((c, r)), "column": np.lexsort((r, c)),
          "random": rng.permutation(len(r))}[order]
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
