"""CSR SpMM without a shape of its own: rows staged per warp, or a warp per row where one row is far
longer than the others; on both sides of that rule, and with strided X and Y."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def _matrix(longest, seed):
    """4,000 rows of about ten nonzeros and one of `longest`."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 20, 4000)
    lens[1234] = longest
    n = 5000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in lens])
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    return M.from_arrays(len(lens), n, rp, ci, v)


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("longest", [20, 41, 5000])   # four times the mean row is 39
@pytest.mark.parametrize("k", [1, 2, 3, 8, 33, 64, 65, 128])
def test_products(cuda, precision, longest, k):
    torch = cuda
    A = _matrix(longest, k)
    fp32 = precision == _abi.PREC_FP32C
    mat = SpMatrix(A, "csr", precision=precision)
    X = M.uniform(A.n * k, seed=5, fp32=True).reshape(A.n, k)
    Xd = torch.from_numpy(X).cuda()
    Xd = Xd.float() if fp32 else Xd
    y = mat.spmm(Xd)
    assert torch.equal(y, mat.spmm(Xd))
    wide = torch.zeros((A.n, k + 3), dtype=Xd.dtype, device="cuda")
    wide[:, 1:k + 1] = Xd
    Y = torch.full((A.m, k + 1), 7.0, dtype=torch.float64, device="cuda")
    mat.spmm(wide[:, 1:k + 1], Y[:, :k])
    assert bool((Y[:, k] == 7.0).all())
    for out in (y.cpu().numpy(), Y[:, :k].cpu().numpy()):
        for c in sorted({0, k // 2, k - 1}):
            yr, ab = O.csr_ref(A.rp, A.ci, A.v, np.ascontiguousarray(X[:, c]))
            assert O.rel_error(np.ascontiguousarray(out[:, c]), yr, ab, 1e-9 if fp32 else 1e-12)[0] == 0


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("m", [1, 31, 13_999, 14_001, 29_999, 30_001])   # a warp per row up to 14,000 or 30,000
@pytest.mark.parametrize("k", [2, 3, 32, 33, 64, 65])
def test_small_matrices_of_even_rows(cuda, precision, m, k):
    torch = cuda
    A = M.banded(m, 8, 6, seed=3) if m > 20 else M.from_arrays(m, m, np.arange(m + 1, dtype=np.int32),
                                                              np.arange(m, dtype=np.int32), np.ones(m))
    fp32 = precision == _abi.PREC_FP32C
    A = M.from_arrays(A.m, A.n, A.rp, A.ci, A.v.astype(np.float32).astype(np.float64))
    mat = SpMatrix(A, "csr", precision=precision)
    X = M.uniform(A.n * k, seed=5, fp32=True).reshape(A.n, k)
    Xd = torch.from_numpy(X).cuda()
    y = mat.spmm(Xd.float() if fp32 else Xd).cpu().numpy()
    for c in (0, k - 1):
        yr, ab = O.csr_ref(A.rp, A.ci, A.v, np.ascontiguousarray(X[:, c]))
        assert O.rel_error(np.ascontiguousarray(y[:, c]), yr, ab, 1e-9 if fp32 else 1e-12)[0] == 0
