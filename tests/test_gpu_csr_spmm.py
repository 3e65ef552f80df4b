"""Plain CSR SpMM in the engine's own shape: rows around a piece of 16 elements, empty and long rows,
row counts around a warp's tile, every columns-per-lane form with odd and even k, padded leading
dimensions, and an X with a non-finite row that no element reads."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def _csr(lens, n, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)])
    ci = np.concatenate([np.sort(1 + rng.choice(n - 1, k, replace=False)) for k in lens])
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    return M.from_arrays(len(lens), n, rp, ci, v)


def _matrices():
    rng = np.random.default_rng(2)
    yield "pieces", _csr([0, 1, 15, 16, 17, 31, 32, 33, 48, 0, 0, 16, 16, 16, 16, 16, 3], 80, 3)
    yield "full_pieces", _csr(np.full(129, 32), 100, 4)
    yield "long", _csr(np.r_[rng.integers(0, 9, 200), 3000, rng.integers(0, 9, 111)], 4000, 5)
    yield "one_row", _csr([5], 9, 6)
    yield "many", _csr(rng.integers(0, 30, 40_000), 3000, 7)


@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("name,A", list(_matrices()), ids=[m[0] for m in _matrices()])
def test_spmm(cuda, name, A, prec):
    torch = cuda
    fp32 = prec == _abi.PREC_FP32C
    mat = SpMatrix(A, "csr", precision=prec)
    for k in (2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128):
        X = np.stack([M.uniform(A.n, seed=20 + j, fp32=True) for j in range(k)], 1)
        Xd = torch.from_numpy(X).cuda()
        Xd[0] = float("nan")  # no element is in column 0
        Xd = Xd.float() if fp32 else Xd
        Y = mat.spmm(Xd)
        assert torch.equal(Y, mat.spmm(Xd))
        Yh = Y.cpu().numpy()
        for j in {0, k // 2, k - 1}:
            yr, ab = O.csr_ref(A.rp, A.ci, A.v, X[:, j].copy())
            assert O.rel_error(Yh[:, j].copy(), yr, ab, 1e-12)[0] == 0, (k, j)
        # leading dimensions of their own, even and odd; what lies past k stays as it was
        for pad in (2, 3):
            Xp = torch.full((A.n, k + pad), float("nan"), dtype=Xd.dtype, device="cuda")
            Xp[:, :k] = Xd
            Yp = torch.full((A.m, k + pad), 7.0, dtype=torch.float64, device="cuda")
            mat.spmm(Xp[:, :k], Yp[:, :k])
            assert torch.equal(Yp[:, :k], Y) and bool((Yp[:, k:] == 7.0).all())
