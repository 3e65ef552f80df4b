"""SELL SpMM at the edges of its pieces and runs: rows of up to a block, a piece and past it, padding
that begins inside a block, empty slices, few and many slices, each lanes-per-row, odd and even k,
and an X whose first row is not finite (padding must not read it)."""
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
    yield "block", _csr(np.full(70, 4), 90, 3)
    yield "piece", _csr(np.r_[np.full(32, 32), np.full(32, 33), np.full(32, 64), np.full(33, 65)], 200, 4)
    yield "ragged", _csr(rng.integers(20, 41, 500), 300, 5)
    yield "empty_slices", _csr(np.r_[np.zeros(64, int), np.full(32, 7), np.zeros(96, int), [3]], 50, 6)
    yield "many_slices", _csr(rng.integers(3, 6, 170_000), 5000, 7)


@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("index", [_abi.INDEX_I32, _abi.INDEX_AUTO])
@pytest.mark.parametrize("name,A", list(_matrices()), ids=[m[0] for m in _matrices()])
def test_pieces(cuda, name, A, index, prec):
    torch = cuda
    fp32 = prec == _abi.PREC_FP32C
    for lanes, ks in ((4, (1, 3, 8, 16, 31, 32)), (8, (2, 5, 32, 64)), (16, (16, 33, 64))):
        mat = SpMatrix(A, "sell", precision=prec, index_mode=index, lanes_per_row=lanes)
        for k in ks:
            X = np.stack([M.uniform(A.n, seed=10 + j, fp32=True) for j in range(k)], 1)
            Xd = torch.from_numpy(X).cuda()
            Xd[0] = float("nan")  # no element is in column 0
            Y = mat.spmm(Xd.float() if fp32 else Xd)
            assert torch.equal(Y, mat.spmm(Xd.float() if fp32 else Xd))
            Yh = Y.cpu().numpy()
            for j in {0, k - 1}:
                yr, ab = O.csr_ref(A.rp, A.ci, A.v, X[:, j].copy())
                assert O.rel_error(Yh[:, j].copy(), yr, ab, 1e-12)[0] == 0, (lanes, k, j)
        mat.close()


@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("lanes", [0, 4, 8, 16])
@pytest.mark.parametrize("per_row", [5, 20])
def test_every_column_count(cuda, per_row, lanes, prec):
    """Each number of columns per lane, whole and partly filled, aligned and not, short and long rows."""
    torch = cuda
    fp32 = prec == _abi.PREC_FP32C
    A = _csr(np.full(300, per_row), 150, 8)
    mat = SpMatrix(A, "sell", precision=prec, lanes_per_row=lanes)
    top = 32 if lanes == 4 else 64
    X = np.stack([M.uniform(A.n, seed=10 + j, fp32=True) for j in range(top)], 1)
    refs = [O.csr_ref(A.rp, A.ci, A.v, X[:, j].copy()) for j in range(top)]
    Xd = torch.from_numpy(X).cuda()
    Xd = Xd.float() if fp32 else Xd
    for k in range(1, top + 1):
        for ld in {k, k + 1, k + 2}:
            Xk = torch.full((A.n, ld), float("nan"), dtype=Xd.dtype, device="cuda")[:, :k]
            Xk.copy_(Xd[:, :k])
            Y = mat.spmm(Xk).cpu().numpy()
            for j in {0, k // 2, k - 1}:
                yr, ab = refs[j]
                assert O.rel_error(Y[:, j].copy(), yr, ab, 1e-12)[0] == 0, (k, ld, j)


@pytest.mark.parametrize("lanes,k", [(0, 3), (4, 32), (16, 64)])
def test_leading_dimension_past_int(cuda, lanes, k):
    torch = cuda
    A = _csr([1, 0, 1] * 20, 2, 9)
    ld = 2**31 + 5
    X = torch.empty(ld + k, dtype=torch.float32, device="cuda").as_strided((2, k), (ld, 1))
    X.copy_(torch.arange(2.0 * k, device="cuda").reshape(2, k))
    mat = SpMatrix(A, "sell", precision=_abi.PREC_FP32C, lanes_per_row=lanes)
    Y = mat.spmm(X).cpu().numpy()
    for j in range(k):
        yr, ab = O.csr_ref(A.rp, A.ci, A.v, X[:, j].double().cpu().numpy().copy())
        assert O.rel_error(Y[:, j].copy(), yr, ab, 1e-12)[0] == 0, j
