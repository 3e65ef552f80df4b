"""SELL SpMM where the pieces' length, the warps per SM, the elements in flight and the lanes per row
change with k, the precision and the columns: rows of a piece of 4 or 8 blocks and around it."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def _matrix(lens, n=250, seed=1):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in lens])
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    return M.from_arrays(len(lens), n, rp, ci, v)


LENS = {"pieces": np.repeat([15, 16, 17, 31, 32, 33, 48, 65], 32), "ragged": np.random.default_rng(4).integers(9, 37, 333),
        "long": np.random.default_rng(5).integers(30, 60, 200), "short": np.random.default_rng(6).integers(3, 6, 200)}


@pytest.mark.parametrize("name", list(LENS))
@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("index", [_abi.INDEX_I32, _abi.INDEX_AUTO])
@pytest.mark.parametrize("lanes,ks", [(0, (13, 14, 16, 49, 56, 63, 64)), (4, (16, 17, 20, 24, 28, 29, 32)), (8, (48, 50, 57, 64))])
def test_shapes(cuda, name, precision, index, lanes, ks):
    torch = cuda
    A = _matrix(LENS[name])
    fp32 = precision == _abi.PREC_FP32C
    mat = SpMatrix(A, "sell", precision=precision, index_mode=index, lanes_per_row=lanes)
    for k in ks:
        X = M.uniform(A.n * k, seed=k, fp32=True).reshape(A.n, k)
        Xd = torch.from_numpy(X).cuda()
        Xd = Xd.float() if fp32 else Xd
        Y = mat.spmm(Xd)
        assert torch.equal(Y, mat.spmm(Xd))
        for c in (0, k // 2, k - 1):
            yr, ab = O.csr_ref(A.rp, A.ci, A.v, np.ascontiguousarray(X[:, c]))
            assert O.rel_error(Y[:, c].contiguous().cpu().numpy(), yr, ab, 1e-12)[0] == 0, (k, c)
