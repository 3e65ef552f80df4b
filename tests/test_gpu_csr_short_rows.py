"""CSR SpMM on row groups whose lanes share a row's elements: rows shorter than the group, the last
round's steps at a half, a quarter and an eighth, and rows of different length in one warp."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("x_window", [0, 1])
@pytest.mark.parametrize("k,kc,kpl", [(2, 2, 1), (4, 4, 1), (7, 8, 1), (13, 8, 2), (31, 16, 2), (33, 16, 4),
                                      (31, 32, 1), (64, 32, 2), (127, 32, 4)])
@pytest.mark.parametrize("lanes", [0, 32])
def test_rows(cuda, precision, x_window, k, kc, kpl, lanes):
    torch = cuda
    lanes = lanes or kc
    rng = np.random.default_rng(k + lanes)
    edges = sorted({e + d for e in (0, lanes // 8, lanes // 4, lanes // 2, lanes, 2 * lanes) for d in (-1, 0, 1)})
    lens = [e for e in edges if e >= 0] * 4
    lens += [e for e in edges if e >= 0 for _ in range(32 // lanes)]  # a warp of rows of one length
    lens = np.array(lens + list(rng.integers(0, 2 * lanes + 3, 41)))
    n = 300
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in lens])
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    A = M.from_arrays(len(lens), n, rp, ci, v)
    mat = SpMatrix(A, "csr", precision=precision, lanes_per_row=lanes, col_lanes=kc, cols_per_lane=kpl,
                   rows_per_tile=128 if x_window else 0, x_window=x_window)
    X = M.uniform(n * k, seed=4, fp32=True).reshape(n, k)
    Xd = torch.from_numpy(X).cuda()
    fp32 = precision == _abi.PREC_FP32C
    y = mat.spmm(Xd.float() if fp32 else Xd).cpu().numpy()
    for c in sorted({0, k // 2, k - 1}):
        yr, ab = O.csr_ref(A.rp, A.ci, A.v, np.ascontiguousarray(X[:, c]))
        assert O.rel_error(np.ascontiguousarray(y[:, c]), yr, ab, 1e-9 if fp32 else 1e-12)[0] == 0  # the stated bounds
