"""Plain CSR SpMV on rows around the lengths where their handling changes: within a group, by the
whole warp (more than 16 elements per lane of the group), by the CTA (more than 1,024), and more
long rows than a warp keeps for the CTA (8)."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def _matrix(lens, n, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens] or [[]])
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    return M.from_arrays(len(lens), n, rp, ci, v)


def _cases():
    rng = np.random.default_rng(3)
    yield "edges", np.array([0, 1, 15, 16, 17, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023,
                             1024, 1025, 4097, 0, 3])
    # 12 rows per warp tile and more, all above 1,024: the lists overflow
    yield "all_long", np.full(40, 1100)
    lens = rng.integers(0, 12, 3000)
    lens[rng.choice(3000, 60, replace=False)] = rng.integers(60, 3000, 60)
    yield "mixed", lens


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("lanes", [0, 1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("name,lens", list(_cases()), ids=[c[0] for c in _cases()])
def test_long_rows(cuda, name, lens, lanes, precision):
    import torch
    A = _matrix(lens, 6000, 5)
    fp32 = precision == _abi.PREC_FP32C
    x = M.uniform(A.n, seed=6, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    xd = torch.from_numpy(x).cuda()
    xd = xd.float() if fp32 else xd
    # one warp takes the whole of "all_long": its list overflows
    rows = 32 // lanes * 64 if lanes and name == "all_long" else 0
    mat = SpMatrix(A, "csr", precision=precision, lanes_per_row=lanes, rows_per_tile=rows)
    y = mat.spmv(xd)
    bound = 1e-9 if fp32 else 1e-12  # the forms' stated bounds
    assert O.rel_error(y.cpu().numpy(), yr, ab, bound)[0] == 0
    assert torch.equal(y, mat.spmv(xd))  # same bits on every call
    # one column of a wider row-major X: strided x and y
    X = torch.zeros((A.n, 3), dtype=xd.dtype, device="cuda")
    X[:, 1] = xd
    Y = torch.full((A.m, 2), 7.0, dtype=torch.float64, device="cuda")
    mat.spmm(X[:, 1:2], Y[:, 1:2])
    assert torch.equal(Y[:, 1], y) and bool((Y[:, 0] == 7.0).all())
