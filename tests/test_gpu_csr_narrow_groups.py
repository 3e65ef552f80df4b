"""Plain CSR SpMV with one, two or four lanes per row where many of a warp's rows are longer than 16
elements per lane: by the groups when that is fewer rounds, else one after the other by the warp."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def _lens(lanes, length, count):
    """Rows of a warp's round (32 / lanes), `count` of them of `length`, the others short."""
    rng = np.random.default_rng(lanes * 10_000 + length + count)
    rows = 32 // lanes
    out = []
    for _ in range(40):
        lens = rng.integers(0, 16 * lanes + 1, rows)
        lens[rng.choice(rows, min(count, rows), replace=False)] = length
        out.append(lens)
    return np.concatenate(out)[:-3]


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("lanes", [1, 2, 4])
@pytest.mark.parametrize("per_lane", [17, 24, 256])
@pytest.mark.parametrize("count", [1, 4, 8, 32])
def test_rounds(cuda, precision, lanes, per_lane, count):
    torch = cuda
    lens = _lens(lanes, lanes * per_lane, count)
    if per_lane == 256:
        lens[::50] = 1025                          # beside rows for the CTA
    rng = np.random.default_rng(9)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n = 3000
    ci = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens])
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    A = M.from_arrays(len(lens), n, rp, ci, v)
    fp32 = precision == _abi.PREC_FP32C
    x = M.uniform(n, seed=6, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    xd = torch.from_numpy(x).cuda()
    xd = xd.float() if fp32 else xd
    mat = SpMatrix(A, "csr", precision=precision, lanes_per_row=lanes)
    y = mat.spmv(xd)
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-9 if fp32 else 1e-12)[0] == 0  # the stated bounds
    assert torch.equal(y, mat.spmv(xd))


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("rows_per_tile,m", [(32, 32 * 7104), (32, 32 * 7104 + 1), (64, 64 * 7104 + 1)])
def test_more_tiles_than_warps(cuda, precision, rows_per_tile, m):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = m // 7104 * (48 * sms) + m % 7104                # 48 warps per SM
    lens = np.full(m, 17)
    lens[::3] = 5
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    rng = np.random.default_rng(3)
    n = 4000
    ci = rng.integers(0, n, int(rp[-1])).astype(np.int32)
    v = rng.normal(size=len(ci)).astype(np.float32).astype(np.float64)
    A = M.from_arrays(m, n, rp, ci, v)
    fp32 = precision == _abi.PREC_FP32C
    x = M.uniform(n, seed=6, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    xd = torch.from_numpy(x).cuda()
    mat = SpMatrix(A, "csr", precision=precision, lanes_per_row=1, rows_per_tile=rows_per_tile)
    y = mat.spmv(xd.float() if fp32 else xd)
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-9 if fp32 else 1e-12)[0] == 0
