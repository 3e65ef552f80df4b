"""CSR5 at the chunk counts where its launch shape changes: one and two waves of 20 or 24 warps per
SM, and one chunk more, each precision and column form; rows that run over chunks."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [20, 24, 40, 48])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("sigma", [8, 12, 32])
@pytest.mark.parametrize("precision,index", [(_abi.PREC_FP64, _abi.INDEX_I32), (_abi.PREC_FP32C, _abi.INDEX_I32),
                                             (_abi.PREC_FP32C, _abi.INDEX_AUTO)])
def test_waves(cuda, warps, more, sigma, precision, index):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chunks = warps * sms + more
    nnz = (chunks - 1) * 32 * sigma + 7       # the last chunk holds seven nonzeros
    rng = np.random.default_rng(chunks)
    lens = rng.integers(1, 25, nnz // 12)
    lens[::997] = 3 * 32 * sigma + 5          # over several chunks
    ends = np.minimum(np.cumsum(lens), nnz)
    ends = ends[: np.searchsorted(ends, nnz) + 1]
    ends[-1] = nnz
    rp = np.concatenate([[0], ends]).astype(np.int32)
    m, n = len(rp) - 1, 4000
    ci = rng.integers(0, n, nnz).astype(np.int32)  # any order, duplicates
    v = rng.normal(size=nnz).astype(np.float32).astype(np.float64)
    A = M.from_arrays(m, n, rp, ci, v)
    fp32 = precision == _abi.PREC_FP32C
    mat = SpMatrix(A, "csr5", sigma=sigma, tiles_per_chunk=1, precision=precision, index_mode=index)
    assert mat.info()["chunks"] == chunks
    x = M.uniform(n, seed=2, fp32=True)
    xd = torch.from_numpy(x).cuda()
    xd = xd.float() if fp32 else xd
    y = mat.spmv(xd)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-9 if fp32 else 1e-12)[0] == 0  # the stated bounds
    assert torch.equal(y, mat.spmv(xd))
