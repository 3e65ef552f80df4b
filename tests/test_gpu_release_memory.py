"""The device memory kept between conversions can be given back; handles that exist keep theirs."""
import pytest

import pava_b200
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_memory_is_given_back(cuda):
    torch = cuda
    A = M.banded(1_000_000, 64, 24)  # 24 M nonzeros: 290 MB a handle
    small = M.laplace2d(50)
    keep = SpMatrix(small, "csr5")
    x = torch.from_numpy(M.uniform(small.n, seed=1)).cuda()
    want = keep.spmv(x).clone()
    pava_b200.release_memory()
    before = _free(torch)
    SpMatrix(A, "csr5").close()
    assert before - _free(torch) > 100 << 20  # kept for the next conversion
    pava_b200.release_memory(keep=200 << 20)
    assert before - _free(torch) <= 264 << 20
    pava_b200.release_memory()
    assert abs(before - _free(torch)) <= 64 << 20
    assert torch.equal(keep.spmv(x), want)
    mat = SpMatrix(A, "cvr")
    xa = torch.from_numpy(M.uniform(A.n, seed=2)).cuda()
    y = mat.spmv(xa).clone()
    pava_b200.release_memory()  # beside a handle in use
    assert torch.equal(mat.spmv(xa), y)
