"""COO -> CSR on a stream that is being captured is refused and leaves the capture whole."""
import ctypes

import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def test_refused_without_ending_the_capture(cuda):
    torch = cuda
    A = M.laplace2d(50)
    mat = SpMatrix(A, "csr5")
    x = torch.from_numpy(M.uniform(A.n, seed=1)).cuda()
    y = torch.zeros(A.m, dtype=torch.float64, device="cuda")
    rows = torch.tensor([0, 1, 1], dtype=torch.int32, device="cuda")
    cols = torch.tensor([1, 0, 1], dtype=torch.int32, device="cuda")
    vals = torch.ones(3, dtype=torch.float64, device="cuda")
    mat.spmv(x, y)
    torch.cuda.synchronize()
    out = _abi.PavaCsr()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st = _abi.gpu().pava_coo_to_csr_device(
            2, 2, 3, rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), 0, 0,
            _abi.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(out))
        mat.spmv(x, y)
    assert st == _abi.E_CUDA
    assert not out.row_ptr
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x.cpu().numpy())
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-12)[0] == 0
    rp, ci, _ = M.coo_to_csr_device(2, 2, rows, cols, vals)
    assert rp.tolist() == [0, 1, 3] and ci.tolist() == [1, 0, 1]
