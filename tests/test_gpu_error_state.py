"""A product that cannot be launched reports it once: calls after it do not see its error again."""
import ctypes

import pytest

from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,k", [("cvr", 1), ("csr5", 1), ("sell", 1), ("csr", 1), ("csr", 8), ("sell", 8)])
def test_after_a_product_on_an_invalid_capture(cuda, fmt, k):
    torch = cuda
    cu = ctypes.CDLL("libcuda.so.1")
    A = M.laplace2d(50)
    mat = SpMatrix(A, fmt)
    x = torch.from_numpy(M.uniform(A.n * k, seed=1)).cuda()
    x = x.reshape(A.n, k) if k > 1 else x
    y = torch.zeros_like(x)
    go = mat.spmm if k > 1 else mat.spmv
    go(x, y)
    want = y.clone()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    stream, graph = ctypes.c_void_p(s.cuda_stream), ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(stream, 0) == 0
    cu.cuCtxSynchronize()  # no capture allows it: it ends this one
    try:
        with pytest.raises(_abi.PavaError) as e:
            go(x, y, s)
    finally:
        cu.cuStreamEndCapture(stream, ctypes.byref(graph))
    assert e.value.status == _abi.E_CUDA
    again = SpMatrix(A, fmt)
    (again.spmm if k > 1 else again.spmv)(x, y)
    torch.cuda.synchronize()
    assert torch.equal(y, want)
