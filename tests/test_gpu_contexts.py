"""Programs that alternate CUDA contexts on a device: each context keeps its pool of device memory, so
that switching leaves nothing behind."""
import ctypes

import pytest

from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


def test_alternating_contexts_keep_one_pool_each(cuda):
    torch = cuda
    cu = ctypes.CDLL("libcuda.so.1")
    A = M.banded(600_000, 64, 24)  # 14.4 M nonzeros: 175 MB a handle, as much for the CSR's copy
    SpMatrix(A, "csr5").close()
    ctx, dev = ctypes.c_void_p(), ctypes.c_int()
    assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev) == 0  # and makes it current
    popped = ctypes.c_void_p()
    try:
        def both():
            SpMatrix(A, "csr5").close()
            assert cu.cuCtxPopCurrent_v2(ctypes.byref(popped)) == 0
            SpMatrix(A, "csr5").close()
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            assert cu.cuCtxPushCurrent_v2(ctx) == 0
            return free

        both()
        before = both()
        for _ in range(4):
            after = both()
        assert before - after < 64 << 20
    finally:
        cu.cuCtxPopCurrent_v2(ctypes.byref(popped))
        cu.cuCtxDestroy_v2(ctx)
    x = torch.from_numpy(M.uniform(A.n, seed=1)).cuda()
    mat = SpMatrix(A, "csr5")
    assert torch.isfinite(mat.spmv(x)).all()
