"""Arrays that pava_coo_to_csr_device returns are ordinary device memory (CUDA IPC takes them), the
pooled form returns the same values; a refused input gives everything back."""
import ctypes

import numpy as np
import pytest

from pava_b200 import _abi
from pava_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _coo(torch, n, nnz, bad=False):
    rng = np.random.default_rng(5)
    r, c = rng.integers(0, n, nnz).astype(np.int32), rng.integers(0, n, nnz).astype(np.int32)
    if bad:
        c[nnz // 2] = n
    return [torch.from_numpy(a).cuda() for a in (r, c, rng.normal(size=nnz))]


def _call(name, n, coo):
    out = _abi.PavaCsr()
    r, c, v = coo
    st = getattr(_abi.gpu(), name)(n, n, r.numel(), r.data_ptr(), c.data_ptr(), v.data_ptr(), 0, 0,
                                   None, ctypes.byref(out))
    return st, out


def test_results_can_be_shared_between_processes(cuda):
    torch = cuda
    cu = ctypes.CDLL("libcuda.so.1")
    st, out = _call("pava_coo_to_csr_device", 5000, _coo(torch, 5000, 60_000))
    assert st == 0
    handle = (ctypes.c_char * 64)()
    for p in (out.row_ptr, out.col_idx, out.vals):
        assert cu.cuIpcGetMemHandle(handle, ctypes.c_uint64(p)) == 0
    assert _abi.gpu().pava_free_device_csr(ctypes.byref(out)) == 0


@pytest.mark.parametrize("n,nnz", [(5000, 60_000), (1, 0), (70, 30_000)])
def test_both_forms_agree(cuda, n, nnz):
    torch = cuda
    coo = _coo(torch, n, nnz)
    got = []
    for name in ("pava_coo_to_csr_device", "pava_coo_to_csr_device_pooled"):
        st, out = _call(name, n, coo)
        assert st == 0 and out.nnz == nnz
        got.append([torch.as_tensor(M._DevView(p, k, t), device="cuda").clone() if k else None
                    for p, k, t in ((out.row_ptr, n + 1, "<i4"), (out.col_idx, nnz, "<i4"),
                                    (out.vals, nnz, "<f8"))])
        _abi.gpu().pava_free_device_csr(ctypes.byref(out))
    assert all(a is b or torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("name", ["pava_coo_to_csr_device", "pava_coo_to_csr_device_pooled"])
def test_refused_input_leaves_nothing(cuda, name):
    torch = cuda
    coo = _coo(torch, 1_000_000, 8_000_000, bad=True)
    assert _call(name, 1_000_000, coo)[0] == _abi.E_INVALID_CSR
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        st, out = _call(name, 1_000_000, coo)
        assert st == _abi.E_INVALID_CSR and not out.row_ptr
    torch.cuda.synchronize()
    assert abs(before - torch.cuda.mem_get_info()[0]) < 8 << 20


def test_freed_in_the_stream_that_still_reads_it(cuda):
    torch = cuda
    coo = _coo(torch, 200_000, 3_000_000)
    want = torch.sort(coo[2]).values
    s = torch.cuda.Stream()
    big = torch.zeros(1 << 26, device="cuda")
    torch.cuda.synchronize()
    got = []
    for _ in range(4):  # the next conversion takes the memory the last one gave back
        st, out = _call("pava_coo_to_csr_device_pooled", 200_000, coo)
        assert st == 0
        with torch.cuda.stream(s):
            for _ in range(20):
                big.add_(1.0)
            got.append(torch.as_tensor(M._DevView(out.vals, out.nnz, "<f8"), device="cuda").clone())
            assert _abi.gpu().pava_free_device_csr_async(ctypes.byref(out), s.cuda_stream) == 0
        assert not out.vals
    torch.cuda.synchronize()
    assert all(torch.equal(torch.sort(g).values, want) for g in got)
