"""Device memory kept between handles: bounded, given back by a failed conversion, safe for work
still in flight, for several threads and streams, and refused (not recorded) during capture."""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu
KEEP = 1 << 30


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_memory_is_bounded(cuda):
    torch = cuda
    A = M.banded(1_200_000, 64, 24)  # 28.8 M nonzeros: 350 MB a handle
    dev = tuple(torch.from_numpy(a).cuda() for a in (A.rp, A.ci, A.v))
    before = _free(torch)
    mats = [SpMatrix(A, "csr5", device_arrays=dev) for _ in range(5)]  # 1.7 GB at once
    for m in mats:
        m.close()
    assert before - _free(torch) <= KEEP + (64 << 20)
    for _ in range(4):
        SpMatrix(A, "cvr", device_arrays=dev).close()
    assert before - _free(torch) <= KEEP + (64 << 20)


def test_close_waits_for_products_in_flight(cuda):
    torch = cuda
    A, B = M.powerlaw(400_000, seed=3), M.powerlaw(400_000, seed=4)
    x = torch.from_numpy(M.uniform(A.n, seed=5)).cuda()
    want = [SpMatrix(Z, "csr5").spmv(x).clone() for Z in (A, B)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    for _ in range(5):
        got = []
        for Z in (A, B):  # the second handle takes the first one's memory
            mat = SpMatrix(Z, "csr5")
            with torch.cuda.stream(s):
                for _ in range(20):
                    y = mat.spmv(x)
            mat.close()
            got.append(y)
        s.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_threads_with_streams_of_their_own(cuda):
    torch = cuda
    mats = [M.powerlaw(60_000 + 7 * i, seed=i) for i in range(4)]
    x = [torch.from_numpy(M.uniform(A.n, seed=9)).cuda() for A in mats]
    want = [SpMatrix(A, "cvr").spmv(v).clone() for A, v in zip(mats, x)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        torch.cuda.set_device(0)
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(15):
                mat = SpMatrix(mats[i], "cvr", stream=s)
                y = mat.spmv(x[i])
                s.synchronize()
                if not torch.equal(y, want[i]):
                    bad.append(i)
                mat.close()

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(mats))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_conversion_on_a_capturing_stream_is_refused(cuda):
    torch = cuda
    A = M.laplace2d(50)
    mat = SpMatrix(A, "csr5")
    x = torch.from_numpy(M.uniform(A.n, seed=1)).cuda()
    y = torch.zeros(A.m, dtype=torch.float64, device="cuda")
    dev = tuple(torch.from_numpy(a).cuda() for a in (A.rp, A.ci, A.v))
    mat.spmv(x, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        with pytest.raises(_abi.PavaError) as e:
            SpMatrix(A, "csr5", device_arrays=dev, stream=torch.cuda.current_stream())
        mat.spmv(x, y)
    assert e.value.status == _abi.E_CUDA
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x.cpu().numpy())
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-12)[0] == 0


@pytest.mark.parametrize("fmt", ["cvr", "csr5", "csr", "sell"])
def test_invalid_matrix_gives_its_memory_back(cuda, fmt):
    torch = cuda
    A = M.banded(1_500_000, 64, 24)
    ci = A.ci.copy()
    ci[12345] = A.n  # out of range
    dev = tuple(torch.from_numpy(a).cuda() for a in (A.rp, ci, A.v))
    host = M.from_arrays(A.m, A.n, A.rp, ci, A.v)
    SpMatrix(M.laplace2d(20), fmt).close()
    before = _free(torch)
    for arrays in (dev, None):
        with pytest.raises(_abi.PavaError) as e:
            SpMatrix(host, fmt, device_arrays=arrays)
        assert e.value.status == _abi.E_INVALID_CSR
        assert abs(before - _free(torch)) < (8 << 20)
