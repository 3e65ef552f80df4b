"""Destroying a handle waits for the device as cudaFree does: beside a stream capture that allows
cudaFree (relaxed, or thread-local in another thread) it leaves the capture whole."""
import threading

import pytest

from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,elsewhere", [("relaxed", False), ("relaxed", True),
                                            ("thread_local", True)])
def test_capture_survives(cuda, mode, elsewhere):
    torch = cuda
    A = M.laplace2d(50)
    keep = SpMatrix(A, "csr5")
    x = torch.from_numpy(M.uniform(A.n, seed=1)).cuda()
    y = torch.zeros(A.m, dtype=torch.float64, device="cuda")
    want = keep.spmv(x).clone()
    gone = [SpMatrix(A, "csr5") for _ in range(2)]
    torch.cuda.synchronize()

    def close():
        for m in gone:
            m.close()

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        keep.spmv(x, y)
        if elsewhere:
            t = threading.Thread(target=close)
            t.start()
            t.join()
        else:
            close()
        keep.spmv(x, y)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert torch.equal(SpMatrix(A, "csr5").spmv(x), want)  # no error is left behind


def test_close_waits_for_the_device(cuda):
    torch = cuda
    A = M.laplace2d(50)
    SpMatrix(A, "csr5").close()
    mat = SpMatrix(A, "csr5")
    big = torch.zeros(1 << 27, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for _ in range(200):  # tens of milliseconds
            big.add_(1.0)
        done = s.record_event()
    mat.close()
    assert done.query()
