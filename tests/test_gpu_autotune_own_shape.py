"""The autotuner times the shape that pava_spmm runs when a handle names none, for every k."""
import pytest

from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import Batch, SpMatrix, autotune

pytestmark = pytest.mark.gpu
SHAPE = ("lanes_per_row", "col_lanes", "cols_per_lane", "rows_per_tile", "x_window")
# the shapes k_csr_spmm.cu runs up to k = 32, as options name them
NAMED = {3: (4, 4, 1, 32, 0), 8: (4, 4, 2, 32, 0), 16: (4, 4, 4, 32, 0), 21: (8, 8, 4, 16, 0), 32: (8, 8, 4, 16, 0)}


@pytest.mark.parametrize("k", [3, 8, 16, 21, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_FP32C])
def test_own_shape_is_timed(cuda, k, prec):
    ents, best = autotune(M.banded(20_000, 64, 24, seed=3), k=k, precision=prec, reps=1)
    shapes = [tuple(e["opts"][o] for o in SHAPE) for e in ents if e["format"] == "csr" and e["status"] == 0]
    assert shapes.count(NAMED.get(k, (0, 0, 0, 0, 0))) == 1
    assert ents[best]["ms"] == min(e["ms"] for e in ents if e["ms"] > 0)


def test_a_batch_takes_it(cuda):
    torch = cuda
    A = M.banded(60_000, 64, 24, seed=4)
    b = Batch([A], "auto", k=128)
    X = torch.rand((A.n, 128), dtype=torch.float64, device="cuda")
    Y, want = b.spmm(X), SpMatrix(A, "csr").spmm(X)
    scale = SpMatrix(M.from_arrays(A.m, A.n, A.rp, A.ci, abs(A.v)), "csr").spmm(X)
    assert ((Y - want).abs() <= 1e-12 * scale).all()
