"""Row tiles dealt over the grid where its size changes: one tile, a share per SM, half a GPU, a full
one, and one tile more than each; the first products of a loop share the GPU with the ones after."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("k,shape", [(1, {}), (2, dict(col_lanes=1, cols_per_lane=2)),
                                     (4, dict(col_lanes=4, cols_per_lane=1))])
def test_tiles(cuda, per_sm, more, k, shape):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = max(1, per_sm * sms * 8 + more)  # a tile of one row per warp, eight warps a CTA
    rng = np.random.default_rng(m)
    lens = rng.integers(0, 40, m)
    lens[rng.integers(0, m, 3)] = 1100  # longer than a warp takes alone
    n = 1500
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in lens] or [[]])
    A = M.from_arrays(m, n, rp, ci, rng.normal(size=int(rp[-1])))
    mat = SpMatrix(A, "csr", lanes_per_row=32, rows_per_tile=1, **shape)
    X = M.uniform(n * k, seed=3).reshape(n, k)
    Xd = torch.from_numpy(X).cuda()
    out = [mat.spmv(Xd[:, 0].contiguous()) if k == 1 else mat.spmm(Xd) for _ in range(12)]
    assert all(torch.equal(out[0], y) for y in out[1:])
    y = out[0].cpu().numpy().reshape(m, k)
    for c in range(k):
        yr, ab = O.csr_ref(A.rp, A.ci, A.v, np.ascontiguousarray(X[:, c]))
        assert O.rel_error(np.ascontiguousarray(y[:, c]), yr, ab, 1e-12)[0] == 0
