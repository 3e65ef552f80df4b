"""A product captured after a fork and a join of two streams, with a product on each of them as its
predecessors: what it reads comes from the other stream's one."""
import pytest

from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 8])
@pytest.mark.parametrize("fmt", ["cvr", "csr5", "sell", "csr"])
@pytest.mark.parametrize("grid", [60, 500])
def test_join_of_two_products(cuda, grid, fmt, k):
    if k > 1 and fmt in ("cvr", "csr5"):
        pytest.skip("one right-hand side")
    torch = cuda
    A = M.laplace2d(grid)
    A.v = A.v / 1000.0
    a, b = SpMatrix(A, fmt), SpMatrix(A, fmt)
    product = (lambda mat, x, y: mat.spmm(x, y)) if k > 1 else (lambda mat, x, y: mat.spmv(x, y))

    def vector(seed):
        x = torch.from_numpy(M.uniform(A.n * k, seed=seed)).cuda()
        return x.reshape(A.n, k) if k > 1 else x

    src = vector(1)
    x, p, q, y, z = (torch.zeros_like(src) for _ in range(5))
    s, other = torch.cuda.Stream(), torch.cuda.Stream()

    def body():
        x.copy_(src)
        other.wait_stream(torch.cuda.current_stream())
        product(a, x, p)
        with torch.cuda.stream(other):
            product(b, x, q)
            product(b, q, z)
            product(b, z, q)
        torch.cuda.current_stream().wait_stream(other)
        product(a, q, y)
        product(a, y, p)

    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        body()
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        body()
    for seed in range(2, 8):
        src.copy_(vector(seed))
        for _ in range(4):
            g.replay()
        torch.cuda.synchronize()
        want = src
        for _ in range(5):
            want = product(a, want, torch.empty_like(want))
            torch.cuda.synchronize()
        assert torch.equal(p, want)
