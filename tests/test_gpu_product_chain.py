"""Products that follow one another closely: each reads the vector the one before wrote, shares its
output and carry buffers, or follows copies, events and other kernels, eagerly and in a graph.
The products overlap their launches, so any missing wait would show as a wrong or changing bit."""
import pytest

from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu

FORMS = [("cvr", {}), ("csr5", {}), ("sell", {}), ("csr", {})]
SIZES = [("small", lambda: M.laplace2d(60)), ("mid", lambda: M.laplace2d(700)),
         ("long_rows", lambda: M.banded(60_000, 900, 300))]


def _scaled(A):
    A.v = A.v / 1000.0  # powers stay finite
    return A


@pytest.mark.parametrize("fmt,kw", FORMS, ids=[f[0] for f in FORMS])
@pytest.mark.parametrize("name,make", SIZES, ids=[s[0] for s in SIZES])
def test_each_product_reads_the_one_before(cuda, name, make, fmt, kw):
    torch = cuda
    A = _scaled(make())
    mat = SpMatrix(A, fmt, index_mode=_abi.INDEX_AUTO if fmt != "csr" else 0, **kw)
    x0 = torch.from_numpy(M.uniform(A.n, seed=2)).cuda()
    want = [x0.clone()]
    for _ in range(12):
        want.append(mat.spmv(want[-1]).clone())
        torch.cuda.synchronize()
    for _ in range(3):
        a, b = x0.clone(), torch.empty_like(x0)
        for _ in range(6):
            mat.spmv(a, b)
            mat.spmv(b, a)
        assert torch.equal(a, want[12])
        # one output buffer for different vectors, copied out in between
        y, out = torch.empty_like(x0), []
        for v in want[:6]:
            mat.spmv(v, y)
            out.append(y.clone())
        assert all(torch.equal(o, w) for o, w in zip(out, want[1:7]))
        # a vector written by another kernel just before, and overwritten just after
        v = torch.zeros_like(x0)
        v.copy_(want[3])
        mat.spmv(v, y)
        v.fill_(float("nan"))
        assert torch.equal(y, want[4])


@pytest.mark.parametrize("fmt,kw", FORMS, ids=[f[0] for f in FORMS])
def test_two_streams_and_events(cuda, fmt, kw):
    torch = cuda
    A = _scaled(M.laplace2d(500))
    mats = [SpMatrix(A, fmt, **kw) for _ in range(2)]
    x0 = torch.from_numpy(M.uniform(A.n, seed=3)).cuda()
    want = mats[0].spmv(mats[0].spmv(x0)).clone()
    big = torch.empty(1 << 28, dtype=torch.float32, device="cuda")
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(10):
        mid, y, v = torch.empty_like(x0), torch.empty_like(x0), torch.zeros_like(x0)
        torch.cuda.synchronize()
        with torch.cuda.stream(s1):
            mats[0].spmv(v, mid)      # a product before the delay, on the stream that delays
            big.zero_()               # a long kernel the other stream has to wait for
            v.copy_(x0)
            mats[0].spmv(v, mid)
            done = s1.record_event()
        with torch.cuda.stream(s2):
            mats[1].spmv(v, y)        # reads whatever v holds; its result is overwritten
            s2.wait_event(done)
            mats[1].spmv(mid, y)
        s2.synchronize()
        assert torch.equal(y, want)


@pytest.mark.parametrize("fmt,kw", FORMS, ids=[f[0] for f in FORMS])
def test_captured_with_other_nodes(cuda, fmt, kw):
    torch = cuda
    A = _scaled(M.laplace2d(300))
    mat = SpMatrix(A, fmt, **kw)
    x = torch.from_numpy(M.uniform(A.n, seed=4)).cuda()
    src = x.clone()
    a, b, y = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)

    def body():
        a.copy_(src)          # a copy node before a product
        mat.spmv(a, b)
        mat.spmv(b, a)
        y.zero_()             # a memset between
        mat.spmv(a, y)
        y.add_(b)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        body()
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        body()
    for seed in range(5, 10):
        src.copy_(torch.from_numpy(M.uniform(A.n, seed=seed)).cuda())
        for _ in range(5):
            g.replay()
        torch.cuda.synchronize()
        first = mat.spmv(src)
        torch.cuda.synchronize()
        want = mat.spmv(mat.spmv(first)) + first
        assert torch.equal(y, want)


@pytest.mark.parametrize("fmt,k", [("csr", 8), ("csr", 3), ("sell", 8), ("sell", 32)])
def test_several_right_hand_sides(cuda, fmt, k):
    torch = cuda
    A = _scaled(M.banded(30_000, 64, 24))
    mat = SpMatrix(A, fmt)
    X = torch.rand((A.n, k), dtype=torch.float64, device="cuda")
    want = [X]
    for _ in range(6):
        want.append(mat.spmm(want[-1]).clone())
        torch.cuda.synchronize()
    for _ in range(5):
        a, b = X.clone(), torch.empty_like(X)
        for _ in range(3):
            mat.spmm(a, b)
            mat.spmm(b, a)
        assert torch.equal(a, want[6])
