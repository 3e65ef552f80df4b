"""Conversion at its edges: unaligned column arrays, chunks of many empty rows, rows spanning many
chunks, and column spans at the reach of 16-bit offsets (65,534) and one past it."""
import numpy as np
import pytest

from oracle import oracle as O
from pava_b200 import _abi
from pava_b200 import matrices as M
from pava_b200.api import SpMatrix

pytestmark = pytest.mark.gpu

FORMS = [("cvr", dict(steps=s)) for s in (32, 64, 128)]
FORMS += [("csr5", dict(sigma=s, tiles_per_chunk=g)) for s in (8, 12, 16, 24, 32) for g in (1, 3)]
FORMS += [("sell", {}), ("csr", {})]


def _csr(rows, n, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    ci = np.concatenate(rows) if rows else np.zeros(0, np.int32)
    v = rng.normal(size=int(rp[-1])).astype(np.float32).astype(np.float64)
    return M.from_arrays(len(rows), n, rp, ci, v)


def _matrices():
    rng = np.random.default_rng(1)
    cols = lambda n, k: np.sort(rng.choice(n, k, replace=False))  # noqa: E731
    yield "empty_runs", _csr([cols(900, int(k)) for k in rng.choice([0, 0, 0, 0, 1, 7, 40], 5000)], 900, 2)
    yield "long_rows", _csr([cols(30000, k) for k in (3, 0, 20000, 0, 1, 4096, 2048, 512, 0, 0, 5)], 30000, 3)
    yield "equal_rows", _csr([cols(700, 37) for _ in range(777)], 700, 4)
    yield "all_empty", _csr([np.zeros(0, np.int32)] * 1000, 10, 5)
    # every chunk starts and ends on a row: 2,048 elements of 64 rows of 32
    yield "aligned", _csr([cols(500, 32) for _ in range(256)], 500, 6)


@pytest.mark.parametrize("index", ["i32", "auto"])
@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("name,A", list(_matrices()), ids=[m[0] for m in _matrices()])
def test_forms_at_the_edges(cuda, name, A, prec, index):
    torch = cuda
    x = M.uniform(A.n, seed=7, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    xd = torch.from_numpy(x).cuda()
    xd = xd.float() if prec == _abi.PREC_FP32C else xd
    # columns and row pointer one int past a 16-byte boundary
    dev = []
    for a in (A.rp, A.ci):
        t = torch.zeros(len(a) + 1, dtype=torch.int32, device="cuda")
        t[1:] = torch.from_numpy(a)
        dev.append(t[1:])
    dev.append(torch.from_numpy(A.v).cuda())
    for fmt, kw in FORMS:
        if fmt == "sell" and not M.sell_accepts(A):
            continue
        mode = _abi.INDEX_AUTO if index == "auto" else _abi.INDEX_I32
        mat = SpMatrix(A, fmt, device_arrays=tuple(dev), precision=prec, index_mode=mode, **kw)
        bound = 1e-9 if prec == _abi.PREC_FP32C else 1e-12
        y = mat.spmv(xd).cpu().numpy()
        assert O.rel_error(y, yr, ab, bound)[0] == 0, (fmt, kw)
        mat.close()


@pytest.mark.parametrize("fmt,kw", [("cvr", {}), ("csr5", {}), ("sell", {})])
@pytest.mark.parametrize("span", [65533, 65534, 65535])
def test_reach_of_16_bit_offsets(cuda, fmt, kw, span):
    torch = cuda
    n, base = 70000, 123
    rows = [np.array([base, base + 5, base + span], np.int32) for _ in range(320)]
    A = _csr(rows, n, 8)
    x = M.uniform(n, seed=9)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    xd = torch.from_numpy(x).cuda()
    fits = span <= 65534
    mat = SpMatrix(A, fmt, index_mode=_abi.INDEX_AUTO, **kw)
    assert mat.info()["index_mode"] == (_abi.INDEX_DELTA16 if fits else _abi.INDEX_I32)
    assert O.rel_error(mat.spmv(xd).cpu().numpy(), yr, ab, 1e-12)[0] == 0
    plain = SpMatrix(A, fmt, **kw).info()["device_bytes"]
    if fits:
        SpMatrix(A, fmt, index_mode=_abi.INDEX_DELTA16, **kw)
    else:
        assert mat.info()["device_bytes"] == plain
        with pytest.raises(_abi.PavaError) as e:
            SpMatrix(A, fmt, index_mode=_abi.INDEX_DELTA16, **kw)
        assert e.value.status == _abi.E_UNSUPPORTED_PARAMS


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("where", [0, 1, 2, 3, 4, -5, -3, -2, -1])
def test_bad_column_found_at_any_alignment(cuda, shift, where):
    torch = cuda
    A = M.banded(3001, 20, 7)
    for bad in (-1, A.n):
        ci = A.ci.copy()
        ci[where] = bad
        t = torch.zeros(len(ci) + shift, dtype=torch.int32, device="cuda")
        t[shift:] = torch.from_numpy(ci)
        dev = (torch.from_numpy(A.rp).cuda(), t[shift:], torch.from_numpy(A.v).cuda())
        with pytest.raises(_abi.PavaError) as e:
            SpMatrix(A, "csr5", device_arrays=dev)
        assert e.value.status == _abi.E_INVALID_CSR


@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_FP32C])
@pytest.mark.parametrize("sigma", [8, 12, 16, 24, 32])
@pytest.mark.parametrize("rows", [60, 61, 4000])  # below and above one sample of 1,024 nonzeros
def test_scattered_columns(cuda, rows, sigma, prec):
    torch = cuda
    rng = np.random.default_rng(rows)
    A = _csr([np.sort(rng.choice(200_000, 17, replace=False)) for _ in range(rows)], 200_000, 10)
    x = M.uniform(A.n, seed=11, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    xd = torch.from_numpy(x).cuda()
    xd = xd.float() if prec == _abi.PREC_FP32C else xd
    mat = SpMatrix(A, "csr5", sigma=sigma, precision=prec)
    y = mat.spmv(xd)
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-9 if prec else 1e-12)[0] == 0
    assert torch.equal(y, mat.spmv(xd))


@pytest.mark.parametrize("extra", [-1, 0, 1, 3, 900])
def test_cvr_chunks_around_a_full_gpu(cuda, extra):
    """16 warps per SM hold one chunk each; 16-bit columns take another launch shape beyond that."""
    torch = cuda
    chunks = 16 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    m = chunks * 32                       # rows of 31 or 33 nonzeros: 1,024 elements to a chunk
    lens = np.where(np.arange(m) % 2, 33, 31)
    lens[-1] -= 1                         # not a whole number of elements
    rp = np.concatenate([[0], np.cumsum(lens)])
    k = np.arange(rp[-1]) - np.repeat(rp[:-1], lens)
    ci = (np.repeat(np.arange(m), lens) // 32 * 5 + k * 7) % 20011
    A = M.from_arrays(m, 20011, rp, ci.astype(np.int32), M.uniform(int(rp[-1]), seed=12, fp32=True))
    x = M.uniform(A.n, seed=13, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    for prec, bound in ((_abi.PREC_FP64, 1e-12), (_abi.PREC_FP32C, 1e-9)):
        for mode in (_abi.INDEX_DELTA16, _abi.INDEX_I32):
            mat = SpMatrix(A, "cvr", precision=prec, index_mode=mode, steps=32)
            xd = torch.from_numpy(x).cuda()
            y = mat.spmv(xd.float() if prec == _abi.PREC_FP32C else xd).cpu().numpy()
            assert O.rel_error(y, yr, ab, bound)[0] == 0, (prec, mode)
            mat.close()


@pytest.mark.parametrize("units", [1, 2, 147, 149, 443, 445, 591, 593, 739, 741, 2367, 2369, 3553, 4737])
def test_every_chunk_is_taken_once(cuda, units):
    """Chunk and slice counts around the CTAs and the warps that 148 SMs hold in each kernel."""
    torch = cuda
    rng = np.random.default_rng(units)
    m = 32 * units - 5                    # rows of 8: CSR5 chunks of 256 elements, slices of 32 rows
    ci = np.sort((np.arange(m)[:, None] * 3 + np.arange(8) * 11 + rng.integers(0, 11, (m, 8))) % 4999, 1)
    A = M.from_arrays(m, 4999, np.arange(0, 8 * m + 1, 8), ci.ravel().astype(np.int32),
                      M.uniform(8 * m, seed=14, fp32=True))
    x = M.uniform(A.n, seed=15, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    for fmt, kw in (("cvr", dict(steps=32)), ("csr5", dict(sigma=8, tiles_per_chunk=1)), ("sell", {})):
        for prec, bound in ((_abi.PREC_FP64, 1e-12), (_abi.PREC_FP32C, 1e-9)):
            for mode in (_abi.INDEX_DELTA16, _abi.INDEX_I32):
                mat = SpMatrix(A, fmt, precision=prec, index_mode=mode, **kw)
                xd = torch.from_numpy(x).cuda()
                y = torch.full((m,), float("nan"), dtype=torch.float64, device="cuda")
                mat.spmv(xd.float() if prec == _abi.PREC_FP32C else xd, y)
                assert O.rel_error(y.cpu().numpy(), yr, ab, bound)[0] == 0, (fmt, prec, mode)
                mat.close()


@pytest.mark.parametrize("fmt,kw", [("cvr", dict(steps=32)), ("csr5", dict(sigma=8, tiles_per_chunk=4))])
def test_rows_over_a_few_chunks(cuda, fmt, kw):
    """Rows over 1 to 40 chunks of 1,024 elements, neighbours ending in the same 32 chunks."""
    torch = cuda
    rng = np.random.default_rng(16)
    spans = [s for s in range(1, 12) for _ in range(5)] + [40, 33, 32, 31, 2, 2, 9, 8, 7]
    lens = [int(s * 1024 + rng.integers(-500, 500)) for s in rng.permutation(spans)]
    A = _csr([np.sort(rng.choice(50_000, k, replace=False)) for k in lens], 50_000, 17)
    x = M.uniform(A.n, seed=18, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    for prec, bound in ((_abi.PREC_FP64, 1e-12), (_abi.PREC_FP32C, 1e-9)):
        mat = SpMatrix(A, fmt, precision=prec, **kw)
        xd = torch.from_numpy(x).cuda()
        y = mat.spmv(xd.float() if prec == _abi.PREC_FP32C else xd)
        assert O.rel_error(y.cpu().numpy(), yr, ab, bound)[0] == 0, prec
        mat.close()


@pytest.mark.parametrize("units", [2369, 2960, 4001])
def test_cvr_scattered_16_bit_columns(cuda, units):
    """Random columns within 30,000: more chunks than 16 warps per SM hold, in one CTA per SM."""
    torch = cuda
    rng = np.random.default_rng(units)
    m = 64 * units                        # 16 nonzeros per row, 1,024 elements to a chunk
    ci = rng.integers(0, 30_000, 16 * m, dtype=np.int32)
    A = M.from_arrays(m, 30_000, np.arange(0, 16 * m + 1, 16), ci, M.uniform(16 * m, seed=20, fp32=True))
    x = M.uniform(A.n, seed=21, fp32=True)
    yr, ab = O.csr_ref(A.rp, A.ci, A.v, x)
    mat = SpMatrix(A, "cvr", index_mode=_abi.INDEX_DELTA16, steps=32)
    xd = torch.from_numpy(x).cuda()
    y = mat.spmv(xd)
    assert O.rel_error(y.cpu().numpy(), yr, ab, 1e-12)[0] == 0
    assert torch.equal(y, mat.spmv(xd))
