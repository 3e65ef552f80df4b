"""The work this engine's users have it do, as cases that can be timed and compared.

Each case is one call (or one short sequence of calls) of the public Python interface on a
seeded synthetic matrix of the families the repository benchmarks on:

* ``spmv``    y = A x on a converted matrix that is kept (SpMatrix.spmv): the timed loop of the
              benchmark driver and the inner step of an iterative solver
* ``spmm``    Y = A X for k right-hand sides on a kept matrix (SpMatrix.spmm)
* ``batch``   many uneven small matrices, one launch replayed from a CUDA graph (Batch.replay)
* ``convert`` a CSR on the device converted into a form, multiplied once and dropped: the
              "convert" column of the benchmark's Performance line, paid for each new matrix
* ``coo``     the loader's COO -> sorted CSR conversion on the device (coo_to_csr_device)
* ``train``   full-batch training of the form selector's network (Network.train): forward,
              backward and Adam steps from given weights

Matrices are generated with torch on the GPU: row lengths from the case (so that the work is the
same for every seed), columns, values and vectors from the seed alone.
"""
import math

import numpy as np
import torch

from pava_b200 import _abi
from pava_b200.api import Batch, SpMatrix
from pava_b200.matrices import CSR, coo_to_csr_device
from pava_b200.selector import Network

PREC = {"fp64": _abi.PREC_FP64, "fp32c": _abi.PREC_FP32C}
INDEX = {"i32": _abi.INDEX_I32, "auto": _abi.INDEX_AUTO}
DEV = "cuda"


def listed():
    return [
        # the plain drop-in on a 512 x 512 grid's 5-point Laplacian: the smallest product, where
        # launches and latency count
        {"name": "laplacian_cvr", "op": "spmv", "family": "laplace", "size": 512, "form": "cvr",
         "precision": "fp64", "index": "auto"},
        # the headline: irregular power-law matrix, 4,194,304 rows, about 66 M nonzeros
        {"name": "powerlaw_cvr", "op": "spmv", "family": "powerlaw", "size": 4194304,
         "form": "cvr", "precision": "fp64", "index": "auto"},
        # the same family in the other drop-in form, ordinary size, odd row count
        {"name": "powerlaw_csr5", "op": "spmv", "family": "powerlaw", "size": 1300021,
         "form": "csr5", "precision": "fp64", "index": "auto"},
        # regular matrix in the drop-in form: 27-point stencil on a 128^3 grid
        {"name": "stencil_csr5", "op": "spmv", "family": "stencil27", "size": 128,
         "form": "csr5", "precision": "fp64", "index": "auto"},
        # the single-precision storage form on the same stencil, in the form the autotuner picks
        {"name": "stencil_sell_fp32c", "op": "spmv", "family": "stencil27", "size": 128,
         "form": "sell", "precision": "fp32c", "index": "auto"},
        # plain CSR rows of very uneven length (no conversion beyond a copy)
        {"name": "powerlaw_csr", "op": "spmv", "family": "powerlaw", "size": 700001,
         "form": "csr", "precision": "fp64", "index": "i32"},
        # several right-hand sides: banded matrix of 1,048,576 rows, 24 nonzeros per row
        {"name": "banded_csr_k8", "op": "spmm", "family": "banded", "size": 1048576,
         "form": "csr", "precision": "fp64", "index": "i32", "k": 8},
        {"name": "banded_sell_k32", "op": "spmm", "family": "banded", "size": 1048576,
         "form": "sell", "precision": "fp64", "index": "auto", "k": 32},
        # a batch of uneven random matrices (256 to 32,768 rows, 12 nonzeros per row on
        # average) replayed from a graph, single-precision storage
        {"name": "batch_csr5_fp32c", "op": "batch", "count": 256, "form": "csr5",
         "precision": "fp32c", "index": "auto"},
        # a new matrix every time: convert and multiply once
        {"name": "convert_csr5", "op": "convert", "family": "stencil27", "size": 97,
         "form": "csr5", "precision": "fp64", "index": "auto"},
        # a symmetric Matrix Market file's triangle, 1-based and column-major, expanded to CSR
        {"name": "coo_symmetric", "op": "coo", "family": "stencil27", "size": 80,
         "symmetric": True, "shuffled": False},
        # 40 training steps of the selector's network on 2,000 samples
        {"name": "selector_train", "op": "train", "samples": 2000, "epochs": 40},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_matrix(rng, lo, hi, families):
    """A family and a size giving about lo .. hi nonzeros."""
    family = rng.choice(families)
    nnz = _log(rng, lo, hi)
    if family == "laplace":
        return family, max(3, int(math.sqrt(nnz / 5)))
    if family == "stencil27":
        return family, max(3, int((nnz / 27) ** (1 / 3)))
    return family, int(nnz / {"banded": 24, "powerlaw": 16, "blocks": 42}[family])


def draw(rng):
    op = rng.choice(["spmv"] * 5 + ["spmm"] * 2 + ["batch", "convert", "coo", "train"])
    if op == "train":
        return {"op": op, "samples": int(_log(rng, 500, 4000)), "epochs": rng.randint(10, 40)}
    prec = rng.choice(["fp64", "fp64", "fp32c"])
    if op == "batch":
        form = rng.choice(["cvr", "csr5", "csr"])
        return {"op": op, "count": int(_log(rng, 64, 300)), "form": form, "precision": prec,
                "index": "i32" if form == "csr" else "auto"}
    if op == "coo":
        family, size = _draw_matrix(rng, 2e6, 1.5e7, ["stencil27", "banded", "blocks", "powerlaw"])
        return {"op": op, "family": family, "size": size,
                "symmetric": family != "powerlaw" and rng.random() < 0.5,
                "shuffled": rng.random() < 0.3}
    if op == "spmm":
        family, size = _draw_matrix(rng, 2.5e6, 2.5e7, ["banded", "stencil27", "blocks"])
        return {"op": op, "family": family, "size": size, "form": rng.choice(["csr", "sell"]),
                "precision": prec, "index": "i32", "k": rng.choice([2, 4, 5, 8, 12, 16, 21, 32])}
    forms = ["cvr", "csr5", "csr", "sell"]
    form = rng.choice(forms)
    families = ["laplace", "stencil27", "banded", "blocks"] + ([] if form == "sell" else ["powerlaw"] * 3)
    lo, hi = (1.3e6, 5.5e7) if op == "spmv" else (2e6, 3e7)
    family, size = _draw_matrix(rng, lo, hi, families)
    return {"op": op, "family": family, "size": size, "form": form, "precision": prec,
            "index": "i32" if form == "csr" else rng.choice(["auto", "auto", "i32"])}


# ---- matrices ------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _lattice(g, dims, offsets):
    """Row pointer and sorted columns of a stencil on a g^dims grid."""
    m = g ** dims
    r = torch.arange(m, device=DEV, dtype=torch.int32)
    coords = [(r // g ** (dims - 1 - d)) % g for d in range(dims)]
    cols = torch.empty((m, len(offsets)), device=DEV, dtype=torch.int32)
    ok = torch.ones((m, len(offsets)), device=DEV, dtype=torch.bool)
    for j, off in enumerate(offsets):
        shift = 0
        for d in range(dims):
            shift = shift * g + off[d]
            if off[d]:
                c = coords[d] + off[d]
                ok[:, j] &= (c >= 0) & (c < g)
        cols[:, j] = r + shift
    length = ok.sum(1)
    return m, length, cols[ok]


def _strata(lo, width, count, j, u):
    """Column j of `count` distinct ascending ones in [lo, lo + width): one per stratum."""
    a = j * width // count
    b = (j + 1) * width // count
    return lo + a + torch.minimum((u * (b - a)).long(), b - a - 1)


def _rp(length):
    rp = torch.zeros(length.numel() + 1, device=DEV, dtype=torch.int32)
    rp[1:] = torch.cumsum(length, 0)
    return rp


def _spread(length, lo, width, g):
    """Columns of rows of the given lengths, spread over each row's [lo, lo + width)."""
    m = length.numel()
    rp = torch.zeros(m + 1, device=DEV, dtype=torch.int64)
    rp[1:] = torch.cumsum(length, 0)
    nnz = int(rp[-1])
    ci = torch.empty(nnz, device=DEV, dtype=torch.int32)
    for r0 in range(0, m, 1 << 20):  # bounded temporaries
        r1 = min(m, r0 + (1 << 20))
        a, b = int(rp[r0]), int(rp[r1])
        row = torch.repeat_interleave(torch.arange(r0, r1, device=DEV), length[r0:r1])
        j = torch.arange(a, b, device=DEV) - rp[row]
        u = torch.rand(b - a, device=DEV, generator=g, dtype=torch.float64)
        ci[a:b] = _strata(lo[row], width[row], length[row], j, u).int()
    return rp.int(), ci


def _matrix(family, size, seed, fp32):
    """(m, n, row pointer, columns, FP64 values) on the GPU; fp32: FP32-representable values."""
    g = _gen(seed)
    if family in ("laplace", "stencil27"):
        if family == "laplace":
            m, length, ci = _lattice(size, 2, [(-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)])
        else:
            m, length, ci = _lattice(size, 3, [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1)
                                               for c in (-1, 0, 1)])
        rp = _rp(length)
        row = torch.repeat_interleave(torch.arange(m, device=DEV), length)
        diag = ci == row
        if family == "laplace":  # 4 on the diagonal, -1 beside it
            v = torch.where(diag, 4.0, -1.0).double()
        else:  # off-diagonals U[-1, 0], diagonal 1.01 times the absolute row sum, FP32 values
            v = -torch.rand(ci.numel(), device=DEV, generator=g, dtype=torch.float32).double()
            v[diag] = 0.0
            s = torch.zeros(m, device=DEV, dtype=torch.float64).index_add_(0, row, v.abs())
            v[diag] = (1.01 * s).float().double()
        return m, m, rp, ci, v
    m = int(size)
    gl = _gen(m)  # row lengths belong to the case, columns and values to the seed
    if family == "banded":  # 24 per row within 64 of the diagonal
        w = min(129, m)
        length = torch.full((m,), min(24, w), device=DEV, dtype=torch.int64)
        lo = (torch.arange(m, device=DEV) - 64).clamp(0, m - w)
        rp, ci = _spread(length, lo, torch.full_like(lo, w), g)
    elif family == "powerlaw":  # lognormal lengths: mean 16, sigma 1.5, cap 200,000, 2 % empty
        z = torch.randn(m, device=DEV, generator=gl, dtype=torch.float64)
        length = torch.exp(math.log(16.0) - 1.125 + 1.5 * z).round().clamp(1, min(m, 200000)).long()
        length[torch.rand(m, device=DEV, generator=gl) < 0.02] = 0
        rp, ci = _spread(length, torch.zeros_like(length), torch.full_like(length, m), g)
    else:  # dense diagonal blocks of 8 .. 64 rows
        sizes = torch.randint(8, 65, (m // 8 + 1,), device=DEV, generator=gl)
        ends = torch.cumsum(sizes, 0).clamp(max=m)
        row = torch.arange(m, device=DEV)
        blk = torch.searchsorted(ends, row, right=True)
        lo = torch.where(blk > 0, ends[(blk - 1).clamp(min=0)], torch.zeros_like(row))
        length = ends[blk] - lo
        rp, ci = _spread(length, lo, length, g)
    v = torch.randn(ci.numel(), device=DEV, generator=g, dtype=torch.float64)
    return m, m, rp, ci, v.float().double() if fp32 else v


def _vector(shape, seed, fp32):
    x = torch.rand(shape, device=DEV, generator=_gen(seed + 7919), dtype=torch.float64) * 2 - 1
    return x.float() if fp32 else x


def _batch_sizes(case):
    """Rows of each matrix of a batch: log-uniform in [256, 32,768] (the same for every seed)."""
    r = np.random.default_rng(case["count"])
    return np.exp(r.uniform(math.log(256), math.log(32768), case["count"])).astype(np.int64)


def _batch_union(case, seed):
    """The batch's matrices stacked: sizes, Poisson(12) row lengths, local columns, values."""
    g = _gen(seed)
    sizes = _batch_sizes(case)
    n_row = torch.repeat_interleave(torch.from_numpy(sizes).to(DEV), torch.from_numpy(sizes).to(DEV))
    mean = torch.full((n_row.numel(),), 12.0, device=DEV)
    length = torch.poisson(mean, generator=_gen(case["count"])).long()
    rp, ci = _spread(length, torch.zeros_like(n_row), n_row, g)
    v = torch.randn(ci.numel(), device=DEV, generator=g, dtype=torch.float64)
    return sizes, rp, ci, v.float().double() if case["precision"] == "fp32c" else v


def _coo(case, seed):
    """1-based COO arrays: the lower triangle (symmetric) or every entry, column-major as Matrix
    Market files are written, or in random order."""
    m, n, rp, ci, v = _matrix(case["family"], case["size"], seed, False)
    row = torch.repeat_interleave(torch.arange(m, device=DEV), (rp[1:] - rp[:-1]).long())
    col = ci.long()
    if case["symmetric"]:
        keep = row >= col
        row, col, v = row[keep], col[keep], v[keep]
    if case["shuffled"]:
        order = torch.randperm(row.numel(), device=DEV, generator=_gen(seed + 1))
    else:
        order = torch.argsort(col, stable=True)
    return m, n, (row[order] + 1).int(), (col[order] + 1).int(), v[order].contiguous()


def _train_data(case, seed):
    r = np.random.default_rng(seed)
    B = case["samples"]
    X = r.normal(size=(B, _abi.MLP_IN)).astype(np.float32)
    W = r.normal(size=(_abi.MLP_IN, _abi.MLP_OUT)) / 4
    T = (np.tanh(X @ W) + 0.1 * r.normal(size=(B, _abi.MLP_OUT))).astype(np.float32)
    mask = (r.uniform(size=(B, _abi.MLP_OUT)) > 0.05).astype(np.float32)
    P = np.concatenate([(r.uniform(-1, 1, o * i) * math.sqrt(6 / i)).tolist() + [0.0] * o
                        for o, i in ((64, 12), (64, 64), (32, 64))]).astype(np.float32)
    return X, T, mask, P


LR = 3e-3


# ---- the cases ------------------------------------------------------------------------------

def prepare(case, seed):
    op = case["op"]
    if op == "train":
        X, T, mask, P = _train_data(case, seed)
        net = Network(0)
        net.set_batch(X, T, mask)
        return {"op": op, "net": net, "P": P, "epochs": case["epochs"]}
    if op == "coo":
        return {"op": op, "coo": _coo(case, seed), "symmetric": case["symmetric"]}
    fp32 = case["precision"] == "fp32c"
    opts = {"precision": PREC[case["precision"]], "index_mode": INDEX[case["index"]]}
    if op == "batch":
        sizes, rp, ci, v = _batch_union(case, seed)
        rp, ci, v = rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()
        mats, r0 = [], 0
        for n in sizes.tolist():
            a, b = rp[r0], rp[r0 + n]
            mats.append(CSR(n, n, rp[r0:r0 + n + 1] - a, ci[a:b], v[a:b]))
            r0 += n
        if case["form"] == "cvr":
            opts["steps"] = 128  # the forms the autotuner picks for such batches
        elif case["form"] == "csr5":
            opts["sigma"] = 32
        batch = Batch(mats, case["form"], **opts)
        x = _vector(batch.n, seed, fp32)
        y = torch.empty(batch.m, dtype=torch.float64, device=DEV)
        batch.capture(x, y)
        return {"op": op, "batch": batch, "x": x, "y": y}
    m, n, rp, ci, v = _matrix(case["family"], case["size"], seed, fp32)
    host = CSR(m, n, rp.cpu().numpy(), None, None)
    if op == "convert":
        return {"op": op, "host": host, "arrays": (rp, ci, v), "form": case["form"],
                "opts": opts, "x": _vector(n, seed, fp32)}
    mat = SpMatrix(host, case["form"], device_arrays=(rp, ci, v), **opts)
    shape = (case["k"],) if op == "spmm" else ()
    return {"op": op, "mat": mat, "x": _vector((n,) + shape, seed, fp32),
            "y": torch.empty((m,) + shape, dtype=torch.float64, device=DEV)}


def run(s):
    op = s["op"]
    if op == "spmv":
        return s["mat"].spmv(s["x"], s["y"])
    if op == "spmm":
        return s["mat"].spmm(s["x"], s["y"])
    if op == "batch":
        s["batch"].replay()
        return s["y"]
    if op == "convert":
        mat = SpMatrix(s["host"], s["form"], device_arrays=s["arrays"], **s["opts"])
        y = mat.spmv(s["x"])
        mat.close()
        return y
    if op == "coo":
        m, n, rows, cols, vals = s["coo"]
        return coo_to_csr_device(m, n, rows, cols, vals, 1, s["symmetric"])
    net = s["net"]
    net.set_params(s["P"])
    losses = net.train(s["epochs"], LR)
    return {"losses": losses, "params": net.params()[0]}


def _nnz(case):
    """Nonzeros of a case's matrix (expected ones, for the random families)."""
    f, z = case["family"], case["size"]
    if f == "laplace":
        return 5 * z * z - 4 * z
    if f == "stencil27":
        return (3 * z - 2) ** 3
    return z * {"banded": 24, "powerlaw": 15.75, "blocks": 41.0}[f]


def _rows(case):
    return case["size"] ** {"laplace": 2, "stencil27": 3}.get(case["family"], 1)


def work(case):
    op = case["op"]
    if op == "train":
        B, e = case["samples"], case["epochs"]
        # forward, and twice that backward; inputs, targets and mask read once a step
        return {"bytes": e * B * 4.0 * (12 + 2 * 32), "flops": e * 6.0 * B * (64 * 12 + 64 * 64 + 32 * 64)}
    if op == "coo":
        out = _nnz(case)
        nin = (out + _rows(case)) / 2 if case["symmetric"] else out
        return {"bytes": 16.0 * nin + 12.0 * out + 4.0 * _rows(case), "flops": 0.0}
    sv = 4.0 if case["precision"] == "fp32c" else 8.0
    if op == "batch":
        m = float(_batch_sizes(case).sum())
        # columns within one small matrix: 16-bit offsets are enough, but not for plain CSR
        si = 4.0 if case["index"] == "i32" else 2.0
        return {"bytes": 12 * m * (sv + si) + 4 * m + (sv + 8) * m, "flops": 24 * m}
    nnz, m = float(_nnz(case)), float(_rows(case))
    k = case.get("k", 1)
    si = 2.0 if case["index"] == "auto" and case["family"] != "powerlaw" else 4.0
    b = nnz * (sv + si) + 4 * m + (sv + 8) * m * k
    if op == "convert":  # the CSR read, the form written, x read and y written
        b += nnz * 12.0 + 4 * m
    return {"bytes": b, "flops": 2.0 * nnz * k}


# ---- the same in 64 bits, by torch alone ------------------------------------------------------

def _product(m, n, rp, ci, v, x):
    A = torch.sparse_csr_tensor(rp.long(), ci.long(), v, size=(m, n))
    x = x.double()
    return A @ x if x.dim() == 2 else (A @ x.unsqueeze(1)).squeeze(1)


def exact(case, seed):
    op = case["op"]
    if op == "train":
        return _train_exact(case, seed)
    if op == "coo":
        m, n, rows, cols, vals = _coo(case, seed)
        r, c, v = rows.long() - 1, cols.long() - 1, vals
        if case["symmetric"]:
            off = r != c
            r, c, v = torch.cat([r, c[off]]), torch.cat([c, r[off]]), torch.cat([v, v[off]])
        order = torch.argsort(r * n + c, stable=True)
        rp = torch.zeros(m + 1, device=DEV, dtype=torch.int64)
        rp[1:] = torch.cumsum(torch.bincount(r, minlength=m), 0)
        return (rp.int(), c[order].int(), v[order])
    fp32 = case["precision"] == "fp32c"
    if op == "batch":
        sizes, rp, ci, v = _batch_union(case, seed)
        s = torch.from_numpy(sizes).to(DEV)
        start = torch.cumsum(s, 0) - s  # first row (and column) of each matrix in the union
        row_len = (rp[1:] - rp[:-1]).long()
        shift = torch.repeat_interleave(torch.repeat_interleave(start, s), row_len)
        m = int(sizes.sum())
        return _product(m, m, rp, ci.long() + shift, v, _vector(m, seed, fp32))
    m, n, rp, ci, v = _matrix(case["family"], case["size"], seed, fp32)
    shape = (n, case["k"]) if op == "spmm" else (n,)
    return _product(m, n, rp, ci, v, _vector(shape, seed, fp32))


def _train_exact(case, seed):
    X, T, mask, P = (torch.from_numpy(a).double() for a in _train_data(case, seed))
    p = P.clone().requires_grad_(True)
    m1, m2 = torch.zeros_like(P), torch.zeros_like(P)
    lr = float(np.float32(LR))
    b1, b2, eps = (float(np.float32(t)) for t in (0.9, 0.999, 1e-8))
    losses = []
    for step in range(1, case["epochs"] + 1):
        at, h = 0, X
        for o, i in ((64, 12), (64, 64), (32, 64)):
            h = h @ p[at:at + o * i].view(o, i).T + p[at + o * i:at + o * i + o]
            at += o * i + o
            if o == 64:
                h = torch.relu(h)
        loss = (mask * (h - T) ** 2).sum() / mask.sum()
        (g,) = torch.autograd.grad(loss, p)
        losses.append(loss.detach())
        with torch.no_grad():
            m1 = b1 * m1 + (1 - b1) * g
            m2 = b2 * m2 + (1 - b2) * g * g
            p -= lr * (m1 / (1 - b1 ** step)) / (torch.sqrt(m2 / (1 - b2 ** step)) + eps)
    return {"losses": torch.stack(losses), "params": p.detach()}
