"""Kernels that start while the kernel before them runs (griddepcontrol) must not read what that
kernel writes through the read-only path: ld.global.nc, or a const __restrict__ pointer that lets the
compiler choose it, holds for data that nothing writes during the kernel.  Read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pava_b200", "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _dependents():
    """(file, kernel, parameters) of the __global__ functions that wait for the kernel before."""
    out = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        t = _text(name)
        heads = list(re.finditer(r"__global__[^;{]*?(\w+)\(((?:[^(){]|\([^()]*\))*)\)\s*\{", t))
        for h, nxt in zip(heads, heads[1:] + [None]):
            body = t[h.end(): nxt.start() if nxt else len(t)]
            if "pdl_wait()" in body:
                out.append((name, h.group(1), h.group(2)))
    return out


def test_the_products_are_found():
    names = {k for _, k, _ in _dependents()}
    assert {"cvr_spmv_kernel", "csr5_spmv_kernel", "csr5_spmv_f32_kernel", "sell_spmv_kernel",
            "sell_spmm_kernel", "csr_spmm_kernel", "csr_spmv_kernel", "csr_group_kernel",
            "csr_window_kernel", "carry_fixup_kernel"} <= names


@pytest.mark.parametrize("name,kernel,params", _dependents(), ids=lambda v: v if len(v) < 40 else "")
def test_no_read_only_promise_on_what_the_kernel_before_writes(name, kernel, params):
    written = {"x", "X", "carry_head", "carry_tail"}  # x may be the y of the product before
    if kernel == "carry_fixup_kernel":
        written |= {"meta", "arp"}  # the allocation-free product writes the headers too
    for p in params.split(","):
        if "const " in p and p.split()[-1].lstrip("*") in written:
            assert "__restrict__" not in p, f"{name}: {kernel}: {p.strip()}"


@pytest.mark.parametrize("name,load", [("pava_common.cuh", "ld_x"), ("k_stream.cuh", "ld_x2")])
def test_x_is_read_by_ordinary_loads(name, load):
    t = _text(name)
    found = re.findall(r"\b%s\(const \w+ \*p, uint64_t pol\) \{(.*?)\n\}" % load, t, re.S)
    assert len(found) == 2  # FP64 and FP32
    for body in found:
        assert "ld.global" in body and ".nc" not in body
