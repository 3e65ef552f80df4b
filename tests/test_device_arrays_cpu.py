"""Device variables that kernels read as vectors state the alignment those reads need: the linker may
place a double array at any multiple of 8.  Read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pava_b200", "csrc")


def _zero_rows():
    """(file, declaration) of the device arrays that SpMM kernels read in place of a row of X."""
    out = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                t = f.read()
            for var in re.findall(r"reinterpret_cast<const VT \*>\((g_\w+)\)", t):
                out += [(name, d) for d in re.findall(r"^__device__[^;]*\b%s\[[^;]*;" % var, t, re.M)]
    return out


def test_both_kernels_are_found():
    assert {n for n, _ in _zero_rows()} == {"k_csr_spmm.cu", "k_sell_spmm.cu"}


@pytest.mark.parametrize("name,decl", _zero_rows())
def test_rows_read_in_pairs_are_aligned(name, decl):
    m = re.search(r"(?:__align__|alignas)\((\d+)\)", decl)
    assert m and int(m.group(1)) % 16 == 0, f"{name}: {decl}"
