"""A thread whose wait for a slice's elements gave up must not store that slice's rows: the wait is
reported, and y keeps no partial sums.  Read from the source, since no test may make a copy fail."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pava_b200", "csrc")


def test_sell_spmm_stores_sums_only_after_a_wait_that_held():
    with open(os.path.join(CSRC, "k_sell_spmm.cu")) as f:
        t = re.sub(r"//[^\n]*", "", f.read())
    wait = t.index("const bool ok = mbar_wait(")
    loop = t[wait: t.index("__syncthreads_or(!ok)")]
    stores = re.findall(r"[^\n]*store_row\([^\n]*acc\)[^\n]*", loop)
    assert len(stores) == 1 and stores[0].strip().startswith("if (ok) store_row(")
