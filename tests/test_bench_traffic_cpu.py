"""bench.py's measured DRAM traffic belongs to the matrix it times: a capture of the same kernel on
another matrix is not reported."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_only_the_timed_matrix(tmp_path):
    f = tmp_path / "traffic.txt"
    f.write_text("# bytes\npowerlaw_100_1600.csr5_sigma32_main = 21000\n")
    assert bench.traffic_from_profiles("powerlaw_100_1600", "csr5_sigma32_main", str(f)) == 21000.0
    assert bench.traffic_from_profiles("powerlaw_101_1600", "csr5_sigma32_main", str(f)) is None
    assert bench.traffic_from_profiles("powerlaw_100_1600", "cvr_steps128_main", str(f)) is None


def test_committed_captures_name_the_matrix_and_exceed_its_streams():
    with open(os.path.join(ROOT, "profiles", "traffic.txt")) as f:
        lines = [s for s in f if s.strip() and not s.startswith("#")]
    assert lines
    for s in lines:
        key, _, value = s.partition("=")
        matrix, kernel = key.strip().split(".")
        family, rows, nnz = matrix.split("_")
        assert family == "powerlaw" and kernel.endswith("_main")
        assert float(value.split()[0]) >= 12 * int(nnz)  # values and columns, each read once
