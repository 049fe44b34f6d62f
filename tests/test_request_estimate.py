"""The admission estimate counts what the density rule's selection on the device holds
per candidate beside the list itself: exact value (4 bytes), approximate value (4),
class (1), index (4) and exact value by index (4), of 2^20 candidates."""
import pytest

import cuda_newest20160331_gb300 as bna


@pytest.mark.parametrize("precision,per", [("bf16x3", 17), ("tf32", 17), ("auto", 17), ("fp32", 4)])
def test_density_estimate_counts_the_selection(precision, per):
    n, t, nnz = 20000, 300, bna.density_nnz(20000, 0.5)
    d = bna.request_bytes(n, t, mode="density", value=0.5, precision=precision, cap=nnz)
    r = bna.request_bytes(n, t, mode="r_ge", value=0.5, precision=precision, cap=nnz)
    assert d - r == per << 20
