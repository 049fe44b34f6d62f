"""Exact density on networks whose correlated voxels lie together (few tiles hold
the edges), at sizes whose histogram covers every tile: one histogram, one count
pass and the selection, alone and in a batch, and the plain FP32 form's graph."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna

pytestmark = pytest.mark.gpu


def _networks(n, t, seed, block=500, nets=60):
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((t, nets)).astype(np.float32)
    x = rng.standard_normal((t, n), dtype=np.float32)
    return x + f[:, (np.arange(n) // block) % nets]


@pytest.mark.parametrize("n", [11800, 12289, 22000])
def test_one_histogram_finds_the_window(n):
    import torch
    d = torch.from_numpy(_networks(n, 200, n)).cuda()
    with bna.Builder(0) as b:
        for percent in (0.2, 0.6):
            for _ in range(2):  # the first call may repeat its count pass to size the lists
                one = b.corr_csr(d, mode="density", value=percent, precision="bf16x3")
            assert one.stats["passes"] == 3, (percent, one.stats["passes"])
            assert one.nnz == bna.density_nnz(n, percent)
            two = b.corr_csr_batch([d, d], mode="density", value=percent)
            want = b.corr_csr(d, mode="density", value=percent, precision="fp32").numpy()
            for g in [one] + two:
                g = g.numpy()
                assert np.array_equal(g.row_ptr, want.row_ptr)
                assert np.array_equal(g.col_idx, want.col_idx)
