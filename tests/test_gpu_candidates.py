"""Pairs near the threshold (candidates) from flag to CSR, at the sizes where the
kernels change: parts of a sub-tile with more than the 64 entries read ahead and
more than a round of 256, series shorter and longer than a group of lanes takes,
a list that outgrows its first allocation; and re-thresholding and degrees over
rows shorter and longer than a flag word or a turn of 32 values.

With delta = 2 every pair of a signed rule is a candidate, so every stored value
has to be the reference's; the tolerance is one float spacing below 1."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24


@pytest.fixture(scope="module")
def builder():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    b = bna.Builder(0)
    yield b
    b.close()


def _bold(N, T, seed):
    b = np.rint(bna.synth_bold(N, T, 6, seed) * 40 + 500).astype(np.float32)
    b[:, N // 2] = 7.0  # a voxel without variance
    return b


@pytest.mark.parametrize("precision", ["fp32", "bf16x3", "tf32"])
@pytest.mark.parametrize("N,T", [(2, 9), (129, 31), (300, 33), (1500, 47), (200, 1600), (200, 1601)])
def test_every_pair_a_candidate(builder, N, T, precision):
    import torch
    b = _bold(N, T, N + T)
    P = oracle.cormat_packed(oracle.zscore(b))
    R, C, V = oracle.threshold_csr(P, N, "r_ge", 0.1)
    res = builder.corr_csr(torch.from_numpy(b).cuda(), mode="r_ge", value=0.1, precision=precision,
                           delta=2.0)
    g = res.numpy()
    assert res.stats["band_candidates"] == N * (N - 1) // 2
    assert np.array_equal(g.row_ptr, R) and np.array_equal(g.col_idx, C)
    assert len(V) == 0 or np.max(np.abs(g.val - V)) <= ULP


@pytest.mark.parametrize("delta", [1e-5, 0.05, 2.0])
@pytest.mark.parametrize("N,T,K", [(33, 20, 2), (700, 40, 3), (3000, 60, 2)])
def test_rethreshold_and_degree(builder, N, T, K, delta):
    import torch
    b = np.rint(bna.synth_bold(N, T, K, 3) * 40 + 500).astype(np.float32)
    base = builder.corr_csr(torch.from_numpy(b).cuda(), mode="r_ge", value=0.0, precision="bf16x3",
                            delta=max(delta, 2.0 ** -13))
    P = oracle.cormat_packed(oracle.zscore(b))
    tol = ULP if delta == 2.0 else base.stats["delta"]
    for tau in (0.0, 0.25, 0.6, 1.5):
        g = builder.rethreshold(base, "r_gt", tau)
        deg = builder.degree(g).cpu().numpy()
        g = g.numpy()
        R, C, V = oracle.threshold_csr(P, N, "r_gt", tau)
        assert np.array_equal(g.row_ptr, R) and np.array_equal(g.col_idx, C)
        assert len(V) == 0 or np.max(np.abs(g.val - V)) <= tol
        want = [np.add.accumulate(g.val[R[k]:R[k + 1]], dtype=np.float32)[-1] if R[k + 1] > R[k]
                else 0.0 for k in range(N)]
        assert np.array_equal(deg, np.array(want, np.float32))


@pytest.mark.parametrize("N", [4095, 4096, 4097, 8193])
def test_row_offsets_over_blocks_of_rows(builder, N):
    """Row offsets where the rows fill the scan's blocks of 4,096, or spill one
    over; a dense corner gives some sub-tiles the dense fill."""
    import torch
    rng = np.random.default_rng(N)
    b = rng.integers(400, 600, (24, N)).astype(np.float32)
    b[:, -200:] = b[:, -1:] + rng.integers(-9, 10, (24, 200))
    P = oracle.cormat_packed(oracle.zscore(b))
    R, C, V = oracle.threshold_csr(P, N, "r_gt", 0.7)
    res = builder.corr_csr(torch.from_numpy(b).cuda(), mode="r_gt", value=0.7, precision="bf16x3")
    g = res.numpy()
    assert np.array_equal(g.row_ptr, R) and np.array_equal(g.col_idx, C)
    assert np.max(np.abs(g.val - V)) <= res.stats["delta"]
