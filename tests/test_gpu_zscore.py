"""Z-scores whose norm comes from integer sums: bit-identical to the oracle at the edges of the
time slices and of the 32-voxel blocks, and on enough samples that some take the exact path."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle

pytestmark = pytest.mark.gpu


def _series(kind, N, T, seed):
    rng = np.random.default_rng(seed)
    if kind == "model":
        return rng.standard_normal((T, N)).astype(np.float32)
    if kind == "scanner":  # integer samples about a baseline; some equal their mean
        base = rng.integers(500, 12000, N)
        return (base + np.round(rng.standard_normal((T, N)) * 9)).astype(np.float32)
    if kind == "spread":  # sample sizes over many binades: other units per slice
        return (rng.standard_normal((T, N)) * 2.0 ** rng.integers(-30, 30, (T, N))).astype(np.float32)
    # near-constant: neighbouring floats about a large mean
    one = np.nextafter(np.float32(3e6), np.float32(np.inf))
    return np.where(rng.random((T, N)) < 0.5, np.float32(3e6), one).astype(np.float32)


@pytest.mark.parametrize("kind", ["model", "scanner", "spread", "near_constant"])
@pytest.mark.parametrize("N,T", [(1, 1), (31, 2), (33, 7), (127, 8), (129, 9), (100, 63),
                                 (64, 65), (257, 513), (4096, 1200)])
def test_zscore_bit_exact(kind, N, T):
    import torch
    x = _series(kind, N, T, 7 * N + T)
    x[:, N // 2] = x[0, N // 2]  # a constant voxel
    with bna.Builder(0) as b:
        z = b.zscore(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = oracle.zscore(x)
    assert np.array_equal(z[:, :T].view(np.uint32)[~np.isnan(ref)], ref.view(np.uint32)[~np.isnan(ref)])
    assert np.array_equal(np.isnan(z[:, :T]), np.isnan(ref))
    assert not z[:, T:].any()
