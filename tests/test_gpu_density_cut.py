"""The density histogram leaves out values far below the wanted one (by the spread
of unrelated series): graphs where the wanted value lies above that cut, below it
(orthogonal series: nearly every correlation is 0, so the histogram has to be
taken again), and shares so large that there is no cut, one subject and in a
batch, against the oracle."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle

pytestmark = pytest.mark.gpu
N, T = 1000, 241


def _series(kind):
    rng = np.random.default_rng(4)
    if kind == "normal":
        x = bna.synth_bold(N, T, 8, 3)
    else:  # each of T - 1 orthogonal cosines for about four voxels
        k = np.arange(N) % (T - 1) + 1
        x = np.cos(np.pi * (np.arange(T)[:, None] + 0.5) * k[None, :] / T)
    x = np.rint(x * 1000 + 5000).astype(np.float32)
    x[:, 17] = 3.0  # without variance
    return x


@pytest.mark.parametrize("precision", ["bf16x3", "tf32"])
@pytest.mark.parametrize("kind,percent", [("normal", 0.2), ("normal", 1.0), ("normal", 30.0),
                                          ("orthogonal", 0.2), ("orthogonal", 1.0),
                                          ("orthogonal", 40.0)])
def test_density_above_and_below_the_cut(kind, percent, precision):
    import torch
    x = _series(kind)
    P = oracle.cormat_packed(oracle.zscore(x))
    tau, _, drop = oracle.density(P, N, percent)
    R, C, V = oracle.threshold_csr(P, N, "r_ge", tau, drop=drop)
    d = torch.from_numpy(x).cuda()
    with bna.Builder(0) as b:
        res = [b.corr_csr(d, mode="density", value=percent, precision=precision)]
        res += b.corr_csr_batch([d, d], mode="density", value=percent, precision=precision)
        delta = res[0].stats["delta"]
        for r in res:
            g = r.numpy()
            assert np.array_equal(g.row_ptr, R) and np.array_equal(g.col_idx, C)
            assert np.max(np.abs(g.val - V)) <= delta
