"""The multi-subject average, tile by tile in registers: against the oracle's packed average at
the edges of the 128-voxel blocks and of the subject count, with values beyond 1/2 (the Fisher
transform's other branch), duplicated voxels (r = 1) and a voxel without variance in one subject."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle

pytestmark = pytest.mark.gpu


def _subjects(N, S, seed):
    out = []
    for k in range(S):
        T = 40 + 37 * ((3 * k + seed) % 5)
        b = bna.synth_bold(N, T, 6, 100 * seed + k, load_sd=0.6)
        if N > 4:
            b[:, N // 3] = b[:, N // 2]          # r = 1 in every subject
            b[:, N - 2] = 2.0 * b[:, 1] + 0.05 * b[:, N - 2]  # r near 1
        if k == S - 1 and N > 6:
            b[:, 2] = 1.0                        # NaN z-scores in one subject
        out.append(b)
    return out


def _pairs(rp, ci):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    return {(i, j) for i, j in zip(rows.tolist(), ci.tolist()) if i < j}


@pytest.mark.parametrize("precision", ["bf16x3", "tf32"])
@pytest.mark.parametrize("N,S,mode,value", [
    (2, 1, "r_gt", -1.0), (5, 2, "r_ge", 0.2), (127, 3, "r_gt", 0.3), (128, 1, "abs_gt", 0.4),
    (129, 4, "abs_ge", 0.25), (257, 5, "r_gt", 0.0), (385, 2, "r_ge", 0.5), (700, 7, "density", 2.0),
])
@pytest.mark.parametrize("fisher", [False, True])
def test_average_matches_oracle(precision, N, S, mode, value, fisher):
    import torch
    bolds = _subjects(N, S, N + S)
    A = oracle.avg_packed(bolds, fisher=fisher)
    with bna.Builder(0) as b:
        res = b.corr_csr_avg([torch.from_numpy(x).cuda() for x in bolds], mode=mode, value=value,
                             precision=precision, fisher=fisher)
    delta = res.stats["delta"]
    g = res.numpy()
    drop = None
    tau = value
    if mode == "density":
        tau, _, drop = oracle.density(A, N, value)
    R, C, V = oracle.threshold_csr(A, N, "r_ge" if mode == "density" else mode, tau, drop=drop)
    if not fisher:  # float arithmetic on both sides: the same graph
        assert np.array_equal(g.row_ptr, R) and np.array_equal(g.col_idx, C)
        assert len(V) == 0 or np.max(np.abs(g.val - V)) <= delta
        return
    # the transforms come from different math libraries: pairs within 1e-5 may differ
    for i, j in _pairs(g.row_ptr, g.col_idx) ^ _pairs(R, C):
        v = A[i * (2 * N - i - 1) // 2 + j - i - 1]
        assert abs((abs(v) if mode.startswith("abs") else v) - tau) <= 1e-5, (i, j, v)
    rows = np.repeat(np.arange(N), np.diff(g.row_ptr))
    i, j = np.minimum(rows, g.col_idx).astype(np.int64), np.maximum(rows, g.col_idx)
    v = A[i * (2 * N - i - 1) // 2 + j - i - 1]
    assert len(v) == 0 or np.max(np.abs(g.val - v)) <= delta + 1e-5
