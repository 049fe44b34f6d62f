"""The tile screen of the count pass: graphs equal to the oracle's where most tiles are screened
out, where all hold edges, and where edges sit on the edges of the screened 256 x 256 tiles."""
from functools import lru_cache

import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle

pytestmark = pytest.mark.gpu
N, T = 12401, 520  # 97 blocks (an odd count), 2,449 count tiles: just above the screen's rule


def _series(kind):
    rng = np.random.default_rng(5)
    x = rng.standard_normal((T, N)).astype(np.float32)
    if kind == "clusters":  # 300-voxel clusters, three networks
        f = rng.standard_normal((T, 3)).astype(np.float32)
        for k, a in enumerate(range(0, N - 300, 1500)):
            x[:, a:a + 300] += 1.1 * f[:, [k % 3]]
    elif kind == "pairs":  # single pairs at tile corners, the threshold just met or missed
        r = rng.permutation(N // 256)
        for k in range(0, len(r) - 1, 2):
            i, j = r[k] * 256 + (255 if k % 4 else 0), r[k + 1] * 256 + (0 if k % 4 else 255)
            x[:, j] = x[:, i] + np.float32(1.0 + 0.25 * (k % 7)) * x[:, j]
        x[:, N - 1] = -x[:, 3] + 0.9 * x[:, N - 1]
        x[:, 77] = 4.0          # no variance
        x[200, 500] += 900.0    # one spike: a large 8-bit error in its row
    else:
        f = rng.standard_normal((T, 4)).astype(np.float32)
        x += f @ (0.7 * rng.standard_normal((4, N))).astype(np.float32)
    return x


@lru_cache(maxsize=1)
def _case(kind):
    x = _series(kind)
    return x, oracle.cormat_packed(oracle.zscore(x))


@pytest.mark.parametrize("precision,mode,value", [
    ("bf16x3", "r_ge", 0.45), ("tf32", "r_gt", 0.45), ("bf16x3", "abs_ge", 0.5),
    ("bf16x3", "density", 0.3)])
@pytest.mark.parametrize("kind", ["clusters", "pairs", "everywhere"])
def test_screened_graph_matches_oracle(kind, precision, mode, value):
    import torch
    x, A = _case(kind)
    drop, tau = None, value
    if mode == "density":
        tau, _, drop = oracle.density(A, N, value)
    R, C, V = oracle.threshold_csr(A, N, "r_ge" if mode == "density" else mode, tau, drop=drop)
    d = torch.from_numpy(x).cuda()
    with bna.Builder(0) as b:
        res = b.corr_csr(d, mode=mode, value=value, precision=precision)
        b.set_option("tiles_per_launch", 200)
        cut = b.corr_csr(d, mode=mode, value=value, precision=precision)
    delta = res.stats["delta"]
    for g in (res.numpy(), cut.numpy()):
        assert np.array_equal(g.row_ptr, R) and np.array_equal(g.col_idx, C)
        assert len(V) == 0 or np.max(np.abs(g.val - V)) <= delta


def test_budget_without_room_for_optional_workspaces():
    """A server whose budget holds a request only without the tile screen's and
    the streamed centrality's workspaces still takes it: the same graph, the
    same centrality within the two forms' rounding (float-float row sums of
    2^-38)."""
    n, t = 17000, 520
    x = bna.synth_bold(n, t, 12, 5)
    need = bna.request_bytes(n, t, mode="density", value=1.0,
                             cap=bna.density_nnz(n, 1.0))
    got = []
    for budget in (2 * need, need - 1):
        with bna.Server(0, slots=1, hbm_budget=budget) as s:
            got.append(s.wait(s.submit(x, mode="density", value=1.0, precision="bf16x3")))
    a, b = got
    assert a.status == b.status == 0 and a.nnz == b.nnz >= 65 * n
    assert np.array_equal(a.row_ptr, b.row_ptr) and np.array_equal(a.col_idx, b.col_idx)
    assert np.array_equal(a.val, b.val) and a.ec_iters == b.ec_iters
    assert np.max(np.abs(a.ec - b.ec)) <= 1e-9 * np.max(np.abs(a.ec))
