"""The tile screen from its smallest problems on (40 count tiles per SM: 155 blocks of
128 voxels on 152 SMs), odd and even block counts, whole and in bounded launches,
where most tiles are screened out, where all hold edges, and where edges sit at the
corners of the screened 256 x 256 tiles: the plain FP32 form's graph, which no
screen touches."""
from functools import lru_cache

import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna

pytestmark = pytest.mark.gpu
T = 520


def _series(kind, n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((T, n), dtype=np.float32)
    if kind == "clusters":  # 300-voxel clusters, three networks
        f = rng.standard_normal((T, 3)).astype(np.float32)
        for k, a in enumerate(range(0, n - 300, 1500)):
            x[:, a:a + 300] += 1.1 * f[:, [k % 3]]
    elif kind == "corners":
        r = rng.permutation(n // 256)
        for k in range(0, len(r) - 1, 2):
            i, j = r[k] * 256 + (255 if k % 4 else 0), r[k + 1] * 256 + (0 if k % 4 else 255)
            x[:, j] = x[:, i] + np.float32(1.0 + 0.25 * (k % 7)) * x[:, j]
        x[:, n - 1] = -x[:, 3] + 0.9 * x[:, n - 1]
        x[:, 77] = 4.0          # no variance
        x[200, 500] += 900.0    # one spike: a large 8-bit error in its row
    else:
        f = rng.standard_normal((T, 4)).astype(np.float32)
        x += f @ (0.7 * rng.standard_normal((4, n))).astype(np.float32)
    return x


@lru_cache(maxsize=1)
def _case(kind, n):
    import torch
    return torch.from_numpy(_series(kind, n)).cuda()


@pytest.mark.parametrize("precision,mode,value", [
    ("bf16x3", "r_ge", 0.45), ("tf32", "abs_gt", 0.5), ("bf16x3", "density", 0.3)])
@pytest.mark.parametrize("n", [19713, 19900, 25000])
@pytest.mark.parametrize("kind", ["clusters", "corners", "everywhere"])
def test_screened_graph_is_the_plain_forms(kind, n, precision, mode, value):
    d = _case(kind, n)
    with bna.Builder(0) as b:
        want = b.corr_csr(d, mode=mode, value=value, precision="fp32").numpy()
        one = b.corr_csr(d, mode=mode, value=value, precision=precision)
        got = [one.numpy()]
        b.set_option("tiles_per_launch", 700)
        got.append(b.corr_csr(d, mode=mode, value=value, precision=precision).numpy())
    nb = (n + 127) // 128
    tiles = sum((nb + 1) // 2 - i // 2 for i in range(nb))
    assert one.stats["screen_tiles"] > 0 or mode == "density"  # a density's limit may be too low
    assert 0 < one.stats["count_tiles"] <= tiles
    if kind != "everywhere" and one.stats["screen_tiles"]:
        assert one.stats["count_tiles"] < tiles // 2
    for g in got:
        assert np.array_equal(g.row_ptr, want.row_ptr) and np.array_equal(g.col_idx, want.col_idx)
