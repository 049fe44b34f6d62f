"""Tile lists that a context keeps from call to call live in its arena: after a
call that moved their buffers a smaller problem gets its list anew.  The middle
call makes the buffers larger without using the tile screen (a large density,
whose threshold lies below what the screen can tell from chance)."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna

pytestmark = pytest.mark.gpu
T = 520


def _clusters(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((T, n)).astype(np.float32)
    f = rng.standard_normal((T, 3)).astype(np.float32)
    for k, a in enumerate(range(0, n - 300, 1500)):
        x[:, a:a + 300] += 1.1 * f[:, [k % 3]]
    return x


@pytest.mark.parametrize("precision", ["bf16x3", "tf32"])
def test_screened_build_after_a_larger_unscreened_one(precision):
    import torch
    n, m = 19800, 21500
    ds, dl = torch.from_numpy(_clusters(n, 5)).cuda(), torch.from_numpy(_clusters(m, 6)).cuda()
    with bna.Builder(0) as b:  # the plain FP32 form, which has no lists
        want = b.corr_csr(ds, mode="r_ge", value=0.45, precision="fp32").numpy()
    with bna.Builder(0) as b:
        first = b.corr_csr(ds, mode="r_ge", value=0.45, precision=precision)
        mid = b.corr_csr(dl, mode="density", value=20.0, precision=precision)
        again = b.corr_csr(ds, mode="r_ge", value=0.45, precision=precision)
    assert first.stats["screen_tiles"] == again.stats["screen_tiles"] > 0
    assert mid.stats["screen_tiles"] == 0
    assert mid.nnz == bna.density_nnz(m, 20.0) and want.nnz > n
    for g in (first.numpy(), again.numpy()):
        assert np.array_equal(g.row_ptr, want.row_ptr) and np.array_equal(g.col_idx, want.col_idx)


def test_batches_of_changing_sizes():
    import torch
    x = [torch.from_numpy(bna.synth_bold(n, 130, 8, n)).cuda() for n in (700, 1500, 400)]
    with bna.Builder(0) as one:
        want = [one.corr_csr(d, mode="r_ge", value=0.35, precision="bf16x3").numpy() for d in x]
    with bna.Builder(0) as b:
        for take in ([0, 2], [0, 1, 2], [0, 2], None, [0, 2], [2]):
            if take is None:  # the arena goes back: the same sizes again on a new one
                b.trim()
                continue
            got = b.corr_csr_batch([x[k] for k in take], mode="r_ge", value=0.35)
            for k, g in zip(take, got):
                g = g.numpy()
                assert np.array_equal(g.row_ptr, want[k].row_ptr)
                assert np.array_equal(g.col_idx, want[k].col_idx)
