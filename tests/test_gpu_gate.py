"""The launch gate behind the tile screen and with the centrality of graphs beyond the
persistent kernel: `done` never goes back within a phase, replays hold an even
number of iterations, and nothing of the results changes."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,T,screened", [(25001, 240, False), (19800, 520, True)])
def test_gate_of_screened_passes_and_replays(N, T, screened):
    import torch
    x = torch.from_numpy(bna.synth_bold(N, T, 20, 508)).cuda()
    calls = []
    with bna.Builder(0) as b:
        whole = b.corr_csr(x, mode="r_gt", value=0.45, precision="bf16x3")
        ec0, lam0, it0, _ = b.ec(whole, max_iter=200)
        b.set_option("tiles_per_launch", 500)
        b.set_option("ec_iters_per_launch", 3)
        b.set_gate(lambda stream, phase, done: calls.append((phase, done)))
        gated = b.corr_csr(x, mode="r_gt", value=0.45, precision="bf16x3")
        n_corr = len(calls)
        ec1, lam1, it1, _ = b.ec(gated, max_iter=200)
        b.set_gate(None)
    w, g = whole.numpy(), gated.numpy()
    assert w.nnz > N and np.array_equal(w.row_ptr, g.row_ptr)
    assert np.array_equal(w.col_idx, g.col_idx) and np.array_equal(w.val, g.val)
    assert it1 == it0 and lam1 == lam0 and torch.equal(ec0, ec1)
    for phase in (0, 1):
        done = [d for p, d in calls[:n_corr] if p == phase]
        assert len(done) >= 3 and done == sorted(set(done))
    assert (whole.stats["screen_tiles"] > 0) == screened
    if screened:  # the screen's launches of 750 super-tiles, then the kept tiles'
        nsup = ((N + 127) // 128 + 1) // 2
        assert max(d for p, d in calls[:n_corr] if p == 0) >= nsup * (nsup + 1) // 2
    ec_calls = calls[n_corr:]
    assert all(p == 2 for p, _ in ec_calls)
    done = [d for _, d in ec_calls]
    assert done == sorted(done) and len(done) >= (it0 - 1) // 4
    if N > 24576:
        assert all(d % 4 == 0 for d in done)
