"""Degrees of graphs whose rows differ in length within a warp's 32: rows taken
together, rows taken by themselves (256 values or more, far longer than the
others), and their edges.  Bit-identical to the sequential float sum."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [
    [0] * 31 + [1], [255] + [1] * 40, [256] + [0] * 70, [257, 3, 0, 511, 512, 513],
    [2000] * 3 + [3] * 30, [2000] * 7 + [3] * 30, [2000] * 15 + [3] * 30, [5] * 40 + [40000, 1, 0] + [300] * 30,
    [1025, 1024, 1023] + [7] * 61])
def test_degree_rows(lens):
    import torch
    rng = np.random.default_rng(len(lens))
    R = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n, nnz = len(lens), int(R[-1])
    V = rng.uniform(-1, 1, nnz).astype(np.float32)
    V[rng.integers(0, max(nnz, 1), 5) % max(nnz, 1)] = -0.0
    csr = bna.CsrResult(n, nnz, torch.from_numpy(R).cuda(), torch.zeros(nnz, dtype=torch.int32).cuda(),
                        torch.from_numpy(V).cuda(), {})
    with bna.Builder(0) as b:
        got = b.degree(csr).cpu().numpy()
    want = np.array([np.add.accumulate(np.concatenate([[np.float32(0)], V[a:e]]))[-1]
                     for a, e in zip(R[:-1], R[1:])], np.float32)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
