"""Groups whose nodes without edges shrink below 2^-1000 in thousands of power
steps: all threads of a block leave the common factor in the same step, so
repeated runs give the same labels, step counts and eigenvalues to the last
bit, equal to the oracle's rounds."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle
from sparse_graphs import random_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 3000])
def test_factor_of_nodes_without_edges_runs_deep(n):
    import torch
    R, C, _ = random_graph(n, 2, 3 * n + 2)
    log_o = []
    lab_o, q_o, m_o, _ = oracle.modularity(R, C, log=log_o)
    assert (np.diff(R) == 0).sum() > 100 and max(max(r["iters"]) for r in log_o) > 5000
    runs = []
    with bna.Builder(0) as b:
        csr = bna.CsrResult(n, len(C), torch.from_numpy(R).cuda(), torch.from_numpy(C).cuda(),
                            None, {})
        for _ in range(4):
            log = []
            labels, m, q = b.modularity(csr, log=log)
            runs.append((labels.cpu().numpy(), m, q, log))
    for labels, m, q, log in runs:
        assert m == m_o and np.array_equal(labels, lab_o)
        assert log == runs[0][3] and q == runs[0][2]
