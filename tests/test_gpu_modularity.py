"""Modularity groups at the edges of the kernel's forms: one block or several, a thread per node
or not (1,024 nodes in one block), each lane count of the row sums, nodes without edges carried as
a factor through thousands of steps.  Labels and rounds against the oracle."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle
from sparse_graphs import random_graph, sym_csr

pytestmark = pytest.mark.gpu


def _planted(n, comm, p_in, p_out, isolated, seed):
    rng = np.random.default_rng(seed)
    c = np.sort(rng.integers(0, comm, n))
    i, j = np.triu_indices(n, 1)
    keep = rng.random(len(i)) < np.where(c[i] == c[j], p_in, p_out)
    keep &= (rng.random(n) >= isolated)[i] & (rng.random(n) >= isolated)[j]
    return sym_csr(n, list(zip(i[keep], j[keep])))


@pytest.mark.parametrize("kind,n,deg", [
    ("random", 40, 3), ("random", 1000, 4), ("random", 1024, 5), ("random", 1030, 5),
    ("random", 1400, 2), ("planted", 300, 0), ("planted", 700, 0), ("hub", 1200, 0),
])
def test_modularity_matches_oracle(kind, n, deg):
    import torch
    if kind == "random":
        R, C, _ = random_graph(n, deg, 3 * n + deg)
    elif kind == "planted":
        R, C = _planted(n, 6, 60.0 / n, 6.0 / n, 0.1, n)
    else:  # rows from 2 to n / 2 entries
        rng = np.random.default_rng(n)
        e = [(0, i) for i in range(1, n // 2)] + [tuple(x) for x in rng.integers(0, n, (4 * n, 2))]
        R, C = sym_csr(n, e)
    with bna.Builder(0) as b:
        csr = bna.CsrResult(n, len(C), torch.from_numpy(R).cuda(), torch.from_numpy(C).cuda(),
                            None, {})
        log, log_o = [], []
        labels, m, q = b.modularity(csr, log=log)
    lab_o, q_o, m_o, _ = oracle.modularity(R, C, log=log_o)
    assert m == m_o and np.array_equal(labels.cpu().numpy(), lab_o)
    assert abs(q - q_o) <= 1e-9 * abs(q_o)
    assert [(r["round"], r["nodes"], r["divided"]) for r in log] == \
        [(r["round"], r["nodes"], r["divided"]) for r in log_o]
    for r, o in zip(log, log_o):
        assert all(abs(x - y) <= 1 for x, y in zip(r["iters"], o["iters"])), (r, o)
        assert abs(r["lambda"] - o["lambda"]) <= 1e-6 * max(1.0, abs(o["lambda"])), (r, o)
