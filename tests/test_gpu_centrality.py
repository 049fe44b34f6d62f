"""Centrality against the FP64 oracle at the sizes where the kernels change: the
persistent kernel takes up to 24,576 vertices; the streamed form
holds the iterate 24,576 columns at a time (up to four times) and gives every
warp a range of rows; the ranged form gives every block one.  Empty rows, rows
joined to everything, an odd number of entries and unsorted columns are in it."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle
from sparse_graphs import random_graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def builder():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    b = bna.Builder(0)
    yield b
    b.close()


def _graph(n, deg, kind, seed):
    """Rows of deg entries at the same random distances from the diagonal
    ("near": within 2 deg of it), a row joined to everything, runs of empty
    rows at both ends and inside, an odd number of entries."""
    rng = np.random.default_rng(seed)
    span = 2 * deg if kind == "near" else n
    offs = rng.choice(span, deg, replace=False)
    cols = np.sort((np.arange(n)[:, None] + offs[None, :]) % n, axis=1).astype(np.int32)
    keep = np.ones(n, bool)
    keep[:3] = keep[n // 2:n // 2 + 400] = keep[n - 2:] = False
    hub = n // 3
    C = np.concatenate([cols[:hub][keep[:hub]].ravel(), np.arange(n, dtype=np.int32),
                        cols[hub + 1:][keep[hub + 1:]].ravel()])
    lens = np.where(keep, deg, 0)
    lens[hub] = n
    lens[n - 3] -= 1 - len(C) % 2  # an odd count, whose last entry is unused
    C = C[:len(C) - 1 + len(C) % 2]
    R = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    assert len(C) == R[-1] and len(C) % 2 == 1
    if kind == "unsorted":
        C[R[9]:R[10]] = C[R[9]:R[10]][::-1].copy()
    return R, C, rng.uniform(0.05, 1.0, len(C)).astype(np.float32)


@pytest.mark.parametrize("n,deg,kind", [(16385, 70, "far"), (24576, 71, "far"),
                                        (24577, 131, "far"), (49153, 200, "far"),
                                        (98304, 261, "far"), (24577, 125, "far"),
                                        (98305, 40, "far"), (24577, 131, "unsorted"),
                                        (16385, 70, "near"), (98305, 40, "near")])
def test_centrality_forms_match_the_oracle(builder, n, deg, kind):
    """40 iterations, double, float and no values.  A row sum carries 2^-38 of
    its magnitude in float-float, and 40 iterations with positive entries do not
    amplify it beyond 1e-9."""
    import torch
    R, C, V = _graph(n, deg, kind, n)
    Vd = V.astype(np.float64) * (1.0 + 2.0 ** -30)  # not a float
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    for vals in (V, None):
        want, lam_o, it_o, conv_o = oracle.ec(R, C, None if vals is None else vals.astype(np.float64),
                                              max_iter=40)
        csr = bna.CsrResult(n, len(C), d(R), d(C), None if vals is None else d(vals), {})
        ec, lam, it, conv = builder.ec(csr, max_iter=40)
        assert it == it_o and conv == conv_o
        assert np.max(np.abs(ec.cpu().numpy() - want)) <= 1e-9 * np.max(np.abs(want))
        assert abs(lam - lam_o) <= 1e-9 * abs(lam_o)
    # to the end, with double values from the host ("near" takes thousands of iterations)
    if kind == "near":
        return
    want, lam_o, it_o, conv_o = oracle.ec(R, C, Vd, max_iter=10000)
    ec, lam, it, conv = builder.lead_vector(R, C, Vd)
    assert it == it_o and conv == conv_o
    assert np.max(np.abs(ec - want)) <= 1e-9 * np.max(np.abs(want))


@pytest.mark.parametrize("n,deg", [(30000, 1), (30000, 3), (30001, 9)])
def test_centrality_of_sparse_rows(builder, n, deg):
    """Either side of the average row lengths at which rows go from a thread
    to a warp each (2 entries)."""
    import torch
    R, C, V = random_graph(n, deg, deg)
    want, lam_o, it_o, conv_o = oracle.ec(R, C, V.astype(np.float64), max_iter=60)
    csr = bna.CsrResult(n, len(C), *(torch.from_numpy(a).cuda() for a in (R, C, V)), {})
    ec, lam, it, conv = builder.ec(csr, max_iter=60)
    assert it == it_o and conv == conv_o
    assert np.max(np.abs(ec.cpu().numpy() - want)) <= 1e-9 * np.max(np.abs(want))


@pytest.mark.parametrize("n,deg", [(2, 1), (65, 20), (65, 60), (2433, 49), (2433, 51), (9729, 70),
                                   (16384, 30), (16384, 60), (24576, 49), (24576, 51)])
def test_persistent_kernel(builder, n, deg):
    """Either side of the row length from which the iterate is staged in shared
    memory, one block and all of them, rows that do not fill a group of four; a
    run cut into segments of 7 iterations gives the same bits."""
    import torch
    rng = np.random.default_rng(n + deg)
    offs = rng.choice(n, deg, replace=False)
    C = np.sort((np.arange(n)[:, None] + offs[None, :]) % n, axis=1).astype(np.int32)
    keep = rng.random(n) > 0.05  # some rows are empty
    keep[0] = True
    lens = np.where(keep, deg, 0)
    R = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    C = np.ascontiguousarray(C[keep].ravel())
    V = rng.uniform(0.05, 1.0, len(C)).astype(np.float32)
    d = lambda a: torch.from_numpy(a).cuda()
    for vals in (V, None):
        want, lam_o, it_o, conv_o = oracle.ec(R, C, None if vals is None else vals.astype(np.float64),
                                              max_iter=40)
        csr = bna.CsrResult(n, len(C), d(R), d(C), None if vals is None else d(vals), {})
        ec, lam, it, conv = builder.ec(csr, max_iter=40)
        ec = ec.cpu().numpy()
        assert it == it_o and conv == conv_o
        assert np.max(np.abs(ec - want)) <= 1e-9 * np.max(np.abs(want))
        assert abs(lam - lam_o) <= 1e-9 * abs(lam_o)
        builder.set_option("ec_iters_per_launch", 7)
        try:
            cut = builder.ec(csr, max_iter=40)
        finally:
            builder.set_option("ec_iters_per_launch", 0)
        assert np.array_equal(cut[0].cpu().numpy(), ec) and cut[1:] == (lam, it, conv)
    Vd = V.astype(np.float64) * (1.0 + 2.0 ** -30)
    want, lam_o, it_o, conv_o = oracle.ec(R, C, Vd)
    ec, lam, it, conv = builder.lead_vector(R, C, Vd)
    assert abs(it - it_o) <= 1 and conv == conv_o
    assert np.max(np.abs(ec - want)) <= 1e-5 * np.max(np.abs(want))
