"""Centrality of graphs whose rows differ in length: the persistent kernel's wide
rows (over 1,024 entries and four times the mean) shared out to a block's warps,
more of them in a block than its list holds, groups of rows of unlike lengths; and
dense graphs of 16,385 to 24,576 vertices, which take the forms of larger graphs.
40 iterations against the FP64 oracle; both entry points; two runs bit-equal."""
import ctypes as C

import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle
from cuda_newest20160331_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _graph(lens, n, seed, near=False):
    """Rows of the given lengths, columns ascending at random distances."""
    rng = np.random.default_rng(seed)
    R = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    row = np.repeat(np.arange(n), lens)
    k = np.arange(R[-1]) - R[row]
    step = np.maximum((3 if near else n // np.maximum(lens, 1)), 1)[row] if not near else 1
    c = k * step + rng.integers(0, 1 << 30, len(k)) % step
    if near:
        c = np.minimum(np.maximum(row - lens[row] // 2, 0), n - lens[row]) + k
    return (R.astype(np.int32), c.astype(np.int32),
            rng.uniform(0.05, 1.0, len(c)).astype(np.float32))


def _check(R, Cc, V, iters=40, to_the_end=True):
    import torch
    n = len(R) - 1
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    with bna.Builder(0) as b:
        for vals in (V, None):
            want, lam_o, it_o, _ = oracle.ec(R, Cc, None if vals is None else vals.astype(np.float64),
                                             max_iter=iters)
            csr = bna.CsrResult(n, len(Cc), d(R), d(Cc), None if vals is None else d(vals), {})
            ec, lam, it, _ = b.ec(csr, max_iter=iters)
            again, _, _, _ = b.ec(csr, max_iter=iters)
            c = L.Csr(n=n, nnz=len(Cc), row_ptr=csr.row_ptr.data_ptr(),
                      col_idx=csr.col_idx.data_ptr(),
                      val=csr.val.data_ptr() if csr.val is not None else None)
            na = torch.empty(n, dtype=torch.float64, device="cuda")
            bna.lib().bna_ec_noalloc(C.byref(c), iters, 1e-6, C.c_void_p(na.data_ptr()), None, None,
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert it == it_o and abs(lam - lam_o) <= 1e-9 * abs(lam_o)
            assert torch.equal(ec, again)
            for e in (ec, na):  # row sums of 2^-38, positive entries
                assert np.max(np.abs(e.cpu().numpy() - want)) <= 1e-9 * np.max(np.abs(want))
        if not to_the_end:  # rows near the diagonal: thousands of iterations
            return
        Vd = V.astype(np.float64) * (1.0 + 2.0 ** -30)
        want, lam_o, it_o, conv_o = oracle.ec(R, Cc, Vd)
        ec, lam, it, conv = b.lead_vector(R, Cc, Vd)
        assert it == it_o and conv == conv_o
        assert np.max(np.abs(ec - want)) <= 1e-9 * np.max(np.abs(want))


@pytest.mark.parametrize("n,base,wide", [
    (1500, 5, [1024, 1025, 1500]), (3000, 60, [2999] * 5 + [1026] * 3),
    (9729, 20, [9729, 5000, 1040, 0, 1025]), (20000, 100, [20000] * 3 + [1500] * 40),
    (24576, 3, [24576, 24575, 1031])])
def test_wide_rows(n, base, wide):
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 2 * base + 1, n)
    lens[rng.permutation(n)[:len(wide)]] = wide
    _check(*_graph(lens, n, n))


def test_more_wide_rows_than_a_block_lists():
    """Rows 0 .. 15 of every 152 x 16 belong to one block: all of its 162 wide."""
    n = 24576
    lens = np.full(n, 40)
    lens[np.arange(n) % (152 * 16) < 16] = 1500
    _check(*_graph(lens, n, 3))


def test_groups_of_unlike_rows():
    rng = np.random.default_rng(8)
    n = 5000
    lens = np.minimum((rng.pareto(0.8, n) * 20).astype(np.int64), 1000)
    _check(*_graph(lens, n, 4))


@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("n,deg", [(16385, 701), (16385, 699), (24576, 720)])
def test_dense_graphs_above_16384_vertices(n, deg, near):
    rng = np.random.default_rng(n + deg)
    lens = np.full(n, deg) + rng.integers(-3, 4, n)
    lens[:2] = lens[n // 2] = 0
    _check(*_graph(lens, n, deg, near), iters=16, to_the_end=not near)
    _check(*_graph(lens, n, deg, near), iters=3, to_the_end=False)  # the persistent kernel
