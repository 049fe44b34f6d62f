"""Workspaces that only save time (the tile screen's, the streamed centrality's) give
their memory to what a call cannot do without: in the call that took them, and in
later calls of the context.  The device's limit is played by a ceiling on the
context's arena, at which an allocation fails as the driver's would."""
import ctypes as C

import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna

pytestmark = pytest.mark.gpu


def _limit(b, nbytes):
    f = bna.lib().bna_ctx_limit_arena
    f.restype, f.argtypes = None, [C.c_void_p, C.c_int64]
    f(b._h, int(nbytes))


def _lean(b, on):
    f = bna.lib()._ZN3bna12ctx_set_leanEP7bna_ctxb
    f.restype, f.argtypes = None, [C.c_void_p, C.c_bool]
    f(b._h, on)


def _same(a, b):
    a, b = a.numpy(), b.numpy()
    assert a.nnz == b.nnz > 0
    assert np.array_equal(a.row_ptr, b.row_ptr) and np.array_equal(a.col_idx, b.col_idx)
    assert np.array_equal(a.val, b.val)


def _far(n, deg, seed):  # columns ascending, each in a sector of its own
    import torch
    rng = np.random.default_rng(seed)
    c = np.arange(deg)[None, :] * (n // deg) + rng.integers(0, n // deg, (n, deg))
    return bna.CsrResult(n, n * deg, torch.arange(0, n * deg + 1, deg, dtype=torch.int32).cuda(),
                         torch.from_numpy(c.astype(np.int32).ravel()).cuda(),
                         torch.from_numpy(rng.uniform(0.1, 1, n * deg).astype(np.float32)).cuda(),
                         {})


@pytest.mark.parametrize("mode,value", [("r_ge", 0.4), ("density", 0.4)])
def test_build_without_room_for_the_screen(mode, value):
    import torch
    x = torch.from_numpy(bna.synth_bold(19800, 520, 12, 5)).cuda()
    kw = dict(mode=mode, value=value, precision="bf16x3")
    with bna.Builder(0) as b:
        want = b.corr_csr(x, **kw)
        most = b.arena_bytes
    assert want.stats["screen_tiles"] > 0 or mode == "density"
    with bna.Builder(0) as b:
        _lean(b, True)  # without the screen's buffers, and without headroom
        _same(want, b.corr_csr(x, **kw))
        least = b.arena_bytes
    assert least + least // 8 + (12 << 20) < most
    for room in (most - (12 << 20), most - (2 << 20), most):
        with bna.Builder(0) as b:
            _limit(b, room)
            for _ in range(2):
                _same(want, b.corr_csr(x, **kw))
                assert b.arena_bytes <= room
    with bna.Builder(0) as b:  # what never fitted still does not, and the context goes on
        _limit(b, least // 2)
        with pytest.raises(bna.BnaError) as e:
            b.corr_csr(x, **kw)
        assert e.value.status == 2  # BNA_OOM
        _limit(b, 0)
        _same(want, b.corr_csr(x, **kw))


def test_build_after_a_streamed_centrality():
    import torch
    g = _far(26000, 400, 3)
    x = torch.from_numpy(bna.synth_bold(5000, 300, 12, 6)).cuda()
    kw = dict(mode="r_ge", value=0.3, precision="bf16x3")
    with bna.Builder(0) as b:
        _lean(b, True)
        e0 = b.ec(g, max_iter=40)
        want = b.corr_csr(x, **kw)
        least = b.arena_bytes
    with bna.Builder(0) as b:
        e1 = b.ec(g, max_iter=40)
        room = least + least // 8  # the headroom of what the centrality keeps
        assert b.arena_bytes + least > room + (8 << 20)
        _limit(b, room)
        _same(want, b.corr_csr(x, **kw))
        assert b.arena_bytes <= room
        e2 = b.ec(g, max_iter=40)  # without its copy of the graph now, or with it again
        _limit(b, 0)
        e3 = b.ec(g, max_iter=40)
    for e in (e1, e2, e3):
        assert e[2] == e0[2] and abs(e[1] - e0[1]) <= 1e-9 * e0[1]
        assert torch.max(torch.abs(e[0] - e0[0])) <= 1e-9 * torch.max(torch.abs(e0[0]))


def test_lean_request_after_one_that_was_not():
    """One slot: a screened request with a streamed centrality, then one that the
    budget holds only without those workspaces.  The slot gives back what it still
    has of them, so it stays within the budget."""
    a, t = 25600, 520  # (from 25,100 voxels on the edge lists come in long chunks)
    b, need = 31000, {}
    for n in (a, b):
        need[n] = bna.request_bytes(n, t, mode="density", value=0.6, cap=bna.density_nnz(n, 0.6))
    x = {n: bna.synth_bold(n, t, 12, n) for n in (a, b)}
    with bna.Server(0, slots=1, hbm_budget=2 * need[b]) as s:
        want = {n: s.wait(s.submit(x[n], mode="density", value=0.6, precision="bf16x3"))
                for n in (a, b)}
    budget = need[b] - 1
    assert need[a] < budget
    with bna.Server(0, slots=1, hbm_budget=budget) as s:
        for n in (a, b):
            r = s.wait(s.submit(x[n], mode="density", value=0.6, precision="bf16x3"))
            assert r.status == 0 and r.nnz == want[n].nnz
            assert np.array_equal(r.row_ptr, want[n].row_ptr)
            assert np.array_equal(r.col_idx, want[n].col_idx)
        assert s.device_bytes <= budget
