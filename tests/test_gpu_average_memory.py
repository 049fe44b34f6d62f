"""Multi-subject averages where the subjects' operands do not fit beside their
z-scores: a subject's at a time, the sums kept in memory between them.  Same
graph, values and packed matrix to the last bit as with all operands at once.
The device's limit is played by a ceiling on the context's arena."""
import ctypes as C

import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
from cuda_newest20160331_gb300 import _lib as L

pytestmark = pytest.mark.gpu
N, S = 1501, 24


def _subjects():
    import torch
    out = []
    for k in range(S):
        x = bna.synth_bold(N, 400 + 7 * (k % 5), 6, 3)[:400 + k]
        x = x + np.random.default_rng(k).standard_normal(x.shape).astype(np.float32)
        x[:, 5] = x[:, 4]           # r = 1 in every subject
        if k == 3:
            x[:, 700] = 2.0         # no variance in one of them
        out.append(torch.from_numpy(np.ascontiguousarray(x)).cuda())
    return out


def _limit(b, nbytes):
    f = bna.lib().bna_ctx_limit_arena
    f.restype, f.argtypes = None, [C.c_void_p, C.c_int64]
    f(b._h, int(nbytes))


def _packed(b, xs, fisher, precision):
    import torch
    out = torch.empty(N * (N - 1) // 2, dtype=torch.float32, device="cuda")
    s = bna.lib().bna_corr_packed(
        b._h, len(xs), (C.c_void_p * S)(*[x.data_ptr() for x in xs]), N,
        (C.c_int32 * S)(*[x.shape[0] for x in xs]), 1 if fisher else 0, L.PRECISIONS[precision],
        C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert s == 0, bna.lib().bna_ctx_last_error(b._h)
    return out


@pytest.mark.parametrize("fisher", [False, True])
@pytest.mark.parametrize("mode,value", [("r_ge", 0.25), ("abs_gt", 0.2), ("density", 2.0)])
def test_average_without_room_for_all_operands(mode, value, fisher):
    import torch
    xs = _subjects()
    kw = dict(mode=mode, value=value, fisher=fisher, precision="bf16x3")
    with bna.Builder(0) as b:
        want = b.corr_csr_avg(xs, **kw)
        most = b.arena_bytes
        packed = _packed(b, xs, fisher, "bf16x3")
    operands = sum(1536 * ((x.shape[0] + 63) // 64 * 64) * 4 for x in xs)
    room = most * 8 // 9 - operands // 2  # (an eighth of every buffer is headroom)
    with bna.Builder(0) as b:
        _limit(b, room)
        for per in (0, 20):
            b.set_option("tiles_per_launch", per)
            got = b.corr_csr_avg(xs, **kw)
            assert b.arena_bytes <= room and got.nnz == want.nnz > 0
            assert torch.equal(got.row_ptr, want.row_ptr)
            assert torch.equal(got.col_idx, want.col_idx) and torch.equal(got.val, want.val)
            assert got.stats["band_candidates"] == want.stats["band_candidates"]
            assert torch.equal(_packed(b, xs, fisher, "bf16x3"), packed)
