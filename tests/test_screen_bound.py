"""What the tile screen leaves for the tensor core's rounding grows with the length
of the series: a step of K = 32 loses less than 33 x 2^-25 + 2^-23 of products and
sums below 2."""
import ctypes as C

import pytest

import cuda_newest20160331_gb300 as bna
from cuda_newest20160331_gb300 import _lib as L


class _Threshold(C.Structure):
    _fields_ = [("mode", C.c_int), ("tau", C.c_float), ("delta", C.c_float)]


@pytest.mark.parametrize("T", [512, 1200, 2656, 10000, 100000, 400000, 2000000])
def test_screen_leaves_room_for_the_accumulator(T):
    f = bna.lib()._ZN3bna12screen_limitERKNS_9ThresholdEdi
    f.restype, f.argtypes = C.c_float, [C.POINTER(_Threshold), C.c_double, C.c_int]
    th = _Threshold(L.THR_MODES["r_ge"], 0.9, 0.001)
    left = 0.9 - 0.001 - 0.0005 - f(C.byref(th), 0.0005, T)
    need = (33 * 2.0 ** -25 + 2.0 ** -23) * ((T + 31) // 32)
    assert left >= max(need, 0.01) - 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["r_ge", "abs_gt"])
def test_long_series_keep_pairs_just_over_the_rule(mode):
    """Pairs at the threshold in tiles that hold nothing else, 2,720 steps: the
    graph of the plain FP32 form, which no screen touches."""
    import numpy as np
    import torch
    N, T, tau = 20225, 2720, 0.45
    rng = np.random.default_rng(9)
    x = torch.from_numpy(rng.standard_normal((T, N), dtype=np.float32)).cuda()
    x -= x.mean(0)
    x /= x.norm(dim=0)
    pick = rng.permutation(N // 128)[:120] * 128 + rng.integers(0, 128, 120)
    for k in range(0, 120, 2):  # r from just below tau to just above
        i, j = int(pick[k]), int(pick[k + 1])
        y = x[:, j] - (x[:, j] @ x[:, i]) * x[:, i]
        y /= y.norm()
        r = tau + (k - 60) * 1e-5
        x[:, j] = (r if mode == "r_ge" or k % 4 else -r) * x[:, i] + (1 - r * r) ** 0.5 * y
    x = (x * 1000).contiguous()
    with bna.Builder(0) as b:
        want = b.corr_csr(x, mode=mode, value=tau, precision="fp32").numpy()
        got = [b.corr_csr(x, mode=mode, value=tau, precision=p) for p in ("bf16x3", "tf32")]
    assert all(g.stats["screen_tiles"] > 0 for g in got)
    got = [g.numpy() for g in got]
    assert want.nnz >= 50
    for g in got:
        assert np.array_equal(g.row_ptr, want.row_ptr) and np.array_equal(g.col_idx, want.col_idx)
