"""Z-scores of series whose values repeat exactly: two levels over 4^k samples
(every z is a power of two, where the next float below is half as far as the
one above), steps, and levels that differ in their last bit.  Bit-identical to
the oracle, and in a time near that of ordinary series: no element of them
needs the reference's sums added again."""
import numpy as np
import pytest

import cuda_newest20160331_gb300 as bna
import oracle

pytestmark = pytest.mark.gpu


def _levels(kind, N, T):
    rng = np.random.default_rng(N + T)
    base = rng.integers(-2000, 9000, N).astype(np.float32)
    if kind == "alternating":  # z = +-1 / sqrt(T)
        s = np.where(np.arange(T) % 2, 1.0, -1.0)[:, None]
    elif kind == "block":  # one quarter high: mean and distances in quarters
        s = np.where(np.arange(T) % 4 == 0, 3.0, -1.0)[:, None]
    else:  # powers of two of both signs, symmetric
        k = rng.integers(0, 12, T // 2)
        s = np.concatenate([2.0 ** k, -2.0 ** k])[:, None]
    return (base + s * 2.0 ** rng.integers(-3, 4, N)).astype(np.float32)


@pytest.mark.parametrize("kind", ["alternating", "block", "powers"])
@pytest.mark.parametrize("N,T", [(33, 4), (130, 16), (65, 64), (129, 250), (500, 256), (70, 1024),
                                 (40, 4096)])
def test_levels_bit_exact(kind, N, T):
    import torch
    x = _levels(kind, N, T)
    with bna.Builder(0) as b:
        z = b.zscore(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = oracle.zscore(x)
    assert np.array_equal(z[:, :T].view(np.uint32), ref.view(np.uint32))


def test_levels_take_no_longer_than_other_series():
    """One warp-wide repair per element would take some hundred times longer."""
    import torch
    N, T = 8192, 1024

    def best(x):
        d = torch.from_numpy(x).cuda()
        ms = []
        with bna.Builder(0) as b:
            for _ in range(4):
                a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                b.zscore(d)
                e.record()
                torch.cuda.synchronize()
                ms.append(a.elapsed_time(e))
        return min(ms)
    other = np.random.default_rng(1).standard_normal((T, N)).astype(np.float32)
    assert best(_levels("alternating", N, T)) <= 4 * best(other)
