"""GPU: the FP64 re-solve takes exactly the units that the gap test has to flag,
on either side of the list lengths where the grids change (112 units, or a full
wave of 304).  A flagged unit has two relevant eigenvalues 1e-5 apart, the others
five that lie far from each other, the rest on the floor; the threshold between."""
import numpy as np
import pytest

from test_gpu_transform import _unpack, pack, transform64

pytestmark = pytest.mark.gpu


def _unit(k, rng, close):
    lam = k * np.array([1.0, 2.0, 3.0, 4.0, 5.0])[:min(5, k - 1)]
    if close:
        lam[0] = lam[-1] * (1.0 - 1e-5)
    Q = np.linalg.qr(rng.standard_normal((k, k)))[0][:, :len(lam)]
    return (Q * lam) @ Q.T, rng.standard_normal(k)


@pytest.mark.parametrize("flagged", [1, 112, 113, 304, 305])
@pytest.mark.parametrize("k", [6, 16, 20, 24, 32, 37, 48, 64, 90])
def test_flagged_exactly(k, flagged):
    from letkf_gb300 import Solver
    rng = np.random.default_rng(1000 * k + flagged)
    kinds = [[_unit(k, rng, close) for _ in range(4)] for close in (False, True)]
    packed = [[pack(G, b) for G, b in us] for us in kinds]
    ref = [[transform64(*_unpack(p, k)) for p in us] for us in packed]
    close = np.zeros(2 * flagged + 37, bool)
    close[rng.permutation(len(close))[:flagged]] = True
    which = rng.integers(0, 4, len(close))
    batch = np.stack([packed[int(c)][w] for c, w in zip(close, which)])
    with Solver(0) as s:
        s.set_precision("fp32")
        T32 = s.debug_transform(batch)
        s.set_precision("fp32_resolve", 1e-3)
        T = s.debug_transform(batch)
        assert s.timings()["fp64_units"] == flagged
    for t, t32, c, w in zip(T, T32, close, which):
        if c:
            # the FP32 storage of T (condition 6)
            assert np.abs(t - ref[1][w]).max() < 1e-6 * max(1.0, np.abs(ref[1][w]).max())
        else:
            assert np.array_equal(t, t32)
