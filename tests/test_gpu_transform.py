"""GPU: the transform stage (lgpu_debug_transform) at the edges of its lane
grids and outside the spectrum of Gram matrices.

Bars, as in test_gpu_eig and test_gpu_precision: FP32 within the larger of
2e-5, four times float32 LAPACK's error and 2 eps32 kappa of float64 numpy
(max norm over max(1, |T|)); FP64 within 1e-6 (the FP32 storage of T) plus
4 eps64 kappa."""
import numpy as np
import pytest

from test_gpu_eig import cases, pack, transform32, transform64

pytestmark = pytest.mark.gpu


def _unpack(p, k):
    iu = np.triu_indices(k)
    G = np.zeros((k, k))
    G[iu] = p[: len(iu[0])]
    return G + np.triu(G, 1).T, p[len(iu[0]):].astype(np.float64)


def _below_floor(k, rng):
    """A = G + (k-1) I positive definite with eigenvalues far below k - 1: no
    Gram matrix, so the lower bound of the spectrum has to be found."""
    out = []
    for lo in (0.5, 1e-2, 1e-3):
        Q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        lam = (k - 1) * np.geomspace(lo, 30.0, k)
        out.append(((Q * (lam - (k - 1))) @ Q.T, rng.standard_normal(k)))
    return out


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
@pytest.mark.parametrize("k", [2, 3, 8, 9, 16, 17, 24, 25, 32, 41, 48, 49, 57, 65, 72, 73, 80, 81, 96, 97, 104, 112,
                               113, 121, 128])
def test_grid_edges(k, mode):
    from letkf_gb300 import Solver
    rng = np.random.default_rng(300 + k)
    cs = [c for c in cases(k, rng)] + _below_floor(k, rng)
    packed = np.stack([pack(G, b) for G, b in cs])
    with Solver(0) as s:
        s.set_precision(mode)
        T = s.debug_transform(packed)
        again = s.debug_transform(packed[::-1])[::-1]
    assert np.array_equal(T, again)   # no dependence on the unit's place in the grid
    bad = []
    for ci, (p, t) in enumerate(zip(packed, T)):
        G, b = _unpack(p, k)
        ref = transform64(G, b)
        scale = max(1.0, np.abs(ref).max())
        err = np.abs(t - ref).max() / scale
        lam = np.linalg.eigvalsh(G + (k - 1) * np.eye(k))
        kappa = lam[-1] / lam[0]
        if mode == "fp64":
            tol = 1e-6 + 4 * 2.3e-16 * kappa
        else:
            tol = max(2e-5, 4.0 * np.abs(transform32(G, b) - ref).max() / scale, 2.0 * 5.96e-8 * kappa)
        if not err < tol:
            bad.append((ci, err, tol))
    assert not bad, (k, mode, bad)


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
@pytest.mark.parametrize("k", [7, 40, 100])
def test_refusals(k, mode):
    """An indefinite A and a non-finite one are errors, whichever unit of the batch they are."""
    from letkf_gb300 import LgpuError, Solver
    rng = np.random.default_rng(400 + k)
    good = [pack(G, b) for G, b in cases(k, rng)[:4]]
    Q, _ = np.linalg.qr(rng.standard_normal((k, k)))
    lam = np.linspace(1.0, 3.0, k) * k
    lam[k // 2] = -0.25 * k
    for wrong in (pack((Q * (lam - (k - 1))) @ Q.T, rng.standard_normal(k)), np.full_like(good[0], np.nan)):
        for at in (0, 3):
            batch = good[:at] + [wrong] + good[at:]
            with Solver(0) as s:
                s.set_precision(mode)
                with pytest.raises(LgpuError) as e:
                    s.debug_transform(np.stack(batch))
                assert e.value.code == 9


@pytest.mark.parametrize("k,copies", [(k, 7) for k in (2, 8, 16, 17, 32, 33, 37, 48, 49, 64, 65, 100, 128)]
                         + [(k, 120) for k in (16, 37, 64)])   # lists below and above one wave of units
def test_resolve_of_flagged_units(k, copies):
    """FP32_RESOLVE with a gap threshold just below 1 flags every unit that
    has two relevant eigenvalues; these get the FP64 form's accuracy, in any
    batch, and the others keep FP32's."""
    from letkf_gb300 import Solver
    rng = np.random.default_rng(500 + k)
    cs = cases(k, rng)
    packed = np.stack([pack(G, b) for G, b in cs] * copies)   # several blocks of the gap test, the last one part filled
    with Solver(0) as s:
        s.set_precision("fp32")
        T32 = s.debug_transform(packed)
        s.set_precision("fp32_resolve", 0.999)
        T = s.debug_transform(packed)
        again = s.debug_transform(packed[::-1])[::-1]
    assert np.array_equal(T, again)
    flagged = expected = 0
    for p, t, t32 in zip(packed, T, T32):
        G, b = _unpack(p, k)
        lam = np.linalg.eigvalsh(G + (k - 1) * np.eye(k))
        # a relevant eigenvalue (clear of the floor) with a neighbour within the threshold
        expected += bool(np.any((lam[:-1] > k - 1 + 1e-2 * lam[-1]) & (np.diff(lam) < 0.99 * lam[-1])))
        if np.array_equal(t, t32):
            continue
        flagged += 1
        ref = transform64(G, b)
        tol = 1e-6 + 4 * 2.3e-16 * lam[-1] / lam[0]
        assert np.abs(t - ref).max() / max(1.0, np.abs(ref).max()) < tol
    assert flagged > 0 or expected == 0
