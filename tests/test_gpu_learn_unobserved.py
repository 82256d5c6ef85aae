"""GPU: the learned form where lattice columns keep no observation.  Their
transform is the identity in an analysis (the update keeps their background) and
zero in the training rows, whatever the handle or the memory held before: an
analysis and a training run have to be those of a handle that saw nothing else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOC = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 500.0e3}]}}


def _problem(seed, half, k):
    from letkf_gb300 import synth
    p = synth.generate("c3", nx=48, ny=24, nz=2, n_obs=1200, k=k)
    p = synth.observe(p, seed=seed, n_obs=1200)
    if half:
        keep = p.olon < 180.0
        for f in ("olat", "olon", "oz", "otime", "oval", "oerr", "oobsid", "oplatid", "hx", "hx_mean"):
            setattr(p, f, np.ascontiguousarray(getattr(p, f)[keep]))
    return p


def _handle(p, gate):
    from letkf_gb300 import Solver
    s = Solver(0)
    s.solver_init({})
    s.loc_init(LOC, p.vars)
    s.set_variant("plain")
    s.set_problem(p)
    s.learn_init(p.nx, p.ny, stride=2, hidden=32, judge_frac=0.0, gate_frac=gate, sample_frac=1.0, train_cap=5000,
                 seed=3)
    return s


@pytest.mark.parametrize("precision", ["fp32", "fp32_resolve", "fp64"])
@pytest.mark.parametrize("k", [6, 16])   # lattice Gram: plain, the faster one
def test_analysis_does_not_depend_on_the_one_before(k, precision):
    full, half = _problem(11, False, k), _problem(12, True, k)
    out = []
    for first in (full, half):
        with _handle(first, 0.2) as s:
            s.set_precision(precision)
            s.learn_collect()
            s.learn_train(epochs=1, batch=256, lr=1e-3)
            s.learn_set_network(False)   # the interpolation alone: no parameters of the first analysis
            s.set_variant("learned")
            s.run()
            s.set_problem(half)
            s.run()
            out.append(s.get_state())
            s.set_variant("plain")
            s.run()
            kept = s.get_diag()["lg_obscount"][0]
            exact = s.get_state()
    act = half.mask == 0
    lattice = np.zeros((half.ny, half.nx), bool)
    lattice[::2, ::2] = True
    bare = lattice.ravel() & act & (kept == 0)
    assert bare.sum() > 20 and (lattice.ravel() & act & (kept > 0)).sum() > 20
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) < 2e-5 * np.linalg.norm(b)   # either Gram form: 1e-5 of the oracle each
    # between the identity and an exact transform, nothing leaves the spread's scale
    d = np.abs(out[0][1] - exact[1])[act] / np.maximum(half.sprd[act], 1e-6)
    assert d.max() < 5.0


def test_training_does_not_depend_on_the_analysis_before():
    full, half = _problem(11, False, 16), _problem(12, True, 16)
    params = []
    for first in (full, half):
        with _handle(first, 0.0) as s:
            if first is full:
                s.learn_collect()   # fills the transforms of every column
                s.set_problem(half)
                s.learn_init(half.nx, half.ny, stride=2, hidden=32, judge_frac=0.0, gate_frac=0.0, sample_frac=1.0,
                             train_cap=5000, seed=3)
            s.learn_collect()
            s.learn_train(epochs=2, batch=256, lr=1e-3)
            params.append(s.learn_params())
    assert np.all(np.isfinite(params[0])) and np.array_equal(*params)
