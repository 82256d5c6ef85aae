"""GPU: the batched Gram's accumulations in tensor memory against 64 bits.  Each
MMA cuts its sum off at the accumulator's last bit, which shows as a bias of the
analysed spread.  In the runs that AUTO would give to the plain FP32 Gram if the
batched one were slower, and on the learned form's lattice (which was plain
before), the batched form may be at most 4/3 as far from 64 bits as the plain
one: 3.2e-7 to 2.4e-7, where the first workload stood with the plain form and
the transform of that time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RATIO = 4.0 / 3.0


def _spread_error(s, ref, cols):
    a = s.get_state()[2][cols].astype(np.float64)
    return np.linalg.norm(a - ref) / np.linalg.norm(ref)


def _oracle(p, loc, cols):
    from helpers import oracle_for
    with_ref = oracle_for(p, loc)
    ref = with_ref.run(precision=64, cols=cols)["sprd"].astype(np.float64)
    with_ref.close()
    return ref


def test_small_run():
    from letkf_gb300 import Solver, synth
    p = synth.generate("c2", nx=144, ny=72, nz=10, k=40, n_swaths=10, swath_len=466, n_profiles=466)
    loc = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 800.0e3},
                                                                                 {"lat": 90.0, "radius": 200.0e3}]}}
    cols = np.nonzero(p.mask == 0)[0][::11].astype(np.int32)
    ref = _oracle(p, loc, cols)
    err = {}
    for v in ("plain", "batched"):
        with Solver(0) as s:
            s.set_variant(v)
            s.solver_init({})
            s.loc_init(loc, p.vars, p.lev_depth)
            s.set_problem(p)
            s.run()
            err[v] = _spread_error(s, ref, cols)
    print(err)
    assert err["batched"] <= RATIO * err["plain"]


def test_lattice():
    from letkf_gb300 import Solver, synth
    p = synth.generate("c3", nx=360, ny=180, nz=5, n_obs=40000, k=32)
    loc = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 400.0e3}]}}
    lattice = np.zeros((p.ny, p.nx), bool)
    lattice[::2, ::2] = True
    cols = np.nonzero(lattice.ravel() & (p.mask == 0))[0][::13].astype(np.int32)
    ref = _oracle(p, loc, cols)
    with Solver(0) as s:
        s.set_variant("plain")
        s.solver_init({})
        s.loc_init(loc, p.vars)
        s.set_problem(p)
        s.learn_init(p.nx, p.ny, stride=2, hidden=32, judge_frac=0.0, gate_frac=0.0, sample_frac=0.01, train_cap=5000,
                     seed=3)
        s.learn_collect()
        s.learn_train(epochs=1, batch=64, lr=1e-3)
        s.learn_set_network(False)
        s.run()
        plain = _spread_error(s, ref, cols)
        s.set_variant("learned")
        s.run()
        lat, bits = _spread_error(s, ref, cols), s.debug_gram_operands()
    print(plain, lat, bits)
    assert lat <= RATIO * plain
