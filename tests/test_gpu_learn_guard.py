"""GPU: the learned form runs on what lgpu_learn_init was given.  Its buffers
hold one row per active column for one ensemble size and one group, so another
localizer class, ensemble size or set of active columns has to be refused, and
new radii or coordinates have to be taken."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNSUPPORTED, ORDER = 10, 6


def _loc(radius):
    return {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": radius}]}}


def _refused(s, code):
    from letkf_gb300 import LgpuError
    for call in (s.run, s.learn_collect):
        with pytest.raises(LgpuError) as e:
            call()
        assert e.value.code == code


def test_learned_form_of_another_configuration():
    from letkf_gb300 import Solver, synth
    p = synth.generate("c3", nx=48, ny=24, nz=5, n_obs=1500, k=10)
    with Solver(0) as s:
        s.solver_init({})
        s.loc_init(_loc(1000.0e3), p.vars)
        s.set_problem(p)
        s.learn_init(p.nx, p.ny, stride=2, hidden=32, judge_frac=0.0, gate_frac=0.0, sample_frac=1.0, train_cap=5000,
                     seed=5)
        s.learn_collect()
        s.learn_train(epochs=1, batch=256, lr=1e-3)
        s.set_variant("learned")
        s.run()
        first = s.get_state()

        def again():
            # (either Gram form of the lattice may be measured faster: 1e-5 of the oracle each)
            s.run()
            x = s.get_state()
            for a, b in zip(x, first):
                assert np.linalg.norm(a - b) < 2e-5 * np.linalg.norm(b)

        # another localizer class, with more groups than the lattice's stride leaves rows for
        vtgc = dict(_loc(1000.0e3), vtloc=200.0)
        vtgc["class"] = "loc_vtgc"
        s.loc_init(vtgc, p.vars, np.linspace(5.0, 500.0, 10).astype(np.float32))
        _refused(s, UNSUPPORTED)
        s.loc_init(_loc(1000.0e3), p.vars)
        again()
        # another ensemble size
        for k in (8, 14):
            s.set_problem(synth.generate("c3", nx=48, ny=24, nz=5, n_obs=1500, k=k))
            _refused(s, ORDER)
        s.set_problem(p)
        again()
        # another set of active columns, of another grid and of the same one
        s.set_problem(synth.generate("c3", nx=96, ny=48, nz=5, n_obs=1500, k=10))
        _refused(s, ORDER)
        q = copy.copy(p)
        q.mask = p.mask.copy()
        q.mask[np.nonzero(p.mask == 0)[0][7]] = 1
        s.set_problem(q)
        _refused(s, ORDER)
        s.set_problem(p)
        again()
        # other radii
        s.loc_init(_loc(1400.0e3), p.vars)
        s.run()
        assert not np.array_equal(s.get_state()[0], first[0])
        s.loc_init(_loc(1000.0e3), p.vars)
        again()
        # the sphere turned as a whole: without the network (whose inputs count
        # observations in fixed cells) the same analysis to the rounding of the
        # positions, 3 m of 1,000 km
        s.learn_set_network(False)
        s.run()
        plain = s.get_state()
        q = copy.copy(p)
        q.lon, q.olon = p.lon + np.float32(7.5), p.olon + np.float32(7.5)
        s.set_problem(q)
        s.run()
        for a, b in zip(s.get_state(), plain):
            assert np.linalg.norm(a - b) < 1e-4 * np.linalg.norm(b)
