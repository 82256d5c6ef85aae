"""GPU: runs on a device without room for their work buffers.  The transforms
then take fewer units at a time, with the same bits; the learned form's lattice
takes the plain Gram."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOC = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 900.0e3}]}}
NOMEM = 3
# bytes, between what 32 units and what the grid's take (transforms at k = 16:
# 0.13 and 1 MB, at k = 70 2.0 and 19 MB; training rows at k = 16: 0.2 and 5.5 MB)
LIMIT = {16: 256 << 10, 37: 2 << 20, 70: 2 << 20}


def _solver(p, variant="plain"):
    from letkf_gb300 import Solver
    s = Solver(0)
    s.solver_init({})
    s.loc_init(LOC, p.vars)
    s.set_variant(variant)
    s.set_problem(p)
    return s


def _problem(k):
    from letkf_gb300 import synth
    return synth.generate("c3", nx=48, ny=24, nz=2, n_obs=1200, k=k)


@pytest.mark.parametrize("precision", ["fp32", "fp32_resolve", "fp64"])
@pytest.mark.parametrize("k", [16, 37, 70])
def test_transforms_in_parts(k, precision):
    with _solver(_problem(k)) as s:
        s.set_precision(precision, 0.5)   # many units flagged
        s.run()
        want = s.get_state()
        s.debug_alloc_limit(LIMIT[k])
        s.run()
        for a, b in zip(s.get_state(), want):
            assert np.array_equal(a, b)


def test_no_room_at_all():
    from letkf_gb300 import LgpuError
    with _solver(_problem(16)) as s:
        s.debug_alloc_limit(1)
        with pytest.raises(LgpuError) as e:
            s.run()
        assert e.value.code == NOMEM
        s.debug_alloc_limit(0)
        s.run()


def test_training_rows_in_parts():
    params = []
    for limit in (0, LIMIT[16]):
        with _solver(_problem(16)) as s:
            s.learn_init(48, 24, stride=2, hidden=32, judge_frac=0.0, gate_frac=0.0, sample_frac=1.0, train_cap=5000,
                         seed=3)
            s.debug_alloc_limit(limit)
            s.learn_collect()
            s.learn_train(epochs=1, batch=256, lr=1e-3)
            params.append(s.learn_params())
    assert np.array_equal(*params)


@pytest.mark.parametrize("first", [True, False])   # the analysis that measures the Gram forms, and a later one
def test_lattice_without_room_for_the_streams(first):
    with _solver(_problem(16)) as s:
        s.learn_init(48, 24, stride=2, hidden=32, judge_frac=0.0, gate_frac=0.0, sample_frac=1.0, train_cap=5000,
                     seed=3)
        s.learn_collect()
        s.learn_train(epochs=1, batch=256, lr=1e-3)
        s.learn_set_network(False)
        s.set_variant("learned")
        s.run()
        want = s.get_state()
        if first:
            # other radii and back: the forms are measured again
            s.loc_init(dict(LOC, hzloc={"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 950.0e3}]}),
                       _problem(16).vars)
            s.loc_init(LOC, _problem(16).vars)
        s.debug_alloc_limit(64 << 10)   # the lattice's two tiles take 150 KB each
        s.run()
        for a, b in zip(s.get_state(), want):
            assert np.linalg.norm(a - b) < 2e-5 * np.linalg.norm(b)   # either Gram form: 1e-5 of the oracle each
