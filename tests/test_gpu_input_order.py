"""GPU: an analysis on a state of another grid's size, or on observations of
another ensemble size, is refused: the device buffers have the sizes their
calls found."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOC = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 900.0e3}]}}
ORDER = 6


def test_inputs_of_another_size():
    from letkf_gb300 import LgpuError, Solver, synth
    p = synth.generate("c3", nx=36, ny=18, nz=2, n_obs=500, k=8)
    big = synth.generate("c3", nx=60, ny=30, nz=2, n_obs=500, k=12)

    def refused(call):
        with pytest.raises(LgpuError) as e:
            call()
        assert e.value.code == ORDER

    with Solver(0) as s:
        s.solver_init({})
        s.loc_init(LOC, p.vars)
        s.set_problem(p)
        s.run()
        want = s.get_state()
        # a larger ensemble, the observations still with 8 members
        s.set_grid(big.lat, big.lon, big.mask)
        s.set_state(big.state, big.mean, big.sprd, big.vars)
        refused(s.run)
        refused(s.get_obs_prepared)
        # a larger grid, the state still of the smaller
        s.set_problem(p)
        s.set_grid(big.lat, big.lon, big.mask)
        refused(s.run)
        refused(s.get_background)
        # a mask of the same grid needs no new state, no observations no ensemble size
        s.set_problem(p)
        s.set_grid(p.lat, p.lon, p.mask)
        s.run()
        for a, b in zip(s.get_state(), want):
            assert np.linalg.norm(a - b) < 2e-5 * np.linalg.norm(b)   # either Gram form: 1e-5 of the oracle each
        none = np.empty(0, np.float32)
        s.set_obs(*[none] * 6, *[np.empty(0, np.int32)] * 2, np.empty((0, 8), np.float32), none)
        s.set_grid(big.lat, big.lon, big.mask)
        s.set_state(big.state, big.mean, big.sprd, big.vars)
        s.run()
        assert not np.any(s.get_diag()["obscount"])
