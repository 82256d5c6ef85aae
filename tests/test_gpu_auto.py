"""GPU: the first analysis of a configuration runs both Gram forms, the batched
one twice where it allocated; what it returns has to be what the following
analyses return, its counters included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,k,radius", [(36, 18, 20, 500.0e3), (96, 48, 12, 900.0e3), (96, 48, 40, 900.0e3)])
def test_first_analysis(nx, ny, k, radius):
    from letkf_gb300 import Solver, synth
    p = synth.generate("c3", nx=nx, ny=ny, nz=2, n_obs=nx * ny, k=k)
    with Solver(0) as s:
        s.solver_init({})
        s.loc_init({"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": radius}]}},
                   p.vars)
        s.set_problem(p)
        out = []
        for _ in range(3):
            s.run()
            t = s.timings()
            out.append((t["variant"], t["mma_chunks"], s.debug_gram_operands(), s.get_state(), s.get_diag()))
    for v, n, bits, x, d in out[1:]:
        assert (v, n, bits) == out[0][:3]
        assert (v == 2) == (n > 0) == (bits > 0)
        for a, b in zip(x, out[0][3]):
            assert np.array_equal(a, b)
        for q in d:
            assert np.array_equal(d[q], out[0][4][q])
