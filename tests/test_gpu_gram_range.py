"""GPU: the batched Gram's operand types over the range of observation
magnitudes.  The analysis has to agree with the plain (FP32, per-column) Gram's
whether the magnitudes take FP16 or TF32 operands; each form is within 1e-5 of
the 64-bit oracle (test_gpu_parity), so the two are within 2e-5 of each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _analysis(prob, variant):
    from letkf_gb300 import Solver
    loc = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 700.0e3}]}}
    with Solver(0) as s:
        s.set_variant(variant)
        s.solver_init({})
        s.loc_init(loc, prob.vars, prob.lev_depth)
        s.set_problem(prob)
        s.run()
        return s.get_state()


# half of the globe's observations with their perturbations and departures times
# `scale` and their errors times `err` (largest feature over error: scale^2 / err)
@pytest.mark.parametrize("k", [20, 29, 37, 40, 60])   # one to four feature passes, ragged rows
@pytest.mark.parametrize("scale,err", [
    (1.0, 1.0),
    (2.0 ** -6, 1.0),              # 2^-12: within FP16's range
    (2.0 ** -12, 1.0),             # 2^-24: beyond it
    (2.0 ** 12, 2.0 ** 24),        # large values, the same features
    (2.0 ** -70, 2.0 ** -60),      # 2^-80
    (0.0, 1.0),                    # no perturbations at all: no information
])
def test_operand_range(k, scale, err):
    from letkf_gb300 import synth
    p = synth.generate("c3", nx=72, ny=36, nz=2, n_obs=2500, k=k)
    half = p.olon < 180.0
    p.hx[half] *= np.float32(scale)
    p.oval[half] = p.hx_mean[half] + np.float32(scale) * (p.oval[half] - p.hx_mean[half])
    p.oerr[half] *= np.float32(err)
    a, b = _analysis(p, "batched"), _analysis(p, "plain")
    act = p.mask == 0
    pa, pb = [x[0][act] - x[1][act][:, :, None] for x in (a, b)]
    assert np.linalg.norm(pa - pb) < 2e-5 * np.linalg.norm(pb)
    # (the mean's own scale: its increments)
    assert np.linalg.norm(a[1][act] - b[1][act]) < 2e-5 * np.linalg.norm(b[1][act])
    # columns of each half by themselves: the far interior sees one half's observations only
    lon = p.lon[act]
    for part in ((lon > 60.0) & (lon < 120.0), (lon > 240.0) & (lon < 300.0)):
        assert np.linalg.norm(pa[part] - pb[part]) < 2e-5 * np.linalg.norm(pb[part])
