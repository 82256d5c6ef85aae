"""GPU: which operands the batched Gram takes, and its accuracy on both sides of
the rule.  The grid's active columns are one tile and every observation lies
within its cap, so the rule's two magnitudes can be formed here.  No column sees
the `other` observations: with their features scaled up, the analysis shows what
the tile's common scale leaves of the rest (y^2 / err about 1)."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOC = {"class": "loc_novrt", "hzloc": {"type": "linearinterp_lat", "value": [{"lat": 0.0, "radius": 700.0e3}]}}
RANGE = 17   # powers of two between the tile's largest feature and the smallest of the largest y_i^2 / err


def _unit(lat, lon):
    la, lo = np.deg2rad(np.asarray(lat, np.float64)), np.deg2rad(np.asarray(lon, np.float64))
    return np.stack([np.cos(la) * np.cos(lo), np.cos(la) * np.sin(lo), np.sin(la)], axis=1)


def _problem(k):
    from letkf_gb300 import synth
    p = synth.generate("c3", nx=12, ny=10, nz=2, n_obs=1500, k=k)
    p = synth.observe(p, seed=5, n_obs=1500)
    act = (p.mask == 0) & (p.lon > 60.0) & (p.lon < 120.0) & (np.abs(p.lat) < 70.0)
    p.mask = np.where(act, 0, 1).astype(p.mask.dtype)
    u, o = _unit(p.lat[act], p.lon[act]), _unit(p.olat, p.olon)
    reach = 700.0e3 * np.sqrt(40.0 / 3.0) / 6371.0e3
    centre = u.mean(axis=0) / np.linalg.norm(u.mean(axis=0))
    cap = np.arccos(u @ centre).max() + reach
    seen = np.arccos(np.clip(u @ o.T, -1.0, 1.0)).min(axis=0) < 1.02 * reach
    keep = seen | (np.arccos(np.clip(o @ centre, -1.0, 1.0)) < 0.97 * cap)
    for f in ("olat", "olon", "oz", "otime", "oval", "oerr", "oobsid", "oplatid", "hx", "hx_mean"):
        setattr(p, f, np.ascontiguousarray(getattr(p, f)[keep]))
    return p, ~seen[keep]


def _span(p):
    """exponent of the largest feature less that of the smallest candidate's largest y_i^2 / err"""
    f = np.float32
    y, d = np.abs(p.hx).max(axis=1).astype(f), np.abs((p.oval - p.hx_mean).astype(f))
    s = (y / p.oerr.astype(f)).astype(f)
    top, own = (s * np.maximum(y, d)).astype(f), (s * y).astype(f)
    return int(np.floor(np.log2(top.max()))) - int(np.floor(np.log2(own[own > 0].min())))


def _analyses(p):
    from letkf_gb300 import Solver
    out, bits = [], []
    for variant in ("batched", "plain"):
        with Solver(0) as s:
            s.set_variant(variant)
            s.solver_init({})
            s.loc_init(LOC, p.vars)
            s.set_problem(p)
            s.run()
            out.append(s.get_state())
            bits.append(s.debug_gram_operands())
    assert bits[1] == 0
    return out, bits[0]


def _compare(p, out, tol):
    (xa, ma, _), (xb, mb, _) = out
    cols = p.mask == 0
    pa, pb = [(x - m[:, :, None])[cols] for x, m in ((xa, ma), (xb, mb))]
    assert np.linalg.norm(pa - pb) < tol * np.linalg.norm(pb)
    inc = np.linalg.norm((mb - p.mean)[cols])
    # the means themselves are rounded to 2^-24 of their values
    assert np.linalg.norm((ma - mb)[cols]) < tol * inc + 2.0 ** -23 * np.linalg.norm(p.mean[cols])


def _scaled(p, other, up):
    q = copy.copy(p)
    q.oerr = p.oerr.copy()
    q.oerr[other] *= np.float32(2.0 ** -up)   # y y / err and y dep / err
    return q


@pytest.mark.parametrize("k", [20, 29, 40])
@pytest.mark.parametrize("up", [0, 6, "in", "out", 24, 40])   # powers of two of the other features
def test_common_scale(k, up):
    p, other = _problem(k)
    if up in ("in", "out"):
        # the last span that takes FP16 operands, and the next one
        span = RANGE + (up == "out")
        up = next(u for u in range(1, 40) if _span(_scaled(p, other, u)) == span)
    q = _scaled(p, other, up)
    out, bits = _analyses(q)
    assert bits == (16 if _span(q) <= RANGE else 32)
    # either form is within 1e-5 of the 64-bit oracle (test_gpu_parity)
    _compare(q, out, 2e-5)


@pytest.mark.parametrize("k", [20, 40])
@pytest.mark.parametrize("far", [0, 6, 12, 20])   # powers of two of the departures alone
@pytest.mark.parametrize("whose", ["other", "all"])
def test_departures_beyond_the_perturbations(k, far, whose):
    """y_i dep sets the tile's scale, y_i y_j lie a further |dep| / |y| below."""
    p, other = _problem(k)
    at = other if whose == "other" else np.ones(len(other), bool)
    p.oval = p.oval.copy()
    p.oval[at] = p.hx_mean[at] + np.float32(2.0 ** far) * (p.oval[at] - p.hx_mean[at])
    out, bits = _analyses(p)
    assert bits == (16 if _span(p) <= RANGE else 32)
    if far in (0, 20):
        assert bits == (32 if far else 16)
    if whose == "other":
        _compare(p, out, 2e-5)
    else:
        # the members carry increments far beyond the spread, and its roundings: the means alone
        d = (out[0][1] - out[1][1])[p.mask == 0]
        assert np.linalg.norm(d) < 2e-5 * np.linalg.norm((out[1][1] - p.mean)[p.mask == 0])
