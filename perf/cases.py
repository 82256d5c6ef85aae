"""The measured workloads of the analysis library.

listed() holds the workloads by what they are in use; draw() gives more of the
same ranges.  prepare() builds what a cycling program keeps (the solver handle
with its grid, localizer and inputs set, tuned by one analysis), run() is one
analysis (or one network training epoch) through the public Python interface
with its results read back into the program's own page-locked arrays, and
exact() is the same analysis in 64 bits in plain torch and numpy.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "umd-letkf_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from letkf_gb300 import Solver, synth  # noqa: E402

EARTH_RADIUS_M = 6371000.0
NO_BOUND = 9.99e36


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # a coastal or lake model: a few hundred columns, a small ensemble;
        # launches and host latency are most of it
        _analysis("regional_36x18_k20", "c2", 36, 18, 5, 20, obs=700, r0=800.0, r90=200.0),
        # the reference's own regression test (test/simple3d): two observations,
        # nearly every column keeps its background
        _analysis("simple3d_k50", "simple3d", 180, 90, 5, 50, obs=2, r0=500.0, r90=50.0),
        # point observations with vertical localisation, one transform per
        # column and level, relaxation to the prior spread
        _analysis("vtgc_90x45x10_k20", "c1", 90, 45, 10, 20, obs=5000, r0=500.0, loc="loc_vtgc", vtloc=200.0,
                  rtps=0.6),
        # one whole assimilation cycle of a coarse ocean model: members and raw
        # observations uploaded, statistics and QC on the device, the analysis,
        # and the analysed ensemble read back
        dict(_analysis("cycle_144x72x10_k40", "c2", 144, 72, 10, 40, obs=14000, r0=800.0, r90=200.0), kind="cycle"),
        # a regional model whose sizes fit no tile: odd grid and ensemble,
        # relaxation to the prior perturbations, physical bounds, FP64 re-solve
        # of near-degenerate columns
        _analysis("odd_101x53x7_k37_resolve", "c2", 101, 53, 7, 37, obs=9001, r0=600.0, r90=250.0, rtpp=0.5,
                  precision="fp32_resolve", bounds=True),
        # the ocean localizer: mixed-layer split (two transforms per column),
        # temporal localisation, separate radii for swath and profile data
        _analysis("ocean_144x72x10_k40", "c2", 144, 72, 10, 40, obs=14000, r0=800.0, r90=200.0, loc="loc_ocean",
                  rs0=500.0, rs90=100.0),
        # clustered observations, short localisation, mid resolution: many
        # columns with few observations each
        _analysis("clustered_360x180x10_k32", "c3", 360, 180, 10, 32, obs=125000, r0=100.0),
        # the same network with a 64-member ensemble
        _analysis("clustered_240x120x10_k64", "c3", 240, 120, 10, 64, obs=60000, r0=150.0),
        # a hundred members: the eigensolve dominates
        _analysis("ensemble_240x120x10_k100", "c4", 240, 120, 10, 100, obs=40000, r0=150.0),
        # the headline horizontal grid, ensemble, localisation and network
        _analysis("global_720x360x10_k40", "c2", 720, 360, 10, 40, obs=260000, r0=800.0, r90=200.0),
        # the learned form: exact solves on a lattice and a judged sample, the
        # network on every other column (no column sent back to the exact solve)
        _learned("learned_360x180x5_k32", "learned", 360, 180, 5, 32, obs=40000, r0=400.0),
        # the learned form's training: one epoch over the collected rows
        _learned("train_180x90x5_k32", "train", 180, 90, 5, 32, obs=10000, r0=400.0),
    ]


def _analysis(name, gen, nx, ny, nz, k, obs, r0, r90=0.0, loc="loc_novrt", vtloc=0.0, rs0=0.0, rs90=0.0, rtps=0.0,
              rtpp=0.0, precision="fp32", bounds=False):
    c = dict(kind="analysis", gen=gen, nx=nx, ny=ny, nz=nz, k=k, obs=obs, loc=loc, r0=r0, r90=r90, rs0=rs0, rs90=rs90,
             vtloc=vtloc, rtps=rtps, rtpp=rtpp, precision=precision, bounds=bounds)
    if name:
        c["name"] = name
    return c


def _learned(name, kind, nx, ny, nz, k, obs, r0):
    c = _analysis(name, "c3", nx, ny, nz, k, obs, r0)
    c["kind"] = kind
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        c = _draw_one(rng)
        if _columns_cost(c) <= 206084 * 40.0 ** 2 * 1.5 and c["nx"] * c["ny"] * (2 * c["nz"] + 1) * c["k"] < 2.0e8:
            return c


def _draw_one(rng):
    kind = rng.choice(["novrt", "novrt", "novrt", "clustered", "clustered", "vtgc", "ocean", "cycle"])
    nx = _log_int(rng, 36, 480)
    ny = max(8, int(nx * rng.uniform(0.4, 0.6)))
    nz = rng.randint(1, 20)
    k = _log_int(rng, 10, 100)
    infl = rng.choice([{}, {}, {"rtps": round(rng.uniform(0.2, 0.9), 2)}, {"rtpp": round(rng.uniform(0.2, 0.9), 2)}])
    prec = rng.choice(["fp32", "fp32", "fp32", "fp32_resolve"])
    per_column = rng.uniform(0.3, 1.5)
    obs = max(50, int(nx * ny * per_column))
    r0 = round(rng.uniform(400.0, 900.0), 1)
    if kind == "vtgc":
        nx = min(nx, 180)
        ny = min(ny, 90)
        return _analysis(None, "c1", nx, ny, max(2, nz // 2), min(k, 40), obs=nx * ny, r0=r0, loc="loc_vtgc",
                         vtloc=round(rng.uniform(100.0, 400.0), 1), **infl)
    if kind == "ocean":
        nx = min(nx, 240)
        ny = min(ny, 120)
        return _analysis(None, "c2", nx, ny, max(2, nz), k, obs=nx * ny, r0=r0, r90=200.0, loc="loc_ocean",
                         rs0=round(rng.uniform(300.0, 600.0), 1), rs90=100.0, **infl)
    if kind == "clustered":
        return _analysis(None, rng.choice(["c3", "c4"]), nx, ny, nz, k, obs=min(obs, 200000),
                         r0=round(rng.uniform(80.0, 200.0), 1), precision=prec, **infl)
    c = _analysis(None, "c2", nx, ny, nz, k, obs=min(obs, 260000), r0=r0, r90=200.0, precision=prec,
                  bounds=rng.random() < 0.3, **infl)
    if kind == "cycle":
        c["kind"] = "cycle"
        c["nx"], c["ny"] = min(nx, 240), min(ny, 120)
    return c


def _columns_cost(c):
    """Units (column, group) times k^2, and the observations they read."""
    groups = c["nz"] if c["loc"] == "loc_vtgc" else 2 if c["loc"] == "loc_ocean" else 1
    units = c["nx"] * c["ny"] * 0.8 * groups
    return units * c["k"] ** 2 * max(1.0, c["k"] / 40.0)


# ----------------------------------------------------------------- inputs --
def _problem(case, seed):
    over = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], k=case["k"])
    if case["gen"] == "c2":
        # a third of the observations are swath pairs, the rest profiles of T and S on every level
        swath = max(1, case["obs"] // 60)
        over.update(n_swaths=10, swath_len=swath * 2, n_profiles=max(1, (case["obs"] * 2 // 3) // (2 * case["nz"])))
    elif case["gen"] in ("c1", "c3", "c4"):
        over.update(n_obs=case["obs"])
    return synth.generate(case["gen"], seed=int(seed) % (1 << 60) + 1, **over)


def _table(r0, r90):
    pts = [{"lat": 0.0, "radius": r0 * 1e3}]
    if r90 > 0.0:
        pts.append({"lat": 90.0, "radius": r90 * 1e3})
    return {"type": "linearinterp_lat", "value": pts}


def _localization(case):
    if case["loc"] == "loc_vtgc":
        return {"class": "loc_vtgc", "hzloc": _table(case["r0"], case["r90"]), "vtloc": case["vtloc"]}
    if case["loc"] == "loc_ocean":
        return {"class": "loc_ocean", "hzloc_prof": _table(case["r0"], case["r90"]),
                "hzloc_sat": _table(case["rs0"], case["rs90"]), "tloc_prof": 2.0, "tloc_sat": 1.5,
                "sat_obs": [3], "sat_plats": [2],
                "vtloc_surf": {"type": "bkg_t", "bkg_t_delta": 0.2, "bkg_t_var": 0}}
    return {"class": "loc_novrt", "hzloc": _table(case["r0"], case["r90"])}


def _variables(case, prob):
    out = [dict(v) for v in prob.vars]
    if case["bounds"]:
        out[0].update(ana_inc_max=2.0, ana_bounds=(-2.0, 35.0))
    return out


def _pinned(a, dtype=np.float32):
    """A page-locked copy of an array, as a program keeps what it exchanges with the GPU."""
    p = _pinned_empty(a.shape, torch.int32 if dtype == np.int32 else torch.float32)
    p[...] = a
    return p


def _pinned_empty(shape, dtype=torch.float32):
    return torch.empty(tuple(shape), dtype=dtype, pin_memory=True).numpy()


class _State:
    pass


def prepare(case, seed):
    prob = _problem(case, seed)
    variables = _variables(case, prob)
    s = _State()
    s.kind = case["kind"]
    s.variables = variables
    s.solver = Solver(0)
    s.solver.solver_init({"inflation": {"rtps": case["rtps"], "rtpp": case["rtpp"]}})
    s.solver.loc_init(_localization(case), variables, prob.lev_depth)
    if case["precision"] != "fp32":
        s.solver.set_precision(case["precision"])
    if s.kind == "cycle":
        # full member values, as the forecast model and its observation operators leave them
        s.members = _pinned(prob.state + prob.mean[:, :, None])
        s.hx = _pinned(prob.hx + prob.hx_mean[:, None])
        s.obs = [_pinned(a) for a in (prob.olat, prob.olon, prob.oz, prob.otime, prob.oval, prob.oerr)]
        s.ids = [_pinned(a, np.int32) for a in (prob.oobsid, prob.oplatid)]
        # one observation in sixteen is rejected by quality control
        s.qc = _pinned((np.random.default_rng(seed).integers(0, 16, prob.nobs) == 0).astype(np.int32), np.int32)
        s.solver.set_grid(prob.lat, prob.lon, prob.mask)
        _upload(s)
    else:
        s.solver.set_problem(prob, variables)
    if s.kind in ("learned", "train"):
        s.solver.set_variant("plain")
        s.solver.learn_init(prob.nx, prob.ny, stride=2, hidden=512, judge_frac=0.02, gate_frac=0.0, sample_frac=0.5,
                            train_cap=30000, seed=5)
        s.solver.learn_collect()
        # the first epoch settles the optimizer's moments at a negligible rate
        s.solver.learn_train(epochs=1, batch=512, lr=1e-12 if s.kind == "train" else 1e-3)
        if s.kind == "train":
            return s
        # the analysed cycle has observations the network was not trained on
        cyc = synth.observe(prob, seed=int(seed) % (1 << 60) + 7, n_obs=case["obs"])
        s.solver.set_obs(cyc.olat, cyc.olon, cyc.oz, cyc.otime, cyc.oval, cyc.oerr, cyc.oobsid, cyc.oplatid, cyc.hx,
                         cyc.hx_mean)
        s.solver.set_variant("learned")
    s.out = tuple(_pinned_empty(a.shape) for a in (prob.state, prob.mean, prob.sprd))
    # a cycling program's handle has been tuned by its first analysis
    s.solver.run()
    return s


def _upload(s):
    s.solver.set_state_members(s.members, s.variables)
    s.solver.set_obs_raw(*s.obs, *s.ids, s.hx, s.qc)


def run(state):
    if state.kind == "train":
        loss = state.solver.learn_train(epochs=1, batch=512, lr=1e-3)
        return {"loss": loss, "params": state.solver.learn_params()}
    if state.kind == "cycle":
        _upload(state)
    state.solver.run()
    x, m, sp = state.solver.get_state(state.out)
    return {"state": x, "mean": m, "sprd": sp}


def work(case):
    """What one pass cannot do without: the background read and the analysis
    written once (and carried over the host link in the whole cycle), the
    observations read once, and per (column, group) the k(k+3) operations of
    each kept observation and, where a column keeps any, the 13 k^3 of the
    eigensolve by its usual count and the members' product."""
    k, ncol = case["k"], case["nx"] * case["ny"]
    if case["kind"] == "train":
        din, h, dout = k * k + k + 16, 512, k * k + k
        params = h * din + h * h + dout * h
        rows = 0.5 * 0.75 * ncol * 0.79
        return {"bytes": 4.0 * rows * (din + dout) + 28.0 * params, "flops": 6.0 * rows * params}
    nvar_slabs = {"c1": 1, "simple3d": 3, "c4": 2}.get(case["gen"], 2) * case["nz"]
    ns = nvar_slabs + (0 if case["gen"] in ("c1", "simple3d", "c4") else 1)
    land = 0.0 if case["gen"] in ("c1", "simple3d") else 0.205
    cols = ncol * (1.0 - land)
    groups = case["nz"] if case["loc"] == "loc_vtgc" else 2 if case["loc"] == "loc_ocean" else 1
    r = 1e3 * (case["r0"] + (case["r90"] or case["r0"])) / 2.0
    share = math.sin(min(1.5, 3.65 * r / EARTH_RADIUS_M / 2.0)) ** 2
    kept = case["obs"] * share
    nbytes = ncol * ns * (8.0 * k + 16.0) + case["obs"] * (4.0 * k + 36.0)
    solved = cols * min(1.0, kept)
    return {"bytes": nbytes, "flops": solved * (groups * (kept * k * (k + 3.0) + 13.0 * k ** 3) + 2.0 * ns * k * k)}


# ------------------------------------------------------- 64-bit reference --
def exact(case, seed):
    """The analysis of every column in 64 bits: the search within
    sqrt(40/3) length scales, Gaspari-Cohn weights kept above 1e-4, the
    ensemble transform and the relaxation, clipping and recentring that follow
    it.  The learned form and its training approximate the analysis and have
    no such value."""
    if case["kind"] in ("learned", "train"):
        return None
    prob = _problem(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    f64 = dict(dtype=torch.float64, device=dev)
    mean_b = prob.mean
    pert_b = prob.state
    hx, hxm, keep_obs = prob.hx, prob.hx_mean.astype(np.float64), np.ones(prob.nobs, bool)
    if case["kind"] == "cycle":
        # the float32 values a program hands over, split again in 64 bits
        keep_obs = np.random.default_rng(seed).integers(0, 16, prob.nobs) != 0
        full = (prob.state + prob.mean[:, :, None]).astype(np.float64)
        mean_b = full.mean(axis=2)
        pert_b = full - mean_b[:, :, None]
        h = (prob.hx + prob.hx_mean[:, None]).astype(np.float64)
        hxm = h.mean(axis=1)
        hx = h - hxm[:, None]
    sprd_b = prob.sprd.astype(np.float64)
    if case["kind"] == "cycle":
        sprd_b = np.sqrt((pert_b ** 2).sum(axis=2) / (prob.k - 1))
    o = dict(u=_unit(prob.olat, prob.olon), y=hx, dep=prob.oval.astype(np.float64) - hxm, err=prob.oerr, time=prob.otime,
             z=prob.oz, surf=((prob.oobsid == 3) & (prob.oplatid == 2)).astype(np.float64))
    o = {q: torch.as_tensor(np.asarray(v)[keep_obs], **f64) for q, v in o.items()}
    act = np.nonzero(prob.mask == 0)[0]
    if case["loc"] == "loc_vtgc":
        slab_group = np.concatenate([np.arange(v["levels"]) for v in prob.vars])[None, :].repeat(len(act), 0)
        groups = list(range(prob.nz))
    elif case["loc"] == "loc_ocean":
        t = prob.mean[act][:, :prob.vars[0]["levels"]]
        below = np.abs(t[:, :1] - t) > np.float32(0.2)
        depth = np.where(below.any(axis=1), below.argmax(axis=1), t.shape[1])
        level = np.concatenate([np.arange(v["levels"]) for v in prob.vars])
        slab_group = (level[None, :] >= depth[:, None]).astype(np.int64)
        groups = [0, 1]
    else:
        slab_group = np.zeros((len(act), prob.ns), np.int64)
        groups = [0]
    xa = pert_b.astype(np.float64, copy=True)
    lens = _length_scales(case, prob.lat)
    uc = _unit(prob.lat, prob.lon)
    row_of = np.full(prob.ncol, -1)
    row_of[act] = np.arange(len(act))
    for cols in _tiles(act, uc):
        T, n = _transforms(case, prob, o, cols, uc, lens, groups, dev)
        x = torch.as_tensor(pert_b[cols], **f64)
        sg = torch.as_tensor(slab_group[row_of[cols]], device=dev)
        new = x.clone()
        for g in range(len(groups)):
            sel = (sg == g) & (n[g] > 0)[:, None]
            new = torch.where(sel[:, :, None], x @ T[g], new)
        xa[cols] = new.cpu().numpy()
    ana, mean, sprd = pert_b + np.asarray(mean_b, np.float64)[:, :, None], mean_b, sprd_b
    ana, mean, sprd = ana.astype(np.float64), np.array(mean, np.float64), np.array(sprd, np.float64)
    if case["kind"] != "cycle":
        # masked columns are carried over as they were given
        ana[prob.mask != 0] = prob.state[prob.mask != 0]
    else:
        ana[prob.mask != 0] = pert_b[prob.mask != 0]
    for lo in range(0, len(act), 16384):
        c = act[lo:lo + 16384]
        ana[c], mean[c], sprd[c] = _epilogue(case, _variables(case, prob), xa[c], pert_b[c].astype(np.float64),
                                             np.asarray(mean_b[c], np.float64), sprd_b[c], prob.k)
    return {"state": ana, "mean": mean, "sprd": sprd}


def _unit(lat, lon):
    p, l = np.deg2rad(np.asarray(lat, np.float64)), np.deg2rad(np.asarray(lon, np.float64))
    return np.stack([np.cos(p) * np.cos(l), np.cos(p) * np.sin(l), np.sin(p)], axis=1)


def _length_scales(case, lat):
    """Length scales (m) by latitude: of the localizer and, for loc_ocean, of the swath data."""
    a = np.abs(np.asarray(lat, np.float64)) / 90.0
    first = 1e3 * (case["r0"] + a * ((case["r90"] or case["r0"]) - case["r0"]))
    if case["loc"] != "loc_ocean":
        return first, None
    return first, 1e3 * (case["rs0"] + a * ((case["rs90"] or case["rs0"]) - case["rs0"]))


def _tiles(cols, u):
    """Neighbouring columns in blocks of at most 128."""
    todo, out = [cols], []
    while todo:
        c = todo.pop()
        if len(c) <= 128:
            out.append(c)
            continue
        axis = np.argmax(np.ptp(u[c], axis=0))
        c = c[np.argsort(u[c, axis], kind="stable")]
        todo += [c[:len(c) // 2], c[len(c) // 2:]]
    return out


def _gc(z, scale):
    """Gaspari-Cohn with the reference's truncated coefficients."""
    c = scale / math.sqrt(0.3)
    z = z.abs() / c
    inner = 1.0 + z * z * (-1.66667 + z * (0.625 + z * (0.5 - 0.25 * z)))
    zo = z.clamp(min=1.0)
    outer = 4.0 + zo * (-5.0 + zo * (1.66667 + zo * (0.625 + zo * (-0.5 + 0.08333 * zo)))) - 0.66667 / zo
    return torch.where(z >= 2.0, torch.zeros_like(z), torch.where(z > 1.0, outer, inner))


def _transforms(case, prob, o, cols, uc, lens, groups, dev):
    """The transforms [group][column, k, k] and kept counts [group][column] of a block of columns."""
    f64 = dict(dtype=torch.float64, device=dev)
    k, nc = prob.k, len(cols)
    u = torch.as_tensor(uc[cols], **f64)
    l1 = torch.as_tensor(lens[0][cols], **f64)[:, None]
    l2 = None if lens[1] is None else torch.as_tensor(lens[1][cols], **f64)[:, None]
    rmax = (l1 if l2 is None else torch.maximum(l1, l2)) * math.sqrt(40.0 / 3.0)
    centre = u.mean(dim=0)
    centre = centre / centre.norm()
    ang = 2.0 * torch.asin(((u - centre).norm(dim=1) / 2.0).clamp(max=1.0)).max() + float(rmax.max()) / EARTH_RADIUS_M
    if float(ang) < math.pi:
        near = torch.nonzero((o["u"] @ centre) >= math.cos(float(ang)) - 1e-9).flatten()
    else:
        near = torch.arange(len(o["dep"]), device=dev)
    q = {n: v[near] for n, v in o.items()}
    dx = torch.zeros(nc, len(near), **f64)
    for d in range(3):
        dx += (u[:, d, None] - q["u"][None, :, d]) ** 2
    dist = 2.0 * EARTH_RADIUS_M * torch.asin((dx.sqrt() / 2.0).clamp(max=1.0))
    iu, ju = torch.triu_indices(k, k, device=dev)
    feat = torch.cat([q["y"][:, iu] * q["y"][:, ju], q["y"] * q["dep"][:, None]], dim=1) / q["err"][:, None]
    Ts, ns = [], []
    for g in groups:
        if case["loc"] == "loc_vtgc":
            rho = _gc(dist, l1) * _gc(q["z"] - float(prob.lev_depth[g]), case["vtloc"])[None, :]
        elif case["loc"] == "loc_ocean":
            prof = _gc(dist, l1) * _gc(q["time"], 2.0)[None, :]
            sat = _gc(dist, l2) * _gc(q["time"], 1.5)[None, :] * (1.0 if g == 0 else 0.0)
            rho = torch.where(q["surf"][None, :] > 0, sat, prof)
        else:
            rho = _gc(dist, l1)
        rho = torch.where((dist <= rmax) & (rho > 1e-4), rho, torch.zeros_like(rho))
        G = rho @ feat
        A = torch.zeros(nc, k, k, **f64)
        A[:, iu, ju] = G[:, :len(iu)]
        A[:, ju, iu] = G[:, :len(iu)]
        A[:, range(k), range(k)] += k - 1.0
        n = (rho > 0).sum(dim=1)
        on = torch.nonzero(n).flatten()   # a column without observations has no transform
        T = torch.zeros(nc, k, k, **f64)
        if len(on):
            root = _inverse_root(A[on])
            T[on] = math.sqrt(k - 1.0) * root + root @ (root @ G[on][:, len(iu):, None])
        Ts.append(T)
        ns.append(n)
    return Ts, ns


def _inverse_root(A):
    """A^(-1/2) of symmetric positive definite matrices by the coupled Newton-Schulz iteration."""
    k = A.shape[1]
    eye = torch.eye(k, dtype=A.dtype, device=A.device)
    scale = A.flatten(1).norm(dim=1)[:, None, None]
    Y, Z = A / scale, eye.expand_as(A).clone()
    for _ in range(80):
        R = Z @ Y
        if float((R - eye).abs().max()) < 1e-12:
            break
        M = 1.5 * eye - 0.5 * R
        Y, Z = Y @ M, M @ Z
    return (Z + Z.transpose(1, 2)) / (2.0 * scale.sqrt())


def _epilogue(case, variables, x, xb, mb, sb, k):
    """Recentring, increment and value bounds, relaxation, spread."""
    full = x + mb[:, :, None]
    m = full.mean(axis=2)
    x = full - m[:, :, None]
    lo, hi, inc = (np.empty(x.shape[1]) for _ in range(3))
    for v in variables:
        s = slice(v["grid_s_idx"], v["grid_s_idx"] + v["levels"])
        lo[s], hi[s] = v.get("ana_bounds", (-NO_BOUND, NO_BOUND))
        inc[s] = v.get("ana_inc_max", NO_BOUND)
    m = np.clip(np.clip(m - mb, -inc, inc), lo - mb, hi - mb) + mb
    if case["rtps"] > 0.0:
        sa = np.sqrt((x ** 2).sum(axis=2) / (k - 1))
        f = np.where(sa > 0.0, case["rtps"] * (sb - sa) / np.where(sa > 0.0, sa, 1.0) + 1.0, 1.0)
        x = x * f[:, :, None]
    if case["rtpp"] > 0.0:
        x = case["rtpp"] * xb + (1.0 - case["rtpp"]) * x
    x = np.clip(x, (lo - m)[:, :, None], (hi - m)[:, :, None])
    r = x.mean(axis=2)
    x = x - r[:, :, None]
    m = m + r
    sp = np.sqrt((x ** 2).sum(axis=2) / (k - 1))
    return x + m[:, :, None], m, sp
