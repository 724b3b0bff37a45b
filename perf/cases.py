"""Timed cases of the forward model, over the range its users run it on.

A case is a dict of plain values.  Kinds:

  pencil     formod_pencil(): one ray through caller structs
  formod     formod(): the drop-in call on one observation struct
  kernel     kernel(): the retrieval's finite-difference Jacobian
  graph      GraphBatch: a fixed-size request replayed from a CUDA graph
  batch      Batch upload + run + download: clear air ("none"), aerosol
             extinction ("ext"), single scattering ("sca1"), depth-2
             scattering ("sca2"), or single scattering with a trained
             surrogate ("sur")
  train      Surrogate: create, train, read the weights back
  mie        read_aero + get_opt_prop: Mie optical properties

Profiles, geometry and emissivity tables follow jscat.synth (the workloads
of the benchmark and the tests).  Tables belong to the instrument, not to a
request: they have one fixed seed and are written once per process tree into
the temporary folder; a Model of them is kept between preparations, as a
program that serves requests keeps it.
"""
import os
import re
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "jurassic-scatter_b200"))

from jscat import api, synth  # noqa: E402
from jscat import structs as S  # noqa: E402

TABLE_SEED = 20261203
EMITTERS = synth.CFG1_EMITTERS + ["F11", "F12", "SF6", "OCS"]
NUS = synth.CFG1_NU                      # 64 channels, 700-1400 cm-1
RET = dict(rett_zmin=5.0, rett_zmax=60.0, retq_zmin=[10.0, 5.0], retq_zmax=[50.0, 40.0],
           retk_zmin=[5.0], retk_zmax=[30.0])


def listed():
    return [
        # one pencil beam, as the reference's other modules call it
        dict(name="pencil", kind="pencil", rays=1, nd=4, ng=2),
        # limb scan of a retrieval's forward model through the drop-in call
        dict(name="limb_scan", kind="formod", rays=61, nd=4, ng=2),
        # the Jacobian of that scan: 160 forward models in one call
        dict(name="jacobian", kind="kernel", rays=61, nd=4, ng=2),
        # a serving request of ordinary size, replayed from a CUDA graph
        dict(name="graph_request", kind="graph", rays=777, per_atm=37, nd=16, ng=2, aero="none"),
        # a request with odd sizes everywhere and profiles of uneven length
        dict(name="clear_odd", kind="batch", rays=2003, per_atm=19, nd=37, ng=5, aero="none",
             ragged=True),
        # the headline workload's shape (8 emitters, 64 channels), 20k rays
        dict(name="clear_large", kind="batch", rays=20000, per_atm=50, nd=64, ng=8, aero="none",
             ragged=False),
        # cloud extinction without scattering
        dict(name="extinction", kind="batch", rays=3000, per_atm=100, nd=16, ng=2, aero="ext",
             ragged=False),
        # plain single scattering through a sulfate layer, 20 pencils a point
        dict(name="single_scattering", kind="batch", rays=400, per_atm=400, nd=16, ng=2,
             aero="sca1", nalpha=20, ragged=False),
        # depth-2 scattering through an ice cloud, 20 and 10 pencils a point
        dict(name="double_scattering", kind="batch", rays=12, per_atm=12, nd=8, ng=2,
             aero="sca2", nalpha=20, ragged=False),
        # single scattering with the learned source, 1 point in 256 checked
        dict(name="surrogate_step", kind="batch", rays=4000, per_atm=4000, nd=16, ng=2,
             aero="sur", nalpha=20, ragged=False),
        # training of the learned source on plain-path samples
        dict(name="surrogate_train", kind="train", samples=65536, batch=4096, epochs=8, nd=16),
        # optical properties of an ice cloud (size parameters to about 800)
        dict(name="optical_properties", kind="mie", nd=8, layer="ice"),
    ]


def _log(rng, lo, hi):
    """A whole number, spread over the logarithm of lo..hi."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["pencil", "formod", "kernel", "graph", "batch", "batch", "batch", "ext",
                       "sca1", "sca1", "sca2", "sur", "train", "mie"])
    if kind in ("pencil", "formod", "kernel"):
        top = {"pencil": 1, "formod": 1000, "kernel": 61}[kind]
        return dict(kind=kind, rays=1 if top == 1 else _log(rng, 5, top), nd=_log(rng, 1, 4 if kind == "kernel" else 16),
                    ng=2 if kind == "kernel" else rng.randint(2, 8))
    if kind == "train":
        return dict(kind=kind, samples=_log(rng, 8192, 65536), batch=rng.choice([512, 1000, 2048, 4096]),
                    epochs=rng.randint(1, 6), nd=_log(rng, 1, 20))
    if kind == "mie":
        return dict(kind=kind, nd=_log(rng, 1, 8), layer=rng.choice(["ice", "sulfate", "layers"]))
    if kind == "graph":
        return dict(kind=kind, rays=_log(rng, 50, 5000), per_atm=_log(rng, 10, 100), nd=_log(rng, 4, 32), ng=2,
                    aero=rng.choice(["none", "ext"]))
    c = dict(kind="batch", aero="none" if kind == "batch" else kind, ragged=rng.random() < 0.5)
    if kind == "batch":
        return dict(c, rays=_log(rng, 50, 10000), per_atm=_log(rng, 1, 200), nd=_log(rng, 1, 64),
                    ng=rng.choice([1, 2, 3, 4, 5, 7, 8, 12]))
    if kind == "sca2":
        return dict(c, rays=rng.randint(1, 8), per_atm=8, nd=_log(rng, 2, 8), ng=2,
                    nalpha=rng.choice([10, 20]))
    rays = {"ext": _log(rng, 50, 3000), "sca1": _log(rng, 5, 300), "sur": _log(rng, 200, 4000)}[kind]
    nd = 16 if kind == "sur" else _log(rng, 1, 20)
    if kind == "sur":
        return dict(c, rays=rays, per_atm=rays, nd=nd, ng=2, nalpha=20)
    c = dict(c, rays=rays, per_atm=_log(rng, 20, 400), nd=nd, ng=rng.choice([2, 2, 4]))
    return dict(c, nalpha=rng.choice([10, 20, 28])) if kind == "sca1" else c


# ------------------------------------------------------------------ inputs --

def _folder():
    d = os.path.join(tempfile.gettempdir(), "jsc_cases_%d" % os.getuid())
    os.makedirs(d, exist_ok=True)
    return d


def _channels(nd):
    return [NUS[i] for i in np.linspace(0, len(NUS) - 1, nd + 2).round().astype(int)[1:-1]] if nd < 63 else NUS[:nd]


def _tables(emitters, nus):
    """Table and filter files of these emitters and channels (those that are
    missing are written); returns their common path prefix."""
    base = os.path.join(_folder(), "synth")

    def put(path, write):
        if not os.path.exists(path):
            write("%s.%d" % (path, os.getpid()))
            os.replace("%s.%d" % (path, os.getpid()), path)

    for nu in nus:
        put("%s_%.4f.filt" % (base, nu), lambda f, nu=nu: synth.write_filter(f, nu))
        for g in emitters:
            put("%s_%.4f_%s.bin" % (base, nu, g), lambda f, nu=nu, g=g: synth.write_table_bin(
                f, *synth.emissivity_table(g, nu, TABLE_SEED)))
    return base


def _control(case):
    aero = case.get("aero", "none")
    emitters, nus = EMITTERS[:case["ng"]], _channels(case["nd"])
    kw = dict(emitters=emitters, nus=nus, tblbase=_tables(emitters, nus), hydz=0.0)
    if aero != "none":
        kw.update(sca_n=1, sca_mult={"ext": 0, "sca1": 1, "sca2": 2, "sur": 1}[aero])
    if aero == "sca2":   # finite depth-2 sources need these continua off
        kw.update(ctm_co2=0, ctm_h2o=0)
    if case["kind"] == "kernel":
        kw.update(RET)
    return S.make_ctl(**kw)


def _profiles_and_rays(case, seed):
    rng = np.random.default_rng([int(seed), 7])
    n, per = case["rays"], case.get("per_atm", case["rays"])
    aero = case.get("aero", "none")
    atms = []
    for _ in range((n + per - 1) // per):
        z = np.linspace(0.0, 120.0, int(rng.integers(61, 122))) if case.get("ragged") else synth.Z_GRID
        many = n > per
        atms.append(synth.atmosphere(EMITTERS[:case["ng"]], rng, t_sigma=5.0 if many else 1.0,
                                     vmr_sigma=0.2 if many else 0.05, z=z))
    if case["kind"] in ("pencil", "formod", "kernel"):
        geom = synth.limb_geometry(np.sort(rng.uniform(5.0, 35.0, n)))
    elif aero == "sca2":
        geom = synth.limb_geometry(rng.uniform(6.0, 14.0, n))
    elif aero in ("sca1", "sur"):
        geom = synth.limb_geometry(rng.uniform(8.0, 30.0, n))
    else:                # limb and nadir rays in turn
        a = synth.limb_geometry(rng.uniform(5.0, 60.0, n))
        b = synth.nadir_geometry(rng.uniform(0.0, 60.0, n))
        odd = np.arange(n) % 2 == 1
        geom = {k: np.where(odd, b[k], a[k]) for k in a}
    if aero in ("sca1", "sca2", "sur"):
        geom["time"] = rng.uniform(0.0, 86400.0, n)
    return atms, np.arange(n) // per, geom


def _aero_file(layer):
    make = {"ice": synth.ice_layer_files, "sulfate": synth.sulfate_layer_files,
            "layers": synth.layered_aero_files}[layer]
    d = os.path.join(_folder(), "aero_%d" % os.getpid())
    return os.path.join(d, make(d))


def _aero(ctl, layer):
    return api.get_opt_prop(ctl, api.read_aero(ctl, _aero_file(layer)))


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


_kept = {}   # the last Model, and the trained surrogate


def _model(ctl, case):
    key = (case["nd"], case["ng"])
    if _kept.get("key") != key:
        _kept.pop("model", None)
        _kept.update(key=key, model=api.Model(ctl))
    return _kept["model"]


def _surrogate(case, ctl, model):
    """Surrogate trained on the plain sources of two batches of other rays."""
    if "sur" not in _kept:
        feats, srcs = [], []
        for seed in (901, 902):
            atms, ray_atm, geom = _profiles_and_rays(dict(case, rays=400, per_atm=400, ragged=False), seed)
            inp = synth.batch_from(atms, ray_atm, geom)
            b = api.Batch(model, ctl, 1, len(inp["z"]), 400)
            b.set_aero(_aero(ctl, "sulfate"))
            b.set_nalpha(20)
            b.upload(inp)
            b.run()
            b.download()
            f, s = b.scatter_samples()
            feats.append(f)
            srcs.append(s)
            b.close()
        sur = api.Surrogate(ctl.nd, seed=5)
        sur.train(np.concatenate(feats), np.concatenate(srcs), epochs=60, batch=512, lr=3e-3)
        _kept["sur"] = sur
    return _kept["sur"]


def _training_set(case, seed):
    """Features with the ranges of the scattering points of limb rays
    through a layer at 15-20 km, and smooth positive sources of them."""
    rng = np.random.default_rng([int(seed), 11])
    n, nd = case["samples"], case["nd"]
    z = rng.uniform(14.9, 20.1, n)
    sza = rng.uniform(0.0, np.pi, n)
    x = np.stack([z, rng.uniform(-0.07, 0.07, n), 216.5 + 0.3 * (z - 15.0) + rng.normal(0, 1, n),
                  np.log(1013.25) - z / 7.0, np.cos(sza), rng.uniform(-1, 1, n), np.zeros(n),
                  90.0 - np.degrees(sza) + 4.0], axis=1)
    u = (x - x.mean(0)) / np.maximum(x.std(0), 1e-6)
    w = rng.normal(0, 0.4, (8, nd))
    y = np.tanh(u @ w) + 0.3 * np.sin(u[:, :1] + np.linspace(0, 2, nd)) - 8.0
    return x.astype(np.float32), np.exp(y)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, src = _training_set(case, seed)
        return dict(case=case, x=x, src=src)
    if kind == "mie":
        nus = [float(v) for v in np.linspace(780.0, 1220.0, case["nd"]) + (seed % 97) * 0.25]
        ctl = S.make_ctl(["CO2"], nus, "-", sca_n=1)
        return dict(case=case, ctl=ctl, file=_aero_file(case["layer"]))
    ctl = _control(case)
    atms, ray_atm, geom = _profiles_and_rays(case, seed)
    if kind in ("pencil", "formod", "kernel"):
        a = atms[0]
        return dict(case=case, ctl=ctl, atm=S.make_atm(a["z"], a["p"], a["t"], a["q"], a["k"]),
                    obs=S.make_obs(geom["obsz"], geom["obslat"], geom["vpz"], geom["vplat"]))
    model = _model(ctl, case)
    inp = {k: _pinned(v) for k, v in synth.batch_from(atms, ray_atm, geom).items()}
    aero = case["aero"]
    layers = None if aero == "none" else _aero(ctl, "ice" if aero == "sca2" else "sulfate")
    n, nd = case["rays"], case["nd"]
    if kind == "graph":
        stream = torch.cuda.Stream()
        g = api.GraphBatch(model, ctl, inp, stream.cuda_stream, _pinned, aero=layers)
        return dict(case=case, graph=g, stream=stream, inp=inp)
    b = api.Batch(model, ctl, len(atms), len(inp["z"]), n)
    if layers is not None:
        b.set_aero(layers)
    if "nalpha" in case:
        b.set_nalpha(case["nalpha"])
    if aero == "sca2":
        b.set_nalpha_depth(1, 10)
    if aero == "sur":
        b.set_surrogate(_surrogate(case, ctl, model), tol_rel=0.2,
                        check_stride=api.SURROGATE_CHECK_STRIDE)
    out = {k: _pinned(np.empty((n, nd) if k in ("rad", "tau") else n, np.int32 if k == "nlos" else float))
           for k in ("rad", "tau", "tpz", "tplon", "tplat", "nlos")}
    return dict(case=case, batch=b, inp=inp, out=out)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        sur = api.Surrogate(case["nd"], seed=5)
        losses = sur.train(state["x"], state["src"], epochs=case["epochs"], batch=case["batch"], lr=3e-3)
        weights = sur.get_params()
        sur.close()
        return dict(losses=losses, weights=weights)
    if kind == "mie":
        ctl = state["ctl"]
        aero = api.get_opt_prop(ctl, api.read_aero(ctl, state["file"]))
        return {k: S.arr(getattr(aero, k))[:aero.nl, :ctl.nd].copy() for k in ("beta_e", "beta_s", "beta_a", "p")}
    if kind == "batch":
        b = state["batch"]
        b.upload(state["inp"])
        b.run()
        return b.download(out=state["out"])
    if kind == "graph":
        state["graph"].launch(state["inp"])
        state["stream"].synchronize()
        state["graph"].status()
        return state["graph"].out
    ctl, atm, obs = state["ctl"], state["atm"], state["obs"]
    if kind == "kernel":
        return dict(jacobian=api.kernel(ctl, atm, obs))
    if kind == "pencil":
        api.formod_pencil(ctl, atm, obs)
    else:
        api.formod(ctl, atm, obs)
    n, nd = obs.nr, ctl.nd
    return dict(rad=S.arr(obs.rad)[:nd, :n], tau=S.arr(obs.tau)[:nd, :n], tpz=S.arr(obs.tpz)[:n],
                tplon=S.arr(obs.tplon)[:n], tplat=S.arr(obs.tplat)[:n])


# -------------------------------------------------------------------- work --

def work(case):
    """Inputs and outputs once, the table intervals that the evaluations
    touch (at most the whole tables) and the floating-point operations:
    about 60 for an emissivity evaluation (four corners, each an inverse and
    a forward interpolation, then three more), 30 for a channel's continuum,
    Planck and transfer step and 400 for tracing a line-of-sight point."""
    kind, nd = case["kind"], case["nd"]
    if kind == "train":
        n, steps = case["samples"], case["epochs"] * (case["samples"] // case["batch"])
        w = 8 * 128 + 2 * 128 * 128 + 128 * nd
        return dict(bytes=n * (8 * 4 + nd * 8) + 4 * w, flops=6.0 * steps * case["batch"] * w)
    if kind == "mie":
        modes, terms = {"ice": (1, 200), "sulfate": (1, 20), "layers": (2, 20)}[case["layer"]]
        return dict(bytes=modes * nd * (181 + 3) * 8, flops=170.0 * nd * modes * terms * 181 * 40)
    n, ng, aero = case["rays"], case["ng"], case.get("aero", "none")
    models = 160 if kind == "kernel" else 1
    limb = kind in ("pencil", "formod", "kernel") or aero in ("sca1", "sca2", "sur")
    points = n * models * (240 if limb else 180)
    pencils = 0
    if aero == "sca1":
        pencils = n * 29 * case["nalpha"]
    elif aero == "sca2":
        pencils = n * 29 * case["nalpha"] * (1 + 12 * 10)
    elif aero == "sur":
        pencils = n * 29 / 256 * case["nalpha"]
    points += pencils * 60
    evals = points * nd * ng
    levels = 121 * ((n + case.get("per_atm", n) - 1) // case.get("per_atm", n)) * models
    tables = min(nd * ng * 40 * 30 * 300 * 8, evals * 64)
    return dict(bytes=levels * (6 + ng) * 8 + n * models * (7 * 8 + 3 * 8 + 16 * nd) + tables,
                flops=60.0 * evals + 30.0 * points * nd + 400.0 * points)


# ------------------------------------------------------------- 64-bit values --

def exact(case, seed):
    """What run() returns, in plain numpy: the clear-air forward model, the
    surrogate's training and the Mie series.  None where it takes too long
    (large batches, Jacobians, scattering)."""
    kind = case["kind"]
    if kind == "train":
        w = 8 * 128 + 2 * 128 * 128 + 128 * case["nd"]
        steps = case["epochs"] * (case["samples"] // case["batch"])
        return _exact_train(case, seed) if 6.0 * steps * case["batch"] * w < 3e11 else None
    if kind == "mie":
        return _exact_mie(case, seed)
    if kind == "kernel" or case.get("aero", "none") != "none" or case["rays"] * case["nd"] * case["ng"] > 30000:
        return None
    out = _exact_clear(case, seed)
    if kind in ("pencil", "formod"):
        return dict(rad=out["rad"].T, tau=out["tau"].T, tpz=out["tpz"], tplon=out["tplon"], tplat=out["tplat"])
    return dict(out, nlos=None)


def _lin(x0, y0, x1, y1, x):
    return y0 + (y1 - y0) / (x1 - x0) * (x - x0)


def _planck(t, nu):
    return 1.19104259e-8 * nu ** 3 / np.expm1(1.43877506 * nu / t)


def _cart(z, lon, lat):
    r, lon, lat = z + synth.RE, np.radians(lon), np.radians(lat)
    return np.stack([r * np.cos(lat) * np.cos(lon), r * np.cos(lat) * np.sin(lon), r * np.sin(lat)], -1)


def _geo(x):
    r = np.sqrt((x * x).sum(-1))
    return r - synth.RE, np.degrees(np.arctan2(x[..., 1], x[..., 0])), np.degrees(np.arcsin(x[..., 2] / r))


def _hydrostatic(a, water):
    """Pressure from the lowest level up (src/atmosphere.c:188-243)."""
    s1, s2 = np.sin(np.radians(a["lat"][0])), np.sin(np.radians(2 * a["lat"][0]))
    g0 = 9.780318 * (1 + 0.0053024 * s1 * s1 - 0.0000058 * s2 * s2)
    p, f = a["p"].copy(), np.arange(20) / 19.0
    for i in range(1, len(p)):
        z0, z1 = a["z"][i - 1], a["z"][i]
        e = water[i - 1] + (water[i] - water[i - 1]) * f
        t = a["t"][i - 1] + (a["t"][i] - a["t"][i - 1]) * f
        mass = e * 18.0153e-3 + (1 - e) * 28.96456e-3
        mean = np.mean(mass * (g0 - 3.086e-3 * (z0 + (z1 - z0) * f)) / 8.314472 / t)
        p[i] = np.exp(np.log(p[i - 1]) - mean * 1000 * (z1 - z0))
    return p


def _line_of_sight(atms, ray_atm, geom, water, balance):
    """Refracted lines of sight of all rays (src/lineofsight.c:5-190): the
    state of point i of every ray, the number of points, the surface
    temperature and the tangent points."""
    n, top = len(ray_atm), max(len(a["z"]) for a in atms)
    pad = {k: np.zeros((len(atms), top)) for k in ("z", "p", "t")}
    q = np.zeros((len(atms), atms[0]["q"].shape[0], top))
    size = np.array([len(a["z"]) for a in atms])
    for i, a in enumerate(atms):
        pad["z"][i], pad["z"][i, :size[i]] = np.inf, a["z"]
        pad["p"][i, :size[i]] = _hydrostatic(a, water(a)) if balance else a["p"]
        pad["t"][i, :size[i]], q[i, :, :size[i]] = a["t"], a["q"]
    ia = np.asarray(ray_atm)

    def state(z, full=False, who=slice(None)):
        w = ia[who]
        i = np.clip((pad["z"][w] <= z[:, None]).sum(1) - 1, 0, size[w] - 2)
        z0, z1 = pad["z"][w, i], pad["z"][w, i + 1]
        p0, p1 = pad["p"][w, i], pad["p"][w, i + 1]
        p = p0 * np.exp(np.log(p1 / p0) / (z1 - z0) * (z - z0))
        t = _lin(z0, pad["t"][w, i], z1, pad["t"][w, i + 1], z)
        if not full:
            return p, t
        return p, t, _lin(z0[:, None], q[w, :, i], z1[:, None], q[w, :, i + 1], z[:, None])

    zmin, zmax = pad["z"][ia, 0], pad["z"][ia, size[ia] - 1]
    obs, vp = _cart(geom["obsz"], geom["obslon"], geom["obslat"]), _cart(geom["vpz"], geom["vplon"], geom["vplat"])
    e0 = vp - obs
    far = np.sqrt((e0 * e0).sum(1))
    e0 /= far[:, None]
    x, lo, hi, seek = obs.copy(), np.zeros(n), far.copy(), geom["obsz"] > zmax
    while seek.any():      # entry into the atmosphere
        seek &= np.abs(lo - hi) > 0.001
        d = (lo + hi) / 2
        x[seek] = (obs + d[:, None] * e0)[seek]
        z = _geo(x)[0]
        seek &= ~((z <= zmax) & (z > zmax - 0.001))
        below = z < zmax - 0.0005
        hi, lo = np.where(seek & below, d, hi), np.where(seek & ~below, d, lo)
    pts, live = [], np.ones(n, bool)
    count, tsurf, smooth = np.zeros(n, int), np.full(n, -999.0), np.zeros(n)
    before, seen = np.zeros((n, 3)), np.zeros(n)
    while live.any():
        r = np.sqrt((x * x).sum(1))
        cosa = np.abs((e0 * x).sum(1) / r)
        ds = np.minimum(10.0, 1.0 / np.maximum(cosa, 1e-300))
        z, lon, lat = _geo(x)
        out = (z < zmin + 0.001) | (z > zmax + 0.001)
        here = np.stack([z, lon, lat], 1)
        past = np.where((count > 0)[:, None], before, here)
        edge = np.where(z < zmin + 0.001, zmin, zmax)
        with np.errstate(all="ignore"):
            f = (past[:, 0] - edge) / (past[:, 0] - z)
        a, b = _cart(*past.T), _cart(z, lon, lat)
        with np.errstate(all="ignore"):
            here = np.where(out[:, None], np.stack(_geo(a + f[:, None] * (b - a)), 1), here)
        here = np.where(np.isfinite(here), here, 0.0)
        raw = np.where(out, 0.0, ds)
        smooth = 0.5 * (smooth + raw)      # the step before the first is 0
        p, t, qq = state(here[:, 0], full=True)
        pts.append(dict(p=p, t=t, q=qq, ds=smooth, raw=raw, geo=here, live=live.copy()))
        count += live
        # a ray that ends on the ground keeps the temperature it looked up
        # last, that of its last refraction step (src/lineofsight.c:98-166)
        tsurf = np.where(live & out & (z < zmin + 0.001), seen, tsurf)
        seen = t.copy()
        before, live = np.where(live[:, None], here, before), live & ~out
        bend = live & (z <= 60.0)
        e1 = e0 * np.where(bend, 1 + 7.753e-05 * p / t, 1.0)[:, None]
        w = np.flatnonzero(bend)
        if len(w):
            mid = x[w] + 0.5 * ds[w, None] * e0[w]
            p0, t0 = state(_geo(mid)[0], who=w)
            for i in range(3):
                step = mid.copy()
                step[:, i] += 0.02
                p1, t1 = state(_geo(step)[0], who=w)
                e1[w, i] += ds[w] * 7.753e-05 * (p1 / t1 - p0 / t0) / 0.02
            seen[w] = t1
        e1 /= np.sqrt((e1 * e1).sum(1))[:, None]
        x = np.where(live[:, None], x + 0.5 * ds[:, None] * (e0 + e1), x)
        e0 = np.where(live[:, None], e1, e0)
    raws, geo = np.array([s["raw"] for s in pts]), np.array([s["geo"] for s in pts])
    tp = np.zeros((n, 3))
    for r in range(n):
        if count[r] >= 3 and raws[count[r] - 2, r] < 1e-3:
            count[r] -= 1
        g, c = geo[:count[r], r], count[r]
        m = int(np.argmin(g[:, 0]))
        if m <= 0 or m >= c - 1:
            tp[r] = g[-1]
            continue
        y0, y1, y2 = g[m - 1, 0], g[m, 0], g[m + 1, 0]
        x1 = np.sqrt(raws[m, r] ** 2 - (y1 - y0) ** 2)
        x2 = x1 + np.sqrt(raws[m + 1, r] ** 2 - (y2 - y1) ** 2)
        aa = 1 / (x1 - x2) * (-(y0 - y1) / x1 + (y0 - y2) / x2)
        bb = -(y0 - y1) / x1 - aa * x1
        xx = -bb / (2 * aa)
        v = _lin(0.0, _cart(*g[m - 1]), x2, _cart(*g[m + 1]), xx)
        tp[r] = (aa * xx * xx + bb * xx + y0,) + _geo(v)[1:]
    return pts, count, tsurf, tp


def _continuum_tables():
    """The measured continuum coefficients (numbers only)."""
    text = open(os.path.join(os.getcwd(), "jurassic-scatter_b200", "csrc", "ckd_tables.h")).read()
    return {m.group(1): np.array([float(v) for v in re.findall(r"[-+0-9.eE]+", m.group(2))])
            for m in re.finditer(r"jsc_(\w+)\[\d+\] = \{([^}]*)\}", text)}


def _continua(nus, p, t, ds, qw, u_co2, u_h2o):
    """Continuum extinction [ray][channel] (src/continua.c:5-2049)."""
    c = _kept.setdefault("ckd", None) or _continuum_tables()
    _kept["ckd"] = c
    nu = np.asarray(nus)
    p, t, ds, qw, u_co2, u_h2o = (v[:, None] for v in (p, t, ds, qw, u_co2, u_h2o))

    def at(name, step):
        x = nu / step
        i = x.astype(int)
        return (1 - (x - i)) * c[name][i] + (x - i) * c[name][i + 1]

    ctw = ((t - 260) * 5.050505e-4 * (t - 296) * at("ckd_co2_t230", 2) - (t - 230) * 9.259259e-4 * (t - 296) *
           at("ckd_co2_t260", 2) + (t - 230) * 4.208754e-4 * (t - 260) * at("ckd_co2_t296", 2))
    beta = u_co2 / 6.02214199e23 / 1000 * p / 1013.25 * ctw / ds
    inside = (nu > 820) & (nu < 960)
    sfac = np.where(inside, np.interp((nu - 820) / 10, np.arange(15), c["ckd_h2o_xfc"]), 1.0)
    w296, w260 = at("ckd_h2o_t296", 10), at("ckd_h2o_t260", 10)
    v2 = (nu - 370) ** 2
    frn = at("ckd_h2o_frn", 10) * (36100 / (v2 + v2 ** 3 * 1e-8 + 36100) * -0.25 + 1)
    self_ = sfac * w296 * (w260 / w296) ** ((296 - t) / 36)
    beta = beta + (nu * u_h2o * np.tanh(0.7193876 / t * nu) * (296 / t) *
                   (p / 1013.25 * (qw * self_ + (1 - qw) * frn) * 1e-20)) / ds
    on = (nu >= c["o2_nu"][0]) & (nu <= c["o2_nu"][-1])
    b, be = np.interp(nu, c["o2_nu"], c["o2_b"]), np.interp(nu, c["o2_nu"], c["o2_beta"])
    return beta + np.where(on, 0.1 * (p / 1013.25) ** 2 * (273 / t) ** 2 * 0.21 * b * np.exp(be * (1 / 296 - 1 / t)), 0.0)


def _bracket(keys, last, x):
    """Largest i <= last with keys[..., i] <= x, else 0."""
    lo, hi = np.zeros(x.shape, int), last + 1
    while (hi > lo + 1).any():
        mid = (lo + hi) >> 1
        above = np.take_along_axis(keys, mid[..., None], -1)[..., 0] > x
        hi, lo = np.where(above & (hi > lo + 1), mid, hi), np.where(~above & (hi > lo + 1), mid, lo)
    return lo


def _exact_clear(case, seed):
    atms, ray_atm, geom = _profiles_and_rays(case, seed)
    emitters, nus = EMITTERS[:case["ng"]], _channels(case["nd"])
    iw = emitters.index("H2O") if "H2O" in emitters else -1
    pts, count, tsurf, tp = _line_of_sight(atms, ray_atm, geom, lambda a: a["q"][iw] if iw >= 0 else 0 * a["z"],
                                           case["kind"] != "pencil")   # a pencil takes the pressures as given
    nr, nd, ng = case["rays"], case["nd"], case["ng"]
    lut_p, lut_t, nu_pts = synth.LUT_P, synth.LUT_T, len(synth.LUT_U)
    eps = np.full((nd, ng, len(lut_p), len(lut_t), nu_pts), np.inf)
    cnt = np.zeros((nd, ng, len(lut_p), len(lut_t)), int)
    for d, nu in enumerate(nus):
        for g, e in enumerate(emitters):
            for i, rows in enumerate(synth.emissivity_table(e, nu, TABLE_SEED)[2]):
                for j, (u, v) in enumerate(rows):
                    eps[d, g, i, j, :len(v)], cnt[d, g, i, j] = v, len(v)
    col = synth.LUT_U.astype(np.float32).astype(np.float64)
    temps = 100.0 + 0.25 * np.arange(1201)
    plk = np.empty((nd, 1201))
    for d, nu in enumerate(nus):
        x = np.arange(nu - 0.6, nu + 0.6 + 0.0025, 0.005)
        f = (np.abs(x - nu) <= 0.5 + 1e-9).astype(float)
        x = np.array([float("%.4f" % v) for v in x])
        plk[d] = (f[:, None] * _planck(temps[None], x[:, None])).sum(0) / f.sum()

    def planck_at(t):
        i = np.clip(((t - 100.0) * 4.0).astype(int), 0, 1199)
        return (plk[:, i] + (plk[:, i + 1] - plk[:, i]) / 0.25 * (t - temps[i])).T

    rad, tau, path = np.zeros((nr, nd)), np.ones((nr, nd)), np.ones((nr, nd, ng))
    dd, gg = np.arange(nd)[None, :, None], np.arange(ng)[None, None, :]
    for k, s in enumerate(pts):
        w = np.flatnonzero(count > k)
        if not len(w):
            break
        p, t, ds, q = s["p"][w], s["t"][w], s["ds"][w], s["q"][w]
        u = 10 * q * (p / (1.3806504e-23 * t) * ds)[:, None]
        tpath = path[w]
        ip = np.clip(np.searchsorted(lut_p, p, "right") - 1, 0, len(lut_p) - 2)
        it = np.clip(np.searchsorted(lut_t, t, "right") - 1, 0, len(lut_t) - 2)
        corner = []
        for a in (0, 1):
            for b in (0, 1):
                i, j = (ip + a)[:, None, None], (it + b)[:, None, None]
                row, n = eps[dd, gg, i, j], cnt[dd, gg, i, j]
                x1 = 1 - tpath
                m = _bracket(row, n - 2, x1)
                e0, e1 = (np.take_along_axis(row, (m + o)[..., None], -1)[..., 0] for o in (0, 1))
                x2 = _lin(e0, col[m], e1, col[m + 1], x1) + u[:, None, :]
                m = _bracket(np.broadcast_to(col, row.shape), n - 2, x2)
                e0, e1 = (np.take_along_axis(row, (m + o)[..., None], -1)[..., 0] for o in (0, 1))
                corner.append(np.clip(_lin(col[m], e0, col[m + 1], e1, x2), 0, 1))
        tt, pp = t[:, None, None], p[:, None, None]
        t0, t1 = lut_t[it][:, None, None], lut_t[it + 1][:, None, None]
        ea = np.clip(_lin(t0, corner[0], t1, corner[1], tt), 0, 1)
        eb = np.clip(_lin(t0, corner[2], t1, corner[3], tt), 0, 1)
        ea = np.clip(_lin(lut_p[ip][:, None, None], ea, lut_p[ip + 1][:, None, None], eb, pp), 0, 1)
        with np.errstate(all="ignore"):
            seg = np.where(tpath < 1e-9, 0.0, (1 - ea) / tpath)
        path[w] = tpath * seg
        gas = seg.prod(-1)
        none = np.zeros(len(w))
        beta = _continua(nus, p, t, ds, q[:, iw] if iw >= 0 else none, u[:, emitters.index("CO2")],
                         u[:, iw] if iw >= 0 else none)
        e = 1 - gas * np.exp(-beta * ds[:, None])
        step = gas > 0
        rad[w] += np.where(step, planck_at(t) * e * tau[w], 0.0)
        tau[w] *= np.where(step, 1 - e, 1.0)
    hit = tsurf > 0
    rad[hit] += planck_at(tsurf[hit]) * tau[hit]
    return dict(rad=rad, tau=tau, tpz=tp[:, 0], tplon=tp[:, 1], tplat=tp[:, 2])


def _mix(state):
    m = (1 << 64) - 1
    state = (state + 0x9E3779B97F4A7C15) & m
    z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return state, z ^ (z >> 31)


def _exact_train(case, seed):
    """The training recipe (standardised log sources, shuffled minibatches,
    Adam with cosine decay) in 64 bits."""
    x, src = _training_set(case, seed)
    n, nd, batch, epochs = case["samples"], case["nd"], case["batch"], case["epochs"]
    x = x.astype(np.float64)
    xs = x.std(0)
    x = (x - x.mean(0)) / np.where(xs * xs > 1e-12, xs, 1.0)
    y = np.log(src)
    y = (y - y.mean(0)) / y.std(0)
    state, w = 5, []
    for i, o in ((8, 128), (128, 128), (128, 128), (128, nd)):
        r = np.empty(i * o)
        for k in range(i * o):
            state, v = _mix(state)
            r[k] = (v >> 11) * 2.0 ** -53
        w += [(np.sqrt(6.0 / (i + o)) * (2 * r - 1)).reshape(o, i).astype(np.float32).astype(float), np.zeros(o)]
    m, v, step = [0 * a for a in w], [0 * a for a in w], 0
    losses, state = [], 7
    for ep in range(epochs):
        perm = list(range(n))
        for i in range(n - 1, 0, -1):
            state, z = _mix(state)
            j = z % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        perm = np.array(perm)
        lr = 3e-3 * 0.5 * (1 + np.cos(np.pi * ep / epochs))
        for b0 in range(0, n - batch + 1, batch):
            h = [x[perm[b0:b0 + batch]]]
            for k in range(4):
                a = h[-1] @ w[2 * k].T + w[2 * k + 1]
                h.append(np.tanh(a) if k < 3 else a)
            d = h[4] - y[perm[b0:b0 + batch]]
            loss, d, grad = (d * d).sum() / batch, 2 * d / batch, [None] * 8
            for k in (3, 2, 1, 0):
                grad[2 * k], grad[2 * k + 1] = d.T @ h[k], d.sum(0)
                if k:
                    d = (d @ w[2 * k]) * (1 - h[k] ** 2)
            step += 1
            for k in range(8):
                m[k] = 0.9 * m[k] + 0.1 * grad[k]
                v[k] = 0.999 * v[k] + 0.001 * grad[k] ** 2
                w[k] = w[k] - lr * (m[k] / (1 - 0.9 ** step)) / (np.sqrt(v[k] / (1 - 0.999 ** step)) + 1e-8)
        losses.append(loss)
    return dict(losses=np.array(losses), weights=np.concatenate([a.ravel() for a in w]))


def _mie_series(x, m):
    """Q_ext, Q_sca and the normalised phase function at 0..180 degrees of
    spheres with size parameters x and refractive indices m (Bohren and
    Huffman 1983, appendix A)."""
    nstop = (x + 4 * x ** 0.3333 + 2).astype(int)
    nmx = int(max(nstop.max(), np.abs(x * m).max())) + 16
    y = x * m
    log_d = np.zeros((nmx + 1, len(x)), complex)
    for n in range(nmx, 1, -1):
        log_d[n - 1] = n / y - 1 / (log_d[n] + n / y)
    mu = np.cos(np.radians(np.arange(181.0)))[:, None]
    pi0, pi1 = np.zeros((181, 1)), np.ones((181, 1))
    s1 = s2 = np.zeros((181, len(x)), complex)
    psi0, psi1, chi0, chi1 = np.cos(x), np.sin(x), -np.sin(x), np.cos(x)
    qsca = np.zeros(len(x))
    for n in range(1, int(nstop.max()) + 1):
        use = n <= nstop
        with np.errstate(all="ignore"):
            psi, chi = (2 * n - 1) * psi1 / x - psi0, (2 * n - 1) * chi1 / x - chi0
            xi, xi1 = psi - 1j * chi, psi1 - 1j * chi1
            a = ((log_d[n] / m + n / x) * psi - psi1) / ((log_d[n] / m + n / x) * xi - xi1)
            b = ((log_d[n] * m + n / x) * psi - psi1) / ((log_d[n] * m + n / x) * xi - xi1)
        a, b = np.where(use, a, 0), np.where(use, b, 0)
        psi0, psi1 = psi1, np.where(use, psi, psi1)
        chi0, chi1 = chi1, np.where(use, chi, chi1)
        f = (2 * n + 1) / (n * (n + 1))
        tau = n * mu * pi1 - (n + 1) * pi0
        s1, s2 = s1 + f * (a * pi1 + b * tau), s2 + f * (a * tau + b * pi1)
        qsca += (2 * n + 1) * (np.abs(a) ** 2 + np.abs(b) ** 2)
        pi0, pi1 = pi1, ((2 * n + 1) * mu * pi1 - (n + 1) * pi0) / n
    qs = 2 / x ** 2 * qsca
    return 4 / x ** 2 * s1[0].real, qs, 2 / (x * x * qs) * (np.abs(s1) ** 2 + np.abs(s2) ** 2)


def _exact_mie(case, seed):
    ctl = prepare(case, seed)["ctl"]
    nus = np.array(ctl.nu[:ctl.nd])
    if case["layer"] == "layers":     # a database layer among the Mie modes: host look-up
        return None
    ice = case["layer"] == "ice"
    count, radius, width = (0.1, 10.0, 1.8) if ice else (10.0, 0.1, 1.5)
    grid = np.arange(600.0, 1500.5, 1.0)
    n, k = (synth.ice_refractive_index if ice else synth.sulfate_refractive_index)(grid)
    n, k = (np.array([float("%.8f" % v) for v in a]) for a in (n, k))
    m = np.interp(nus, grid, n) + 1j * np.interp(nus, grid, k)
    z, w = np.polynomial.hermite.hermgauss(170)
    be, bs, ph = np.zeros(len(nus)), np.zeros(len(nus)), np.zeros((len(nus), 181))
    r = np.exp(np.sqrt(2) * np.log(width) * z + np.log(radius))
    keep = (r >= 0.001) & (r <= 1000.0)
    r, w = r[keep], w[keep]
    for d in range(len(nus)):
        qe, qs, p = _mie_series(2 * np.pi * r * nus[d] * 1e-4, np.full(len(r), m[d]))
        f = count * 1e-3 * np.sqrt(np.pi) * r ** 2 * w
        be[d], bs[d], ph[d] = (f * qe).sum(), (f * qs).sum(), (f * qs * p).sum(1)
        ph[d] /= bs[d]
    return dict(beta_e=be[None], beta_s=bs[None], beta_a=(be - bs)[None], p=ph[None])
