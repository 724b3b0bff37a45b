"""Edge sizes of the batch kernels against host restatements: sizes at the
ends of a kernel's tiles, remainders and the branches that a rule on sizes
selects."""
import numpy as np
import pytest

from helpers import max_rel

pytestmark = pytest.mark.gpu


def _hydrostatic(z, lon, lat, t, qh, p, hydz):
    """src/atmosphere.c:163-243 in numpy, column by column."""
    p = p.copy()
    cut = [0] + [i for i in range(1, len(z)) if lon[i] != lon[i - 1] or lat[i] != lat[i - 1]] + [len(z)]
    f = np.arange(20) / 19.0
    for i0, i1 in zip(cut[:-1], cut[1:]):
        ref = i0 + int(np.argmin(np.abs(z[i0:i1] - hydz)))
        s1, s2 = np.sin(np.radians(lat[ref])), np.sin(2 * np.radians(lat[ref]))
        g0 = 9.780318 * (1 + 0.0053024 * s1 * s1 - 0.0000058 * s2 * s2)
        for d, span in ((1, range(ref + 1, i1)), (-1, range(ref - 1, i0 - 1, -1))):
            for i in span:
                j = i - d
                e, tt = qh[j] + (qh[i] - qh[j]) * f, t[j] + (t[i] - t[j]) * f
                g = g0 - 3.086e-3 * (z[j] + (z[i] - z[j]) * f)
                mean = np.mean((e * 18.0153e-3 + (1 - e) * 28.96456e-3) * g / 8.314472 / tt)
                p[i] = np.exp(np.log(p[j]) - mean * 1000 * (z[i] - z[j]))
    return p


def _limb_inputs(workdir, z, n_rays=5, seed=3):
    from jscat import synth
    rng = np.random.default_rng(seed)
    atm = synth.atmosphere(synth.CFG0_EMITTERS, rng, t_sigma=0.0, z=z)
    geom = synth.limb_geometry(np.linspace(6.0, 40.0, n_rays))
    base = synth.write_tables(workdir, synth.CFG0_EMITTERS, synth.CFG0_NU, 20261203)
    return dict(emitters=synth.CFG0_EMITTERS, nus=synth.CFG0_NU, tblbase=base), atm, geom


@pytest.mark.parametrize("levels,hydz,columns", [(2, 0.0, 1), (3, 55.0, 1), (128, 0.0, 1), (129, 0.0, 1),
                                                 (130, 120.0, 1), (300, 41.7, 1), (121, 0.0, 2)])
def test_hydrostatic_levels(workdir, levels, hydz, columns):
    """The device's balance (a block per profile, 128 levels at a time)
    gives the radiances of a profile balanced on the host: 1e-9, the bound
    of the parity tests (log and exp differ by last bits)."""
    from jscat import api, synth, structs as S
    z = np.linspace(0.0, 120.0, levels)
    kw, atm, geom = _limb_inputs(workdir, z)
    more = {}
    if columns == 2:   # the points of one IP=3 atmosphere: each column is balanced by itself
        more = dict(ip=3, cz=1.5, cx=20000.0)
        for k in ("z", "lon", "lat", "p", "t"):
            atm[k] = np.concatenate([atm[k], atm[k]])
        atm["q"], atm["k"] = np.tile(atm["q"], 2), np.tile(atm["k"], 2)
        atm["lat"][levels:] = 20.0
    done = dict(atm, p=_hydrostatic(atm["z"], atm["lon"], atm["lat"], atm["t"], atm["q"][1], atm["p"], hydz))
    n = len(geom["obsz"])
    got = api.formod_batch(S.make_ctl(hydz=hydz, **kw, **more), synth.batch_from([atm], np.zeros(n, np.int32), geom))
    want = api.formod_batch(S.make_ctl(hydz=-999.0, **kw, **more), synth.batch_from([done], np.zeros(n, np.int32), geom))
    np.testing.assert_array_equal(got["nlos"], want["nlos"])
    assert np.all(want["rad"] > 0)
    assert max_rel(got["rad"], want["rad"]) <= 1e-9
    assert max_rel(got["tau"], want["tau"]) <= 1e-9
