"""Edge sizes of the batch kernels against host restatements: sizes at the
ends of a kernel's tiles, remainders and the branches that a rule on sizes
selects."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
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


def _mixed_rays(n, seed=5):
    from jscat import synth
    rng = np.random.default_rng(seed)
    a = synth.limb_geometry(rng.uniform(4.0, 70.0, n))
    b = synth.nadir_geometry(rng.uniform(0.0, 75.0, n))
    odd = np.arange(n) % 2 == 1
    geom = {k: np.where(odd, b[k], a[k]) for k in a}
    geom["obsz"][::7] = 30.0                       # observers inside the atmosphere
    geom["vpz"][3::11] = 130.0                     # and rays that miss it
    return geom


@pytest.mark.parametrize("grid", ["even", "uneven", "descending", "doubled", "two"])
@pytest.mark.parametrize("hydz", [0.0, -999.0])
def test_march_against_two_pass_tracing(workdir, grid, hydz):
    """The march over level records and its records of points against the
    counting and storing passes that jsc_formod_batch_noalloc keeps: the same
    operations, so the same bits, on profiles whose altitudes are evenly
    spaced, uneven, descending, doubled, or only two."""
    from jscat import api, synth, structs as S
    z = {"even": np.arange(0.0, 121.0), "uneven": 120.0 * np.linspace(0, 1, 90) ** 1.7,
         "descending": np.arange(120.0, -1.0, -1.0), "two": np.array([0.0, 120.0]),
         "doubled": np.sort(np.concatenate([np.arange(0.0, 121.0, 2.0), [14.0, 50.0]]))}[grid]
    kw, atm, _ = _limb_inputs(workdir, z)
    ctl = S.make_ctl(hydz=hydz, **kw)
    geom = _mixed_rays(97)
    inp = synth.batch_from([atm, dict(atm, t=atm["t"] + 3.0)], np.arange(97) % 2, geom)
    m = api.Model(ctl)
    got, want = api.formod_batch(ctl, inp, model=m), api.formod_batch_noalloc(ctl, inp, m)
    for k in ("nlos", "rad", "tau", "tpz", "tplon", "tplat"):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("refine", [False, True])
def test_march_lanes_and_pool(workdir, refine):
    """A thread per ray (above 16384 rays) and eight lanes per ray give the
    same bits, and so does a pool that starts too small and grows."""
    from jscat import api, synth, structs as S
    kw, atm, _ = _limb_inputs(workdir, np.arange(0.0, 121.0))
    aero = None
    if refine:
        aero = S.AeroT.from_buffer_copy(np.load(os.path.join(GOLDEN, "aero_ice8.npz"))["aero"].tobytes())
        kw.update(sca_n=1, sca_mult=0)
    ctl = S.make_ctl(hydz=0.0, **kw)
    n = 16385
    geom = _mixed_rays(n)
    m = api.Model(ctl)
    inp = synth.batch_from([atm], np.zeros(n, np.int32), geom)
    many = api.formod_batch(ctl, inp, model=m, aero=aero)
    for k in (1, 15, 17):
        part = synth.batch_from([atm], np.zeros(k, np.int32), {c: v[n - k:] for c, v in geom.items()})
        few = api.formod_batch(ctl, part, model=m, aero=aero)
        for c in few:
            np.testing.assert_array_equal(few[c], many[c][n - k:])
        b = api.Batch(m, ctl, 1, len(inp["z"]), k, max_seg=600 if refine else 1)
        try:
            if aero is not None:
                b.set_aero(aero)
            b.upload(part)
            b.run()
            few = b.download()
        finally:
            b.close()
        for c in few:
            np.testing.assert_array_equal(few[c], many[c][n - k:])


@pytest.mark.parametrize("nd,nalpha,layer", [(1, 10, "aero_sulfate16"), (16, 28, "aero_sulfate16"), (8, 20, "aero_ice8")])
def test_source_integral_against_port(workdir, nd, nalpha, layer):
    """Single-scattering radiances (source integral over pencil intervals)
    against the C restatement, which evaluates every direction: channel
    counts of one, part of and a whole channel pass, the fewest and the most
    pencils, a limb and an oblique ray and one that looks straight down,
    where the scattering frame is degenerate.  1e-9, the parity bound."""
    from jscat import api, synth, structs as S
    from oracle import refrun
    g = np.load(os.path.join(GOLDEN, layer + ".npz"))
    full = S.AeroT.from_buffer_copy(g["aero"].tobytes())
    kw, atm, _ = _limb_inputs(workdir, np.arange(0.0, 121.0))
    nus = [float(v) for v in g["nus"]][:nd]
    kw.update(nus=nus, tblbase=synth.write_tables(workdir, kw["emitters"], [float(v) for v in g["nus"]], 20261203),
              sca_n=1, sca_mult=1, hydz=0.0, ctm_co2=0, ctm_h2o=0)
    geom = {k: np.concatenate([a, b]) for (k, a), b in zip(
        synth.limb_geometry([17.3 if "sulfate" in layer else 9.7]).items(),
        synth.nadir_geometry([0.0, 41.0]).values())}
    geom["time"] = np.array([3600.0, 40000.0, 43200.0])
    inp = synth.batch_from([atm], np.zeros(3, np.int32), geom)
    got = api.formod_batch(S.make_ctl(**kw), inp, aero=full, nalpha=nalpha)
    ref = refrun.run_port(kw, [atm], np.zeros(3, int), geom, aero=bytes(full), threads=os.cpu_count(),
                          nalpha=nalpha, timeout=900)
    assert np.all(np.isfinite(ref["rad"])) and np.all(ref["rad"] > 0)
    assert max_rel(got["rad"], ref["rad"]) <= 1e-9
    assert max_rel(got["tau"], ref["tau"]) <= 1e-9


@pytest.mark.parametrize("nd", [7, 9, 17, 24, 25, 33])
def test_source_integral_channel_passes(workdir, nd):
    """Channel counts around the passes of 8 and 16: channels repeated from a
    run of 16, whose radiances are compared with the C restatement above.
    The passes add the same 180 polar steps of one sign in other groups:
    180 x 2 x 2^-53."""
    from jscat import api, synth, structs as S
    g = np.load(os.path.join(GOLDEN, "aero_sulfate16.npz"))
    full = S.AeroT.from_buffer_copy(g["aero"].tobytes())
    all_nus = [float(v) for v in g["nus"]]
    kw, atm, _ = _limb_inputs(workdir, np.arange(0.0, 121.0))
    base = synth.write_tables(workdir, kw["emitters"], all_nus, 20261203)
    geom = synth.limb_geometry([17.3, 12.1])
    inp = synth.batch_from([atm], np.zeros(2, np.int32), geom)

    def run(ch):
        aero = S.AeroT.from_buffer_copy(bytes(full))
        for il in range(full.nl):
            for j, i in enumerate(ch):
                aero.beta_e[il][j] = full.beta_e[il][i]
                aero.beta_s[il][j] = full.beta_s[il][i]
                aero.beta_a[il][j] = full.beta_a[il][i]
                for a in range(181):
                    aero.p[il][j][a] = full.p[il][i][a]
        kw.update(nus=[all_nus[i] for i in ch], tblbase=base, sca_n=1, sca_mult=1, hydz=0.0,
                  ctm_co2=0, ctm_h2o=0)
        return api.formod_batch(S.make_ctl(**kw), inp, aero=aero, nalpha=20)

    want, got = run(range(16)), run([i % 16 for i in range(nd)])
    for k in ("rad", "tau"):
        ref = want[k][:, [i % 16 for i in range(nd)]]
        assert np.all(np.isfinite(ref)) and np.any(ref > 0)
        assert max_rel(got[k], ref) <= 2 * 180 * 2.0 ** -53


@pytest.mark.parametrize("ng,nd,n", [(1, 1, 1), (2, 3, 7), (3, 2, 8), (5, 4, 9), (8, 2, 33), (9, 2, 17), (16, 1, 8),
                                     (17, 2, 9), (25, 1, 5)])
def test_window_variants_against_others(workdir, ng, nd, n):
    """The window lookups (four lanes and one lane per ray) against the
    thread-per-channel kernel, which
    computes the same operations in the same order: the same bits and table
    indices at emitter counts of every block size and rays at the edges of
    a tile of 8 and of 32."""
    from jscat import api, synth, structs as S
    emitters = (synth.CFG1_EMITTERS + ["X%02d" % i for i in range(25)])[:ng]
    nus = synth.CFG1_NU[5::20][:nd]
    ctlkw, atms, ray_atm, geom = synth.batched_case(workdir, n_rays=n, rays_per_atm=4, seed=77,
                                                    emitters=emitters, nus=nus)
    ctl = S.make_ctl(**ctlkw)
    inp = synth.batch_from(atms, ray_atm, geom)
    m = api.Model(ctl)
    four, one, want = (api.formod_batch(ctl, inp, model=m, digest=True, variant=v) for v in (21, 22, 6))
    for k in want:
        np.testing.assert_array_equal(four[k], want[k])
        np.testing.assert_array_equal(one[k], want[k])


@pytest.mark.parametrize("n,variant", [(900, 21), (1500, 21), (3000, 22)])
def test_default_variant_by_points(workdir, n, variant):
    """Limb and nadir rays in turn on both sides of the rule: rays count by
    their length against the longest, and either side gives the bits of the
    other."""
    from jscat import api, synth, structs as S
    emitters, nus = synth.CFG1_EMITTERS[:2], synth.CFG1_NU[::2]
    base = synth.write_tables(workdir, emitters, nus, 20261203)
    atm = synth.atmosphere(emitters, np.random.default_rng(1), t_sigma=0.0)
    a, c = (synth.limb_geometry(np.linspace(5.0, 60.0, n)), synth.nadir_geometry(np.linspace(0.0, 60.0, n)))
    geom = {k: np.where(np.arange(n) % 2 == 1, c[k], a[k]) for k in a}
    ctl = S.make_ctl(emitters, nus, base, hydz=0.0)
    inp = synth.batch_from([atm], np.zeros(n, np.int32), geom)
    m = api.Model(ctl)
    b = api.Batch(m, ctl, 1, len(inp["z"]), n)
    try:
        b.upload(inp)
        b.run()
        got = b.download()
        points, longest = int(got["nlos"].sum()), int(got["nlos"].max())
        warps = (points // longest + 31) // 32 * len(nus) * 2
        assert (warps <= 2048) == (variant == 21)
        assert b.variant()["variant"] == variant
    finally:
        b.close()
    want = api.formod_batch(ctl, inp, model=m, variant=43 - variant)
    for k in ("rad", "tau", "nlos"):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("kind", ["uneven", "ties", "shifted", "grids", "short"])
def test_gas_variants_on_irregular_tables(workdir, kind):
    """The default kernels' rules on tables (evenly spaced columns, strictly
    increasing rows, one grid) against the thread-per-channel kernel on
    tables that miss each of them: unevenly spaced columns, rows with equal
    neighbours, columns that differ by row, another (p, T) grid per emitter,
    and rows of two, one or no point.  The same bits and table indices."""
    from jscat import api, synth, structs as S
    rng = np.random.default_rng(11)
    d = os.path.join(workdir, "irregular_%s" % kind)
    os.makedirs(d, exist_ok=True)
    base, nu, emitters = os.path.join(d, "tab"), 800.0, ["CO2", "H2O", "O3"]
    synth.write_filter("%s_%.4f.filt" % (base, nu), nu)
    for e in emitters:
        p, t, rows = synth.emissivity_table(e, nu, 20261203)
        step = 1 + (kind == "grids") * emitters.index(e)
        p, t, rows = p[::step], t, rows[::step]
        for i, line in enumerate(rows):
            for j, (u, v) in enumerate(line):
                if kind == "uneven":
                    keep = np.sort(rng.choice(len(u), max(2, len(u) // 3), replace=False))
                    line[j] = (u[keep], v[keep])
                elif kind == "ties":
                    line[j] = (u, np.minimum(v, np.float32(0.6)))
                elif kind == "shifted":
                    line[j] = (u[(i + j) % 7:], v[(i + j) % 7:])
                elif kind == "short" and (i * 30 + j) % 5 == 0:
                    n = (i + j) % 3
                    line[j] = (u[150:150 + n], v[150:150 + n])
        synth.write_table_bin("%s_%.4f_%s.bin" % (base, nu, e), p, t, rows)
    ctl = S.make_ctl(emitters, [nu], base, hydz=0.0)
    atms = [synth.atmosphere(emitters, rng, t_sigma=5.0, vmr_sigma=0.2) for _ in range(3)]
    n = 41
    inp = synth.batch_from(atms, np.arange(n) % 3, _mixed_rays(n))
    m = api.Model(ctl)
    four, one, want = (api.formod_batch(ctl, inp, model=m, digest=True, variant=v) for v in (21, 22, 6))
    assert np.any(want["tau"] < 0.9)
    for k in want:
        np.testing.assert_array_equal(four[k], want[k])
        np.testing.assert_array_equal(one[k], want[k])


@pytest.mark.parametrize("n,nd", [(1, 1), (31, 5), (32, 16), (33, 3), (64, 64), (129, 33), (1000, 16), (4159, 7)])
def test_training_gradients_at_tile_edges(n, nd):
    """Gradients of one minibatch against the FP64 restatement at batches
    around the row tiles (32), the slices (64) and their remainders, and
    output widths that are no multiple of four.  Bounds as in the gradient
    check of the surrogate's tests: FP32 sums of n products, relative to the
    largest gradient."""
    from jscat import api
    from oracle import mlp_ref
    rng = np.random.default_rng(n * 100 + nd)
    s = api.Surrogate(nd=nd, seed=3)
    try:
        p = s.get_params()
        p = (p + rng.normal(0, 0.05, p.shape)).astype(np.float32)
        s.set_params(p)
        x = rng.normal(0, 1, (n, 8)).astype(np.float32)
        t = rng.normal(0, 1, (n, nd)).astype(np.float32)
        loss, g = s.loss_grad(x, t)
        ref_loss, ref_g = mlp_ref.loss_and_grads(s.layers(p.astype(np.float64)), x, t)
        assert abs(loss - ref_loss) <= 1e-4 * abs(ref_loss)
        flat = np.concatenate([np.concatenate([gw.ravel(), gb]) for gw, gb in ref_g])
        assert np.max(np.abs(g - flat)) <= 2e-4 * np.max(np.abs(flat))
    finally:
        s.close()


@pytest.mark.parametrize("n,nd", [(16, 1), (297, 3), (1000, 16), (4099, 64)])
def test_training_set_standardisation(n, nd):
    """Loss of the untrained network on the whole training set, whose targets
    are the standardised logarithms: against numpy in 64 bits, at sample
    counts below, at and past the rows of the statistics' blocks.  Tolerance:
    three sums of 128 products in FP32 (3 x 128 x 2^-24)."""
    from jscat import api
    rng = np.random.default_rng(n)
    x = (rng.normal(size=(n, 8)) * 10.0 ** np.arange(-3, 5)).astype(np.float32)
    x[:, 3] = 7.25                                 # a feature without spread
    src = np.exp(rng.normal(size=(n, nd)) - 30.0)
    src[0, 0] = 0.0                                # bounded below
    sur = api.Surrogate(nd, seed=3)
    got = sur.train(x, src, epochs=1, batch=n, lr=0.0)
    par = sur.get_params().astype(np.float64)
    sur.close()
    h = x.astype(np.float64)
    sd = h.std(0)
    h = (h - h.mean(0)) / np.where(sd * sd > 1e-12, sd, 1.0)
    y = np.log(np.maximum(src, 1e-300))
    y = (y - y.mean(0)) / y.std(0)
    o = 0
    for k, (a, b) in enumerate(((8, 128), (128, 128), (128, 128), (128, nd))):
        h = h @ par[o:o + a * b].reshape(b, a).T + par[o + a * b:o + a * b + b]
        o += a * b + b
        h = np.tanh(h) if k < 3 else h
    want = ((h - y) ** 2).sum() / n
    assert abs(got[0] - want) <= 3 * 128 * 2.0 ** -24 * want


def _mie_numpy(x, m):
    """Q_ext, Q_sca and phase function of spheres (Bohren and Huffman 1983,
    appendix A, whose downward recurrence starts 15 orders above the larger
    of the last order and |x m|), all orders of all spheres at once."""
    nstop = (x + 4 * x ** 0.3333 + 2).astype(int)
    nmx = (np.maximum(x + 4 * x ** 0.3333 + 2, np.abs(x * m)) + 15).astype(int)
    d = np.zeros((nmx.max() + 1, len(x)), complex)
    for n in range(nmx.max(), 1, -1):
        d[n - 1] = np.where(n <= nmx, n / (x * m) - 1 / (d[n] + n / (x * m)), 0)
    mu = np.cos(np.radians(np.arange(181.0)))[:, None]
    p0, p1 = np.zeros((181, 1)), np.ones((181, 1))
    s1, s2 = np.zeros((181, len(x)), complex), np.zeros((181, len(x)), complex)
    psi0, psi1, chi0, chi1, q = np.cos(x), np.sin(x), -np.sin(x), np.cos(x), np.zeros(len(x))
    for n in range(1, int(nstop.max()) + 1):
        use = n <= nstop
        with np.errstate(all="ignore"):
            psi, chi = (2 * n - 1) * psi1 / x - psi0, (2 * n - 1) * chi1 / x - chi0
            xi, xi1 = psi - 1j * chi, psi1 - 1j * chi1
            a = ((d[n] / m + n / x) * psi - psi1) / ((d[n] / m + n / x) * xi - xi1)
            b = ((d[n] * m + n / x) * psi - psi1) / ((d[n] * m + n / x) * xi - xi1)
        a, b = np.where(use, a, 0), np.where(use, b, 0)
        psi0, psi1 = psi1, np.where(use, psi, psi1)
        chi0, chi1 = chi1, np.where(use, chi, chi1)
        f, t = (2 * n + 1) / (n * (n + 1)), n * mu * p1 - (n + 1) * p0
        s1, s2 = s1 + f * (a * p1 + b * t), s2 + f * (a * t + b * p1)
        q += (2 * n + 1) * (np.abs(a) ** 2 + np.abs(b) ** 2)
        p0, p1 = p1, ((2 * n + 1) * mu * p1 - (n + 1) * p0) / n
    qs = 2 / x ** 2 * q
    return 4 / x ** 2 * s1[0].real, qs, 2 / (x * x * qs) * (np.abs(s1) ** 2 + np.abs(s2) ** 2)


@pytest.mark.parametrize("nr,ni", [(1.31, 0.0), (1.45, 1e-3), (2.5, 1.2)])
def test_mie_series_at_its_ends(nr, ni):
    """The Mie kernel's series against numpy from one order to some hundred
    and at odd and even last orders, without and with absorption.  1e-10 of
    the phase function's largest value: the recurrences lose about as many
    bits as they have hundreds of orders, from 2e-16."""
    import ctypes as C
    from jscat import lib as L
    lib = L.load()
    lib.jsc_mie_eval.restype = C.c_int
    x = np.concatenate([np.logspace(-3, 0, 9), np.arange(1.0, 12.0, 0.5), [63.2, 64.8, 127.1, 300.3, 701.0]])
    n = len(x)
    out = np.empty((n, 183))
    arr = [np.ascontiguousarray(v, dtype=np.float64) for v in (x, np.full(n, nr), np.full(n, ni))]
    dp = C.POINTER(C.c_double)
    assert lib.jsc_mie_eval(0, n, *[a.ctypes.data_as(dp) for a in arr], out.ctypes.data_as(dp)) == 0
    qe, qs, ph = _mie_numpy(x, np.full(n, nr + 1j * ni))
    assert max_rel(out[:, 1], qs) <= 1e-10
    big = x > 0.05          # extinction of a tiny sphere cancels to its last bits
    assert max_rel(out[big, 0], qe[big]) <= 1e-10
    assert np.max(np.abs(out[:, 2:] - ph.T) / ph.T.max(axis=1, keepdims=True)) <= 1e-10


@pytest.mark.parametrize("n", [3, 1300])
def test_mie_series_beyond_shared_memory(n):
    """Size parameters whose orders fit shared memory, alone and in a call
    with one whose orders do not (all tasks then keep them in device memory,
    in several launches from 1185 tasks on): the same operations, the same
    bits."""
    import ctypes as C
    from jscat import lib as L
    lib = L.load()
    lib.jsc_mie_eval.restype = C.c_int
    dp = C.POINTER(C.c_double)

    def run(x):
        out = np.empty((len(x), 183))
        arr = [np.ascontiguousarray(v) for v in (x, np.full(len(x), 1.33), np.full(len(x), 1e-4))]
        assert lib.jsc_mie_eval(0, len(x), *[a.ctypes.data_as(dp) for a in arr], out.ctypes.data_as(dp)) == 0
        return out

    x = np.random.default_rng(n).uniform(0.1, 400.0, n)
    want, got = run(x), run(np.append(x, 5400.0))
    assert np.all(np.isfinite(got))
    np.testing.assert_array_equal(got[:n], want)
