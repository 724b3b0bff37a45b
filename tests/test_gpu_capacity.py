"""Fixed-capacity batches whose lines of sight exceed the capacity given at
their creation: the run reports it, the rays inside the buffers keep their
results, the others are cut, and the next request that fits is unaffected."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

NLOS_STATUS = 5   # JSC_ERR_NLOS
KEYS = ("rad", "tau", "tpz", "tplon", "tplat", "nlos")


def _rays(n, seed=5):
    from jscat import synth
    rng = np.random.default_rng(seed)
    a, b = synth.limb_geometry(rng.uniform(6.0, 50.0, n)), synth.nadir_geometry(rng.uniform(0.0, 60.0, n))
    odd = np.arange(n) % 3 == 1
    geom = {k: np.where(odd, b[k], a[k]) for k in a}
    geom["vpz"][4::13] = 130.0    # rays that miss the atmosphere
    return geom


def _case(workdir, nd, n, aero=False, **kw):
    from jscat import synth, structs as S
    rng = np.random.default_rng(3)
    atms = [synth.atmosphere(synth.CFG0_EMITTERS, rng, t_sigma=1.0) for _ in range(2)]
    base = synth.write_tables(workdir, synth.CFG0_EMITTERS, synth.CFG0_NU, 20261203)
    layers = None
    if aero:
        layers = S.AeroT.from_buffer_copy(np.load(os.path.join(GOLDEN, "aero_ice8.npz"))["aero"].tobytes())
        kw = dict(dict(sca_n=1, sca_mult=0), **kw)
    ctl = S.make_ctl(synth.CFG0_EMITTERS, synth.CFG0_NU[:nd], base, hydz=0.0, **kw)
    geom = _rays(n)
    return ctl, synth.batch_from(atms, np.arange(n) % 2, geom), layers


def _missing(inp, rays):
    """The same request with some of its rays above the atmosphere."""
    out = {k: np.array(v) for k, v in inp.items()}
    out["vpz"][rays] = 130.0
    return out


def _overflowing(ctl, inp, layers, model, cap, variant=-1):
    """Outputs of a fixed run that has to report the capacity, then those of
    the same batch on rays that fit."""
    from jscat import api, lib as L
    n, nd = len(inp["ray_atm"]), ctl.nd
    b = api.Batch(model, ctl, len(inp["atm_off"]) - 1, len(inp["z"]), n, max_seg=cap)
    out = {k: np.full((n, nd) if k in ("rad", "tau") else n, -7, np.int32 if k == "nlos" else float) for k in KEYS}
    try:
        if layers is not None:
            b.set_aero(layers)
        b.set_variant(variant)
        L.check(L.load().jsc_batch_set_fixed(b.h, 1), "jsc_batch_set_fixed")
        b.upload(inp)
        b.run()
        with pytest.raises(L.JscError) as e:
            b.download(out=out)
        assert e.value.status == NLOS_STATUS
        first = int(np.argmin(out["nlos"] == api.formod_batch(ctl, inp, model=model, aero=layers)["nlos"]))
        fits = _missing(inp, np.arange(n) >= max(first, 1) // 2 + 1)
        b.upload(fits)
        b.run()
        again = b.download()
        want = api.formod_batch(ctl, fits, model=model, aero=layers)
        for k in KEYS:
            np.testing.assert_array_equal(again[k], want[k])
    finally:
        b.close()
    return out


def _cut_chains(points, n, cap, nd):
    """The march has to run out of chunks of 32 points: more of them than the
    pool holds (a chunk of 1284 bytes per ray and per 32 points of the
    capacity, or the continuum array if that is larger)."""
    pool = max((n + cap // 32 + 1) * 1284 // 8 + 1, cap * nd) * 8 // 1284
    return np.sum((points + 31) // 32) > pool


@pytest.mark.parametrize("nd,n,variant,part", [(1, 64, -1, 0.3), (2, 64, 21, 0.3), (2, 64, 22, 0.4), (2, 200, 6, 0.02),
                                               (1, 33, -1, 0.97), (4, 40, 21, 0.9), (2, 20000, -1, 0.5)])
def test_clear_air_past_capacity(workdir, nd, n, variant, part):
    """Rays inside the capacity keep the bits of an ordinary run, the one
    across its end keeps its points inside, later ones none; where the
    capacity is a fraction of the points the march's pool runs out as well
    (a thread per ray above 16384 rays)."""
    from jscat import api
    ctl, inp, _ = _case(workdir, nd, n)
    m = api.Model(ctl)
    full = api.formod_batch(ctl, inp, model=m)
    end = np.cumsum(full["nlos"])
    cap = int(part * end[-1])
    cut = int(np.argmax(end > cap))
    if part <= 0.5:
        assert _cut_chains(full["nlos"], n, cap, nd)
    out = _overflowing(ctl, inp, None, m, cap, variant)
    for k in KEYS:
        np.testing.assert_array_equal(out[k][:cut], full[k][:cut])
    assert out["nlos"][cut] == cap - (end[cut] - full["nlos"][cut])
    assert np.all(out["nlos"][cut + 1:] == 0)
    for k, v in (("tpz", "vpz"), ("tplon", "vplon"), ("tplat", "vplat")):
        np.testing.assert_array_equal(out[k][cut:], inp[v][cut:])


@pytest.mark.parametrize("mult,nd,n,variant,part", [(0, 1, 48, -1, 0.3), (0, 2, 48, 22, 0.3), (0, 4, 30, -1, 0.9),
                                                    (1, 2, 9, -1, 0.6), (1, 4, 5, 22, 0.9)])
def test_layers_past_capacity(workdir, mult, nd, n, variant, part):
    """The same with layer edges between the points and single scattering:
    the ray across the end of the buffers keeps nothing."""
    from jscat import api
    ctl, inp, layers = _case(workdir, nd, n, True, sca_mult=mult)
    m = api.Model(ctl)
    full = api.formod_batch(ctl, inp, model=m, aero=layers)
    end = np.cumsum(full["nlos"])
    cap = int(part * end[-1])
    cut = int(np.argmax(end > cap))
    clear, _, _ = _case(workdir, nd, n)
    marched = api.formod_batch(clear, inp, model=m)["nlos"]
    assert np.all(np.cumsum(marched)[:cut] <= cap)
    if part <= 0.3:
        assert _cut_chains(marched, n, cap, nd)
    out = _overflowing(ctl, inp, layers, m, cap, variant)
    for k in KEYS:
        np.testing.assert_array_equal(out[k][:cut], full[k][:cut])
    assert np.all(out["nlos"][cut:] == 0)
    past = np.cumsum(marched) > cap
    for k, v in (("tpz", "vpz"), ("tplon", "vplon"), ("tplat", "vplat")):
        np.testing.assert_array_equal(out[k][~past], full[k][~past])
        np.testing.assert_array_equal(out[k][past], inp[v][past])


@pytest.mark.parametrize("layers", [False, True])
@pytest.mark.parametrize("variant", [9, 13, 14, 17])
def test_continuum_pass_past_capacity(workdir, layers, variant):
    """The lane and ray-tile variants, whose pass over all (point, channel)
    pairs takes their number from the device: not more than the buffers
    hold."""
    from jscat import api
    n = 24
    ctl, inp, aero = _case(workdir, 4, n, layers)
    m = api.Model(ctl)
    full = api.formod_batch(ctl, inp, model=m, aero=aero)
    end = np.cumsum(full["nlos"])
    cap = int(0.5 * end[-1])
    cut = int(np.argmax(end > cap))
    out = _overflowing(ctl, inp, aero, m, cap, variant)
    for k in KEYS:
        np.testing.assert_array_equal(out[k][:cut], full[k][:cut])


@pytest.mark.parametrize("layers", [False, True])
def test_graph_past_capacity(workdir, layers):
    """A captured graph: a replay past the capacity reports it, the replay
    after it gives the bits of an ordinary run."""
    import torch
    from jscat import api, lib as L
    n = 64
    ctl, inp, aero = _case(workdir, 2, n, layers)
    m = api.Model(ctl)
    full = api.formod_batch(ctl, inp, model=m, aero=aero)
    end = np.cumsum(full["nlos"])
    cap = int(0.4 * end[-1])
    cut = int(np.argmax(end > cap))
    fits = _missing(inp, np.arange(n) >= cut)
    want = api.formod_batch(ctl, fits, model=m, aero=aero)
    stream = torch.cuda.Stream()
    pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()   # noqa: E731
    gb = api.GraphBatch(m, ctl, fits, stream.cuda_stream, pin, max_seg=cap, aero=aero)
    try:
        for _ in range(2):
            gb.launch(inp)
            stream.synchronize()
            with pytest.raises(L.JscError) as e:
                gb.status()
            assert e.value.status == NLOS_STATUS
            np.testing.assert_array_equal(gb.out["rad"][:cut], full["rad"][:cut])
            gb.launch(fits)
            stream.synchronize()
            gb.status()
            for k in KEYS:
                np.testing.assert_array_equal(gb.out[k], want[k])
    finally:
        gb.close()


@pytest.mark.parametrize("ip,mult", [(2, None), (2, 0), (3, 0)])
def test_horizontally_varying_past_capacity(workdir, ip, mult):
    """IP 2 and 3, without and with layers, whose edges are a pass over the
    stored points: the ray across the end keeps its points inside in clear
    air and nothing with layers."""
    from jscat import api, synth, structs as S
    ctlkw, atm, geom = synth.curtain_case(workdir)
    geom = {k: v[::4] for k, v in geom.items()}
    n, layers = len(geom["obsz"]), None
    kw = dict(ctlkw, nus=ctlkw["nus"][:2], ip=ip, **(dict(cz=1.5, cx=900.0) if ip == 3 else {}))
    if mult is not None:
        layers = S.AeroT.from_buffer_copy(np.load(os.path.join(GOLDEN, "aero_ice8.npz"))["aero"].tobytes())
        kw.update(sca_n=1, sca_mult=mult)
    atms = [{k: v[..., 121 * i:121 * i + 121] for k, v in atm.items()} for i in range(5)] if ip == 2 else [atm]
    ctl, inp = S.make_ctl(**kw), synth.batch_from(atms, np.zeros(n, np.int32), geom)
    m = api.Model(ctl)
    full = api.formod_batch(ctl, inp, model=m, aero=layers)
    end = np.cumsum(full["nlos"])
    cap = int(0.6 * end[-1])
    cut = int(np.argmax(end > cap))
    out = _overflowing(ctl, inp, layers, m, cap)
    for k in KEYS:
        np.testing.assert_array_equal(out[k][:cut], full[k][:cut])
    assert out["nlos"][cut] == (cap - (end[cut] - full["nlos"][cut]) if mult is None else 0)
    assert np.all(out["nlos"][cut + 1:] == 0)


@pytest.mark.parametrize("ip,n,cap", [(1, 1, 1), (1, 17, 1), (1, 17, 200), (2, 5, 1), (3, 3, 100)])
def test_buffers_grow_with_layers(workdir, ip, n, cap):
    """Ordinary runs whose rays, each by itself, have more points with the
    layer edges than the batch starts with room for: the buffers grow, as
    they do in clear air."""
    from jscat import api, synth, structs as S
    ctlkw, atm, geom = synth.curtain_case(workdir)
    geom = {k: v[:n] for k, v in geom.items()}
    layers = S.AeroT.from_buffer_copy(np.load(os.path.join(GOLDEN, "aero_ice8.npz"))["aero"].tobytes())
    kw = dict(ctlkw, sca_n=1, sca_mult=0, ip=ip, **(dict(cz=1.5, cx=900.0) if ip == 3 else {}))
    cols = [{k: v[..., 121 * i:121 * i + 121] for k, v in atm.items()} for i in range(5)]
    atms = [atm] if ip == 3 else cols
    ctl, inp = S.make_ctl(**kw), synth.batch_from(atms, np.zeros(n, np.int32), geom)
    m = api.Model(ctl)

    def run(max_seg):
        b = api.Batch(m, ctl, len(atms), len(inp["z"]), n, max_seg=max_seg)
        try:
            b.set_aero(layers)
            b.upload(inp)
            b.run()
            return b.download()
        finally:
            b.close()

    want, got = run(4096 * n), run(cap)
    assert want["nlos"].min() > cap
    for k in KEYS:
        np.testing.assert_array_equal(got[k], want[k])


def test_one_ray_above_the_default_capacity(workdir):
    """One pencil whose line of sight, with short steps and a layer, exceeds
    the 512 points a one-ray batch starts with."""
    from jscat import api
    ctl, inp, layers = _case(workdir, 2, 1, True, raydz=0.2, rayds=2.0)
    out = api.formod_batch(ctl, inp, aero=layers)
    assert out["nlos"][0] > 512
    assert np.all(out["rad"] > 0)


def _curtain(workdir, ip, n, mult=None):
    from jscat import synth, structs as S
    ctlkw, atm, geom = synth.curtain_case(workdir)
    geom = {k: v[:n] for k, v in geom.items()}
    kw, layers = dict(ctlkw, ip=ip), None
    if mult is not None:
        layers = S.AeroT.from_buffer_copy(np.load(os.path.join(GOLDEN, "aero_ice8.npz"))["aero"].tobytes())
        kw.update(sca_n=1, sca_mult=mult)
    atms = [{k: v[..., 121 * i:121 * i + 121] for k, v in atm.items()} for i in range(5)]
    return S.make_ctl(**kw), synth.batch_from(atms, np.zeros(n, np.int32), geom), layers


@pytest.mark.parametrize("ip,mult", [(1, None), (1, 0), (1, 1), (2, None), (2, 0)])
def test_run_after_a_failed_growth(workdir, ip, mult):
    """Each allocation of a run whose buffers have to grow fails in turn
    (an error code on the host, before any use of the memory): the call
    reports it, and the next one allocates again and gives the results."""
    from jscat import api, lib as L
    ctl, inp, layers = _curtain(workdir, ip, 3, mult)
    m, lib = api.Model(ctl), L.load()
    want = api.formod_batch(ctl, inp, model=m, aero=layers)
    failed = 0
    for k in range(1, 40):
        b = api.Batch(m, ctl, len(inp["atm_off"]) - 1, len(inp["z"]), 3, max_seg=1)
        try:
            if layers is not None:
                b.set_aero(layers)
            b.upload(inp)
            L.check(lib.jsc_batch_fail_alloc(b.h, k))
            try:
                b.run()
            except L.JscError as e:
                assert e.status == 10   # JSC_ERR_NOMEM
                failed += 1
            else:
                break
            b.run()
            got = b.download()
            for c in KEYS:
                np.testing.assert_array_equal(got[c], want[c])
        finally:
            b.close()
    assert failed == {(1, None): 6, (1, 0): 6, (1, 1): 12, (2, None): 4, (2, 0): 6}[ip, mult]


def test_layers_after_a_failed_allocation(workdir):
    """jsc_batch_set_aero with each of its allocations failing in turn: no
    run takes half of the layers, and the next call sets them."""
    from jscat import api, lib as L
    ctl, inp, layers = _case(workdir, 2, 5, True)
    m, lib = api.Model(ctl), L.load()
    want = api.formod_batch(ctl, inp, model=m, aero=layers)
    for before in (False, True):
        for k in range(3 if before else 1, 7):
            b = api.Batch(m, ctl, 2, len(inp["z"]), 5)
            try:
                if before:
                    b.set_aero(layers)
                L.check(lib.jsc_batch_fail_alloc(b.h, k - 2 if before else k))
                with pytest.raises(L.JscError) as e:
                    b.set_aero(layers)
                assert e.value.status == 10
                b.upload(inp)
                with pytest.raises(L.JscError) as e:
                    b.run()
                assert e.value.status == 1   # JSC_ERR_ARG: a run with layers needs them
                b.set_aero(layers)
                b.run()
                got = b.download()
                for c in KEYS:
                    np.testing.assert_array_equal(got[c], want[c])
            finally:
                b.close()
