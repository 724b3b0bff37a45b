"""A single-scattering batch between fixed-capacity and ordinary runs: each
kind has its own way to run the secondary and solar pencils, and neither may
take over what the other left."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

KEYS = ("rad", "tau", "nlos")


def _case(workdir, n):
    from jscat import synth, structs as S
    layers = S.AeroT.from_buffer_copy(np.load(os.path.join(GOLDEN, "aero_ice8.npz"))["aero"].tobytes())
    atm = synth.atmosphere(synth.CFG0_EMITTERS, np.random.default_rng(3))
    base = synth.write_tables(workdir, synth.CFG0_EMITTERS, synth.CFG0_NU, 20261203)
    ctl = S.make_ctl(synth.CFG0_EMITTERS, synth.CFG0_NU[:2], base, hydz=0.0, sca_n=1, sca_mult=1)
    geom = synth.limb_geometry(np.linspace(7.0, 10.5, n))
    geom["time"][:] = 43200.0
    return ctl, synth.batch_from([atm], np.zeros(n, np.int32), geom), layers


def _above(inp, rays):
    out = {k: np.array(v) for k, v in inp.items()}
    out["vpz"][rays] = 130.0
    return out


def _run(b, inp):
    b.upload(inp)
    b.run()
    return b.download()


def test_ordinary_runs_after_fixed_ones(workdir):
    """The last fixed run scatters at few points; the ordinary one after it
    at all of them, and the fixed one after that again."""
    from jscat import api, lib as L
    ctl, inp, layers = _case(workdir, 4)
    m, lib = api.Model(ctl), L.load()
    few = _above(inp, np.arange(4) > 0)
    want, wfew = (api.formod_batch(ctl, i, model=m, aero=layers) for i in (inp, few))
    b = api.Batch(m, ctl, 1, len(inp["z"]), 4)
    try:
        b.set_aero(layers)
        for _ in range(2):
            L.check(lib.jsc_batch_set_fixed_points(b.h, 400))
            L.check(lib.jsc_batch_set_fixed(b.h, 1))
            got = _run(b, few)
            for k in KEYS:
                np.testing.assert_array_equal(got[k], wfew[k])
            L.check(lib.jsc_batch_set_fixed(b.h, 0))
            got = _run(b, inp)
            for k in KEYS:
                np.testing.assert_array_equal(got[k], want[k])
    finally:
        b.close()
        m.close()


def test_scatter_points_of_a_fixed_batch(workdir):
    """jsc_batch_scatter_points on a batch in fixed-capacity mode, with fewer
    and with more points than a round of its runs holds: the sources of an
    ordinary batch, and the fixed runs go on."""
    from jscat import api, synth, lib as L
    ctl, inp, layers = _case(workdir, 2)
    m, lib = api.Model(ctl), L.load()
    few = _above(inp, [1])
    wfew = api.formod_batch(ctl, few, model=m, aero=layers)
    dp, ip = C.POINTER(C.c_double), C.POINTER(C.c_int)

    def sources(b, n):
        x = np.zeros((n, 3))
        x[:, 0] = synth.RE + 9.0 + 0.01 * np.arange(n)
        dx = np.tile([0.1, 1.0, 0.2], (n, 1))
        layer, sec, src = np.zeros(n, np.int32), np.full(n, 43200.0), np.zeros((n, ctl.nd))
        L.check(lib.jsc_batch_scatter_points(b.h, n, x.ctypes.data_as(dp), dx.ctypes.data_as(dp), layer.ctypes.data_as(ip),
                                             sec.ctypes.data_as(dp), None, src.ctypes.data_as(dp), None))
        return src

    b, plain = (api.Batch(m, ctl, 1, len(inp["z"]), 2) for _ in range(2))
    try:
        for c in (b, plain):
            c.set_aero(layers)
            c.upload(inp)
        L.check(lib.jsc_batch_set_fixed_points(b.h, 100))
        L.check(lib.jsc_batch_set_fixed(b.h, 1))
        for n in (3, 150):
            got = _run(b, few)
            for k in KEYS:
                np.testing.assert_array_equal(got[k], wfew[k])
            b.upload(inp)
            np.testing.assert_array_equal(sources(b, n), sources(plain, n))
        got = _run(b, few)
        for k in KEYS:
            np.testing.assert_array_equal(got[k], wfew[k])
    finally:
        b.close()
        plain.close()
        m.close()


def test_pencil_count_after_fixed_mode(workdir):
    """jsc_batch_set_nalpha drops what the fixed-capacity runs had prepared:
    the next one says so, until jsc_batch_set_fixed prepares it again."""
    from jscat import api, lib as L
    ctl, inp, layers = _case(workdir, 2)
    m, lib = api.Model(ctl), L.load()
    want = api.formod_batch(ctl, inp, model=m, aero=layers, nalpha=10)
    b = api.Batch(m, ctl, 1, len(inp["z"]), 2)
    try:
        b.set_aero(layers)
        L.check(lib.jsc_batch_set_fixed_points(b.h, 200))
        L.check(lib.jsc_batch_set_fixed(b.h, 1))
        b.set_nalpha(10)
        b.upload(inp)
        with pytest.raises(L.JscError) as e:
            b.run()
        assert "jsc_batch_set_fixed" in str(e.value)
        L.check(lib.jsc_batch_set_fixed(b.h, 1))
        got = _run(b, inp)
        for k in KEYS:
            np.testing.assert_array_equal(got[k], want[k])
    finally:
        b.close()
        m.close()


@pytest.mark.parametrize("change", ["layers", "pencils", "growth"])
def test_graph_of_another_state(workdir, change):
    """A launch of a graph whose batch has other layers, another number of
    pencils or other buffers since is refused on the host; a new capture runs
    with the new state."""
    import torch
    from jscat import api, lib as L
    ctl, inp, layers = _case(workdir, 2)
    if change != "pencils":
        ctl.sca_mult = 0
    m, lib = api.Model(ctl), L.load()
    few = _above(inp, [0, 1])
    pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()   # noqa: E731
    stream = torch.cuda.Stream()
    gb = api.GraphBatch(m, ctl, few if change == "growth" else inp, stream.cuda_stream, pin, aero=layers,
                        fixed_points=400, max_seg=16 if change == "growth" else 0)
    nalpha = None
    try:
        gb.launch()
        stream.synchronize()
        gb.status()
        if change == "layers":
            layers = type(layers).from_buffer_copy(bytes(layers))
            layers.trans[0] = 0.5
            gb.batch.set_aero(layers)
        elif change == "pencils":
            nalpha = 10
            gb.batch.set_nalpha(nalpha)
        else:
            L.check(lib.jsc_batch_set_fixed(gb.batch.h, 0))
            _run(gb.batch, inp)
        with pytest.raises(L.JscError) as e:
            gb.launch()
        assert e.value.status == 1 and "capture again" in str(e.value)   # JSC_ERR_ARG
        L.check(lib.jsc_batch_set_fixed(gb.batch.h, 1))
        bi, bo = gb._keep
        for k in gb._KEYS:
            gb.host[k][...] = inp[k]
        L.check(lib.jsc_batch_graph_capture(gb.batch.h, C.byref(bi), C.byref(bo), stream.cuda_stream))
        gb.launch()
        stream.synchronize()
        gb.status()
        want = api.formod_batch(ctl, inp, model=m, aero=layers, nalpha=nalpha)
        for k in KEYS:
            np.testing.assert_array_equal(gb.out[k], want[k])
    finally:
        gb.close()
        m.close()


def test_failed_preparation(workdir):
    """A larger point capacity whose allocations fail in turn: the call
    reports it and leaves an ordinary batch, not a fixed-capacity one without
    its buffers; the next call prepares it."""
    from jscat import api, lib as L
    ctl, inp, layers = _case(workdir, 2)
    m, lib = api.Model(ctl), L.load()
    want = api.formod_batch(ctl, inp, model=m, aero=layers)
    failed = 0
    for k in range(1, 20):
        b = api.Batch(m, ctl, 1, len(inp["z"]), 2)
        try:
            b.set_aero(layers)
            L.check(lib.jsc_batch_set_fixed_points(b.h, 50))
            L.check(lib.jsc_batch_set_fixed(b.h, 1))
            L.check(lib.jsc_batch_set_fixed_points(b.h, 1200))
            L.check(lib.jsc_batch_fail_alloc(b.h, k))
            st = lib.jsc_batch_set_fixed(b.h, 1)
            L.check(lib.jsc_batch_fail_alloc(b.h, 0))
            if st == 0:
                break
            assert st == 10   # JSC_ERR_NOMEM
            failed += 1
            for _ in range(2):   # as an ordinary batch, then prepared
                got = _run(b, inp)
                for c in KEYS:
                    np.testing.assert_array_equal(got[c], want[c])
                L.check(lib.jsc_batch_set_fixed(b.h, 1))
            got = _run(b, inp)
            for c in KEYS:
                np.testing.assert_array_equal(got[c], want[c])
        finally:
            b.close()
    assert failed == 3   # point records, their profiles, their sources
    m.close()
