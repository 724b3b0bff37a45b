"""Launch variants: what the autotuner times, and the default ones with layers
and scattering."""
import numpy as np
import pytest

from test_gpu_parity import shape_case  # noqa: F401  (the fixture)
from test_gpu_parity import test_every_launch_variant as _against_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng", [2, 17])
def test_autotune_times_whole_variants(workdir, ng):
    """The tuner launches for each variant what a run with it launches: its
    order of the rays, its continuum pass, its transfer.  Counted: the
    launches of a run less those before them (a run of variant 0 has one
    kernel after them)."""
    from jscat import api, synth, structs as S
    emitters = (synth.CFG1_EMITTERS + ["X%02d" % i for i in range(25)])[:ng]
    ctlkw, atms, ray_atm, geom = synth.batched_case(workdir, n_rays=40, rays_per_atm=20, seed=7, emitters=emitters,
                                                    nus=synth.CFG1_NU[5::40])
    ctl = S.make_ctl(**ctlkw)
    inp = synth.batch_from(atms, ray_atm, geom)
    m = api.Model(ctl)
    b = api.Batch(m, ctl, len(atms), len(inp["z"]), 40)

    def launches(f):
        n = api.launch_count()
        f()
        return api.launch_count() - n

    try:
        b.upload(inp)
        b.run()
        run = {}
        for v in range(-1, 23):
            b.set_variant(v)
            run[v] = launches(b.run)
        before = run[0] - 1
        assert run[9] == before + 2 and run[21] == run[22] > run[9]
        b.set_variant(-1)
        assert launches(b.autotune) == run[-1] + sum(run[v] - before for v in range(23))
    finally:
        b.close()
        m.close()


@pytest.mark.parametrize("layer,mult,n,nd", [("aero_ice8", 0, 70, 8), ("aero_sulfate16", 0, 33, 5), ("aero_ice8", 1, 3, 3),
                                             ("aero_sulfate16", 1, 2, 16), ("aero_ice8", 2, 1, 2)])
def test_gas_variants_with_layers(workdir, layer, mult, n, nd):
    """Four lanes and one lane per ray (21, 22) against the
    thread-per-channel kernel (6) through aerosol and cloud layers and with
    scattering sources, whose child batches run the same variant: the same
    operations in the same order, so the same bits."""
    import os
    from conftest import GOLDEN
    from jscat import api, synth, structs as S
    g = np.load(os.path.join(GOLDEN, layer + ".npz"))
    aero = S.AeroT.from_buffer_copy(g["aero"].tobytes())
    nus = [float(v) for v in g["nus"]]
    rng = np.random.default_rng(n)
    atms = [synth.atmosphere(synth.CFG0_EMITTERS, rng, t_sigma=3.0) for _ in range(2)]
    base = synth.write_tables(workdir, synth.CFG0_EMITTERS, nus, 20261203)
    ctl = S.make_ctl(synth.CFG0_EMITTERS, nus[:nd], base, hydz=0.0, sca_n=1, sca_mult=mult)
    a, b = synth.limb_geometry(rng.uniform(6.0, 30.0, n)), synth.nadir_geometry(rng.uniform(0.0, 60.0, n))
    geom = {k: np.where(np.arange(n) % 3 == 2, b[k], a[k]) for k in a}
    geom["time"] = np.linspace(20000.0, 43200.0, n)
    inp = synth.batch_from(atms, np.arange(n) % 2, geom)
    m = api.Model(ctl)
    try:
        want, four, one = (api.formod_batch(ctl, inp, model=m, aero=aero, digest=True, variant=v, nalpha=10)
                           for v in (6, 21, 22))
    finally:
        m.close()
    assert np.all(np.isfinite(want["rad"])) and np.any(want["tau"] < 0.9)
    for k in want:
        np.testing.assert_array_equal(four[k], want[k])
        np.testing.assert_array_equal(one[k], want[k])


@pytest.mark.parametrize("variant", [21, 22])
def test_gas_variants_on_reference_shapes(shape_case, variant):   # noqa: F811
    """The shapes on which the parity tests run the variants 0-20: counts and
    table indices of the reference, radiances within its bounds."""
    _against_reference(shape_case, variant)
