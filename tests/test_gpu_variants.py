"""Launch variants: what the autotuner times, and the default ones with layers
and scattering."""
import numpy as np
import pytest

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
