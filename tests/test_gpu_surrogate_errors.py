"""Errors of the surrogate's training: what the caller reads, and the call after."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_training_reports_its_own_error():
    """A copy that the runtime refuses (the legacy stream while another one
    is being captured): the message is that of the call, not one left from an
    earlier call, and the next training is not disturbed."""
    from cuda.bindings import runtime as rt
    from jscat import api, lib as L
    rng = np.random.default_rng(1)
    x = rng.normal(size=(64, 8)).astype(np.float32)
    src = np.exp(rng.normal(size=(64, 3)) - 20.0)
    want = api.Surrogate(3, seed=3)
    want.train(x, src, epochs=1, batch=32)
    sur = api.Surrogate(3, seed=3)
    with pytest.raises(L.JscError) as e:
        sur.train(x, src, epochs=1, batch=1)
    assert "invalid arguments" in str(e.value)
    err, stream = rt.cudaStreamCreate()
    assert err == 0
    assert rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0] == 0
    try:
        with pytest.raises(L.JscError) as e:
            sur.train(x, src, epochs=1, batch=32)
        assert "invalid arguments" not in str(e.value)
        assert "captur" in str(e.value)
    finally:
        rt.cudaStreamEndCapture(stream)
        rt.cudaGetLastError()
        rt.cudaStreamDestroy(stream)
    sur.train(x, src, epochs=1, batch=32)
    np.testing.assert_array_equal(sur.get_params(), want.get_params())
    sur.close()
    want.close()
