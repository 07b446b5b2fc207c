"""Uploaded FP64 arrays arrive rounded to FP32, on the host or on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 128 rows: the largest arrays rounded on the host; 256: on the device, the
# air flow's N + 1 values in two pieces.  Rounding is IEEE's, so exact.
@pytest.mark.parametrize("nT", [8, 128, 256])
@pytest.mark.parametrize("name", ["u_theta", "u_phi", "eta_delta", "uair", "vair", "eta"])
def test_uploads_round_to_nearest(gpulib, nT, name):
    from soapbubble_gb300.bubble import GpuBubble, make_params
    rng = np.random.Generator(np.random.PCG64(nT))
    with GpuBubble(make_params(nT, 0.005)) as gb:
        shape = gb.shape(name)
        a = rng.normal(size=shape) * 10.0 ** rng.integers(-30, 30, size=shape)
        flat = a.reshape(-1)
        flat[:8] = [np.nan, np.inf, -np.inf, -0.0, 1e-45, 1e300, 1 + 2.0 ** -24, 1 + 3 * 2.0 ** -24]
        flat[-1] = 1.0 / 3.0
        with np.errstate(over="ignore"):
            want = a.astype(np.float32)
        other = gb.download("gamma")
        gb.upload(name, a)
        got = gb.download(name).astype(np.float32)
        np.testing.assert_array_equal(got.view(np.uint32)[~np.isnan(want)], want.view(np.uint32)[~np.isnan(want)])
        assert np.isnan(got[np.isnan(want)]).all()
        np.testing.assert_array_equal(gb.download("gamma"), other)
