"""The transfer behind the learned gas optics forms a column's band fields
with the bands along half warps and the layers in ten ranges: layer counts at
the edges of those ranges (empty and short ones), every ice option, the
diagnostic cloud and both vertical orders.  Doubled CO2 sends every layer to
plain FP32 taumol, so the FP32 path is the reference: the cloud optical depth
is formed in FP64 by both (the sums may contract differently, 1e-14), and a
flux differs by the FP16 copies of optical depths, fractions and transmittance
records, three roundings of 2^-11 that no g-point exceeds."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lw():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ccpp_physics_b200 import rrtmg_lw, surrogate
    rc, msg = rrtmg_lw.rlwinit(device=0)
    assert rc == 0, msg
    surrogate.load()
    return rrtmg_lw


@pytest.mark.parametrize("nlay,flags,cloudy,flip", [
    (1, {}, True, False), (2, dict(ilwcice=1), True, False), (9, {}, True, False), (10, dict(ilwcice=2), True, True),
    (11, dict(ilwcice=3), True, False), (20, {}, False, False), (21, dict(iovr=3), True, True),
    (91, dict(ilwcice=1), True, False), (126, dict(ilwcice=2), True, False), (127, dict(iovr=4), True, True),
])
def test_band_fields_match_the_fp32_path(lw, nlay, flags, cloudy, flip):
    n = 37
    prof = synthetic.make_profiles(n, nlay, seed=60 + nlay, cloudy=cloudy)
    prof["gasvmr_co2"] = prof["gasvmr_co2"] * 2.0
    flags = dict(flags)
    if flip:
        prof = {k: (np.ascontiguousarray(v[::-1]) if isinstance(v, np.ndarray) and v.ndim == 2 else v)
                for k, v in prof.items()}
        for k in ("aeraod", "aerssa"):
            prof[k] = np.ascontiguousarray(prof[k][:, ::-1])
        flags["top_at_1"] = 1
    got, want = (abi.alloc_outputs(n, nlay, hlw0=True) for _ in range(2))
    for out, precision in ((got, "surrogate"), (want, "fp32")):
        msg, err = lw.run_profile(prof, out, precision=precision, flags=flags)
        assert err == 0, msg
    np.testing.assert_allclose(got["cldtau"], want["cldtau"], rtol=1e-14, atol=0)
    for k in ("topflx", "sfcflx"):
        assert np.max(np.abs(got[k] - want[k]) / np.maximum(np.abs(want[k]), 1e-3)) <= 3 * 2.0 ** -11, k
