"""The FP64 longwave transfer (a thread per g-point, four layers at a time) at
the edges of its loops: layer counts around the four-layer blocks, the 32-layer
cloud-flag words and the supported maximum, both vertical orders, clear and
cloudy columns; and the gas optics' pairs of g-points against the same oracle."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,nlay,flags,cloudy", [
    (1, 1, {}, True), (2, 2, {}, True), (3, 3, dict(iovr=3), True), (5, 4, {}, True), (3, 5, {}, False),
    (7, 31, dict(iovr=4), True), (4, 32, {}, True), (6, 33, dict(iovr=0), True), (9, 61, dict(isubclw=1), True),
    (2, 127, dict(iovr=2), True), (3, 128, {}, True), (2, 255, {}, True),
])
def test_transfer_matches_oracle(npts, nlay, flags, cloudy):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import oracle
    rc, msg = lw.rlwinit(device=0)
    assert rc == 0, msg
    rc, msg = oracle.rlwinit()
    assert rc == 0, msg
    prof = synthetic.make_profiles(npts, nlay, seed=300 + nlay, cloudy=cloudy)
    rng = np.random.default_rng(nlay)
    prof["aeraod"] = rng.uniform(0.0, 0.05, prof["aeraod"].shape)
    prof["aerssa"] = rng.uniform(0.2, 0.9, prof["aerssa"].shape)
    rc, msg, ref = oracle.rrtmg_lw_run(prof, flags=flags, hlw0=True, flxprf=True)
    assert rc == 0, msg
    out = abi.alloc_outputs(npts, nlay, hlw0=True, flxprf=True)
    msg, err = lw.run_profile(prof, out, flags=flags)
    assert err == 0, msg
    # the bars of tests/test_gpu_parity.py: the g-point sums run in another order
    for k in ("topflx", "sfcflx", "flxprf"):
        assert np.max(np.abs(out[k] - ref[k]) / np.maximum(np.abs(ref[k]), 1e-300)) <= 1e-10, k
    for k in ("hlwc", "hlw0"):
        assert np.max(np.abs(out[k] - ref[k]) / np.maximum(np.abs(ref[k]), 1.0)) <= 1e-9, k
