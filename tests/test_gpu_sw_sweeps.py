"""The shortwave transfer kernels at the edges of their loops and of their
launch rule: layer counts around the four-layer blocks of the optical depths,
the two-layer record pipeline of the way down and the 32-layer cloud-flag
words; column counts either side of the first whole wave of the upward kernel
(4 x 148 columns on B200), with and without the band fluxes."""
import numpy as np
import pytest

from ccpp_physics_b200 import rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,nlay,flags,hswb", [
    (1, 1, {}, True), (2, 2, {}, False), (3, 3, dict(iovr=3), True), (5, 4, dict(isubcsw=0), True),
    (7, 5, {}, False), (9, 31, dict(top_at_1=1), False), (11, 33, dict(isubcsw=0, top_at_1=1), False),
    (6, 65, {}, True), (591, 33, {}, False), (592, 32, dict(isubcsw=0), False), (595, 34, dict(iovr=3), True),
    (681, 5, {}, True),
])
def test_sweeps_match_oracle(npts, nlay, flags, hswb):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import oracle_sw
    sw.rswinit(device=0)
    rc, msg = oracle_sw.rswinit()
    assert rc == 0, msg
    prof = sw.add_sw_inputs(synthetic.make_profiles(npts, nlay, seed=100 + nlay), seed=100 + nlay, precip=True)
    ref = sw.alloc_outputs(npts, nlay, hswb=hswb, flxprf=True)
    rc, msg = oracle_sw.run(prof, ref, flags=flags)
    assert rc == 0, msg
    out = sw.alloc_outputs(npts, nlay, hswb=hswb, flxprf=True)
    sw.rrtmg_sw_run(prof, out, flags=flags)
    # the bars of tests/test_gpu_sw.py: fluxes differ by the order of the
    # g-point sums, heating rates by that over the layer thickness
    for k in ("topflx", "sfcflx", "fdncmp", "flxprf"):
        assert np.max(np.abs(out[k] - ref[k]) / np.maximum(np.abs(ref[k]), 1e-300)) <= 1e-10, k
    for k in ("hswc", "hsw0", "hswb"):
        if k in out:
            assert np.max(np.abs(out[k] - ref[k]) / np.maximum(np.abs(ref[k]), 1.0)) <= 1e-9, k
    assert np.array_equal(out["cldtau"], ref["cldtau"])
