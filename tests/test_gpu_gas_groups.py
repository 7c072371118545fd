"""The gas optics split a column's segments into one, two, four or eight band
groups by the size of the call; the split changes no bit: the first columns of
calls at each side of the rule's lines equal calls of a few columns, in FP64
and FP32."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,nlay", [(110, 64), (112, 64), (222, 61), (223, 61), (448, 33), (900, 33), (1800, 33),
                                       (600, 127)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_results_do_not_depend_on_the_band_groups(npts, nlay, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rc, msg = lw.rlwinit(device=0)
    assert rc == 0, msg

    def run(n):
        prof = synthetic.make_profiles(n, nlay, seed=77)
        out = abi.alloc_outputs(n, nlay, hlw0=True)
        msg, err = lw.run_profile(prof, out, precision=precision)
        assert err == 0, msg
        return out
    few, many = run(5), run(npts)
    for k in ("hlwc", "hlw0", "cldtau"):
        assert np.array_equal(few[k], many[k][:, :5]), k
    for k in ("topflx", "sfcflx"):
        assert np.array_equal(few[k], many[k][:5]), k
