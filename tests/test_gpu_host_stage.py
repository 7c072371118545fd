"""Host-array calls either side of the pinned-staging limit (16 MiB of
arguments: about 270 longwave or 240 shortwave columns of 127 layers) give the
device-resident call's results bit for bit, and leave the columns beyond npts
of arrays with ldim > npts as they were."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("npts,nlay", [(1, 64), (31, 127), (400, 127)])
def test_lw_host_matches_device(npts, nlay):
    torch = _cuda()
    assert lw.rlwinit(device=0)[0] == 0
    prof = synthetic.make_profiles(npts, nlay, seed=9)
    host = abi.alloc_outputs(npts, nlay, hlw0=True, flxprf=True)
    msg, err = lw.run_profile(prof, host)
    assert err == 0, msg
    dev = abi.alloc_outputs(npts, nlay, hlw0=True, flxprf=True, like="cuda")
    msg, err = lw.run_profile(lw.to_device(prof), dev)
    assert err == 0, msg
    torch.cuda.synchronize()
    for k, v in dev.items():
        assert np.array_equal(host[k], v.cpu().numpy()), k


@pytest.mark.parametrize("npts,nlay", [(1, 64), (31, 127), (300, 127)])
def test_sw_host_matches_device(npts, nlay):
    torch = _cuda()
    sw.rswinit(device=0)
    prof = sw.add_sw_inputs(synthetic.make_profiles(npts, nlay, seed=9), seed=9, night_fraction=0.3, precip=True)
    if not len(prof["idxday"]):
        prof["cosz"][0], prof["idxday"] = 0.5, np.ones(1, np.int32)
    host = sw.alloc_outputs(npts, nlay, flxprf=True, hswb=True)
    sw.rrtmg_sw_run(prof, host)
    dprof = {k: torch.as_tensor(v).cuda() if isinstance(v, np.ndarray) else v for k, v in prof.items()}
    dev = sw.alloc_outputs(npts, nlay, flxprf=True, hswb=True, like=dprof["plyr"])
    torch.cuda.synchronize()
    sw.rrtmg_sw_run(dprof, dev, device_memory=True)
    for k, v in dev.items():
        assert np.array_equal(host[k], v.cpu().numpy()), k


def test_padding_columns_untouched():
    _cuda()
    assert lw.rlwinit(device=0)[0] == 0
    n, ld, nlay = 17, 23, 40
    prof = synthetic.make_profiles(ld, nlay, seed=4)
    full = abi.alloc_outputs(ld, nlay, hlw0=True, flxprf=True)
    msg, err = lw.run_profile(prof, full)
    assert err == 0, msg
    out = abi.alloc_outputs(ld, nlay, hlw0=True, flxprf=True)
    part = dict(prof, npts=n, flags=dict(prof["flags"], ldim=ld))
    msg, err = lw.run_profile(part, out)
    assert err == 0, msg
    for k in ("hlwc", "hlw0", "cldtau"):
        assert np.array_equal(out[k][:, :n], full[k][:, :n]) and np.isnan(out[k][:, n:]).all(), k
    assert np.array_equal(out["flxprf"][:, :n], full["flxprf"][:, :n]) and np.isnan(out["flxprf"][:, n:]).all()
    for k in ("topflx", "sfcflx"):
        assert np.array_equal(out[k][:n], full[k][:n]) and np.isnan(out[k][n:]).all(), k
