"""Host arrays with ldim > npts: the columns beyond npts are the caller's and
stay as they were, whichever way the call's size takes the arrays to the
device: one pinned buffer (up to 12 MiB of arguments), a copy per array, or
chunks of 4,096 columns (from 8,192 columns on)."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu

# (columns, ldim, layers): staged, per array, pipelined
SIZES = [(17, 23, 40), (400, 431, 127), (8200, 8209, 12)]


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _check(part, full, n):
    for k, v in part.items():
        axis = 0 if k in ("topflx", "sfcflx", "fdncmp") else v.ndim - (2 if k == "flxprf" else 1)
        got, want = np.moveaxis(v, axis, 0), np.moveaxis(full[k], axis, 0)
        assert np.array_equal(got[:n], want[:n]), k
        assert np.isnan(got[n:]).all(), k


@pytest.mark.parametrize("n,ld,nlay", SIZES)
def test_longwave(n, ld, nlay):
    _cuda()
    assert lw.rlwinit(device=0)[0] == 0
    prof = synthetic.make_profiles(ld, nlay, seed=4)
    new = lambda: abi.alloc_outputs(ld, nlay, hlw0=True, hlwb=True, flxprf=True)  # noqa: E731
    full, part = new(), new()
    for v in part.values():
        v.fill(np.nan)
    msg, err = lw.run_profile(prof, full)
    assert err == 0, msg
    msg, err = lw.run_profile(dict(prof, npts=n, flags=dict(prof["flags"], ldim=ld)), part)
    assert err == 0, msg
    _check(part, full, n)


def test_longwave_missing_arguments():
    """cldtau is zeroed (npts columns of it) when the optional cloud arguments are missing."""
    _cuda()
    assert lw.rlwinit(device=0)[0] == 0
    n, ld, nlay = 17, 23, 40
    prof = {k: v for k, v in synthetic.make_profiles(ld, nlay, seed=4).items() if not k.startswith("cld_")
            or k == "cld_cf"}
    out = abi.alloc_outputs(ld, nlay)
    for v in out.values():
        v.fill(np.nan)
    _, err = lw.run_profile(dict(prof, npts=n, flags=dict(prof["flags"], ldim=ld)), out)
    assert err == 1
    assert (out["cldtau"][:, :n] == 0).all() and np.isnan(out["cldtau"][:, n:]).all()


@pytest.mark.parametrize("n,ld,nlay", SIZES)
def test_shortwave(n, ld, nlay):
    _cuda()
    sw.rswinit(device=0)
    prof = sw.add_sw_inputs(synthetic.make_profiles(ld, nlay, seed=4), seed=4, night_fraction=0.3, precip=True)
    new = lambda: sw.alloc_outputs(ld, nlay, hswb=True, flxprf=True)  # noqa: E731
    full, part = new(), new()
    for v in part.values():
        v.fill(np.nan)
    sw.rrtmg_sw_run(prof, full)
    idx = prof["idxday"]
    sw.rrtmg_sw_run(dict(prof, npts=n, idxday=idx[idx <= n]), part, ldim=ld)
    _check(part, full, n)
