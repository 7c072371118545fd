"""Optical depths that are not numbers: every table index they lead to stays
inside its table (the conversion of NaN to an integer is INT_MIN), and the columns
beside them are untouched.  Where the longwave's FP64 transfer gives numbers for
the spoilt columns, they are those of the general transfer, which clamps its
indices and runs where hlwb is asked for."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu

N, NLAY = 9, 40
BAD = [1, 4, 7]   # columns
CASES = [("aeraod", np.nan), ("aeraod", -np.nan), ("aeraod", np.inf), ("cld_od", np.nan), ("cld_od", -np.nan),
         ("cld_od", np.inf), ("cld_rwp", np.nan), ("cld_rwp", np.inf)]


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _spoil(prof, field, value):
    """Cloud in layers 14..16 of every column, `value` in layer 15 of the bad columns."""
    cf = np.zeros((NLAY, N))
    cf[14:17] = 0.7
    prof["cld_cf"] = cf
    for k in ("cld_lwp", "cld_rwp"):
        prof[k] = np.where(cf > 0, 5.0, 0.0)
    prof["cld_od"] = np.where(cf > 0, 2.0, 0.0)
    prof["cld_ssa"], prof["cld_asy"] = np.full((NLAY, N), 0.9), np.full((NLAY, N), 0.8)
    prof["aeraod"] = np.array(prof["aeraod"])
    clean = dict(prof)
    prof[field] = np.array(prof[field])
    prof[field][..., 15, BAD] = value
    return clean, prof


def _others_same(got, want):
    good = [c for c in range(N) if c not in BAD]
    for k, v in got.items():
        axis = 0 if k in ("topflx", "sfcflx", "fdncmp") else v.ndim - (2 if k == "flxprf" else 1)
        assert np.array_equal(v.take(good, axis), want[k].take(good, axis)), k


@pytest.mark.parametrize("field,value", CASES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_longwave(field, value, precision):
    torch = _cuda()
    assert lw.rlwinit(device=0)[0] == 0
    clean, prof = _spoil(synthetic.make_profiles(N, NLAY, seed=2), field, value)
    flags = dict(prof["flags"], ilwcliq=0 if field == "cld_od" else 1)
    got, want = (abi.alloc_outputs(N, NLAY, flxprf=True) for _ in range(2))
    for p, o in ((clean, want), (prof, got)):
        msg, err = lw.run_profile(dict(p, flags=flags), o, precision=precision)
        assert err == 0, msg
    torch.cuda.synchronize()
    _others_same(got, want)
    if precision == "fp64":
        ref = abi.alloc_outputs(N, NLAY, hlwb=True, flxprf=True)
        msg, err = lw.run_profile(dict(prof, flags=flags), ref)
        assert err == 0, msg
        for k in ("topflx", "sfcflx", "flxprf"):
            both = np.isfinite(got[k]) & np.isfinite(ref[k])
            np.testing.assert_allclose(got[k][both], ref[k][both], rtol=1e-10, atol=1e-9, err_msg=k)


@pytest.mark.parametrize("field,value", CASES)
@pytest.mark.parametrize("n", [N, 620])
def test_shortwave(field, value, n):
    """n = 620: the upward kernel with its table in shared memory (four columns per SM or more)."""
    torch = _cuda()
    sw.rswinit(device=0)
    clean, prof = _spoil(sw.add_sw_inputs(synthetic.make_profiles(N, NLAY, seed=2), seed=2), field, value)
    fl = dict(sw.DEFAULT_FLAGS, iswcliq=0 if field == "cld_od" else 1)
    got, want = (sw.alloc_outputs(n, NLAY, flxprf=True) for _ in range(2))
    reps = -(-n // N)
    for p, o in ((clean, want), (prof, got)):
        p = {k: np.ascontiguousarray(np.tile(v, (1,) * (v.ndim - 1) + (reps,))[..., :n])
             if isinstance(v, np.ndarray) and v.shape[-1] == N else v for k, v in p.items()}
        p.update(npts=n, cosz=np.full(n, 0.6), idxday=np.arange(1, n + 1, dtype=np.int32), sw_flags=fl)
        sw.rrtmg_sw_run(p, o)
    torch.cuda.synchronize()
    _others_same({k: v[..., :N] if v.shape[-1] == n else (v[:, :N] if k == "flxprf" else v[:N]) for k, v in got.items()},
                 {k: v[..., :N] if v.shape[-1] == n else (v[:, :N] if k == "flxprf" else v[:N]) for k, v in want.items()})
    full = np.arange(n) % N
    good = ~np.isin(full, BAD)
    assert np.array_equal(got["sfcflx"][good], want["sfcflx"][good])
