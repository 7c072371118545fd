"""The FP64 helpers of the transfer kernels by themselves (csrc/fp64_util.cuh),
against IEEE division and square root.

pade_index (behind finite_od, as its callers have it) has to equal int(z / (bpade + z) * 10000 + 0.5) everywhere: on a
dense logarithmic grid, within 64 units in the last place of each of the 10,000
ties, and at the ends of the range.  The quotient and the root come from an
estimate good to 2^-20, two Newton steps (error below 2^-80 before the last
rounding) and a residual step, so they may miss the nearest value only where the
exact one lies within a rounding error of the estimate of a midpoint: at most
one unit in the last place, and seldom.  The reciprocal without that step is
likewise within one unit."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "ccpp_physics_b200", "csrc")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    so = str(tmp_path_factory.mktemp("probe") / "fp64_util_probe.so")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", "-o", so, os.path.join(HERE, "fp64_util_probe.cu")], check=True)
    lib = C.CDLL(so)
    lib.probe.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong] + [C.c_void_p] * 4

    def run(a, b, what):
        a, b = (torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda() for x in (a, b))
        out = torch.zeros(a.numel(), dtype=torch.int32 if what == "index" else torch.float64, device="cuda")
        ptr = [out.data_ptr() if w == what else None for w in ("div", "rec", "root", "index")]
        torch.cuda.synchronize()
        assert lib.probe(a.data_ptr(), b.data_ptr(), a.numel(), *ptr) == 0
        return out.cpu().numpy()
    return run


def _index(z):
    bpade = 1.0 / 0.278
    with np.errstate(over="ignore"):
        return (z / (bpade + z) * 10000 + 0.5).astype(np.int64)


def _ulps(got, want):
    """Distance in representable values (both positive and finite)."""
    return np.abs(got.view(np.int64) - want.view(np.int64))


def _operands(lo, hi, n, seed):
    rng = np.random.default_rng(seed)
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    # mantissas next to the powers of two and to one half
    m = np.array([1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5, np.nextafter(1.5, 1.0)])
    e = 2.0 ** np.arange(np.ceil(np.log2(lo)), np.floor(np.log2(hi)))
    return np.concatenate([x, np.outer(m, e).ravel()])


def test_index_grid(probe):
    z = np.exp(np.linspace(np.log(1e-9), np.log(1e9), 8_000_001))
    assert np.array_equal(probe(z, z, "index"), _index(z))


def test_index_ties(probe):
    q = (np.arange(10000) + 0.5) / 10000.0
    z = q / (1.0 - q) / 0.278
    z = (z.view(np.int64)[:, None] + np.arange(-64, 65)).view(np.float64).ravel()
    assert np.array_equal(probe(z, z, "index"), _index(z))


def test_index_ends(probe):
    z = np.concatenate([10.0 ** np.arange(-307, 309), 2.0 ** np.arange(-1022.0, 1024.0),
                        [5e-324, 1.7976931348623157e308]])
    assert np.array_equal(probe(z, z, "index"), _index(z))


def test_quotient(probe):
    a = _operands(1e-30, 1e30, 4_000_000, 1)
    b = np.random.default_rng(2).permutation(_operands(1e-30, 1e30, 4_000_000, 3))
    u = _ulps(probe(a, b, "div"), a / b)
    assert u.max() <= 1 and (u != 0).mean() < 1e-4, (u.max(), (u != 0).mean())
    assert np.all(probe(np.zeros(4), np.array([1e-12, 1.0, 3.0, 1e12]), "div") == 0.0)


def test_reciprocal(probe):
    b = _operands(1e-30, 1e30, 4_000_000, 4)
    u = _ulps(probe(b, b, "rec"), 1.0 / b)
    assert u.max() <= 1, u.max()


def test_root(probe):
    b = _operands(1e-30, 1e30, 4_000_000, 5)
    u = _ulps(probe(b, b, "root"), np.sqrt(b))
    assert u.max() <= 1 and (u != 0).mean() < 1e-4, (u.max(), (u != 0).mean())


def _profiles(clouds):
    """Four columns, three with an optical depth beyond 2^1022 in a layer: of
    aerosol, or of cloud (given as optical depths)."""
    from ccpp_physics_b200 import rrtmg_sw as sw, synthetic
    n, nlay = 4, 40
    lwp = synthetic.make_profiles(n, nlay, seed=2)
    swp = sw.add_sw_inputs(synthetic.make_profiles(n, nlay, seed=2), seed=2)
    swp["cosz"], swp["idxday"] = np.full(n, 0.9), np.arange(1, n + 1, dtype=np.int32)
    lwp["aerssa"] = np.zeros_like(np.array(lwp["aeraod"]))
    if not clouds:
        for p in (lwp, swp):
            p["aeraod"] = np.array(p["aeraod"])
            p["aeraod"][:, 15, 1:] = 6e307
        return lwp, swp
    cf = np.zeros((nlay, n))
    cf[14:17] = 1.0
    od = np.where(cf > 0, 2.0, 0.0)
    od[15, 1:] = 6e307
    for p in (lwp, swp):
        p["cld_cf"], p["cld_od"] = cf, od
        p["cld_ssa"], p["cld_asy"] = np.full((nlay, n), 0.9), np.full((nlay, n), 0.8)
    lwp["flags"] = dict(lwp["flags"], ilwcliq=0)
    swp["sw_flags"] = dict(sw.DEFAULT_FLAGS, iswcliq=0)
    return lwp, swp


@pytest.mark.parametrize("clouds", [False, True])
def test_optical_depth_at_the_end_of_the_range(oracle_lib, clouds):
    """Such a layer is opaque in both schemes."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ccpp_physics_b200 import abi, rrtmg_lw as lw, rrtmg_sw as sw
    from oracle import oracle_sw
    lwp, swp = _profiles(clouds)
    n, nlay = lwp["npts"], lwp["nlay"]
    assert lw.rlwinit(device=0)[0] == 0
    got = abi.alloc_outputs(n, nlay, flxprf=True)
    msg, err = lw.run_profile(lwp, got)
    assert err == 0, msg
    err, msg, want = oracle_lib.rrtmg_lw_run(lwp, flxprf=True)
    assert err == 0, msg
    for k in ("topflx", "sfcflx", "flxprf", "cldtau"):
        np.testing.assert_allclose(got[k], want[k], rtol=1e-12, atol=1e-10, err_msg=k)
    sw.rswinit(device=0)
    assert oracle_sw.rswinit()[0] == 0
    got, want = sw.alloc_outputs(n, nlay, flxprf=True), sw.alloc_outputs(n, nlay, flxprf=True)
    sw.rrtmg_sw_run(swp, got)
    assert oracle_sw.run(swp, want)[0] == 0
    for k in ("topflx", "sfcflx", "flxprf", "cldtau"):
        np.testing.assert_allclose(got[k], want[k], rtol=1e-12, atol=1e-10, err_msg=k)
