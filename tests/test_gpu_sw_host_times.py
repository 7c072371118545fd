"""kernel_ms of a shortwave call on host arrays large enough to travel in
chunks of 4,096 columns covers all of them, a first chunk without a daytime
point among them."""
import numpy as np
import pytest

from ccpp_physics_b200 import rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu


def _profile(n, nlay):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sw.rswinit(device=0)
    return sw.add_sw_inputs(synthetic.make_profiles(n, nlay, seed=9), seed=9, precip=True)


def test_host_times_cover_all_chunks():
    torch = pytest.importorskip("torch")
    n, nlay = 12288, 40
    prof = _profile(n, nlay)
    dprof = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v
             for k, v in prof.items()}
    out, dout = sw.alloc_outputs(n, nlay), sw.alloc_outputs(n, nlay, like=dprof["tlyr"])
    host, dev = [], []
    for _ in range(3):
        km = []
        sw.rrtmg_sw_run(prof, out, kernel_ms=km)
        host.append(km)
        km = []
        sw.rrtmg_sw_run(dprof, dout, device_memory=True, kernel_ms=km)
        dev.append(km)
    # the same columns by the same kernels: one chunk of three would read a third
    for h, d in zip(np.min(host, 0), np.min(dev, 0)):
        assert 0.6 * d < h < 2.0 * d, (host, dev)


def test_night_in_front():
    n, nlay = 8300, 40
    prof = _profile(n, nlay)
    idx = np.asarray(prof["idxday"])
    prof["idxday"] = idx[idx > 4096]
    km = []
    sw.rrtmg_sw_run(prof, sw.alloc_outputs(n, nlay), kernel_ms=km)
    assert all(t > 0 for t in km), km
