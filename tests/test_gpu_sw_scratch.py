"""Shortwave calls where memory is short: the scratch of a call (up to 1.55 MB per
column of 127 layers) shrinks to what the device has left, or to
RRTMG_SW_GPU_SCRATCH_MB, and the results stay the same."""
import numpy as np
import pytest

from ccpp_physics_b200 import rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu

N, NLAY = 3000, 127


@pytest.fixture(scope="module")
def case():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sw.rswinit(device=0)
    prof = sw.add_sw_inputs(synthetic.make_profiles(N, NLAY, seed=9), seed=9, precip=True)
    prof = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v
            for k, v in prof.items()}
    want = sw.alloc_outputs(N, NLAY, flxprf=True, like=prof["tlyr"])
    sw.rrtmg_sw_run(prof, want, device_memory=True)
    return torch, prof, want


def _same(torch, prof, want, run):
    got = sw.alloc_outputs(N, NLAY, flxprf=True, like=prof["tlyr"])
    run(got)
    torch.cuda.synchronize()
    for k, v in want.items():
        assert torch.equal(got[k], v), k


@pytest.fixture
def fresh():
    """A library without workspaces, before and after."""
    sw.lib().rrtmg_sw_gpu_finalize()
    sw.rswinit(device=0)
    yield
    sw.lib().rrtmg_sw_gpu_finalize()
    sw.rswinit(device=0)


def test_less_memory_than_asked_for(case, fresh):
    torch, prof, want = case
    torch.cuda.empty_cache()
    got = sw.alloc_outputs(N, NLAY, flxprf=True, like=prof["tlyr"])
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - (3 << 30), dtype=torch.uint8, device="cuda")   # 3 GiB left; 5.8 GB would be asked for
    try:
        sw.rrtmg_sw_run(prof, got, device_memory=True)
        sw.rrtmg_sw_run_blocks([prof], [got])
        torch.cuda.synchronize()
    finally:
        del taken
        torch.cuda.empty_cache()
    for k, v in want.items():
        assert torch.equal(got[k], v), k


@pytest.mark.parametrize("mb", ["1", "700", "2500"])
def test_budget(case, fresh, monkeypatch, mb):
    torch, prof, want = case
    monkeypatch.setenv("RRTMG_SW_GPU_SCRATCH_MB", mb)
    if mb == "1":   # a column at a time: a few columns are enough
        prof = dict(prof, idxday=prof["idxday"][:3])
        got = sw.alloc_outputs(N, NLAY, flxprf=True, like=prof["tlyr"])
        sw.rrtmg_sw_run(prof, got, device_memory=True)
        torch.cuda.synchronize()
        i = (prof["idxday"] - 1).long()
        assert torch.equal(got["flxprf"][:, i], want["flxprf"][:, i])
        return
    _same(torch, prof, want, lambda got: sw.rrtmg_sw_run(prof, got, device_memory=True))
