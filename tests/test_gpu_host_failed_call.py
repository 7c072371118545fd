"""A host-array call that fails behind its staging (no device memory left for its
scratch) reports it, and the next call, on another stream, gives the right
results: the staging buffer is at rest when the failed call returns."""
import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, synthetic

pytestmark = pytest.mark.gpu


def test_call_after_a_failed_one():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, nlay = 180, 127   # 11.5 MiB of arguments: staged
    profs = [synthetic.make_profiles(n, nlay, seed=s) for s in (5, 6)]
    outs = [abi.alloc_outputs(n, nlay) for _ in range(4)]
    assert lw.rlwinit(device=0)[0] == 0
    assert lw.run_profile(profs[1], outs[0])[1] == 0
    lw.lib().rrtmg_lw_gpu_finalize()   # drops the workspaces
    assert lw.rlwinit(device=0)[0] == 0
    torch.cuda.empty_cache()
    other = torch.cuda.Stream()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - (40 << 20), dtype=torch.uint8, device="cuda")   # the scratch alone would take 76 MB
    try:
        msg, err = lw.run_profile(profs[0], outs[1])
    finally:
        del taken
        torch.cuda.empty_cache()
    assert err == 1 and "scratch" in msg, (err, msg)
    msg, err = lw.run_profile(profs[1], outs[2], stream=other.cuda_stream)
    assert err == 0, msg
    for k, v in outs[0].items():
        assert np.array_equal(outs[2][k], v), k
    assert lw.run_profile(profs[0], outs[3])[1] == 0
