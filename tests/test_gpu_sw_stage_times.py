"""kernel_ms of a shortwave call covers every chunk of the scratch budget: 5,000
columns of 200 layers take two, so the stages add up to nearly the whole of the
call, where one chunk's are about half."""
import numpy as np
import pytest

from ccpp_physics_b200 import rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu


def test_stage_times_cover_all_chunks():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sw.rswinit(device=0)
    n, nlay = 5000, 200
    prof = sw.add_sw_inputs(synthetic.make_profiles(n, nlay, seed=9), seed=9, precip=True)
    prof = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v
            for k, v in prof.items()}
    out = sw.alloc_outputs(n, nlay, like=prof["tlyr"])
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 0.0
    for _ in range(3):
        km = []
        torch.cuda.synchronize()
        ev[0].record()
        sw.rrtmg_sw_run(prof, out, device_memory=True, kernel_ms=km)
        ev[1].record()
        torch.cuda.synchronize()
        best = max(best, sum(km) / ev[0].elapsed_time(ev[1]))
    assert 0.75 <= best <= 1.01, best
