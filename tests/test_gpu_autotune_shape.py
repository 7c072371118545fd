"""The autotuner only chooses between transfer CTAs where the kernel has the
choice: FP64 without hlwb runs a CTA per column whatever rt_warps says, and the
recorded shape, which a later hlwb call takes, keeps the default."""
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw, synthetic

pytestmark = pytest.mark.gpu


def test_rt_warps_stays_at_its_default():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert rrtmg_lw.rlwinit(device=0)[0] == 0
    n, nlay = 300, 40
    prof = synthetic.make_profiles(n, nlay, seed=3, device="cuda")
    try:
        for _ in range(8):   # equal candidates are told apart by noise: once is not enough
            best, _ = rrtmg_lw.autotune(prof, abi.alloc_outputs(n, nlay, like="cuda"), [n], precision="fp64")
            assert best["rt_warps"] == 4
        out = abi.alloc_outputs(n, nlay, hlwb=True, like="cuda")
        best, _ = rrtmg_lw.autotune(prof, out, [n], precision="fp64")
        assert best["rt_warps"] in (1, 2, 4)
    finally:
        rrtmg_lw.set_tuning(nlay, "fp64", None)
