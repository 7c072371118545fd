"""The decorrelation-length and exponential overlaps (iovr 3..5) of both
generators, flag for flag against the oracles: layer counts around the
32-layer words, columns whose clouds end low, reach the top or are missing
(the longwave walk stops above the last cloudy layer), thresholds that lie on
draws, and a draw of exactly 1 above the clouds."""
import ctypes as C

import numpy as np
import pytest

from ccpp_physics_b200 import rrtmg_lw as lw, rrtmg_sw as sw

pytestmark = pytest.mark.gpu
OVERLAPS = (3, 4, 5)


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    rc, msg = lw.rlwinit(device=0)
    assert rc == 0, msg
    return t


@pytest.fixture(scope="module")
def orc():
    from oracle import oracle
    rc, msg = oracle.rlwinit()
    assert rc == 0, msg
    return oracle


def _columns(rng, nlay, n):
    """Cloud fractions: column 0 clear, 1 cloudy at the surface, 2 at the top,
    3 overcast throughout, 4 in the lower third, the rest scattered."""
    cldf = rng.random((nlay, n)) * (rng.random((nlay, n)) < 0.3)
    cldf[:, :5] = 0.0
    cldf[0, 1] = 0.7
    cldf[-1, 2] = 0.7
    cldf[:, 3] = 1.0
    cldf[:max(1, nlay // 3), 4] = 0.5
    return cldf


def _lw_flags(torch, cldf, seeds, iovr, dz, de_lgth, alpha):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    nlay = cldf.shape[0]
    bits = lw.mcica_bits(t(cldf), t(seeds), iovr=iovr, dz=t(dz), de_lgth=t(de_lgth), alpha=t(alpha))
    bits = bits.cpu().numpy().view(np.uint32)
    k = np.arange(nlay)
    return ((bits[:, :, k >> 5] >> (k & 31)) & 1).astype(bool).transpose(0, 2, 1)   # (column, layer, g-point)


@pytest.mark.parametrize("nlay", [1, 2, 31, 32, 33, 64, 65, 96, 254, 255])
def test_longwave_layer_counts(torch, orc, nlay):
    n = 9
    rng = np.random.default_rng(nlay)
    cldf = _columns(rng, nlay, n)
    seeds = rng.integers(-2**31, 2**31 - 1, n).astype(np.int32)
    dz, dl = rng.uniform(0.05, 1.0, (nlay, n)), rng.uniform(0.2, 6.0, n)
    alpha = rng.uniform(0.0, 1.0, (nlay, n))
    for iovr in OVERLAPS:
        got = _lw_flags(torch, cldf, seeds, iovr, dz, dl, alpha)
        for i in range(n):
            want = orc.mcica(cldf[:, i], int(seeds[i]), iovr=iovr, dz=dz[:, i], de_lgth=float(dl[i]),
                             alpha=alpha[:, i])
            assert np.array_equal(got[i], want), (iovr, i)


@pytest.mark.parametrize("seed,draw", [(2944804, 2448), (3658552, 3428), (2093810, 7220)])
def test_longwave_draw_of_one_above_the_clouds(torch, orc, seed, draw):
    """Draw `draw` of these seeds is 1: g-point draw % 140 of layer draw // 140,
    above the six cloudy layers.  It flags that clear layer (unlinked layers,
    column 0) and, under iovr 3, the run linked to it (column 1)."""
    nlay, k, g = 127, draw // 140, draw % 140
    u, _, _ = orc.mt_stream(seed, draw + 1)
    assert u[draw] == 0xFFFFFFFF
    cldf = np.zeros((nlay, 2))
    cldf[:6] = 0.4
    seeds = np.array([seed, seed], dtype=np.int32)
    dz, dl = np.full((nlay, 2), 0.5), np.array([1e-3, 5.0])
    alpha = np.stack([np.zeros(nlay), np.full(nlay, 0.9)], axis=1)
    for iovr in OVERLAPS:
        got = _lw_flags(torch, cldf, seeds, iovr, dz, dl, alpha)
        for i in range(2):
            want = orc.mcica(cldf[:, i], seed, iovr=iovr, dz=dz[:, i], de_lgth=float(dl[i]), alpha=alpha[:, i])
            assert i == 1 or want[k, g]
            assert np.array_equal(got[i], want), (iovr, i)


@pytest.mark.parametrize("nlay", [2, 31, 32, 65, 128, 199])
def test_shortwave_layer_counts(torch, nlay):
    from oracle import oracle_sw as osw
    n = 9
    rng = np.random.default_rng(1000 + nlay)
    cldf = _columns(rng, nlay, n)
    seeds = rng.integers(-2**31, 2**31 - 1, n).astype(np.int32)
    dz, dl = rng.uniform(0.05, 1.0, (nlay, n)), rng.uniform(0.2, 6.0, n)
    alpha = rng.uniform(0.0, 1.0, (nlay, n))
    alpha[::3, 5], alpha[1::3, 5], alpha[2::3, 5] = 1.5, -0.5, np.nan
    alpha[:, 6], alpha[:, 7] = 1.0, 0.0
    nw = (nlay + 31) // 32
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    args = [t(a) for a in (seeds, cldf, dz, dl, alpha)]
    sw.rswinit(device=0)
    for iovr in OVERLAPS:
        bits = torch.zeros(n * 112 * nw, dtype=torch.int32, device="cuda")
        err = C.create_string_buffer(256)
        rc = sw.lib().rrtmg_sw_gpu_mcica(n, nlay, 0, iovr, *[a.data_ptr() for a in args], bits.data_ptr(), None, err,
                                         256)
        assert rc == 0, err.value
        torch.cuda.synchronize()
        got = bits.cpu().numpy().view(np.uint32).reshape(n, 112, nw)
        for i in range(n):
            want = osw.mcica_bits(nlay, int(seeds[i]), iovr, cldf[:, i], dz=dz[:, i], de_lgth=float(dl[i]),
                                  alpha=alpha[:, i])
            assert np.array_equal(got[i], want), (iovr, i)
