"""Several optimiser steps against a numpy Adam that is fed the gradients of the
same batch: every step has to start from zeroed sums, in a training call after
a gradient check on another stream too.

One batch holds all the samples, so a step's gradient does not depend on the
epoch's permutation but for the order of the reductions.  Tolerances: the
gradients of two passes differ by at most 1e-4 of their norm
(test_gpu_train_batch.py), and rounding the weights to BF16 can turn a last-bit
difference of a weight into 2^-8 of it, which over the few steps stays within
a few per cent of the tensors' norms; sums carried over from the step before
double the second step's gradient, which test_carried_sums_would_show shows to
be far outside."""
import numpy as np
import pytest

from ccpp_physics_b200 import surrogate as sg

pytestmark = pytest.mark.gpu

BATCH, STEPS, LR = 1024, 4, 1e-3
B1, B2, EPS = 0.9, 0.999, 1e-8


def _adam(st, g):
    t = st["step"] + 1
    m = B1 * st["m"] + (1 - B1) * g
    v = B2 * st["v"] + (1 - B2) * g * g
    p = st["params"] - LR * (m / (1 - B1 ** t)) / (np.sqrt(v / (1 - B2 ** t)) + EPS)
    return dict(st, params=np.where(v > 0, p, st["params"]), m=m, v=v, step=t)


def _off(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.fixture(scope="module")
def run():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ccpp_physics_b200 import rrtmg_lw as lw
    rc, msg = lw.rlwinit(device=0)
    assert rc == 0, msg
    feats, targ = sg.make_dataset(BATCH, seed=5)
    feats, targ = feats[:BATCH].contiguous(), targ[:BATCH]
    norm = sg.normalisation(feats, targ)
    y = sg.normalise_targets(targ, norm)
    sg.init(norm, seed=3)
    start = sg.get_state()
    sg.grads(feats, y, BATCH)   # leaves sums behind, on the current stream
    with torch.cuda.stream(torch.cuda.Stream()):
        sg.train(feats, y, epochs=STEPS, batch=BATCH, lr=LR, lr_final=LR)
    got = sg.get_state()
    want = carried = {k: (np.asarray(v, np.float64) if k in ("params", "m", "v") else v) for k, v in start.items()}
    past = 0.0
    for _ in range(STEPS):
        g = {}
        for name, st in (("want", want), ("carried", carried)):
            sg.set_state(**{k: st[k] for k in ("params", "m", "v", "step", "norm")})
            g[name] = sg.grads(feats, y, BATCH)[0].astype(np.float64)
        past = past + g["carried"]
        want, carried = _adam(want, g["want"]), _adam(carried, past)
    return start, got, want, carried


def test_steps_match_adam(run):
    start, got, want, _ = run
    assert got["step"] == STEPS
    assert _off(got["m"], want["m"]) < 0.05 and _off(got["v"], want["v"]) < 0.05
    assert _off(got["params"] - start["params"], want["params"] - start["params"]) < 0.1


def test_carried_sums_would_show(run):
    _, _, want, carried = run
    assert _off(carried["m"], want["m"]) > 0.5 and _off(carried["v"], want["v"]) > 0.5
