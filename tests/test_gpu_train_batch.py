"""The backward products at the edges of their K slices and chunks: batches of
one tile, of an odd number of tiles, of one CTA per slice and of slices longer
than a staged chunk.  Gradients against the numpy oracle with the tolerance of
tests/test_gpu_surrogate.py (3 % of the tensor's norm: BF16 operands)."""
import numpy as np
import pytest

from ccpp_physics_b200 import surrogate as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [128, 384, 1152, 8192, 24576])
def test_gradients_any_batch(batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ccpp_physics_b200 import rrtmg_lw as lw
    from oracle import mlp_oracle as mo
    rc, msg = lw.rlwinit(device=0)
    assert rc == 0, msg
    feats, targ = sg.make_dataset(batch, seed=5)
    feats, targ = feats[:batch].contiguous(), targ[:batch]
    norm = sg.normalisation(feats, targ)
    y = sg.normalise_targets(targ, norm)
    sg.init(norm, seed=3)
    got, loss = sg.grads(feats, y, batch)
    again, loss2 = sg.grads(feats, y, batch)
    # a second pass starts from zeroed sums: only the order of the reductions differs
    assert np.linalg.norm(again - got) <= 1e-4 * np.linalg.norm(got) and abs(loss2 - loss) <= 1e-4 * loss
    w, n = sg.get_weights()
    ref_loss, ref = mo.loss_and_grads(mo.normalise(feats.cpu().numpy(), n), y.cpu().numpy().astype(np.float64),
                                      mo.unpack(w))
    want = mo.pack_grads(ref)
    assert abs(loss - ref_loss) <= 2e-3 * ref_loss
    for name, lo, hi in (("w1", 0, 1024), ("w2", 1024, 17408), ("b2", 17408, 17536), ("w3", 17536, 54400),
                         ("b3", 54400, 54688)):
        off = np.linalg.norm(got[lo:hi] - want[lo:hi]) / np.linalg.norm(want[lo:hi])
        assert off < 3e-2, (name, off)
