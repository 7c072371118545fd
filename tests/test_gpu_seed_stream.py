"""Column seeds of faces whose random stream one CTA walks, is cut into jumped
segments, and needs several rounds of them: stream lengths (two draws per grid
point) at the edges of a segment (20,592 words), of the single walk (four
segments) and of a round (sixteen), against the oracle's serial twister."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cnx,cny", [
    (1, 1), (8, 39), (312, 66), (313, 66), (144, 143), (144, 286), (203, 203), (234, 220), (235, 220), (384, 384),
    (312, 528), (313, 528), (768, 576),
])
def test_seeds_of_whole_faces(cnx, cny):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ccpp_physics_b200 import rad_time_vary as rtv
    from oracle import oracle
    i, j = np.meshgrid(np.arange(1, cnx + 1), np.arange(1, cny + 1), indexing="ij")
    keep = np.random.default_rng(cnx * cny).permutation(cnx * cny)[:20000]
    keep = np.append(keep, [0, cnx * cny - 1])      # the first and the last draw of each field
    imap, jmap = i.ravel()[keep].astype(np.int32), j.ravel()[keep].astype(np.int32)
    for sec, ipsd0 in ((3600.0, 35063), (54321.0, 7)):
        rc, sw_ref, lw_ref = oracle.seeds(sec=sec, ipsd0=ipsd0, ipsdlim=100000000, cnx=cnx, cny=cny, isc=1, jsc=1,
                                          imap=imap, jmap=jmap)
        assert rc == 0
        im, jm = torch.from_numpy(imap).cuda(), torch.from_numpy(jmap).cuda()
        sw, lw = (torch.zeros(imap.size, dtype=torch.int32, device="cuda") for _ in range(2))
        msg, err = rtv.gfs_rad_time_vary_seeds(False, None, True, True, 2, 2, sw, lw, cnx, cny, 1, 1, im, jm, sec,
                                               ipsd0, 100000000)
        assert err == 0, msg
        assert np.array_equal(sw.cpu().numpy(), sw_ref) and np.array_equal(lw.cpu().numpy(), lw_ref)
