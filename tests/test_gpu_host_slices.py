"""Host arrays that are slices of a parent's columns, ptr = parent + c0 with
ldim the parent's: the last row's npts columns end where the parent ends, and
nothing behind them is read or written.  Every array ends at the end of a page
whose neighbour is not accessible."""
import ctypes as C
import mmap

import numpy as np
import pytest

from ccpp_physics_b200 import abi, rrtmg_lw as lw, rrtmg_sw as sw, synthetic

pytestmark = pytest.mark.gpu

# (columns, ldim, layers): staged, per array, pipelined
SIZES = [(17, 23, 40), (400, 431, 127), (8200, 8209, 12)]
_libc = C.CDLL(None, use_errno=True)
_libc.mprotect.argtypes = [C.c_void_p, C.c_size_t, C.c_int]


class Guarded:
    """Arrays in maps of their own, the page behind each closed."""

    def __init__(self):
        self.maps = []

    def array(self, values):
        page = mmap.PAGESIZE
        room = -(-values.nbytes // page) * page
        m = mmap.mmap(-1, room + page)
        whole = np.frombuffer(m, np.uint8)
        assert _libc.mprotect(whole.ctypes.data + room, page, 0) == 0
        self.maps.append((m, whole, room))
        out = whole[room - values.nbytes:room].view(values.dtype)
        out[:] = values
        return out

    def close(self):
        for _, whole, room in self.maps:
            assert _libc.mprotect(whole.ctypes.data + room, mmap.PAGESIZE, mmap.PROT_READ | mmap.PROT_WRITE) == 0


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _sliced(arrays, c0, ld, guarded):
    """Columns c0 .. of every array over the columns, flat."""
    out = {}
    for k, v in arrays.items():
        if not isinstance(v, np.ndarray) or ld not in v.shape:
            out[k] = v
        else:
            record = v.shape[-1] if v.shape[-1] != ld else 1
            out[k] = guarded.array(np.ascontiguousarray(v).reshape(-1)[c0 * record:])
    return out


def _compare(part, full, c0, ld):
    for k, v in part.items():
        record = full[k].shape[-1] if full[k].shape[-1] != ld else 1
        want = full[k].reshape(-1, ld, record)
        got = np.concatenate([np.zeros(c0 * record), v]).reshape(want.shape)
        assert np.array_equal(got[:, c0:], want[:, c0:]), k


@pytest.mark.parametrize("n,ld,nlay", SIZES)
def test_longwave(n, ld, nlay):
    _cuda()
    assert lw.rlwinit(device=0)[0] == 0
    c0 = ld - n
    prof = synthetic.make_profiles(ld, nlay, seed=4)
    full = abi.alloc_outputs(ld, nlay, hlw0=True, flxprf=True)
    msg, err = lw.run_profile(prof, full)
    assert err == 0, msg
    gd = Guarded()
    part = _sliced(abi.alloc_outputs(ld, nlay, hlw0=True, flxprf=True), c0, ld, gd)
    msg, err = lw.run_profile(dict(_sliced(prof, c0, ld, gd), npts=n, flags=dict(prof["flags"], ldim=ld)), part)
    gd.close()
    assert err == 0, msg
    _compare(part, full, c0, ld)


@pytest.mark.parametrize("n,ld,nlay", SIZES)
def test_shortwave(n, ld, nlay):
    _cuda()
    sw.rswinit(device=0)
    c0 = ld - n
    prof = sw.add_sw_inputs(synthetic.make_profiles(ld, nlay, seed=4), seed=4, night_fraction=0.3, precip=True)
    full = sw.alloc_outputs(ld, nlay, flxprf=True)
    sw.rrtmg_sw_run(prof, full)
    idx = np.asarray(prof["idxday"])
    gd = Guarded()
    part = _sliced(sw.alloc_outputs(ld, nlay, flxprf=True), c0, ld, gd)
    inputs = _sliced({k: v for k, v in prof.items() if k != "idxday"}, c0, ld, gd)
    sw.rrtmg_sw_run(dict(inputs, npts=n, idxday=(idx[idx > c0] - c0).astype(np.int32)), part, ldim=ld)
    gd.close()
    _compare(part, full, c0, ld)
