"""lbx_download_mv into planes that lie behind one another on the host, some of
them page-locked by the caller: no copy reaches from one kind of memory into
the other."""
import mmap

import numpy as np
import pytest

import lbx

pytestmark = pytest.mark.gpu


def _pages(count):
    """Page-aligned host memory of `count` floats."""
    return np.frombuffer(mmap.mmap(-1, 4 * count), np.float32)


@pytest.mark.parametrize("locked", [(), (0,), (1,), (0, 2), (0, 1, 2, 3), (3,)])
@pytest.mark.parametrize("n", [4096, 4096 * 64, 4096 * 640])
def test_some_planes_page_locked(locked, n):
    import torch
    from lbx.batch import Batch
    rt = torch.cuda.cudart()
    assert torch.cuda.is_available() and torch.zeros(1, device="cuda").item() == 0
    out = _pages(4 * n).reshape(4, n)
    mv = np.random.default_rng(n).random((1, 4, n)).astype(np.float32)
    p = lbx.Params(dims=3, LX=n, LY=1, LZ=1, precision=4, layout=lbx.LBX_LAYOUT_DENSE)
    lib = lbx.load_library()
    for c in locked:
        assert int(rt.cudaHostRegister(out[c].ctypes.data, 4 * n, 0)) == 0
    try:
        ptrs = [out[c].ctypes.data for c in range(4)]
        with lbx.Domain(p, np.zeros(n, np.uint8)) as d:
            d.upload_mv(mv)
            for _ in range(2):
                out[:] = -1
                assert lib.lbx_download_mv(d._h, 0, *ptrs) == 0
                assert np.array_equal(out, mv[0])
            out[:] = -1
            assert lib.lbx_download_mv(d._h, 0, ptrs[0], None, ptrs[2], ptrs[3]) == 0
            assert np.array_equal(out[[0, 2, 3]], mv[0, [0, 2, 3]]) and (out[1] == -1).all()
        with Batch([p], [np.zeros(n, np.uint8)]) as b:
            b.init_equilibrium(0, mv[0, 0])
            b.run(0, 2, 2)
            out[:] = -1
            assert lib.lbx_batch_download_mv(b._h, 0, *ptrs) == 0
            want = b.download_mv(0)
            assert np.array_equal(out, want)
    finally:
        for c in locked:
            rt.cudaHostUnregister(out[c].ctypes.data)
