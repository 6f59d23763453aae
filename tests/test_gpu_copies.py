"""Large copies to and from pageable host buffers go through page-locked
chunks on several threads: every byte arrives, around the size where that
starts and at chunk remainders, ordered after the stream's work, from several
host threads at once, and after the last domain gave the chunks back."""
import threading

import numpy as np
import pytest

import lbx

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _domain(n):
    p = lbx.Params(dims=3, LX=n, LY=1, LZ=1, precision=4, layout=lbx.LBX_LAYOUT_DENSE)
    return lbx.Domain(p, np.zeros(n, np.uint8))


# bytes of [19][n] floats: below, at and above 4 MB, one with a ragged last chunk
@pytest.mark.parametrize("n", [4 * MB // 76 - 3, 4 * MB // 76 + 1, 4 * MB // 76 + 13797 * 3 + 1,
                               500_001])
def test_populations_round_trip(n):
    f = np.random.default_rng(n).random((1, 19, n)).astype(np.float32)
    with _domain(n) as d:
        d.upload_f(f)
        assert np.array_equal(d.download_f(), f)


def test_fields_after_a_step():
    """The staged copy waits for the step that writes the fields."""
    n = 1_200_007
    with _domain(n) as d:
        d.init_equilibrium(0, np.linspace(0.9, 1.1, n))
        d.run(0, 20, 20)
        a = d.download_mv()
        d.sync()
        assert np.isfinite(a).all() and np.array_equal(a, d.download_mv())
        parts = [np.empty(n, np.float32) for _ in range(4)]       # planes apart on the host
        lib = lbx.load_library()
        assert lib.lbx_download_mv(d._h, 0, *[x.ctypes.data for x in parts]) == 0
        assert all(np.array_equal(x, a[0, c]) for c, x in enumerate(parts))


def test_threads_and_reuse():
    n = 400_000
    fs = [np.random.default_rng(s).random((1, 19, n)).astype(np.float32) for s in range(3)]
    for _ in range(2):
        out = [None] * 3

        def work(i):
            with _domain(n) as d:
                for _ in range(3):
                    d.upload_f(fs[i])
                    out[i] = d.download_f()

        ts = [threading.Thread(target=work, args=(i,)) for i in range(3)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert all(np.array_equal(o, f) for o, f in zip(out, fs))


def test_batch_samples():
    from lbx.batch import Batch
    edges = [40, 97]
    ps = [lbx.Params(dims=3, LX=e, LY=e, LZ=e, precision=4) for e in edges]
    rng = np.random.default_rng(2)
    ms = [(rng.random(p.NN) < 0.3).astype(np.uint8) for p in ps]
    with Batch(ps, ms) as b:
        fs = [rng.random((19, p.NN)).astype(np.float32) for p in ps]
        for i, f in enumerate(fs):
            b.upload_f(i, f)
        assert all(np.array_equal(b.download_f(i), f) for i, f in enumerate(fs))
