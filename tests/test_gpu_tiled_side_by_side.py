"""Tiled runs of several small 2D domains on streams of their own: they share
the GPU instead of taking it in turns, and every domain's results are those
of its run alone, from one host thread or several."""
import threading
import time

import numpy as np
import pytest

import lbx

pytestmark = pytest.mark.gpu


def _make(shape, real, seed, nsubs=1):
    LX, LY = shape
    p = lbx.Params(dims=2, LX=LX, LY=LY, LZ=1, precision=real, nsubs=nsubs, tau=(0.8, 0.9),
                   gaccel=(1e-6, 2e-6, 0, 0, 0, 0), sigma_t_on=0, sigma_t_off=1 << 30)
    rng = np.random.default_rng(seed)
    d = lbx.Domain(p, (rng.random(p.NN) < 0.35).astype(np.uint8))
    f = rng.standard_normal((nsubs, 9, p.NN)) * 1e-4
    if nsubs == 2:
        f[1] += 0.1
    d.upload_f(f.astype(p.dtype))
    return d


def _state(d):
    d.sync()
    return d.download_f(), d.download_mv()


@pytest.mark.parametrize("threads", [False, True])
@pytest.mark.parametrize("real,nsubs", [(8, 1), (4, 1), (8, 2)])
def test_results_do_not_depend_on_the_others(real, nsubs, threads):
    shapes = [(48, 67), (30, 30), (100, 64), (128, 128), (17, 41), (64, 64), (200, 90), (300, 300),
              (256, 256)]
    calls = [(40, 40), (20, 60), (200, 0), (6, 266), (34, 300)]

    def go(d):
        t = 0
        for steps, rate in calls:
            d.run(t, steps, rate)
            t += steps

    alone = []
    for i, s in enumerate(shapes):
        with _make(s, real, i, nsubs) as d:
            go(d)
            alone.append(_state(d))
    for _ in range(2):
        ds = [_make(s, real, i, nsubs) for i, s in enumerate(shapes)]
        if threads:
            ts = [threading.Thread(target=go, args=(d,)) for d in ds]
            [t.start() for t in ts]
            [t.join() for t in ts]
        else:
            t = 0
            for steps, rate in calls:
                for d in ds:
                    d.run(t, steps, rate)
                t += steps
        for d, (f, mv) in zip(ds, alone):
            g, nv = _state(d)
            assert np.array_equal(g, f) and np.array_equal(nv, mv)
            d.close()


@pytest.mark.parametrize("real", [8, 4])
def test_small_domains_share_the_gpu(real):
    """Eight domains take less than five times as long as one."""
    n = 2000

    def took(ds):
        r = 1.0
        for q in range(8):
            at = time.perf_counter()
            for d in ds:
                d.run(q * n, n, 0)
            for d in ds:
                d.sync()
            r = min(r, time.perf_counter() - at)
        return r

    ds = [_make((48, 67), real, i) for i in range(8)]
    one = _make((48, 67), real, 99)
    alone, all8 = took([one]), took(ds)
    [d.close() for d in ds + [one]]
    assert all8 < 5 * alone, (alone, all8)
