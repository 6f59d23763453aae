"""A frame that ends a tiled stretch writes the macro variables at every tile
plan: lattices near what the tiles hold, whose rounds are two steps long, and
stretches of few pairs.  The macro variables are overwritten before each
stretch, so that an unwritten frame cannot pass.  FP64 equals the per-step
path bit for bit (the same arithmetic per node); FP32 to its rounding over
the steps run."""
import numpy as np
import pytest

import lbx

pytestmark = pytest.mark.gpu

PAIRS = (2, 3, 5, 15, 25)


def _run(mode, real, edge, nsubs):
    p = lbx.Params(dims=2, LX=edge, LY=edge, LZ=1, nsubs=nsubs, precision=real, tau=(0.9, 0.8),
                   gaccel=(1e-5, 2e-6, 0, 0, 0, 0), sigma_t_on=0, sigma_t_off=1 << 30)
    rng = np.random.default_rng(edge)
    sol = (rng.random(p.NN) < 0.35).astype(np.uint8)
    f0 = rng.standard_normal((nsubs, 9, p.NN)) * 1e-4
    if nsubs == 2:
        f0[1] += 0.1
    poison = np.full((nsubs, 1 + p.dims, p.NN), -7.0, p.dtype)
    with lbx.Domain(p, sol) as d:
        d.set_run_mode(mode)
        d.upload_f(f0.astype(p.dtype))
        t, out, launches = 0, [], []
        for pairs in PAIRS:
            d.upload_mv(poison)
            n0 = d.launch_count()
            d.run(t, 2 * pairs, t + 2 * pairs)          # the last step is a frame
            d.sync()
            t += 2 * pairs
            launches.append(d.launch_count() - n0)
            out.append(d.download_mv()[:, :, sol == 0])
        return d.download_f()[:, :, sol == 0], out, launches


@pytest.mark.parametrize("mode,real,edge,nsubs", [
    ("auto", 4, 560, 2), ("auto", 4, 780, 1), ("tiled", 8, 560, 1), ("tiled", 8, 380, 2),
    ("auto", 8, 200, 1), ("tiled", 4, 200, 2)])
def test_frame_after_any_number_of_pairs(mode, real, edge, nsubs):
    a = _run(mode, real, edge, nsubs)
    b = _run("steps", real, edge, nsubs)
    assert a[2][1:] == [1] * (len(PAIRS) - 1)           # one launch a stretch (the first plans)

    def same(x, y):
        if real == 8:
            return np.array_equal(x, y)
        return np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)

    for pairs, x, y in zip(PAIRS, a[1], b[1]):
        for s in range(nsubs):
            for c in range(3):
                assert same(x[s, c], y[s, c]), (pairs, s, c)
    for s in range(nsubs):
        assert same(a[0][s], b[0][s])
