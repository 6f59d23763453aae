"""The tiled run of small 2D lattices: two substances, stretches of any
number of pairs (rounds of uneven length), a frame's step inside the stretch,
columns of uneven width.  FP64 equals the per-step path bit for bit (the same
arithmetic per node); FP32 to its rounding over the steps run."""
import numpy as np
import pytest

import lbx
from lbx import geometry

pytestmark = pytest.mark.gpu


def _run(mode, real, shape, nsubs, calls, layout, faces=True):
    LX, LY = shape
    kw = dict(pressure_s_in=(1, 0), pressure_n_out=(1, 0), rho_in=1.001, rho_out=1.0,
              zeroconcgrad_n=1 if nsubs == 2 else 0) if faces else dict(
                  gaccel=(1e-5, 2e-6, 0, 0, 0, 0))
    p = lbx.Params(dims=2, LX=LX, LY=LY, LZ=1, nsubs=nsubs, precision=real, tau=(0.9, 0.8),
                   sink=1e-3, sigma_t_on=0, sigma_t_off=1 << 30, layout=layout, **kw)
    sol = geometry.transpose_2d(geometry.disc_pack(LY, LX, radius=3, porosity=0.7, seed=4), LY, LX)
    rng = np.random.default_rng(8)
    f0 = rng.standard_normal((nsubs, 9, p.NN)) * 1e-4
    if nsubs == 2:
        f0[1] += 0.1
    with lbx.Domain(p, sol) as d:
        d.set_run_mode(mode)
        d.upload_f(f0.astype(p.dtype))
        out, t = [], 0
        n0 = d.launch_count()
        for steps, rate in calls:
            d.run(t, steps, rate)
            t += steps
            d.sync()
            out.append(d.download_mv())
        n = d.launch_count() - n0
        return d.download_f(), out, n


@pytest.mark.parametrize("layout", [lbx.LBX_LAYOUT_DENSE, lbx.LBX_LAYOUT_COMPACT])
@pytest.mark.parametrize("nsubs,faces", [(1, True), (2, True), (2, False)])
@pytest.mark.parametrize("shape", [(48, 67), (301, 21), (7, 5)])
@pytest.mark.parametrize("calls", [((4, 4), (6, 0), (26, 13), (2, 2), (34, 34)), ((90, 30),)])
def test_tiled_equals_steps(shape, nsubs, faces, calls, layout):
    a = _run("tiled", 8, shape, nsubs, calls, layout, faces)
    b = _run("steps", 8, shape, nsubs, calls, layout, faces)
    assert np.isfinite(a[0]).all()
    assert np.array_equal(a[0], b[0])
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)
    assert a[2] < b[2]


@pytest.mark.parametrize("nsubs", [1, 2])
def test_tiled_fp32_close_to_steps(nsubs):
    a = _run("tiled", 4, (61, 50), nsubs, ((60, 20),), lbx.LBX_LAYOUT_COMPACT)
    b = _run("steps", 4, (61, 50), nsubs, ((60, 20),), lbx.LBX_LAYOUT_COMPACT)
    for s in range(nsubs):
        assert np.linalg.norm(a[0][s] - b[0][s]) <= 1e-5 * np.linalg.norm(b[0][s])
