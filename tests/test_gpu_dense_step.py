"""The dense layout's step kernel at the edges of its blocks: node counts
around multiples of 256, rows of one to a few nodes, warps with and without
a node next to a solid, one and two substances, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 7, 5), (2, 3, 1), (3, 5, 17), (17, 3, 5), (16, 16, 1),
                                   (257, 1, 1), (64, 4, 8), (61, 23, 9)])
@pytest.mark.parametrize("real,nsubs", [(8, 1), (8, 2), (4, 1), (4, 2)])
def test_dense_step_equals_oracle(shape, real, nsubs):
    import lbx
    import pyoracle as po
    LX, LY, LZ = shape
    kw = dict(dims=3, LX=LX, LY=LY, LZ=LZ, nsubs=nsubs, tau=(0.8, 0.7),
              gaccel=(1e-5, 2e-5, -1e-5, 0, 0, 0), sink=1e-3, sigma_t_on=0, sigma_t_off=100)
    p = po.Params(**kw)
    rng = np.random.default_rng(LX * 100 + LZ)
    sol = np.zeros(p.NN, np.uint8)
    sol[rng.choice(p.NN, max(1, p.NN // 40), replace=False)] = 1
    dt = np.float64 if real == 8 else np.float32
    f0 = (rng.standard_normal((nsubs, 19, p.NN)) * 1e-3).astype(dt)
    if nsubs == 2:
        f0[1] += dt(0.05)
    with lbx.Domain(lbx.Params(precision=real, layout=lbx.LBX_LAYOUT_DENSE, **kw), sol) as d:
        d.upload_f(f0)
        d.run(0, 7, 7)
        d.sync()
        f, mv = d.download_f(), d.download_mv()
    fo, mvo = po.run_oracle(p, f0.copy(), sol, 0, 7, 7)
    fluid = sol != 1
    tol = 1e-12 if real == 8 else 1e-5
    for s in range(nsubs):
        ref = fo[s][:, fluid]
        assert np.linalg.norm(f[s][:, fluid] - ref) <= tol * np.linalg.norm(ref)
        ref = mvo[s][:, fluid]
        assert np.linalg.norm(mv[s][:, fluid] - ref) <= tol * np.linalg.norm(ref)
    assert np.array_equal(f[:, :, ~fluid], f0[:, :, ~fluid])
