"""The dense layout's step at its block sizes: node counts around 16384, where
a launch goes from blocks of 64 (D2Q9 128) threads to larger ones, and
remainders of those, plain and with Walsh nodes, against the oracle."""
import dataclasses

import numpy as np
import pytest

import lbx
import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(129, 127, 1), (128, 128, 1), (29, 113, 5), (131, 126, 0),
                                   (128, 128, 0), (151, 129, 0)])
@pytest.mark.parametrize("real,nsubs", [(8, 1), (8, 2), (4, 1), (4, 2)])
@pytest.mark.parametrize("walsh", [False, True])
def test_dense_blocks_equal_oracle(shape, real, nsubs, walsh):
    LX, LY, LZ = shape
    kw = dict(dims=3 if LZ else 2, LX=LX, LY=LY, LZ=LZ or 1, nsubs=nsubs, tau=(0.8, 0.7),
              gaccel=(1e-5, 2e-5, -1e-5 if LZ else 0, 0, 0, 0), sink=1e-3, sigma_t_on=0,
              sigma_t_off=100)
    p = po.Params(**kw)
    rng = np.random.default_rng(LX)
    sol = (rng.random(p.NN) < 0.02).astype(np.uint8)
    ns = rng.random(p.NN) * 0.5
    dt = np.float64 if real == 8 else np.float32
    f0 = (rng.standard_normal((nsubs, 19 if LZ else 9, p.NN)) * 1e-3).astype(dt)
    if nsubs == 2:
        f0[1] += dt(0.05)
    lp = lbx.Params(precision=real, layout=lbx.LBX_LAYOUT_DENSE, walsh=int(walsh), **kw)
    with lbx.Domain(lp, sol) as d:
        if walsh:
            d.set_ns(ns)
        d.set_run_mode("steps")
        d.upload_f(f0)
        d.run(0, 6, 6)
        d.sync()
        f, mv = d.download_f(), d.download_mv()
    if walsh:
        p = dataclasses.replace(p, walsh=1, ns=ns)
    fo, mvo = po.run_oracle(p, f0.copy(), sol, 0, 6, 6)
    fluid = np.ones(p.NN, bool) if walsh else sol != 1
    tol = 1e-12 if real == 8 else 1e-5
    for s in range(nsubs):
        ref = fo[s][:, fluid]
        assert np.linalg.norm(f[s][:, fluid] - ref) <= tol * np.linalg.norm(ref)
        ref = mvo[s][:, fluid]
        assert np.linalg.norm(mv[s][:, fluid] - ref) <= tol * np.linalg.norm(ref)
