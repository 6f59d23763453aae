"""lbx_run's host work grows with the number of steps, not with its square,
on every stream."""
import time

import numpy as np
import pytest

import lbx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("default_stream", [False, True])
def test_time_is_linear_in_the_steps(default_stream):
    """Four times the steps: four times as long, sixteen where each step
    looks at all that follow."""
    p = lbx.Params(dims=2, LX=16, LY=16, LZ=1, precision=8, tau=(0.8, 1.0))
    with lbx.Domain(p, np.zeros(p.NN, np.uint8)) as d:
        d.set_run_mode("steps")
        if default_stream:
            d.set_stream(0)
        d.init_equilibrium(0, 1.0)
        t0 = 0

        def run(n):
            nonlocal t0
            at = time.perf_counter()
            d.run(t0, n, 0)
            d.sync()
            t0 += n
            return time.perf_counter() - at

        run(200)
        assert min(run(16000) for _ in range(3)) < 9 * min(run(4000) for _ in range(3))


def test_a_repeated_short_stretch_is_replayed():
    """A stretch too short to pay for capturing its graph is launched step by
    step; the same one again and again is not: its host time drops, and the
    results stay the same."""
    p = lbx.Params(dims=3, LX=72, LY=70, LZ=75, nsubs=2, precision=8, tau=(0.9, 0.8),
                   pressure_b_in=(1, 0), pressure_t_out=(1, 0), rho_in=1.0005, rho_out=1.0,
                   constcon_b_in=1, zeroconcgrad_t=1, rho_sigma_in=1.0, sigma_t_on=0,
                   sigma_t_off=1 << 30)
    rng = np.random.default_rng(1)
    sol = (rng.random((p.LZ, p.LX * p.LY)) < 0.2).astype(np.uint8)
    sol[[0, -1]] = 0
    with lbx.Domain(p, sol.reshape(-1)) as a, lbx.Domain(p, sol.reshape(-1)) as b:
        host, launches = [], []
        for d in (a, b):
            d.init_equilibrium(0, 1.0)
            d.init_equilibrium(1, 0.0)
        for k in range(8):
            n0 = a.launch_count()
            at = time.perf_counter()
            a.run(60 * k, 60, 0)
            host.append(time.perf_counter() - at)
            a.sync()
            launches.append(a.launch_count() - n0)
        for t in range(1, 481):
            b.step(t)
        a.sync(), b.sync()
        assert np.array_equal(a.download_f(), b.download_f())
        assert len(set(launches)) == 1
        assert min(host[4:]) < 0.5 * min(host[:2])
