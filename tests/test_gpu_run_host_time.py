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
