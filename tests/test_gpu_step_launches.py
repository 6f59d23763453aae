"""How steps are launched does not change what they compute: close to one
another in a stream (own, a caller's, the CUDA default stream), captured by
the caller into a graph, a short stretch of a large lattice launched directly
by lbx_run, one substance initialised beside a stepped one."""
import numpy as np
import pytest

import lbx

pytestmark = pytest.mark.gpu


def _make(dims, real, layout, edge=20, nsubs=1, solid=0.3):
    LX, LY, LZ = (edge + 3, edge, edge if dims == 3 else 1)
    p = lbx.Params(dims=dims, LX=LX, LY=LY, LZ=LZ, precision=real, layout=layout, nsubs=nsubs,
                   tau=(0.8, 0.9), gaccel=(1e-5, 0, 0, 0, 0, 0), sigma_t_on=0,
                   sigma_t_off=1 << 30)
    rng = np.random.default_rng(dims + real)
    sol = (rng.random(p.NN) < solid).astype(np.uint8)
    f = (rng.standard_normal((nsubs, p.Q, p.NN)) * 1e-4).astype(p.dtype)
    d = lbx.Domain(p, sol)
    d.set_run_mode("steps")
    d.upload_f(f)
    return d


CASES = [(2, 8, lbx.LBX_LAYOUT_COMPACT, 1), (3, 4, lbx.LBX_LAYOUT_COMPACT, 1),
         (3, 8, lbx.LBX_LAYOUT_DENSE, 1), (3, 4, lbx.LBX_LAYOUT_COMPACT, 2),
         (2, 8, lbx.LBX_LAYOUT_DENSE, 2)]


@pytest.mark.parametrize("dims,real,layout,nsubs", CASES)
def test_streams_and_capture(dims, real, layout, nsubs):
    import torch
    out = []
    for how in ("plain", "caller", "default", "capture", "captured run"):
        with _make(dims, real, layout, nsubs=nsubs) as d:
            if how == "plain":
                for t in range(1, 21):
                    d.step(t, write_mv=t == 20)
                    d.sync()                       # every step on its own
            elif how.startswith("capture"):
                d.set_run_mode("auto")
                s = torch.cuda.Stream()
                d.set_stream(s.cuda_stream)
                g = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(g, stream=s):
                    if how == "capture":
                        for t in range(1, 11):
                            d.step(t, write_mv=True)
                    else:
                        d.run(0, 10, 10)
                for _ in range(2):
                    g.replay()
                torch.cuda.synchronize()
            else:
                s = torch.cuda.Stream()
                d.set_stream(s.cuda_stream if how == "caller" else 0)
                for t in range(1, 21):
                    d.step(t, write_mv=t == 20)
            d.sync()
            out.append((d.download_f(), d.download_mv()))
    for f, mv in out[1:]:
        assert np.array_equal(f, out[0][0]) and np.array_equal(mv, out[0][1])


@pytest.mark.parametrize("real,edge", [(8, 74), (4, 94)])
def test_short_stretch_of_a_large_lattice(real, edge):
    """64-65 MB of populations: lbx_run launches 5 pairs directly."""
    with _make(3, real, lbx.LBX_LAYOUT_DENSE, edge, solid=0.02) as a, \
            _make(3, real, lbx.LBX_LAYOUT_DENSE, edge, solid=0.02) as b:
        a.run(0, 10, 0)
        a.run(10, 6, 6)
        for t in range(1, 17):
            b.step(t, write_mv=t in (12,))
        a.sync(), b.sync()
        assert np.array_equal(a.download_f(), b.download_f())
        assert np.array_equal(a.download_mv(), b.download_mv())


@pytest.mark.parametrize("layout", [lbx.LBX_LAYOUT_DENSE, lbx.LBX_LAYOUT_COMPACT])
def test_one_substance_set_beside_a_stepped_one(layout):
    """The other substance's stepped state comes back from the download."""
    with _make(3, 8, layout, nsubs=2) as d:
        d.run(0, 6, 0)
        before = d.download_f()
        d.run(6, 6, 0)
        stepped = d.download_f()
        d.run(12, 4, 0)
        d.upload_f(before[1], subs=1)              # the flow is stale in the exchange array
        f = d.download_f()
        assert np.array_equal(f[1], before[1])
        assert not np.array_equal(f[0], stepped[0])
        d.upload_f(stepped)
        d.run(0, 4, 0)
        assert np.array_equal(d.download_f()[0], f[0])
