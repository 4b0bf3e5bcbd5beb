"""States read back through the gather: a mesh's leaves in their order, whatever their slots, against
the blocks written one by one; and the run goes on from a read state as without the read."""
import numpy as np
import pytest

from shaderous_b200 import Config, Problem
from shaderous_b200.amr import AmrConfig, AmrSim

pytestmark = pytest.mark.gpu


def _run(ndim, bins, read):
    hyd = Config(gamma=1.4, bc_lo=(1, 2, 0), bc_hi=(1, 1, 0), recon="mc", isentropic=False, cfl=0.4, p_floor=1e-12)
    cfg = AmrConfig(hydro=hyd, ndim=ndim, nr=2, max_level=2, cap=900 if ndim == 3 else 120, refine_hi=0.1, refine_lo=0.05,
                    regrid_every=4, time_bins=bins, time_bins_always=bins > 0)
    with AmrSim(cfg) as a:
        a.reset(Problem("blast", a=(1, 10, 1, 0.1, 0.15)))
        for _ in range(6):
            a.step(3)
            if read:
                a.leaves_state()
        return a.leaves(), a.leaves_state()


@pytest.mark.parametrize("ndim,bins", [(2, 0), (3, 0), (3, 2)])
def test_reading_the_state_leaves_the_run_as_it_is(ndim, bins):
    (s0, l0, c0), (u0, v0) = _run(ndim, bins, False)
    (s1, l1, c1), (u1, v1) = _run(ndim, bins, True)
    assert (s0 == s1).all() and (l0 == l1).all() and (c0 == c1).all()
    assert np.array_equal(u0, u1) and np.array_equal(v0, v1)


@pytest.mark.parametrize("ndim", [2, 3])
def test_leaves_come_back_as_they_were_written(ndim):
    hyd = Config(gamma=1.4, recon="mc", cfl=0.4)
    cfg = AmrConfig(hydro=hyd, ndim=ndim, nr=2, max_level=2, cap=900 if ndim == 3 else 120, regrid_every=4)
    with AmrSim(cfg) as a:
        a.reset(Problem("blast", a=(1, 10, 1, 0.1, 0.15)))
        a.step(9)
        n, cb = len(a.leaves()[0]), cfg.cells_per_block
        rng = np.random.default_rng(1)
        u = rng.random((2, n, cb, 4), dtype=np.float32)
        a.set_leaves_state(u[0], u[1])
        got = a.leaves_state()
        assert np.array_equal(got[0], u[0]) and np.array_equal(got[1], u[1])
