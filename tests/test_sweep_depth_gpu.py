"""The march's depth is fitted to the grid (few columns: shallow marches, so that every SM has work).
Every depth is the same kernel and gives the same bits: the fitted one against pinned ones, at
shapes with one column, ragged columns, fewer planes than any depth, and long thin grids."""
import numpy as np
import pytest

from shaderous_b200 import Config, Problem, Sim, tune

pytestmark = pytest.mark.gpu


def _run(n, recon, bc, depth):
    tune.reset()
    if depth is not None:
        tune.pin("uniform_sweep", 0, depth)
    try:
        cfg = Config(n=n, gamma=1.4, bc_lo=(bc, bc, bc if n[2] > 1 else 0), bc_hi=(bc, bc, bc if n[2] > 1 else 0), cfl=0.4,
                     recon=recon, p_floor=1e-12)
        with Sim(cfg) as s:
            s.reset(Problem("blast", a=(1.0, 10.0, 1.0, 0.1, 0.2)))
            s.run(steps=7)
            return s.read_state(), s.clock()
    finally:
        tune.pin("uniform_sweep", None)


@pytest.mark.parametrize("n,recon,bc", [
    ((16, 12, 3), "ppm", 0), ((17, 13, 2), "koren", 1), ((45, 52, 61), "koren", 2), ((5, 7, 300), "ppm", 1),
    ((131, 9, 33), "mc", 0), ((512, 515, 1), "koren", 1), ((700, 513, 1), "ppm", 0),
])
def test_fitted_depth_gives_the_pinned_depths_bits(n, recon, bc):
    (a1, a2), clk = _run(n, recon, bc, None)
    for depth in (1, 7, 64):
        (b1, b2), c = _run(n, recon, bc, depth)
        assert c == clk and np.array_equal(a1, b1) and np.array_equal(a2, b2), depth


@pytest.mark.parametrize("n,caps", [((45, 52, 112), (64, 32)), ((40, 24, 273), (64, 32, 128, 256)),
                                    ((512, 515, 1), (16, 8, 32, 64))])
def test_equal_depths_leave_the_largest_bound(n, caps):
    """Shapes whose fitted depth is below every candidate bound: all bounds are the same launch, and the one
    kept for the size class is the largest, however their timings fall."""
    b = tuple(1 if k > 1 else 0 for k in n)
    cfg = Config(n=n, gamma=1.4, bc_lo=b, bc_hi=b, cfl=0.4, recon="mc", isentropic=False, p_floor=1e-12)
    for _ in range(5):
        tune.reset()
        with Sim(cfg) as s:
            s.reset(Problem("blast", a=(1.0, 10.0, 1.0, 0.1, 0.2)))
            s.run(steps=2)
        ent, = [e for e in tune.entries() if e["kernel"] == "uniform_sweep"]
        assert ent["tz"] == max(caps) and ent["candidates"] == len(caps)
    tune.reset()
