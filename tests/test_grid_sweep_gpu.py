"""Served blocks: a block's march is split over several CTAs where a batch has few blocks, and so is the
first pass of its assemble. A request alone (few blocks, the finest split) and beside a grid that fills
the GPU (whole blocks) ends in the same state, bit for bit; and in the plain step's within rounding."""
import numpy as np
import pytest

from shaderous_b200 import Config, Problem, Sim, tune
from shaderous_b200.serve import Request, Server, ServerConfig

pytestmark = pytest.mark.gpu

KH = Problem("kh", a=(2, 1, 0.5, 2.5, 0.01, 1e-3), seed=11)
BLAST = Problem("blast", a=(3.0, 50.0, 1.0, 1.0, 0.15))


def _served(hyd, reqs):
    cfg = ServerConfig(hydro=hyd, budget_bytes=3e9, max_grids=8, round_steps=4, keep_states=True)
    with Server(cfg) as s:
        ids = [s.submit(r) for r in reqs]
        s.drain()
        return [s.state(i, r) for i, r in zip(ids, reqs)]


@pytest.mark.parametrize("recon,isen,bc,prob", [
    ("koren", True, 1, BLAST), ("koren", True, 2, BLAST), ("mc", False, 0, KH), ("vanleer", True, 2, BLAST),
    ("minmod", False, 1, BLAST),
])
def test_split_blocks_give_the_whole_blocks_bits(recon, isen, bc, prob):
    hyd = Config(recon=recon, isentropic=isen, cfl=0.4, p_floor=1e-12)
    small = [Request(ndim=3, n=n, steps=9, problem=prob, gamma=1.4, bc=bc) for n in (16, 48)]
    small.append(Request(ndim=2, n=48, steps=9, problem=prob, gamma=1.4, bc=bc))
    alone = [_served(hyd, [r])[0] for r in small]
    mixed = _served(hyd, small + [Request(ndim=3, n=112, steps=9, problem=prob, gamma=1.4, bc=bc)])
    for (a1, a2), (b1, b2) in zip(alone, mixed):
        assert np.array_equal(a1, b1) and np.array_equal(a2, b2)
    r = small[1]
    cfg = Config(**{**hyd.__dict__, "n": (48, 48, 48), "gamma": 1.4, "bc_lo": (bc,) * 3, "bc_hi": (bc,) * 3})
    with Sim(cfg) as s:
        s.reset(prob)
        s.run(steps=9)
        p1, p2 = s.read_state()
    # nine steps of the same arithmetic in two kernels: a few float32 roundings of the largest values
    for got, ref in zip(alone[1], (p1, p2)):
        assert np.abs(got - ref).max() <= 9 * 8 * 2.0 ** -24 * np.abs(ref).max()


# Requests beside one of a single 3D block, the blocks of the whole batch, and the planes of a block a CTA
# marches there: of 16, 8, 4 and 2 the p with the least (p + 4) (c / 2 + 0.65 (c mod 2)), c the CTAs of the
# fullest of 148 SMs (two run side by side on one).
BATCHES = [((), 1, 2), ((32, 32), 17, 2), ((32, 32, 32), 25, 4), ((64,), 65, 8), ((96,), 217, 8), ((96, 32), 225, 16),
           ((112, 48), 371, 16)]


def _planes(n):
    def cost(p):
        c = -(-n * (16 // p) // 148)
        return (p + 4) * (c // 2 + 0.65 * (c % 2))

    return min((16, 8, 4, 2), key=cost)


@pytest.mark.parametrize("bc", [0, 1, 2])
def test_every_split_gives_the_same_bits(bc):
    hyd = Config(recon="koren", isentropic=True, cfl=0.4, p_floor=1e-12)
    one = Request(ndim=3, n=16, steps=8, problem=BLAST, gamma=1.4, bc=bc)
    first, splits = None, set()
    for beside, blocks, planes in BATCHES:
        assert 1 + sum((n // 16) ** 3 for n in beside) == blocks and _planes(blocks) == planes
        splits.add(planes)
        got = _served(hyd, [one] + [Request(ndim=3, n=n, steps=8, problem=BLAST, gamma=1.4, bc=bc) for n in beside])[0]
        first = first or got
        assert np.array_equal(first[0], got[0]) and np.array_equal(first[1], got[1]), beside
    assert splits == {2, 4, 8, 16}


def test_a_pinned_grid_gives_the_same_bits():
    """The block sweep's pinned CTAs per SM hold for served grids too. At one an SM a CTA takes several
    blocks, one after another, in 2D and in 3D."""
    hyd = Config(recon="koren", isentropic=True, cfl=0.4, p_floor=1e-12)
    reqs = [Request(ndim=3, n=112, steps=5, problem=BLAST, gamma=1.4, bc=2),
            Request(ndim=2, n=400, steps=7, problem=BLAST, gamma=1.4, bc=1),
            Request(ndim=3, n=16, steps=3, problem=BLAST, gamma=1.4, bc=1)]  # held while the others run on
    ref = _served(hyd, reqs)
    for per_sm in (1, 2):
        tune.pin("amr_sweep", 0, per_sm)
        try:
            got = _served(hyd, reqs)
        finally:
            tune.pin("amr_sweep", None)
        for (a1, a2), (b1, b2) in zip(ref, got):
            assert np.array_equal(a1, b1) and np.array_equal(a2, b2), per_sm
