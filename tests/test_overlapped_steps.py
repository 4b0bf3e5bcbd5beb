"""Uniform steps whose launches overlap (a sweep is resident while the step before still writes the state
it will read). On the CPU: the sweeps read the state by coherent loads only. On the GPU: many steps
enqueued at once end where the same steps end with a wait after each, bit for bit."""
import re
from pathlib import Path

import numpy as np
import pytest

from shaderous_b200 import Config, Problem, Sim

CSRC = Path(__file__).resolve().parent.parent / "shaderous_b200" / "csrc"


@pytest.mark.parametrize("name,end", [("sweep.cu", "__global__ void rate_kernel"), ("sweep_rows.cu", None)])
def test_sweeps_read_the_state_by_coherent_loads(name, end):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    text = text[: text.index(end)] if end else text
    assert "ld_state(u1 +" in text and "ld_state(u2 +" in text
    # neither the read-only path nor a plain read of the state's pointers
    assert "__ldg" not in text and not re.search(r"\bu[12]\s*\[|\*\s*u[12]\b(?!\s*[,)])", text)


@pytest.mark.gpu
@pytest.mark.parametrize("n,recon,bc", [((512, 1, 1), "koren", 1), ((126, 1, 1), "ppm", 2), ((64, 64, 1), "mc", 0),
                                        ((33, 17, 1), "koren", 2), ((513, 512, 1), "minmod", 1), ((17, 13, 9), "koren", 1),
                                        ((40, 36, 21), "ppm", 0)])
def test_steps_at_once_end_where_steps_one_by_one_end(n, recon, bc):
    b = tuple(bc if k > 1 else 0 for k in n)
    cfg = Config(n=n, gamma=1.4, bc_lo=b, bc_hi=b, cfl=0.4, recon=recon, p_floor=1e-12)
    out = []
    for batch in (120, 1):
        with Sim(cfg) as s:
            s.reset(Problem("blast", a=(1.0, 10.0, 1.0, 0.1, 0.2)))
            for _ in range(120 // batch):
                s.step(batch)
                s.sync()
            out.append((s.read_state(), s.clock()))
    (a, ca), (c, cc) = out
    assert ca == cc and np.array_equal(a[0], c[0]) and np.array_equal(a[1], c[1])
