"""Logging a grid's Newton solves does not change what it computes: states and
solver counters of the exact solver with the log on equal those with it off."""
import numpy as np
import pytest

import dragon_b200 as dg
from dragon_b200 import problems

pytestmark = pytest.mark.gpu


def grid(dim):
    cfg = dg.Config(riemann=dg.RIEMANN_EXACT, limiter=dg.LIMITER_MC)
    if dim == 1:
        w, dx = problems.sod_1d(700, ghosts=2)
        G = dg.Grid1D(700, dx, ghosts=2, config=cfg)
    elif dim == 2:
        w, dx, dy = problems.kelvin_helmholtz_2d(72, ghosts=2, seed=3)
        G = dg.Grid2D(72, 72, dx, dy, ghosts=2, config=cfg)
        G.boundary = dg.Periodic()
    else:
        w, d = problems.blast_3d(40, ghosts=2, p_in=300.0)
        G = dg.Grid3D(40, 40, 40, d, d, d, ghosts=2, config=cfg)
    G.w[...] = w
    return G


@pytest.mark.parametrize("dim,steps", [(1, 40), (2, 10), (3, 25)])
def test_logging_leaves_the_solution_alone(dim, steps):
    a, b = grid(dim), grid(dim)
    b.newton_log(1 << 20, 3)
    a.advance_steps(steps)
    b.advance_steps(steps)
    sa, sb = a.newton_stats(), b.newton_stats()
    seen, stored = sb.pop("log_seen"), sb.pop("log_stored")
    assert seen == sb["exact_calls"] - sb["cap_hits"] > 100 and stored == -(-seen // 3)
    assert {k: sa[k] for k in sb} == sb
    assert np.array_equal(a.w, b.w)
    rows = b.newton_log_rows()
    assert (rows[:, 6] > 0).all() and (rows[:, 7] >= 1).all()
