"""The three tiles of the FP64 2D hydro step (6 x 14, 6 x 30, 16 x 24 cells,
chosen by the grid's extents) at the sizes where one gives way to the next and
at their remainders, against the C restatement of the reference, bit for bit."""
import numpy as np
import pytest

import dragon_b200 as dg
from dragon_b200 import problems
from oracle import port

pytestmark = pytest.mark.gpu


# (nx, ny): a cell or two, one tile and its neighbours, the last 6 x 14 grid
# (148 tiles) and the first 6 x 30 one, the last 6 x 30 grid (740) and the first of 16 x 24
@pytest.mark.parametrize("nx,ny", [(2, 3), (6, 14), (7, 15), (12, 13), (222, 56), (223, 56), (24, 518), (24, 519),
                                   (444, 300), (445, 300), (60, 2220), (61, 2221)])
@pytest.mark.parametrize("walls", [False, True])
def test_tiles_equal_the_restatement(nx, ny, walls):
    w0, dx, dy = problems.kelvin_helmholtz_2d(nx, ghosts=2, seed=5, amp=0.1, ny=ny)
    G = dg.Grid2D(nx, ny, dx, dy, ghosts=2, config=dg.Config(riemann=dg.RIEMANN_HLLC, limiter=dg.LIMITER_VANLEER))
    G.w[...] = w0
    G.boundary = (dg.boundary.Reflective("X") + dg.Periodic("Y")) if walls else dg.Periodic()
    assert G.advance_steps(2).steps == 2
    bc = [(3, 3, 1, None), (4, 12, 1, None)] if walls else [(4, 63, 1, None)]
    ref = port.run_steps_2d(w0, dx, dy, steps=2, riemann=dg.RIEMANN_HLLC, limiter=dg.LIMITER_VANLEER, boundary=bc)
    assert np.array_equal(G.w, ref)
