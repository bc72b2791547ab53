"""The one-pass ghost fill (k_prologue_direct) against the fill that runs the
list pass after pass (forced by the test hook), bit for bit over the whole
padded arrays, and the dt after each: every type, order of entries, dimension
and physics the one pass accepts, extents down to its smallest, ragged ones and
lists it hands on (corner ghosts off, Reflective and Fixed MHD faces)."""
import numpy as np
import pytest

import dragon_b200 as dg
from dragon_b200.boundary import Fixed, Ignore, Outflow, Periodic, Reflective

pytestmark = pytest.mark.gpu
NO_COOP = 2

LISTS = {
    "implicit outflow": lambda mhd: None,
    "periodic": lambda mhd: Periodic(),
    "walls and periodic": lambda mhd: Reflective("X") + Periodic("YZ"),
    "periodic then outflow": lambda mhd: Periodic("Y") + Outflow("XZ"),
    "gated": lambda mhd: Outflow.Gated("XY") + Periodic("Z"),
    "one side each": lambda mhd: Outflow("X-") + Reflective("X+Y") + Outflow.Gated("Z-"),
    "ignored faces": lambda mhd: Ignore("X-") + Periodic("Y"),
    "fixed inflow": lambda mhd: Fixed(state(mhd), "X-") + Reflective("Y") + Outflow("X+Z"),
    "written twice": lambda mhd: Outflow() + Periodic("Y") + Reflective("X-"),
    "no corners": lambda mhd: Periodic(corner_ghosts=False),
}
SIZES = [(2, (4, 5)), (2, (37, 130)), (3, (5, 4, 6)), (3, (17, 9, 40))]


def state(mhd):
    return [1.1, 0.7, 0.3, -0.2, 0.1, 0.4, 0.5, 0.6][:8 if mhd else 5]


def filled(dim, n, mhd, name, slow):
    rng = np.random.default_rng(4)
    cls = dg.Grid2D if dim == 2 else dg.Grid3D
    G = cls(*n, *([0.1, 0.13, 0.07][:dim]), ghosts=3 if mhd else 2,
            config=dg.Config(mhd=mhd, riemann=dg.RIEMANN_HLLD if mhd else dg.RIEMANN_HLLC))
    w = G.w
    w[...] = rng.uniform(-1, 1, w.shape)
    w[..., :2] = rng.uniform(0.5, 1.5, w.shape[:-1] + (2,))
    if mhd:
        G.B[...] = rng.uniform(-1, 1, G.B.shape)
    b = LISTS[name](mhd)
    if b is not None:
        G.boundary = b
    if slow:
        assert G._lib.dragon_gpu_debug_set(G._h, NO_COOP, 1) == 0
    G.apply_boundary()
    dt = G.cfl_time()
    return G.w.copy(), G.B.copy() if mhd else None, dt


@pytest.mark.parametrize("mhd", [False, True])
@pytest.mark.parametrize("name", list(LISTS))
@pytest.mark.parametrize("dim,n", SIZES)
def test_one_pass_fill_equals_the_passes(dim, n, mhd, name):
    a, b = filled(dim, n, mhd, name, False), filled(dim, n, mhd, name, True)
    assert np.array_equal(a[0], b[0])
    if mhd:
        assert np.array_equal(a[1], b[1])
    assert a[2] == b[2]
