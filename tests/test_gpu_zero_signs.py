"""Signs of zero through a split step: a sweep adds (F_left - F_right) dt / dx to
the conserved state (applyFluxes order, Splitting.cpp), so a momentum of -0
between equal fluxes becomes +0, as -0 + 0 does."""
import numpy as np
import pytest

import dragon_b200 as dg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("riemann", [dg.RIEMANN_HLLC, dg.RIEMANN_HLL, dg.RIEMANN_ROE, dg.RIEMANN_EXACT])
@pytest.mark.parametrize("n", [(13, 9), (7, 6, 5)])
def test_negative_zero_momentum(n, riemann):
    dim = len(n)
    G = (dg.Grid2D if dim == 2 else dg.Grid3D)(*n, *([0.1] * dim), ghosts=2,
                                               config=dg.Config(riemann=riemann, limiter=dg.LIMITER_MC))
    G.w[..., :2] = 1.0, 0.7
    G.w[..., 2:] = -0.0
    G.boundary = dg.Periodic()
    G.split_step(0.01)
    inside = G.w[tuple(slice(2, -2) for _ in n)]
    assert (inside[..., 2:] == 0).all() and not np.signbit(inside[..., 2:]).any()
    assert (inside[..., 0] == 1.0).all()
