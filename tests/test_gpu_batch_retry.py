"""Batch members whose steps fail and are retried at half the dt end where their
own advance_steps ends, retry for retry. A retried member's control block goes
up on the member's stream, and the next replay reads it on the batch's."""
import numpy as np
import pytest

import dragon_b200 as dg
from dragon_b200 import batch, problems

pytestmark = pytest.mark.gpu


def tubes(count):
    """Tubes of uneven length; with CFL_coeff = 2 most steps are rejected once."""
    grids = []
    for k in range(count):
        n = 32 + 7 * k
        w0, dx = problems.sod_1d(n, ghosts=2, left=(1.0, 0.0, 1000.0), right=(1.0, 0.0, 0.01))
        G = dg.Grid1D(n, dx, ghosts=2, config=dg.Config(riemann=dg.RIEMANN_HLLC, limiter=dg.LIMITER_SUPERBEE,
                                                        cfl_coeff=2.0 if k % 3 else 0.3))
        G.w[...] = w0
        G.boundary = dg.Outflow()
        grids.append(G)
    return grids


@pytest.mark.parametrize("count,steps", [(1, 3), (40, 5)])
def test_retried_members_match_their_own_advance(count, steps):
    ref, grids = tubes(count + 1), tubes(count + 1)
    b = batch.Batch(grids)
    for _ in range(3):  # an advance whose last step was retried hands over to the next
        retries = sum(G.advance_steps(steps).retries for G in ref)
        assert b.advance_steps(steps)["retries"] == retries
        for G, R in zip(grids, ref):
            np.testing.assert_array_equal(G.w, R.w)
        assert retries > 0
