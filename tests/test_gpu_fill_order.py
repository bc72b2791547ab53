"""Boundary lists of MHD grids with a Periodic entry over an Outflow face: the
outermost face point keeps the value Outflow extrapolated before Periodic wrote
the face it came from, so these lists run pass after pass; the arrays and the
dt equal the forced passes bit for bit."""
import numpy as np
import pytest

from dragon_b200.boundary import Outflow, Periodic
from test_gpu_direct_fill import LISTS, filled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [Outflow, Outflow.Gated])
@pytest.mark.parametrize("dim,n,faces", [(2, (4, 5), "Y"), (2, (37, 130), "XY"), (3, (17, 9, 40), "Z")])
def test_periodic_over_outflow(monkeypatch, dim, n, faces, first):
    monkeypatch.setitem(LISTS, "periodic over outflow", lambda mhd: first() + Periodic(faces))
    a, b = (filled(dim, n, True, "periodic over outflow", slow) for slow in (False, True))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert a[2] == b[2]
