"""Tiles of a 2D MHD phase per work item of a batch: a number that was set is the
number that runs (seen in the count of work items), an untuned batch takes
fewer where its members have few tiles, and members end where their own advance
ends with several tiles per item and a remainder in the last one."""
import numpy as np
import pytest

import dragon_b200 as dg
from dragon_b200 import batch, problems

pytestmark = pytest.mark.gpu


def grids_of(sizes, seed=6):
    out = []
    for spec in problems.batch_instances(n1d=0, n2d=len(sizes), seed=seed, sizes_1d=(16, 32), sizes_2d=sizes)[1]:
        n = spec["n"]
        G = dg.Grid2D(n, n, spec["dx"], spec["dx"], ghosts=3, config=dg.Config(mhd=True, riemann=dg.RIEMANN_HLLX))
        G.w[...] = spec["w"]
        G.B[...] = spec["B"]
        G.boundary = dg.Periodic()
        G.initialize_B_fields()
        out.append(G)
    return out


def phase_items(grids, group):
    """Work items of the seven sweeps: 8 x 32 tiles of their cell ranges, `group` to an item."""
    return sum(-(-(-(-(G.n[0] + e) // 8) * -(-(G.n[1] + e) // 32)) // group) for G in grids for e in (4, 4, 3, 2, 2, 1, 0))


def same(grids, ref):
    for G, R in zip(grids, ref):
        np.testing.assert_array_equal(G.w, R.w)
        np.testing.assert_array_equal(G.B, R.B)


@pytest.mark.parametrize("group", [2, 4, 8])
def test_a_set_number_runs(group):
    sizes = (16, 40, 72)
    grids, ref = grids_of(sizes), grids_of(sizes)
    b = batch.Batch(grids)
    b.tuning = batch.Tuning(graph_steps=4, mhd_tiles=1)
    one = b.advance_steps(1)["work_items"]
    b.tuning = batch.Tuning(graph_steps=4, mhd_tiles=group)
    assert b.tuning.mhd_tiles == group
    items = b.advance_steps(5)["work_items"]
    assert one - items == phase_items(grids, 1) - phase_items(grids, group) > 0
    for R in ref:
        R.advance_steps(6)
    same(grids, ref)


@pytest.mark.parametrize("sizes,group", [((16, 40, 72), 1), ((256, 256, 256), 3)])
def test_an_untuned_batch_chooses(sizes, group):
    grids, ref = grids_of(sizes), grids_of(sizes)
    b = batch.Batch(grids)
    items = b.advance_steps(3)["work_items"]
    b.tuning = batch.Tuning(mhd_tiles=1)
    one = b.advance_steps(1)["work_items"]
    assert one - items == phase_items(grids, 1) - phase_items(grids, group)
    for R in ref:
        R.advance_steps(4)
    same(grids, ref)
