"""The tile list where its rows are unusual: long rows (coarse sort cells leave
clusters with boxes as large as the cell), rows longer than the search's
buffer, both tile shapes, with and without pruning at the rebuild, rectangular
and triclinic cells, a system of less than one warp of clusters, and the cells
of a sort that end inside a scan chunk or exactly at its edge.

A list only decides which pairs are looked at: forces agree with the default
list's to the rounding of sums taken in another order (1e-6 relative RMS, five
times what two orders show), and the in-cutoff pair count is the same.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def evaluated(system, state, tuning):
    from mdb200 import steploop

    loop = steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(seed=3, tuning=tuning))
    loop.run(7)  # a rebuild or two on the way
    x = loop.positions()
    loop.set_positions(state.positions)  # and one at the same positions for every list
    energies, forces = loop.evaluate()
    flags = loop.verlet_flags()
    loop.destroy()
    return energies, forces, flags, x


@pytest.mark.parametrize("shape,width,waters", [("cube", 4.6, None), ("octahedron", 5.0, None),
                                                ("dodecahedron", 3.1, None), ("cube", 2.1, 60)])
@pytest.mark.parametrize("tile", [8, 32])
@pytest.mark.parametrize("prune", [1, 2])
@pytest.mark.parametrize("inner", [-1.0, 0.08])
def test_long_rows(shape, width, waters, tile, prune, inner):
    from mdb200 import synth

    system, state = synth.water_box(width=width, shape=shape, seed=8, n_waters=waters)
    e0, f0, flags0, x0 = evaluated(system, state, None)
    e1, f1, flags1, x1 = evaluated(system, state, [(0.2, 1.5, tile, prune, inner)])
    if tile == 8 and prune == 2 and width > 4:
        assert flags1["tiles"] > 1.5 * flags0["tiles"]  # the coarse sort's boxes reach much further
    assert np.isfinite(x1).all() and np.abs(x1 - x0).max() < 0.01
    assert e0["pairs_within_cutoff"] == e1["pairs_within_cutoff"]
    assert np.sqrt(((f1 - f0) ** 2).sum() / (f0**2).sum()) < 1e-6


ROW_BUFFER, ROW_TASKS = 512, 8192  # the search's buffer (candidates) and the warps it wants at least


def tiles_within_the_buffer(supers, copies, tile):
    """The most tiles a system's list can have while no stretch of a row has more candidates than the buffer.  Rows are
    cut in half, down to 8 super-clusters, until the engine has ROW_TASKS stretches."""
    per, sub = supers, 32 // tile
    while per > 8 and copies * supers * sub * (-(-supers // per) + 1) // 2 < ROW_TASKS:
        per = max(8, (per + 1) // 2)
    most, clusters = 0, supers * sub
    for start in range(0, clusters, per * sub):
        end = min(clusters, start + per * sub)
        most += sum(min(ROW_BUFFER, end - max(start, row)) for row in range(end))
    return most


@pytest.mark.parametrize("tile,copies,width", [(8, 1, 6.5), (8, 16, 5.6), (32, 16, 5.6)])
def test_rows_past_the_buffer(tile, copies, width):
    """Waters in no order and one sort cell: a cluster's box is most of the cell, and nearly every cluster near every
    other.  One system in the one-launch list, and batches whose rows are whole and whose phases are separate
    launches; with the tiles as found (the count shows the buffer is passed) and pruned."""
    from mdb200 import steploop, synth
    from mdb200.system import State

    system, state = synth.water_box(width=width, seed=10)
    order = np.random.default_rng(1).permutation(system.particle_count // 3)
    state = State(positions=state.positions.reshape(-1, 3, 3)[order].reshape(-1, 3), box=state.box,
                  velocities=state.velocities)
    e0, f0, _, _ = evaluated(system, state, None)
    for prune in (2, 1):
        loop = steploop.StepLoop.batch([system] * copies, [state] * copies,
                                       steploop.RunOptions(seed=3, tuning=[(0.15, width, tile, prune, -1.0)] * copies))
        if prune == 2:
            supers = -(-system.particle_count // 32)
            assert loop.verlet_flags()["tiles"] > tiles_within_the_buffer(supers, copies, tile)
        loop.run(3)
        loop.set_positions(state.positions, copies - 1)
        e1, f1 = loop.evaluate(copies - 1)
        loop.destroy()
        assert e0["pairs_within_cutoff"] == e1["pairs_within_cutoff"]
        assert np.sqrt(((f1 - f0) ** 2).sum() / (f0**2).sum()) < 1e-6


@pytest.mark.parametrize("width,cell", [(4.0, 0.5), (4.0, 0.25), (4.05, 0.58), (2.05, 2.0)])
def test_sort_chunks(width, cell):
    """8^3 = 512 cells fill one chunk, 16^3 eight, 6^3 part of one; one cell."""
    from mdb200 import synth

    system, state = synth.water_box(width=width, seed=9)
    _, f0, _, x0 = evaluated(system, state, None)
    _, f1, _, x1 = evaluated(system, state, [(0.2, cell, 8, 1, -1.0)])
    assert np.isfinite(x1).all() and np.abs(x1 - x0).max() < 0.01
    assert np.sqrt(((f1 - f0) ** 2).sum() / (f0**2).sum()) < 1e-6
