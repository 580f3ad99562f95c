"""The tile list where its rows are unusual: rows longer than the search's
buffer (coarse sort cells leave clusters with boxes as large as the cell), both
tile shapes, with and without pruning at the rebuild, rectangular and
triclinic cells, a system that fills less than one warp of clusters, and the
cells of a sort that end inside a scan chunk or exactly at its edge.

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


@pytest.mark.parametrize("shape,width", [("cube", 4.6), ("octahedron", 5.0), ("dodecahedron", 3.1)])
@pytest.mark.parametrize("tile", [8, 32])
@pytest.mark.parametrize("prune", [1, 2])
@pytest.mark.parametrize("inner", [-1.0, 0.08])
def test_long_rows(shape, width, tile, prune, inner):
    from mdb200 import synth

    system, state = synth.water_box(width=width, shape=shape, seed=8)
    e0, f0, flags0, x0 = evaluated(system, state, None)
    e1, f1, flags1, x1 = evaluated(system, state, [(0.2, 1.5, tile, prune, inner)])
    if tile == 8 and prune == 2 and width > 4:
        assert flags1["tiles"] > 1.5 * flags0["tiles"]  # the coarse sort's boxes reach much further
    assert np.isfinite(x1).all() and np.abs(x1 - x0).max() < 0.01
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
