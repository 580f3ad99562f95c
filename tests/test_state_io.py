"""States and forces between the caller's arrays and the device's tables: the
conversion kernels at sizes that end inside a block, the second system of a
batch, values at the edges of the fixed-point range, and what a refused call
leaves behind.

Positions are multiples of 2^-32 nm on the device: what goes in comes back
rounded to the nearest one (half away from zero, as the host rounds), so a
round trip is within 2^-33 and a second one exact; velocities come back as the
f32 they are.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch():
    from mdb200 import steploop, synth

    members = [synth.water_box(n_waters=n, width=2.8, seed=60 + n) for n in (601, 683)]
    loop = steploop.StepLoop.batch([m[0] for m in members], [m[1] for m in members], steploop.RunOptions(seed=4))
    yield loop, members
    loop.destroy()


@pytest.mark.parametrize("system", [0, 1])
def test_round_trips(batch, system):
    loop, members = batch
    other = 1 - system
    x_other, v_other = loop.positions(other), loop.velocities(other)
    x = members[system][1].positions.copy()
    x[0] = [-3.25, 900000.0, 2.0**-33]  # negative; near the range's edge; half a unit
    x[-1] = [-(2.0**-33), 3 * 2.0**-33, 0.1]
    loop.set_positions(x, system)
    got = loop.positions(system)
    assert np.abs(got - x).max() <= 2.0**-33
    assert got[0, 2] == 2.0**-32 and got[-1, 0] == -(2.0**-32) and got[-1, 1] == 2.0**-31
    loop.set_positions(got, system)
    assert np.array_equal(loop.positions(system), got)
    v = np.random.default_rng(3).normal(size=x.shape)
    loop.set_velocities(v, system)
    assert np.array_equal(loop.velocities(system), v.astype(np.float32).astype(np.float64))
    assert np.array_equal(loop.positions(other), x_other) and np.array_equal(loop.velocities(other), v_other)
    loop.set_positions(members[system][1].positions, system)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1.1e6])
def test_refused_positions_change_nothing(batch, bad):
    from mdb200 import steploop

    loop, members = batch
    before = loop.positions(1)
    x = members[1][1].positions.copy()
    x[7, 1] = bad
    with pytest.raises(steploop.EngineError):
        loop.set_positions(x, 1)
    with pytest.raises(steploop.EngineError):
        loop.potential(x, 1)
    assert np.array_equal(loop.positions(1), before)


@pytest.mark.parametrize("system", [0, 1])
def test_forces_come_by_atom(batch, system):
    """Each system's forces and energies in its own atom order, against the
    system alone; a trial evaluation leaves the state."""
    from mdb200 import steploop

    loop, members = batch
    s, st = members[system]
    alone = steploop.StepLoop.from_parsed(s, st, steploop.RunOptions(seed=4))
    loop.set_positions(st.positions, system)
    loop.set_velocities(st.velocities, system)
    e0, f0 = alone.evaluate()
    e1, f1 = loop.evaluate(system)
    assert np.array_equal(f0, f1)  # the same fixed-point sums
    assert e0["direct_coulomb"] == e1["direct_coulomb"] and e0["kinetic"] == e1["kinetic"]
    before = loop.positions(system)
    trial = st.positions + 0.001
    energy, forces = loop.potential(trial, system)
    assert np.array_equal(loop.positions(system), before)
    want, want_forces = alone.potential(trial)
    assert np.array_equal(forces, want_forces) and energy == want
    alone.destroy()
