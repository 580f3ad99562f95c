"""X-H_n clusters (one to three spokes) under the integrator: the multipliers
come from their linear system (velocities) and Newton's method (positions).

Checked on free clusters at temperatures up to 10,000 K, where a step turns a
bond by up to 30 degrees and Newton's method needs several rounds (much hotter
and the equations have no solution): the
positions meet every constraint within the solver's window (1e-6 relative, in
f32 displacements: 2e-6), and one step agrees with the f64 oracle's Jacobi
sweeps, which stop inside the same window (so within 2e-6 of a 0.1 nm bond
plus the f32 rounding of a displacement).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stars(spokes: int, temperature: float, seed: int = 3):
    from mdb200 import synth
    from mdb200.system import Nonbonded, State, System

    rng = np.random.default_rng(seed)
    g = (np.arange(5) + 0.5) * 0.8
    centres = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    arms = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1]])[:spokes] / np.sqrt(3) * 0.109
    pos, masses, p1, p2 = [], [], [], []
    for c in centres:
        base = len(masses)
        pos += [c, *(c + arms)]
        masses += [12.011] + [1.008] * spokes
        p1 += [base] * spokes
        p2 += [base + 1 + k for k in range(spokes)]
    n = len(masses)
    zero = np.zeros(0, dtype=np.int32)
    system = System(masses=np.array(masses), box=np.eye(3) * 4.0, constraint_p1=np.array(p1, dtype=np.int32),
                    constraint_p2=np.array(p2, dtype=np.int32), constraint_distance=np.full(len(p1), 0.109),
                    nonbonded=Nonbonded(cutoff=1.0, ewald_tolerance=5e-4, charge=np.zeros(n), sigma=np.full(n, 0.3),
                                        epsilon=np.zeros(n), exception_p1=zero, exception_p2=zero,
                                        exception_charge_prod=np.zeros(0), exception_sigma=np.zeros(0),
                                        exception_epsilon=np.zeros(0), use_dispersion_correction=False))
    state = State(positions=np.array(pos), box=np.eye(3) * 4.0,
                  velocities=synth.maxwell_boltzmann(system, temperature, rng))
    return system, state


@pytest.mark.parametrize("spokes", [1, 2, 3])
@pytest.mark.parametrize("temperature", [300.0, 10000.0])
def test_star_step_meets_its_constraints(spokes, temperature):
    from mdb200 import steploop
    from oracle import oracle

    system, state = stars(spokes, temperature)
    loop = steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(friction=0.0, seed=2))
    loop.run(1)
    x = loop.positions()
    want, _, _ = oracle.run(system, state, 1, friction=0.0, seed=2)
    assert np.abs(x - want).max() < 4e-7
    loop.run(20)
    x = loop.positions()
    length = np.linalg.norm(x[system.constraint_p1] - x[system.constraint_p2], axis=1)
    assert np.abs(length / 0.109 - 1).max() < 2e-6
    loop.destroy()


def test_massless_spokes_in_one_plane():
    """Three fixed atoms around a moving one, in a plane with it: the velocity equations have no unique solution and
    Jacobi's sweeps leave the motion out of the plane alone, which nothing constrains.  One slow step (lengths stay
    inside the solver's window) against the oracle; the step moves an atom about 4e-5 nm."""
    from mdb200 import steploop
    from mdb200.system import State
    from oracle import oracle

    system, state = stars(3, 300.0)
    rng = np.random.default_rng(5)
    pos, vel = state.positions.copy(), np.zeros_like(state.positions)
    for base in range(0, len(pos), 4):
        u, v, w = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        for k in range(3):
            angle = 2 * np.pi * k / 3
            pos[base + 1 + k] = pos[base] + 0.109 * (np.cos(angle) * u + np.sin(angle) * v)
        vel[base] = 0.02 * (w + 0.3 * rng.normal(size=3))
        system.masses[base + 1 : base + 4] = 0.0
    state = State(positions=pos, box=state.box, velocities=vel)
    loop = steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(friction=0.0, seed=2))
    loop.run(1)
    want, _, _ = oracle.run(system, state, 1, friction=0.0, seed=2)
    assert np.abs(want[::4] - pos[::4]).max() > 2e-5
    assert np.abs(loop.positions() - want).max() < 4e-7
    loop.destroy()
