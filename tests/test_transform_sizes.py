"""The mesh transforms and the charge spread at the sizes where they can go
wrong: axes of one to four stages, odd planes (whose last z line has no
partner), planes that fit shared memory and planes that do not, charges past
the range of the spread's sums in shared memory, and spread blocks that hold
the end of one system and the start of the next.

Bounds: reciprocal forces against the f64 oracle at the 1e-5 relative RMS the
oracle's own PME forces are pinned to (an f32 transform of n points loses
about log2(n) 2^-24, a few 1e-7); grids are integers, so routes that only
differ in the order of the spread agree to the bit.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import ENERGY_REL, RECIPROCAL_FORCE_REL_RMS, separated_charges

pytestmark = pytest.mark.gpu

# one stage; odd; three stages on x, on y and z of whole planes (75, 98, 112; 75 is odd) and in strips; both sides
# of the plane kernels' shared memory; the largest
MESHES = [(10, 9, 8), (21, 15, 25), (35, 27, 49), (98, 27, 14), (12, 75, 75), (9, 98, 50), (9, 30, 112), (20, 100, 128),
          (18, 125, 63), (64, 64, 64)]


@pytest.mark.parametrize("mesh", MESHES)
def test_mesh_forces_and_energy(mesh):
    import torch

    from mdb200 import abi
    from oracle import oracle

    system, state, alpha = separated_charges()
    want, want_forces = oracle.potential(system, state.positions, grid=mesh)
    n = system.particle_count
    pos, q = torch.from_numpy(state.positions).cuda(), torch.from_numpy(system.nonbonded.charge).cuda()
    forces = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda")
    energy = torch.full((1,), 7.0, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second call finds the first one's scratch
        status = abi.load().mdb_reciprocal_noalloc(
            n, pos.data_ptr(), q.data_ptr(), (C.c_double * 9)(*np.asarray(state.box).reshape(9)), alpha,
            (C.c_int32 * 3)(*mesh), forces.data_ptr(), energy.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert status == abi.OK
        got = forces.cpu().numpy()
        # the charges are farther apart than the cutoff: direct forces are zero
        assert np.sqrt(((got - want_forces) ** 2).sum() / (want_forces**2).sum()) < RECIPROCAL_FORCE_REL_RMS
        assert abs(energy.item() - want["reciprocal_mesh"]) < ENERGY_REL * abs(want["reciprocal_mesh"])


@pytest.mark.parametrize("mesh", [(21, 15, 25), (75, 84, 96), (96, 98, 75), (25, 105, 112), (24, 30, 375),
                                  (375, 24, 27), (24, 120, 120)])
@pytest.mark.parametrize("charge", [1.0, 1500.0])
def test_engine_mesh_forces(mesh, charge):
    """The engine's own passes, at ordinary charges and beyond 1,000 e: whole planes of two-stage and of three-stage
    axes, four stages, and strips."""
    from mdb200 import steploop
    from oracle import oracle

    system, state, _ = separated_charges()
    system.nonbonded.charge = system.nonbonded.charge * charge
    _, want = oracle.potential(system, state.positions, grid=mesh)
    loop = steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(mesh=mesh))
    _, got = loop.evaluate()
    loop.destroy()
    # a force is the difference of neighbouring points' f32 potentials over their distance: past 100 points on these
    # 3 nm the potentials' rounding grows with the points (375 points: 2.3e-5, with radices up to 5 3.8e-5)
    bound = RECIPROCAL_FORCE_REL_RMS * max(1.0, max(mesh) / 100)
    assert np.sqrt(((got - want) ** 2).sum() / (want**2).sum()) < bound


@pytest.mark.parametrize("counts", [(672, 700), (672, 683, 691, 705, 672, 690, 750)])
def test_spread_blocks_across_systems(counts):
    """Systems whose slots are no multiple of a spread block's: the batch
    moves each as it moves alone, to the bit."""
    from mdb200 import steploop, synth

    members = [synth.water_box(n_waters=n, width=2.9, seed=40 + k, grid=(28, 27, 30)) for k, n in enumerate(counts)]
    batch = steploop.StepLoop.batch([m[0] for m in members], [m[1] for m in members], steploop.RunOptions(seed=5))
    batch.run(12)
    for k, (system, state) in enumerate(members):
        alone = steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(seed=5))
        alone.run(12)
        assert np.array_equal(batch.positions(k), alone.positions()), k
        alone.destroy()
    batch.destroy()


@pytest.mark.parametrize("charge", [1.0, 990.0, 1010.0, 1e5, 1e7])
def test_large_charges_close_together(charge):
    """Two clumps of 32 like charges, each a compact block of the spread: below 1,000 e their sums meet in shared
    memory, 32 bits at a time, from there they go straight to the 64-bit grid.  The mesh energy against the oracle's."""
    from mdb200 import steploop
    from mdb200.system import State
    from oracle import oracle

    system, state, _ = separated_charges()
    rng = np.random.default_rng(4)
    corner = np.stack(np.meshgrid(range(4), range(4), range(2), indexing="ij"), -1).reshape(-1, 3) * 0.1
    width = state.box[0][0]
    pos = np.concatenate([corner + 0.2 * width, corner + 0.6 * width]) + rng.uniform(-0.02, 0.02, size=(64, 3))
    system.nonbonded.charge = charge * np.repeat([1.0, -0.9], 32) * rng.uniform(0.99, 1.01, size=64)
    state = State(positions=pos, box=state.box)
    want, _ = oracle.potential(system, pos, grid=(40, 36, 42))
    loop = steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(mesh=(40, 36, 42)))
    got, _ = loop.evaluate()
    loop.destroy()
    assert abs(got["reciprocal_mesh"] - want["reciprocal_mesh"]) < ENERGY_REL * abs(want["reciprocal_mesh"])


@pytest.mark.parametrize("short", [0, 1, 2])
@pytest.mark.parametrize("corner", range(8))
def test_spread_on_an_axis_of_five_points(short, corner):
    """Uncharged atoms share a block with charged ones and come first in it for some corner: on an axis as short as
    the stencil the charged ones' unwrapped points then start as much as six points from the mesh's first.  The mesh
    energy against the oracle's."""
    from mdb200 import steploop
    from mdb200.system import Nonbonded, State, System
    from oracle import oracle

    rng = np.random.default_rng(6)
    width, n, empty = 3.0, 32, np.zeros(0, dtype=np.int32)
    mesh = [24, 27, 28]
    mesh[short] = 5
    place = np.array([(corner >> k) & 1 for k in range(3)]) * 0.9 + 0.05
    pos = np.tile(place, (n, 1)) + rng.uniform(-0.03, 0.03, size=(n, 3))  # of the box
    charge = rng.uniform(0.5, 1.0, size=n)
    charge[: n // 2] = 0.0
    pos[: n // 2, short] = rng.uniform(0.62, 0.78, size=n // 2)  # base 4 of the five
    pos[n // 2 :, short] = rng.uniform(0.02, 0.18, size=n // 2)  # base 1
    order = rng.permutation(n)
    pos, charge = pos[order] * width, charge[order]
    box = np.eye(3) * width
    system = System(masses=np.full(n, 10.0), box=box,
                    nonbonded=Nonbonded(cutoff=0.5, ewald_tolerance=5e-4, charge=charge, sigma=np.full(n, 0.3),
                                        epsilon=np.zeros(n), exception_p1=empty, exception_p2=empty,
                                        exception_charge_prod=np.zeros(0), exception_sigma=np.zeros(0),
                                        exception_epsilon=np.zeros(0), use_dispersion_correction=False))
    want, _ = oracle.potential(system, pos, grid=tuple(mesh))
    loop = steploop.StepLoop.from_parsed(system, State(positions=pos, box=box), steploop.RunOptions(mesh=mesh))
    got, _ = loop.evaluate()
    loop.destroy()
    assert abs(got["reciprocal_mesh"] - want["reciprocal_mesh"]) < ENERGY_REL * abs(want["reciprocal_mesh"])
