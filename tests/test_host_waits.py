"""The engine's host code against a CUDA runtime that records missing waits.

The engine's streams do not order with the legacy default stream, where a
device memset and a copy from pageable memory may still be at work when their
calls return.  So what a call leaves behind has to be waited for, or queued on
the engine's own stream, before the next launch reads it.  Kernels do nothing
here (host_runtime/): the host code of csrc/ is compiled against the fakes and
taken through every call that touches a live engine's tables.
"""

from __future__ import annotations

import ctypes as C
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
PACKAGE = ROOT / "making-it-rain-webgpu_b200"
FAKES = Path(__file__).resolve().parent / "host_runtime"


@pytest.fixture(scope="module")
def host_library(tmp_path_factory):
    import sys

    sys.path.insert(0, str(PACKAGE))
    import build

    out = tmp_path_factory.mktemp("host_runtime")
    sources = [PACKAGE / "csrc" / "engine.cu", PACKAGE / "csrc" / "prep.cu", FAKES / "fake_launchers.cu",
               FAKES / "fake_cuda.cpp"]

    def compile_one(source: Path) -> Path:
        made = out / (source.stem + ".o")
        include = ["-I", str(ROOT / "include"), "-I", str(PACKAGE / "csrc")]
        if source.suffix == ".cu":
            cmd = [build.nvcc(), *build.host_compiler(), *build.ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
                   "--expt-relaxed-constexpr", *include]
        else:
            toolkit = Path(build.nvcc()).resolve().parent.parent
            cmd = ["/usr/bin/g++", "-O1", "-std=c++17", "-fPIC", "-I", str(toolkit / "include")]
        subprocess.run([*cmd, "-c", str(source), "-o", str(made)], check=True, capture_output=True)
        return made

    with ThreadPoolExecutor() as pool:
        objects = list(pool.map(compile_one, sources))
    library = out / "libmdb_host.so"
    subprocess.run(["/usr/bin/g++", "-shared", "-o", str(library), *map(str, objects), "-Wl,-Bsymbolic"], check=True)
    return library


@pytest.fixture
def fake(host_library, monkeypatch):
    from mdb200 import abi

    for name in [n for n in abi.EXPORTS if n.startswith(("mdb_mlp", "mdb_reciprocal"))]:
        monkeypatch.delitem(abi.EXPORTS, name)  # kernel files' own entry points, not built here
    lib = abi.load(host_library)
    lib.fake_first_fault.restype = C.c_char_p
    monkeypatch.setattr(abi, "_library", lib)
    lib.fake_reset()
    lib.cudaSetDevice(0)
    yield lib
    assert lib.fake_faults() == 0, lib.fake_first_fault().decode()


def water(barostat=None, **options):
    from mdb200 import steploop, synth

    system, state = synth.water_box(n_waters=300, width=3.0, seed=1, barostat=barostat)
    options = steploop.RunOptions(seed=1, max_batch=1, **options)
    return steploop.StepLoop.batch([system, system], [state, state], options), state


@pytest.mark.parametrize("overflows", [1, 2])
def test_overflowing_lists(fake, overflows):
    """The halt word, the capacities and the new list's arrays are as the next launch needs them."""
    loop, state = water()
    fake.fake_overflow_lists(overflows)
    loop.run(2)
    fake.fake_overflow_lists(overflows)
    loop.evaluate(1)
    assert loop.verlet_flags(0)["listGrown"] == 2 * overflows
    loop.destroy()


def test_creation_with_an_overflowing_list(fake):
    fake.fake_overflow_lists(1)
    loop, _ = water()
    loop.run(1)
    loop.destroy()


def test_state_and_box_calls(fake):
    loop, state = water()
    loop.set_positions(state.positions, 1)
    loop.set_box(np.asarray(state.box) * 1.001, 1)
    loop.set_velocities(state.velocities, 0)
    loop.run(3)
    loop.set_box(np.asarray(state.box), 0)
    loop.evaluate(0)
    loop.advance_step_count(7)
    loop.run(2)
    loop.potential(state.positions, 1)
    loop.positions(0), loop.velocities(1)
    loop.verlet_flags(1)
    loop.run(1)
    loop.destroy()


def test_timed_out_list(fake):
    from mdb200 import steploop

    loop, state = water()
    fake.fake_time_out()
    with pytest.raises(steploop.EngineError):
        loop.run(1)
    loop.run(1)
    loop.destroy()


@pytest.mark.parametrize("surrogate_attempts", [0, 130])
def test_volume_moves(fake, surrogate_attempts):
    """Boxes move one by one and together, a box that has drifted by more than a hundredth asks for a rebuild
    inside a round, and a screening network is trained and used."""
    loop, _ = water(barostat=(1.0, 300.0, 1), surrogate_attempts=surrogate_attempts)
    for _ in range(100):
        loop.run(1)
    assert np.abs(loop.box_vectors(0) / 3.0 - np.eye(3)).max() > 0.01
    loop.destroy()


def test_engines_on_two_devices(fake):
    """Every call reaches its engine's device whichever is current, and leaves the caller's."""
    from mdb200 import steploop, synth

    system, state = synth.water_box(n_waters=300, width=3.0, seed=1)
    loops = [steploop.StepLoop.from_parsed(system, state, steploop.RunOptions(seed=1, device=k)) for k in (0, 1)]
    for current in (1, 0):
        fake.cudaSetDevice(current)
        for loop in loops:
            loop.positions(), loop.velocities()
            loop.set_positions(state.positions)
            loop.set_velocities(state.velocities)
            loop.set_box(state.box)
            loop.run(2)
            loop.run_timed(1)
            loop.evaluate(), loop.potential(state.positions)
            loop.profile_step(1)
            loop.advance_step_count(3)
            now = C.c_int(-1)
            fake.cudaGetDevice(C.byref(now))
            assert now.value == current
    for loop in loops:
        loop.destroy()
