"""Bearing projection gathered by body, against the oracle (0 ULP): odd and even
numbers of passes (the velocities alternate between two buffers), mechanisms
with and without a dynamic root, bodies without bearings beside them, ticks with
and without active contacts."""
import dataclasses

import numpy as np
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_mechanism import _compare, _pair

pytestmark = pytest.mark.gpu


def _scene(static_root, height):
    chains = scenes.bearing_chains(40, 5, seed=3, closure_fraction=0.3, height=height)
    if static_root:
        masses = chains.masses.copy()
        masses[chains.root_flags == 1] = np.zeros(1, masses.dtype)
        chains = dataclasses.replace(chains, masses=masses, has_dynamic_root=0)
    cubes = scenes.translated(scenes.falling_cubes(300, seed=5, box=3.0), (60.0, height, 0.0))
    return scenes.concatenate([chains, cubes])[0]


@pytest.mark.parametrize("iterations", [1, 3, 8])
@pytest.mark.parametrize("static_root", [False, True])
@pytest.mark.parametrize("height", [0.3, 20.0], ids=["contacts", "in_flight"])
def test_bearing_passes_bitexact(cuda_lib, iterations, static_root, height):
    gpu, orc = _pair(_scene(static_root, height), GpuPhysicsConfig(solver_iterations=iterations))
    for tick in range(1, 6):
        _compare(gpu, orc, tick, f"{iterations} passes")


@pytest.mark.parametrize("spokes", [31, 32, 33, 70])
def test_hub_bodies_bitexact(cuda_lib, spokes):
    """A body of 32 bearings fills a warp's lanes; more take the warp-per-body path."""
    scene = scenes.dense_grid(spokes + 1)
    tr = scene.transforms.copy()
    ring = np.arange(1, spokes + 1) * (2.0 * np.pi / spokes)
    tr["position"][0, :3] = (0.0, 30.0, 0.0)
    tr["position"][1:, 0], tr["position"][1:, 1], tr["position"][1:, 2] = 40.0 * np.cos(ring), 30.0, 40.0 * np.sin(ring)
    vel = scene.velocities.copy()
    vel["linear"][:, :3] = scenes.Rng(spokes).normal("v", 3 * (spokes + 1)).reshape(-1, 3)
    scene = dataclasses.replace(scene, transforms=tr, velocities=vel)
    pos = tr["position"][:, :3].astype(np.float64)
    axes = np.tile([0.0, 1.0, 0.0], (spokes, 1))
    scene = scenes.compile_mechanism(scene, np.zeros(spokes, np.int64), np.arange(1, spokes + 1),
                                     0.5 * (pos[:1] + pos[1:]), axes)
    gpu, orc = _pair(scene, GpuPhysicsConfig())
    for tick in range(1, 4):
        _compare(gpu, orc, tick, f"{spokes} spokes")
