"""Bodies with hundreds of bearings: their sides in chunks of one block each, against the
oracle (0 ULP) at the edges of a chunk, and the time of a pass with thousands."""
import dataclasses

import numpy as np
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysics, GpuPhysicsConfig

from test_gpu_mechanism import _compare, _pair

pytestmark = pytest.mark.gpu


def _star(spokes, static=False):
    """A cube with `spokes` bearings to cubes on a ring around it."""
    scene = scenes.dense_grid(spokes + 1)
    tr = scene.transforms.copy()
    ring, radius = np.arange(1, spokes + 1) * (2.0 * np.pi / spokes), max(40.0, 0.3 * spokes)
    tr["position"][0, :3] = (0.0, 30.0, 0.0)
    tr["position"][1:, 0], tr["position"][1:, 1], tr["position"][1:, 2] = radius * np.cos(ring), 30.0, radius * np.sin(ring)
    vel, masses = scene.velocities.copy(), scene.masses.copy()
    vel["linear"][:, :3] = scenes.Rng(spokes).normal("v", 3 * (spokes + 1)).reshape(-1, 3)
    if static:
        masses[:1] = np.zeros(1, masses.dtype)
    scene = dataclasses.replace(scene, transforms=tr, velocities=vel, masses=masses)
    pos = tr["position"][:, :3].astype(np.float64)
    return scenes.compile_mechanism(scene, np.zeros(spokes, np.int64), np.arange(1, spokes + 1),
                                    0.5 * (pos[:1] + pos[1:]), np.tile([0.0, 1.0, 0.0], (spokes, 1)))


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("iterations", [3, 8])
@pytest.mark.parametrize("spokes", [(127,), (128,), (129,), (385,), (40, 300, 256)])
def test_hub_chunks_bitexact(cuda_lib, spokes, iterations, static):
    parts = [scenes.translated(_star(n, static), (0.0, 4.0 * k, 0.0)) for k, n in enumerate(spokes)]
    scene = parts[0] if len(parts) == 1 else scenes.concatenate(parts)[0]
    gpu, orc = _pair(scene, GpuPhysicsConfig(solver_iterations=iterations))
    for tick in range(1, 4):
        _compare(gpu, orc, tick, f"{spokes} spokes")
    gpu.close()


def test_a_hub_of_thousands_does_not_hold_up_the_passes(cuda_lib):
    """5,000 bearings on one body against 5,000 in chains of six: mechanism stages of about 65 us each; one
    warp on the hub took 1,600, a thread per bearing with atomics 225."""
    stage = []
    for scene in (_star(5000), scenes.bearing_chains(1000, 6, seed=1, closure_fraction=0.0, height=20.0)):
        gpu = GpuPhysics(scene, GpuPhysicsConfig(), capacities={"pair_capacity": 1 << 18})
        us = []
        for tick in range(1, 9):
            gpu.dispatch_tick(tick)
            us.append(gpu.read_last_tick().kernel_timings.mechanism_ms * 1e3)
        gpu.close()
        stage.append(min(us[2:]))
    assert stage[0] < 2.0 * stage[1]
