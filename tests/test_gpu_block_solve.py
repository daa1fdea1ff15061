"""The contact solve of a few contacts by one block, against the oracle (0 ULP).

Cubes that rest a little inside the ground have one active contact each, so the
number of cubes sets the number of active contacts: the block takes up to 1,024
of them on ticks of up to 4,096 contacts; static cubes add contacts that are not
active.
"""
import dataclasses

import numpy as np
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu


def _resting(dynamic, static=0, stacked=0):
    """`dynamic` cubes on the ground, `stacked` of them with another cube on top, and `static` fixed ones."""
    n = dynamic + static + stacked
    scene = scenes.falling_cubes(n, seed=n)
    tr, masses = scene.transforms.copy(), scene.masses.copy()
    i = np.arange(dynamic + static)
    tr["position"][:dynamic + static, :3] = np.stack([i % 70 * 0.5, np.full(len(i), 0.12), i // 70 * 0.5], 1)
    top = tr["position"][:stacked].copy()
    top[:, 1] += 0.24
    tr["position"][dynamic + static:] = top
    tr["rotation"][:] = (0.0, 0.0, 0.0, 1.0)
    masses[dynamic:dynamic + static] = np.zeros(1, masses.dtype)
    vel = scene.velocities.copy()
    vel["linear"] *= 0.1
    vel["angular"] *= 0.1
    return dataclasses.replace(scene, transforms=tr, masses=masses, velocities=vel)


@pytest.mark.parametrize("residual", [False, True], ids=["passes", "residual"])
@pytest.mark.parametrize("dynamic,static,stacked", [(1, 0, 0), (33, 0, 1), (1000, 0, 11), (1023, 0, 0), (1024, 0, 0),
                                                    (1025, 0, 0), (70, 4050, 20)])
def test_block_solve_bitexact(cuda_lib, dynamic, static, stacked, residual):
    cfg = GpuPhysicsConfig(contact_tolerance=1e-5, contact_max_iterations=24) if residual else GpuPhysicsConfig()
    gpu, orc = make_pair(_resting(dynamic, static, stacked), cfg)
    most = 0
    for tick in range(1, 4):
        compare_tick(gpu, orc, tick, check_tree=False)
        rb = gpu.read_last_tick()
        most = max(most, rb.active_contact_count)
        if residual:
            st = orc.solve_stats()
            assert rb.contact_iterations == st["iterations"]
            assert rb.contact_relative_residual == st["relative_residual"]
    assert most >= dynamic
