"""Where the one-block contact solve hands over to the grid: both sides of the line against
the oracle (0 ULP), and the time of a tick above it."""
import dataclasses

import numpy as np
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysics, GpuPhysicsConfig

from test_gpu_block_solve import _resting
from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu


def _pairs(n):
    """n cubes, each a millimetre inside a static cube of its own: n contacts on 2 n bodies."""
    base = _resting(n)
    col = base.colliders.copy()
    col["local_rotation"][:] = (0.0, 0.0, 0.0, 1.0)
    low, high = base.transforms.copy(), base.transforms.copy()
    low["position"][:, 1] = 5.0
    high["position"][:, 1] = 5.249
    static = dataclasses.replace(base, transforms=low, colliders=col, masses=np.zeros(n, base.masses.dtype))
    return scenes.concatenate([dataclasses.replace(base, transforms=high, colliders=col), static])[0]


@pytest.mark.parametrize("n", [383, 384, 385, 386, 700])
def test_both_sides_of_the_line_bitexact(cuda_lib, n):
    """The line lies at 768 sides of contacts: 384 contacts between bodies."""
    gpu, orc = make_pair(_pairs(n), GpuPhysicsConfig(), pair_capacity=1 << 16)
    for tick in (1, 2, 3):
        compare_tick(gpu, orc, tick, check_tree=False)
        assert tick == 1 or gpu.read_last_tick().active_contact_count in (n, n - 1)   # (a few fly apart at first)
    gpu.close()


@pytest.mark.parametrize("n", [768, 769])
def test_ground_contacts_at_the_line_bitexact(cuda_lib, n):
    gpu, orc = make_pair(_resting(n), GpuPhysicsConfig(), pair_capacity=1 << 16)
    for tick in (1, 2, 3):
        compare_tick(gpu, orc, tick, check_tree=False)
    gpu.close()


def stage_us(scene, cfg, ticks=10):
    """The shortest contact stage of the ticks after the second, and that tick's passes."""
    gpu = GpuPhysics(scene, cfg, capacities={"pair_capacity": 1 << 18})
    stage = []
    for tick in range(1, ticks + 1):
        gpu.dispatch_tick(tick)
        rb = gpu.read_last_tick()
        assert rb.error_flags == 0
        stage.append((rb.kernel_timings.contact_solver_ms * 1e3, rb.contact_iterations))
    gpu.close()
    return min(stage[2:])


def test_a_thousand_contacts_are_not_left_to_one_block(cuda_lib):
    """Eight fixed passes over 1,000 contacts on the grid against 384 in the block (47 and 45 us); left to
    the block, 1,000 took 80."""
    many, few = (stage_us(_pairs(n), GpuPhysicsConfig())[0] for n in (1000, 384))
    assert many < 1.35 * few
