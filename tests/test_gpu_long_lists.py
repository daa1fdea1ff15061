"""Bodies that touch far more contacts than the others (floors and platforms), against the
oracle (0 ULP): the heavy solve at each width it gives the other bodies' lists, with
lists on either side of the chunks'.

Boxes lie a little inside static plates, four clipped contacts each.  The plates come
last, so that they are body b of every contact.
"""
import dataclasses

import numpy as np
import pytest

from mechanic_b200 import abi, physics, scenes
from mechanic_b200.physics import GpuPhysics, GpuPhysicsConfig

from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu

CLIPPED = GpuPhysicsConfig(contact_manifold=abi.MANIFOLD_CLIPPED)


def _platforms(counts, sink=0.005, beside=()):
    """A static plate under each number of 0.25 m cubes on a 0.5 m grid, `beside` them other scenes."""
    plate = scenes.take_bodies(scenes.dense_grid(1), 1)
    cubes, plates = list(beside), []
    for k, n in enumerate(counts):
        cols = max(1, int(np.ceil(np.sqrt(n))))
        i, at = np.arange(n), 30.0 + 0.75 * cols + 40.0 * k
        c = scenes.falling_cubes(n, seed=k)
        tr = c.transforms.copy()
        tr["position"][:, :3] = np.stack([i % cols * 0.5, np.full(n, 20.625 - sink), at + i // cols * 0.5], 1)
        tr["rotation"][:] = (0.0, 0.0, 0.0, 1.0)
        v, col = c.velocities.copy(), c.colliders.copy()
        v["linear"] *= 0.01
        v["angular"] *= 0.01
        col["local_rotation"][:] = (0.0, 0.0, 0.0, 1.0)
        cubes.append(dataclasses.replace(c, transforms=tr, velocities=v, colliders=col))
        tr, col = plate.transforms.copy(), plate.colliders.copy()
        tr["position"][0, :3] = (0.25 * cols, 20.0, at + 0.25 * cols)
        col["half_extents"][0, :3] = (0.25 * cols + 1.0, 0.5, 0.25 * cols + 1.0)
        plates.append(dataclasses.replace(plate, transforms=tr, colliders=col,
                                          masses=np.zeros(1, plate.masses.dtype)))
    return scenes.concatenate(cubes + plates)[0]


@pytest.mark.parametrize("counts,box,cubes", [
    ((32, 33, 128, 129, 256), 0.0, 0),      # 128, 132, 512, 516 and 1,024 entries; cut above 128 (4 lanes)
    ((257, 600), 0.0, 0),                   # 1,028 and 2,400 entries
    ((20, 128, 129, 300), 0.8, 500),        # 16 lanes: cut above 512 entries
    ((512, 513, 700), 0.1, 500),            # a warp per body: above 2,048
])
def test_heavy_solve_with_long_lists_bitexact(cuda_lib, counts, box, cubes):
    beside = [scenes.falling_cubes(cubes, seed=5, box=box)] if cubes else []
    gpu, orc = make_pair(_platforms(counts, beside=beside), CLIPPED)
    for tick in (1, 2, 3):
        compare_tick(gpu, orc, tick, check_tree=False)
        if tick == 1:
            assert gpu.read_last_tick().active_contact_count > max(1024, 2 * gpu.body_count())
    gpu.close()


def _stage_us(scene, cfg, heavy):
    """The shortest contact stage of eight ticks, heavy ones only if asked."""
    gpu = GpuPhysics(scene, cfg, capacities={"pair_capacity": 1 << 18})
    stage = []
    for tick in range(1, 9):
        gpu.dispatch_tick(tick)
        rb = gpu.read_last_tick()
        assert rb.error_flags == 0
        if tick > 2 and (not heavy or rb.active_contact_count > 2 * gpu.body_count()):
            stage.append(rb.kernel_timings.contact_solver_ms * 1e3)
    gpu.close()
    return min(stage)


def test_one_long_list_does_not_hold_up_the_heavy_solve(cuda_lib):
    """20,000 boxes on one plate: 80,000 entries.  The contact stage takes 0.42 ms; with four lanes on
    that list it took 57 ms, with a warp 3.6, and the gather form, which has a warp, takes 3.9."""
    scene = _platforms((20_000,))
    split = _stage_us(scene, CLIPPED, True)
    prev = physics.set_tuning(physics.TUNE_HEAVY_SOLVE, 2)
    try:
        gather = _stage_us(scene, CLIPPED, True)
    finally:
        physics.set_tuning(physics.TUNE_HEAVY_SOLVE, max(prev, 0))
    assert split < 0.5 * gather


def test_lists_are_counted_for_the_split_solve_only(cuda_lib):
    """The residual solve uses no lists: one pass over 80,000 contacts on one plate takes 47 us, about as
    on 160 plates; counted all the same, one atomic after the other on the plate's word, it took 92."""
    cfg = GpuPhysicsConfig(contact_manifold=abi.MANIFOLD_CLIPPED, contact_tolerance=1e-5, contact_max_iterations=1)
    one, many = (_stage_us(_platforms(counts), cfg, False) for counts in ((20_000,), (125,) * 160))
    assert one < 1.4 * many
