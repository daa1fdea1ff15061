"""The one-block contact solve with a body that touches most of the others, against the
oracle (0 ULP): a static plate under cubes, as body b of their contacts and as body a,
with lists on either side of what one thread sums."""
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysics, GpuPhysicsConfig

from test_gpu_long_lists import _platforms
from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu


def _scene(counts, plates_first):
    scene = _platforms(counts)
    if not plates_first:
        return scene
    n = scene.body_count - len(counts)   # (cubes, then plates)
    cubes = scenes.take_bodies(scene, n)
    order = [_platforms((c,)) for c in counts]
    plates = [_last(s) for s in order]
    for k, plate in enumerate(plates):
        plate.transforms["position"][0] = scene.transforms["position"][n + k]
    return scenes.concatenate(plates + [cubes])[0]


def _last(scene):
    """The last body of a scene with one collider per body."""
    import dataclasses
    col = scene.colliders[-1:].copy()
    col["metadata"][:, :2] = 0
    return dataclasses.replace(scene, transforms=scene.transforms[-1:].copy(), velocities=scene.velocities[-1:],
                               masses=scene.masses[-1:], spatial_inertias=scene.spatial_inertias[-1:], colliders=col,
                               root_flags=scene.root_flags[-1:], body_components=scene.body_components[:1])


@pytest.mark.parametrize("residual", [False, True], ids=["passes", "residual"])
@pytest.mark.parametrize("plates_first", [False, True], ids=["body_b", "body_a"])
@pytest.mark.parametrize("counts", [(31, 32, 33), (64, 200), (448,), (33,) * 13, (1024,), (33,) * 31])
def test_block_solve_long_lists_bitexact(cuda_lib, counts, plates_first, residual):
    cfg = GpuPhysicsConfig(contact_tolerance=1e-5, contact_max_iterations=24) if residual else GpuPhysicsConfig()
    gpu, orc = make_pair(_scene(counts, plates_first), cfg, pair_capacity=1 << 18)
    for tick in (1, 2, 3):
        compare_tick(gpu, orc, tick, check_tree=False)
        rb = gpu.read_last_tick()
        assert rb.active_contact_count == sum(counts)
        if residual:
            assert rb.contact_iterations == orc.solve_stats()["iterations"]
    gpu.close()


@pytest.mark.parametrize("cubes,residual,limit_us", [(440, False, 61.0), (1000, True, 1620.0)],
                         ids=["passes", "residual"])
def test_one_long_list_does_not_hold_up_the_block(cuda_lib, cubes, residual, limit_us):
    """Cubes on one plate: the contact stage in at most 1.25 times the 49 us that the whole grid takes
    for eight passes and 1.5 times its 1,080 for 81; one thread per component took 66 and 1,949 us."""
    cfg = GpuPhysicsConfig(contact_tolerance=1e-5, contact_max_iterations=81) if residual else GpuPhysicsConfig()
    gpu = GpuPhysics(_platforms((cubes,), sink=0.001), cfg, capacities={"pair_capacity": 1 << 16})
    stage = []
    for tick in range(1, 11):
        gpu.dispatch_tick(tick)
        rb = gpu.read_last_tick()
        assert rb.active_contact_count == cubes
        stage.append(rb.kernel_timings.contact_solver_ms * 1e3)
    gpu.close()
    assert min(stage[2:]) < limit_us
