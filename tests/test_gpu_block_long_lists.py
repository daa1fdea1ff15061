"""The one-block contact solve with a body that touches most of the others, against the
oracle (0 ULP): a static plate under cubes, as body b of their contacts and as body a,
with lists on either side of what one thread sums."""
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_block_line import _pairs, stage_us
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
@pytest.mark.parametrize("counts", [(31, 32, 33), (64, 200), (384,), (33,) * 11, (1024,), (33,) * 31])
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


@pytest.mark.parametrize("cubes,residual,ratio", [(380, False, 1.2), (1000, True, 1.5)], ids=["passes", "residual"])
def test_one_long_list_does_not_hold_up_the_block(cuda_lib, cubes, residual, ratio):
    """Cubes on one plate against as many on a cube each, per pass: 45 us and 49 for eight passes, 6.6 us
    and 8.2 for one to a residual; with one thread per component the plate took 66 and 24."""
    cfg = GpuPhysicsConfig(contact_tolerance=1e-5, contact_max_iterations=81) if residual else GpuPhysicsConfig()
    (plate, n), (pairs, m) = (stage_us(s, cfg) for s in (_platforms((cubes,), sink=0.001), _pairs(cubes)))
    assert plate / n < ratio * pairs / m
