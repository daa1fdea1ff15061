"""Collider trees at the edges of the refit's chunks (32 leaves), super-chunks (1,024) and
block forms (one super-chunk, one block per SM, more blocks than SMs), against the oracle."""
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cubes,box", [(1, 1.0), (2, 0.3), (3, 0.3), (31, 1.0), (32, 1.0), (33, 1.0), (65, 1.5),
                                       (1023, 4.0), (1024, 4.0), (1025, 4.0), (2049, 6.0), (151552, 60.0),
                                       (151553, 60.0)])
def test_tree_of_size_bitexact(cuda_lib, cubes, box):
    gpu, orc = make_pair(scenes.falling_cubes(cubes, seed=cubes, box=box), GpuPhysicsConfig())
    for tick in (1, 2):
        compare_tick(gpu, orc, tick)
    gpu.close()
