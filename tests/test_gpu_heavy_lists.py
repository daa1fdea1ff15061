"""Heavy contact ticks at each number of lanes that the split solve gives a body's list
of contacts: 4, 8 and 16 lanes, and the whole warp above 64 entries per body."""
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cubes,box,low,high", [(1500, 2.7, 2, 8), (900, 1.4, 8, 24), (500, 0.8, 24, 64),
                                                (260, 0.1, 66, 200)])
def test_lists_of_each_length_bitexact(cuda_lib, cubes, box, low, high):
    gpu, orc = make_pair(scenes.falling_cubes(cubes, seed=5, box=box), GpuPhysicsConfig())
    for tick in (1, 2):
        compare_tick(gpu, orc, tick, check_tree=False)
        assert low * cubes < gpu.read_last_tick().active_contact_count < high * cubes
    gpu.close()
