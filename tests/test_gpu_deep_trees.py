"""Deep mechanisms: velocities reconstructed by one block's walk over the depth
levels, against the oracle (0 ULP), and the closure columns of a converged wide
lattice, which the loop itself does not need."""
import numpy as np
import pytest

from mechanic_b200 import abi, learned, scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_mechanism import _compare, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains,links", [(1, 18), (3, 17), (1025, 18), (1500, 20)])
def test_level_walk_bitexact(cuda_lib, chains, links):
    """Levels of 1 body, of one round of 1,024 and of more; 17 links (16 levels) keep the launches."""
    gpu, orc = _pair(scenes.bearing_chains(chains, links, seed=links, closure_fraction=0.0, height=0.6),
                     GpuPhysicsConfig())
    for tick in range(1, 4):
        _compare(gpu, orc, tick, f"{chains} x {links}")


def test_columns_of_a_converged_lattice(cuda_lib):
    scene = scenes.loops_grid(20, 20, 3)
    got = []
    for cfg in (GpuPhysicsConfig(), learned.closure_config(preconditioner=abi.PRECOND_DIAGONAL)):
        gpu, _ = _pair(scene, cfg)
        gpu.dispatch_tick(1)
        assert gpu.read_last_tick().error_flags == 0
        got.append(gpu.closure_slots()[:3])
    for a, b in zip(*got):
        np.testing.assert_array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))
