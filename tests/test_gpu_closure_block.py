"""The closure solves in one block's shared memory, against the oracle (0 ULP).

Closures of unequal length (the columns' order is by falling length), systems
on either side of the serial dot product's 512 coordinates and of a chunk's
1,024, in one block and spread over a cluster of blocks.
"""
import pytest

from mechanic_b200 import abi, learned, scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_closure_pcg import _run
from test_gpu_mechanism import _compare, _pair

pytestmark = pytest.mark.gpu

MIXES = {   # chains, links, closed share
    "one_loop": [(1, 3, 1.0), (3, 5, 0.0)],
    "unequal": [(12, 3, 0.5), (9, 9, 0.7), (15, 5, 0.4), (2, 12, 1.0)],
    "coords_516": [(129, 5, 1.0)],
    "coords_1020_unequal": [(100, 5, 1.0), (70, 9, 0.9), (20, 3, 0.5)],
    "coords_1500": [(375, 5, 1.0)],
}


def _mix(name):
    parts = [scenes.translated(scenes.bearing_chains(n, links, seed=7 + i, closure_fraction=closed, height=0.5),
                               (0.0, 0.0, 40.0 * i)) for i, (n, links, closed) in enumerate(MIXES[name])]
    return parts[0] if len(parts) == 1 else scenes.concatenate(parts)[0]


@pytest.mark.parametrize("mode", ["reference", "loop_blocks", "diagonal"])
@pytest.mark.parametrize("mix", list(MIXES))
def test_block_closure_solve_bitexact(cuda_lib, mix, mode):
    if mode == "reference":
        gpu, orc = _pair(_mix(mix), GpuPhysicsConfig())
        for tick in range(1, 4):
            _compare(gpu, orc, tick, mix)
        return
    precond = abi.PRECOND_DIAGONAL if mode == "diagonal" else abi.PRECOND_BLOCK_JACOBI
    _run(_mix(mix), learned.closure_config(max_iterations=12, preconditioner=precond), 3)
