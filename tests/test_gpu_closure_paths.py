"""Which kernels a closure system takes, and systems that do not fit one block's shared
memory and have too few closures for the grid, against the oracle (0 ULP).

The tuning's "one block" and "grid" are the forms that keep their vectors in global
memory; by size, systems that fit are solved in shared memory.
"""
import numpy as np
import pytest

from mechanic_b200 import abi, learned, physics, scenes
from mechanic_b200.physics import GpuPhysics, GpuPhysicsConfig

from test_gpu_closure_block import MIXES, _mix
from test_gpu_closure_pcg import _run
from test_gpu_mechanism import _compare, _pair

pytestmark = pytest.mark.gpu


def _kernels(scene, cfg, mode):
    prev = physics.set_tuning(physics.TUNE_CLOSURE_GRID, mode)
    try:
        gpu = GpuPhysics(scene, cfg, capacities={"pair_capacity": 1 << 18})
    finally:
        physics.set_tuning(physics.TUNE_CLOSURE_GRID, max(prev, 0))
    gpu.dispatch_tick(1)
    gpu.wait()
    n = gpu.tick_kernel_count()
    gpu.close()
    return n


@pytest.mark.parametrize("mix", list(MIXES))
def test_forced_forms_do_not_take_the_shared_memory_solve(cuda_lib, mix):
    """To a residual, twelve Newton steps are one launch there and two or three each elsewhere; its
    memory holds the reference's loop wherever it holds this one."""
    scene, cfg = _mix(mix), learned.closure_config(max_iterations=12)
    by_size, one_block, grid = (_kernels(scene, cfg, mode) for mode in (0, 1, 2))
    assert one_block >= by_size + 23 and grid >= by_size + 23


def _in_motion(scene, seed=0):
    coords = np.zeros(scene.coordinate_count, abi.MECHANISM_COORDINATE)
    coords["angle"] = np.random.default_rng(seed).normal(0.0, 1e-4, len(coords)).astype(np.float32)
    return coords


def _narrow():   # 214 loops of 16 bodies, 3,210 closure coordinates
    return scenes.bearing_chains(214, 16, seed=3, closure_fraction=1.0, height=20.0, pitch_x=5.0)


def _wide():   # 361 closures of dozens of joints each; the first rows' coordinates are on hundreds of branches
    return scenes.loops_grid(20, 20, 1)


@pytest.mark.parametrize("make", [_narrow, _wide], ids=["narrow", "wide"])
def test_reference_loop_of_systems_that_do_not_fit_bitexact(cuda_lib, make):
    scene = make()
    assert scene.closure_count < 512
    gpu, orc = _pair(scene, GpuPhysicsConfig())
    coords = _in_motion(scene)
    gpu.initialize_mechanism_coordinates(coords)
    orc.set_coordinates(coords)
    for tick in (1, 2, 3):
        rb = _compare(gpu, orc, tick, "does not fit")
    assert rb.closure_iterations > 0   # unconverged steps: columns, long runs and rounds
    gpu.close()


@pytest.mark.parametrize("precond", [abi.PRECOND_BLOCK_JACOBI, abi.PRECOND_DIAGONAL], ids=["loop_blocks", "diagonal"])
@pytest.mark.parametrize("make", [_narrow, _wide], ids=["narrow", "wide"])
def test_pcg_of_systems_that_do_not_fit_bitexact(cuda_lib, make, precond):
    scene, cfg = make(), learned.closure_config(max_iterations=12, preconditioner=precond)
    assert _kernels(scene, cfg, 0) == _kernels(scene, cfg, 1)
    _run(scene, cfg, 2, coords=_in_motion(scene))


def test_block_solve_of_many_closures_bitexact(cuda_lib):
    """600 loops of three bodies, above the closures from which the rest takes the grid."""
    scene = scenes.bearing_chains(600, 3, seed=5, closure_fraction=1.0, height=0.5)
    gpu, orc = _pair(scene, GpuPhysicsConfig())
    for tick in (1, 2, 3):
        _compare(gpu, orc, tick, "600 loops")
    cfg = learned.closure_config(max_iterations=12)
    assert _kernels(scene, cfg, 0) < _kernels(scene, cfg, 2)
    _run(scene, cfg, 3)
