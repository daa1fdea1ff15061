"""Sorts of at most 4,096 keys by rank: stable order over ties, digits above the
sorted bits ignored, odd counts, and pair lists on both sides of the limit."""
import numpy as np
import pytest

from mechanic_b200 import scenes
from mechanic_b200.physics import GpuPhysicsConfig

from test_gpu_parity import compare_tick, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 24, 39, 63])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 4095, 4096])
def test_rank_sort_is_the_stable_sort(cuda_lib, n, bits):
    import torch
    from mechanic_b200 import ops
    rng = np.random.default_rng(n * 64 + bits)
    keys = rng.integers(0, 1 << 63, n, dtype=np.uint64)   # bits above the sorted ones too
    keys[rng.random(n) < 0.4] = keys[0]
    vals = rng.permutation(n).astype(np.uint32)
    k_out, v_out = ops.sort_keys(torch.from_numpy(keys.view(np.int64)).cuda(),
                                 torch.from_numpy(vals.view(np.int32)).cuda(), key_bits=bits)
    passes = (bits + 7) // 8
    order = np.argsort(keys & np.uint64((1 << (8 * passes)) - 1), kind="stable")
    assert np.array_equal(k_out.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(v_out.cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("cubes", [500, 1200, 1500, 4000])
def test_pair_lists_around_the_limit(cuda_lib, cubes):
    """Cubes packed into one box: a few hundred to tens of thousands of pairs."""
    gpu, orc = make_pair(scenes.falling_cubes(cubes, seed=9, box=2.6), GpuPhysicsConfig())
    for tick in (1, 2):
        compare_tick(gpu, orc, tick, check_tree=False)
