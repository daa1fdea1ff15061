"""The network's launches at their edges: forward passes around 1, 2, 4 and 8 tiles beside one
another per CTA and at several row widths, parameters that are only 4-byte aligned, and training
runs of more steps than one launch takes."""
import pytest
import torch

from mechanic_b200 import ops

from test_gpu_mlp import _data, _params

pytestmark = pytest.mark.gpu

WAVE = 148 * 128   # samples of one tile per SM


@pytest.mark.parametrize("n,cols", [(WAVE, 1), (WAVE + 1, 3), (2 * WAVE + 1, 4), (4 * WAVE, 5), (4 * WAVE + 1, 2),
                                    (8 * WAVE + 129, 4), (17 * WAVE + 5, 1), (1000, 8), (129, 15), (257, 12)])
def test_forward_tiles_and_row_widths(cuda_lib, n, cols):
    """A sample's outputs depend neither on its tile's place nor on the row width: the same
    bits as in calls of 1,000 samples and 16 columns."""
    x = torch.from_numpy(_data(n, seed=n)[0]).cuda()
    p = torch.from_numpy(_params(4)).cuda()
    y = ops.mlp_forward(p, x, y_cols=cols)
    small = torch.cat([ops.mlp_forward(p, part)[:, :cols] for part in x.split(1000)])
    assert y.shape == (n, cols) and torch.equal(y, small)


def test_unaligned_parameters_give_the_same_bits(cuda_lib):
    x, t, w = (torch.from_numpy(a).cuda() for a in _data(3000, seed=5))
    p = torch.from_numpy(_params(5)).cuda()
    shifted = torch.cat([p[:1], p])[1:]   # 4 bytes past an aligned address
    assert shifted.data_ptr() % 16 == 4
    assert torch.equal(ops.mlp_forward(p, x), ops.mlp_forward(shifted, x))
    assert torch.equal(ops.mlp_gradient(p, x, t, w)[0], ops.mlp_gradient(shifted, x, t, w)[0])


@pytest.mark.parametrize("n,steps", [(200, 256), (200, 257), (20000, 300)])
def test_training_in_one_call_or_step_by_step(cuda_lib, n, steps):
    x, t, w = (torch.from_numpy(a).cuda() for a in _data(n, seed=6))
    runs = []
    for per_call in (steps, 1):
        p = torch.from_numpy(_params(6)).cuda()
        m, v = torch.zeros_like(p), torch.zeros_like(p)
        losses = [ops.mlp_train(p, m, v, x, t, w, steps=per_call, batch=n, lr=1e-3, first_step=k)
                  for k in range(0, steps, per_call)]
        runs.append((torch.cat([q.reshape(-1) for q in losses]), p, m, v))
    for one, many in zip(*runs):
        assert torch.equal(one, many)
