"""The standalone SAT where the answer's axis is decided late or not at all: parallel boxes
(degenerate cross axes), boxes separated along each of the 15 axes, ties, zero extents and
degenerate frames, all against the oracle's bits."""
import numpy as np
import pytest

import oracle
from mechanic_b200 import scenes

pytestmark = pytest.mark.gpu


def _boxes(center, half, axes):
    n = len(center)
    b = np.zeros((n, 4, 4), np.float32)
    b[:, 0, :3] = center
    b[:, 0, 3], b[:, 1, 3], b[:, 2, 3] = half[:, 0], half[:, 1], half[:, 2]
    b[:, 1, :3], b[:, 2, :3], b[:, 3, :3] = axes[:, 0], axes[:, 1], axes[:, 2]
    return b


@pytest.mark.parametrize("kind", ["parallel", "separated", "flat", "no_frame"])
def test_sat_axis_of_every_kind(cuda_lib, kind):
    import torch
    from mechanic_b200 import ops
    rng = np.random.default_rng(len(kind))
    n = 3000
    frames = [scenes.quat_matrix(scenes.Rng(s).unit_quaternions("q", n)).astype(np.float32).transpose(0, 2, 1)
              for s in (11, 12)]
    half = [rng.uniform(0.05, 0.3, (n, 3)).astype(np.float32) for _ in range(2)]
    delta = rng.uniform(-0.4, 0.4, (n, 3)).astype(np.float32)
    if kind == "parallel":
        frames[1] = frames[0][:, [1, 2, 0]]
        delta[::3] = 0.0   # concentric: every face axis ties with its opposite
    elif kind == "separated":   # pushed apart along a random cross or face axis
        pick = rng.integers(0, 15, n)
        u = frames[0][np.arange(n), np.where(pick < 3, pick, (pick - 6) % 3)]
        v = frames[1][np.arange(n), np.where(pick < 6, pick % 3, (pick - 6) // 3 % 3)]
        axis = np.where((pick < 3)[:, None], u, np.where((pick < 6)[:, None], v, np.cross(u, v)))
        delta = (axis * rng.choice([0.3, 0.5, 0.7], (n, 1))).astype(np.float32)
    elif kind == "flat":
        half[0][:, 1] = 0.0
        half[1][::2] = 0.0
    else:
        frames[1][::2, 1] = 0.0
        frames[0][1::4] = 0.0
        frames[1][1::4] = 0.0   # no axis at all
    a = _boxes(np.zeros((n, 3)), half[0], frames[0])
    b = _boxes(delta, half[1], frames[1])
    out, feat = ops.obb_sat(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    out, feat = out.cpu().numpy(), feat.cpu().numpy().view(np.uint32)
    for i in range(n):
        ref, f = oracle.obb_sat(a[i].reshape(-1), b[i].reshape(-1))
        assert f == feat[i], i
        assert np.array_equal(ref.view(np.uint32), out[i].view(np.uint32)), i
