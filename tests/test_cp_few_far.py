"""Calls of fewer than 32 closest points far away from the shape (where the rounding of the
distances spans it) and with single non-finite or overflowing coordinates, bit for bit as the
walk in the reference's order."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("prims", [1, 2, 5120])
def test_far_and_nonfinite_points(dim, prims):
    v, f = W.icosphere(4, amplitude=0.2, seed=2) if dim == 3 else W.star_polyline(5120, seed=2)
    s = Scene(v, f[:prims], dim, device=0, build_snch=False)
    q = np.concatenate([W.sphere_dirs(20, dim, seed=k) * 10.0 ** k for k in range(0, 9)]).astype(np.float32)
    odd = W.uniform_points(40, dim, seed=1)
    odd[np.arange(40), np.arange(40) % dim] = np.resize(np.float32([np.nan, np.inf, -np.inf, 1e19, 1e30, -3e38]), 40)
    q = torch.as_tensor(np.concatenate([q, odd])).cuda()
    exact = to_np(s.closest_point(q, variant="exact"))
    for at in range(0, q.shape[0], 20):
        got = to_np(s.closest_point(q[at:at + 20].t().contiguous(), variant="coherent"))
        assert_bitwise(got, {k: x[..., at:at + 20] for k, x in exact.items()}, list(got), f"{at} ")
    assert s.device_error() == 0
