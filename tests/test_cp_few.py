"""Calls of fewer than 32 closest points (one query per warp) against the per-lane walk in the
reference's order, bit for bit in every field: uniform, on and near vertices and at the
centre of the shape, on plain, shifted and snapped geometry (exact ties, coplanar and zero-area
primitives), on single primitives and on device-built trees."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu


def _shape(dim, size, kind):
    v, f = W.icosphere(size, amplitude=0.2, seed=size) if dim == 3 else W.star_polyline(20 * 4 ** size, seed=size)
    if kind == "shifted":
        v = v + 100
    elif kind == "snapped":
        v = np.round(v * 8) / 8
    elif kind == "single":
        f = f[:1]
    return v.astype(np.float32), f


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("size,kind,build", [(2, "plain", {}), (5, "plain", {}), (5, "shifted", {}), (4, "snapped", {}),
                                             (1, "single", {}), (5, "plain", dict(gpu_build=True))])
def test_few_queries_equal_the_reference_order(dim, size, kind, build):
    v, f = _shape(dim, size, kind)
    s = Scene(v, f, dim, device=0, build_snch=False, **build)
    rng = np.random.default_rng(size)
    lo, hi = v.min(0), v.max(0)
    pick = lambda n: v[rng.integers(0, len(v), n)]  # noqa: E731
    q = np.concatenate([rng.uniform(2 * lo - hi, 2 * hi - lo, (300, dim)), pick(100), pick(200) + rng.normal(0, 0.01, (200, dim)),
                        (lo + hi)[None] / 2, [[np.nan] * dim, [np.inf] * dim]]).astype(np.float32)
    q = torch.as_tensor(q).cuda()
    exact = to_np(s.closest_point(q, variant="exact"))
    at = 0
    while at < q.shape[0]:
        n = min(int(rng.choice([1, 2, 5, 31])), q.shape[0] - at)
        part = q[at:at + n].t().contiguous() if n <= dim else q[at:at + n]
        got = to_np(s.closest_point(part, variant="coherent"))
        assert_bitwise(got, {k: x[..., at:at + n] for k, x in exact.items()}, list(got), f"{at} {n} ")
        at += n
    assert s.device_error() == 0
