"""The default ray walk over the 8-wide nodes against the per-lane walk it stands in for, bit
for bit: a stack limit at the compiled size keeps a scene's rays on the per-lane walk.
Rays with zero, tiny and huge direction components, along box faces, with and without
r_max, on meshes with repeated faces (exact ties) and open polylines; call sizes around a
warp and around the number of rays the GPU holds."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu

CAP = 96  # GQ_STACK_WIDE: limits nothing


def _scene(kind):
    if kind == "mesh":
        v, f = W.icosphere(4, amplitude=0.2, seed=3)
        f = np.concatenate([f, f[100:400]]).astype(np.int32)
    elif kind == "box":  # axis-aligned faces: edges and faces on box planes
        k = np.arange(9, dtype=np.float32) / 4 - 1
        x, y = (a.reshape(-1) for a in np.meshgrid(k, k))
        v = np.concatenate([np.stack([x, y, np.full_like(x, z)], 1) for z in (-1, 1)]).astype(np.float32)
        i = np.array([a * 9 + b for a in range(8) for b in range(8)])
        f = np.concatenate([np.stack([i, i + 1, i + 9], 1), np.stack([i + 1, i + 10, i + 9], 1)])
        f = np.concatenate([f, f + 81]).astype(np.int32)
    else:
        v, f = W.star_polyline(3000, seed=2)
        f = np.concatenate([f[:2500], f[200:300]]).astype(np.int32)
    return Scene(v, f, v.shape[1], device=0, build_snch=False), v


def _rays(v, n, seed):
    rng = np.random.default_rng(seed)
    dim = v.shape[1]
    o = rng.uniform(-2, 2, (n, dim))
    d = rng.standard_normal((n, dim))
    k = rng.integers(0, 8, n)
    d[k == 1] = np.eye(dim)[rng.integers(0, dim, n)][k == 1]         # along an axis
    d[k == 2, 0] = 0.0
    d[k == 3] *= 1e-20
    d[k == 4] *= 1e12
    d[k == 5] = (v[rng.integers(0, len(v), n)] - o)[k == 5]          # at a vertex
    o[k == 6] = v[rng.integers(0, len(v), n)][k == 6]                # from a vertex
    d[(k == 7) & (rng.random(n) < 0.1)] = 0.0
    return (torch.as_tensor(x.astype(np.float32)).cuda() for x in (o, d))


@pytest.mark.parametrize("kind", ["mesh", "box", "line"])
@pytest.mark.parametrize("n", [1, 31, 33, 5003, 300_007])
def test_default_rays_equal_the_per_lane_walk(kind, n):
    s, v = _scene(kind)
    fields = ["valid", "p", "n", "t" if s.dim == 2 else "uv", "d", "prim_id", "on_boundary"]
    o, d = _rays(v, n, n)
    r = torch.rand(n, device=o.device) * 3
    for r_max in (float("inf"), r):
        for a, b in ((o, d), (o.t().contiguous(), d.t().contiguous())) if n > 3 else ((o.t(), d.t()),):
            s.set_stack_limit(CAP)
            want = to_np(s.intersect(a, b, r_max, variant="wide8"))
            s.set_stack_limit(0)
            assert_bitwise(to_np(s.intersect(a, b, r_max, variant="wide8")), want, fields, f"{kind} {n} ")
            assert_bitwise(to_np(s.intersect(a, b, r_max, variant="wide8", sort=False)), want, fields, f"{kind} {n} ")
    assert s.device_error() == 0
