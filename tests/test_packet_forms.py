"""The two forms of the 3D warp-coherent closest point (few queries: pairs of a triangle and a
lane; many queries: bounding cylinders before the triangle tests) against each other and
against the exact walk, on geometry where the bounds can go wrong: slivers and zero-area
triangles (which bound nothing), meshes far from the origin and tiny ones, leaves larger
than a run, device-built trees."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu

FIELDS = ["valid", "p", "n", "uv", "d", "prim_id"]
DENSE_FROM = 1 << 21  # queries of a call from which the dense form runs
EPS32 = 2.0 ** -24


def _mesh(kind):
    v, f = W.icosphere(4, amplitude=0.3, seed=5)
    if kind == "slivers":
        v = v * np.array([1.0, 1.0, 1e-4], np.float32)
        f = np.concatenate([f, np.stack([f[:50, 0], f[:50, 0], f[:50, 1]], 1)]).astype(np.int32)
    elif kind == "far":
        v = v + np.float32(300.0)
    elif kind == "tiny":
        v = v * np.float32(1e-6)
    return np.ascontiguousarray(v, np.float32), f


def _queries(v, n, seed):
    rng = np.random.default_rng(seed)
    mid, half = (v.max(0) + v.min(0)) / 2, (v.max(0) - v.min(0)).max()
    box = mid + rng.uniform(-1.0, 1.0, (n, 3)) * half
    near = v[rng.integers(0, len(v), n)] + rng.normal(0, 0.01, (n, 3)) * half
    return np.where(rng.random((n, 1)) < 0.5, box, near).astype(np.float32)


@pytest.mark.parametrize("kind,build", [("plain", {}), ("plain", dict(gpu_build=True)), ("plain", dict(max_prims_in_node=1)),
                                        ("slivers", {}), ("far", {}), ("tiny", {})])
def test_forms_agree_bitwise_and_with_exact(kind, build):
    v, f = _mesh(kind)
    s = Scene(v, f, 3, device=0, build_snch=False, **build)
    sizes = (33, 64, 4099)
    q = torch.as_tensor(_queries(v, DENSE_FROM, 7)).cuda()
    dense = to_np(s.closest_point(q, variant="coherent", sort=False))  # tiles of 32 in input order
    for n in sizes:
        part = to_np(s.closest_point(q[:n], variant="coherent", sort=False))
        whole = n - n % 32  # the last, shorter tile walks alone here
        assert_bitwise({k: part[k][..., :whole] for k in FIELDS}, {k: dense[k][..., :whole] for k in FIELDS}, FIELDS,
                       f"{kind} {n} ")
    exact = to_np(s.closest_point(q[:4099], variant="exact"))
    assert np.array_equal(exact["valid"], dense["valid"][:4099])
    # both closest points are formed with a few roundings of the coordinates' size
    tol = 16 * EPS32 * float(np.abs(v).max() + q.abs().max().item())
    assert np.abs(exact["d"].astype(np.float64) - dense["d"][:4099]).max() <= tol


@pytest.mark.parametrize("segments,large", [(3, 1 << 16), (300, 1 << 16), (20_000, 1 << 21)])
def test_2d_forms_agree_bitwise(segments, large):
    """The 2D walk with and without its children brought ahead: by call size, on small polylines
    from 65,536 points on, on large ones from 2,097,152."""
    v, e = W.star_polyline(segments, seed=segments)
    s = Scene(v, e, 2, device=0, build_snch=False)
    q = torch.as_tensor(W.uniform_points(large + 5, 2, seed=8)).cuda()
    fields = ["valid", "p", "n", "t", "d", "prim_id"]
    whole = to_np(s.closest_point(q, variant="coherent", sort=False))
    for n in (64, 4096):
        part = to_np(s.closest_point(q[:n], variant="coherent", sort=False))
        assert_bitwise(part, {k: whole[k][..., :n] for k in fields}, fields, f"{segments} {n} ")
