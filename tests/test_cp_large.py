"""3D closest points in calls of 4,194,304 and more, which fetch nothing ahead and, sorted, start the
tiles in the middle of the scene first: bit for bit what calls of a few thousand give for
the same tiles, and what the query order passed in by the caller gives; a last tile that
is not full.  On geometry whose bounding cylinders are flat, bound nothing, far from the
origin or tiny, with leaves larger than a run, and on device-built trees (no runs)."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu

FIELDS = ["valid", "p", "n", "uv", "d", "prim_id"]
N = (1 << 22) + 5


def _mesh(kind):
    v, f = W.icosphere(4, amplitude=0.3, seed=5)
    if kind == "slivers":
        v = v * np.array([1.0, 1.0, 1e-4], np.float32)
        f = np.concatenate([f, np.stack([f[:50, 0], f[:50, 0], f[:50, 1]], 1)]).astype(np.int32)
    elif kind == "far":
        v = v + np.float32(300.0)
    elif kind == "tiny":
        v = v * np.float32(1e-6)
    elif kind == "stacked":  # leaves larger than a run
        f = np.concatenate([f, np.repeat(f[:20], 30, 0)]).astype(np.int32)
    return np.ascontiguousarray(v, np.float32), f


@pytest.mark.parametrize("kind,build", [("plain", {}), ("plain", dict(gpu_build=True)), ("plain", dict(max_prims_in_node=1)),
                                        ("slivers", {}), ("far", {}), ("tiny", {}), ("stacked", dict(max_prims_in_node=40))])
def test_large_calls(kind, build):
    v, f = _mesh(kind)
    s = Scene(v, f, 3, device=0, build_snch=False, **build)
    rng = np.random.default_rng(7)
    mid, half = (v.max(0) + v.min(0)) / 2, (v.max(0) - v.min(0)).max()
    q = mid + rng.uniform(-1.0, 1.0, (N, 3)) * half
    q[::3] = v[rng.integers(0, len(v), len(q[::3]))] + rng.normal(0, 0.01, (len(q[::3]), 3)) * half
    q = torch.as_tensor(q.astype(np.float32)).cuda()
    plain = to_np(s.closest_point(q, variant="coherent", sort=False))
    assert plain["valid"].all()
    tail = N - N % 32 - 32  # a full tile and the short one
    for at, n in ((0, 64), (32 * 777, 4096), (tail, N - tail)):
        part = to_np(s.closest_point(q[at:at + n], variant="coherent", sort=False))
        assert_bitwise({k: plain[k][..., at:at + n] for k in FIELDS}, part, FIELDS, f"{kind} {at} ")
    tiles = to_np(s.closest_point(q, variant="coherent", sort=True))
    given = to_np(s.closest_point(q, variant="coherent", order=s.order(q)))
    assert_bitwise(tiles, given, FIELDS, f"{kind} sorted ")
    exact = to_np(s.closest_point(q[tail:], variant="exact"))
    # both closest points are formed with a few roundings of the coordinates' size
    tol = 16 * 2.0 ** -24 * float(np.abs(v).max() + q.abs().max().item())
    assert np.abs(exact["d"].astype(np.float64) - plain["d"][tail:]).max() <= tol
    assert s.device_error() == 0
