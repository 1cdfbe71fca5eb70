"""Default rays on scenes whose tree is a single leaf (no nodes at all): a few primitives, many at one
place, device-built ones; alone and in a batch beside larger scenes.  Against the walk in the
reference's order, and the per-lane walk bit for bit."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.batch import SceneBatch
from gquery_b200.scene import Scene
from parity import assert_bitwise, tie_report, to_np

pytestmark = pytest.mark.gpu

CAP = 96  # GQ_STACK_WIDE: limits nothing, keeps the rays on the per-lane walk


def _scene(dim, prims, **build):
    v, f = W.icosphere(1, amplitude=0.2, seed=1) if dim == 3 else W.star_polyline(40, seed=1)
    f = np.tile(f[:1], (40, 1)) if prims == "one place" else f[:prims]
    return Scene(v, np.ascontiguousarray(f, np.int32), dim, device=0, build_snch=False, **build)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("prims,build", [(1, {}), (2, {}), (10, {}), ("one place", {}),
                                         (1, dict(gpu_build=True)), (2, dict(gpu_build=True))])
def test_one_leaf(dim, prims, build):
    s = _scene(dim, prims, **build)
    if prims in (1, "one place"):
        assert s.info["n_wide_nodes"] == 0
    fields = ["valid", "p", "n", "t" if dim == 2 else "uv", "d", "prim_id", "on_boundary"]
    rng = np.random.default_rng(3)
    big = Scene(*(W.icosphere(3, amplitude=0.2, seed=1) if dim == 3 else W.star_polyline(900, seed=1)), dim, device=0,
                build_snch=False)
    b = SceneBatch([s, big], 5003)
    for n in (1, 33, 5003):
        at = s.vertices_host[s.indices_host[rng.integers(0, len(s.indices_host), n)]].mean(1)
        o = rng.uniform(-2, 2, (n, dim))
        d = at + rng.normal(0, 0.05, (n, dim)) - o
        o, d = (torch.as_tensor(x.astype(np.float32).T.copy()).cuda() for x in (o, d))
        r = torch.rand(n, device=o.device) * 3
        ids = torch.arange(n, dtype=torch.int32, device=o.device) % 2
        for r_max in (float("inf"), r):
            got = to_np(s.intersect(o, d, r_max))
            assert n < 33 or got["valid"].any()
            rep = tie_report(got, to_np(s.intersect(o, d, r_max, variant="exact")))
            assert rep["valid_mismatch"] == 0 and rep["prim_mismatch_not_tie"] == 0, rep
            s.set_stack_limit(CAP)
            want = to_np(s.intersect(o, d, r_max, variant="wide8"))
            s.set_stack_limit(0)
            assert_bitwise(got, want, fields, f"{prims} {n} ")
            res = to_np(b.run(ray=(o, d, ids) + ((r,) if r_max is r else ())).ray)
            torch.cuda.synchronize()
            assert_bitwise({k: x[..., 0:n:2] for k, x in res.items()}, {k: x[..., 0:n:2] for k, x in want.items()}, fields,
                           f"batch {prims} {n} ")
    assert s.device_error() == 0 and b.device_error() == 0
