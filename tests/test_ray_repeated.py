"""Default rays on shapes that list their faces several times: equal hits within one leaf, whose
order decides, and in different leaves, where the per-lane walk does.  Against that walk bit
for bit (a stack limit at the compiled size keeps a scene's rays on it); alone and in a
batch, on host-built and device-built trees."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.batch import SceneBatch
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu

CAP = 96  # GQ_STACK_WIDE: limits nothing


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("times", [2, 3, 7, 40])
@pytest.mark.parametrize("build", [{}, dict(gpu_build=True), dict(max_prims_in_node=1)])
def test_repeated_faces(dim, times, build):
    v, f = W.icosphere(3, amplitude=0.2, seed=2) if dim == 3 else W.star_polyline(800, seed=2)
    f = np.concatenate([f if k % 2 == 0 else f[::-1] for k in range(times)]).astype(np.int32)
    if times == 3:
        f[len(f) // 2:] = f[len(f) // 2:, ::-1]  # the other orientation: equal up to rounding
    if times == 40 and "max_prims_in_node" in build:
        pytest.skip("forty equal boxes one below the other")
    s = Scene(v, f, dim, device=0, build_snch=False, **build)
    fields = ["valid", "p", "n", "t" if dim == 2 else "uv", "d", "prim_id", "on_boundary"]
    b = SceneBatch([s], 5003)
    for n in (31, 5003):
        o, d = (torch.as_tensor(x.T.copy()).cuda() for x in W.rays(n, dim, seed=n))
        r = torch.linspace(0, 4, n, device=o.device)
        for r_max in (float("inf"), r):
            got = to_np(s.intersect(o, d, r_max))
            s.set_stack_limit(CAP)
            want = to_np(s.intersect(o, d, r_max, variant="wide8"))
            s.set_stack_limit(0)
            assert_bitwise(got, want, fields, f"{times} {n} ")
            ids = torch.zeros(n, dtype=torch.int32, device=o.device)
            res = to_np(b.run(ray=(o, d, ids) + ((r,) if r_max is r else ())).ray)
            torch.cuda.synchronize()
            assert_bitwise(res, want, fields, f"batch {times} {n} ")
    assert s.device_error() == 0 and b.device_error() == 0
