"""Default rays at the ends of the float range: directions up to the largest float and down to
subnormal ones, with unequal and infinite components, origins far away, tiny scenes; alone
and in a batch.  Against the per-lane walk bit for bit (a stack limit at the compiled size
keeps a scene's rays on it) and, in which rays hit, against the reference's order."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.batch import SceneBatch
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu

CAP = 96  # GQ_STACK_WIDE: limits nothing
LENGTHS = [1e-44, 1e-38, 1e-30, 1e-20, 1e20, 1e30, 8e37, 1e38, 3e38]


def _rays(v, n, dim, size):
    """Towards points of the shape, of every length, some along an axis, some with an infinite
    component."""
    rng = np.random.default_rng(n)
    o = rng.uniform(-2, 2, (n, dim)) * size
    at = v[rng.integers(0, len(v), n)].astype(np.float64) * 0.9
    o[::5] = at[::5] * rng.uniform(0, 1, (len(o[::5]), 1))  # from inside
    d = at - o
    d[::7] = np.eye(dim)[rng.integers(0, dim, len(d[::7]))]
    d /= np.abs(d).max(1, keepdims=True)
    d *= np.array(LENGTHS)[np.arange(n) % len(LENGTHS), None]
    d = d.astype(np.float32)
    d[3::11, 0] = np.inf
    d[4::11, 1] = -np.inf
    o[5::13] += 1e6 * size
    return (torch.as_tensor(np.ascontiguousarray(x.T, np.float32)).cuda() for x in (o, d))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("size", [1.0, 1e-12])
def test_directions_over_the_float_range(dim, size):
    v, f = W.icosphere(4, amplitude=0.2, seed=2) if dim == 3 else W.star_polyline(2000, seed=2)
    v = (v * size).astype(np.float32)
    s = Scene(v, f, dim, device=0, build_snch=False)
    fields = ["valid", "p", "n", "t" if dim == 2 else "uv", "d", "prim_id", "on_boundary"]
    b = SceneBatch([s], 5003)
    for n in (31, 5003):
        o, d = _rays(v, n, dim, size)
        got = to_np(s.intersect(o, d))
        s.set_stack_limit(CAP)
        want = to_np(s.intersect(o, d, variant="wide8"))
        s.set_stack_limit(0)
        assert_bitwise(got, want, fields, f"{n} ")
        normal = (d.abs().amax(0) >= torch.finfo(torch.float32).tiny).cpu().numpy()
        exact = to_np(s.intersect(o, d, variant="exact"))
        assert np.array_equal(got["valid"][normal], exact["valid"][normal])
        if size == 1.0 and n > 31:  # long ones hit
            assert got["valid"][np.isin(np.arange(n) % len(LENGTHS), (6, 7))].mean() > 0.3
        res = to_np(b.run(ray=(o, d, torch.zeros(n, dtype=torch.int32, device=o.device))).ray)
        torch.cuda.synchronize()
        assert_bitwise(res, want, fields, f"batch {n} ")
    assert s.device_error() == 0 and b.device_error() == 0
