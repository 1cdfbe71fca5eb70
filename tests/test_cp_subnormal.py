"""3D closest points whose squared distances are below the smallest normal number: the cylinder
bounds leave no nearer triangle out.  The error of a distance is then that of a subnormal
square, sqrt(4 * 2^-149), beside some roundings of the coordinates."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-16, 1e-17, 1e-18])
@pytest.mark.parametrize("n", [4099, (1 << 22) + 5])
def test_subnormal_squares(scale, n):
    v, f = W.icosphere(4, amplitude=0.2, seed=3)
    v = (v.astype(np.float64) * scale).astype(np.float32)
    s = Scene(v, f, 3, device=0, build_snch=False)
    rng = np.random.default_rng(1)
    m = 20_000
    q = v[rng.integers(0, len(v), m)] + rng.normal(0, 1.0, (m, 3)) * 10.0 ** rng.uniform(-23, -18, (m, 1))
    q = torch.as_tensor(np.resize(q.astype(np.float32), (n, 3))).cuda()
    got = s.closest_point(q, variant="coherent")
    want = s.closest_point(q[:m], variant="exact")
    k = min(n, m)
    tol = 16 * 2.0 ** -24 * float(np.abs(v).max() + 1e-18) + 2 * (4 * 2.0 ** -149) ** 0.5
    worst = (got.d[:k].double() - want.d[:k].double()).abs().max().item()
    assert worst <= tol, (worst, tol)
    assert bool(got.valid.all())
