"""Silhouettes with radii at, just below and just above the distances of boxes and vertices: the
2D walks compare squared box distances with the largest square whose root is within r_max.
The coherent and one-query-per-warp walks against the exact walk and the brute-force list."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_sil_variant, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,size,n", [(2, 300, 33), (2, 5000, 4099), (3, 3, 4099), (3, 4, 300_001)])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12])
def test_radii_on_the_edge(dim, size, n, scale):
    v, f = W.star_polyline(size, seed=size) if dim == 2 else W.icosphere(size, amplitude=0.3, seed=size)
    s = Scene((v * np.float32(scale)).astype(np.float32), f, dim, device=0)
    x = torch.as_tensor((W.uniform_points(n, dim, seed=5) * np.float32(scale)).astype(np.float32)).cuda()
    d = s.closest_silhouette(x, variant="exact").d
    step = torch.arange(n, device=x.device) % 5
    lo, hi = torch.full_like(d, 0.0), torch.full_like(d, float("inf"))
    r = torch.where(step == 0, d, torch.where(step == 1, torch.nextafter(d, hi), torch.where(
        step == 2, torch.nextafter(d, lo), torch.where(step == 3, 0.5 * d, hi))))
    exact, brute = to_np(s.closest_silhouette(x, r, variant="exact")), to_np(s.closest_silhouette_brute(x, r)) if n < 5000 else None
    for variant in ("coherent", "warp"):
        got = to_np(s.closest_silhouette(x, r, variant=variant))
        assert_sil_variant(exact, got, brute if brute is not None else exact, f"{variant} {scale} ", max_nearer=0.01)
