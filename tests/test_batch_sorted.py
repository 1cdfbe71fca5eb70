"""Batched steps of enough queries of a kind to be sorted where the order does not change their
answers: each answer equal to the single-scene call in the same form."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.batch import SKIP, SceneBatch
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [(1 << 15) - 1, (1 << 15) + 33])
def test_around_the_line(dim, n):
    ss = [Scene(*(W.star_polyline(m, seed=m) if dim == 2 else W.icosphere(m, amplitude=0.2, seed=m)), dim, device=0)
          for m in ((70, 900) if dim == 2 else (2, 3))]
    ids = np.random.default_rng(n).integers(0, 2, n).astype(np.int32)
    ids[::7] = SKIP
    q = torch.as_tensor(W.uniform_points(n, dim, seed=3).T.copy()).cuda()
    o, d = (torch.as_tensor(x.T.copy()).cuda() for x in W.rays(n, dim, seed=4))
    t = torch.as_tensor(ids).cuda()
    b = SceneBatch(ss, n, cp_variant="exact", ray_variant="exact", sil_variant="warp")
    res = b.run(cp=(q, t), ray=(o, d, t), sil=(q, t))
    torch.cuda.synchronize()
    assert b.device_error() == 0
    for k, s in enumerate(ss):
        at = np.nonzero(ids == k)[0]
        col = lambda x: x[:, torch.as_tensor(at).cuda()].contiguous()  # noqa: E731
        for name, got, want in (("cp", res.cp, s.closest_point(col(q), variant="exact")),
                                ("ray", res.ray, s.intersect(col(o), col(d), variant="exact")),
                                ("sil", res.sil, s.closest_silhouette(col(q), variant="warp"))):
            w = to_np(want)
            assert_bitwise({f: x[..., at] for f, x in to_np(got).items()}, w, list(w), f"{name} {k} ")
