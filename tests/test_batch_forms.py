"""Batched steps in every form of their launch: one kind alone or several, queries in the
caller's order or sorted, few queries (few lanes per warp) and many, padding slots and bad
scene indices among them; each answer equal to the single-scene call in the same form."""
import numpy as np
import pytest
import torch

from gquery_b200 import _lib as L
from gquery_b200 import workloads as W
from gquery_b200.batch import SKIP, SceneBatch
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scenes():
    return {2: [Scene(*W.star_polyline(m, seed=m), 2, device=0) for m in (70, 900, 5000)],
            3: [Scene(*W.icosphere(k, amplitude=0.2, seed=k), 3, device=0) for k in (2, 3, 4)]}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [3, 1000, 40_000])
@pytest.mark.parametrize("kinds", ["cp", "ray", "cp ray", "cp ray sil"])
def test_rays_and_ordered_closest_points_equal_single_calls(scenes, dim, n, kinds):
    ss = scenes[dim]
    rng = np.random.default_rng(n)
    ids = rng.integers(0, len(ss), n).astype(np.int32)
    ids[::7] = SKIP
    bad = n > 3
    if bad:
        ids[1] = len(ss)
    q = torch.as_tensor(W.uniform_points(n, dim, seed=3).T.copy()).cuda()
    o, d = (torch.as_tensor(x.T.copy()).cuda() for x in W.rays(n, dim, seed=4))
    r = torch.rand(n, device=q.device) * 4
    t = torch.as_tensor(ids).cuda()
    for cp_form in ("exact", "split"):
        b = SceneBatch(ss, n, cp_variant=cp_form, sil_variant="warp")
        res = b.run(cp=(q, t) if "cp" in kinds else None, ray=(o, d, t, r) if "ray" in kinds else None,
                    sil=(q, t) if "sil" in kinds else None)
        torch.cuda.synchronize()
        assert bool(b.device_error() & L.BATCH_ERR_SCENE) == bad
        for k, s in enumerate(ss):
            at = np.nonzero(ids == k)[0]
            if at.size == 0:
                continue
            sel = torch.as_tensor(at).cuda()
            col = lambda x: x[:, sel].contiguous()  # noqa: E731
            if "ray" in kinds:
                want = to_np(s.intersect(col(o), col(d), r[sel].contiguous(), variant="wide8"))
                assert_bitwise({f: x[..., at] for f, x in to_np(res.ray).items()}, want, list(want), f"ray {k} ")
            if "cp" in kinds:  # a walk past the hand-over budget may keep another primitive at a tie
                want = to_np(s.closest_point(col(q), variant="exact"))
                got = {f: x[..., at] for f, x in to_np(res.cp).items()}
                assert_bitwise(got, want, list(want) if cp_form == "exact" else ["valid", "d"], f"cp {k} ")
            if "sil" in kinds:
                want = to_np(s.closest_silhouette(col(q), variant="warp"))
                assert_bitwise({f: x[..., at] for f, x in to_np(res.sil).items()}, want, list(want), f"sil {k} ")
