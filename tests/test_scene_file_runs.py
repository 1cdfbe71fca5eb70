"""A scene file whose pair records name smaller runs than this build collapses (the larger ones
cleared, which the load check accepts): runs without a bounding cylinder are tested as they
are, and the answers are those of the scene that was saved, up to ties."""
import struct

import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import REL_TOL, tie_report, to_np
from test_scene_file import _layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keep", [0, 1, 3, 4])
def test_smaller_runs(keep, tmp_path):
    v, f = W.icosphere(4, amplitude=0.2, seed=6)
    v = v + np.float32(0.7)  # not around the origin
    a = Scene(v, f, 3, device=0, build_snch=False)
    path = tmp_path / "a.gqs"
    a.save(path)
    raw = bytearray(path.read_bytes())
    _, _, st, sz = _layout(bytes(raw))
    cleared = 0
    for at in range(st[0], st[0] + sz[0], 64):
        for c in (56, 60):
            if struct.unpack_from("<I", raw, at + c)[0] >> 24 > keep:
                struct.pack_into("<I", raw, at + c, 0)
                cleared += 1
    assert cleared > 100
    path.write_bytes(bytes(raw))
    junk = torch.rand(1 << 24, device="cuda")  # the loaded scene's memory may have held anything
    del junk
    torch.cuda.empty_cache()
    b = Scene.load(path)
    q = torch.as_tensor(W.uniform_points((1 << 22) + 5, 3, seed=7)).cuda()
    for n in (4099, q.shape[0]):
        rep = tie_report(to_np(b.closest_point(q[:n], variant="coherent")), to_np(a.closest_point(q[:n], variant="coherent")))
        assert rep["valid_mismatch"] == 0 and rep["prim_mismatch_not_tie"] == 0 and rep["max_rel_d"] <= REL_TOL, rep
    assert b.device_error() == 0
