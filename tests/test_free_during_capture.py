"""Scenes and batches that are freed while a graph is being captured (by a garbage collector, say)
leave the capture and its replays alone."""
import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.batch import SceneBatch
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_free_during_capture(dim):
    v, f = W.icosphere(3, amplitude=0.2, seed=1) if dim == 3 else W.star_polyline(500, seed=1)
    s, other, third = (Scene(v, f, dim, device=0) for _ in range(3))
    q = torch.as_tensor(W.uniform_points(5000, dim, seed=1)).cuda()
    ids = torch.zeros(5000, dtype=torch.int32, device=q.device)
    want = to_np(s.closest_point(q))
    b, gone = SceneBatch([s], 5000), SceneBatch([third], 5000)
    want_b = to_np(b.run(cp=(q, ids)).cp)
    gone.run(cp=(q, ids))
    other.closest_point(q)
    out, out_b = s.alloc_cp(5000), b.alloc(5000, 0, 0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s.closest_point(q, out=out)
        other.close()
        gone.close()
        third.close()
        b.run(cp=(q, ids), out=out_b)
    out.d.zero_()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert_bitwise(to_np(out), want, ["valid", "d", "prim_id"], "scene ")
    assert_bitwise(to_np(out_b.cp), want_b, ["valid", "d", "prim_id"], "batch ")
    assert np.all(want["valid"])
