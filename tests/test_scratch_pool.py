"""The query calls' scratch memory: calls on several streams and threads, calls recorded in a
CUDA graph, and scenes that come and go (the pool goes with the last one)."""
import threading

import numpy as np
import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
from parity import assert_bitwise, to_np

pytestmark = pytest.mark.gpu

FIELDS = ["valid", "p", "n", "uv", "d", "prim_id"]


def _scene(level=3):
    return Scene(*W.icosphere(level, amplitude=0.2, seed=1), 3, device=0, build_snch=False)


@pytest.mark.parametrize("n", [1, 33, 20_000])
def test_threads_streams_and_graphs_give_the_same_answers(n):
    s = _scene()
    q = torch.as_tensor(W.uniform_points(n, 3, seed=n)).cuda()
    want = to_np(s.closest_point(q))
    got = [None] * 4

    def work(k):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for _ in range(8):
                rec = s.closest_point(q)
            st.synchronize()
        got[k] = to_np(rec)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in got:
        assert_bitwise(g, want, FIELDS, "thread ")

    out = s.alloc_cp(n)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s.closest_point(q, out=out)
    out.d.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert_bitwise(to_np(out), want, FIELDS, "graph ")


def test_pool_goes_with_the_last_scene_and_comes_back():
    q = torch.as_tensor(W.uniform_points(5000, 3, seed=2)).cuda()
    a = _scene(2)
    want = to_np(a.closest_point(q))
    b = _scene(2)
    a.close()
    assert_bitwise(to_np(b.closest_point(q)), want, FIELDS, "second scene ")
    b.close()
    c = _scene(2)
    assert_bitwise(to_np(c.closest_point(q)), want, FIELDS, "after the pool went ")
    assert np.all(want["valid"])
