"""The first launches of every form, made by several host threads at once: the number of resident
blocks is published in one step.  By the sources (a thread that sees half of it shows only
by chance), and in a fresh process on the GPU."""
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
DEVICE = ROOT / "gquery_b200" / "csrc" / "device"

WORK = """
import sys, threading
sys.path[:0] = [{root!r}, {tests!r}]
import numpy as np, torch
from gquery_b200 import workloads as W
from gquery_b200.batch import SceneBatch
from gquery_b200.scene import Scene
from parity import to_np
shapes = {{3: W.icosphere(3, amplitude=0.2, seed=1), 2: W.star_polyline(500, seed=1)}}
scenes = {{d: Scene(*g, d, device=0) for d, g in shapes.items()}}
ins = {{d: (torch.as_tensor(W.uniform_points(5000, d, seed=2)).cuda(), torch.as_tensor(W.sphere_dirs(5000, d)).cuda())
       for d in shapes}}
ids = torch.zeros(5000, dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
start, got = threading.Barrier(8), [None] * 8
def work(k):
    d = 2 + k % 2
    s, (q, v) = scenes[d], ins[d]
    b = SceneBatch([s], 5000)
    with torch.cuda.stream(torch.cuda.Stream()):
        start.wait()
        out = [s.intersect(q, v), s.closest_point(q), s.closest_silhouette(q), s.intersect(q, v, variant="exact"),
               s.closest_silhouette(q, variant="coherent"), s.closest_silhouette(q, variant="exact")]
        res = b.run(cp=(q, ids), ray=(q, v, ids), sil=(q, ids))
        torch.cuda.current_stream().synchronize()
    got[k] = [to_np(x) for x in out + [res.cp, res.ray, res.sil]]
ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
[t.start() for t in ts]; [t.join() for t in ts]
assert all(g is not None for g in got), "a thread ended with an error"
for k in range(2, 8):
    for a, b in zip(got[k], got[k % 2]):
        for f in a:
            assert np.array_equal(a[f], b[f], equal_nan=a[f].dtype.kind == "f"), (k, f)
print("ok")
"""


def test_launchers_keep_no_plain_statics():
    for p in sorted(DEVICE.glob("*.cu*")):
        found = re.findall(r"^\s+static (?!std::atomic|constexpr|const |__device__)[\w:<>]+ \w+[^(;]*=", p.read_text(), re.M)
        assert not found, (p.name, found)


@pytest.mark.gpu
def test_threads_launch_first_together():
    code = WORK.format(root=str(ROOT), tests=str(ROOT / "tests"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:] + r.stderr[-2000:]
