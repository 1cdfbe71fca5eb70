"""The scratch pool: a call on one stream does not wait for another stream whose scratch is still
to be released, and the pool's memory goes back with the last scene (seen in a fresh process,
where no other scene lives)."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from gquery_b200 import workloads as W
from gquery_b200.scene import Scene

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


def test_calls_on_two_streams_do_not_wait_for_one_another():
    s = Scene(*W.icosphere(2, seed=1), 3, device=0, build_snch=False)
    q = torch.as_tensor(W.uniform_points(3_000_000, 3, seed=2)).cuda()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    outs = [s.alloc_cp(3_000_000) for _ in range(2)]
    for st, out in zip((a, b), outs):  # the pool holds the scratch of one call
        with torch.cuda.stream(st):
            s.closest_point(q, out=out)
        torch.cuda.synchronize()
    slow = torch.cuda.Event()
    with torch.cuda.stream(a):
        torch.cuda._sleep(1_000_000_000)  # about half a second
        s.closest_point(q, out=outs[0])
        slow.record()
    with torch.cuda.stream(b):
        s.closest_point(q, out=outs[1])
    b.synchronize()
    ended = slow.query()
    torch.cuda.synchronize()
    assert not ended, "the second stream's call waited for the first stream"
    assert torch.equal(outs[0].d, outs[1].d)


LAST = """
import sys
sys.path.insert(0, {root!r})
import torch
from gquery_b200 import workloads as W
from gquery_b200.scene import Scene
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info(0)[0])[1]
n = 2_000_000
q = torch.as_tensor(W.uniform_points(n, 3, seed=2)).cuda()
def one():
    s = Scene(*W.icosphere(2, seed=1), 3, device=0, build_snch=False)
    return s, s.alloc_cp(n)
s, out = one()
before = free()
s.closest_point(q, out=out)
held = before - free()
t = Scene(*W.icosphere(2, seed=1), 3, device=0, build_snch=False)
need = s.scratch_bytes(n)
assert held >= need // 2, (held, need)
s.close()
still = before - free()
assert still >= need // 2, (still, held)
t.close()
after = before - free()
assert after < need // 8, (after, held)
s, out = one()
a = s.closest_point(q).d
assert before - free() >= need // 2
s.close()
print("ok")
"""


def test_pool_memory_goes_with_the_last_scene():
    r = subprocess.run([sys.executable, "-c", LAST.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:] + r.stderr[-2000:]
