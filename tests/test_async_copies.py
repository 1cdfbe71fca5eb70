"""Kernels that start asynchronous copies (the fetch-ahead of the closest-point and silhouette
walks) end them before they return: read from the sources, since a copy that lands late shows
only by chance."""
import re
from pathlib import Path

import pytest

DEVICE = Path(__file__).resolve().parents[1] / "gquery_b200" / "csrc" / "device"


def _functions(text):
    """(name, body) of every __global__ or __noinline__ device function."""
    for m in re.finditer(r"(?:__global__|__noinline__)[^;{]*?\b(k_\w+|\w+_phase)\(", text):
        at = text.index("{", m.end())
        depth, end = 0, at
        while True:
            depth += (text[end] == "{") - (text[end] == "}")
            end += 1
            if depth == 0:
                break
        yield m.group(1), text[at:end]


@pytest.mark.parametrize("source,name,call", [("packet.cu", "k_cp_packet", "closest_point<"),
                                              ("batch.cu", "sil_tiles_phase", "closest_silhouette<")])
def test_callers_of_the_fetch_ahead_wait_for_it(source, name, call):
    body = dict(_functions((DEVICE / source).read_text()))[name]
    assert call in body
    # after the loop over tiles, so once per warp
    assert body.rindex("copies_done()") > body.index(call)


def test_copies_are_started_by_the_two_walks_only():
    users = sorted(p.name for p in DEVICE.iterdir() if "cp.async.ca" in p.read_text())
    assert users == ["packet.cuh", "sil_packet.cuh"]
    # nobody but those callers asks for it
    sinks = sorted(p.name for p in DEVICE.glob("*.cu") if re.search(r"\bsink\[|LeafBuf leaf_buf\[\]", p.read_text()))
    assert sinks == ["batch.cu", "packet.cu"]
    assert "cp.async.wait_all" in (DEVICE / "packet.cuh").read_text()
