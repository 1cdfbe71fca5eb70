"""Ray candidates: the default walk over the 8-wide nodes chooses its own launch, so the fields it
does not read (threads per block, refill budget, persistence) make no second candidate."""
import pytest

from gquery_b200.autotune import candidates, config_key


@pytest.mark.parametrize("dim", [2, 3])
def test_default_ray_walk_is_one_candidate(dim):
    c = candidates("ray", dim, True, 24, 40)
    assert len({config_key(x) for x in c}) == len(c)
    assert len([x for x in c if x["variant"] == "wide8" and x["packet"] == 0 and x["sorted"] == 1]) == 1
    assert {x["variant"] for x in c} == {"exact", "wide8"}
    assert all(x["variant"] == "exact" for x in candidates("ray", dim, False, 24, 0))
