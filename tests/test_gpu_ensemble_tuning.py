"""The launch shape of a new ensemble is one of those that the autotuner
tries (8, 16, 32 or 64 planes a face tile, at most as many blocks per SM as
fit), so that autotuning never leaves an ensemble slower than it was
created."""
import pytest

import cases
from test_gpu_ensemble import CFL, _members

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("members", [slice(0, 1), slice(0, 5)])
def test_default_is_among_the_trials(precision, members):
    import grdzhadzha_b200 as G
    t = G.Ensemble(_members(precision)[members], cfl=CFL).tuning
    assert t["zchunk"] in (8, 16, 32, 64)
    assert 1 <= t["blocks_per_sm"] <= t["max_blocks_per_sm"]


def test_default_of_many_small_members():
    import grdzhadzha_b200 as G
    p, box, s, _ = cases.CASES["michel18"]()
    mem = [(cases.gpu_operator(p), cases.gpu_level(box, s))
           for _ in range(40)]
    assert G.Ensemble(mem, cfl=CFL).tuning["zchunk"] in (8, 16, 32, 64)
