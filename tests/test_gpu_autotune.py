"""The autotuner times no two configurations that make the same launch: work items are at most
target_pairs large, and small batches have smaller ones whatever it says."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import autotune, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("search", ["descent", "grid"])
def test_equal_launches_are_timed_once(search):
    meshes = [synthetic.bumpy_icosphere(level, seed=level) for level in (2, 4)]
    queries = [synthetic.mixed_queries(V, F, 2000, seed=1) for V, F in meshes]
    space = {"qpt": (2,), "target_pairs": (1 << 23, 1 << 21, 1 << 18, 1 << 12)}
    result = autotune.tune(meshes, queries, space=space, use_cache=False, reps=1, search=search)
    pairs = float(sum(len(F) * len(O) for (_, F), O in zip(meshes, queries)))
    made = [autotune._item_pairs(pairs, t["config"]["target_pairs"]) for t in result["trials"]]
    assert len(made) == len(set(made)) == 2  # the first three are one launch
    assert {t["config"]["target_pairs"] for t in result["trials"]} == {1 << 23, 1 << 12}


def test_item_pairs():
    assert autotune._item_pairs(1e3, 1 << 23) == 1 << 17
    assert autotune._item_pairs(1e3, 1 << 10) == 1 << 10
    assert autotune._item_pairs(1e15, 1 << 23) == 1 << 23
    values = [autotune._item_pairs(p, 1 << 23) for p in np.geomspace(1e6, 1e13, 20)]
    assert values == sorted(values)
