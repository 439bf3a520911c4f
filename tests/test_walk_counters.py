"""Counters of a plan whose items are shared between blocks: an item's points and levels are those of its deepest
entry, whichever block walks it. The levels themselves come from libgrpp_b200_level_samples, which
gives an item to one block. (A level L has 2^(L+5) - 1 points in all.)"""
import numpy as np
import pytest

from libgrpp_b200 import synthetic


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 20, 90])
def test_counters_of_shared_items(gpu_lib, n, mode):
    S = synthetic.moderate_heavy_system(3)
    a, b, c = S.all_tasks()
    pick = np.sort(np.random.default_rng(n).choice(len(a), n, replace=False))
    batch = S.batch(a[pick], b[pick], c[pick])
    levels = gpu_lib.level_samples(batch)[1].astype(int)
    walked = levels[levels >= 0]
    plan = gpu_lib.plan(batch, mode)
    for _ in range(2):
        plan.execute()
        got = plan.counters()
        assert got["items"] == len(walked)
        assert got["levels"] == np.sum(walked + 1)
        assert got["points"] == np.sum(2 ** (walked + 5) - 1)
