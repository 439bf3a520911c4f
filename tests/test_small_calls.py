"""A task alone against the same task in a batch: small calls share an item's grid walk between
blocks, cut the screening runs finer and take larger assembly blocks.

Every sum that reaches an output has one order whatever the batch, except the screening estimates
(their last bits decide nothing unless an estimate lies within them of a threshold, when one radial
integral changes by its threshold, 1e-16): the tolerance is 1e-13 of the block's largest value."""
import numpy as np
import pytest

from libgrpp_b200 import synthetic


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("system,pairs", [
    ("heavy", [(0, 0, 0), (0, 4, 1), (3, 7, 0), (3, 7, 1), (2, 9, 1), (7, 6, 0)]),
    ("molecule", [(0, 0, 0), (6, 6, 0), (5, 8, 0), (6, 7, 1), (13, 6, 0)])])
def test_task_alone_equals_batch(gpu_lib, system, pairs, mode):
    S = synthetic.moderate_heavy_system(3) if system == "heavy" else synthetic.config2(9, n_heavy=2, n_h=1, lmax=6, box=9.0, l_proj=5)
    whole = S.batch(*S.all_tasks())
    off = whole.block_offsets()
    ns, nc = len(S.shells), len(S.centres)
    ref = gpu_lib.full_grpp_batch(whole, mode)
    for a, b, c in pairs:
        t = (a * ns + b) * nc + c
        one = gpu_lib.full_grpp_batch(S.batch(*[np.array([x], np.int32) for x in (a, b, c)]), mode)
        for m in range(4):
            want = ref[m][off[t]:off[t + 1]]
            assert np.max(np.abs(one[m] - want)) <= 1e-13 * max(np.max(np.abs(want)), 1e-300), (a, b, c, m)
