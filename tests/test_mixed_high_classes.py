"""Batches that mix classes near the limit of the assembly's shared memory: what runs alone in its range of sizes runs
beside the other ranges, with the same bits, whatever launch group the tasks share."""
import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System


def _system(classes):
    rng = np.random.default_rng(7)
    shells, centres, grpps, tasks = [], [], [], []
    for k, (la, lb, L) in enumerate(classes):
        for l in (la, lb):
            shells.append(Shell(rng.uniform(-0.4, 0.4, 3), l, [0.7], [rng.uniform(0.5, 1.0)]))
        grpps.append(GRPP(arep=[Potential(L, 0, [2], [1.5], [0.9])]))
        centres.append((rng.uniform(-0.4, 0.4, 3), k))
        tasks.append((2 * k, 2 * k + 1, k))
    return System(shells, grpps, centres), np.array(tasks, np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 400])
@pytest.mark.parametrize("classes", [[(0, 5, 10), (5, 6, 8)], [(0, 5, 10), (6, 5, 8)], [(0, 5, 10), (2, 10, 2), (10, 2, 2)]])
def test_ranges_side_by_side(gpu_lib, classes, copies):
    S, tasks = _system(classes)
    alone = [gpu_lib.full_grpp_batch(S.batch(*t[:, None]))[0] for t in tasks]
    both = gpu_lib.full_grpp_batch(S.batch(*np.tile(tasks, (copies, 1)).T.copy()))[0]
    want = np.concatenate(alone)
    assert all(np.abs(x).max() > 0.0 for x in alone)
    assert np.array_equal(both, np.tile(want, copies))


@pytest.mark.gpu
def test_refused_within_a_range(gpu_lib):
    S, tasks = _system([(6, 6, 8), (0, 0, 0)])
    with pytest.raises(RuntimeError, match="assembly tables"):
        gpu_lib.full_grpp_batch(S.batch(*tasks.T.copy()))
