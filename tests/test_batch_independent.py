"""The bits of a block do not depend on what else is in the batch: type 1 items of a small batch are shared
between blocks, those of a large one are not, and both add the same parts in the same order."""
import numpy as np
import pytest

from libgrpp_b200 import synthetic
from libgrpp_b200.system import GRPP, Potential, Shell, System


# candidates: 5 na nb triples; alone, an item is cut into up to min(triples / 64, 16) shares. Among them
# part sizes of 32 and 64, totals that are no multiple of either, one share more and less than parts
# of one kind, and terms of one kind only
@pytest.mark.gpu
@pytest.mark.parametrize("powers", [[0, 1, 2, 2, 1], [2, 2, 2, 2, 2], [0, 0, 1, 1, 0]])
@pytest.mark.parametrize("la,lb,na,nb", [(0, 0, 3, 3), (1, 2, 8, 8), (4, 3, 11, 11), (2, 2, 21, 21), (6, 6, 5, 5), (6, 6, 9, 9), (5, 6, 13, 7),
                                         (6, 5, 21, 23), (0, 0, 64, 64), (7, 4, 17, 16), (3, 6, 64, 5)])
def test_type1_items_shared_or_not(gpu_lib, la, lb, na, nb, powers):
    rng = np.random.default_rng(1000 * la + 100 * lb + na + nb)
    al = lambda n, top: np.exp(rng.uniform(np.log(0.2), np.log(top), n))
    A = Shell([0.0, 0.1, -0.2], la, rng.uniform(-1.0, 1.0, na), al(na, 300.0))
    B = Shell([1.7, -0.3, 2.4], lb, rng.uniform(-1.0, 1.0, nb), al(nb, 300.0))  # far enough that tight triples are dropped
    U = Potential(0, 0, powers, rng.uniform(0.5, 2.0, 5), al(5, 30.0))
    S = System(shells=[A, B], grpps=[GRPP(UL=U)], centres=[(np.array([0.2, 0.3, 0.1]), 0)])
    task = [np.array([x], np.int32) for x in (0, 1, 0)]
    want = gpu_lib.full_grpp_batch(S.batch(*[np.repeat(x, 600) for x in task]))[0].reshape(600, -1)
    assert np.abs(want[0]).max() > 0.0 and np.all(want == want[0])
    for n in (1, 2, 5, 40):  # fewer shares the more items there are
        got = gpu_lib.full_grpp_batch(S.batch(*[np.repeat(x, n) for x in task]))[0].reshape(n, -1)
        assert np.array_equal(got, np.repeat(want[:1], n, axis=0)), n


@pytest.mark.gpu
@pytest.mark.parametrize("system", ["heavy", "molecule"])
def test_tasks_alone_and_in_a_batch(gpu_lib, system):
    S = synthetic.moderate_heavy_system(3) if system == "heavy" else synthetic.config2(9, n_heavy=2, n_h=1, lmax=6, box=9.0, l_proj=5)
    a, b, c = S.all_tasks()
    whole = S.batch(a, b, c)
    off = whole.block_offsets()
    ref = gpu_lib.full_grpp_batch(whole)
    for t in np.random.default_rng(1).choice(len(a), 12, replace=False):
        one = gpu_lib.full_grpp_batch(S.batch(a[t:t + 1], b[t:t + 1], c[t:t + 1]))
        for m in range(4):
            assert np.array_equal(one[m], ref[m][off[t]:off[t + 1]]), (t, m)


@pytest.mark.gpu
def test_no_triple_left(gpu_lib):
    """Every triple dropped: the block is zero, whatever the output held before."""
    A, B = Shell([0.0, 0.0, 0.0], 1, [1.0], [40.0]), Shell([0.0, 0.0, 30.0], 2, [1.0], [50.0])
    U = Potential(0, 0, [2, 1], [1.0, 1.0], [3.0, 4.0])
    near = Shell([0.0, 0.1, 0.2], 2, [1.0], [0.5])
    S = System(shells=[A, B, near], grpps=[GRPP(UL=U)], centres=[(np.zeros(3), 0)])
    z = np.zeros(9, np.int32)
    assert np.abs(gpu_lib.full_grpp_batch(S.batch(z, z + 2, z))[0]).max() > 0.0
    for n in (1, 9):
        assert np.all(gpu_lib.full_grpp_batch(S.batch(z[:n], z[:n] + 1, z[:n]))[0] == 0.0)
