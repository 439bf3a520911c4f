"""The allocation-free entry point up to L = 10: classes whose assembly tables fit only when each task's own
sides are counted, alone and beside smaller ones, against the engine: 1e-9 of the block's largest value (the blocks are
small, so this is below the tolerance of record)."""
import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System


@pytest.mark.gpu
@pytest.mark.parametrize("pairs,Ls", [([(10, 4)], [1]), ([(4, 10)], [1]), ([(10, 4), (0, 2), (4, 4)], [1, 0]), ([(10, 1)], [0]), ([(9, 4)], [1]),
                                      ([(8, 5)], [2])])
def test_high_shells(gpu_lib, pairs, Ls):
    rng = np.random.default_rng(len(pairs) + 10 * len(Ls))
    shells = [Shell(rng.uniform(-0.4, 0.4, 3), l, [1e-3 ** (l / 4)], [0.4 + 0.1 * k]) for k, l in enumerate(sum(map(list, pairs), []))]
    S = System(shells, [GRPP(arep=[Potential(L, 0, [2, 1], [1.5, -0.7], [0.9, 2.5]) for L in Ls])], [(np.zeros(3), 0)])
    n = len(pairs)
    batch = S.batch(np.arange(0, 2 * n, 2, dtype=np.int32), np.arange(1, 2 * n, 2, dtype=np.int32), np.zeros(n, np.int32))
    want, got = gpu_lib.full_grpp_batch(batch)[0], gpu_lib.type2_batch_noalloc(batch)
    off = batch.block_offsets()
    for t in range(n):
        w, g = want[off[t]:off[t + 1]], got[off[t]:off[t + 1]]
        assert np.abs(w).max() > 0.0 and np.abs(g - w).max() <= min(1e-10, 1e-9 * np.abs(w).max())
