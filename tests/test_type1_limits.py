"""Angular momenta of type 1 blocks: what is supported runs, the rest is refused with a message that names the
limits (the largest L and the largest L_A + L_B of the batch count)."""
import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System


def _batch(pairs):
    shells = [Shell([0.1 * k, -0.2, 0.3 * k], l, [1.0], [0.8 + 0.1 * k]) for k, l in enumerate(sum(map(list, pairs), []))]
    U = Potential(0, 0, [2, 1, 0], [1.0, -0.5, 0.3], [0.9, 1.3, 2.0])
    S = System(shells, [GRPP(UL=U)], [(np.array([0.2, 0.0, 0.1]), 0)])
    n = len(pairs)
    return S.batch(np.arange(0, 2 * n, 2, dtype=np.int32), np.arange(1, 2 * n, 2, dtype=np.int32), np.zeros(n, np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("pairs", [[(6, 6), (0, 0)], [(7, 4), (6, 5)], [(4, 7)], [(8, 0), (4, 4)], [(0, 8)]])
def test_supported(gpu_lib, pairs):
    out = gpu_lib.full_grpp_batch(_batch(pairs))[0]
    assert np.all(np.isfinite(out)) and np.abs(out).max() > 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("pairs", [[(7, 5)], [(8, 1)], [(1, 8)], [(9, 0)], [(7, 0), (6, 6)], [(8, 0), (5, 4)]])
def test_refused(gpu_lib, pairs):
    with pytest.raises(RuntimeError, match=r"L_A \+ L_B <= 11"):
        gpu_lib.full_grpp_batch(_batch(pairs))
