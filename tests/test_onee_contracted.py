"""One-electron blocks of contracted shells against their primitives: a warp tabulates up to ten
primitive pairs at a time, fewer for high angular momenta (one lane per pair and axis). A block is
the sum over its pairs in order: n eps of the terms' moduli. Angular momenta to 10 and up to 25
pairs cross every batch size."""
import numpy as np
import pytest

from libgrpp_b200.system import System, Shell

EPS = 2.3e-16


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("la,lb,na,nb", [(0, 0, 1, 1), (0, 0, 3, 4), (1, 0, 5, 5), (4, 4, 3, 2), (4, 4, 7, 1), (6, 5, 2, 3),
                                         (10, 10, 2, 2), (0, 10, 1, 11)])
def test_contracted_equals_primitives(gpu_lib, kind, la, lb, na, nb):
    rng = np.random.default_rng(1000 * la + 100 * lb + na + nb)
    al = lambda n: np.exp(rng.uniform(np.log(0.3), np.log(6.0), n))
    A = Shell([0.1, -0.2, 0.3], la, rng.uniform(0.3, 1.0, na), al(na))
    B = Shell([-0.6, 0.5, 0.9], lb, rng.uniform(0.3, 1.0, nb), al(nb))
    prims = [Shell(s.origin, s.L, [1.0], [x]) for s in (A, B) for x in s.alpha]
    S = System(shells=[A, B] + prims, grpps=[], centres=[(np.zeros(3), 0)])
    pa, pb = 2 + np.arange(na), 2 + na + np.arange(nb)
    a = np.array([0] + [i for i in pa for _ in pb], np.int32)
    b = np.array([1] + [j for _ in pa for j in pb], np.int32)
    cc = (A.coeffs[:, None] * B.coeffs[None, :]).reshape(-1, 1)
    for out in gpu_lib.onee_batch(S.batch(a, b, np.zeros(len(a), np.int32)), kind):
        out = out.reshape(1 + na * nb, -1)
        terms = cc * out[1:]
        assert np.all(np.abs(out[0] - terms.sum(axis=0)) <= (na * nb + 2) * EPS * np.abs(terms).sum(axis=0))
        assert np.abs(out[0]).max() > 0.0
