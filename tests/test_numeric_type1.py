"""Numeric type 1 integrals of contracted shells against their primitives: a block adds the
primitive pairs' contributions c_i c_j <i|V|j> in order, groups of four pairs share an assembly
block, one lane holds one radial sum up to L_A + L_B = 9 and two above, 1024 centres or 256 MB of
scratch make a chunk. The contributions of one pair do not depend on what else is in the batch, so
the two sides differ by the rounding of n products and additions, n eps of the terms' moduli."""
import numpy as np
import pytest

from libgrpp_b200.system import System, Shell

GAUSS = 2
EPS = 2.3e-16


def _system(la, lb, na, nb, centres):
    rng = np.random.default_rng(100 * la + 10 * lb + na + nb)
    al = lambda n: np.exp(rng.uniform(np.log(0.3), np.log(6.0), n))
    A = Shell(np.array([0.1, -0.2, 0.3]), la, rng.uniform(0.3, 1.0, na), al(na))
    B = Shell(np.array([-0.6, 0.5, 0.9]), lb, rng.uniform(0.3, 1.0, nb), al(nb))
    prims = [Shell(s.origin, s.L, [1.0], [x]) for s in (A, B) for x in s.alpha]
    S = System(shells=[A, B] + prims, grpps=[], centres=[])
    xyz = rng.uniform(-1.5, 1.5, (centres, 3))
    xyz[0] = A.origin
    return S, A, B, xyz


@pytest.mark.gpu
@pytest.mark.parametrize("la,lb,na,nb", [(0, 0, 1, 1), (1, 2, 3, 1), (2, 0, 5, 1), (4, 4, 2, 4), (4, 5, 1, 3), (5, 5, 3, 3),
                                         (6, 6, 2, 2)])
def test_contracted_equals_primitives(gpu_lib, la, lb, na, nb):
    S, A, B, xyz = _system(la, lb, na, nb, 2)
    _compare(gpu_lib, S, A, B, xyz)


@pytest.mark.gpu
@pytest.mark.parametrize("centres", [1023, 1024, 1025])
def test_many_centres(gpu_lib, centres):
    S, A, B, xyz = _system(1, 1, 2, 1, centres)
    _compare(gpu_lib, S, A, B, xyz)


def _compare(lib, S, A, B, xyz):
    S.centres = [(x, 0) for x in xyz]
    na, nb, nc = len(A.alpha), len(B.alpha), len(xyz)
    Z = np.linspace(1.0, 9.0, nc)
    par = np.tile([0.4, 0.0, 0.0], (nc, 1))
    pa, pb = 2 + np.arange(na), 2 + na + np.arange(nb)
    a, b, c = [], [], []
    for k in range(nc):
        a += [0] + [i for i in pa for _ in pb]
        b += [1] + [j for _ in pa for j in pb]
        c += [k] * (1 + na * nb)
    out = lib.nuclear_attraction_batch(S.batch(*[np.array(x, np.int32) for x in (a, b, c)]), GAUSS, Z, par)
    out = out.reshape(nc, 1 + na * nb, -1)
    cc = (A.coeffs[:, None] * B.coeffs[None, :]).reshape(1, -1, 1)
    terms = cc * out[:, 1:]
    tol = (na * nb + 2) * EPS * np.abs(terms).sum(axis=1)
    assert np.all(np.abs(out[:, 0] - terms.sum(axis=1)) <= tol)
    assert np.abs(out).max() > 0.0
