"""The engine's screening (triples dropped by a bound, ratios from tables, lanes shared between
entries and triples) against the general path: libgrpp_b200_type2_batch_noalloc screens every
entry of the whole (l1, l2, N) box with libgrpp's expressions, one thread per entry.

Shells l <= 1 only: their re-centring sums have at most four terms, so that exponents up to 1e5
and distances up to 40 bohr, where most triples are dropped, can be compared (on higher shells
such exponents amplify last-bit differences of any two implementations without bound; the
fixture tests cover those). The tolerance of record, max(1e-10, 1e-9 |ref|)."""
import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System
from tests.util import strict_tol


def _system(L, n_prim, amax, dist, seed):
    """s and p shells of n_prim primitives on the centre and on two other atoms; two projectors."""
    rng = np.random.default_rng(seed)
    xyz = [np.zeros(3), np.array([0.3, -0.2, 1.0]) * dist, np.array([-0.8, 0.5, 0.1]) * dist]
    shells = []
    for l, o in [(0, 1), (1, 1), (0, 2), (1, 2), (0, 0), (1, 0)]:
        shells.append(Shell(xyz[o], l, rng.uniform(-1, 1, n_prim), np.exp(rng.uniform(np.log(0.05), np.log(amax), n_prim))))
    arep = [Potential(q, 0, rng.integers(0, 3, n), rng.uniform(-10, 10, n), np.exp(rng.uniform(np.log(0.05), np.log(50.0), n)))
            for q, n in ((L, 3), (0, 1))]
    return System(shells, [GRPP(arep=arep)], [(xyz[0], 0)])


@pytest.mark.gpu
@pytest.mark.parametrize("L,n_prim,amax,dist", [
    (0, 1, 5.0, 1.0), (4, 8, 50.0, 2.0), (3, 7, 5e3, 0.7), (5, 9, 5e3, 3.0), (1, 3, 5e3, 12.0), (10, 5, 20.0, 1.5),
    (2, 8, 5e3, 40.0), (2, 4, 1e5, 1e-3), (6, 17, 1e5, 5.0)])
def test_screening_against_general_path(gpu_lib, L, n_prim, amax, dist):
    S = _system(L, n_prim, amax, dist, seed=100 * n_prim + L)
    batch = S.batch(*S.all_tasks())
    got, want = gpu_lib.full_grpp_batch(batch)[0], gpu_lib.type2_batch_noalloc(batch)
    err = np.abs(got - want)
    print(f"L {L} {n_prim} primitives to {amax:g}, {dist:g} bohr: max abs {err.max():.2e} of {np.abs(want).max():.2e}")
    assert np.all(err <= strict_tol(want)), float((err / strict_tol(want)).max())
