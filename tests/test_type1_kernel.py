"""The type 1 kernel at the edges of its batches: one to several groups of 64 triples, partial
batches, potentials with terms of one power only and of all three, dropped triples, s x s up to
the largest classes of its tables.

Compared with the oracle at the tolerance of record, max(1e-10, 1e-9 |ref|): the exponents lie
in [0.1, 5], where libgrpp's own type 1 sums keep 12 or more digits."""
import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System
from tests.util import strict_tol

POWERS = {"boys": [1], "overlap": [2], "g": [0], "all": [2, 0, 1, 2, 0, 1, 1]}


def _system(la, lb, n_a, n_b, powers, far, seed=11):
    rng = np.random.default_rng(seed)

    def shell(o, L, n):
        return Shell(np.array(o), L, rng.uniform(-1, 1, n), np.exp(rng.uniform(np.log(0.1), np.log(5.0), n)))

    A, B, C = [0.0, 0.1, -0.2], [0.7, -0.5, 1.1], [-0.9, 0.4, 0.6 + far]
    shells = [shell(A, la, n_a), shell(B, lb, n_b), shell(C, max(la, lb), 3)]
    shells[0].coeffs[-1] = 0.0  # a primitive that libgrpp leaves out
    n = len(powers)
    ul = Potential(0, 0, np.array(powers), rng.uniform(-5, 5, n), np.exp(rng.uniform(np.log(0.1), np.log(5.0), n)))
    return System(shells, [GRPP(UL=ul)], [(np.array(C), 0)])


@pytest.mark.gpu
@pytest.mark.parametrize("la,lb,n_a,n_b,powers,far", [
    (0, 0, 2, 1, "boys", 0.0), (0, 0, 17, 16, "all", 0.0), (0, 1, 9, 7, "all", 0.0), (1, 1, 5, 13, "g", 0.0),
    (2, 1, 3, 3, "overlap", 0.0), (3, 2, 9, 9, "all", 0.0), (4, 4, 3, 5, "all", 0.0), (4, 4, 2, 2, "boys", 14.0),
    (5, 2, 2, 9, "g", 0.0), (6, 6, 2, 3, "all", 0.0), (7, 4, 2, 2, "all", 0.0), (0, 7, 3, 1, "all", 14.0)])
def test_type1_blocks(gpu_lib, oracle_lib, la, lb, n_a, n_b, powers, far):
    batch = _system(la, lb, n_a, n_b, POWERS[powers], far).batch(*[np.array(x, np.int32) for x in ([0, 1], [1, 0], [0, 0])])
    got = gpu_lib.full_grpp_batch(batch)[0]
    want = oracle_lib.driver_full_batch(batch, nthreads=1)[0]
    err = np.abs(got - want)
    print(f"({la},{lb}) {n_a}x{n_b} {powers}: max abs {err.max():.2e} of {np.abs(want).max():.2e}")
    assert np.all(err <= strict_tol(want)), float(err.max())
