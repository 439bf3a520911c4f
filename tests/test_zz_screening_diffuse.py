"""Screening of diffuse f..i shells under tight potentials, where libgrpp's quotient of Bessel functions is 0/0 (orders
l >= 6, arguments below 0.005) and the estimate undefined: those entries are walked. Against the
no-allocation path, which screens with libgrpp's expressions entry by entry; the tolerance of record,
max(1e-10, 1e-9 |ref|). Shells within 1.2 bohr of the centre, much less than their extent, so that the
re-centring sums keep their digits.

A potential whose coefficient is NaN makes every element of its blocks NaN, also where none of its
triples could have mattered."""
import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System
from tests.util import strict_tol


def diffuse_system(l_proj, eta, seed):
    rng = np.random.default_rng(seed)
    xyz = [np.zeros(3), np.array([0.5, -0.3, 0.9]), np.array([-0.6, 0.8, 0.2])]
    shells = []
    for l in (3, 4, 5, 6):
        for o in (1, 2):
            al = np.exp(rng.uniform(np.log(0.02), np.log(0.4), 3))
            shells.append(Shell(xyz[o], l, rng.uniform(0.2, 1.0, 3) * al, al))
    arep = [Potential(q, 0, [2, 1, 2], rng.uniform(-5, 5, 3) * eta ** 2, eta * np.array([1.0, 0.3, 4.0])) for q in (l_proj, 1)]
    return System(shells, [GRPP(arep=arep)], [(xyz[0], 0)])


@pytest.mark.gpu
@pytest.mark.parametrize("l_proj,eta", [(3, 2.0), (5, 2.0), (4, 50.0), (2, 1e3), (5, 1e3), (5, 1e5)])
def test_undefined_estimates_are_walked(gpu_lib, l_proj, eta):
    S = diffuse_system(l_proj, eta, seed=l_proj)
    batch = S.batch(*S.all_tasks())
    got, want = gpu_lib.full_grpp_batch(batch)[0], gpu_lib.type2_batch_noalloc(batch)
    err = np.abs(got - want)
    print(f"projector {l_proj}, exponents {eta:g}: max abs {err.max():.2e} of {np.abs(want).max():.2e}")
    assert np.all(np.isfinite(want)) and np.abs(want).max() > 0.0
    assert np.all(err <= strict_tol(want)), float((err / strict_tol(want)).max())


@pytest.mark.gpu
@pytest.mark.parametrize("distance", [1.0, 30.0])
def test_nan_coefficient_reaches_the_result(gpu_lib, distance):
    xyz = np.array([0.0, 0.3, 1.0]) * distance
    shells = [Shell(xyz, l, [0.7, 0.4], [3.0, 8.0]) for l in (0, 1)]
    arep = [Potential(1, 0, [2, 2], [1.0, np.nan], [5.0, 9.0])]
    S = System(shells, [GRPP(arep=arep)], [(np.zeros(3), 0)])
    out = gpu_lib.full_grpp_batch(S.batch(*S.all_tasks()))[0]
    assert np.all(np.isnan(out))
