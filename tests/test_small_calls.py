"""A task alone against the same task in a batch: small calls share an item's grid walk between
blocks, cut the screening runs finer and take larger assembly blocks.

Every sum that reaches an output has one order whatever the batch, except the type 1 sums of items
that several blocks share (last bits) and the screening estimates (their last bits decide nothing unless an estimate lies within them of a threshold, when one radial
integral changes by its threshold, 1e-16): the tolerance is 1e-13 of the block's largest value."""
import numpy as np
import pytest

from libgrpp_b200 import synthetic
from libgrpp_b200.system import GRPP, Potential, Shell, System


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


@pytest.mark.gpu
@pytest.mark.parametrize("n_tasks", [4095, 4096, 4097, 9000])
@pytest.mark.parametrize("symmetric", [False, True])
def test_gradient_of_a_long_list(gpu_lib, n_tasks, symmetric):
    """The gradient runs its list in chunks, the host one chunk ahead: a list that repeats a few
    tasks gives their weighted sum. n equal addends in any order: n eps of the addends' sum."""
    S = synthetic.config2(9, n_heavy=1, n_h=2, lmax=2, box=7.0, l_proj=2)
    a, b, c = S.all_tasks()
    n = S.n_basis()
    D = np.random.default_rng(4).uniform(-1, 1, (n, n))
    D = 0.5 * (D + D.T)
    pick = np.arange(min(7, len(a)))
    idx = pick[np.arange(n_tasks) % len(pick)]
    got = gpu_lib.grad_contract(S, S.batch(a[idx], b[idx], c[idx]), D, symmetric=symmetric)
    want, size = np.zeros_like(got), np.zeros_like(got)
    for k, cnt in zip(pick, np.bincount(idx, minlength=len(pick))):
        one = gpu_lib.grad_contract(S, S.batch(a[k:k + 1], b[k:k + 1], c[k:k + 1]), D, symmetric=symmetric)
        want += cnt * one
        size += cnt * np.abs(one)
    assert np.all(np.abs(got - want) <= n_tasks * 2.3e-16 * size + 1e-13 * size.max())


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 227, 228, 400])
def test_outputs_with_the_status_or_after_it(gpu_lib, copies):
    """Up to 8192 numbers per array return with the status words, more are copied on their own
    (a block of two d shells: 36 numbers, the line at 227 copies)."""
    S = synthetic.config2(9, n_heavy=1, n_h=2, lmax=2, box=7.0, l_proj=2)
    a, b, c = S.all_tasks()
    ncart = np.array([(s.L + 1) * (s.L + 2) // 2 for s in S.shells])
    k = int(np.argmax(ncart[a] * ncart[b]))
    one = gpu_lib.full_grpp_batch(S.batch(a[k:k + 1], b[k:k + 1], c[k:k + 1]))
    assert len(one[0]) == 36
    many = gpu_lib.full_grpp_batch(S.batch(*[np.repeat(x[k:k + 1], copies) for x in (a, b, c)]))
    for x, y in zip(one, many):
        y = y.reshape(copies, 36)
        assert np.max(np.abs(y - x)) <= 1e-13 * max(np.max(np.abs(x)), 1e-300)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("which", ["all", "one_centre", "local_only", "one_task"])
def test_three_streams_equal_one(gpu_lib, which, mode):
    """A batched call spreads its kernels over three streams, a kept plan runs them one after
    another: the same operations in the same order, so the same bits."""
    S = synthetic.moderate_heavy_system(3)
    a, b, c = S.all_tasks()
    if which == "one_centre":
        at = np.array([[np.allclose(s.origin, x) for x, _ in S.centres] for s in S.shells])
        keep = at[a, c] & at[b, c]
        a, b, c = a[keep], b[keep], c[keep]
    elif which == "local_only":
        for g in S.grpps:
            g.arep, g.so, g.oc = [], [], []
    elif which == "one_task":
        a, b, c = a[17:18], b[17:18], c[17:18]
    batch = S.batch(a, b, c)
    got = gpu_lib.full_grpp_batch(batch, mode)
    plan = gpu_lib.plan(batch, mode)
    plan.execute()
    want = plan.outputs()
    assert len(a) and max(np.abs(x).max() for x in want) > 0.0
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("la,lb,nprim", [(0, 0, 3), (1, 2, 8), (4, 3, 11), (6, 6, 5), (6, 6, 9)])
def test_shared_type1_items(gpu_lib, la, lb, nprim):
    """A few type 1 items are cut into shares of their triples, many are not: one task against 700
    copies of it. Coefficients of one sign, so the shares' sums do not cancel: the orders differ
    by at most n_triples eps of the terms, which the block's largest element bounds within a factor of 10."""
    rng = np.random.default_rng(10 * la + lb + nprim)
    al = lambda n: np.exp(rng.uniform(np.log(0.2), np.log(3.0), n))
    A = Shell([0.0, 0.1, -0.2], la, rng.uniform(0.2, 1.0, nprim), al(nprim))
    B = Shell([0.7, -0.3, 0.4], lb, rng.uniform(0.2, 1.0, nprim), al(nprim))
    U = Potential(0, 0, [0, 1, 2, 2, 1], rng.uniform(0.5, 2.0, 5), al(5))
    S = System(shells=[A, B], grpps=[GRPP(UL=U)], centres=[(np.array([0.2, 0.3, 0.1]), 0)])
    task = [np.array([x], np.int32) for x in (0, 1, 0)]
    one = gpu_lib.full_grpp_batch(S.batch(*task))[0]
    many = gpu_lib.full_grpp_batch(S.batch(*[np.repeat(x, 700) for x in task]))[0].reshape(700, -1)
    tol = 10 * 5 * nprim * nprim * 2.3e-16 * np.abs(one).max()
    assert np.abs(one).max() > 0.0
    assert np.all(many == many[0])
    assert np.max(np.abs(many[0] - one)) <= tol
