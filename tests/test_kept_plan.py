"""A kept plan after other calls on its device. The angular tensors of a device grow with the classes
(L, l) that its batches bring and move to a larger allocation; a plan made before must read them where
they are when it runs. In a process of its own, so that the growth happens in between."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import numpy as np
from tests.util import load_product
from libgrpp_b200.system import GRPP, Potential, Shell, System


def slots(L, l):
    low = lambda n: L - n if L >= n else (L + n) & 1
    return max((L + n - low(n)) // 2 + 1 for n in range(l + 1))


def tensor_bytes(L, l):  # [abc][slot][mu][m]
    return 8 * (l + 1) * (l + 2) * (l + 3) // 6 * slots(L, l) * (2 * (L + l) + 1) * (2 * L + 1)


def system(ls, Ls):
    rng = np.random.default_rng(len(ls))
    shells = [Shell(rng.uniform(-0.5, 0.5, 3), l, [0.01], [0.7]) for l in ls]
    arep = [Potential(L, 0, [2], [1.0], [1.5]) for L in Ls]
    return System(shells, [GRPP(arep=arep)], [(np.zeros(3), 0)])


lib = load_product()
small, large = system([0, 1, 2], [0, 1, 2]), system([0, 6, 7, 8], [3, 4, 5])
first = 8 << 20  # the first allocation
assert sum(tensor_bytes(L, l) for L in range(3) for l in range(3)) < first < sum(tensor_bytes(L, l) for L in (3, 4, 5) for l in (6, 7, 8))
batch = small.batch(*small.all_tasks())
high = [np.array(x, np.int32) for x in ([0, 0, 0], [1, 2, 3], [0, 0, 0])]  # s with i, k and l shells
for mode in (0, 1):
    plan = lib.plan(batch, mode)
    plan.execute()
    before = plan.outputs()
    if mode == 0:
        kept, want = plan, before
lib.full_grpp_batch(large.batch(*high))
# whatever is allocated next may lie where the tensors were
other = lib.plan(large.batch(*high), 0)
other.execute()
for p, w in ((kept, want), (plan, before)):
    p.execute()
    assert max(np.abs(x).max() for x in w) > 0.0
    for x, y in zip(p.outputs(), w):
        assert np.array_equal(x, y)
print("same")
"""


@pytest.mark.gpu
def test_plan_after_the_tensors_have_grown(gpu_lib):
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("same\n"), r.stdout[-2000:] + r.stderr[-2000:]
