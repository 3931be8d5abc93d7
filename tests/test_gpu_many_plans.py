"""More plans alive than there are page-locked places for their results (64):
every plan's build returns its own energy, in any order and after others have
gone, from two host threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from nukexc_b200 import api as A  # noqa: E402


def test_each_plan_returns_its_own_result():
    c, Z = np.zeros((1, 3)), np.ones(1, np.int32)
    b = A.make_manual_basis([(1, 0, 0, 1.0, 0.0, 0.0, 0.0)])
    pts = np.random.default_rng(0).normal(size=(100, 3))
    make = lambda k: A.FockBuilder(c, Z, b, (pts, np.full(100, 1.0 + k)), func_ids=("LDA_X",))  # noqa: E731
    energy = lambda fb, p: fb.build([np.ones((1, 1))], [np.ones(1)], precision=p)[0]  # noqa: E731
    plans = {k: make(k) for k in range(70)}
    e = energy(plans[0], "fp64")
    for k in list(range(0, 70, 3)):
        plans.pop(k).close()
    for k in range(70, 80):
        plans[k] = make(k)
    bad = []

    def run(keys, precision):
        for _ in range(5):
            for k in keys:
                if not abs(energy(plans[k], precision) - (1.0 + k) * e) <= 1e-6 * abs((1.0 + k) * e):
                    bad.append(k)
    keys = sorted(plans)
    t = [threading.Thread(target=run, args=(keys[0::2], "fp64")), threading.Thread(target=run, args=(keys[1::2], "mixed"))]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not bad
    for fb in plans.values():
        fb.close()
