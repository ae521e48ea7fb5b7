"""Reparametrizations of strings of different lengths from two threads: the
shared memory that one plan may use is no setting that the other's launch loses."""
import threading

import numpy as np
import pytest

from mepgl_gb300.problem import StringState
from mepgl_gb300.workloads import random_state
from test_gpu_strips import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cubic", [False, True])
def test_plans_of_two_lengths_at_once(cubic):
    from mepgl_gb300 import native
    rng = np.random.default_rng(9)
    prob = problem(rng, 6, 5, False, False, True, 0.0)
    ends = random_state(rng, prob, images=2, amp=0.3)
    errors, done = [], []

    def work(images, rounds):
        try:
            t = np.linspace(0, 1, images)[:, None, None, None] ** 1.2
            st = StringState(a=(1 - t) * ends.a[:1] + t * ends.a[1:], psi_1=(1 - t) * ends.psi_1[:1] + t * ends.psi_1[1:],
                             psi_2=None)
            c = native.StringContext(prob, images, "fp64")
            c.set_state(st)
            for _ in range(rounds):
                (c.redistribute_cubic if cubic else c.redistribute_linear)()
            done.append(np.all(np.isfinite(c.compute_free_energy())))
            c.close()
        except native.MepglError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=a) for a in ((750, 600), (2000, 300))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert done == [True, True]
