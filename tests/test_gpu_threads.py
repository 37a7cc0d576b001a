"""Solves on two host threads at once: each returns what it returns alone."""
import threading

import numpy as np
import pytest

from pdhcg_b200 import instances, native
from test_gpu_resident import _problem

pytestmark = pytest.mark.gpu


def _dense(k, n):
    rng = np.random.default_rng(k)
    p = _problem(n, n, n // 4, True)
    p.R_dense = rng.standard_normal((k, n)) / np.sqrt(n)
    return p


# Two sizes of shared memory of one kernel each: ranks 64 and 10 of the dense
# inner solve, PSD blocks of order 20 and 5 (step and residual)
@pytest.mark.parametrize("big,small", [
    (lambda: _dense(64, 4000), lambda: _dense(10, 4000)),
    (lambda: instances.psd_lp(seed=41, orders=(20,) * 8), lambda: instances.psd_lp(seed=42, orders=(5,) * 8)),
], ids=["dense rank", "psd order"])
def test_two_sizes_at_once(lib, big, small):
    prm = {"termination_criteria.iteration_limit": 400, "termination_criteria.eps_optimal_relative": 1e-15,
           "termination_criteria.eps_feasible_relative": 1e-15}
    probs = [big(), small()]
    alone = [native.solve(p, prm) for p in probs]
    got, errors = [[], []], []

    def work(i):
        try:
            for _ in range(4):
                got[i].append(native.solve(probs[i], prm))
        except Exception as e:  # a launch that failed ends its solve
            errors.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, solves in zip(alone, got):
        for d in solves:  # every sum has a fixed order
            np.testing.assert_array_equal(d["x"], a["x"])
            np.testing.assert_array_equal(d["y"], a["y"])
