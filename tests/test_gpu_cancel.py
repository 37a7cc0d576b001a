"""Cancelling a solve whose main loop runs in persistent launches."""
import threading
import time

import numpy as np
import pytest

from pdhcg_b200 import native
from test_gpu_resident import _problem

pytestmark = pytest.mark.gpu


@pytest.fixture
def flag(lib):
    lib.pdhcg_b200_request_cancel(0)
    yield lib.pdhcg_b200_request_cancel
    lib.pdhcg_b200_request_cancel(0)


def _params(limit, **more):
    return {"termination_criteria.iteration_limit": limit, "termination_criteria.eps_optimal_relative": 1e-15,
            "termination_criteria.eps_feasible_relative": 1e-15, **more}


def test_cancel_during_the_last_launch(lib, flag):
    """2300 iterations are two launches of 200 and one of 1900 (20 of the 25 ms on
    this problem): a flag set in the middle of the last one, with the iteration
    limit at its end, still ends the solve as interrupted."""
    p, prm = _problem(5, 150000, 75000, False), _params(2300)
    native.solve(p, prm)
    seen = []
    for _ in range(5):  # the host may stall between the clock and the flag
        t0 = time.perf_counter()
        native.solve(p, prm)
        timer = threading.Timer(0.75 * (time.perf_counter() - t0), flag, (1,))
        timer.start()
        d = native.solve(p, prm)
        timer.join()
        flag(0)
        seen.append(d["status"])
        if d["status"] == "USER_INTERRUPT":
            assert np.isfinite(d["x"]).all() and d["total_count"] <= 2300
            break
    assert seen[-1] == "USER_INTERRUPT", seen


def test_time_limit_within_a_launch(lib):
    """A limit that ends half way through a launch of 2000 iterations (20 ms): the
    solve stops at an evaluation soon after it."""
    p, prm = _problem(6, 150000, 75000, False), _params(20000)
    native.solve(p, dict(prm, **{"termination_criteria.iteration_limit": 400}))
    limit = 0.012
    over = []
    for _ in range(5):  # the host may stall
        d = native.solve(p, dict(prm, **{"termination_criteria.time_sec_limit": limit}))
        assert d["status"] == "TIME_LIMIT"
        over.append(d["cumulative_time_sec"] - limit)
    assert min(over) <= 0.005, over
