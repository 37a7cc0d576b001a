"""The step's cone launches, blocks of several kinds side by side and PSD
blocks of every order, against the oracle's iteration."""
import numpy as np
import pytest

from pdhcg_b200 import instances
from test_gpu_solver import _solve_gpu, _solve_oracle

pytestmark = pytest.mark.gpu

PRM = {"termination_criteria.iteration_limit": 60, "termination_criteria.eps_optimal_relative": 1e-15,
       "termination_criteria.eps_feasible_relative": 1e-15}


@pytest.mark.parametrize("make", [
    lambda: instances.psd_lp(seed=31, orders=(2,)),
    lambda: instances.psd_lp(seed=32, orders=(1, 2, 3, 7, 15, 16, 17)),
    lambda: instances.psd_lp(seed=33, orders=(22, 21, 5)),
    lambda: instances.psd_lp(seed=34, orders=(23, 33), with_q=True),
    lambda: instances.conic_lp(seed=35, nfree=1, nsoc=1, nrsoc=1, nexp=1, npow=1),
    lambda: instances.conic_lp(seed=36, nfree=400, nsoc=70, soc_len=33, nrsoc=5, rsoc_len=65, nexp=300, npow=300),
    lambda: instances.conic_lp(seed=37, nfree=0, nsoc=0, nrsoc=0, nexp=40, npow=33, with_q=True),
], ids=["psd2", "psd to 17", "psd to 22", "psd past the registers", "one of each", "many", "three-slot only"])
def test_iterates_follow_the_oracle(lib, oracle, make):
    """60 iterations agree to 1e-7 of the largest entry: an eigenvalue or
    multiplier is accurate to 1e-12 on either side (Jacobi's and the searches'
    stopping bounds), the projections are nonexpansive, and the ill-conditioned
    exponential blocks get the remaining digits."""
    p = make()
    a, b = _solve_gpu(lib, p, PRM), _solve_oracle(oracle, lib, p, PRM)
    assert a["termination_reason"] == b["termination_reason"]
    for key in ("x", "y"):
        np.testing.assert_allclose(a[key], b[key], rtol=0, atol=1e-7 * max(1.0, np.abs(b[key]).max()))
