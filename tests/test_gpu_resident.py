"""The persistent main loop (LP and diagonal QP without cones) against the
oracle's iteration."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdhcg_b200.capi import CsrMatrix, Problem
from test_gpu_solver import _solve_gpu, _solve_oracle

pytestmark = pytest.mark.gpu


def _problem(seed, n, m, with_q, per_row=6):
    rng = np.random.default_rng(seed)
    w = min(per_row, n)
    cols = np.concatenate([rng.choice(n, w, replace=False) for _ in range(m)])
    A = sp.csr_matrix((rng.standard_normal(m * w), (np.repeat(np.arange(m), w), cols)), shape=(m, n))
    A.sort_indices()
    ax = A @ rng.uniform(-1, 1, n)
    lo, up = ax - rng.uniform(0, 1, m), ax + rng.uniform(0, 1, m)
    eq = rng.random(m) < 0.3
    lo[eq] = up[eq] = ax[eq]
    Q = None
    if with_q:
        Q = CsrMatrix(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), rng.uniform(0.05, 1.0, n))
    return Problem(c=rng.standard_normal(n), A=CsrMatrix.from_scipy(A), con_lb=lo, con_ub=up, var_lb=np.full(n, -2.0),
                   var_ub=np.full(n, 2.0), Q=Q)


# one block, one block's edge, several blocks, more than shared memory holds
@pytest.mark.parametrize("n,m", [(1, 1), (2, 1), (1, 3), (31, 33), (511, 200), (512, 513), (513, 511), (1350, 700),
                                 (5000, 2500), (60000, 30000)])
@pytest.mark.parametrize("with_q", [False, True])
def test_iterates_follow_the_oracle(lib, oracle, n, m, with_q):
    """After 170 iterations (restarts among them) x and y agree to 1e-8 of
    their largest entry: the iteration is nonexpansive in the step's metric,
    so the roundings of 170 steps, 1e-16 times the few hundred terms of a
    row's work each, add up to about 1e-11; the primal weight's logarithms and
    ratios at a restart leave three digits of room."""
    p = _problem(n + m, n, m, with_q)
    prm = {"termination_criteria.iteration_limit": 170, "termination_criteria.eps_optimal_relative": 1e-15,
           "termination_criteria.eps_feasible_relative": 1e-15}
    a, b = _solve_gpu(lib, p, prm), _solve_oracle(oracle, lib, p, prm)
    if a["termination_reason"] != b["termination_reason"]:  # a tiny problem may be solved exactly on one side first
        assert n * m <= 4
    for key in ("x", "y"):
        np.testing.assert_allclose(a[key], b[key], rtol=0, atol=1e-8 * max(1.0, np.abs(b[key]).max()))
