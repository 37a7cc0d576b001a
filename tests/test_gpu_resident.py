"""The persistent main loop (LP and diagonal QP without cones) against the
oracle's iteration."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdhcg_b200 import native
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


# one block, one block's edge, several blocks, a block per SM
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


def _iterates_follow(lib, oracle, p, persistent):
    """As above over 70 iterations, and which loop took them: the persistent one
    launches kernels only at its evaluations, the other two a step."""
    prm = {"termination_criteria.iteration_limit": 70, "termination_criteria.eps_optimal_relative": 1e-15,
           "termination_criteria.eps_feasible_relative": 1e-15}
    a = _solve_gpu(lib, p, prm)
    first = native.last_stats()["kernel_launches"]
    b = _solve_oracle(oracle, lib, p, prm)
    for key in ("x", "y"):
        np.testing.assert_allclose(a[key], b[key], rtol=0, atol=1e-8 * max(1.0, np.abs(b[key]).max()))
    _solve_gpu(lib, p, dict(prm, **{"termination_criteria.iteration_limit": 150}))
    assert (native.last_stats()["kernel_launches"] - first < 80) == persistent


# the most variables of a block (1024 on each of 148 SMs), and one past it
@pytest.mark.parametrize("n,m,persistent", [(151552, 300, True), (151553, 300, False), (75000, 151552, True),
                                            (75000, 151553, False)])
def test_largest_problem_of_the_persistent_loop(lib, oracle, n, m, persistent):
    _iterates_follow(lib, oracle, _problem(n + m, n, m, False, per_row=3 if m > n else 6), persistent)


# rows (columns) of very different lengths side by side: the fullest block's
# share fits its shared memory, or the persistent loop is not taken
@pytest.mark.parametrize("lens,other,columns,persistent", [
    (((200, 50), (2800, 3)), 1500, True, True), (((1000, 60), (20000, 3)), 25000, False, True),
    (((10000, 30), (10000, 2)), 10000, True, True), (((1350, 60), (98650, 3)), 50000, True, False),
    (((1350, 60), (98650, 3)), 100000, False, False)])
def test_uneven_rows(lib, oracle, lens, other, columns, persistent):
    rng = np.random.default_rng(len(lens) + other)
    k = np.concatenate([np.full(c, w) for c, w in lens])
    # distinct columns of a row: a random start and a stride coprime to the width
    rows = np.repeat(np.arange(k.size), k)
    at = np.arange(rows.size) - np.repeat(np.cumsum(k) - k, k)
    cols = (rng.integers(0, other, k.size)[rows] + at * 7919) % other
    M = sp.csr_matrix((rng.standard_normal(rows.size), (rows, cols)), shape=(k.size, other))
    M = sp.csr_matrix(M.T if columns else M)
    M.sort_indices()
    p = _problem(1, M.shape[1], 1, False)
    ax = M @ rng.uniform(-1, 1, M.shape[1])
    p.A, p.con_lb, p.con_ub = CsrMatrix.from_scipy(M), ax - 0.5, ax + 0.5
    _iterates_follow(lib, oracle, p, persistent)
