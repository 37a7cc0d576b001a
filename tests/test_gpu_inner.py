"""The inner solves with their own kernels, sparse Q of short rows and dense
low-rank terms, against the oracle at the sizes where their launch shape, tile
grouping or dispatch changes."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdhcg_b200 import instances, native
from pdhcg_b200.capi import CONE_EXPONENTIAL, CONE_STANDARD_SOC, Cone, CsrMatrix
from test_gpu_resident import _problem
from test_gpu_solver import _solve_gpu, _solve_oracle

pytestmark = pytest.mark.gpu

# An inner solve ends by a test on its step (relative 1e-3 of the start's and
# tighter as the outer solve goes on), which rounding may pass one inner
# iteration apart; such a step is below the outer error of 45 iterations by
# far more than the 1e-6 asked for here.
PRM = {"termination_criteria.iteration_limit": 45, "termination_criteria.eps_optimal_relative": 1e-15,
       "termination_criteria.eps_feasible_relative": 1e-15}


def _compare(lib, oracle, p):
    a, b = _solve_gpu(lib, p, PRM), _solve_oracle(oracle, lib, p, PRM)
    assert a["termination_reason"] == b["termination_reason"]
    for key in ("x", "y"):
        np.testing.assert_allclose(a[key], b[key], rtol=0, atol=1e-6 * max(1.0, np.abs(b[key]).max()))


# n and half bandwidth of Q.  Cluster form (up to 64 K entries off the
# diagonal): 128, 512, 1024 variables a block; grid form beyond, 128, 256 a
# block; past the register forms the general kernel
@pytest.mark.parametrize("n,band", [(2, 1), (127, 1), (128, 2), (129, 3), (2048, 1), (2049, 2), (8192, 2), (8193, 2),
                                    (16384, 1), (16385, 1), (8193, 3), (8193, 4), (18944, 2), (18945, 2), (20000, 7),
                                    (40000, 8)])
def test_sparse_q(lib, oracle, n, band):
    rng = np.random.default_rng(n + band)
    p = _problem(n, n, max(1, n // 2), False)
    diags = [np.full(n, 2.0 * band)] + [rng.uniform(-0.9, 0.9, n - d) for d in range(1, band + 1) if d < n]
    Q = sp.diags(diags, range(len(diags)), format="csr")
    p.Q = CsrMatrix.from_scipy(sp.csr_matrix(Q + sp.triu(Q, 1).T))
    _compare(lib, oracle, p)


# more than 16 entries a row: the general kernel, 32 lanes a row, on one block per
# SM up to 148 * 256 / 32 rows and on two beyond
@pytest.mark.parametrize("n", [1184, 1185])
def test_general_kernel_on_one_and_two_blocks_per_sm(lib, oracle, n):
    test_sparse_q(lib, oracle, n, 20)


# The first rows of Q are long (half bandwidth `wide`), the others tridiagonal:
# the fullest block's share fits its shared memory (cluster form, grid form
# where the cluster's 16 blocks do not) or the general kernel is taken
@pytest.mark.parametrize("n,stretch,wide", [(3000, 150, 30), (10000, 500, 30), (60000, 3000, 8), (60000, 3000, 30)])
def test_sparse_q_with_a_dense_stretch(lib, oracle, n, stretch, wide):
    _compare(lib, oracle, _dense_stretch(n, stretch, wide))


def _dense_stretch(n, stretch, wide):
    rng = np.random.default_rng(n + wide)
    p = _problem(n, n, max(1, n // 2), False)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.full(n, 2.0 * wide)]
    for d in range(1, wide + 1):
        at = np.arange(n - 1 if d == 1 else stretch - d)
        v = rng.uniform(-0.9, 0.9, at.size)
        rows += [at, at + d]
        cols += [at + d, at]
        vals += [v, v]
    p.Q = CsrMatrix.from_scipy(sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))),
                                             shape=(n, n)))
    return p


def test_dense_stretch_keeps_its_time(lib):
    """An inner iteration on rows of 61 entries side by side takes no more than
    1.2 times that of the same rows spread over the matrix (the same entries, an
    even share of them in every block)."""
    p = _dense_stretch(10000, 500, 30)
    perm = np.random.default_rng(0).permutation(10000)
    spread = _dense_stretch(10000, 500, 30)
    Q = p.Q.to_scipy()[perm][:, perm]
    Q.sort_indices()
    spread.Q = CsrMatrix.from_scipy(sp.csr_matrix(Q))
    prm = dict(PRM, **{"termination_criteria.iteration_limit": 300})

    def per_inner(q):
        best = np.inf
        for _ in range(3):
            d = native.solve(q, prm)
            best = min(best, native.last_stats()["loop_ms"] / d["total_inner_count"])
        return best

    assert per_inner(p) <= 1.2 * per_inner(spread)


# rows of R around the 16 warps, 4, 8 and 16 rows a warp and the limit of 256
# (FP64 groups of 4 tiles to 64 rows, 2 to 108); widths around the 32 columns
# of a tile and the groups of tiles a block takes
@pytest.mark.parametrize("k,n", [(1, 31), (1, 33), (15, 32), (16, 64), (17, 300), (64, 5000), (65, 5000), (108, 9500),
                                 (109, 4737), (128, 3000), (129, 3000), (256, 700), (257, 700)])
@pytest.mark.parametrize("with_q", [False, True])
def test_dense_low_rank(lib, oracle, k, n, with_q):
    rng = np.random.default_rng(k * 10000 + n)
    p = _problem(n, n, max(1, n // 4), with_q)
    p.R_dense = rng.standard_normal((k, n)) / np.sqrt(n)
    _compare(lib, oracle, p)


# a dense R with a dense middle matrix: up to 64 rows the dense kernel (every block
# applies D in every pass), beyond it the general one; a diagonal one at any rank
@pytest.mark.parametrize("k,dense", [(3, True), (64, True), (65, True), (65, False)])
def test_dense_low_rank_with_a_middle_matrix(lib, oracle, k, dense):
    rng = np.random.default_rng(k)
    p = _problem(k, 900, 200, True)
    p.R_dense = rng.standard_normal((k, 900)) / 30.0
    if dense:
        B = rng.standard_normal((k, k)) / np.sqrt(k)
        p.D = CsrMatrix.from_dense(B @ B.T + 0.1 * np.eye(k))
    else:
        p.D = CsrMatrix.from_scipy(sp.diags(rng.uniform(0.5, 2.0, k), format="csr"))
    _compare(lib, oracle, p)


def _with_tail(k, width, n, cones=()):
    """R over the leading `width` of n variables and of `cones` (type, count,
    slots) behind them."""
    rng = np.random.default_rng(k + width + n)
    p = _problem(k, n + sum(c * w for _, c, w in cones), max(1, n // 8), True, per_row=3)
    p.R_dense = np.zeros((k, p.n))
    p.R_dense[:, :width] = rng.standard_normal((k, width)) / np.sqrt(width)
    at = n
    for kind, count, slots in cones:
        for _ in range(count):
            p.cones.append(Cone(kind, at, 1 if kind == CONE_EXPONENTIAL else slots - 2))
            at += slots
    p.var_lb[n:], p.var_ub[n:] = -np.inf, np.inf
    return p


# variables and cones past R's width: few (the dense kernel), many (the general
# one), and to either side of the line between them
@pytest.mark.parametrize("k,width,n,cones", [
    (64, 1000, 1000, ()), (64, 1000, 1001, ()), (64, 1000, 16000, ()), (64, 1000, 21000, ()), (64, 1000, 100000, ()),
    (64, 20000, 20000, ((CONE_STANDARD_SOC, 500, 12),)), (64, 20000, 20000, ((CONE_STANDARD_SOC, 2000, 12),)),
    (20, 3000, 5000, ((CONE_STANDARD_SOC, 30, 40), (CONE_EXPONENTIAL, 60, 3))),
    (20, 3000, 5000, ((CONE_STANDARD_SOC, 30, 40), (CONE_EXPONENTIAL, 900, 3)))])
def test_dense_low_rank_with_a_tail(lib, oracle, k, width, n, cones):
    _compare(lib, oracle, _with_tail(k, width, n, cones))


def test_a_long_tail_keeps_its_time(lib):
    """R over 1000 of 200000 columns: an inner iteration at rank 64 takes no more
    than 1.3 times one at rank 300 (the general kernel at any tail)."""
    prm = dict(PRM, **{"termination_criteria.iteration_limit": 200})

    def per_inner(q):
        best = np.inf
        for _ in range(3):
            d = native.solve(q, prm)
            best = min(best, native.last_stats()["loop_ms"] / d["total_inner_count"])
        return best

    assert per_inner(_with_tail(64, 1000, 200000)) <= 1.3 * per_inner(_with_tail(300, 1000, 200000))


def test_portfolio_with_columns_of_middle_length(lib, oracle):
    """The exposure rows make every column of A 70 entries long (the product
    with A^T by a warp a column); cone slots follow the columns of R."""
    _compare(lib, oracle, instances.portfolio(seed=11, scale=0.05, rank=70, sectors=40))
