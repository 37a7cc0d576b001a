"""The step's cone launches, blocks of several kinds side by side and PSD
blocks of every order, against the oracle's iteration."""
import ctypes as C

import numpy as np
import pytest
import torch

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


# 402 and 952 thread blocks of free variables and cones (one launch up to 888), PSD
# blocks on 128 threads (to order 20) and on 256
@pytest.mark.parametrize("make", [
    lambda: instances.conic_lp(seed=38, nfree=400, nsoc=1600, soc_len=5, nrsoc=1, nexp=800, npow=800),
    lambda: instances.conic_lp(seed=39, nfree=400, nsoc=3600, soc_len=5, nrsoc=1, nexp=2000, npow=2000),
    lambda: instances.psd_lp(seed=40, orders=(20, 20)), lambda: instances.psd_lp(seed=41, orders=(21, 20, 2)),
    lambda: instances.psd_lp(seed=42, orders=(40,))],
    ids=["one launch", "a launch per kind", "128 threads", "256 threads", "order 40"])
def test_iterates_at_the_launch_rules(lib, oracle, make):
    """As above over 40 iterations: among 2000 random exponential blocks one is so
    ill-conditioned that its two projections are 3e-9 apart, which the primal weight
    of a restart after 40 multiplies by a thousand."""
    p = make()
    prm = dict(PRM, **{"termination_criteria.iteration_limit": 40})
    a, b = _solve_gpu(lib, p, prm), _solve_oracle(oracle, lib, p, prm)
    for key in ("x", "y"):
        np.testing.assert_allclose(a[key], b[key], rtol=0, atol=1e-7 * max(1.0, np.abs(b[key]).max()))


# the largest PSD block that a thread block takes in the residual (83) and in the
# step (112), and the first that a warp takes on device scratch instead
@pytest.mark.parametrize("orders", [(83,), (84,), (112,), (113, 4)])
def test_psd_blocks_past_a_thread_blocks_shared_memory(lib, oracle, orders):
    p = instances.psd_lp(seed=sum(orders), nfree=20, orders=orders)
    prm = dict(PRM, **{"termination_criteria.iteration_limit": 12})
    a, b = _solve_gpu(lib, p, prm), _solve_oracle(oracle, lib, p, prm)
    assert a["termination_reason"] == b["termination_reason"]
    for key in ("x", "y"):
        np.testing.assert_allclose(a[key], b[key], rtol=0, atol=1e-7 * max(1.0, np.abs(b[key]).max()))
    for key in ("relative_primal_residual", "relative_dual_residual"):
        assert abs(a[key] - b[key]) <= 1e-7 * max(1.0, abs(b[key]))


def _positive_part(A):
    """The projection of a symmetric matrix by cyclic Jacobi in extended precision."""
    A, n = A.copy(), len(A)
    V = np.eye(n, dtype=A.dtype)
    for _ in range(40):
        off = A - np.diag(np.diag(A))
        if np.sqrt((off * off).sum()) <= 1e-21 * np.sqrt((A * A).sum()):
            break
        for p in range(n - 1):
            for q in range(p + 1, n):
                if A[p, q] == 0:
                    continue
                h, a = A[q, q] - A[p, p], 2 * A[p, q]
                t = a / (h + np.copysign(np.sqrt(h * h + a * a), h))
                c = 1 / np.sqrt(1 + t * t)
                J = np.array([[c, t * c], [-t * c, c]])
                A[:, [p, q]] = A[:, [p, q]] @ J
                A[[p, q], :] = J.T @ A[[p, q], :]
                V[:, [p, q]] = V[:, [p, q]] @ J
    return (V * np.maximum(np.diag(A), 0)) @ V.T


def test_psd_projection_error(lib):
    """Nearly diagonal matrices of orders 2 to 22 that one sweep diagonalises as far
    as its angles are good: the mean error of the projection, relative to the
    matrix.  It is 1.8e-15 for cyclic Jacobi with the same stopping bound and 3.5e-16
    in round-robin order with angles good to 1e-13; a tangent formed in FP32 alone
    leaves 1e-7 of each entry behind and gives 4.8e-16."""
    rng = np.random.default_rng(5)
    orders, mats, x = [], [], []
    for n in [k for k in range(2, 23) for _ in range(3)]:
        E = 1e-7 * rng.standard_normal((n, n))
        M = np.diag(rng.standard_normal(n)) + E + E.T
        svec = np.concatenate([np.r_[M[c, c], np.sqrt(2) * M[c + 1:, c]] for c in range(n)])
        full, i = np.zeros((n, n), np.longdouble), 0
        for c in range(n):  # the matrix that the rounded svec stands for
            full[c:, c] = full[c, c:] = np.r_[svec[i], svec[i + 1:i + n - c] / np.sqrt(np.longdouble(2))]
            i += n - c
        orders.append(n), mats.append(full), x.append(svec)
    start = np.cumsum([0] + [len(v) for v in x])
    dev = lambda a, t: torch.tensor(np.asarray(a), dtype=t, device="cuda")
    xd, st, vd, ty = dev(np.concatenate(x), torch.float64), dev(start[:-1], torch.int32), dev(orders, torch.int32), \
        dev([4] * len(orders), torch.int32)
    ptr = lambda t: C.c_void_p(t.data_ptr())
    d = torch.ones_like(xd)
    assert lib.pdhcg_b200_project_cones(len(orders), ptr(st), ptr(vd), ptr(ty), None, ptr(xd), ptr(d), None, 0.0, None) == 0
    got, err = xd.cpu().numpy(), []
    for k, (n, M) in enumerate(zip(orders, mats)):
        P = _positive_part(M)
        want = np.concatenate([np.r_[P[c, c], np.sqrt(np.longdouble(2)) * P[c + 1:, c]] for c in range(n)])
        err.append(float(np.sqrt(((got[start[k]:start[k + 1]] - want) ** 2).sum() / (M * M).sum())))
    assert np.mean(err) <= 4.2e-16, (np.mean(err), max(err))
