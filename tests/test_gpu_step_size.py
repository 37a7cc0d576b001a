"""The step size from a Lanczos process against the oracle's power method."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from pdhcg_b200 import capi, native
from pdhcg_b200.capi import CsrMatrix, Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,kind", [(1, 1, "random"), (1, 40, "random"), (2, 3, "random"), (33, 20, "random"),
                                      (60, 50, "rank one"), (50, 50, "identity"), (700, 900, "random")])
def test_step_size_is_the_power_methods(lib, oracle, m, n, kind, max_iter=5000):
    """0.998 / sigma with the oracle's power method on the same matrix: the
    Lanczos process reproduces its stopping iterate to rounding (1e-9 leaves
    room for the stopping test falling one iterate apart, where the quotients
    differ by the square of the tolerance)."""
    rng = np.random.default_rng(m * 1000 + n)
    if kind == "identity":
        M = sp.identity(n, format="csr")
    elif kind == "rank one":
        M = sp.csr_matrix(np.outer(rng.standard_normal(m), rng.standard_normal(n)))
    else:
        M = sp.random(m, n, density=min(1.0, 8.0 / n), random_state=3, format="csr") + sp.csr_matrix(
            (np.ones(min(m, n)), (np.arange(min(m, n)), np.arange(min(m, n)))), shape=(m, n))
    A = CsrMatrix.from_scipy(sp.csr_matrix(M))
    p = Problem(c=np.ones(n), A=A, con_lb=np.zeros(m), con_ub=np.ones(m), var_lb=np.zeros(n), var_ub=np.ones(n))
    prm = {"l_inf_ruiz_iterations": 0, "has_pock_chambolle_alpha": False, "bound_objective_rescaling": False,
           "termination_criteria.iteration_limit": 1, "sv_max_iter": max_iter}
    native.solve(p, prm)
    full = capi.default_params(lib, **prm)
    dp, ip = C.POINTER(C.c_double), C.POINTER(C.c_int)
    sv = oracle.oracle_sigma_max(m, n, A.row_ptr.ctypes.data_as(ip), A.col_ind.ctypes.data_as(ip),
                                 A.val.ctypes.data_as(dp), full.sv_max_iter, full.sv_tol)
    assert abs(native.last_stats()["step_size"] * sv - 0.998) <= 1e-9


@pytest.mark.parametrize("max_iter", [1, 2**30, 2**31 - 1])  # the last: no limit but the tolerance
def test_iteration_limits_of_the_power_method(lib, oracle, max_iter):
    test_step_size_is_the_power_methods(lib, oracle, 33, 20, "random", max_iter)
