"""The work that a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes what a program holds
before the call (inputs from the seed alone, problem objects, device handles,
networks), ``run`` takes one pass through the public entry points of
``pdhcg_b200`` and returns all of its outputs.

Every kind stands for one use of the framework:

- ``lp``         a small LP or diagonal QP through ``native.solve``: problem
                 build, solve and result copies, where launches and latency count
- ``family``     one instance of a parametric QP family from host buffers with a
                 warm start, a primal weight and the family's step size
- ``conic``      an LP or diagonal QP with SOC, rotated-SOC, exponential and power blocks
- ``sdp``        an LP with PSD blocks of several orders
- ``soc``        the SOC-constrained QP, resident on the device or from host
                 buffers, in FP64 or mixed precision
- ``sparse_q``   a QP with a sparse Q (inner Barzilai-Borwein solve)
- ``portfolio``  a low-rank portfolio QP with dense rows (inner solve over a dense R)
- ``mpc``        a batch of uneven MPC QPs in one call
- ``train``      fit of the warm-start network: forward, backward, Adam
- ``predict``    one prediction of the warm-start network
- ``spmv``       the CSR product on device arrays

Whole solves run to the relative KKT error that is named (or to the iteration
limit that bounds a drawn case).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from pdhcg_b200 import capi, instances, native, warmstart
from pdhcg_b200.capi import Cone, CsrMatrix, Problem

DEV = "cuda"


def listed():
    return [
        # the smallest solve: an LP of a few hundred rows at the default tolerance
        {"name": "lp_small", "kind": "lp", "n": 300, "m": 150, "with_q": False},
        # one instance of a parametric family, warm-started as WarmStart.solve does
        {"name": "family_warm", "kind": "family", "n": 50000, "dim": 32},
        # every kind of small cone block beside free variables, diagonal Q, cold start
        {"name": "conic_mixed_blocks", "kind": "conic", "nfree": 2000, "nsoc": 200, "soc_len": 30, "nrsoc": 60,
         "rsoc_len": 16, "nexp": 60, "npow": 60, "with_q": True},
        # PSD blocks of orders 2 to 20
        {"name": "sdp_blocks", "kind": "sdp", "nfree": 200, "blocks": 38, "max_order": 20},
        # the headline instance: 1e6 variables in 20000 blocks, mixed precision, resident
        {"name": "soc_resident_mixed", "kind": "soc", "blocks": 20000, "block": 50, "mixed": True, "host": False},
        # the same kind at a fifth of the size from host buffers, plain FP64
        {"name": "soc_host_fp64", "kind": "soc", "blocks": 4000, "block": 50, "mixed": False, "host": True},
        # the sparse convex QP of 1e4 variables
        {"name": "sparse_q", "kind": "sparse_q", "scale": 1.0, "mixed": False},
        # 2e5 assets, rank 100: the largest working set
        {"name": "portfolio", "kind": "portfolio", "n": 200000, "rank": 100, "sectors": 500, "mixed": False},
        # a batch of control problems with horizons 10 to 100
        {"name": "mpc_batch", "kind": "mpc", "count": 1024, "tmin": 10, "tmax": 100},
        # the warm-start network over 256 collected solves, minibatches of 64
        {"name": "mlp_train", "kind": "train", "in": 32, "hidden": 512, "rank": 64, "out": 75000, "count": 256,
         "batch": 64, "epochs": 40},
        # one parameter vector to one starting point
        {"name": "mlp_predict", "kind": "predict", "in": 32, "hidden": 512, "rank": 64, "out": 75000, "batch": 1},
        # the headline instance's matrix times a vector
        {"name": "spmv", "kind": "spmv", "m": 500000, "n": 1000000, "per_row": 10, "ragged": False},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["lp", "family", "conic", "sdp", "soc", "soc", "sparse_q", "portfolio", "mpc", "train", "predict",
                       "spmv"])
    if kind == "lp":
        n = log(40, 4000)
        return {"kind": kind, "n": n, "m": max(5, int(n * rng.uniform(0.2, 0.8))), "with_q": rng.random() < 0.5}
    if kind == "family":
        return {"kind": kind, "n": 2 * log(1000, 25000), "dim": rng.randint(4, 32)}
    if kind == "conic":
        return {"kind": kind, "nfree": log(30, 2000), "nsoc": log(4, 200), "soc_len": rng.randint(4, 60),
                "nrsoc": log(2, 60), "rsoc_len": rng.randint(4, 40), "nexp": rng.randint(0, 60),
                "npow": rng.randint(0, 60), "with_q": rng.random() < 0.7}
    if kind == "sdp":
        return {"kind": kind, "nfree": log(20, 200), "blocks": log(3, 38), "max_order": rng.randint(3, 20)}
    if kind == "soc":
        block = rng.randint(8, 100)
        return {"kind": kind, "blocks": log(100, 1000000 // block), "block": block, "mixed": rng.random() < 0.5,
                "host": rng.random() < 0.5}
    if kind == "sparse_q":
        return {"kind": kind, "scale": math.exp(rng.uniform(math.log(0.03), 0.0)), "mixed": rng.random() < 0.3}
    if kind == "portfolio":
        return {"kind": kind, "n": log(4000, 150000), "rank": rng.randint(8, 100), "sectors": rng.randint(10, 500),
                "mixed": rng.random() < 0.5}
    if kind == "mpc":
        tmin = rng.randint(5, 40)
        return {"kind": kind, "count": log(8, 700), "tmin": tmin, "tmax": rng.randint(tmin, 100)}
    if kind == "train":
        batch = rng.randint(8, 64)
        return {"kind": kind, "in": rng.randint(4, 48), "hidden": rng.randint(32, 512), "rank": rng.randint(8, 64),
                "out": log(1500, 75000), "count": batch * rng.randint(1, 4) + rng.randint(0, 7), "batch": batch,
                "epochs": rng.randint(2, 30)}
    if kind == "predict":
        return {"kind": kind, "in": rng.randint(4, 48), "hidden": rng.randint(32, 512), "rank": rng.randint(8, 64),
                "out": log(1500, 75000), "batch": log(1, 64)}
    m = log(5000, 500000)
    per_row = min(rng.randint(2, 40), max(2, 5000000 // m))
    return {"kind": "spmv", "m": m, "n": max(50, int(m * rng.uniform(0.5, 2.0))), "per_row": per_row,
            "ragged": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _random_cols(g, m, n, k):
    """m x k distinct sorted uniform columns, as instances.random_csr draws them."""
    cols = torch.randint(0, n, (m, k), generator=g, device=DEV, dtype=torch.int32).sort(1).values
    for _ in range(64):
        dup = torch.zeros_like(cols, dtype=torch.bool)
        dup[:, 1:] = cols[:, 1:] == cols[:, :-1]
        nd = int(dup.sum())
        if nd == 0:
            break
        cols[dup] = torch.randint(0, n, (nd,), generator=g, device=DEV, dtype=torch.int32)
        cols = cols.sort(1).values
    return cols


def _np(t):
    return t.cpu().numpy()


def _diag(n, q):
    return CsrMatrix(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), q)


def _soc_problem(case, seed):
    """instances.soc_qp's shapes and distributions, drawn on the device."""
    g = _gen(seed)
    nb, L = case["blocks"], case["block"]
    n = nb * L
    m = n // 2
    k = min(10, n)
    cols = _random_cols(g, m, n, k)
    vals = torch.randn((m, k), generator=g, device=DEV, dtype=torch.float64)
    q = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 0.99 + 0.01
    c = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    x0 = torch.randn((nb, L), generator=g, device=DEV, dtype=torch.float64)
    x0[:, -1] = x0[:, :-1].norm(dim=1) + 1.0
    b = _np((vals * x0.reshape(-1)[cols.long()]).sum(1))
    A = CsrMatrix(m, n, np.arange(0, (m + 1) * k, k, dtype=np.int32), _np(cols).reshape(-1), _np(vals).reshape(-1))
    return Problem(c=_np(c), A=A, con_lb=b, con_ub=b.copy(), var_lb=np.full(n, -np.inf), var_ub=np.full(n, np.inf),
                   Q=_diag(n, _np(q)), cones=[Cone(capi.CONE_STANDARD_SOC, i * L, L - 2) for i in range(nb)])


def _portfolio_problem(case, seed):
    """instances.portfolio's shapes and distributions, the CSR arrays laid out directly."""
    g = _gen(seed)
    rng = np.random.default_rng(seed)
    n, k = case["n"], case["rank"]
    nsec = max(2, min(case["sectors"], n // 20))
    R = _np(torch.randn((k, n), generator=g, device=DEV, dtype=torch.float64) / math.sqrt(n))
    Dd = rng.uniform(0.5, 2.0, k)
    N = n + k + 2
    sec = rng.integers(0, nsec, n)
    z0 = np.sqrt(Dd) * R.mean(1)
    te2 = 1.5 * float(z0 @ z0) + 1e-8
    base = 1 + nsec
    m = base + k + 2
    expo_c = np.tile(np.arange(n + 1, dtype=np.int32), (k, 1))
    expo_c[:, n] += np.arange(k, dtype=np.int32)
    expo_v = np.concatenate([-np.sqrt(Dd)[:, None] * R, np.ones((k, 1))], axis=1)
    counts = np.concatenate([[n], np.bincount(sec, minlength=nsec), np.full(k, n + 1), [1, 1]])
    A = CsrMatrix(m, N, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32),
                  np.concatenate([np.arange(n, dtype=np.int32), np.argsort(sec, kind="stable").astype(np.int32),
                                  expo_c.ravel(), np.array([n + k, n + k + 1], np.int32)]),
                  np.concatenate([np.ones(2 * n), expo_v.ravel(), np.ones(2)]))
    lo, up = np.full(m, -np.inf), np.full(m, np.inf)
    lo[0] = up[0] = 1.0
    up[1:base] = 0.05 * 500.0 / nsec  # the cap of 500 sectors, scaled so that fewer sectors stay feasible
    lo[base:base + k] = up[base:base + k] = 0.0
    lo[base + k] = up[base + k] = 0.5 * te2
    lo[base + k + 1] = up[base + k + 1] = 1.0
    Rfull = np.zeros((k, N))
    Rfull[:, :n] = R
    Q = CsrMatrix(N, N, np.concatenate([np.arange(n + 1), np.full(k + 2, n)]).astype(np.int32),
                  np.arange(n, dtype=np.int32), rng.uniform(1e-4, 1e-2, n))
    return Problem(c=np.concatenate([-rng.uniform(0.0, 1e-3, n), np.zeros(k + 2)]), A=A, con_lb=lo, con_ub=up,
                   var_lb=np.concatenate([np.zeros(n), np.full(k + 2, -np.inf)]),
                   var_ub=np.concatenate([np.full(n, 0.02 * max(1.0, 2e5 / n / 40)), np.full(k + 2, np.inf)]),
                   Q=Q, R_dense=Rfull, D=CsrMatrix(k, k, np.arange(k + 1, dtype=np.int32), np.arange(k, dtype=np.int32), Dd),
                   cones=[Cone(capi.CONE_ROTATED_SOC, n, k)])


def _problem(case, seed):
    kind = case["kind"]
    if kind == "lp":
        make = instances.diag_qp if case["with_q"] else instances.box_lp
        return make(seed, case["n"], case["m"])
    if kind == "conic":
        return instances.conic_lp(seed, **{k: case[k] for k in ("nfree", "nsoc", "soc_len", "nrsoc", "rsoc_len", "nexp",
                                                                "npow", "with_q")})
    if kind == "sdp":
        orders = [2 + i % (case["max_order"] - 1) for i in range(case["blocks"])]
        return instances.psd_lp(seed, case["nfree"], orders)
    if kind == "soc":
        return _soc_problem(case, seed)
    if kind == "sparse_q":
        return instances.sparse_qp(seed, case["scale"])
    return _portfolio_problem(case, seed)


# eps and iteration limit of every kind's solves: the default tolerance for the
# small problems, 1e-6 for the benchmark's workloads, 1e-5 for the batch.  The
# limits leave the listed cases room to converge and bound the drawn ones.
EPS = {"lp": 1e-4, "family": 1e-6, "conic": 1e-4, "sdp": 1e-4, "soc": 1e-6, "sparse_q": 1e-6, "portfolio": 1e-6,
       "mpc": 1e-5}
LIMIT = {"lp": 20000, "family": 6000, "conic": 2500, "sdp": 1000, "soc": 4000, "sparse_q": 1300, "portfolio": 3000,
         "mpc": 4000}


def _params(kind):
    return {"termination_criteria.eps_optimal_relative": EPS[kind],
            "termination_criteria.eps_feasible_relative": EPS[kind],
            "termination_criteria.iteration_limit": LIMIT[kind]}


class _DeviceArray:
    """float64 device memory of the library, for torch.as_tensor; a tensor
    over it keeps its owner."""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (int(ptr), False), "version": 3}


class _State:
    """What one prepared case holds; library objects go back with it."""

    def __init__(self):
        self.lib = native.load()
        self.probs, self.handle, self.net = [], None, None

    def __del__(self):
        for p in self.probs:
            self.lib.qp_problem_free(p)
        if self.handle:
            self.lib.pdhcg_b200_device_problem_free(self.handle)
        if self.net:
            self.lib.pdhcg_b200_mlp_free(self.net)


def _fptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def _params_of(net, lib):
    out = np.empty(lib.pdhcg_b200_mlp_num_params(net), np.float32)
    if lib.pdhcg_b200_mlp_get_params(net, _fptr(out)) != 0:
        raise RuntimeError("pdhcg_b200_mlp_get_params failed")
    return out


def _weights(case, seed):
    """Packed initial parameters, uniform of the layers' fan-in, small biases."""
    rng = np.random.default_rng(int(seed) + 77)
    i, h, r, o = case["in"], case["hidden"], case["rank"], case["out"]
    parts = []
    for fan_in, fan_out, relu in ((i, h, True), (h, h, True), (h, r, False), (r, o, False), (h, 1, False)):
        a = math.sqrt(6.0 / fan_in) if relu else math.sqrt(6.0 / (fan_in + fan_out))
        parts.append(a * (2.0 * rng.random(fan_in * fan_out, dtype=np.float32) - 1.0))
        parts.append(0.02 * rng.standard_normal(fan_out, dtype=np.float32))
    return np.concatenate(parts).astype(np.float32)


def _train_data(case, seed):
    """Parameters, normalised targets that follow them, log primal weights."""
    rng = np.random.default_rng(seed)
    B, d, o = case["count"], case["in"], case["out"]
    theta = rng.standard_normal((B, d)).astype(np.float32)
    mix = rng.standard_normal((d, o)).astype(np.float32) / np.float32(math.sqrt(d))
    target = (np.tanh(theta @ mix) + 0.1 * rng.standard_normal((B, o), dtype=np.float32)).astype(np.float32)
    return theta, target, (0.3 * theta[:, 0] + 0.1 * rng.standard_normal(B)).astype(np.float32)


def _spmv_data(case, seed):
    g = _gen(seed)
    m, n, k = case["m"], case["n"], case["per_row"]
    if case["ragged"]:  # row lengths 0 .. 2k, columns with repeats allowed
        lens = torch.randint(0, 2 * k + 1, (m,), generator=g, device=DEV)
        rp = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
        rp[1:] = lens.cumsum(0)
        cols = torch.randint(0, n, (int(rp[-1]),), generator=g, device=DEV, dtype=torch.int32)
    else:
        rp = torch.arange(m + 1, device=DEV, dtype=torch.int64) * k
        cols = _random_cols(g, m, n, k).reshape(-1)
    val = torch.randn(cols.numel(), generator=g, device=DEV, dtype=torch.float64)
    x = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    return rp.to(torch.int32), cols.contiguous(), val, x


def prepare(case, seed):
    kind = case["kind"]
    s = _State()
    lib = s.lib
    s.case = case
    if kind == "spmv":
        s.rp, s.cols, s.val, s.x = _spmv_data(case, seed)
        s.y = torch.empty(case["m"], dtype=torch.float64, device=DEV)
        torch.cuda.synchronize()
        return s
    if kind in ("train", "predict"):
        s.net = lib.pdhcg_b200_mlp_create(case["in"], case["hidden"], case["rank"], case["out"], int(seed) & 0xffffffff)
        if not s.net or lib.pdhcg_b200_mlp_set_params(s.net, _fptr(_weights(case, seed))) != 0:
            raise RuntimeError("pdhcg_b200_mlp_create failed")
        if kind == "train":
            s.theta, s.target, s.lw = _train_data(case, seed)
        else:
            s.theta = np.random.default_rng(seed).standard_normal((case["batch"], case["in"])).astype(np.float32)
            s.out = np.empty((case["batch"], case["out"]), np.float32)
            s.lw = np.empty(case["batch"], np.float32)
        return s
    s.prm = capi.default_params(lib, **_params(kind))
    s.opts = native.default_options()
    if kind == "mpc":
        hor = np.random.default_rng(4).integers(case["tmin"], case["tmax"] + 1, size=case["count"])
        qps = [instances.mpc_qp(int(seed) * 1000003 + i, int(t)) for i, t in enumerate(hor)]
        s.keep = [capi.build(lib, p) for p in qps]
        s.probs = [b[0] for b in s.keep]
        s.arr = (C.POINTER(capi.QpProblem) * len(qps))(*s.probs)
        s.sizes = [(p.n, p.A.m) for p in qps]
        s.bopts = native.BatchOptions()
        lib.pdhcg_b200_default_batch_options(C.byref(s.bopts))
        return s
    if kind == "family":
        fam = warmstart.ParametricQP(seed=int(seed) % (1 << 31), n=case["n"], dim=case["dim"])
        mid, off = fam.thetas(2, int(seed) + 1)
        first = native.solve(fam.problem(mid), _params(kind))  # a neighbouring solved instance
        st = native.last_stats()
        s.problem = fam.problem(mid + 0.3 * off)
        s.problem.primal_start, s.problem.dual_start = first["x"], first["y"]
        s.opts.has_initial_primal_weight, s.opts.initial_primal_weight = 1, st["primal_weight"]
        s.opts.has_initial_step_size, s.opts.initial_step_size = 1, st["step_size"]
    else:
        s.problem = _problem(case, seed)
    s.n, s.m = s.problem.n, s.problem.A.m
    if kind == "lp":
        return s
    if case.get("mixed"):
        s.opts.precision = 1
    prob, s.keep = capi.build(lib, s.problem)
    if not prob:
        raise RuntimeError("create_qp_problem rejected the problem")
    s.probs = [prob]
    if kind == "portfolio" or (kind == "soc" and not case["host"]):
        s.opts.solution_on_device = 1
        s.handle = lib.pdhcg_b200_upload(prob)
        if not s.handle:
            raise RuntimeError("pdhcg_b200_upload failed")
        lib.qp_problem_free(prob)
        s.probs, s.problem, s.keep = [], None, None
    return s


def run(s):
    case, lib = s.case, s.lib
    kind = case["kind"]
    if kind == "spmv":
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if lib.pdhcg_b200_csr_spmv(case["m"], s.rp.data_ptr(), s.cols.data_ptr(), s.val.data_ptr(), s.x.data_ptr(),
                                   s.y.data_ptr(), stream) != 0:
            raise RuntimeError("pdhcg_b200_csr_spmv failed")
        return s.y
    if kind == "train":
        loss = C.c_double()
        if lib.pdhcg_b200_mlp_train(s.net, case["count"], _fptr(s.theta), _fptr(s.target), _fptr(s.lw), case["epochs"],
                                    case["batch"], 1e-3, C.byref(loss)) != 0:
            raise RuntimeError("pdhcg_b200_mlp_train failed")
        return {"params": _params_of(s.net, lib), "loss": loss.value}
    if kind == "predict":
        if lib.pdhcg_b200_mlp_predict(s.net, case["batch"], _fptr(s.theta), _fptr(s.out), _fptr(s.lw)) != 0:
            raise RuntimeError("pdhcg_b200_mlp_predict failed")
        return {"out": s.out, "logw": s.lw}
    if kind == "mpc":
        res = (C.POINTER(capi.PdhcgResult) * len(s.sizes))()
        if lib.pdhcg_b200_solve_batch(len(s.sizes), s.arr, C.byref(s.prm), C.byref(s.bopts), res) != 0:
            raise RuntimeError("pdhcg_b200_solve_batch failed")
        x = np.empty(sum(n for n, _ in s.sizes))
        y = np.empty(sum(m for _, m in s.sizes))
        px, py = x.ctypes.data, y.ctypes.data
        for r, (n, m) in zip(res, s.sizes):
            c = r.contents
            C.memmove(px, c.primal_solution, 8 * n)
            C.memmove(py, c.dual_solution, 8 * m)
            px += 8 * n
            py += 8 * m
            lib.pdhcg_result_free(r)
        return {"x": x, "y": y}
    if kind == "lp":
        d = native.solve(s.problem, _params(kind), s.opts)
        return {k: d[k] for k in ("x", "y", "rc")}
    if s.handle:
        r = lib.pdhcg_b200_solve_device(s.handle, C.byref(s.prm), C.byref(s.opts))
        if not r:
            raise RuntimeError("pdhcg_b200_solve_device failed")
        lib.pdhcg_result_free(r)
        p = [C.c_void_p() for _ in range(3)]
        if lib.pdhcg_b200_device_solution(s.handle, *[C.byref(v) for v in p]) != 0:
            raise RuntimeError("pdhcg_b200_device_solution failed")
        return {k: torch.as_tensor(_DeviceArray(s, v.value, n), device=DEV)
                for k, v, n in zip(("x", "y", "rc"), p, (s.n, s.m, s.n))}
    r = lib.pdhcg_b200_solve(s.probs[0], C.byref(s.prm), C.byref(s.opts))
    if not r:
        raise RuntimeError("pdhcg_b200_solve failed")
    d = capi.result_dict(r, s.n, s.m)
    lib.pdhcg_result_free(r)
    return {k: d[k] for k in ("x", "y", "rc")}


# ---- what a pass cannot do without ------------------------------------------

# iterations that a solve of the kind takes to its tolerance (inner ones too
# where there is an inner solve), for the work below: each reads the matrices
# once per product and its vectors once
ITERS = {"lp": 600, "family": 500, "conic": 1200, "sdp": 500, "soc": 1900, "sparse_q": 1100, "portfolio": 2700,
         "mpc": 540}
INNER = {"sparse_q": 56, "portfolio": 4.2}  # passes over the quadratic term per outer iteration


def work(case):
    kind = case["kind"]
    if kind == "spmv":
        nnz = case["m"] * case["per_row"]
        return {"bytes": 12 * nnz + 4 * (case["m"] + 1) + 8 * (case["m"] + case["n"]), "flops": 2 * nnz}
    if kind in ("train", "predict"):
        i, h, r, o = case["in"], case["hidden"], case["rank"], case["out"]
        weights = h * i + h * h + r * h + o * r
        params = weights + 2 * h + r + o + h + 1
        if kind == "predict":
            return {"bytes": 2 * weights + 4 * (params - weights) + 4 * case["batch"] * (i + o + 1),
                    "flops": 2 * case["batch"] * weights}
        steps = case["count"] // case["batch"] * case["epochs"]
        # a step reads and writes weight, momentum and velocity, reads the BF16 copy and the targets
        return {"bytes": steps * (24 * params + 4 * weights + 4 * case["batch"] * (o + i + 1)),
                "flops": steps * 6 * case["batch"] * weights}
    its = ITERS[kind]
    vb = 4 if case.get("mixed") else 8
    if kind == "mpc":  # an instance is read once and solved on chip
        t = 0.5 * (case["tmin"] + case["tmax"])
        nnz, n, m = instances.mpc_nnz(int(t)), 12 * t, 8 * t
        return {"bytes": case["count"] * (12 * nnz + 8 * (6 * n + 4 * m)),
                "flops": case["count"] * its * (4 * nnz + 20 * (n + m))}
    extra = 0.0
    if kind == "lp":
        n, m, nnz = case["n"], case["m"], 6 * case["m"]
    elif kind == "family":
        n, m, nnz = case["n"], case["n"] // 2, 3 * case["n"]
    elif kind == "conic":
        n = (case["nfree"] + case["nsoc"] * case["soc_len"] + case["nrsoc"] * case["rsoc_len"] +
             3 * (case["nexp"] + case["npow"]))
        m, nnz = n // 3, 5 * (n // 3)
    elif kind == "sdp":
        orders = [2 + i % (case["max_order"] - 1) for i in range(case["blocks"])]
        n = case["nfree"] + sum(k * (k + 1) // 2 for k in orders)
        m, nnz = n // 3, 5 * (n // 3)
    elif kind == "soc":
        n = case["blocks"] * case["block"]
        m, nnz = n // 2, 10 * (n // 2)
    elif kind == "sparse_q":
        n = max(20, int(10000 * case["scale"]))
        m, nnz = n // 2, 8 * (n // 2)
        extra = INNER[kind] * (4.2 * n * (vb + 4) + 40 * n)
    else:
        n, k = case["n"], case["rank"]
        m, nnz = case["sectors"] + k + 3, n * (2 + k)
        extra = INNER[kind] * (k * n * vb + 40 * n)
    step = 2 * nnz * (vb + 4) + 9 * n * vb + 6 * m * vb + extra
    return {"bytes": its * step, "flops": its * (4 * nnz + 20 * (n + m) + extra / 4)}


def tolerance(case):
    return TOL[case["kind"]]


# Whole solves: about four times the largest relative change of x, y or the
# reduced cost seen over seeds when A's rows (and, in lp and sparse_q, the
# variables) are permuted, so that every product and reduction adds in another
# order: lp 7e-7, conic 1.5e-6, sdp 2e-11, soc 1.4e-8 (mixed), sparse_q 4e-7,
# portfolio 9e-4 (y only: its sector rows are nearly degenerate), with room in
# the small ones for a seed whose restart falls on another evaluation.  The
# batch holds FP32 iterates and an instance may stop one evaluation earlier or
# later.  The network: BF16 weights, whose rounding a training run carries on
# (1e-3 against 64 bits), 5e-6 in one prediction.
TOL = {"lp": {"rel": 1e-5, "max": 1e-3}, "family": {"rel": 1e-5, "max": 1e-3}, "conic": {"rel": 1e-5, "max": 1e-3},
       "sdp": {"rel": 1e-7, "max": 1e-5}, "soc": {"rel": 1e-6, "max": 1e-4}, "sparse_q": {"rel": 5e-6, "max": 5e-4},
       "portfolio": {"rel": 4e-3, "max": 5e-2}, "mpc": {"rel": 1e-3, "max": 5e-2}, "train": {"rel": 4e-3, "max": 0.5},
       "predict": {"rel": 2.5e-5, "max": 1e-3}, "spmv": {"rel": 1e-14, "max": 1e-11}}


# ---- the same in 64 bits -----------------------------------------------------

def _layers(case, p):
    """The packed parameters (W1, b1, W2, b2, W3, b3, U, bu, wp, bp) as views."""
    i, h, r, o = case["in"], case["hidden"], case["rank"], case["out"]
    shapes = [(h, i), (h,), (h, h), (h,), (r, h), (r,), (o, r), (o,), (h,), (1,)]
    out, at = [], 0
    for sh in shapes:
        k = math.prod(sh)
        out.append(p[at:at + k].view(sh))
        at += k
    return out


def _bf16(w):
    """The BF16 copy of a weight that the products read."""
    return w.float().bfloat16().double()


def _forward(layers, x):
    W1, b1, W2, b2, W3, b3, U, bu, wp, bp = layers
    h1 = torch.relu(x @ _bf16(W1).T + b1)
    h2 = torch.relu(h1 @ _bf16(W2).T + b2)
    z = h2 @ _bf16(W3).T + b3
    return h1, h2, z, z @ _bf16(U).T + bu, h2 @ wp + bp


def exact(case, seed):
    """None for whole solves: any point within the tolerance is an answer, and
    which one it is depends on where the iteration stops."""
    kind = case["kind"]
    if kind == "spmv":
        rp, cols, val, x = _spmv_data(case, seed)
        rows = torch.repeat_interleave(torch.arange(case["m"], device=DEV), (rp[1:] - rp[:-1]).long())
        return torch.zeros(case["m"], dtype=torch.float64, device=DEV).index_add_(0, rows, val * x[cols.long()])
    if kind == "predict":
        theta = np.random.default_rng(seed).standard_normal((case["batch"], case["in"])).astype(np.float32)
        o = _forward(_layers(case, torch.from_numpy(_weights(case, seed)).to(DEV).double()), torch.from_numpy(theta).to(DEV).double())
        return {"out": o[3], "logw": o[4]}
    if kind != "train":
        return None
    theta, target, lw = (torch.from_numpy(a).to(DEV).double() for a in _train_data(case, seed))
    p = torch.from_numpy(_weights(case, seed)).to(DEV).double()
    mom, vel = torch.zeros_like(p), torch.zeros_like(p)
    grad = torch.zeros_like(p)
    B, step = case["batch"], 0
    for _ in range(case["epochs"]):
        for b0 in range(0, case["count"] - B + 1, B):
            x, t, tl = theta[b0:b0 + B], target[b0:b0 + B], lw[b0:b0 + B]
            L, G = _layers(case, p), _layers(case, grad)
            h1, h2, z, o, l = _forward(L, x)
            dO, dl = 2.0 * (o - t) / o.numel(), 2.0 * (l - tl) / B
            dz = dO @ _bf16(L[6])
            d2 = (dz @ _bf16(L[4]) + dl[:, None] * L[8]) * (h2 > 0)
            d1 = d2 @ _bf16(L[2]) * (h1 > 0)
            for at, v in enumerate((d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), dz.T @ h2, dz.sum(0), dO.T @ z,
                                    dO.sum(0), dl @ h2, dl.sum().view(1))):
                G[at].copy_(v)
            step += 1
            mom.mul_(0.9).add_(grad, alpha=0.1)
            vel.mul_(0.999).addcmul_(grad, grad, value=0.001)
            p -= 1e-3 * (mom / (1 - 0.9 ** step)) / ((vel / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"params": p, "loss": None}  # the loss follows the parameters' path and has no value of its own
