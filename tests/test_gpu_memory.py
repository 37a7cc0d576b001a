"""A dense low-rank solve on a device with too little memory left for the tiled
copy of R: it runs on the general kernel, which needs none."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
RANK, N = 120, 250000  # 240 MB of tiles
CHILD = r"""
import ctypes as C, sys
import numpy as np, torch
from pdhcg_b200 import capi, native
from test_gpu_resident import _problem
rank, n, take = (int(a) for a in sys.argv[1:4])
p = _problem(1, n, n // 4, True, per_row=2)
p.R_dense = np.random.default_rng(0).standard_normal((rank, n)) / np.sqrt(n)
lib = native.load()
prm = {"termination_criteria.iteration_limit": 6, "termination_criteria.eps_optimal_relative": 1e-15,
       "termination_criteria.eps_feasible_relative": 1e-15}
native.solve(_problem(2, 50, 20, True), prm)
prob, keep = capi.build(lib, p)
full = capi.default_params(lib, **prm)
before = torch.cuda.mem_get_info()[0]
held = torch.empty(before - take, dtype=torch.uint8, device="cuda") if take else None
r = lib.pdhcg_b200_solve(prob, C.byref(full), None)
assert r, "solve failed"
x = capi.result_dict(r, p.n, p.A.m)["x"]
print(before - torch.cuda.mem_get_info()[0], float(np.abs(x).sum()))
"""


def _child(take):
    env = dict(os.environ, CUDA_MODULE_LOADING="EAGER", PYTHONPATH=os.pathsep.join([os.path.dirname(HERE), HERE]))
    out = subprocess.run([sys.executable, "-c", CHILD, str(RANK), str(N), str(take)], env=env, capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    used, total = out.stdout.split()[-2:]
    return int(used), float(total)


def test_without_room_for_the_tiles():
    used, total = _child(0)  # what the solve took from the device, the tiles among it
    _, small = _child(used - RANK * N * 8 // 2)
    assert abs(small - total) <= 1e-6 * total  # another order of the sums
