"""Device memory that a new handle holds after its first solve.  Limits in MB, between what the
handle needs and what it held when every array was twice its estimate: the traversal's stacks
and frontiers are the larger part at these sizes."""
import gc
import importlib

import numpy as np
import pytest
import torch

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nt,limit,kw", [
    (16384, 0, 31, dict(P=6, theta=0.4, precision="f64")),
    (31607, 0, 85, dict(P=10, theta=0.35)),
    (50021, 20011, 160, dict(P=8, theta=0.4, precision="f64")),
    (250007, 0, 180, dict(P=6, theta=0.4, tree="uniform")),
])
def test_first_solve_memory(n, nt, limit, kw):
    rng = np.random.default_rng(1)
    x, q = rng.uniform(-1, 1, (n, 3)), rng.uniform(-1, 1, n)

    def handle():
        s = fmm.Solver(use_ropt=0, **kw)
        if nt:
            s.solve_ij(rng.uniform(-1, 1, (nt, 3)), np.ones(nt), x, q)
        else:
            s.solve(x, q)
        return s

    handle().close()  # the kernels' code is loaded at their first launch in a process
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = handle()
    used = (before - torch.cuda.mem_get_info()[0]) / 1e6
    s.close()
    assert used < limit
