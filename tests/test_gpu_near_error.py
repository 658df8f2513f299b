"""The FP32 near field against 64 bits on leaves of a few bodies, whose targets several lanes share:
the plain runs between compensated folds must not be longer there than they were when a target
had four lanes at most and every chunk was folded.

Limits: the errors of that form on these bodies (relative 2-norm of the potentials, mean of six
draws, measured) and a tenth; with 32 sources summed plainly throughout, the potentials of mixed
charges stand 21-29 % above them."""
import importlib

import numpy as np
import pytest

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncrit,error", [
    (4000, 2, 6.52e-8), (4000, 8, 6.63e-8), (4000, 16, 7.07e-8),
    (30000, 4, 7.67e-8), (30000, 8, 7.76e-8), (30000, 12, 8.15e-8), (30000, 16, 8.27e-8),
    (30000, 24, 8.25e-8), (30000, 64, 9.95e-8), (30000, 128, 1.045e-7)])
def test_near_field_error(n, ncrit, error):
    e = []
    for seed in range(6):
        rng = np.random.default_rng(seed)
        x = rng.uniform(-1, 1, (n, 3)).astype(np.float32).astype(float)
        q = rng.uniform(-1, 1, n).astype(np.float32).astype(float)
        # an opening angle that no pair of cells meets: the near field alone
        s = fmm.Solver(P=4, theta=1e-5, ncrit=ncrit, use_ropt=0)
        got, ref = s.solve(x, q)[:, 0], fmm.direct(x, x, q)[:, 0]
        e.append(np.linalg.norm(got - ref) / np.linalg.norm(ref))
    assert np.mean(e) <= 1.1 * error
