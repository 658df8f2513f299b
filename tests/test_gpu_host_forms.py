"""Host solves in both layouts of the results (p and f apart, 4 n rows): the same bits, for one
set of bodies, a batch and separate target and source sets, empty sets included."""
import importlib

import numpy as np
import pytest

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


def ptr(a):
    return a.ctypes.data


def check(s, n, call_pf, call_rows, got):
    p, f, rows = np.full(n, 1e30), np.full((n, 3), 1e30), np.full((n, 4), 1e30)
    s._check(call_pf(ptr(p), ptr(f)))
    s._check(call_rows(ptr(rows)))
    assert not (rows == 1e30).any()
    assert np.array_equal(rows, np.column_stack([p, f]), equal_nan=True)  # a lone body: 0 / 0
    assert np.array_equal(rows, got, equal_nan=True)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n,m", [(1, 1), (33, 0), (1000, 2500), (5001, 1)])
def test_host_forms(prec, n, m):
    rng = np.random.default_rng(n)
    x, q = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n)
    y, w = rng.uniform(-1, 1, (m, 3)), rng.uniform(0.5, 1, m)
    s = fmm.Solver(P=4, theta=0.5, ncrit=32, precision=prec)
    L, h = s.lib, s.h
    check(s, n, lambda p, f: L.fmm_b200_solve_host(h, n, ptr(x), ptr(q), p, f),
          lambda t: L.fmm_b200_solve_host_trg(h, n, ptr(x), ptr(q), t), s.solve(x, q))
    assert np.array_equal(s.trg(), s.solve(x, q), equal_nan=True)
    counts = np.array([n, 0, m], np.int32)
    xb, qb = np.concatenate([x, y]), np.concatenate([q, w])
    check(s, n + m,
          lambda p, f: L.fmm_b200_solve_batch_host(h, 3, ptr(counts), ptr(xb), ptr(qb), p, f),
          lambda t: L.fmm_b200_solve_batch_host_trg(h, 3, ptr(counts), ptr(xb), ptr(qb), t),
          np.concatenate(s.solve_batch([x, x[:0], y], [q, q[:0], w])))
    check(s, n,
          lambda p, f: L.fmm_b200_solve_ij_host(h, n, ptr(x), ptr(q), m, ptr(y), ptr(w), 1, p, f),
          lambda t: L.fmm_b200_solve_ij_host_trg(h, n, ptr(x), ptr(q), m, ptr(y), ptr(w), 1, t),
          s.solve_ij(x, q, y, w, common_box=True))
