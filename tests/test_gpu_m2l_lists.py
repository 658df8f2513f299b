"""M2L lists at the edges of the kernel's batches of 32 sources, every kernel form, against the
oracle's M2L term by term.

Tolerances: the harmonics' recurrences and the contraction are a few P roundings deep, with
cancellation between the terms of a coefficient: 1e-12 (FP64) and 3e-5 (FP32) of the largest sum
of magnitudes of a degree."""
import importlib

import numpy as np
import pytest

from oracle import SPHERICAL, Oracle

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,P", [("f32", 4), ("f32", 8), ("f32", 9), ("f32", 10), ("f32", 12),
                                    ("f64", 7), ("f64", 8), ("f64", 10)])
def test_m2l_list_lengths(prec, P):
    """Targets with 1, 31, 32, 33, 64 and 65 sources against the oracle's M2L term by term."""
    lengths = [1, 31, 32, 33, 64, 65]
    rng = np.random.default_rng(P)
    nt, ns = len(lengths), max(lengths)
    X = np.concatenate([rng.uniform(-0.3, 0.3, (nt, 3)), np.zeros((ns, 3))])
    d = rng.standard_normal((ns, 3))
    X[nt:] = d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(2.5, 4, (ns, 1))
    if prec == "f32":
        X = X.astype(np.float32).astype(float)
    m, nterm = nt + ns, P * (P + 1) // 2
    M = np.zeros((m, nterm), complex)
    M[nt:] = rng.standard_normal((ns, nterm)) + 1j * rng.standard_normal((ns, nterm))
    scale = np.array([1.0 / np.prod(np.arange(1, 2 * j + 1), dtype=float) ** 0.5
                      for j in range(P) for _ in range(j + 1)])
    M *= scale
    for j in range(P):
        M[:, j * (j + 1) // 2] = M[:, j * (j + 1) // 2].real
    if prec == "f32":
        M = M.real.astype(np.float32).astype(float) + 1j * M.imag.astype(np.float32).astype(float)
    s = fmm.Solver(P=P, precision=prec)
    s.set_bodies(np.zeros((1, 3)), np.ones(1))
    z = np.zeros(m, int)
    s.kernel_set_cells(X, np.ones(m), z, z, z, z, z)
    s.kernel_set_expansion(0, M)
    s.kernel_set_expansion(1, None)
    ci = np.concatenate([np.full(k, t) for t, k in enumerate(lengths)])
    cj = np.concatenate([nt + rng.permutation(ns)[:k] for k in lengths])
    s.kernel_m2l(ci, cj)
    got = s.expansion(1)
    o = Oracle("f64")
    for t, k in enumerate(lengths):
        ref, mag = np.zeros(nterm, complex), np.zeros(nterm)
        for j in cj[ci == t]:
            row = np.stack([M[j].real, M[j].imag], 1).ravel()
            L = o.op_m2l(SPHERICAL, P, X[t], X[j], row, np.zeros(2 * nterm))
            L = L[0::2] + 1j * L[1::2]
            ref += L
            mag += np.abs(L)
        # within a degree every coefficient is a sum of terms of the degree's size
        for n in range(P):
            sl = slice(n * (n + 1) // 2, (n + 1) * (n + 2) // 2)
            tol = (3e-5 if prec == "f32" else 1e-12) * mag[sl].max()
            assert np.abs(got[t, sl] - ref[sl]).max() <= tol, (k, n)
