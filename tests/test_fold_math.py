"""The folded M2L, M2M and L2L contractions the CUDA kernels run, built for the host (tests/native/
fold_host.cpp), against the oracle's operators: every compiled order, the output orders in one
group and split.  FP64 both sides; a sum of at most a few hundred terms each rounded once:
1e-11 of the largest coefficient, as for the other operators."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oracle import SPHERICAL, Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fold") / "libfold.so"
    subprocess.check_call(["/usr/bin/g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w",
                           "-I", os.path.join(ROOT, "exafmm-dev_b200", "csrc"),
                           os.path.join(ROOT, "tests", "native", "fold_host.cpp"), "-o", str(out)])
    f = C.CDLL(str(out))
    f.fold_m2l.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 4
    return f


@pytest.mark.parametrize("split", [0, 1, 2])
@pytest.mark.parametrize("P", [4, 5, 6, 7, 8, 9, 10, 12])
def test_folded_m2l(P, split, lib):
    op = Oracle("f64").lib.oracle_op_m2l
    op.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 4
    rng = np.random.default_rng(P)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    offsets = [rng.uniform(2, 3, 3) * rng.choice([-1, 1], 3) for _ in range(4)]
    # offsets along the axes: sin(alpha) = 0 and cos(alpha) = 0, beta = 0, pi and +-pi / 2
    offsets += [np.array(v) * 2.5 for v in
                ((0, 0, 1.0), (0, 0, -1.0), (1.0, 0, 0), (-1.0, 0, 0), (0, 1.0, 0), (0, -1.0, 0))]
    for d in offsets:
        Xi = np.ascontiguousarray(rng.uniform(-1, 1, 3))
        Xj = np.ascontiguousarray(Xi - d)
        M = rng.standard_normal(P * (P + 1))
        M[1] = 0.0
        ref, got = np.zeros(P * (P + 1)), np.zeros(P * (P + 1))
        op(SPHERICAL, P, ptr(Xi), ptr(Xj), ptr(M), ptr(ref))
        assert lib.fold_m2l(P, split, ptr(Xi), ptr(Xj), ptr(M), ptr(got)) == 0
        assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("up", [1, 0])
@pytest.mark.parametrize("split", [0, 1, 2])
@pytest.mark.parametrize("P", [4, 5, 6, 7, 8, 9, 10, 12])
def test_folded_shift(P, split, up, lib):
    o = Oracle("f64").lib
    op = o.oracle_op_m2m if up else o.oracle_op_l2l
    op.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 4
    lib.fold_shift.argtypes = [C.c_int] * 3 + [C.c_void_p] * 3
    rng = np.random.default_rng(P + 100)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    # the octants of a child, and shifts along the axes
    offsets = [np.array([a, b, c]) * 0.25 for a in (-1, 1) for b in (-1, 1) for c in (-1, 1)]
    offsets += [rng.uniform(-0.3, 0.3, 3) for _ in range(3)]
    offsets += [np.array(v) * 0.25 for v in ((0, 0, 1.0), (0, 0, -1.0), (1.0, 0, 0), (0, -1.0, 0))]
    for d in offsets:
        X = np.ascontiguousarray(rng.uniform(-1, 1, 3))  # the cell written (M2M parent, L2L child)
        Y = np.ascontiguousarray(X - d)
        d = np.ascontiguousarray(X - Y)
        E = rng.standard_normal(P * (P + 1))
        E[1] = 0.0
        ref, got = np.zeros(P * (P + 1)), np.zeros(P * (P + 1))
        op(SPHERICAL, P, ptr(X), ptr(Y), ptr(E), ptr(ref))
        assert lib.fold_shift(P, up, split, ptr(d), ptr(E), ptr(got)) == 0
        assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
