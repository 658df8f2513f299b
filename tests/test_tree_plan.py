"""The sizes that the host works out for the adaptive tree's build (fmm_tree_plan.cuh), built for
the host: every ncrit and every number of bodies that an int holds."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INT_MAX = 2 ** 31 - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "libplan.so"
    subprocess.check_call(["/usr/bin/g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wall",
                           "-I", os.path.join(ROOT, "exafmm-dev_b200", "csrc"),
                           os.path.join(ROOT, "tests", "native", "tree_plan_host.cpp"), "-o", str(out)])
    return C.CDLL(str(out))


@pytest.mark.parametrize("n", [1, 2, 1000, 1 << 20, 1 << 29, INT_MAX])
@pytest.mark.parametrize("ncrit", [1, 64, 1 << 28, 1 << 29, (1 << 29) + 1, 1 << 30, INT_MAX])
def test_tree_blocks(n, ncrit, lib):
    for most in (1, 33, 444):
        assert lib.tree_blocks(n, ncrit, most) == max(1, min(most, -(-n // (4 * ncrit))))
