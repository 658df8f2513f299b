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
    f = C.CDLL(str(out))
    f.tree_first_nodes.argtypes = [C.c_int] * 3 + [C.c_ulonglong]
    f.tree_more_nodes.argtypes = [C.c_ulonglong] * 2
    f.tree_first_nodes.restype = f.tree_more_nodes.restype = C.c_ulonglong
    return f


@pytest.mark.parametrize("n", [1, 2, 1000, 1 << 20, 1 << 29, INT_MAX])
@pytest.mark.parametrize("ncrit", [1, 64, 1 << 28, 1 << 29, (1 << 29) + 1, 1 << 30, INT_MAX])
def test_tree_blocks(n, ncrit, lib):
    for most in (1, 33, 444):
        assert lib.tree_blocks(n, ncrit, most) == max(1, min(most, -(-n // (4 * ncrit))))


@pytest.mark.parametrize("n,ncrit,nroots", [(1, 1, 1), (1000, 64, 1), (1 << 29, 1, 1),
                                            (INT_MAX, 1, 1), (INT_MAX, INT_MAX, 1000000)])
@pytest.mark.parametrize("most", [0, 5000])
def test_tree_nodes(n, ncrit, nroots, most, lib):
    """Room for a tree that never fits: it grows to the limit (0: the builder's own, 2^27 - 1; or a
    lower one), and then there is no more, so the rebuilds end."""
    top = most or 2 ** 27 - 1
    cap = lib.tree_first_nodes(n, ncrit, nroots, most)
    if nroots > top:
        assert cap == 0
        return
    assert cap == min(top, max(1024, 4 * (n // ncrit) + 64 + nroots))
    for _ in range(30):
        more = lib.tree_more_nodes(cap, most)
        if more == 0:
            break
        assert cap < more <= top
        cap = more
    assert more == 0 and cap == top


@pytest.mark.parametrize("sms", [1, 8, 18, 74, 132, 148])
@pytest.mark.parametrize("per", [1, 2, 3, 4])
def test_resident_blocks(sms, per, lib):
    """A launch whose blocks wait on one another never has more than are resident together."""
    most = lib.tree_most(sms, per, 3)
    assert 1 <= most <= sms * per
    for n in (1, 100000, INT_MAX):
        assert 1 <= lib.tree_blocks(n, 1, most) <= sms * per
    assert lib.tree_most(148, per, 3) == 148 * min(per, 3)
