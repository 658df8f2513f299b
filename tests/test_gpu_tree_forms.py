"""The tree kernel at the sizes where it takes another form: leaves a warp ranks with two or four
bodies per lane, or leaves to the sorts; node arrays that overflow; a tree deeper than the
handle's last one; and the traversal in one launch and by steps.  Trees bit for bit the
oracle's, radii of a whole solve bit for bit those of the stages, lists equal in both forms."""
import importlib

import numpy as np
import pytest

from oracle import Oracle

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


def bodies(kind, n, rng, prec):
    x = rng.uniform(-1, 1, (n, 3))
    if kind == "pairs":  # bodies in close pairs: long chains of single-child nodes
        x[1::2] = x[: 2 * (n // 2) : 2] + rng.uniform(-1, 1, (n // 2, 3)) * 1e-5
    if kind == "clump":  # a clump far deeper than the rest
        x[: n // 3] = 0.3 + rng.uniform(-1, 1, (n // 3, 3)) * 1e-3
    if kind == "same":  # more coincident bodies than any leaf holds: split to the last level
        x[: n // 4] = x[0]
    q = rng.uniform(0.5, 1, n)
    if prec == "f32":
        x, q = x.astype(np.float32).astype(float), q.astype(np.float32).astype(float)
    return np.ascontiguousarray(x), q


def check_tree(s, o, keys=("iparent", "ichild", "nchild", "ibody", "nbody", "level", "X")):
    got, ref = s.cells(), o.cells()
    for k in keys:
        assert np.array_equal(got[k], ref[k]), k
    assert np.array_equal(s.order(), o.order())


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("ncrit", [1, 7, 32, 64, 65, 100, 128, 129, 200])
def test_tree_forms(prec, ncrit):
    """One handle through bodies of every kind, each tree against the oracle's."""
    rng = np.random.default_rng(ncrit)
    s = fmm.Solver(P=4, theta=0.5, ncrit=ncrit, precision=prec, use_ropt=0)
    for kind, n in (("cube", 1), ("cube", 3000), ("pairs", 2001), ("clump", 5003), ("cube", 700),
                    ("clump", 40001), ("same", 900)):
        x, q = bodies(kind, n, rng, prec)
        if kind == "same":
            # the reference recurses without end on coincident bodies: against the stages only
            s.solve(x, q)
            c = s.cells()
            assert c["nbody"][0] == n and c["level"].max() == 21
            leaf = c["nchild"] == 0
            assert c["nbody"][leaf].sum() == n
            order = s.order()
            for b, m in zip(c["ibody"][leaf], c["nbody"][leaf]):
                assert (np.diff(order[b:b + m]) > 0).all()
            continue
        o = Oracle(prec).run(x, q, P=4, theta=0.5, ncrit=ncrit, use_ropt=0,
                             kahan=int(prec == "f32"))
        s.set_bodies(x, q)
        s.build_tree()
        check_tree(s, o)
        s.upward_pass()
        R = s.cells()["R"]
        s.solve(x, q)
        check_tree(s, o)
        assert np.array_equal(s.cells()["R"], R), kind
        for got, ref in zip(s.lists(), (o.m2l(), o.p2p())):
            assert np.array_equal(got, np.sort(ref)), kind


def test_traversal_forms():
    """More cells than the one-launch traversal takes: the first solve of a handle runs it all the
    same, the later ones by steps, after other bodies too."""
    rng = np.random.default_rng(3)
    s = fmm.Solver(P=4, theta=0.5, ncrit=16, use_ropt=0)
    first = {}
    for rep in range(3):
        for kind, n in (("cube", 60001), ("clump", 90001), ("cube", 500)):
            x, q = bodies(kind, n, np.random.default_rng(n), "f32")
            s.solve(x, q)
            lists = s.lists()
            if rep == 0:
                alone = fmm.Solver(P=4, theta=0.5, ncrit=16, use_ropt=0)
                alone.solve(x, q)
                first[n] = alone.lists()
                assert n < 1000 or alone.num_cells()[0] > 8192
            for a, b in zip(lists, first[n]):
                assert np.array_equal(a, b), (rep, kind)
