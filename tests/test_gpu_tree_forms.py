"""The tree kernel at the sizes where it takes another form: leaves a warp ranks with two or four
bodies per lane, or leaves to the sorts; node arrays that overflow; a tree deeper than the
handle's last one; and the traversal with stacks and by steps.  Trees bit for bit the
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
            s.set_bodies(x, q)
            s.build_tree()
            s.upward_pass()
            s.traverse()
            R, lists = s.cells()["R"], s.lists()
            s.solve(x, q)
            assert np.array_equal(s.cells()["R"], R)
            for got, ref in zip(s.lists(), lists):
                assert np.array_equal(got, ref)
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
    """More cells than the traversal with stacks takes: a handle's first solve by all steps, the
    later ones by as many as the last took, with stacks in between."""
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


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_traversal_stack_overflow(prec):
    """Eight distant clumps that no pair of cells is far from at this theta: the frontier stays at
    64 pairs down to the clumps, then every pair becomes 64, more than a block's stack holds."""
    rng = np.random.default_rng(8)
    corner = np.array([[i & 1, i >> 1 & 1, i >> 2] for i in range(8)]) - 0.5
    x = np.concatenate([c + rng.uniform(-1, 1, (768, 3)) * 5e-4 for c in corner])
    q = rng.uniform(0.5, 1, len(x))
    s = fmm.Solver(P=4, theta=1e-5, ncrit=16, precision=prec, use_ropt=0, nspawn=1)
    y, w = bodies("cube", 500, rng, prec)
    for rep in range(2):
        s.solve(x, q)
        c = s.cells()
        leaves = np.flatnonzero(c["nchild"] == 0)
        m2l, p2p = s.lists()
        assert len(m2l) == 0
        ref = (leaves[:, None].astype(np.uint64) << np.uint64(32) | leaves.astype(np.uint64)).ravel()
        assert np.array_equal(p2p, ref)
        s.solve(y, w)


@pytest.mark.parametrize("n", [300, 1000, 6000])
def test_small_tree_grouping(n):
    """Both lists of a small tree grouped together, with images and at a theta that no pair of
    cells is far at: every leaf against every leaf in 27 images, from 200 to 14,000 sources a
    target (a warp's, a block's and the global sort)."""
    x, q = bodies("cube", n, np.random.default_rng(n), "f32")
    s = fmm.Solver(P=4, theta=1e-5, ncrit=32, images=1, cycle=2.0, use_ropt=0)
    s.solve(x, q)
    c = s.cells()
    assert len(c["nchild"]) <= 2048
    leaves = np.flatnonzero(c["nchild"] == 0)
    m2l, p2p = s.lists()
    assert len(m2l) == 0
    img = np.arange(27, dtype=np.int64)
    ref = leaves[:, None, None] << 32 | img[None, :, None] << 27 | leaves[None, None, :]
    assert np.array_equal(p2p, ref.ravel())


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("use_rmax", [1, 0])
@pytest.mark.parametrize("use_ropt", [0, 1])
def test_coincident_bodies_radii(prec, use_rmax, use_ropt):
    """More coincident bodies than a warp ranks, on a fresh handle and on one that has solved
    before: radii and lists of a whole solve are those of the stages, results too."""
    kw = dict(P=4, theta=0.5, ncrit=32, precision=prec, use_rmax=use_rmax, use_ropt=use_ropt)
    x, q = bodies("same", 1600, np.random.default_rng(5), prec)
    y, w = bodies("clump", 3000, np.random.default_rng(6), prec)
    ref = fmm.Solver(**kw)
    ref.set_bodies(x, q)
    ref.build_tree()
    ref.upward_pass()
    ref.traverse()
    ref.downward_pass()
    R, lists, trg = ref.cells()["R"], ref.lists(), ref.trg()
    s = fmm.Solver(**kw)
    for rep in range(2):
        got = s.solve(x, q)
        assert s.cells()["level"].max() == 21
        assert np.array_equal(s.cells()["R"], R), rep
        for a, b in zip(s.lists(), lists):
            assert np.array_equal(a, b), rep
        assert np.array_equal(got, trg)
        s.solve(y, w)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("ncrit", [1 << 29, 1 << 30, 2 ** 31 - 1])
def test_one_leaf(prec, ncrit):
    """An ncrit as large as an int holds: one leaf, the direct sum.  FP32 sums of one sign: 2e-6
    of the magnitudes as in the near-field tests, which the potentials are."""
    x, q = bodies("cube", 777, np.random.default_rng(2), prec)
    s = fmm.Solver(P=4, ncrit=ncrit, precision=prec, use_ropt=0)
    t = s.solve(x, q)
    assert s.num_cells() == (1, 0)
    ref = fmm.direct(x, x, q)
    assert (np.abs(t[:, 0] - ref[:, 0]) <= (2e-6 if prec == "f32" else 1e-13) * ref[:, 0]).all()


def test_traversal_after_stack_overflow():
    """A handle whose traversal has overflowed a block's stack takes steps for a while, for inputs
    that would fit too, and then the stacks again: by the kernels that its solves launch."""
    launches = fmm.load_library().fmm_b200_kernel_launches
    rng = np.random.default_rng(9)
    corner = np.array([[i & 1, i >> 1 & 1, i >> 2] for i in range(8)]) - 0.5
    x = np.concatenate([c + rng.uniform(-1, 1, (768, 3)) * 5e-4 for c in corner])
    y, w = bodies("cube", 500, rng, "f32")
    kw = dict(P=4, theta=1e-5, ncrit=16, use_ropt=0, nspawn=1)

    def count(s):
        n = launches()
        s.solve(y, w)
        return launches() - n

    fresh = fmm.Solver(**kw)
    count(fresh)
    few = count(fresh)
    lists = fresh.lists()
    s = fmm.Solver(**kw)
    s.solve(x, np.ones(len(x)))
    counts = [count(s) for _ in range(40)]
    for a, b in zip(s.lists(), lists):
        assert np.array_equal(a, b)
    assert counts[0] > few and counts[-1] == few
