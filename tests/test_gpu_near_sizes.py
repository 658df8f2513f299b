"""The near field at the sizes where its kernel changes form: target leaves at the edges of the
lane mapping, source lists at the edges of the chunks and of the teams of warps.  Cells are set
up by hand, so sizes are exact.

Tolerances.  FP64: sums of up to 1e4 terms of one sign for the potential, each within a few
eps (2.2e-16): 1e-13 of the sum of magnitudes.  FP32: a term's relative error is at most about
12 eps (6e-8; three rounded differences, r^2, a reciprocal square root within 2 ulp cubed); a lane
adds up to 16 terms plainly in either half of its sums, and then the halves, before a compensated
fold, which adds none: 16 eps more, 28 in all or 1.7e-6 of the sum of magnitudes: 2e-6."""
import importlib

import numpy as np
import pytest

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


def pair_sums(xt, xs, qs):
    """Potential and gradient of the pairs with r > 0, and the sums of their magnitudes."""
    d = xs[None] - xt[:, None]
    r2 = (d ** 2).sum(2)
    with np.errstate(divide="ignore"):
        inv = np.where(r2 > 0, 1 / np.sqrt(r2), 0)
    t = np.concatenate([(qs * inv)[..., None], (qs * inv ** 3)[..., None] * d], 2)
    mag = np.stack([np.abs(qs * inv), np.abs(qs) * inv ** 2], 2).sum(1)
    return t.sum(1), mag


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("nb", [1, 4, 5, 8, 9, 12, 13, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 72, 80, 95, 96, 97,
                                129, 145])
@pytest.mark.parametrize("src", [(1,), (31, 0, 1), (33, 0, 0, 5, 64), (700, 41), (40,) * 130])
def test_near_field_sizes(prec, nb, src):
    """One target cell against itself and source cells of the given sizes (empty ones among
    them), one source in the place of a target; alone and with a shifted image."""
    rng = np.random.default_rng(nb * 1000 + len(src))
    n = nb + sum(src)
    x = rng.uniform(-1, 1, (n, 3))
    x[nb] = x[0]  # coincident bodies of two cells: skipped, as r = 0 is
    q = rng.uniform(0.5, 1, n)
    if prec == "f32":
        x, q = x.astype(np.float32).astype(float), q.astype(np.float32).astype(float)
    s = fmm.Solver(P=4, precision=prec, cycle=8.0)
    s.set_bodies(x, q)
    count = np.array((nb,) + src)
    first = np.concatenate([[0], np.cumsum(count)[:-1]])
    m = len(count)
    z = np.zeros(m, int)
    s.kernel_set_cells(np.zeros((m, 3)), np.ones(m), first, count, z, z, z)
    code = 9  # image (1, 0, 0)
    ci, cj = np.zeros(m + 1, int), np.append(np.arange(m), m - 1)
    s.kernel_p2p(ci, cj, np.append(np.zeros(m, int), code))
    got = s.kernel_trg()[:nb]
    last = slice(first[-1], n)
    # the image: (xi - xj) - Xperiodic with Xperiodic = (cycle, 0, 0)
    xs = np.concatenate([x, x[last] + np.array([8.0, 0, 0])])
    ref, mag = pair_sums(x[:nb], xs, np.concatenate([q, q[last]]))
    tol = 2e-6 if prec == "f32" else 1e-13
    assert (np.abs(got[:, 0] - ref[:, 0]) <= tol * mag[:, 0]).all()
    assert (np.abs(got[:, 1:] - ref[:, 1:]).max(1) <= tol * mag[:, 1]).all()
