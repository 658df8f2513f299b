"""FP64 direct sums at the edges of the kernel's target tiles and source slices, against numpy:
each term within a few eps (2.2e-16) and sums of up to 4e4 terms, 1e-13 of the sum of magnitudes."""
import importlib

import numpy as np
import pytest

fmm = importlib.import_module("exafmm-dev_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,ns", [(1, 1), (1, 1000), (63, 255), (64, 256), (65, 257), (65, 0),
                                   (129, 40000), (1000, 2049), (37889, 300)])
@pytest.mark.parametrize("eps2", [0.0, 1e-3])
def test_direct_sizes(nt, ns, eps2):
    rng = np.random.default_rng(nt + ns)
    xt, xs, qs = rng.uniform(-1, 1, (nt, 3)), rng.uniform(-1, 1, (ns, 3)), rng.uniform(-1, 1, ns)
    if ns:
        xt[0] = xs[0]
    got = fmm.direct(xt, xs, qs, eps2)
    pick = np.unique(np.concatenate([np.arange(min(nt, 70)), np.arange(max(0, nt - 70), nt)]))
    d = xs[None] - xt[pick, None]
    r2 = (d ** 2).sum(2) + eps2
    with np.errstate(divide="ignore"):
        inv = np.where(r2 > 0, 1 / np.sqrt(r2), 0)
    ref = np.concatenate([(qs * inv).sum(1)[:, None], ((qs * inv ** 3)[..., None] * d).sum(1)], 1)
    mag = np.concatenate([np.abs(qs * inv).sum(1)[:, None],
                          np.abs((qs * inv ** 3)[..., None] * d).sum(1)], 1)
    assert (np.abs(got[pick] - ref) <= 1e-13 * mag + 1e-300).all()
    if nt <= fmm.DIRECT_NOALLOC_MAX_TARGETS and ns <= fmm.DIRECT_NOALLOC_MAX_SOURCES:
        assert np.array_equal(fmm.direct_noalloc(xt, xs, qs, eps2), got)
