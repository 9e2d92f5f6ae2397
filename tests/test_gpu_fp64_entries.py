"""Plain FP64 with 64-row tiles, entry by entry.

A decaying solution (unit right-hand sides, strong dominance, bands that fill a
tile in part) has entries far below the scales of their tile's rows and columns;
each must come out as a chain of FP64 multiply-adds gives it, not with an error
measured by its neighbours.  The reference is the solution refined in extended
precision, whose Jacobi sweeps contract every entry.  An entry sums terms of
rounding 2^-53 over some tens of steps, and one in a hundred may cancel by two
digits and more: half of the entries within 2^-44, 99 % within 2^-36."""
import numpy as np
import pytest

import hspike_gb300 as hs

pytestmark = pytest.mark.gpu


def extended(rp, ci, a, b, ku, kl, x):
    """x refined entry by entry in extended precision"""
    n, w = len(rp) - 1, kl + ku + 1
    band = np.zeros((n, w), np.longdouble)
    r = np.repeat(np.arange(n), np.diff(rp))
    band[r, ci - r + kl] = a
    diag = band[:, kl].copy()
    band[:, kl] = 0
    x, rhs = x.astype(np.longdouble), b.astype(np.longdouble)
    for _ in range(200):
        pad = np.zeros((n + w, x.shape[1]), np.longdouble)
        pad[kl:kl + n] = x
        y = rhs.copy()
        for j in range(w):
            y -= band[:, j, None] * pad[j:j + n]
        y /= diag[:, None]
        step = np.abs(y - x) / np.maximum(np.abs(y), np.longdouble(1e-290))
        x = y
        if step.max() < 1e-17:
            return x
    raise AssertionError("the reference did not settle")


@pytest.mark.parametrize("p", [1, 4])
@pytest.mark.parametrize("ku,kl", [(64, 64), (40, 40), (64, 35), (33, 60)])
@pytest.mark.parametrize("dom", [1.5, 10.0, 1e4])
def test_small_entries(ku, kl, dom, p):
    n = 1000
    rp, ci, a, _, b0 = hs.gen_banded(n, ku, kl, dom, seed=ku + kl, nrhs=1)
    b = np.zeros((n, 3), order="F")
    b[:, 0] = b0.reshape(-1)
    b[90, 1] = 1.0
    b[n - 17, 2] = 1.0
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, precision=hs.SPIKE_PRECISION_FP64, partitions=p, ctx=ctx)
    ctx.close()
    xe = extended(rp, ci, a, b, ku, kl, x)
    for h in range(3):
        live = np.abs(xe[:, h]) > 1e-250
        err = np.abs(x[live, h] - xe[live, h]) / np.abs(xe[live, h])
        assert np.median(err) <= 2.0 ** -44
        assert np.quantile(err, 0.99) <= 2.0 ** -36
