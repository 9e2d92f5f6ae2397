"""The FP64 residual of full bands with several columns (digit products on the
tensor cores): row and column counts around its tiles, ku != kl, every band
class, and the systems its scales must not spoil -- solutions that decay across
the band, columns scaled far apart, zero columns.  The solve refines with that
residual, so its error shows in the residual the oracle forms."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu
MODES = {"mixed": hs.SPIKE_PRECISION_MIXED, "fp64": hs.SPIKE_PRECISION_FP64}


def solve(rp, ci, a, b, mode):
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, precision=MODES[mode], ctx=ctx)
    info = ctx.info()
    ctx.close()
    return x, info


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("case", [(4096, 64, 64, 8), (4097, 64, 64, 9), (4159, 64, 33, 16), (6000, 12, 12, 2),
                                  (6001, 13, 12, 3), (5003, 24, 40, 17), (3000, 32, 32, 65), (70, 16, 16, 2),
                                  (2050, 50, 1, 4)], ids=lambda c: f"n{c[0]}_k{c[1]}_{c[2]}_r{c[3]}")
def test_shapes(case, mode):
    shapes(case, mode)


def shapes(case, mode):
    n, ku, kl, nrhs = case
    rp, ci, a, xt, b = hs.gen_banded(n, ku, kl, 1.5, seed=n + ku, nrhs=nrhs)
    x, info = solve(rp, ci, a, b, mode)
    true = oracle.residual(rp, ci, a, x, b)
    assert true.max() <= 1e-12
    # the reported residual is the true one, up to what FP64 sums of |A||x| round
    assert abs(info.relres_max - true.max()) <= 1e-15
    assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)


@pytest.mark.parametrize("case", [(9000, 100, 100, 8), (5000, 128, 128, 5), (4000, 65, 128, 2)],
                         ids=lambda c: f"n{c[0]}_k{c[1]}_{c[2]}_r{c[3]}")
def test_shapes_128(case):
    shapes(case, "mixed")


@pytest.mark.parametrize("k,dom", [(16, 1.5), (40, 3.0), (64, 1e4)])
def test_decaying_solutions(k, dom):
    n, nrhs = 3000, 4
    rp, ci, a, _, _ = hs.gen_banded(n, k, k, dom, seed=k, nrhs=1)
    b = np.zeros((n, nrhs), order="F")
    for h in range(nrhs):
        b[h * (n // nrhs) + 17, h] = 1.0  # unit vectors: x falls off on both sides, to nothing
    x, _ = solve(rp, ci, a, b, "mixed")
    xo = oracle.spike(rp, ci, a, b, p=4)
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    # entry by entry, within 2^-20 of each over thirty orders of magnitude
    big = np.abs(xo) > 1e-30
    assert (np.abs(x - xo)[big] / np.abs(xo)[big]).max() <= 2.0 ** -20


@pytest.mark.parametrize("k", [16, 64])
def test_columns_scaled_far_apart(k):
    n, nrhs = 2500, 5
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=k + 1, nrhs=nrhs)
    s = np.where(np.arange(n) % 2 == 0, 2.0 ** 24, 2.0 ** -24)
    x, _ = solve(rp, ci, a * s[ci], b, "fp64")  # the solution is xt / s
    assert np.linalg.norm(x * s[:, None] - xt) <= 1e-12 * np.linalg.norm(xt)


def test_zero_and_tiny_columns():
    n, k = 2000, 32
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=9, nrhs=4)
    b[:, 1] = 0.0
    b[:, 2] *= 1e-200
    x, _ = solve(rp, ci, a, b, "mixed")
    assert not x[:, 1].any()
    for h, f in ((0, 1.0), (3, 1.0)):
        assert np.linalg.norm(x[:, h] - f * xt[:, h]) <= 1e-10 * np.linalg.norm(xt[:, h])
