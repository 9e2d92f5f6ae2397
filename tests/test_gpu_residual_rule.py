"""Which FP64 residual runs, and the smallest systems of the one on the tensor
cores: bands cut by both ends of the matrix, fewer rows than a tile, and right-
hand sides far below one.  The digit products take full bands of three columns
and more with 112 multiply-adds a row and pass of eight columns; above eight
columns they launch once per eight where the other kernel launches once."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


def solve(rp, ci, a, b, precision=hs.SPIKE_PRECISION_MIXED):
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, precision=precision, ctx=ctx)
    info = ctx.info()
    ctx.close()
    return x, info


def launches(ku, kl, nrhs, drop=False):
    """kernel launches of a solve, and its relative residual; `drop` leaves one entry of the band out"""
    n = 3000
    rp, ci, a, _, b = hs.gen_banded(n, ku, kl, 1.5, seed=3, nrhs=nrhs)
    if drop:
        t = rp[1500]  # the row's first entry, below the diagonal
        rp = rp.copy()
        rp[1501:] -= 1
        ci, a = np.delete(ci, t), np.delete(a, t)
    x, info = solve(rp, ci, a, b)
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    return info.kernel_launches, info.refine_sweeps


@pytest.mark.parametrize("ku,kl,nrhs,digits", [(12, 12, 9, True), (12, 11, 9, False), (6, 7, 16, True),
                                               (6, 6, 16, False)] +
                         [(9, 9, 17, False), (12, 12, 17, True), (20, 19, 17, True), (64, 64, 9, True), (100, 90, 9, True)])
def test_rule(ku, kl, nrhs, digits):
    full, sweeps = launches(ku, kl, nrhs)
    sparse, sweeps1 = launches(ku, kl, nrhs, drop=True)  # not a full band: never by digits
    assert sweeps == sweeps1
    passes = -(-nrhs // 8)
    assert full - sparse == ((sweeps + 1) * (passes - 1) if digits else 0)


@pytest.mark.parametrize("n,ku,kl,nrhs", [(20, 19, 19, 8), (33, 32, 32, 3), (70, 16, 16, 4), (64, 63, 40, 5),
                                          (65, 40, 64, 3), (129, 128, 128, 3), (130, 128, 60, 9), (31, 18, 30, 8)])
@pytest.mark.parametrize("mode", [hs.SPIKE_PRECISION_MIXED, hs.SPIKE_PRECISION_FP64])
def test_systems_of_a_tile_or_two(n, ku, kl, nrhs, mode):
    if max(ku, kl) > 64 and mode == hs.SPIKE_PRECISION_FP64:
        pytest.skip("128-row tiles: mixed precision only")
    assert nrhs * (ku + kl + 1) >= 112 * -(-nrhs // 8)
    rp, ci, a, xt, b = hs.gen_banded(n, ku, kl, 1.5, seed=n, nrhs=nrhs)
    x, info = solve(rp, ci, a, b, mode)
    true = oracle.residual(rp, ci, a, x, b).max()
    assert true <= 1e-12
    assert abs(info.relres_max - true) <= 1e-15
    assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)


@pytest.mark.parametrize("mode,f,bar", [(hs.SPIKE_PRECISION_MIXED, 1e-25, 1e-10), (hs.SPIKE_PRECISION_FP64, 1e-25, 1e-12),
                                        (hs.SPIKE_PRECISION_FP64, 1e-200, 1e-12)])
def test_a_tiny_column(mode, f, bar):
    rp, ci, a, xt, b = hs.gen_banded(2000, 32, 32, 1.5, seed=9, nrhs=4)
    b[:, 1] = 0.0
    b[:, 2] *= f
    x, _ = solve(rp, ci, a, b, mode)
    assert not x[:, 1].any()
    for h, s in ((0, 1.0), (2, f), (3, 1.0)):
        assert np.linalg.norm(x[:, h] / s - xt[:, h]) <= bar * np.linalg.norm(xt[:, h])


@pytest.mark.parametrize("n,k,nrhs", [(70_001, 64, 16), (70_000, 24, 5), (40_033, 100, 8), (20_000, 40, 3)])
@pytest.mark.parametrize("every", [1, 40, 400])
def test_localized_sources(n, k, nrhs, every):
    """solutions that fall off between their sources: few, many or nearly all results
    of a tile outside the digits' scales (the larger systems give every CTA several
    tiles, which after such a one go without digits), entry by entry within what
    FP32 factors refined once or more leave (2^-20)"""
    rp, ci, a, _, _ = hs.gen_banded(n, k, k, 20.0, seed=k, nrhs=1)
    b = np.zeros((n, nrhs), order="F")
    for h in range(nrhs):
        b[h * 31 % every::every, h] = 1.0
    x, _ = solve(rp, ci, a, b)
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    xo = oracle.spike(rp, ci, a, b, p=4)
    big = np.abs(xo) > 1e-30
    assert np.quantile(np.abs(x - xo)[big] / np.abs(xo)[big], 0.999) <= 2.0 ** -20
