"""Plain FP64 solves whose 64-row tiles are factored with digit products on the
tensor cores: bandwidths from 33 to 64 on either side, ragged last tiles, one to
many partitions (and with them the levels of the reduced system), and what the
digits' scales and the FP32 start of the tile inverse must not spoil -- rows and
columns scaled far apart, tiles too ill-conditioned for FP32, zero pivots.  The
bar is the solver's contract, a relative residual of 1e-12 in the FP64 residual
that the oracle forms; well-conditioned systems reach it without a refinement
sweep, as factors good to FP64 do."""
import numpy as np
import pytest
import scipy.sparse as sp

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


def solve(rp, ci, a, b, partitions=0):
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, precision=hs.SPIKE_PRECISION_FP64, partitions=partitions, ctx=ctx)
    info = ctx.info()
    ctx.close()
    return x, info


def times(rp, ci, a, x):
    return np.asarray(sp.csr_matrix((a, ci, rp), shape=(len(rp) - 1,) * 2) @ x)


@pytest.mark.parametrize("case", [(64, 40, 40, 1, 1), (500, 64, 64, 1, 1), (1000, 33, 64, 2, 0), (3001, 64, 33, 3, 0),
                                  (4133, 50, 41, 1, 5), (20011, 64, 64, 2, 0), (9000, 48, 64, 1, 33)],
                         ids=lambda c: f"n{c[0]}_k{c[1]}_{c[2]}_r{c[3]}_p{c[4]}")
def test_shapes(case):
    n, ku, kl, nrhs, p = case
    rp, ci, a, xt, b = hs.gen_banded(n, ku, kl, 1.5, seed=n + kl, nrhs=nrhs)
    x, info = solve(rp, ci, a, b, p)
    assert info.refine_sweeps == 0
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    assert np.linalg.norm(x - xt) <= 1e-12 * np.linalg.norm(xt)


@pytest.mark.parametrize("rows,cols", [(30, 0), (0, 30), (25, 25)])
def test_scaled_rows_and_columns(rows, cols):
    n, k = 5000, 60
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=7, nrhs=1)
    r = 2.0 ** (rows * np.sin(np.arange(n)).round())
    c = 2.0 ** (cols * np.cos(3 * np.arange(n)).round())
    i = np.repeat(np.arange(n), np.diff(rp))
    x, _ = solve(rp, ci, a * r[i] * c[ci], b * r.reshape((-1,) + (1,) * (b.ndim - 1)))
    y = x * c.reshape((-1,) + (1,) * (x.ndim - 1))
    assert np.linalg.norm(y - xt) <= 1e-12 * np.linalg.norm(xt)


@pytest.mark.parametrize("n,every", [(700, 64), (6000, 331)])
def test_tiles_beyond_fp32(n, every):
    """pairs of rows that differ by 1e-5: the pivot between them is lost in FP32"""
    k = 64
    rp, ci, a, xt, _ = hs.gen_banded(n, k, k, 1.5, seed=n, nrhs=1)
    for i in range(10, n - 1, every):
        for r in (i, i + 1):
            s = slice(rp[r], rp[r + 1])
            pair = (ci[s] == i) | (ci[s] == i + 1)
            v = a[s] * 1e-7
            v[pair] = 1.0
            a[s] = v
        a[rp[i + 1] + np.flatnonzero(ci[rp[i + 1]:rp[i + 2]] == i + 1)[0]] = 1.0 + 1e-5
    b = times(rp, ci, a, xt)
    x, _ = solve(rp, ci, a, b)
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12


def test_zero_pivot():
    n, k = 900, 64
    rp, ci, a, _, b = hs.gen_banded(n, k, k, 1.5, seed=3, nrhs=1)
    a[rp[0]:rp[1]] = 0.0
    with pytest.raises(hs.SpikeError):
        solve(rp, ci, a, b)
