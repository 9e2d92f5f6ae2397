"""Band tiles from CSR rows: blocks inside a full band are placed by index and
their columns only compared, all others entry by entry.  The patterns sit around
that line -- full bands, a hole, rows of one length whose columns are not one run,
explicit zeros, bands narrower on one side -- for the first solve of a context
(analysed) and the next (validated while the tiles are formed, whose residual
reads no columns where the band is full).  The bar is the solver's contract: a
relative residual of 1e-12 as the oracle forms it, the exact bandwidths, and an
error for columns out of order or out of range."""
import numpy as np
import pytest
import scipy.sparse as sp

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


def system(n, ku, kl, pattern, seed):
    rp, ci, a, xt, _ = hs.gen_banded(n, ku, kl, 1.6, seed=seed, nrhs=1)
    A = sp.csr_matrix((a, ci, rp), shape=(n, n))
    if pattern == "hole":
        A[n // 2, n // 2 + 1] = 0.0
        A.eliminate_zeros()
    elif pattern == "gap":  # rows of one length, column i + 1 missing in every third
        keep = np.ones(len(ci), bool)
        for i in range(n):
            gone = i + 1 if i % 3 == 0 else i + ku
            keep[rp[i]:rp[i + 1]] &= ci[rp[i]:rp[i + 1]] != gone
        i = np.repeat(np.arange(n), np.diff(rp))
        A = sp.csr_matrix((a[keep], (i[keep], ci[keep])), shape=(n, n))
    elif pattern == "zeros":
        A.data[::7] = np.where(A.indices[::7] == np.repeat(np.arange(n), np.diff(rp))[::7], A.data[::7], 0.0)
        A.data[3] = 1e-300
    A.sort_indices()
    return A, np.asarray(A @ xt), xt


@pytest.mark.parametrize("pattern", ["full", "hole", "gap", "zeros"])
@pytest.mark.parametrize("n,ku,kl,nrhs", [(3000, 7, 8, 1), (2500, 16, 9, 2), (4003, 20, 32, 1), (5000, 64, 64, 1),
                                          (4999, 33, 60, 2), (3001, 100, 128, 1)])
def test_patterns(n, ku, kl, nrhs, pattern):
    A, b, xt = system(n, ku, kl, pattern, n + ku)
    b = np.asfortranarray(np.tile(b.reshape(n, 1), nrhs) * (1.0 + np.arange(nrhs)))
    rp, ci, a = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    ctx = hs.Context()
    for _ in range(2):
        x = hs.solve(rp, ci, a, b, ctx=ctx)
        info = ctx.info()
        assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
        i = np.repeat(np.arange(n), np.diff(rp))
        assert (info.ku, info.kl) == ((ci - i).max(), (i - ci).max())
        assert abs(info.relres_max - oracle.residual(rp, ci, a, x, b).max()) <= 1e-15
    ctx.close()


@pytest.mark.parametrize("k", [20, 64])
@pytest.mark.parametrize("fault", ["swap", "range", "twice"])
def test_columns_that_are_wrong(k, fault):
    n = 3000
    rp, ci, a, _, b = hs.gen_banded(n, k, k, 1.6, seed=5, nrhs=1)
    ctx = hs.Context()
    hs.solve(rp, ci, a, b, ctx=ctx)
    bad, t = ci.copy(), rp[n // 2] + 5
    if fault == "swap":
        bad[t], bad[t + 1] = bad[t + 1], bad[t]
    elif fault == "range":
        bad[t] = n + 17
    else:
        bad[t] = bad[t + 1]
    with pytest.raises(hs.SpikeError):
        hs.solve(rp, bad, a, b, ctx=ctx)
    x = hs.solve(rp, ci, a, b, ctx=ctx)  # the context stays usable
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    ctx.close()
