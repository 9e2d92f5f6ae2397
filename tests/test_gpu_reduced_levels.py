"""Factorization of the reduced system of FP32 tiles of 32, 64 and 128 rows: one
interface, level sizes on both sides of the split into finer column slices,
odd and even block counts, and a zero pivot.  The bar is the solver's
contract: a relative residual of 1e-12 as the oracle forms it, and the generated
solution within 1e-10."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,ps", [(24, (2, 3, 20, 311)), (60, (2, 4, 78, 79, 157)), (100, (2, 3, 6, 39, 42, 90)),
                                  (128, (5, 41))])
def test_levels(k, ps):
    kb = next(s for s in (32, 64, 128) if s >= k)
    for p in ps:
        n = 2 * kb * p + p // 3 + 1
        rp, ci, a, xt, b = hs.gen_banded(n, k, k - 3, 1.5, seed=n + p, nrhs=1)
        ctx = hs.Context()
        x = hs.solve(rp, ci, a, b, partitions=p, ctx=ctx)
        assert ctx.info().partitions == p
        assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
        assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)
        ctx.close()


@pytest.mark.parametrize("k", [24, 64, 128])
def test_singular(k):
    n = 6 * k * 4
    rp, ci, a, _, b = hs.gen_banded(n, k, k, 1.5, seed=k, nrhs=1)
    a[rp[n // 2]:rp[n // 2 + 1]] = 0.0
    with pytest.raises(hs.SpikeError):
        hs.solve(rp, ci, a, b)
