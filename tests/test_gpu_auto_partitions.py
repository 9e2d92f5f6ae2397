"""Automatic partition counts of tiles of 32 rows and more at sizes that do not fill
the GPU: one and two tiles, around the counts 2^L + 1, and on both sides of the
size from which every SM has its chains.  The bar is the solver's contract: a
relative residual of 1e-12 as the oracle forms it."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,kb,fill", [(24, 32, 304 * 8 * 32), (64, 64, 304 * 8 * 64), (100, 128, 152 * 4 * 128)])
@pytest.mark.parametrize("mode", [hs.SPIKE_PRECISION_MIXED, hs.SPIKE_PRECISION_FP64])
def test_sizes(k, kb, fill, mode):
    if kb == 128 and mode == hs.SPIKE_PRECISION_FP64:
        pytest.skip("FP64 tiles have up to 64 rows")
    for n in (kb - 1, 2 * kb, 4 * kb - 1, 4 * kb + 1, 9 * kb, 37 * kb + 5, 130 * kb - 3) + ((fill - 1, fill) if k == 24 else ()):
        rp, ci, a, xt, b = hs.gen_banded(n, min(k, n - 1), min(k, n - 1), 1.5, seed=n, nrhs=2)
        ctx = hs.Context()
        x = hs.solve(rp, ci, a, b, precision=mode, ctx=ctx)
        assert ctx.info().partitions <= max(1, n // (2 * kb))
        ctx.close()
        assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
