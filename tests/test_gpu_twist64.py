"""Both spikes of a half together, 64-row FP32 tiles eliminated from both ends: two
partitions (one without W, one without V) and more, the fewest tiles that are
eliminated so, odd and even tile counts, ragged last tiles, narrower bands on
either side.  The bar is the solver's contract -- a relative residual of 1e-12 as
the oracle forms it -- reached in the one refinement sweep that FP32 factors need."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 3, 5])
@pytest.mark.parametrize("tiles,extra", [(8, 0), (9, 0), (9, 17), (12, -1)])
@pytest.mark.parametrize("ku,kl", [(64, 64), (40, 64), (64, 33)])
def test_both_spikes(p, tiles, extra, ku, kl):
    n = (64 * tiles + extra) * p
    rp, ci, a, xt, b = hs.gen_banded(n, ku, kl, 1.5, seed=n + ku, nrhs=2)
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, partitions=p, ctx=ctx)
    info = ctx.info()
    ctx.close()
    assert info.partitions == p and info.twisted and info.refine_sweeps <= 1
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)
