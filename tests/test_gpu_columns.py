"""Tiles of 32 to 128 rows with column counts around the passes of the retrieval
(1, 4, 8 and 16 columns) and of the reduced system's residual (one column, eight
by digit products): every type, ragged last tiles, columns of very different
sizes and a zero one.  The bar is the solver's contract per column: a relative
residual of 1e-12 as the oracle forms it; the zero column stays zero."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu
MODES = {"mixed": hs.SPIKE_PRECISION_MIXED, "fp64": hs.SPIKE_PRECISION_FP64}
CASES = [(k, nrhs, "mixed", False) for k in (24, 64, 100) for nrhs in (1, 2, 4, 5, 8, 9, 16, 19)]
CASES += [(64, nrhs, "fp64", False) for nrhs in (1, 3, 6)] + [(50, nrhs, "mixed", True) for nrhs in (1, 3, 6)]


@pytest.mark.parametrize("k,nrhs,mode,cplx", CASES)
def test_columns(k, nrhs, mode, cplx):
    kb = next(s for s in (32, 64, 128) if s >= k)
    n, p = 2 * kb * 7 + 5 * kb // 3, 7
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=n + nrhs, complex_=cplx, nrhs=nrhs)
    f = 10.0 ** (7.0 * (np.arange(nrhs) % 8) - 20.0)  # within the factor precision's range
    if nrhs > 2:
        f[nrhs // 2] = 0.0
    b = np.asfortranarray(b.reshape(n, nrhs, order="F") * f)
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, precision=MODES[mode], partitions=p, ctx=ctx).reshape(n, nrhs, order="F")
    ctx.close()
    live = f != 0.0
    assert oracle.residual(rp, ci, a, np.asfortranarray(x[:, live]), np.asfortranarray(b[:, live])).max() <= 1e-12
    assert not x[:, ~live].any()
