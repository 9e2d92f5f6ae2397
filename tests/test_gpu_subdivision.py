"""A requested partition count whose partitions are split further for the GPU:
around the shortest partition that is split (two pieces of 16 tiles, 8 from
64-row tiles on), with a long last partition, for every tile size.  Same bar
and the caller's count reported, as for any other count."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu
MODES = {"mixed": hs.SPIKE_PRECISION_MIXED, "fp64": hs.SPIKE_PRECISION_FP64}
# k, rows per partition in tiles, p, rows beyond p equal partitions, nrhs
CASES = [(2, 32, 3, 0, 1), (2, 31, 3, 1, 2), (1, 700, 4, 3, 1), (4, 33, 5, 4, 3), (3, 900, 2, 1, 1), (8, 32, 7, 6, 1),
         (7, 200, 3, 2, 4), (16, 32, 2, 1, 1), (11, 100, 3, 0, 2), (32, 33, 2, 1, 1), (64, 16, 2, 1, 1),
         (50, 17, 3, 2, 2)]


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("case", CASES + [(100, 16, 2, 1, 1)], ids=lambda c: f"k{c[0]}_t{c[1]}_p{c[2]}_r{c[4]}")
def test_requested_partitions_are_split(case, mode):
    k, tiles, p, extra, nrhs = case
    if k > 64 and mode == "fp64":
        pytest.skip("128-row tiles: mixed precision only")
    kb = next(s for s in (2, 4, 8, 16, 32, 64, 128) if s >= k)
    n = kb * tiles * p + extra
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=7 + n, nrhs=nrhs)
    ctx = hs.Context()
    for _ in range(2):  # the second call reuses the plan
        x = hs.solve(rp, ci, a, b, precision=MODES[mode], partitions=p, ctx=ctx)
        assert ctx.info().partitions == p
        assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
        xo = oracle.spike(rp, ci, a, b, p=p)
        assert np.linalg.norm(x - xo) <= 1e-9 * np.linalg.norm(xo)
    ctx.close()
