"""Requested partition counts on the device: exactly p on request, and a split
count on the pipelined path of a repeated call with host arrays."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [hs.SPIKE_PRECISION_MIXED, hs.SPIKE_PRECISION_FP64])
@pytest.mark.parametrize("n,k,p", [(20001, 2, 4), (30000, 12, 3), (60000, 40, 5)])
def test_exact_and_split_counts(n, k, p, mode):
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 2.0, seed=n + k, nrhs=2)
    held = {}
    for split in (1, 0):
        ctx = hs.Context()
        ctx.set_option(hs.SPIKE_OPT_SPLIT_PARTITIONS, split)
        x = hs.solve(rp, ci, a, b, precision=mode, partitions=p, ctx=ctx)
        info = ctx.info()
        ctx.close()
        assert info.partitions == p
        assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
        assert np.linalg.norm(x - xt) <= 1e-11 * np.linalg.norm(xt)
        held[split] = info.device_bytes
    assert held[0] < held[1]  # the pieces' interfaces


def test_split_count_on_the_pipelined_path():
    n, k, p = 140_000, 32, 8  # above the path's entry count; 8 partitions in 34 pieces each
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=5, nrhs=1)
    ctx = hs.Context()
    for call in range(3):  # the first builds the plan, the others take the values range by range
        ac = a * (1.0 + call)
        x = hs.solve(rp, ci, ac, b, partitions=p, ctx=ctx)
        info = ctx.info()
        assert info.partitions == p
        assert bool(info.columns_implied) == (call > 0)
        assert oracle.residual(rp, ci, ac, x, b).max() <= 1e-12
        assert np.linalg.norm(x * (1.0 + call) - xt) <= 1e-10 * np.linalg.norm(xt)
    ctx.close()
