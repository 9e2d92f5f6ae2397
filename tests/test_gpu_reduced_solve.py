"""The reduced system's solve at the edges of its schedule: one interface, the
largest system one CTA takes, one more, segments in one and in several tiers,
ragged last segments, column counts around the kernels' passes, every tile
size.  The bar is the solver's contract: relative residual <= 1e-12 in FP64,
and the generated solution within 1e-10."""
import numpy as np
import pytest

import hspike_gb300 as hs
from oracle import oracle

pytestmark = pytest.mark.gpu
MODES = {"mixed": hs.SPIKE_PRECISION_MIXED, "fp64": hs.SPIKE_PRECISION_FP64}

CASES = [
    # k, p, nrhs
    (1, 2, 1), (2, 3, 5), (2, 129, 1), (2, 130, 4), (1, 257, 3), (2, 1000, 1), (1, 20011, 2),
    (4, 129, 1), (4, 131, 6), (3, 5003, 1), (8, 129, 5), (8, 130, 1), (7, 2500, 4),
    (16, 33, 1), (16, 34, 4), (13, 700, 5), (16, 2050, 1),
    (32, 2, 1), (32, 64, 9), (20, 301, 4), (64, 2, 8), (64, 33, 1), (50, 90, 17),
]
CASES_128 = [(100, 2, 1), (128, 17, 8), (70, 40, 9)]


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"k{c[0]}_p{c[1]}_r{c[2]}")
def test_reduced_solve_schedule(case, mode):
    run(case, mode, False)


@pytest.mark.parametrize("case", CASES_128, ids=lambda c: f"k{c[0]}_p{c[1]}_r{c[2]}")
def test_reduced_solve_schedule_128(case):
    run(case, "mixed", False)


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("case", [(1, 300, 5), (3, 513, 4), (8, 70, 1), (16, 100, 3), (30, 20, 5)],
                         ids=lambda c: f"k{c[0]}_p{c[1]}_r{c[2]}")
def test_reduced_solve_schedule_complex(case, mode):
    run(case, mode, True)


def run(case, mode, cplx):
    k, p, nrhs = case
    kb = next(s for s in (2, 4, 8, 16, 32, 64, 128) if s >= k)
    n = 2 * kb * p + p // 2 + 3
    rp, ci, a, xt, b = hs.gen_banded(n, k, k, 1.5, seed=n + p, complex_=cplx, nrhs=nrhs)
    ctx = hs.Context()
    x = hs.solve(rp, ci, a, b, precision=MODES[mode], partitions=p, ctx=ctx)
    assert ctx.info().partitions == p
    assert oracle.residual(rp, ci, a, x, b).max() <= 1e-12
    assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)
    ctx.close()
