"""The sweeps' strip height (OTM_INFO_STRIP_ROWS) is the order in which the line search's sums are
formed. Lone small FP64 instances take short strips; split precision, whose FP32 fields follow the
last bit of the step, and batches of one register-transform size keep 16 rows and more."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,sizes,rows", [("fp64", (256,), 4), ("fp64", (64, 48, 33), 4), ("split", (256,), 16),
                                                  ("split", (64,), 16), ("split", (64, 48), 16), ("fp64", (64,) * 4, 16),
                                                  ("fp64", (128,) * 4, 16), ("split", (1024,), 32)])
def test_strip_rows(precision, sizes, rows):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    ctx = N.Context(0)
    ctx.set_precision(N.PRECISION_SPLIT if precision == "split" else N.PRECISION_FP64)
    dens = [W.to_cells(W.gaussian_mixture(n, k)) for k, n in enumerate(sizes)]
    ot.solve_batch(dens, ot.SolverOptions(max_iter=2), context=ctx)
    assert ctx.strip_rows() == rows
    ctx.close()
