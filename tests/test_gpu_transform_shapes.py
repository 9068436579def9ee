"""The cosine transforms' launch shapes: a lone instance spreads its rows and columns over the
SMs in narrow blocks (1 to 8 warps), a large batch takes full ones. The arithmetic of a line
does not depend on the block, so one iteration of a density gives the same step alone, in a
small batch and in a batch large enough for full blocks, up to the order of the line search's
sums (1e-13 relative for n^2 <= 2^20 terms of one sign; displacements are below 1)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("n,counts", [(64, (1, 5, 160)), (128, (1, 3, 40)), (256, (1, 4, 20)), (512, (1, 3, 6)),
                                      (1024, (1, 2, 3))])
def test_step_does_not_depend_on_block_shape(n, counts, precision):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    ctx = N.Context(0)
    ctx.set_precision(N.PRECISION_SPLIT if precision == "split" else N.PRECISION_FP64)
    dens = [W.to_cells(W.gaussian_mixture(n, 40 + k)) for k in range(2)]
    opt = ot.SolverOptions(max_iter=1)
    ref = None
    for count in counts:
        maps = ot.solve_batch([dens[k % 2] for k in range(count)], opt, context=ctx)
        if ref is None:
            ref = [maps[0], ot.solve_batch([dens[1]], opt, context=ctx)[0]]
        for k, m in enumerate(maps):
            assert m.stats.iterations == 1
            assert np.abs(m.fwd_mesh() - ref[k % 2].fwd_mesh()).max() <= 1e-13
    ctx.close()
