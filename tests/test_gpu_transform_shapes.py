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


# Sizes around the steps of the block transforms: the powers of two without a register
# transform, the first and last n of each chirp length M (2n - 1 <= M), odd and even, primes and
# composites. One iteration with the fast transform takes the dense products' step: both are
# accurate to about 1e-14 of the potential, whose n/2-scaled differences (potential below 1e-2,
# n <= 2049) are the displacements.
@pytest.mark.parametrize("n", [8, 9, 16, 17, 31, 32, 33, 63, 65, 127, 129, 255, 257, 300, 499, 513, 1000, 1025, 2049])
def test_fast_transform_takes_the_dense_step(n):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    dens = W.to_cells(W.gaussian_mixture(n, n))
    opt = ot.SolverOptions(max_iter=1)
    out = []
    for mode in (N.POISSON_AUTO, N.POISSON_DENSE):
        ctx = N.Context(0)
        ctx.set_poisson(mode)
        out.append(ot.solve_batch([dens], opt, context=ctx)[0].fwd_mesh())
        if mode == N.POISSON_AUTO:  # the same instance beside others of other sizes
            more = ot.solve_batch([W.to_cells(W.gaussian_mixture(m, m)) for m in (40, 64, 100)] + [dens, dens], opt,
                                  context=ctx)
            assert np.abs(more[3].fwd_mesh() - out[0]).max() <= 1e-13
            assert np.array_equal(more[3].fwd_mesh(), more[4].fwd_mesh())
        ctx.close()
    assert np.abs(out[0] - out[1]).max() <= 1e-11
