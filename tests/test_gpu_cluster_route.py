"""Which solves one kernel takes (a thread-block cluster per instance): its launches do not grow
with the iterations, those of the loop of kernels do."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(sizes, max_iter, split=False, loop=0):
    from otmap_b200 import native as N
    from otmap_b200 import otmap as ot
    from otmap_b200 import workloads as W

    ctx = N.Context(0)
    ctx.set_loop(loop)
    if split:
        ctx.set_precision(N.PRECISION_SPLIT)
    dens = [W.to_cells(W.gaussian_mixture(n, 5 + k)) for k, n in enumerate(sizes)]
    opt = ot.SolverOptions(max_iter=max_iter, threshold=0.0)
    ot.solve_batch(dens, opt, context=ctx)  # builds what is kept
    before = ctx.launch_count()
    maps = ot.solve_batch(dens, opt, context=ctx)
    assert all(m.stats.iterations == max_iter and np.isfinite(m.fwd_mesh()).all() for m in maps)
    count = ctx.launch_count() - before
    ctx.close()
    return count


@pytest.mark.parametrize("sizes", [[n] for n in (8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 127)] +
                         [[24] * 2, [64] * 2, [24] * 7, [64] * 7, [100] * 3])
def test_one_kernel(sizes):
    # four kernels of set-up, the loop, a mesh per instance
    for max_iter in (3, 13):
        assert _launches(sizes, max_iter) == 5 + len(sizes)


@pytest.mark.parametrize("sizes,split", [([129], False), ([128], False), ([7], False), ([64], True), ([24] * 40, False),
                                         ([64] * 40, False), ([24, 25], False), ([50, 64], False)])
def test_loop_of_kernels(sizes, split):
    assert _launches(sizes, 13, split) - _launches(sizes, 3, split) >= 10


def test_host_loop():
    assert _launches([64], 13, loop=1) - _launches([64], 3, loop=1) >= 10
